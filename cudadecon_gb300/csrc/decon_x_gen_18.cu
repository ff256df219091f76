// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 225, 378, 576, 840, 1176, 1575.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_18(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 225:
      *done = true;
      return px_fwd_go<PPX225, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 378:
      *done = true;
      return px_fwd_go<PPX378, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 576:
      *done = true;
      return px_fwd_go<PPX576, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 840:
      *done = true;
      return px_fwd_go<PPX840, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1176:
      *done = true;
      return px_fwd_go<PPX1176, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1575:
      *done = true;
      return px_fwd_go<PPX1575, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_18(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 225:
      *done = true;
      return px_ratio_go<PPX225, 2>(g, tw, S, raw, mean, eps, st);
    case 378:
      *done = true;
      return px_ratio_go<PPX378, 2>(g, tw, S, raw, mean, eps, st);
    case 576:
      *done = true;
      return px_ratio_go<PPX576, 2>(g, tw, S, raw, mean, eps, st);
    case 840:
      *done = true;
      return px_ratio_go<PPX840, 2>(g, tw, S, raw, mean, eps, st);
    case 1176:
      *done = true;
      return px_ratio_go<PPX1176, 2>(g, tw, S, raw, mean, eps, st);
    case 1575:
      *done = true;
      return px_ratio_go<PPX1575, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_18(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 225:
      *done = true;
      return px_update_go<PPX225, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 378:
      *done = true;
      return px_update_go<PPX378, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 576:
      *done = true;
      return px_update_go<PPX576, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 840:
      *done = true;
      return px_update_go<PPX840, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1176:
      *done = true;
      return px_update_go<PPX1176, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1575:
      *done = true;
      return px_update_go<PPX1575, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
