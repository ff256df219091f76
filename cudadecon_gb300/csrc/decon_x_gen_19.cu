// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 240, 384, 588, 864, 1200, 1600.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_19(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 240:
      *done = true;
      return px_fwd_go<PPX240, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 384:
      *done = true;
      return px_fwd_go<PPX384, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 588:
      *done = true;
      return px_fwd_go<PPX588, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 864:
      *done = true;
      return px_fwd_go<PPX864, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1200:
      *done = true;
      return px_fwd_go<PPX1200, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1600:
      *done = true;
      return px_fwd_go<PPX1600, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_19(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 240:
      *done = true;
      return px_ratio_go<PPX240, 2>(g, tw, S, raw, mean, eps, st);
    case 384:
      *done = true;
      return px_ratio_go<PPX384, 2>(g, tw, S, raw, mean, eps, st);
    case 588:
      *done = true;
      return px_ratio_go<PPX588, 2>(g, tw, S, raw, mean, eps, st);
    case 864:
      *done = true;
      return px_ratio_go<PPX864, 2>(g, tw, S, raw, mean, eps, st);
    case 1200:
      *done = true;
      return px_ratio_go<PPX1200, 2>(g, tw, S, raw, mean, eps, st);
    case 1600:
      *done = true;
      return px_ratio_go<PPX1600, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_19(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 240:
      *done = true;
      return px_update_go<PPX240, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 384:
      *done = true;
      return px_update_go<PPX384, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 588:
      *done = true;
      return px_update_go<PPX588, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 864:
      *done = true;
      return px_update_go<PPX864, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1200:
      *done = true;
      return px_update_go<PPX1200, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1600:
      *done = true;
      return px_update_go<PPX1600, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
