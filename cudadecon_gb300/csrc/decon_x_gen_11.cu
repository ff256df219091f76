// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 189, 320, 500, 735, 1029, 1440, 1944.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_11(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 189:
      *done = true;
      return px_fwd_go<PPX189, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 320:
      *done = true;
      return px_fwd_go<PPX320, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 500:
      *done = true;
      return px_fwd_go<PPX500, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 735:
      *done = true;
      return px_fwd_go<PPX735, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1029:
      *done = true;
      return px_fwd_go<PPX1029, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1440:
      *done = true;
      return px_fwd_go<PPX1440, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1944:
      *done = true;
      return px_fwd_go<PPX1944, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_11(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 189:
      *done = true;
      return px_ratio_go<PPX189, 2>(g, tw, S, raw, mean, eps, st);
    case 320:
      *done = true;
      return px_ratio_go<PPX320, 2>(g, tw, S, raw, mean, eps, st);
    case 500:
      *done = true;
      return px_ratio_go<PPX500, 2>(g, tw, S, raw, mean, eps, st);
    case 735:
      *done = true;
      return px_ratio_go<PPX735, 2>(g, tw, S, raw, mean, eps, st);
    case 1029:
      *done = true;
      return px_ratio_go<PPX1029, 2>(g, tw, S, raw, mean, eps, st);
    case 1440:
      *done = true;
      return px_ratio_go<PPX1440, 2>(g, tw, S, raw, mean, eps, st);
    case 1944:
      *done = true;
      return px_ratio_go<PPX1944, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_11(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 189:
      *done = true;
      return px_update_go<PPX189, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 320:
      *done = true;
      return px_update_go<PPX320, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 500:
      *done = true;
      return px_update_go<PPX500, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 735:
      *done = true;
      return px_update_go<PPX735, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1029:
      *done = true;
      return px_update_go<PPX1029, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1440:
      *done = true;
      return px_update_go<PPX1440, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1944:
      *done = true;
      return px_update_go<PPX1944, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
