// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 147, 256, 432, 648, 945, 1280, 1750.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_4(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 147:
      *done = true;
      return px_fwd_go<PPX147, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 256:
      *done = true;
      return px_fwd_go<PPX256, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 432:
      *done = true;
      return px_fwd_go<PPX432, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 648:
      *done = true;
      return px_fwd_go<PPX648, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 945:
      *done = true;
      return px_fwd_go<PPX945, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1280:
      *done = true;
      return px_fwd_go<PPX1280, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1750:
      *done = true;
      return px_fwd_go<PPX1750, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_4(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 147:
      *done = true;
      return px_ratio_go<PPX147, 2>(g, tw, S, raw, mean, eps, st);
    case 256:
      *done = true;
      return px_ratio_go<PPX256, 2>(g, tw, S, raw, mean, eps, st);
    case 432:
      *done = true;
      return px_ratio_go<PPX432, 2>(g, tw, S, raw, mean, eps, st);
    case 648:
      *done = true;
      return px_ratio_go<PPX648, 2>(g, tw, S, raw, mean, eps, st);
    case 945:
      *done = true;
      return px_ratio_go<PPX945, 2>(g, tw, S, raw, mean, eps, st);
    case 1280:
      *done = true;
      return px_ratio_go<PPX1280, 2>(g, tw, S, raw, mean, eps, st);
    case 1750:
      *done = true;
      return px_ratio_go<PPX1750, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_4(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 147:
      *done = true;
      return px_update_go<PPX147, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 256:
      *done = true;
      return px_update_go<PPX256, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 432:
      *done = true;
      return px_update_go<PPX432, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 648:
      *done = true;
      return px_update_go<PPX648, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 945:
      *done = true;
      return px_update_go<PPX945, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1280:
      *done = true;
      return px_update_go<PPX1280, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1750:
      *done = true;
      return px_update_go<PPX1750, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
