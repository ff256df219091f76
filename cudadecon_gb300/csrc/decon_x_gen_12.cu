// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 192, 324, 504, 750, 1050, 1458, 1960.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_12(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 192:
      *done = true;
      return px_fwd_go<PPX192, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 324:
      *done = true;
      return px_fwd_go<PPX324, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 504:
      *done = true;
      return px_fwd_go<PPX504, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 750:
      *done = true;
      return px_fwd_go<PPX750, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1050:
      *done = true;
      return px_fwd_go<PPX1050, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1458:
      *done = true;
      return px_fwd_go<PPX1458, 4>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1960:
      *done = true;
      return px_fwd_go<PPX1960, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_12(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 192:
      *done = true;
      return px_ratio_go<PPX192, 2>(g, tw, S, raw, mean, eps, st);
    case 324:
      *done = true;
      return px_ratio_go<PPX324, 2>(g, tw, S, raw, mean, eps, st);
    case 504:
      *done = true;
      return px_ratio_go<PPX504, 2>(g, tw, S, raw, mean, eps, st);
    case 750:
      *done = true;
      return px_ratio_go<PPX750, 2>(g, tw, S, raw, mean, eps, st);
    case 1050:
      *done = true;
      return px_ratio_go<PPX1050, 2>(g, tw, S, raw, mean, eps, st);
    case 1458:
      *done = true;
      return px_ratio_go<PPX1458, 4>(g, tw, S, raw, mean, eps, st);
    case 1960:
      *done = true;
      return px_ratio_go<PPX1960, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_12(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 192:
      *done = true;
      return px_update_go<PPX192, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 324:
      *done = true;
      return px_update_go<PPX324, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 504:
      *done = true;
      return px_update_go<PPX504, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 750:
      *done = true;
      return px_update_go<PPX750, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1050:
      *done = true;
      return px_update_go<PPX1050, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1458:
      *done = true;
      return px_update_go<PPX1458, 4>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1960:
      *done = true;
      return px_update_go<PPX1960, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
