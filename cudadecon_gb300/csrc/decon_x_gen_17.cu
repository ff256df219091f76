// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 224, 375, 567, 810, 1152, 1568.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_17(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 224:
      *done = true;
      return px_fwd_go<PPX224, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 375:
      *done = true;
      return px_fwd_go<PPX375, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 567:
      *done = true;
      return px_fwd_go<PPX567, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 810:
      *done = true;
      return px_fwd_go<PPX810, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1152:
      *done = true;
      return px_fwd_go<PPX1152, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1568:
      *done = true;
      return px_fwd_go<PPX1568, 4>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_17(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 224:
      *done = true;
      return px_ratio_go<PPX224, 2>(g, tw, S, raw, mean, eps, st);
    case 375:
      *done = true;
      return px_ratio_go<PPX375, 2>(g, tw, S, raw, mean, eps, st);
    case 567:
      *done = true;
      return px_ratio_go<PPX567, 2>(g, tw, S, raw, mean, eps, st);
    case 810:
      *done = true;
      return px_ratio_go<PPX810, 2>(g, tw, S, raw, mean, eps, st);
    case 1152:
      *done = true;
      return px_ratio_go<PPX1152, 2>(g, tw, S, raw, mean, eps, st);
    case 1568:
      *done = true;
      return px_ratio_go<PPX1568, 4>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_17(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 224:
      *done = true;
      return px_update_go<PPX224, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 375:
      *done = true;
      return px_update_go<PPX375, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 567:
      *done = true;
      return px_update_go<PPX567, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 810:
      *done = true;
      return px_update_go<PPX810, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1152:
      *done = true;
      return px_update_go<PPX1152, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1568:
      *done = true;
      return px_update_go<PPX1568, 4>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
