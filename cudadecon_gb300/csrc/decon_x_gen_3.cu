// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 144, 252, 420, 640, 900, 1260, 1728.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_3(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 144:
      *done = true;
      return px_fwd_go<PPX144, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 252:
      *done = true;
      return px_fwd_go<PPX252, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 420:
      *done = true;
      return px_fwd_go<PPX420, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 640:
      *done = true;
      return px_fwd_go<PPX640, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 900:
      *done = true;
      return px_fwd_go<PPX900, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1260:
      *done = true;
      return px_fwd_go<PPX1260, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1728:
      *done = true;
      return px_fwd_go<PPX1728, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_3(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 144:
      *done = true;
      return px_ratio_go<PPX144, 2>(g, tw, S, raw, mean, eps, st);
    case 252:
      *done = true;
      return px_ratio_go<PPX252, 2>(g, tw, S, raw, mean, eps, st);
    case 420:
      *done = true;
      return px_ratio_go<PPX420, 2>(g, tw, S, raw, mean, eps, st);
    case 640:
      *done = true;
      return px_ratio_go<PPX640, 2>(g, tw, S, raw, mean, eps, st);
    case 900:
      *done = true;
      return px_ratio_go<PPX900, 2>(g, tw, S, raw, mean, eps, st);
    case 1260:
      *done = true;
      return px_ratio_go<PPX1260, 2>(g, tw, S, raw, mean, eps, st);
    case 1728:
      *done = true;
      return px_ratio_go<PPX1728, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_3(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 144:
      *done = true;
      return px_update_go<PPX144, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 252:
      *done = true;
      return px_update_go<PPX252, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 420:
      *done = true;
      return px_update_go<PPX420, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 640:
      *done = true;
      return px_update_go<PPX640, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 900:
      *done = true;
      return px_update_go<PPX900, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1260:
      *done = true;
      return px_update_go<PPX1260, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1728:
      *done = true;
      return px_update_go<PPX1728, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
