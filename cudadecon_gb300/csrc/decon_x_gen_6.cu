// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 160, 280, 448, 675, 972, 1323, 1792.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_6(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 160:
      *done = true;
      return px_fwd_go<PPX160, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 280:
      *done = true;
      return px_fwd_go<PPX280, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 448:
      *done = true;
      return px_fwd_go<PPX448, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 675:
      *done = true;
      return px_fwd_go<PPX675, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 972:
      *done = true;
      return px_fwd_go<PPX972, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1323:
      *done = true;
      return px_fwd_go<PPX1323, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1792:
      *done = true;
      return px_fwd_go<PPX1792, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_6(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 160:
      *done = true;
      return px_ratio_go<PPX160, 2>(g, tw, S, raw, mean, eps, st);
    case 280:
      *done = true;
      return px_ratio_go<PPX280, 2>(g, tw, S, raw, mean, eps, st);
    case 448:
      *done = true;
      return px_ratio_go<PPX448, 2>(g, tw, S, raw, mean, eps, st);
    case 675:
      *done = true;
      return px_ratio_go<PPX675, 2>(g, tw, S, raw, mean, eps, st);
    case 972:
      *done = true;
      return px_ratio_go<PPX972, 2>(g, tw, S, raw, mean, eps, st);
    case 1323:
      *done = true;
      return px_ratio_go<PPX1323, 2>(g, tw, S, raw, mean, eps, st);
    case 1792:
      *done = true;
      return px_ratio_go<PPX1792, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_6(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 160:
      *done = true;
      return px_update_go<PPX160, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 280:
      *done = true;
      return px_update_go<PPX280, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 448:
      *done = true;
      return px_update_go<PPX448, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 675:
      *done = true;
      return px_update_go<PPX675, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 972:
      *done = true;
      return px_update_go<PPX972, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1323:
      *done = true;
      return px_update_go<PPX1323, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1792:
      *done = true;
      return px_update_go<PPX1792, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
