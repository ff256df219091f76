// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 162, 288, 450, 686, 980, 1344, 1800.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_7(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 162:
      *done = true;
      return px_fwd_go<PPX162, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 288:
      *done = true;
      return px_fwd_go<PPX288, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 450:
      *done = true;
      return px_fwd_go<PPX450, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 686:
      *done = true;
      return px_fwd_go<PPX686, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 980:
      *done = true;
      return px_fwd_go<PPX980, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1344:
      *done = true;
      return px_fwd_go<PPX1344, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1800:
      *done = true;
      return px_fwd_go<PPX1800, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_7(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 162:
      *done = true;
      return px_ratio_go<PPX162, 2>(g, tw, S, raw, mean, eps, st);
    case 288:
      *done = true;
      return px_ratio_go<PPX288, 2>(g, tw, S, raw, mean, eps, st);
    case 450:
      *done = true;
      return px_ratio_go<PPX450, 2>(g, tw, S, raw, mean, eps, st);
    case 686:
      *done = true;
      return px_ratio_go<PPX686, 2>(g, tw, S, raw, mean, eps, st);
    case 980:
      *done = true;
      return px_ratio_go<PPX980, 2>(g, tw, S, raw, mean, eps, st);
    case 1344:
      *done = true;
      return px_ratio_go<PPX1344, 2>(g, tw, S, raw, mean, eps, st);
    case 1800:
      *done = true;
      return px_ratio_go<PPX1800, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_7(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 162:
      *done = true;
      return px_update_go<PPX162, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 288:
      *done = true;
      return px_update_go<PPX288, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 450:
      *done = true;
      return px_update_go<PPX450, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 686:
      *done = true;
      return px_update_go<PPX686, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 980:
      *done = true;
      return px_update_go<PPX980, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1344:
      *done = true;
      return px_update_go<PPX1344, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1800:
      *done = true;
      return px_update_go<PPX1800, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
