// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 210, 350, 540, 784, 1125, 1512, 2025.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_15(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 210:
      *done = true;
      return px_fwd_go<PPX210, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 350:
      *done = true;
      return px_fwd_go<PPX350, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 540:
      *done = true;
      return px_fwd_go<PPX540, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 784:
      *done = true;
      return px_fwd_go<PPX784, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1125:
      *done = true;
      return px_fwd_go<PPX1125, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1512:
      *done = true;
      return px_fwd_go<PPX1512, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 2025:
      *done = true;
      return px_fwd_go<PPX2025, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_15(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 210:
      *done = true;
      return px_ratio_go<PPX210, 2>(g, tw, S, raw, mean, eps, st);
    case 350:
      *done = true;
      return px_ratio_go<PPX350, 2>(g, tw, S, raw, mean, eps, st);
    case 540:
      *done = true;
      return px_ratio_go<PPX540, 2>(g, tw, S, raw, mean, eps, st);
    case 784:
      *done = true;
      return px_ratio_go<PPX784, 2>(g, tw, S, raw, mean, eps, st);
    case 1125:
      *done = true;
      return px_ratio_go<PPX1125, 2>(g, tw, S, raw, mean, eps, st);
    case 1512:
      *done = true;
      return px_ratio_go<PPX1512, 2>(g, tw, S, raw, mean, eps, st);
    case 2025:
      *done = true;
      return px_ratio_go<PPX2025, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_15(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 210:
      *done = true;
      return px_update_go<PPX210, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 350:
      *done = true;
      return px_update_go<PPX350, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 540:
      *done = true;
      return px_update_go<PPX540, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 784:
      *done = true;
      return px_update_go<PPX784, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1125:
      *done = true;
      return px_update_go<PPX1125, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1512:
      *done = true;
      return px_update_go<PPX1512, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 2025:
      *done = true;
      return px_update_go<PPX2025, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
