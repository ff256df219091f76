// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 216, 360, 560, 800, 1134, 1536, 2048.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_16(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 216:
      *done = true;
      return px_fwd_go<PPX216, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 360:
      *done = true;
      return px_fwd_go<PPX360, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 560:
      *done = true;
      return px_fwd_go<PPX560, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 800:
      *done = true;
      return px_fwd_go<PPX800, 4>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1134:
      *done = true;
      return px_fwd_go<PPX1134, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1536:
      *done = true;
      return px_fwd_go<PPX1536, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 2048:
      *done = true;
      return px_fwd_go<PPX2048, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_16(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 216:
      *done = true;
      return px_ratio_go<PPX216, 2>(g, tw, S, raw, mean, eps, st);
    case 360:
      *done = true;
      return px_ratio_go<PPX360, 2>(g, tw, S, raw, mean, eps, st);
    case 560:
      *done = true;
      return px_ratio_go<PPX560, 2>(g, tw, S, raw, mean, eps, st);
    case 800:
      *done = true;
      return px_ratio_go<PPX800, 4>(g, tw, S, raw, mean, eps, st);
    case 1134:
      *done = true;
      return px_ratio_go<PPX1134, 2>(g, tw, S, raw, mean, eps, st);
    case 1536:
      *done = true;
      return px_ratio_go<PPX1536, 2>(g, tw, S, raw, mean, eps, st);
    case 2048:
      *done = true;
      return px_ratio_go<PPX2048, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_16(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 216:
      *done = true;
      return px_update_go<PPX216, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 360:
      *done = true;
      return px_update_go<PPX360, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 560:
      *done = true;
      return px_update_go<PPX560, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 800:
      *done = true;
      return px_update_go<PPX800, 4>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1134:
      *done = true;
      return px_update_go<PPX1134, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1536:
      *done = true;
      return px_update_go<PPX1536, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 2048:
      *done = true;
      return px_update_go<PPX2048, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
