// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 168, 294, 480, 700, 1000, 1350, 1875.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_8(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 168:
      *done = true;
      return px_fwd_go<PPX168, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 294:
      *done = true;
      return px_fwd_go<PPX294, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 480:
      *done = true;
      return px_fwd_go<PPX480, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 700:
      *done = true;
      return px_fwd_go<PPX700, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1000:
      *done = true;
      return px_fwd_go<PPX1000, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1350:
      *done = true;
      return px_fwd_go<PPX1350, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1875:
      *done = true;
      return px_fwd_go<PPX1875, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_8(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 168:
      *done = true;
      return px_ratio_go<PPX168, 2>(g, tw, S, raw, mean, eps, st);
    case 294:
      *done = true;
      return px_ratio_go<PPX294, 2>(g, tw, S, raw, mean, eps, st);
    case 480:
      *done = true;
      return px_ratio_go<PPX480, 2>(g, tw, S, raw, mean, eps, st);
    case 700:
      *done = true;
      return px_ratio_go<PPX700, 2>(g, tw, S, raw, mean, eps, st);
    case 1000:
      *done = true;
      return px_ratio_go<PPX1000, 2>(g, tw, S, raw, mean, eps, st);
    case 1350:
      *done = true;
      return px_ratio_go<PPX1350, 2>(g, tw, S, raw, mean, eps, st);
    case 1875:
      *done = true;
      return px_ratio_go<PPX1875, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_8(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 168:
      *done = true;
      return px_update_go<PPX168, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 294:
      *done = true;
      return px_update_go<PPX294, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 480:
      *done = true;
      return px_update_go<PPX480, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 700:
      *done = true;
      return px_update_go<PPX700, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1000:
      *done = true;
      return px_update_go<PPX1000, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1350:
      *done = true;
      return px_update_go<PPX1350, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1875:
      *done = true;
      return px_update_go<PPX1875, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
