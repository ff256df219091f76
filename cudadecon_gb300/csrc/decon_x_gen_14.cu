// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 200, 343, 525, 768, 1120, 1500, 2016.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_14(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 200:
      *done = true;
      return px_fwd_go<PPX200, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 343:
      *done = true;
      return px_fwd_go<PPX343, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 525:
      *done = true;
      return px_fwd_go<PPX525, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 768:
      *done = true;
      return px_fwd_go<PPX768, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1120:
      *done = true;
      return px_fwd_go<PPX1120, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1500:
      *done = true;
      return px_fwd_go<PPX1500, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 2016:
      *done = true;
      return px_fwd_go<PPX2016, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_14(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 200:
      *done = true;
      return px_ratio_go<PPX200, 2>(g, tw, S, raw, mean, eps, st);
    case 343:
      *done = true;
      return px_ratio_go<PPX343, 2>(g, tw, S, raw, mean, eps, st);
    case 525:
      *done = true;
      return px_ratio_go<PPX525, 2>(g, tw, S, raw, mean, eps, st);
    case 768:
      *done = true;
      return px_ratio_go<PPX768, 2>(g, tw, S, raw, mean, eps, st);
    case 1120:
      *done = true;
      return px_ratio_go<PPX1120, 2>(g, tw, S, raw, mean, eps, st);
    case 1500:
      *done = true;
      return px_ratio_go<PPX1500, 2>(g, tw, S, raw, mean, eps, st);
    case 2016:
      *done = true;
      return px_ratio_go<PPX2016, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_14(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 200:
      *done = true;
      return px_update_go<PPX200, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 343:
      *done = true;
      return px_update_go<PPX343, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 525:
      *done = true;
      return px_update_go<PPX525, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 768:
      *done = true;
      return px_update_go<PPX768, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1120:
      *done = true;
      return px_update_go<PPX1120, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1500:
      *done = true;
      return px_update_go<PPX1500, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 2016:
      *done = true;
      return px_update_go<PPX2016, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
