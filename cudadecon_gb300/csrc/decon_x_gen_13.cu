// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 196, 336, 512, 756, 1080, 1470, 2000.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_13(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 196:
      *done = true;
      return px_fwd_go<PPX196, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 336:
      *done = true;
      return px_fwd_go<PPX336, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 512:
      *done = true;
      return px_fwd_go<PPX512, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 756:
      *done = true;
      return px_fwd_go<PPX756, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1080:
      *done = true;
      return px_fwd_go<PPX1080, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1470:
      *done = true;
      return px_fwd_go<PPX1470, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 2000:
      *done = true;
      return px_fwd_go<PPX2000, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_13(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 196:
      *done = true;
      return px_ratio_go<PPX196, 2>(g, tw, S, raw, mean, eps, st);
    case 336:
      *done = true;
      return px_ratio_go<PPX336, 2>(g, tw, S, raw, mean, eps, st);
    case 512:
      *done = true;
      return px_ratio_go<PPX512, 2>(g, tw, S, raw, mean, eps, st);
    case 756:
      *done = true;
      return px_ratio_go<PPX756, 2>(g, tw, S, raw, mean, eps, st);
    case 1080:
      *done = true;
      return px_ratio_go<PPX1080, 2>(g, tw, S, raw, mean, eps, st);
    case 1470:
      *done = true;
      return px_ratio_go<PPX1470, 2>(g, tw, S, raw, mean, eps, st);
    case 2000:
      *done = true;
      return px_ratio_go<PPX2000, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_13(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 196:
      *done = true;
      return px_update_go<PPX196, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 336:
      *done = true;
      return px_update_go<PPX336, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 512:
      *done = true;
      return px_update_go<PPX512, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 756:
      *done = true;
      return px_update_go<PPX756, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1080:
      *done = true;
      return px_update_go<PPX1080, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1470:
      *done = true;
      return px_update_go<PPX1470, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 2000:
      *done = true;
      return px_update_go<PPX2000, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
