// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 180, 315, 490, 729, 1024, 1400, 1920.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_10(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 180:
      *done = true;
      return px_fwd_go<PPX180, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 315:
      *done = true;
      return px_fwd_go<PPX315, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 490:
      *done = true;
      return px_fwd_go<PPX490, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 729:
      *done = true;
      return px_fwd_go<PPX729, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1024:
      *done = true;
      return px_fwd_go<PPX1024, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1400:
      *done = true;
      return px_fwd_go<PPX1400, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1920:
      *done = true;
      return px_fwd_go<PPX1920, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_10(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 180:
      *done = true;
      return px_ratio_go<PPX180, 2>(g, tw, S, raw, mean, eps, st);
    case 315:
      *done = true;
      return px_ratio_go<PPX315, 2>(g, tw, S, raw, mean, eps, st);
    case 490:
      *done = true;
      return px_ratio_go<PPX490, 2>(g, tw, S, raw, mean, eps, st);
    case 729:
      *done = true;
      return px_ratio_go<PPX729, 2>(g, tw, S, raw, mean, eps, st);
    case 1024:
      *done = true;
      return px_ratio_go<PPX1024, 2>(g, tw, S, raw, mean, eps, st);
    case 1400:
      *done = true;
      return px_ratio_go<PPX1400, 2>(g, tw, S, raw, mean, eps, st);
    case 1920:
      *done = true;
      return px_ratio_go<PPX1920, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_10(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 180:
      *done = true;
      return px_update_go<PPX180, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 315:
      *done = true;
      return px_update_go<PPX315, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 490:
      *done = true;
      return px_update_go<PPX490, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 729:
      *done = true;
      return px_update_go<PPX729, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1024:
      *done = true;
      return px_update_go<PPX1024, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1400:
      *done = true;
      return px_update_go<PPX1400, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1920:
      *done = true;
      return px_update_go<PPX1920, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
