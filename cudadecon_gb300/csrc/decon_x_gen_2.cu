// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 140, 250, 405, 630, 896, 1250, 1701.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_2(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 140:
      *done = true;
      return px_fwd_go<PPX140, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 250:
      *done = true;
      return px_fwd_go<PPX250, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 405:
      *done = true;
      return px_fwd_go<PPX405, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 630:
      *done = true;
      return px_fwd_go<PPX630, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 896:
      *done = true;
      return px_fwd_go<PPX896, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1250:
      *done = true;
      return px_fwd_go<PPX1250, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1701:
      *done = true;
      return px_fwd_go<PPX1701, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_2(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 140:
      *done = true;
      return px_ratio_go<PPX140, 2>(g, tw, S, raw, mean, eps, st);
    case 250:
      *done = true;
      return px_ratio_go<PPX250, 2>(g, tw, S, raw, mean, eps, st);
    case 405:
      *done = true;
      return px_ratio_go<PPX405, 2>(g, tw, S, raw, mean, eps, st);
    case 630:
      *done = true;
      return px_ratio_go<PPX630, 2>(g, tw, S, raw, mean, eps, st);
    case 896:
      *done = true;
      return px_ratio_go<PPX896, 2>(g, tw, S, raw, mean, eps, st);
    case 1250:
      *done = true;
      return px_ratio_go<PPX1250, 2>(g, tw, S, raw, mean, eps, st);
    case 1701:
      *done = true;
      return px_ratio_go<PPX1701, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_2(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 140:
      *done = true;
      return px_update_go<PPX140, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 250:
      *done = true;
      return px_update_go<PPX250, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 405:
      *done = true;
      return px_update_go<PPX405, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 630:
      *done = true;
      return px_update_go<PPX630, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 896:
      *done = true;
      return px_update_go<PPX896, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1250:
      *done = true;
      return px_update_go<PPX1250, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1701:
      *done = true;
      return px_update_go<PPX1701, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
