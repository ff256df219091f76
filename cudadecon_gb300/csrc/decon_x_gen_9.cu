// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 175, 300, 486, 720, 1008, 1372, 1890.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_9(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 175:
      *done = true;
      return px_fwd_go<PPX175, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 300:
      *done = true;
      return px_fwd_go<PPX300, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 486:
      *done = true;
      return px_fwd_go<PPX486, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 720:
      *done = true;
      return px_fwd_go<PPX720, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1008:
      *done = true;
      return px_fwd_go<PPX1008, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1372:
      *done = true;
      return px_fwd_go<PPX1372, 4>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1890:
      *done = true;
      return px_fwd_go<PPX1890, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_9(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 175:
      *done = true;
      return px_ratio_go<PPX175, 2>(g, tw, S, raw, mean, eps, st);
    case 300:
      *done = true;
      return px_ratio_go<PPX300, 2>(g, tw, S, raw, mean, eps, st);
    case 486:
      *done = true;
      return px_ratio_go<PPX486, 2>(g, tw, S, raw, mean, eps, st);
    case 720:
      *done = true;
      return px_ratio_go<PPX720, 2>(g, tw, S, raw, mean, eps, st);
    case 1008:
      *done = true;
      return px_ratio_go<PPX1008, 2>(g, tw, S, raw, mean, eps, st);
    case 1372:
      *done = true;
      return px_ratio_go<PPX1372, 4>(g, tw, S, raw, mean, eps, st);
    case 1890:
      *done = true;
      return px_ratio_go<PPX1890, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_9(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 175:
      *done = true;
      return px_update_go<PPX175, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 300:
      *done = true;
      return px_update_go<PPX300, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 486:
      *done = true;
      return px_update_go<PPX486, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 720:
      *done = true;
      return px_update_go<PPX720, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1008:
      *done = true;
      return px_update_go<PPX1008, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1372:
      *done = true;
      return px_update_go<PPX1372, 4>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1890:
      *done = true;
      return px_update_go<PPX1890, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
