// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 150, 270, 441, 672, 960, 1296, 1764.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_5(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 150:
      *done = true;
      return px_fwd_go<PPX150, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 270:
      *done = true;
      return px_fwd_go<PPX270, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 441:
      *done = true;
      return px_fwd_go<PPX441, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 672:
      *done = true;
      return px_fwd_go<PPX672, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 960:
      *done = true;
      return px_fwd_go<PPX960, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1296:
      *done = true;
      return px_fwd_go<PPX1296, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1764:
      *done = true;
      return px_fwd_go<PPX1764, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_5(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 150:
      *done = true;
      return px_ratio_go<PPX150, 2>(g, tw, S, raw, mean, eps, st);
    case 270:
      *done = true;
      return px_ratio_go<PPX270, 2>(g, tw, S, raw, mean, eps, st);
    case 441:
      *done = true;
      return px_ratio_go<PPX441, 2>(g, tw, S, raw, mean, eps, st);
    case 672:
      *done = true;
      return px_ratio_go<PPX672, 2>(g, tw, S, raw, mean, eps, st);
    case 960:
      *done = true;
      return px_ratio_go<PPX960, 2>(g, tw, S, raw, mean, eps, st);
    case 1296:
      *done = true;
      return px_ratio_go<PPX1296, 2>(g, tw, S, raw, mean, eps, st);
    case 1764:
      *done = true;
      return px_ratio_go<PPX1764, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_5(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 150:
      *done = true;
      return px_update_go<PPX150, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 270:
      *done = true;
      return px_update_go<PPX270, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 441:
      *done = true;
      return px_update_go<PPX441, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 672:
      *done = true;
      return px_update_go<PPX672, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 960:
      *done = true;
      return px_update_go<PPX960, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1296:
      *done = true;
      return px_update_go<PPX1296, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1764:
      *done = true;
      return px_update_go<PPX1764, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
