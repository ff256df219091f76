// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 135, 245, 400, 625, 882, 1225, 1680.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_1(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 135:
      *done = true;
      return px_fwd_go<PPX135, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 245:
      *done = true;
      return px_fwd_go<PPX245, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 400:
      *done = true;
      return px_fwd_go<PPX400, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 625:
      *done = true;
      return px_fwd_go<PPX625, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 882:
      *done = true;
      return px_fwd_go<PPX882, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1225:
      *done = true;
      return px_fwd_go<PPX1225, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1680:
      *done = true;
      return px_fwd_go<PPX1680, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_1(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 135:
      *done = true;
      return px_ratio_go<PPX135, 2>(g, tw, S, raw, mean, eps, st);
    case 245:
      *done = true;
      return px_ratio_go<PPX245, 2>(g, tw, S, raw, mean, eps, st);
    case 400:
      *done = true;
      return px_ratio_go<PPX400, 2>(g, tw, S, raw, mean, eps, st);
    case 625:
      *done = true;
      return px_ratio_go<PPX625, 2>(g, tw, S, raw, mean, eps, st);
    case 882:
      *done = true;
      return px_ratio_go<PPX882, 2>(g, tw, S, raw, mean, eps, st);
    case 1225:
      *done = true;
      return px_ratio_go<PPX1225, 2>(g, tw, S, raw, mean, eps, st);
    case 1680:
      *done = true;
      return px_ratio_go<PPX1680, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_1(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 135:
      *done = true;
      return px_update_go<PPX135, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 245:
      *done = true;
      return px_update_go<PPX245, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 400:
      *done = true;
      return px_update_go<PPX400, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 625:
      *done = true;
      return px_update_go<PPX625, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 882:
      *done = true;
      return px_update_go<PPX882, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1225:
      *done = true;
      return px_update_go<PPX1225, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1680:
      *done = true;
      return px_update_go<PPX1680, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
