// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired x-pass kernels
// of the lengths 128, 243, 392, 600, 875, 1215, 1620.
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pxgen_fwd_0(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 128:
      *done = true;
      return px_fwd_go<PPX128, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 243:
      *done = true;
      return px_fwd_go<PPX243, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 392:
      *done = true;
      return px_fwd_go<PPX392, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 600:
      *done = true;
      return px_fwd_go<PPX600, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 875:
      *done = true;
      return px_fwd_go<PPX875, 3>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1215:
      *done = true;
      return px_fwd_go<PPX1215, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    case 1620:
      *done = true;
      return px_fwd_go<PPX1620, 2>(g, tw, X, Xm1, lam, predict, bg, S, st);
    default:
      return 0;
  }
}

int pxgen_ratio_0(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 128:
      *done = true;
      return px_ratio_go<PPX128, 2>(g, tw, S, raw, mean, eps, st);
    case 243:
      *done = true;
      return px_ratio_go<PPX243, 2>(g, tw, S, raw, mean, eps, st);
    case 392:
      *done = true;
      return px_ratio_go<PPX392, 2>(g, tw, S, raw, mean, eps, st);
    case 600:
      *done = true;
      return px_ratio_go<PPX600, 2>(g, tw, S, raw, mean, eps, st);
    case 875:
      *done = true;
      return px_ratio_go<PPX875, 3>(g, tw, S, raw, mean, eps, st);
    case 1215:
      *done = true;
      return px_ratio_go<PPX1215, 2>(g, tw, S, raw, mean, eps, st);
    case 1620:
      *done = true;
      return px_ratio_go<PPX1620, 2>(g, tw, S, raw, mean, eps, st);
    default:
      return 0;
  }
}

int pxgen_update_0(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  switch (g.nx) {
    case 128:
      *done = true;
      return px_update_go<PPX128, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 243:
      *done = true;
      return px_update_go<PPX243, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 392:
      *done = true;
      return px_update_go<PPX392, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 600:
      *done = true;
      return px_update_go<PPX600, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 875:
      *done = true;
      return px_update_go<PPX875, 3>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1215:
      *done = true;
      return px_update_go<PPX1215, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    case 1620:
      *done = true;
      return px_update_go<PPX1620, 2>(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st);
    default:
      return 0;
  }
}

}  // namespace cdx
