// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 25, 42, 63, 90, 125, 160, 200, 250, 315, 378, 448.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_5(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 25:
      *done = true;
      return pz_mode<PPZ25, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 42:
      *done = true;
      return pz_mode<PPZ42, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 63:
      *done = true;
      return pz_mode<PPZ63, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 90:
      *done = true;
      return pz_mode<PPZ90, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 125:
      *done = true;
      return pz_mode<PPZ125, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 160:
      *done = true;
      return pz_mode<PPZ160, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 200:
      *done = true;
      return pz_mode<PPZ200, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 250:
      *done = true;
      return pz_mode<PPZ250, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 315:
      *done = true;
      return pz_mode<PPZ315, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 378:
      *done = true;
      return pz_mode<PPZ378, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 448:
      *done = true;
      return pz_mode<PPZ448, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
