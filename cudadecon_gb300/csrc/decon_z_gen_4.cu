// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 24, 40, 60, 84, 120, 150, 196, 245, 300, 375, 441, 512.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_4(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 24:
      *done = true;
      return pz_mode<PPZ24, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 40:
      *done = true;
      return pz_mode<PPZ40, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 60:
      *done = true;
      return pz_mode<PPZ60, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 84:
      *done = true;
      return pz_mode<PPZ84, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 120:
      *done = true;
      return pz_mode<PPZ120, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 150:
      *done = true;
      return pz_mode<PPZ150, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 196:
      *done = true;
      return pz_mode<PPZ196, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 245:
      *done = true;
      return pz_mode<PPZ245, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 300:
      *done = true;
      return pz_mode<PPZ300, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 375:
      *done = true;
      return pz_mode<PPZ375, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 441:
      *done = true;
      return pz_mode<PPZ441, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 512:
      *done = true;
      return pz_mode<PPZ512, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
