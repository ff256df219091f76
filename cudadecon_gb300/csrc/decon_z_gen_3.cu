// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 21, 36, 56, 81, 112, 147, 192, 243, 294, 360, 432, 504.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_3(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 21:
      *done = true;
      return pz_mode<PPZ21, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 36:
      *done = true;
      return pz_mode<PPZ36, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 56:
      *done = true;
      return pz_mode<PPZ56, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 81:
      *done = true;
      return pz_mode<PPZ81, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 112:
      *done = true;
      return pz_mode<PPZ112, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 147:
      *done = true;
      return pz_mode<PPZ147, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 192:
      *done = true;
      return pz_mode<PPZ192, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 243:
      *done = true;
      return pz_mode<PPZ243, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 294:
      *done = true;
      return pz_mode<PPZ294, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 360:
      *done = true;
      return pz_mode<PPZ360, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 432:
      *done = true;
      return pz_mode<PPZ432, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 504:
      *done = true;
      return pz_mode<PPZ504, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
