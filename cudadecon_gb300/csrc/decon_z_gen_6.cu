// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 27, 45, 64, 96, 126, 162, 210, 252, 320, 384, 450.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_6(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 27:
      *done = true;
      return pz_mode<PPZ27, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 45:
      *done = true;
      return pz_mode<PPZ45, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 64:
      *done = true;
      return pz_mode<PPZ64, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 96:
      *done = true;
      return pz_mode<PPZ96, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 126:
      *done = true;
      return pz_mode<PPZ126, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 162:
      *done = true;
      return pz_mode<PPZ162, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 210:
      *done = true;
      return pz_mode<PPZ210, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 252:
      *done = true;
      return pz_mode<PPZ252, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 320:
      *done = true;
      return pz_mode<PPZ320, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 384:
      *done = true;
      return pz_mode<PPZ384, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 450:
      *done = true;
      return pz_mode<PPZ450, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
