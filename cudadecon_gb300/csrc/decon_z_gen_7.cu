// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 28, 48, 70, 98, 128, 168, 216, 256, 324, 392, 480.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_7(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 28:
      *done = true;
      return pz_mode<PPZ28, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 48:
      *done = true;
      return pz_mode<PPZ48, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 70:
      *done = true;
      return pz_mode<PPZ70, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 98:
      *done = true;
      return pz_mode<PPZ98, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 128:
      *done = true;
      return pz_mode<PPZ128, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 168:
      *done = true;
      return pz_mode<PPZ168, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 216:
      *done = true;
      return pz_mode<PPZ216, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 256:
      *done = true;
      return pz_mode<PPZ256, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 324:
      *done = true;
      return pz_mode<PPZ324, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 392:
      *done = true;
      return pz_mode<PPZ392, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 480:
      *done = true;
      return pz_mode<PPZ480, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
