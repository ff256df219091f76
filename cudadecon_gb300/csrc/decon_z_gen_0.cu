// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 16, 30, 49, 72, 100, 135, 175, 224, 270, 336, 400, 486.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_0(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 16:
      *done = true;
      return pz_mode<PPZ16, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 30:
      *done = true;
      return pz_mode<PPZ30, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 49:
      *done = true;
      return pz_mode<PPZ49, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 72:
      *done = true;
      return pz_mode<PPZ72, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 100:
      *done = true;
      return pz_mode<PPZ100, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 135:
      *done = true;
      return pz_mode<PPZ135, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 175:
      *done = true;
      return pz_mode<PPZ175, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 224:
      *done = true;
      return pz_mode<PPZ224, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 270:
      *done = true;
      return pz_mode<PPZ270, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 336:
      *done = true;
      return pz_mode<PPZ336, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 400:
      *done = true;
      return pz_mode<PPZ400, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 486:
      *done = true;
      return pz_mode<PPZ486, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
