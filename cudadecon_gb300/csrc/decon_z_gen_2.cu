// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 20, 35, 54, 80, 108, 144, 189, 240, 288, 350, 420, 500.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_2(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 20:
      *done = true;
      return pz_mode<PPZ20, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 35:
      *done = true;
      return pz_mode<PPZ35, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 54:
      *done = true;
      return pz_mode<PPZ54, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 80:
      *done = true;
      return pz_mode<PPZ80, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 108:
      *done = true;
      return pz_mode<PPZ108, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 144:
      *done = true;
      return pz_mode<PPZ144, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 189:
      *done = true;
      return pz_mode<PPZ189, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 240:
      *done = true;
      return pz_mode<PPZ240, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 288:
      *done = true;
      return pz_mode<PPZ288, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 350:
      *done = true;
      return pz_mode<PPZ350, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 420:
      *done = true;
      return pz_mode<PPZ420, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 500:
      *done = true;
      return pz_mode<PPZ500, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
