// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired z-pass kernels
// of the lengths 18, 32, 50, 75, 105, 140, 180, 225, 280, 343, 405, 490.
#include "decon_pz.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pzgen_1(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  switch (g.nz) {
    case 18:
      *done = true;
      return pz_mode<PPZ18, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 32:
      *done = true;
      return pz_mode<PPZ32, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 50:
      *done = true;
      return pz_mode<PPZ50, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 75:
      *done = true;
      return pz_mode<PPZ75, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 105:
      *done = true;
      return pz_mode<PPZ105, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 140:
      *done = true;
      return pz_mode<PPZ140, 16>(g, tw, S, otf, conj, st, fwd_only);
    case 180:
      *done = true;
      return pz_mode<PPZ180, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 225:
      *done = true;
      return pz_mode<PPZ225, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 280:
      *done = true;
      return pz_mode<PPZ280, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 343:
      *done = true;
      return pz_mode<PPZ343, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 405:
      *done = true;
      return pz_mode<PPZ405, 8>(g, tw, S, otf, conj, st, fwd_only);
    case 490:
      *done = true;
      return pz_mode<PPZ490, 8>(g, tw, S, otf, conj, st, fwd_only);
    default:
      return 0;
  }
}

}  // namespace cdx
