// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 12, 27, 45, 64, 96, 126, 162, 210, 252, 320, 384, 450, 540, 640, 735, 864, 980, 1125, 1260, 1440, 1600, 1800, 2025.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_2(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 12:
      *done = true;
      return py_eo_go<PPY12, 32>(g, tw, S, inv, st);
    case 27:
      *done = true;
      return py_zz_go<PPY27, 8>(g, tw, S, inv, st);
    case 45:
      *done = true;
      return py_zz_go<PPY45, 8>(g, tw, S, inv, st);
    case 64:
      *done = true;
      return py_eo_go<PPY64, 16>(g, tw, S, inv, st);
    case 96:
      *done = true;
      return py_eo_go<PPY96, 16>(g, tw, S, inv, st);
    case 126:
      *done = true;
      return py_eo_go<PPY126, 10>(g, tw, S, inv, st);
    case 162:
      *done = true;
      return py_eo_go<PPY162, 10>(g, tw, S, inv, st);
    case 210:
      *done = true;
      return py_eo_go<PPY210, 8>(g, tw, S, inv, st);
    case 252:
      *done = true;
      return py_eo_go<PPY252, 8>(g, tw, S, inv, st);
    case 320:
      *done = true;
      return py_eo_go<PPY320, 8>(g, tw, S, inv, st);
    case 384:
      *done = true;
      return py_eo_go<PPY384, 8>(g, tw, S, inv, st);
    case 450:
      *done = true;
      return py_eo_go<PPY450, 8>(g, tw, S, inv, st);
    case 540:
      *done = true;
      return py_eo_go<PPY540, 6>(g, tw, S, inv, st);
    case 640:
      *done = true;
      return py_eo_go<PPY640, 4>(g, tw, S, inv, st);
    case 735:
      *done = true;
      return py_zz_go<PPY735, 2>(g, tw, S, inv, st);
    case 864:
      *done = true;
      return py_eo_go<PPY864, 2>(g, tw, S, inv, st);
    case 980:
      *done = true;
      return py_eo_go<PPY980, 2>(g, tw, S, inv, st);
    case 1125:
      *done = true;
      return py_zz_go<PPY1125, 1>(g, tw, S, inv, st);
    case 1260:
      *done = true;
      return py_eo_go<PPY1260, 2>(g, tw, S, inv, st);
    case 1440:
      *done = true;
      return py_eo_go<PPY1440, 2>(g, tw, S, inv, st);
    case 1600:
      *done = true;
      return py_eo_go<PPY1600, 2>(g, tw, S, inv, st);
    case 1800:
      *done = true;
      return py_eo_go<PPY1800, 2>(g, tw, S, inv, st);
    case 2025:
      *done = true;
      return py_zz_go<PPY2025, 1>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
