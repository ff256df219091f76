// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 45, 64, 96, 126, 162, 210, 252, 320, 384, 450, 540, 640, 735, 864, 980.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_5(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 45:
      *done = true;
      return py_zz_go<PPY45, 11>(g, tw, S, inv, st);
    case 64:
      *done = true;
      return py_eo_go<PPY64, 16>(g, tw, S, inv, st);
    case 96:
      *done = true;
      return py_eo_go<PPY96, 16>(g, tw, S, inv, st);
    case 126:
      *done = true;
      return py_eo_go<PPY126, 11>(g, tw, S, inv, st);
    case 162:
      *done = true;
      return py_eo_go<PPY162, 11>(g, tw, S, inv, st);
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
      return py_zz_go<PPY735, 4>(g, tw, S, inv, st);
    case 864:
      *done = true;
      return py_eo_go<PPY864, 4>(g, tw, S, inv, st);
    case 980:
      *done = true;
      return py_eo_go<PPY980, 4>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
