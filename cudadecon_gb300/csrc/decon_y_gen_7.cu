// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 21, 36, 56, 81, 112, 147, 192, 243, 294, 360, 432, 504, 600, 700, 800, 945, 1050, 1215, 1350, 1536, 1750, 1960.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_7(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 21:
      *done = true;
      return py_zz_go<PPY21, 8>(g, tw, S, inv, st);
    case 36:
      *done = true;
      return py_eo_go<PPY36, 16>(g, tw, S, inv, st);
    case 56:
      *done = true;
      return py_eo_go<PPY56, 16>(g, tw, S, inv, st);
    case 81:
      *done = true;
      return py_zz_go<PPY81, 8>(g, tw, S, inv, st);
    case 112:
      *done = true;
      return py_eo_go<PPY112, 16>(g, tw, S, inv, st);
    case 147:
      *done = true;
      return py_zz_go<PPY147, 4>(g, tw, S, inv, st);
    case 192:
      *done = true;
      return py_eo_go<PPY192, 10>(g, tw, S, inv, st);
    case 243:
      *done = true;
      return py_zz_go<PPY243, 2>(g, tw, S, inv, st);
    case 294:
      *done = true;
      return py_eo_go<PPY294, 4>(g, tw, S, inv, st);
    case 360:
      *done = true;
      return py_eo_go<PPY360, 8>(g, tw, S, inv, st);
    case 432:
      *done = true;
      return py_eo_go<PPY432, 6>(g, tw, S, inv, st);
    case 504:
      *done = true;
      return py_eo_go<PPY504, 6>(g, tw, S, inv, st);
    case 600:
      *done = true;
      return py_eo_go<PPY600, 4>(g, tw, S, inv, st);
    case 700:
      *done = true;
      return py_eo_go<PPY700, 2>(g, tw, S, inv, st);
    case 800:
      *done = true;
      return py_eo_go<PPY800, 2>(g, tw, S, inv, st);
    case 945:
      *done = true;
      return py_zz_go<PPY945, 2>(g, tw, S, inv, st);
    case 1050:
      *done = true;
      return py_eo_go<PPY1050, 2>(g, tw, S, inv, st);
    case 1215:
      *done = true;
      return py_zz_go<PPY1215, 1>(g, tw, S, inv, st);
    case 1350:
      *done = true;
      return py_eo_go<PPY1350, 2>(g, tw, S, inv, st);
    case 1536:
      *done = true;
      return py_eo_go<PPY1536, 2>(g, tw, S, inv, st);
    case 1750:
      *done = true;
      return py_eo_go<PPY1750, 2>(g, tw, S, inv, st);
    case 1960:
      *done = true;
      return py_eo_go<PPY1960, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
