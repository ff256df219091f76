// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 48, 70, 98, 128, 168, 216, 256, 324, 392, 480, 560, 648, 750, 875, 1000.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_6(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 48:
      *done = true;
      return py_eo_go<PPY48, 16>(g, tw, S, inv, st);
    case 70:
      *done = true;
      return py_eo_go<PPY70, 16>(g, tw, S, inv, st);
    case 98:
      *done = true;
      return py_eo_go<PPY98, 16>(g, tw, S, inv, st);
    case 128:
      *done = true;
      return py_eo_go<PPY128, 16>(g, tw, S, inv, st);
    case 168:
      *done = true;
      return py_eo_go<PPY168, 11>(g, tw, S, inv, st);
    case 216:
      *done = true;
      return py_eo_go<PPY216, 11>(g, tw, S, inv, st);
    case 256:
      *done = true;
      return py_eo_go<PPY256, 8>(g, tw, S, inv, st);
    case 324:
      *done = true;
      return py_eo_go<PPY324, 6>(g, tw, S, inv, st);
    case 392:
      *done = true;
      return py_eo_go<PPY392, 8>(g, tw, S, inv, st);
    case 480:
      *done = true;
      return py_eo_go<PPY480, 8>(g, tw, S, inv, st);
    case 560:
      *done = true;
      return py_eo_go<PPY560, 4>(g, tw, S, inv, st);
    case 648:
      *done = true;
      return py_eo_go<PPY648, 6>(g, tw, S, inv, st);
    case 750:
      *done = true;
      return py_eo_go<PPY750, 4>(g, tw, S, inv, st);
    case 875:
      *done = true;
      return py_zz_go<PPY875, 4>(g, tw, S, inv, st);
    case 1000:
      *done = true;
      return py_eo_go<PPY1000, 4>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
