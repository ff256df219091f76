// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 15, 28, 48, 70, 98, 128, 168, 216, 256, 324, 392, 480, 560, 648, 750, 875, 1000, 1134, 1280, 1458, 1620, 1875, 2048.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_3(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 15:
      *done = true;
      return py_zz_go<PPY15, 8>(g, tw, S, inv, st);
    case 28:
      *done = true;
      return py_eo_go<PPY28, 16>(g, tw, S, inv, st);
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
      return py_eo_go<PPY168, 10>(g, tw, S, inv, st);
    case 216:
      *done = true;
      return py_eo_go<PPY216, 10>(g, tw, S, inv, st);
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
      return py_eo_go<PPY750, 2>(g, tw, S, inv, st);
    case 875:
      *done = true;
      return py_zz_go<PPY875, 2>(g, tw, S, inv, st);
    case 1000:
      *done = true;
      return py_eo_go<PPY1000, 2>(g, tw, S, inv, st);
    case 1134:
      *done = true;
      return py_eo_go<PPY1134, 2>(g, tw, S, inv, st);
    case 1280:
      *done = true;
      return py_eo_go<PPY1280, 2>(g, tw, S, inv, st);
    case 1458:
      *done = true;
      return py_eo_go<PPY1458, 2>(g, tw, S, inv, st);
    case 1620:
      *done = true;
      return py_eo_go<PPY1620, 2>(g, tw, S, inv, st);
    case 1875:
      *done = true;
      return py_zz_go<PPY1875, 1>(g, tw, S, inv, st);
    case 2048:
      *done = true;
      return py_eo_go<PPY2048, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
