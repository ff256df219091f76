// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 35, 54, 80, 108, 144, 189, 240, 288, 350, 420, 500, 588, 686, 784, 900.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_1(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 35:
      *done = true;
      return py_zz_go<PPY35, 16>(g, tw, S, inv, st);
    case 54:
      *done = true;
      return py_eo_go<PPY54, 11>(g, tw, S, inv, st);
    case 80:
      *done = true;
      return py_eo_go<PPY80, 16>(g, tw, S, inv, st);
    case 108:
      *done = true;
      return py_eo_go<PPY108, 11>(g, tw, S, inv, st);
    case 144:
      *done = true;
      return py_eo_go<PPY144, 11>(g, tw, S, inv, st);
    case 189:
      *done = true;
      return py_zz_go<PPY189, 4>(g, tw, S, inv, st);
    case 240:
      *done = true;
      return py_eo_go<PPY240, 11>(g, tw, S, inv, st);
    case 288:
      *done = true;
      return py_eo_go<PPY288, 11>(g, tw, S, inv, st);
    case 350:
      *done = true;
      return py_eo_go<PPY350, 4>(g, tw, S, inv, st);
    case 420:
      *done = true;
      return py_eo_go<PPY420, 8>(g, tw, S, inv, st);
    case 500:
      *done = true;
      return py_eo_go<PPY500, 4>(g, tw, S, inv, st);
    case 588:
      *done = true;
      return py_eo_go<PPY588, 4>(g, tw, S, inv, st);
    case 686:
      *done = true;
      return py_eo_go<PPY686, 4>(g, tw, S, inv, st);
    case 784:
      *done = true;
      return py_eo_go<PPY784, 4>(g, tw, S, inv, st);
    case 900:
      *done = true;
      return py_eo_go<PPY900, 4>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
