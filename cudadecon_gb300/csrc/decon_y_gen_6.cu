// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 20, 35, 54, 80, 108, 144, 189, 240, 288, 350, 420, 500, 588, 686, 784, 900, 1029, 1200, 1344, 1512, 1728, 1944.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_6(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 20:
      *done = true;
      return py_eo_go<PPY20, 16>(g, tw, S, inv, st);
    case 35:
      *done = true;
      return py_zz_go<PPY35, 8>(g, tw, S, inv, st);
    case 54:
      *done = true;
      return py_eo_go<PPY54, 10>(g, tw, S, inv, st);
    case 80:
      *done = true;
      return py_eo_go<PPY80, 16>(g, tw, S, inv, st);
    case 108:
      *done = true;
      return py_eo_go<PPY108, 10>(g, tw, S, inv, st);
    case 144:
      *done = true;
      return py_eo_go<PPY144, 10>(g, tw, S, inv, st);
    case 189:
      *done = true;
      return py_zz_go<PPY189, 2>(g, tw, S, inv, st);
    case 240:
      *done = true;
      return py_eo_go<PPY240, 10>(g, tw, S, inv, st);
    case 288:
      *done = true;
      return py_eo_go<PPY288, 10>(g, tw, S, inv, st);
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
      return py_eo_go<PPY900, 2>(g, tw, S, inv, st);
    case 1029:
      *done = true;
      return py_zz_go<PPY1029, 1>(g, tw, S, inv, st);
    case 1200:
      *done = true;
      return py_eo_go<PPY1200, 2>(g, tw, S, inv, st);
    case 1344:
      *done = true;
      return py_eo_go<PPY1344, 2>(g, tw, S, inv, st);
    case 1512:
      *done = true;
      return py_eo_go<PPY1512, 2>(g, tw, S, inv, st);
    case 1728:
      *done = true;
      return py_eo_go<PPY1728, 2>(g, tw, S, inv, st);
    case 1944:
      *done = true;
      return py_eo_go<PPY1944, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
