// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 18, 32, 50, 75, 105, 140, 180, 225, 280, 343, 405, 490, 576, 675, 768, 896, 1024, 1176, 1323, 1500, 1701, 1920.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_5(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 18:
      *done = true;
      return py_eo_go<PPY18, 32>(g, tw, S, inv, st);
    case 32:
      *done = true;
      return py_eo_go<PPY32, 32>(g, tw, S, inv, st);
    case 50:
      *done = true;
      return py_eo_go<PPY50, 16>(g, tw, S, inv, st);
    case 75:
      *done = true;
      return py_zz_go<PPY75, 8>(g, tw, S, inv, st);
    case 105:
      *done = true;
      return py_zz_go<PPY105, 4>(g, tw, S, inv, st);
    case 140:
      *done = true;
      return py_eo_go<PPY140, 10>(g, tw, S, inv, st);
    case 180:
      *done = true;
      return py_eo_go<PPY180, 10>(g, tw, S, inv, st);
    case 225:
      *done = true;
      return py_zz_go<PPY225, 4>(g, tw, S, inv, st);
    case 280:
      *done = true;
      return py_eo_go<PPY280, 8>(g, tw, S, inv, st);
    case 343:
      *done = true;
      return py_zz_go<PPY343, 2>(g, tw, S, inv, st);
    case 405:
      *done = true;
      return py_zz_go<PPY405, 2>(g, tw, S, inv, st);
    case 490:
      *done = true;
      return py_eo_go<PPY490, 4>(g, tw, S, inv, st);
    case 576:
      *done = true;
      return py_eo_go<PPY576, 6>(g, tw, S, inv, st);
    case 675:
      *done = true;
      return py_zz_go<PPY675, 2>(g, tw, S, inv, st);
    case 768:
      *done = true;
      return py_eo_go<PPY768, 4>(g, tw, S, inv, st);
    case 896:
      *done = true;
      return py_eo_go<PPY896, 4>(g, tw, S, inv, st);
    case 1024:
      *done = true;
      return py_eo_go<PPY1024, 4>(g, tw, S, inv, st);
    case 1176:
      *done = true;
      return py_eo_go<PPY1176, 2>(g, tw, S, inv, st);
    case 1323:
      *done = true;
      return py_zz_go<PPY1323, 1>(g, tw, S, inv, st);
    case 1500:
      *done = true;
      return py_eo_go<PPY1500, 2>(g, tw, S, inv, st);
    case 1701:
      *done = true;
      return py_zz_go<PPY1701, 1>(g, tw, S, inv, st);
    case 1920:
      *done = true;
      return py_eo_go<PPY1920, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
