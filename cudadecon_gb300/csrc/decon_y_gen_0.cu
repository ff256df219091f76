// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 8, 24, 40, 60, 84, 120, 150, 196, 245, 300, 375, 441, 512, 625, 720, 810, 960, 1080, 1225, 1372, 1568, 1764, 2000.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_0(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 8:
      *done = true;
      return py_eo_go<PPY8, 32>(g, tw, S, inv, st);
    case 24:
      *done = true;
      return py_eo_go<PPY24, 32>(g, tw, S, inv, st);
    case 40:
      *done = true;
      return py_eo_go<PPY40, 16>(g, tw, S, inv, st);
    case 60:
      *done = true;
      return py_eo_go<PPY60, 16>(g, tw, S, inv, st);
    case 84:
      *done = true;
      return py_eo_go<PPY84, 16>(g, tw, S, inv, st);
    case 120:
      *done = true;
      return py_eo_go<PPY120, 10>(g, tw, S, inv, st);
    case 150:
      *done = true;
      return py_eo_go<PPY150, 8>(g, tw, S, inv, st);
    case 196:
      *done = true;
      return py_eo_go<PPY196, 8>(g, tw, S, inv, st);
    case 245:
      *done = true;
      return py_zz_go<PPY245, 2>(g, tw, S, inv, st);
    case 300:
      *done = true;
      return py_eo_go<PPY300, 8>(g, tw, S, inv, st);
    case 375:
      *done = true;
      return py_zz_go<PPY375, 4>(g, tw, S, inv, st);
    case 441:
      *done = true;
      return py_zz_go<PPY441, 2>(g, tw, S, inv, st);
    case 512:
      *done = true;
      return py_eo_go<PPY512, 8>(g, tw, S, inv, st);
    case 625:
      *done = true;
      return py_zz_go<PPY625, 2>(g, tw, S, inv, st);
    case 720:
      *done = true;
      return py_eo_go<PPY720, 2>(g, tw, S, inv, st);
    case 810:
      *done = true;
      return py_eo_go<PPY810, 2>(g, tw, S, inv, st);
    case 960:
      *done = true;
      return py_eo_go<PPY960, 2>(g, tw, S, inv, st);
    case 1080:
      *done = true;
      return py_eo_go<PPY1080, 2>(g, tw, S, inv, st);
    case 1225:
      *done = true;
      return py_zz_go<PPY1225, 2>(g, tw, S, inv, st);
    case 1372:
      *done = true;
      return py_eo_go<PPY1372, 2>(g, tw, S, inv, st);
    case 1568:
      *done = true;
      return py_eo_go<PPY1568, 2>(g, tw, S, inv, st);
    case 1764:
      *done = true;
      return py_eo_go<PPY1764, 2>(g, tw, S, inv, st);
    case 2000:
      *done = true;
      return py_eo_go<PPY2000, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
