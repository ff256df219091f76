// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 9, 25, 42, 63, 90, 125, 160, 200, 250, 315, 378, 448, 525, 630, 729, 840, 972, 1120, 1250, 1400, 1575, 1792, 2016.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_1(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 9:
      *done = true;
      return py_zz_go<PPY9, 8>(g, tw, S, inv, st);
    case 25:
      *done = true;
      return py_zz_go<PPY25, 8>(g, tw, S, inv, st);
    case 42:
      *done = true;
      return py_eo_go<PPY42, 16>(g, tw, S, inv, st);
    case 63:
      *done = true;
      return py_zz_go<PPY63, 8>(g, tw, S, inv, st);
    case 90:
      *done = true;
      return py_eo_go<PPY90, 10>(g, tw, S, inv, st);
    case 125:
      *done = true;
      return py_zz_go<PPY125, 4>(g, tw, S, inv, st);
    case 160:
      *done = true;
      return py_eo_go<PPY160, 10>(g, tw, S, inv, st);
    case 200:
      *done = true;
      return py_eo_go<PPY200, 10>(g, tw, S, inv, st);
    case 250:
      *done = true;
      return py_eo_go<PPY250, 4>(g, tw, S, inv, st);
    case 315:
      *done = true;
      return py_zz_go<PPY315, 2>(g, tw, S, inv, st);
    case 378:
      *done = true;
      return py_eo_go<PPY378, 4>(g, tw, S, inv, st);
    case 448:
      *done = true;
      return py_eo_go<PPY448, 8>(g, tw, S, inv, st);
    case 525:
      *done = true;
      return py_zz_go<PPY525, 2>(g, tw, S, inv, st);
    case 630:
      *done = true;
      return py_eo_go<PPY630, 4>(g, tw, S, inv, st);
    case 729:
      *done = true;
      return py_zz_go<PPY729, 2>(g, tw, S, inv, st);
    case 840:
      *done = true;
      return py_eo_go<PPY840, 2>(g, tw, S, inv, st);
    case 972:
      *done = true;
      return py_eo_go<PPY972, 2>(g, tw, S, inv, st);
    case 1120:
      *done = true;
      return py_eo_go<PPY1120, 2>(g, tw, S, inv, st);
    case 1250:
      *done = true;
      return py_eo_go<PPY1250, 4>(g, tw, S, inv, st);
    case 1400:
      *done = true;
      return py_eo_go<PPY1400, 2>(g, tw, S, inv, st);
    case 1575:
      *done = true;
      return py_zz_go<PPY1575, 1>(g, tw, S, inv, st);
    case 1792:
      *done = true;
      return py_eo_go<PPY1792, 2>(g, tw, S, inv, st);
    case 2016:
      *done = true;
      return py_eo_go<PPY2016, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
