// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 42, 63, 90, 125, 160, 200, 250, 315, 378, 448, 525, 630, 729, 840, 972.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_4(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 42:
      *done = true;
      return py_eo_go<PPY42, 16>(g, tw, S, inv, st);
    case 63:
      *done = true;
      return py_zz_go<PPY63, 11>(g, tw, S, inv, st);
    case 90:
      *done = true;
      return py_eo_go<PPY90, 11>(g, tw, S, inv, st);
    case 125:
      *done = true;
      return py_zz_go<PPY125, 5>(g, tw, S, inv, st);
    case 160:
      *done = true;
      return py_eo_go<PPY160, 11>(g, tw, S, inv, st);
    case 200:
      *done = true;
      return py_eo_go<PPY200, 11>(g, tw, S, inv, st);
    case 250:
      *done = true;
      return py_eo_go<PPY250, 5>(g, tw, S, inv, st);
    case 315:
      *done = true;
      return py_zz_go<PPY315, 4>(g, tw, S, inv, st);
    case 378:
      *done = true;
      return py_eo_go<PPY378, 4>(g, tw, S, inv, st);
    case 448:
      *done = true;
      return py_eo_go<PPY448, 8>(g, tw, S, inv, st);
    case 525:
      *done = true;
      return py_zz_go<PPY525, 4>(g, tw, S, inv, st);
    case 630:
      *done = true;
      return py_eo_go<PPY630, 4>(g, tw, S, inv, st);
    case 729:
      *done = true;
      return py_zz_go<PPY729, 4>(g, tw, S, inv, st);
    case 840:
      *done = true;
      return py_eo_go<PPY840, 4>(g, tw, S, inv, st);
    case 972:
      *done = true;
      return py_eo_go<PPY972, 4>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
