// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired y-pass kernels
// of the lengths 16, 30, 49, 72, 100, 135, 175, 224, 270, 336, 400, 486, 567, 672, 756, 882, 1008, 1152, 1296, 1470, 1680, 1890.
#include "decon_py.cuh"
#include "pair_plans_gen.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int pygen_4(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  switch (g.ny) {
    case 16:
      *done = true;
      return py_eo_go<PPY16, 32>(g, tw, S, inv, st);
    case 30:
      *done = true;
      return py_eo_go<PPY30, 16>(g, tw, S, inv, st);
    case 49:
      *done = true;
      return py_zz_go<PPY49, 8>(g, tw, S, inv, st);
    case 72:
      *done = true;
      return py_eo_go<PPY72, 16>(g, tw, S, inv, st);
    case 100:
      *done = true;
      return py_eo_go<PPY100, 10>(g, tw, S, inv, st);
    case 135:
      *done = true;
      return py_zz_go<PPY135, 4>(g, tw, S, inv, st);
    case 175:
      *done = true;
      return py_zz_go<PPY175, 4>(g, tw, S, inv, st);
    case 224:
      *done = true;
      return py_eo_go<PPY224, 8>(g, tw, S, inv, st);
    case 270:
      *done = true;
      return py_eo_go<PPY270, 8>(g, tw, S, inv, st);
    case 336:
      *done = true;
      return py_eo_go<PPY336, 8>(g, tw, S, inv, st);
    case 400:
      *done = true;
      return py_eo_go<PPY400, 4>(g, tw, S, inv, st);
    case 486:
      *done = true;
      return py_eo_go<PPY486, 2>(g, tw, S, inv, st);
    case 567:
      *done = true;
      return py_zz_go<PPY567, 2>(g, tw, S, inv, st);
    case 672:
      *done = true;
      return py_eo_go<PPY672, 4>(g, tw, S, inv, st);
    case 756:
      *done = true;
      return py_eo_go<PPY756, 4>(g, tw, S, inv, st);
    case 882:
      *done = true;
      return py_eo_go<PPY882, 4>(g, tw, S, inv, st);
    case 1008:
      *done = true;
      return py_eo_go<PPY1008, 2>(g, tw, S, inv, st);
    case 1152:
      *done = true;
      return py_eo_go<PPY1152, 2>(g, tw, S, inv, st);
    case 1296:
      *done = true;
      return py_eo_go<PPY1296, 2>(g, tw, S, inv, st);
    case 1470:
      *done = true;
      return py_eo_go<PPY1470, 2>(g, tw, S, inv, st);
    case 1680:
      *done = true;
      return py_eo_go<PPY1680, 2>(g, tw, S, inv, st);
    case 1890:
      *done = true;
      return py_eo_go<PPY1890, 2>(g, tw, S, inv, st);
    default:
      return 0;
  }
}

}  // namespace cdx
