// Registry of the compile-time specialised transform lengths.
//
// CDX_SPLAN_LIST gives each registered length and its radices (their
// product is the length; radices up to 32 points run in registers).  The
// per-axis lists say for which pass kernels a length is instantiated and
// with which tile: y passes with V rows, z passes with W columns.  Other
// lengths use the generic engine.  These passes work on the plain spectrum
// layout, which the tensor-core x passes and the x lengths without a paired
// plan (fft_pair.cuh) use.
#pragma once

#include <vector>

#include "fft_static.cuh"
#include "static_plans_gen.cuh"

#define CDX_SPLAN_LIST(F) \
  F(32, 8, 4)             \
  F(64, 8, 8)             \
  F(100, 10, 10)          \
  F(128, 16, 8)           \
  F(256, 16, 16)          \
  F(512, 32, 16)          \
  F(756, 9, 12, 7)        \
  F(1024, 32, 32)         \
  F(1620, 15, 12, 9)      \
  CDX_GEN_SPLANS(F)

// y entries: F(L, rows per block, extra registers of the launch bounds,
// padding periods of the two stage layouts of a three-radix plan)
#define CDX_Y_PLANS(F) \
  F(128, 16, 0, 0, 0) F(256, 8, 0, 0, 0) F(512, 4, 0, 0, 0) F(1024, 4, 0, 0, 0) CDX_GEN_Y_PLANS(F)
#define CDX_Z_PLANS(F) F(32, 16) F(64, 16) F(100, 16) F(128, 16) F(256, 16)
// generated z plans (types SPZ<L>, twiddles FftLen::gzdev): F(L, columns
// per block, extra registers); instantiated for radially averaged OTFs only
#define CDX_Z_GEN_PLANS(F) CDX_GEN_Z_PLANS(F)

namespace cdx {

#define CDX_DEF_SPLAN(L, ...) using SP##L = SPlan<L, __VA_ARGS__>;
CDX_SPLAN_LIST(CDX_DEF_SPLAN)
#undef CDX_DEF_SPLAN

#define CDX_DEF_GZPLAN(L, ...) using SPZ##L = SPlan<L, __VA_ARGS__>;
CDX_GEN_Z_SPLANS(CDX_DEF_GZPLAN)
#undef CDX_DEF_GZPLAN

// Radices of the registered plan for length L (false when L is not registered).
inline bool static_radices(int L, std::vector<int>& rad) {
  switch (L) {
#define CDX_RAD_CASE(LL, ...) \
  case LL:                    \
    rad = {__VA_ARGS__};      \
    return true;
    CDX_SPLAN_LIST(CDX_RAD_CASE)
#undef CDX_RAD_CASE
    default:
      return false;
  }
}

// Radices of the generated z-pass plan for length L (false when it has none).
inline bool gz_radices(int L, std::vector<int>& rad) {
  switch (L) {
#define CDX_GZ_CASE(LL, ...) \
  case LL:                   \
    rad = {__VA_ARGS__};     \
    return true;
    CDX_GEN_Z_SPLANS(CDX_GZ_CASE)
#undef CDX_GZ_CASE
    default:
      return false;
  }
}

}  // namespace cdx
