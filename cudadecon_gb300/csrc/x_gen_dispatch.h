// Generated by cudadecon_gb300/gen_plans.py (do not edit): dispatch of the
// paired passes to the units decon_{x,y,z}_gen_<k>.cu.  Each function sets
// *done when its length has a plan.
#pragma once

#include "pair_layout.cuh"

namespace cdx {

int pxgen_fwd_0(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_1(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_2(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_3(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_4(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_5(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_6(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_7(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_8(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_9(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_10(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_11(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_12(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_13(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_14(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_15(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_16(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_17(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_18(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_fwd_19(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done);
int pxgen_ratio_0(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_1(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_2(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_3(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_4(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_5(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_6(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_7(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_8(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_9(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_10(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_11(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_12(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_13(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_14(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_15(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_16(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_17(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_18(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_ratio_19(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done);
int pxgen_update_0(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_1(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_2(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_3(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_4(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_5(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_6(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_7(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_8(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_9(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_10(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_11(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_12(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_13(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_14(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_15(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_16(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_17(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_18(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pxgen_update_19(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done);
int pygen_0(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_1(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_2(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_3(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_4(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_5(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_6(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pygen_7(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done);
int pzgen_0(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_1(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_2(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_3(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_4(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_5(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_6(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);
int pzgen_7(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done);

inline int pxgen_fwd(const PairGeom& g, const float2* tw, const float* X, float* Xm1, const float* lam, int predict, float bg, float2* S, cudaStream_t st, bool* done) {
  int rc = 0;
  *done = false;
  if ((rc = pxgen_fwd_0(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_1(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_2(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_3(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_4(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_5(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_6(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_7(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_8(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_9(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_10(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_11(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_12(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_13(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_14(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_15(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_16(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_17(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_18(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  if ((rc = pxgen_fwd_19(g, tw, X, Xm1, lam, predict, bg, S, st, done)) || *done) return rc;
  return 0;
}

inline int pxgen_ratio(const PairGeom& g, const float2* tw, float2* S, const float* raw, const float* mean, float eps, cudaStream_t st, bool* done) {
  int rc = 0;
  *done = false;
  if ((rc = pxgen_ratio_0(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_1(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_2(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_3(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_4(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_5(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_6(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_7(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_8(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_9(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_10(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_11(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_12(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_13(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_14(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_15(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_16(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_17(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_18(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_ratio_19(g, tw, S, raw, mean, eps, st, done)) || *done) return rc;
  return 0;
}

inline int pxgen_update(const PairGeom& g, const float2* tw, const float2* S, const float* Y, float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps, cudaStream_t st, bool* done) {
  int rc = 0;
  *done = false;
  if ((rc = pxgen_update_0(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_1(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_2(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_3(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_4(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_5(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_6(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_7(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_8(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_9(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_10(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_11(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_12(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_13(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_14(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_15(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_16(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_17(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_18(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  if ((rc = pxgen_update_19(g, tw, S, Y, Xout, G, dots, w, lam_next, eps, st, done)) || *done) return rc;
  return 0;
}

inline int pygen(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st, bool* done) {
  int rc = 0;
  *done = false;
  if ((rc = pygen_0(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_1(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_2(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_3(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_4(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_5(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_6(g, tw, S, inv, st, done)) || *done) return rc;
  if ((rc = pygen_7(g, tw, S, inv, st, done)) || *done) return rc;
  return 0;
}

inline int pzgen(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj, cudaStream_t st, bool fwd_only, bool* done) {
  int rc = 0;
  *done = false;
  if ((rc = pzgen_0(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_1(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_2(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_3(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_4(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_5(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_6(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  if ((rc = pzgen_7(g, tw, S, otf, conj, st, fwd_only, done)) || *done) return rc;
  return 0;
}

}  // namespace cdx
