// The x passes on row pairs (plain form): forward with the prediction
// prologue, inverse with the RL ratio and the forward transform of the ratio,
// inverse with the estimate update and the dot products.  Templates over the
// plan (fft_pair.cuh) and the pairs per block; the generated units
// decon_x_gen_*.cu instantiate them for every length with a plan.
//
// A block owns NQ pairs of complex rows (4 NQ real rows) of a slice.  Stage A
// reads and writes the packed spectrum, whose NQ slots of one kx are
// contiguous, straight from registers; stage C reads and writes the real rows
// the same way (consecutive threads on consecutive x).  The shared tile only
// carries the data between the stages: 2 round trips a transform at three
// radices where staging, split and merge took 7 for the two of the ratio
// pass.  Stage 100 x 256 x 756 on a GB300, x ratio: 16.1 M shared wavefronts
// and 74 M warp instructions before.
#pragma once

#include "decon_common.cuh"
#include "fft_pair.cuh"
#include "pair_layout.cuh"

namespace cdx {

// The four real rows of pair m of slice z: offset of row 2m, and whether the
// two rows H further exist.
struct RowQuad {
  long long o;  // row 2m
  long long h;  // H rows further
  bool v2, v3;
};
__device__ __forceinline__ RowQuad row_quad(const PairGeom& g, int z, int m) {
  RowQuad r;
  r.o = ((long long)z * g.zrows + 2 * m) * g.nx;
  r.h = (long long)g.H * g.nx;
  r.v2 = 2 * m + g.H < g.ny;
  r.v3 = 2 * m + 1 + g.H < g.ny;
  return r;
}
// A block's rows in shared memory, copied with cp.async at its start (they are
// read once an iteration: evict-first in L2) and read by stage C: rows 2 m0 ..
// 2 m0 + 2 NQ - 1 of each half, the halves one after the other.
template <int NQ>
__device__ __forceinline__ void prefetch_rows(const PairGeom& g, float* dst, const float* src,
                                              int z, int m0) {
  const long long o = ((long long)z * g.zrows + 2 * m0) * g.nx;
  const int n0 = max(0, min(2 * NQ, g.H - 2 * m0)), n1 = max(0, min(n0, g.ny - g.H - 2 * m0));
  prefetch_floats(dst, src + o, n0 * g.nx, true);
  prefetch_floats(dst + 2 * NQ * g.nx, src + o + (long long)g.H * g.nx, n1 * g.nx, true);
  if (n0 + n1 < 4 * NQ) {  // rows past the volume read as 0
    for (int i = n0 * g.nx + threadIdx.x; i < 2 * NQ * g.nx; i += blockDim.x) dst[i] = 0.f;
    for (int i = n1 * g.nx + threadIdx.x; i < 2 * NQ * g.nx; i += blockDim.x)
      dst[2 * NQ * g.nx + i] = 0.f;
  }
}
// The rows of a block at p as two runs of floats (one per half); whether both
// start and end on 16 bytes.
template <int NQ>
struct RowRuns {
  long long o, h;  // first run, distance to the second
  int n0, n1;      // floats
  __device__ __forceinline__ RowRuns(const PairGeom& g, int z, int m0) {
    o = ((long long)z * g.zrows + 2 * m0) * g.nx;
    h = (long long)g.H * g.nx;
    const int r0 = max(0, min(2 * NQ, g.H - 2 * m0));
    n0 = r0 * g.nx;
    n1 = max(0, min(r0, g.ny - g.H - 2 * m0)) * g.nx;
  }
  __device__ __forceinline__ bool vec(const float* p) const {
    const unsigned long long a = reinterpret_cast<unsigned long long>(p + o);
    return ((a | (unsigned long long)(4 * h) | (unsigned)(4 * n0) | (unsigned)(4 * n1)) & 15) == 0;
  }
};

// Sample x of the four rows of pair q from such a copy.
template <int NQ, int L>
__device__ __forceinline__ C2 lds_rows(const float* rows, int q, int x) {
  const float* p = rows + 2 * q * L + x;
  return {make_float2(p[0], p[L]), make_float2(p[2 * NQ * L], p[2 * NQ * L + L])};
}
template <int NQ, int L>
__device__ __forceinline__ void sts_rows(float* rows, int q, int x, const C2& v) {
  float* p = rows + 2 * q * L + x;
  p[0] = v.re.x;
  p[L] = v.re.y;
  p[2 * NQ * L] = v.im.x;
  p[2 * NQ * L + L] = v.im.y;
}
template <bool STREAM>
__device__ __forceinline__ void st_rows(float* p, const RowQuad& q, int nx, const C2& x) {
  auto st = [](float* a, float v) {
    if (STREAM) __stcs(a, v);
    else *a = v;
  };
  st(p, x.re.x);
  st(p + nx, x.re.y);
  if (q.v2) st(p + q.h, x.im.x);
  if (q.v3) st(p + q.h + nx, x.im.y);
}

// Addresses of the packed spectrum elements e = j + r L/Q0 of pair m: Z[e] for
// e <= L/2, the mirrored row's second half beyond.  Neighbouring e are 4 slots
// apart, so every r is a constant offset.
template <class PL>
struct SpecPtr {
  float4 *lo, *hi;
  int j;
  __device__ __forceinline__ SpecPtr(const PairGeom& g, float4* S, int z, int m, int j_) : j(j_) {
    lo = S + g.slot(j, z, m);
    hi = S + g.slot(PL::L - j, z, g.hp + m);
  }
  template <int R>
  __device__ __forceinline__ float4* at() const {
    constexpr int e0 = R * PL::KA;
    if constexpr (e0 + PL::KA - 1 <= PL::L / 2) return lo + 4 * e0;
    else if constexpr (e0 > PL::L / 2) return hi - 4 * e0;
    else return e0 + j <= PL::L / 2 ? lo + 4 * e0 : hi - 4 * e0;
  }
};

// Shared memory: twiddles, tile, then the copies of the block's rows (R
// arrays of 4 NQ rows).
template <class PL, int NQ>
struct PX {
  static constexpr int T = PL::threads(NQ);
  static constexpr int kTile = NQ * PL::VS;         // float4s
  static constexpr int kRows = (4 * NQ * PL::L + 3) & ~3;  // floats
  // Registers a thread to plan with: the widest butterfly, or in stage C of
  // the ratio and update passes its values and the rows' (8 Q2).  12 more for
  // 1620 (one block per SM instead of two) took x ratio from 1544 to 2103 us,
  // 16 fewer for 810 (spills) x update from 379 to 508 us.
  static constexpr int kRegs =
      8 * PL::Q2 + 12 > 4 * PL::qmax() + 24 ? 8 * PL::Q2 + 12 : 4 * PL::qmax() + 24;
  static constexpr int by_regs(int regs) {
    const int b = 65536 / (T * regs), most = 2048 / T;
    return b < 1 ? 1 : (b < most ? b : most);
  }
  static constexpr int blocks_with(int tw) {
    return resident_blocks(by_regs(kRegs), sizeof(float2) * tw + sizeof(float4) * kTile +
                                               sizeof(float) * kRows);
  }
  // Stage C's twiddles stay in global memory (L1) where their copy would cost
  // a block per SM (its table is L - L/Q2 of the L entries)
  static constexpr int kTwAll = PL::L + (PL::L & 1), kTwB = PL::KC + (PL::KC & 1);
  static constexpr bool kGlobalTw = blocks_with(kTwAll) < blocks_with(kTwB);
  static constexpr int kTw = kGlobalTw ? kTwB : kTwAll;  // float2s
  static constexpr int kBlocks = blocks_with(kTw);
  // its twiddle table: tw in global or stw in shared memory
  __device__ __forceinline__ static const float2* tw_c(const float2* tw, const float2* stw) {
    return kGlobalTw ? tw : stw;
  }
  static constexpr size_t smem(int R) {
    return sizeof(float2) * kTw + sizeof(float4) * kTile + sizeof(float) * kRows * R;
  }
  __device__ __forceinline__ static float4* tile(float2* sm) {
    return reinterpret_cast<float4*>(sm + kTw);
  }
  __device__ __forceinline__ static float* rows(float2* sm, int i) {
    return reinterpret_cast<float*>(tile(sm) + kTile) + i * kRows;
  }
  // forward pass: the rows are read before the tile is written and share its
  // memory, which lets one block more fit an SM
  static constexpr size_t smem_fwd(int R) {
    const size_t rows = sizeof(float) * kRows * R, tile = sizeof(float4) * kTile;
    return sizeof(float2) * kTw + (rows > tile ? rows : tile);
  }
  static constexpr int kBlocksFwd = resident_blocks(by_regs(24 + 4 * PL::qmax()), smem_fwd(2));
  static constexpr int kRegsUpd = 24 + 4 * PL::qmax() > 64 ? 24 + 4 * PL::qmax() : 64;
  // Row arrays (Y, then G) that the update pass of a large volume has in shared
  // memory: as many as fit a block and leave 512 threads an SM, or all that fit
  // beside the blocks there are without them.  One block of two lost 27% of the
  // pass at 800 columns, two of four (448 threads) 9% at 756, three of eight
  // (192) 13% at 625; three of four (672) gained 6% at 700, four of eight (512)
  // 3% at 512.  Against the rule 567 (+3%) and 980 (+1.6% of the pass) lost.
  static constexpr int blocks_upd(int R) { return resident_blocks(by_regs(kRegsUpd), smem(R)); }
  static constexpr bool stages(int R) {
    return blocks_upd(R) > 0 && (blocks_upd(R) * T >= 512 || blocks_upd(R) == blocks_upd(0));
  }
  static constexpr int kStaged = stages(2) ? 2 : (stages(1) ? 1 : 0);
  __device__ __forceinline__ static float* rows_fwd(float2* sm, int i) {
    return reinterpret_cast<float*>(tile(sm)) + i * kRows;
  }
};

// Rows in registers (x[r] = sample k + r KC) -> stages C, B, A forward ->
// packed spectrum in S.  The tile's C addresses are free to write on entry.
template <class PL, int NQ>
__device__ __forceinline__ void rows_to_spec(const PairGeom& g, C2* x, float4* sm,
                                             const float2* tw, const float2* stw, float4* S, int z,
                                             int m0) {
  const int idx = threadIdx.x;
  if (idx < NQ * PL::KC) {
    const int q = idx / PL::KC, k = idx - q * PL::KC;
    using P = PX<PL, NQ>;
    butterfly<PL::Q2, PL::KC, false, true, P::kGlobalTw>(x, P::tw_c(tw, stw), k);
    float4* p = sm + q * PL::VS + pos_c<PL>(k);
#pragma unroll
    for (int r = 0; r < PL::Q2; ++r) stp(p + r, x[r]);
  }
  __syncthreads();
  stage_b<PL, NQ, false, true>(sm, stw);
  grid_dep_launch_small();
  const int j = idx / NQ, q = idx - j * NQ;
  if (j < PL::KA && 2 * (m0 + q) < g.H) {
    const float4* p = sm + q * PL::VS + j;
    C2 y[PL::Q0];
#pragma unroll
    for (int r = 0; r < PL::Q0; ++r) y[r] = ldp(p + r * PL::S0);
    PDft<PL::Q0, false>::run(y);
    const SpecPtr<PL> sp(g, S, z, m0 + q, j);
    static_for<PL::Q0>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      *sp.template at<r>() = pack(y[r]);
    });
  }
}

// Packed spectrum -> stages A and B inverse; the tile then holds stage C's
// inputs.  Waits for the thread's async copies (twiddles, rows), all but
// the last KEEP groups, before its first barrier; then() runs before its last.
template <class PL, int NQ, bool LAST, int KEEP = 0, class Then>
__device__ __forceinline__ void spec_to_tile(const PairGeom& g, float4* sm, const float2* stw,
                                             float4* S, int z, int m0, const Then& then) {
  const int idx = threadIdx.x;
  const int j = idx / NQ, q = idx - j * NQ;
  if (j < PL::KA) {
    C2 y[PL::Q0];
    if (2 * (m0 + q) < g.H) {
      const SpecPtr<PL> sp(g, S, z, m0 + q, j);
      static_for<PL::Q0>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        const float4 v = LAST ? __ldcs(sp.template at<r>()) : *sp.template at<r>();
        y[r] = {make_float2(v.x, v.y), make_float2(v.z, v.w)};
      });
    } else {
#pragma unroll
      for (int r = 0; r < PL::Q0; ++r) y[r] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    }
    PDft<PL::Q0, true>::run(y);
    float4* p = sm + q * PL::VS + j;
#pragma unroll
    for (int r = 0; r < PL::Q0; ++r) stp(p + r * PL::S0, y[r]);
  }
  cp_async_wait<KEEP>();
  if constexpr (PL::Q1 == 1) then();
  __syncthreads();
  stage_b<PL, NQ, true, false>(sm, stw, then);
}

// ---------------------------------------------------------------- forward
template <class PL, int NQ>
__global__ void __launch_bounds__(PX<PL, NQ>::T, PX<PL, NQ>::kBlocksFwd)
k_px_fwd(PairGeom g, const float2* __restrict__ tw, const float* X, float* Xm1, const float* lamp,
         int predict, float bg, float4* S) {
  using P = PX<PL, NQ>;
  extern __shared__ __align__(16) float2 smem[];
  float2* stw = smem;
  float4* sm = P::tile(smem);
  const int z = blockIdx.y, m0 = blockIdx.x * NQ;
  copy_twiddles<P::kTw>(tw, stw);
  if (!predict) grid_dep_wait();
  // predict: the previous kernel only sums lambda; it passed its own wait, so
  // the update pass before it, which wrote these rows, has completed
  prefetch_rows<NQ>(g, P::rows_fwd(smem, 0), X, z, m0);
  if (predict) prefetch_rows<NQ>(g, P::rows_fwd(smem, 1), Xm1, z, m0);
  cp_async_commit();
  if (predict) grid_dep_wait();
  const int idx = threadIdx.x;
  const int q = idx / PL::KC, k = idx - q * PL::KC;
  const RowQuad rq = row_quad(g, z, m0 + q);
  // (a plain load: the read-only path promises that nobody writes while the kernel
  // is resident; past L1 it takes every warp to one L2 line)
  const float2 lam = dup2(predict ? *lamp : 0.f);
  cp_async_wait_all();
  __syncthreads();
  C2 x[PL::Q2];
  if (q < NQ && 2 * (m0 + q) < g.H) {
#pragma unroll
    for (int r = 0; r < PL::Q2; ++r)
      x[r] = lds_rows<NQ, PL::L>(P::rows_fwd(smem, 0), q, k + r * PL::KC);
    if (predict) {
      // prediction of updatePrediction_kernel (RLgpuImpl.cu:658-666), written
      // over X_{k-1}
      float* pm = Xm1 + rq.o + k;
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r) {
        const C2 o = lds_rows<NQ, PL::L>(P::rows_fwd(smem, 1), q, k + r * PL::KC);
        x[r].re = relu2(fma2(lam, sub2(x[r].re, o.re), x[r].re));
        x[r].im = relu2(fma2(lam, sub2(x[r].im, o.im), x[r].im));
        st_rows<true>(pm + r * PL::KC, rq, PL::L, x[r]);
      }
    } else if (bg != 0.f) {  // rows past the volume stay 0
      const float2 im = make_float2(rq.v2 ? -bg : 0.f, rq.v3 ? -bg : 0.f);
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r) x[r] = {add2(x[r].re, dup2(-bg)), add2(x[r].im, im)};
    }
  } else {
#pragma unroll
    for (int r = 0; r < PL::Q2; ++r) x[r] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  }
  __syncthreads();
  rows_to_spec<PL, NQ>(g, x, sm, tw, stw, S, z, m0);
}

// ---------------------------------------------------------------- ratio
// The RL ratio of the reference's LRcore_kernel (RLgpuImpl.cu:416-434), raw / c
// + eps clamped to +-10, for the two lanes of c and raw in the range that
// ratio_range accepts.  The quotient by Newton's method on the reciprocal with
// one residual correction of the quotient (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990), two
// lanes per instruction: 14 instructions a pair where two IEEE divisions with
// their selects took about 50, over half of the pass's inner stage.
__device__ __forceinline__ float2 rl_ratio2(float2 c, float2 raw, float eps) {
  float2 r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(c.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(c.y));
  const float2 nc = neg2(c);
  r = fma2(r, fma2(nc, r, dup2(1.f)), r);
  float2 u = mul2(raw, r);
  u = add2(fma2(fma2(nc, u, raw), r, u), dup2(eps));
  return make_float2(fmaxf(fminf(u.x, 10.f), -10.f), fmaxf(fminf(u.y, 10.f), -10.f));
}
// Smallest and largest magnitude of the c and largest of the raw values seen;
// NaN propagates.  Zero, tiny, huge, infinite and NaN operands fall outside:
// a thread that holds one takes the IEEE division for all of its values.
struct RatioRange {
  float lo = 1.f, hi = 1.f, top = 0.f;
  __device__ __forceinline__ static float min_nan(float a, float b) {
    float d;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
  }
  __device__ __forceinline__ static float max_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
  }
  __device__ __forceinline__ void see(float2 c, float2 raw) {
    lo = min_nan(lo, min_nan(fabsf(c.x), fabsf(c.y)));
    hi = max_nan(hi, max_nan(fabsf(c.x), fabsf(c.y)));
    top = max_nan(top, max_nan(fabsf(raw.x), fabsf(raw.y)));
  }
  __device__ __forceinline__ bool plain() const {
    return lo >= 0x1p-60f && hi <= 0x1p60f && top <= 0x1p60f;
  }
};

template <class PL, int NQ>
__global__ void __launch_bounds__(PX<PL, NQ>::T, PX<PL, NQ>::kBlocks)
k_px_ratio(PairGeom g, const float2* __restrict__ tw, float4* S, const float* __restrict__ raw,
           const float* mean, float eps) {
  using P = PX<PL, NQ>;
  extern __shared__ __align__(16) float2 smem[];
  float2* stw = smem;
  float4* sm = P::tile(smem);
  const int z = blockIdx.y, m0 = blockIdx.x * NQ;
  copy_twiddles<P::kTw>(tw, stw);
  prefetch_rows<NQ>(g, P::rows(smem, 0), raw, z, m0);  // written before the iterations
  cp_async_commit();
  grid_dep_wait();
  float off = 0.f;
  spec_to_tile<PL, NQ, false>(g, sm, stw, S, z, m0, [&] { off = -__ldg(mean); });
  const int idx = threadIdx.x;
  const int q = idx / PL::KC, k = idx - q * PL::KC;
  C2 x[PL::Q2];
  if (q < NQ) {
    const RowQuad rq = row_quad(g, z, m0 + q);
    const float4* p = sm + q * PL::VS + pos_c<PL>(k);
#pragma unroll
    for (int r = 0; r < PL::Q2; ++r) x[r] = ldp(p + r);
    butterfly<PL::Q2, PL::KC, true, false, P::kGlobalTw>(x, P::tw_c(tw, stw), k);
    C2 d[PL::Q2];
    RatioRange range;
#pragma unroll
    for (int r = 0; r < PL::Q2; ++r) {
      d[r] = lds_rows<NQ, PL::L>(P::rows(smem, 0), q, k + r * PL::KC);
      range.see(x[r].re, d[r].re);
      range.see(x[r].im, d[r].im);
    }
    if (range.plain()) {
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r)
        x[r] = {rl_ratio2(x[r].re, d[r].re, eps), rl_ratio2(x[r].im, d[r].im, eps)};
    } else {
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r) {
        x[r].re = make_float2(rl_ratio(x[r].re.x, d[r].re.x, eps), rl_ratio(x[r].re.y, d[r].re.y, eps));
        x[r].im = make_float2(rl_ratio(x[r].im.x, d[r].im.x, eps), rl_ratio(x[r].im.y, d[r].im.y, eps));
      }
    }
    // The ratio goes on less a constant m: what the second convolution does to a
    // constant is known (m times the OTF at frequency 0, added back by the update
    // pass), and its transforms round in proportion to the root mean square of
    // what they are given.  That is smallest, and never more than the ratio's own,
    // with m the ratio's mean.  The mean of an earlier iteration's ratio is close to
    // it and at hand in the z pass, as frequency 0 of that spectrum (rl_loop).
    // The ratio is about 1 where the image is above the background and about 0
    // where it is empty, so m lies near 1 in crowded images and near 0 in dark
    // ones; a fixed 1 took the error of images with nine tenths of zeros up 1.5
    // to 4 times.
#pragma unroll
    for (int r = 0; r < PL::Q2; ++r) x[r] = {add2(x[r].re, dup2(off)), add2(x[r].im, dup2(off))};
    if (!(rq.v2 && rq.v3)) {
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r) {
        if (!rq.v2) x[r].im.x = 0.f;
        if (!rq.v3) x[r].im.y = 0.f;
      }
    }
  }
  rows_to_spec<PL, NQ>(g, x, sm, tw, stw, S, z, m0);
}

// ---------------------------------------------------------------- update
__device__ __forceinline__ void l2_prefetch(const float* p, int bytes) {
  if (bytes > 0)
    asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(p), "r"(bytes),
                 "l"(l2_evict_first_policy())
                 : "memory");
}
// Float-float sums of two lanes at once (acc_add per lane).
__device__ __forceinline__ void acc_add2(float2& hi, float2& lo, float2 p) {
  const float2 s = add2(hi, p);
  const float2 bb = sub2(s, hi);
  const float2 err = add2(sub2(hi, sub2(s, bb)), sub2(p, bb));
  hi = s;
  lo = add2(lo, err);
}

// Y == nullptr: the plain inverse transform, written to Xout; otherwise *addp is
// what the convolution made of the constant that k_px_ratio took off.
template <class PL, int NQ, int STAGED>
__global__ void __launch_bounds__(PX<PL, NQ>::T, PX<PL, NQ>::blocks_upd(STAGED))
k_px_update(PairGeom g, const float2* __restrict__ tw, float4* S, const float* Y, float* Xout,
            float* G, int dots, float4* partials, const float* addp) {
  using P = PX<PL, NQ>;
  extern __shared__ __align__(16) float2 smem[];
  __shared__ float4 red[32];
  float2* stw = smem;
  float4* sm = P::tile(smem);
  const int z = blockIdx.y, m0 = blockIdx.x * NQ;
  copy_twiddles<P::kTw>(tw, stw);
  cp_async_commit();
  const RowRuns<NQ> runs(g, z, m0);
  // (the halves of the rows in shared memory are 2 NQ L floats apart)
  const bool vec = NQ * PL::L % 2 == 0 && Y && runs.vec(Xout) && runs.vec(Y) && runs.vec(G);
  // Y and G were written by kernels that completed before the previous pass
  // passed its own wait: ask for them now, in shared memory (the first STAGED of
  // them) or in L2 (16-byte walk only: the prefetch takes whole 16-byte units)
  if constexpr (STAGED > 0) {
    prefetch_rows<NQ>(g, P::rows(smem, 0), Y, z, m0);
    if (STAGED > 1 && dots) prefetch_rows<NQ>(g, P::rows(smem, 1), G, z, m0);
    cp_async_commit();
  }
  if (vec && threadIdx.x == 0) {
    if (STAGED < 1) {
      l2_prefetch(Y + runs.o, 4 * runs.n0);
      l2_prefetch(Y + runs.o + runs.h, 4 * runs.n1);
    }
    if (STAGED < 2 && dots) {
      l2_prefetch(G + runs.o, 4 * runs.n0);
      l2_prefetch(G + runs.o + runs.h, 4 * runs.n1);
    }
  }
  grid_dep_wait();
  spec_to_tile<PL, NQ, true, STAGED ? 1 : 0>(g, sm, stw, S, z, m0, [] {});
  // stage C, its samples as rows over the tile (all of it read by then)
  const int idx = threadIdx.x;
  const int q = idx / PL::KC, k = idx - q * PL::KC;
  const bool in = q < NQ && 2 * (m0 + q) < g.H;
  float* rows = reinterpret_cast<float*>(sm);
  static_assert(P::kRows <= 4 * P::kTile, "the rows fit the tile");
  {
    C2 x[PL::Q2];
    if (in) {
      const float4* p = sm + q * PL::VS + pos_c<PL>(k);
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r) x[r] = ldp(p + r);
    }
    __syncthreads();
    if (in) {
      butterfly<PL::Q2, PL::KC, true, false, P::kGlobalTw>(x, P::tw_c(tw, stw), k);
#pragma unroll
      for (int r = 0; r < PL::Q2; ++r) sts_rows<NQ, PL::L>(rows, q, k + r * PL::KC, x[r]);
    }
  }
  if constexpr (STAGED > 0) cp_async_wait_all();
  __syncthreads();
  grid_dep_launch_small();
  // Estimate update (currEstimate_kernel + currPrevDiff_kernel,
  // RLgpuImpl.cu:462-470, 501-508) and the Biggs-Andrews dot products of
  // innerProduct_kernel (RLgpuImpl.cu:571-633), as one walk over the rows,
  // 16 bytes an access where they are aligned.  X is read next
  // by the x forward pass (kept in L2), G only by the next iteration's update.
  float2 s1h = make_float2(0.f, 0.f), s1l = s1h, s2h = s1h, s2l = s1h;
  const float2 add = dup2(Y ? __ldg(addp) : 0.f);
  auto update = [&](float2 cc, float2 y, float2 go, float2& xn, float2& gn) {
    xn = relu2(mul2(add2(cc, add), y));
    gn = sub2(xn, y);
    if (dots) {
      acc_add2(s1h, s1l, mul2(gn, go));
      acc_add2(s2h, s2l, mul2(go, go));
    }
  };
  const int total = runs.n0 + runs.n1;
  if (!Y) {  // plain transform
    for (int e = idx; e < total; e += P::T) {
      const bool second = e >= runs.n0;
      const int f = second ? e - runs.n0 : e;
      Xout[runs.o + (second ? runs.h : 0) + f] = rows[f + (second ? 2 * NQ * PL::L : 0)];
    }
    return;
  }
  if (vec) {
    constexpr int U = 2;  // accesses in flight per thread and array
    // from the block's first row, which is what lies on 16 bytes
    const int n0 = runs.n0 >> 2, n = total >> 2, o1 = (int)(runs.h >> 2) - n0;
    const float4* Y4 = reinterpret_cast<const float4*>(Y + runs.o);
    float4* X4 = reinterpret_cast<float4*>(Xout + runs.o);
    float4* G4 = reinterpret_cast<float4*>(G + runs.o);
    const float4* r4 = reinterpret_cast<const float4*>(rows);
    for (int i0 = idx; i0 < n; i0 += U * P::T) {
      float4 y[U], go[U];
      int at[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * P::T;
        at[u] = i < n0 ? i : o1 + i;
        if (i < n) {
          const int f = i < n0 ? i : i - n0 + NQ * PL::L / 2;
          y[u] = STAGED > 0 ? reinterpret_cast<const float4*>(P::rows(smem, 0))[f]
                            : __ldcs(Y4 + at[u]);
          if (dots)
            go[u] = STAGED > 1 ? reinterpret_cast<const float4*>(P::rows(smem, 1))[f]
                               : __ldcs(G4 + at[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * P::T;
        if (i >= n) break;
        const float4 c = r4[i < n0 ? i : i - n0 + NQ * PL::L / 2];
        float2 xa, xb, ga, gb;
        update(make_float2(c.x, c.y), make_float2(y[u].x, y[u].y), make_float2(go[u].x, go[u].y), xa,
               ga);
        update(make_float2(c.z, c.w), make_float2(y[u].z, y[u].w), make_float2(go[u].z, go[u].w), xb,
               gb);
        X4[at[u]] = make_float4(xa.x, xa.y, xb.x, xb.y);
        __stcs(G4 + at[u], make_float4(ga.x, ga.y, gb.x, gb.y));
      }
    }
  } else {
    constexpr int U = 4;
    const long long o1 = runs.o + runs.h - runs.n0;
    for (int i0 = idx; i0 < total; i0 += U * P::T) {
      float2 y[U / 2], go[U / 2];  // two accesses a lane pair
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * P::T;
        float v = 0.f, w = 0.f;
        if (i < total) {
          const long long at = (i < runs.n0 ? runs.o : o1) + i;
          const int f = i < runs.n0 ? i : i - runs.n0 + 2 * NQ * PL::L;
          v = STAGED > 0 ? P::rows(smem, 0)[f] : __ldcs(Y + at);
          if (dots) w = STAGED > 1 ? P::rows(smem, 1)[f] : __ldcs(G + at);
        }
        (u & 1 ? y[u / 2].y : y[u / 2].x) = v;
        (u & 1 ? go[u / 2].y : go[u / 2].x) = w;
      }
#pragma unroll
      for (int u = 0; u < U; u += 2) {
        const int i = i0 + u * P::T, j = i + P::T;
        if (i >= total) break;
        auto row = [&](int e) { return rows[e < runs.n0 ? e : e - runs.n0 + 2 * NQ * PL::L]; };
        float2 xn, gn;
        update(make_float2(row(i), j < total ? row(j) : 0.f), y[u / 2], go[u / 2], xn, gn);
        const long long at = (i < runs.n0 ? runs.o : o1) + i;
        Xout[at] = xn.x;
        __stcs(G + at, gn.x);
        if (j < total) {
          const long long bt = (j < runs.n0 ? runs.o : o1) + j;
          Xout[bt] = xn.y;
          __stcs(G + bt, gn.y);
        }
      }
    }
  }
  if (!dots) return;
  float ah = s1h.x, al = s1l.x, bh = s2h.x, bl = s2l.x;
  acc_add(ah, al, s1h.y);
  al = __fadd_rn(al, s1l.y);
  acc_add(bh, bl, s2h.y);
  bl = __fadd_rn(bl, s2l.y);
  const float4 sum = block_sum2_ff(ah, al, bh, bl, red);
  if (threadIdx.x == 0) partials[blockIdx.y * gridDim.x + blockIdx.x] = sum;
}

// ---------------------------------------------------------------- launches
template <class PL, int NQ>
static int px_fwd_go(const PairGeom& g, const float2* tw, const float* X, float* Xm1,
                     const float* lam, int predict, float bg, float2* S, cudaStream_t st) {
  using P = PX<PL, NQ>;
  static_assert(P::kBlocksFwd > 0, "an SM holds a block");
  auto kern = k_px_fwd<PL, NQ>;
  const size_t smem = P::smem_fwd(predict ? 2 : 1);
  if (int rc = smem_optin(kern, smem)) return rc;
  CDX_CHECK(launch_pdl(kern, dim3(ceil_div(g.H / 2, NQ), g.nz), dim3(P::T), smem, st, g, tw, X,
                       Xm1, lam, predict, bg, reinterpret_cast<float4*>(S)));
  CDX_LAUNCH_CHECK("k_px_fwd");
  return 0;
}

template <class PL, int NQ>
static int px_ratio_go(const PairGeom& g, const float2* tw, float2* S, const float* raw,
                       const float* mean, float eps, cudaStream_t st) {
  using P = PX<PL, NQ>;
  static_assert(P::kBlocks > 0, "an SM holds a block");
  auto kern = k_px_ratio<PL, NQ>;
  const size_t smem = P::smem(1);
  if (int rc = smem_optin(kern, smem)) return rc;
  CDX_CHECK(launch_pdl(kern, dim3(ceil_div(g.H / 2, NQ), g.nz), dim3(P::T), smem, st, g, tw,
                       reinterpret_cast<float4*>(S), raw, mean, eps));
  CDX_LAUNCH_CHECK("k_px_ratio");
  return 0;
}

template <class PL, int NQ>
static int px_update_go(const PairGeom& g, const float2* tw, const float2* S, const float* Y,
                        float* Xout, float* G, int dots, RLWork* w, float* lam_next, float eps,
                        cudaStream_t st) {
  using P = PX<PL, NQ>;
  static_assert(P::blocks_upd(0) > 0 && P::blocks_upd(P::kStaged) > 0, "an SM holds a block");
  const dim3 grid(ceil_div(g.H / 2, NQ), g.nz);
  const int nblk = grid.x * grid.y;
  if (dots && nblk > w->max_blocks) {
    set_error("launch_x_inv_update", "partials buffer too small");
    return cudaErrorInvalidValue;
  }
  // Y and G come through shared memory where the arrays of an iteration do not
  // stay in L2, which takes about 6 M voxels: the copies then run under the
  // transform, where a prefetch into L2 leaves its latency to the walk.
  // 108x324x525 takes 101 us against 111, 100x256x756 85.2 (Y alone) against
  // 89.8, 64x500x1620 249 against 261; below it costs shared memory for
  // nothing: 81x180x180 20.7 us against 18.9, 150x270x252 (10 M) 44.6 against 43.4.
  const bool stage = Y && (long long)g.nx * g.ny * g.nz >= 12 << 20;
  auto kern = stage ? k_px_update<PL, NQ, P::kStaged> : k_px_update<PL, NQ, 0>;
  const size_t smem = P::smem(stage ? P::kStaged : 0);
  if (int rc = smem_optin(kern, smem)) return rc;
  float4* part = dots ? reinterpret_cast<float4*>(w->partials) : nullptr;
  const float* add = w ? w->add : nullptr;
  CDX_CHECK(launch_pdl(kern, grid, dim3(P::T), smem, st, g, tw,
                       reinterpret_cast<float4*>(const_cast<float2*>(S)), Y, Xout, G, dots, part,
                       add));
  CDX_LAUNCH_CHECK("k_px_update");
  if (dots) return launch_lambda(part, nblk, lam_next, eps, st);
  return 0;
}

}  // namespace cdx
