// z pass on the paired layout: forward transform along z, OTF multiply,
// inverse transform, for two columns (the lanes of a slot) per thread.
//
// The transform ends in the registers where the inverse begins, so the OTF is
// applied in between without touching shared memory, and the first and last
// stages read and write global memory directly: at two radices a tile makes
// two shared round trips, where staging both ways and the OTF store made four.
#pragma once

#include <algorithm>

#include "decon_common.cuh"
#include "fft_pair.cuh"
#include "pair_layout.cuh"

namespace cdx {

template <class PL, int W>
struct PZ {
  static constexpr int T = (W * PL::kmax() + 31) / 32 * 32;
  static constexpr int kTw = PL::L + (PL::L & 1);
  static constexpr int kTile = W * PL::L;  // float4s
  static constexpr size_t kSmem = sizeof(float2) * kTw + 2 * sizeof(float4) * kTile;
  static constexpr int kBlocks = resident_blocks(PL::blocks(W, 56 /*Z*/), kSmem);
  static_assert(T % W == 0 && kBlocks > 0, "a thread copies one column, an SM holds a block");
};

// The mean of the ratio whose spectrum the z pass is given, for the next iteration
// (k_px_ratio): what was taken off it plus what is left at frequency 0, the sum of
// column (0, 0) over z (twice the transform, as the paired passes have it).  One
// warp calls this before the column is overwritten: its values lie `step` floats
// apart from p, in shared or global memory; before, h0: what was taken off and the
// OTF at frequency 0.  The ratio lies within 10; a mean that does not (NaN, when the
// image holds one) gives 0.
__device__ __forceinline__ void store_ratio_mean(const OtfDev& otf, const float* p, int nz,
                                                 long long step, float before, float h0) {
  float sum = 0.f;
#pragma unroll 4
  for (int z = threadIdx.x; z < nz; z += 32) sum += p[z * step];
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (threadIdx.x) return;
  float m = __fmaf_rn(sum, otf.inv2n, before);
  m = fabsf(m) <= 10.f ? m : 0.f;
  otf.mean_next[0] = m;
  otf.mean_next[3] = m * h0;
}

// MODE 0: radially averaged table (CONJ: its conjugate); 1: full 3D array in
// the paired layout, conjugated when conj, or with fwd_only the forward
// transform alone.
//
// A block walks over tiles: while it transforms one, the copies of the next
// are on their way into the other half of its tile memory, so the latency of
// global memory, which a block that loads, transforms and stores one tile
// waits out (a third of its time), is hidden.
template <class PL, int W, int MODE, bool CONJ, bool MEAN>
__global__ void __launch_bounds__(PZ<PL, W>::T, PZ<PL, W>::kBlocks)
k_pz(PairGeom g, const float2* __restrict__ tw, float4* S, OtfDev otf, int conj, int fwd_only,
     int ntiles) {
  using P = PZ<PL, W>;
  constexpr int Q0 = PL::Q0, Q1 = PL::Q1, Q2 = PL::Q2, KA = PL::KA, KC = PL::KC;
  extern __shared__ __align__(16) float2 smem[];
  float2* stw = smem;
  float4* bufs = reinterpret_cast<float4*>(smem + P::kTw);
  copy_twiddles<P::kTw>(tw, stw);
  const int c = threadIdx.x % W, b = threadIdx.x / W;  // column pair, butterfly
  const int nf = (4 * g.nxh + W - 1) / W;  // tiles per slot block
  // W neighbouring (kx, slot % 4) of a slot block
  auto place = [&](int t, int& kx, int& s) {
    const int sb = t / nf, f = (t - sb * nf) * W + c;
    kx = f >> 2;
    s = sb * 4 + (f & 3);
    return (long long)sb * g.nxh * 4 + f;
  };
  auto copy = [&](int t, float4* buf) {
    int kx, s;
    const float4* src = S + place(t, kx, s);
    if (kx < g.nxh && s < g.slots) {
#pragma unroll 4
      for (int z = b; z < PL::L; z += P::T / W)
        cp_async16(buf + z * W + c, src + (long long)z * g.zstep);
    }
    cp_async_commit();
  };
  int t = blockIdx.x;
  grid_dep_wait();
  if (t < ntiles) copy(t, bufs);
  // Kernels of their own store the ratio's mean (MEAN), for two passes of a loop: in
  // the others, never reached, the code cost 64 x 256 x 384 0.9% of an iteration.
  float before = 0.f, h0 = 0.f;
  if (MEAN && blockIdx.x == 0) {
    before = __ldcg(otf.mean);
    h0 = __ldg(otf.h0);
  }
  for (int half = 0; t < ntiles; t += gridDim.x, half ^= 1) {
    float4* tc = bufs + half * P::kTile + c;
    int kx, s;
    const long long col_at = place(t, kx, s);
    const bool in = kx < g.nxh && s < g.slots;
    float4* col = S + col_at;
    cp_async_wait_all();
    __syncthreads();
    if (MEAN && t == 0) {  // column (0, 0) is the tile's first
      if (threadIdx.x < 32)
        store_ratio_mean(otf, reinterpret_cast<const float*>(bufs), PL::L, 4 * W, before, h0);
      __syncthreads();
    }
    if (t + gridDim.x < ntiles) copy(t + gridDim.x, bufs + (half ^ 1) * P::kTile);
    if (b < KA) {
      C2 x[Q0];
#pragma unroll
      for (int r = 0; r < Q0; ++r) x[r] = ldp(tc + (r * KA + b) * W);
      PDft<Q0, false>::run(x);
#pragma unroll
      for (int r = 0; r < Q0; ++r) stp(tc + (r * KA + b) * W, x[r]);
    }
    __syncthreads();
    auto mid = [&](auto invc) {
      constexpr bool INV = decltype(invc)::value;
      if constexpr (Q1 > 1) {
        if (b < PL::KB) {
          const int b0 = b / Q2, a2 = b - b0 * Q2;
          float4* p = tc + (b0 * KA + a2) * W;
          C2 x[Q1];
#pragma unroll
          for (int r = 0; r < Q1; ++r) x[r] = ldp(p + r * Q2 * W);
          butterfly<Q1, Q0, INV, INV>(x, stw, b0);
#pragma unroll
          for (int r = 0; r < Q1; ++r) stp(p + r * Q2 * W, x[r]);
        }
        __syncthreads();
      }
    };
    mid(std::false_type{});
    if (b < KC) {
      const int b1 = b / Q0, b0 = b - b1 * Q0;
      float4* p = tc + (b0 * KA + b1 * Q2) * W;
      C2 x[Q2];
#pragma unroll
      for (int r = 0; r < Q2; ++r) x[r] = ldp(p + r * W);
      butterfly<Q2, KC, false, false>(x, stw, b);
      if (MODE == 1 && fwd_only) {
        if (in) {
#pragma unroll
          for (int r = 0; r < Q2; ++r) stp(col + (long long)(b + r * KC) * g.zstep, x[r]);
        }
      } else {
        if constexpr (MODE == 0) {
          // radius of the two columns, then the pair (value at ir, at ir + 1)
          // per kz (dev_otfinterpolate RA branch, RLgpuImpl.cu:238-273)
          int ir0 = 0, ir1 = 0;
          float ar0 = 0.f, ar1 = 0.f;
          // (a slot without columns has its first so far out that no radius reaches it)
          int y0 = g.per * s, y1 = y0 + g.step;
          if (g.kc) {
            y0 = g.col(s);
            y1 = y0 + g.col_step(s);
          }
          const bool in0 = in && otf_radius(otf, kx, y0, g.ny, ir0, ar0);
          const bool in1 = in && y1 < g.ny && otf_radius(otf, kx, y1, g.ny, ir1, ar1);
          const float4* t0 = otf.tz + (long long)b * otf.nr + ir0;
          const float4* t1 = otf.tz + (long long)b * otf.nr + ir1;
#pragma unroll
          for (int r = 0; r < Q2; ++r) {
            float2 u = make_float2(0.f, 0.f), v = make_float2(0.f, 0.f);
            if (in0) u = otf_lerp(__ldg(t0 + r * KC * otf.nr), ar0);
            if (in1) v = otf_lerp(__ldg(t1 + r * KC * otf.nr), ar1);
            x[r] = cmul2<CONJ>(x[r], C2{make_float2(u.x, v.x), make_float2(u.y, v.y)});
          }
        } else if (in) {
          const float4* full = reinterpret_cast<const float4*>(otf.full) + col_at;
#pragma unroll
          for (int r = 0; r < Q2; ++r) {
            const float4 o = __ldg(full + (long long)(b + r * KC) * g.zstep);
            const float2 oi = make_float2(o.z, o.w);
            x[r] = cmul2<false>(x[r], C2{make_float2(o.x, o.y), conj ? neg2(oi) : oi});
          }
        }
        butterfly<Q2, KC, true, true>(x, stw, b);
#pragma unroll
        for (int r = 0; r < Q2; ++r) stp(p + r * W, x[r]);
      }
    }
    if (MODE == 1 && fwd_only) continue;
    __syncthreads();
    mid(std::true_type{});
    if (t + gridDim.x >= ntiles) grid_dep_launch_small();
    if (b < KA && in) {
      C2 x[Q0];
#pragma unroll
      for (int r = 0; r < Q0; ++r) x[r] = ldp(tc + (r * KA + b) * W);
      PDft<Q0, true>::run(x);
#pragma unroll
      for (int r = 0; r < Q0; ++r) stp(col + (long long)(b + r * KA) * g.zstep, x[r]);
    }
  }
}

// ---------------------------------------------------------------- launches
template <class PL, int W, int MODE, bool CONJ, bool MEAN = false>
static int pz_go(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf,
                 bool conj, cudaStream_t st, bool fwd_only) {
  using P = PZ<PL, W>;
  auto kern = k_pz<PL, W, MODE, CONJ, MEAN>;
  if (int rc = smem_optin(kern, P::kSmem)) return rc;
  const int ntiles = ceil_div(4 * g.nxh, W) * ceil_div(g.slots, 4);
  const int grid = std::min(ntiles, P::kBlocks * sm_count());
  CDX_CHECK(launch_pdl(kern, dim3(grid), dim3(P::T), P::kSmem, st, g, tw,
                       reinterpret_cast<float4*>(S), otf, conj ? 1 : 0, fwd_only ? 1 : 0, ntiles));
  CDX_LAUNCH_CHECK("k_pz");
  return 0;
}

template <class PL, int W>
static int pz_mode(const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, bool conj,
                   cudaStream_t st, bool fwd_only) {
  if (fwd_only || otf.mode == 1) return pz_go<PL, W, 1, false>(g, tw, S, otf, conj, st, fwd_only);
  if (otf.mean_next) return pz_go<PL, W, 0, true, true>(g, tw, S, otf, conj, st, false);
  return conj ? pz_go<PL, W, 0, true>(g, tw, S, otf, conj, st, false)
              : pz_go<PL, W, 0, false>(g, tw, S, otf, conj, st, false);
}

}  // namespace cdx
