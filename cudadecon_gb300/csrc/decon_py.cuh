// y pass on the paired layout (pair_layout.cuh): separates the packed rows'
// spectra, transforms along y, and back.
//
// Three forms:
//   eo   (even ny, plan of ny / 2 points): the lanes are the even and the odd
//        rows, which is how the x pass stores them; two ny/2-point transforms
//        run in the lanes and one radix-2 step across the lanes finishes
//        (starts) the ny-point one.
//   zz   (odd ny with a plan): the lanes are two z slices.
//   generic engine (decon_py.cu): any supported length.
#pragma once

#include "decon_common.cuh"
#include "fft_pair.cuh"
#include "pair_layout.cuh"

namespace cdx {

// Rows (kx, z) whose mirror image is the row itself.
__device__ __forceinline__ bool self_row(const PairGeom& g, int kx) {
  return kx == 0 || 2 * kx == g.nx;
}

// Spectra of the two real rows from the packed ones, times 2 (the OTF carries
// the 1/2): a = Z[kx] + conj Z[-kx], b = -i (Z[kx] - conj Z[-kx]).
__device__ __forceinline__ void split_rows(const C2& zp, const C2& zm, C2& a, C2& b) {
  a = {add2(zp.re, zm.re), sub2(zp.im, zm.im)};
  b = {add2(zp.im, zm.im), sub2(zm.re, zp.re)};
}
// and back: Z[kx] = a + i b, Z[-kx] = conj a + i conj b.  A row that is its
// own mirror image has real a and b (their imaginary parts are rounding,
// dropped as a C2R transform does).
__device__ __forceinline__ void merge_rows(const C2& a, const C2& b, bool self, C2& zp, C2& zm) {
  zp = {sub2(a.re, b.im), add2(a.im, b.re)};
  zm = {add2(a.re, b.im), sub2(b.re, a.im)};
  if (self) zp = {a.re, b.re};
}

// A block transforms V neighbouring kx of one slice.  Butterfly index i of the
// stages that touch global memory: consecutive threads take 4 consecutive
// slots, then the next kx (64 V contiguous bytes), then the next 4 slots.
template <int V, int E>
__device__ __forceinline__ void slot_order(int i, int& e, int& v) {
  e = i / (E * V) * E + i % E;
  v = i / E % V;
}
__host__ __device__ constexpr int round_up(int n, int m) { return (n + m - 1) / m * m; }

// ---------------------------------------------------------------- even/odd
template <class PL, int V>
struct PYE {
  static constexpr int KA4 = round_up(PL::KA, 4), KC4 = round_up(PL::KC, 4);
  static constexpr int kmax = KA4 > KC4 ? (KA4 > PL::KB || PL::Q1 == 1 ? KA4 : PL::KB)
                                        : (KC4 > PL::KB || PL::Q1 == 1 ? KC4 : PL::KB);
  static constexpr int T = round_up(V * kmax, 32);
  static constexpr int kTw = 2 * PL::L;  // plan twiddles, then w_ny^k for k < L
  static constexpr size_t kSmem = sizeof(float2) * kTw + sizeof(float4) * V * PL::VS;
  // pairs of the first half of the rows; kSame: rows m and m + HP are elements
  // of one stage A butterfly (ny % 4 == 0)
  static constexpr int HP = pair_split(2 * PL::L) / 2;
  static constexpr bool kSame = PL::L % 2 == 0;
  // 40 (inverse 28) registers beside the widest butterfly and 64 at least:
  // with 16 the inverse spilled (12.8 us against 11.0 on 64 x 256 x 256)
  template <bool INV>
  static constexpr int blocks() {
    const int regs = 4 * PL::qmax() + (INV ? 28 : 40);
    const int b = 65536 / (T * (regs < 64 ? 64 : regs)), most = 2048 / T;
    return b < 1 ? 1 : (b < most ? b : most);
  }
};

template <class PL, int V, bool INV>
__global__ void __launch_bounds__(PYE<PL, V>::T, PYE<PL, V>::template blocks<INV>())
k_py_eo(PairGeom g, const float2* __restrict__ tw, float4* S) {
  using P = PYE<PL, V>;
  constexpr int Q0 = PL::Q0, Q2 = PL::Q2, HP = P::HP;
  constexpr bool kSame = P::kSame;
  static_assert(!kSame || Q0 % 2 == 0, "stage A holds rows m and m + L/2");
  extern __shared__ __align__(16) float2 smem[];
  float2* stw = smem;
  const float2* wny = smem + PL::L;
  float4* sm = reinterpret_cast<float4*>(smem + P::kTw);
  copy_twiddles<P::kTw>(tw, stw);
  cp_async_commit();
  const int idx = threadIdx.x, kx0 = blockIdx.x * V;
  float4* slice = S + (long long)blockIdx.y * g.zstep;
  // slot s + r STEP of row kx; whole blocks of 4 slots apart for the usual STEP
  auto slot = [&](int kx, int s, auto stepc, int r) {
    constexpr int STEP = decltype(stepc)::value;
    if constexpr (STEP % 4 == 0)
      return slice + (((s >> 2) * g.nxh + kx) * 4 + (s & 3)) + r * (STEP * g.nxh);
    s += r * STEP;
    return slice + (((s >> 2) * g.nxh + kx) * 4 + (s & 3));
  };
  using StepA = std::integral_constant<int, PL::KA>;
  using StepC = std::integral_constant<int, PL::KC>;
  int j, va, k, vc;
  slot_order<V, 4>(idx, j, va);
  slot_order<V, 4>(idx, k, vc);
  const int kxa = kx0 + va, kxc = kx0 + vc;
  const bool act_a = j < PL::KA && kxa < g.nxh, act_c = k < PL::KC && kxc < g.nxh;
  const bool self = self_row(g, kxa);
  grid_dep_wait();
  if (!INV) {
    if constexpr (!kSame) {
      // rows m and m + HP belong to different butterflies: they go through the
      // tile, so that every slot is read once (each butterfly reading its half of
      // the slots it needs took 86 us on 96 x 486 x 525, all from DRAM twice)
      constexpr int kSlots = round_up(HP, 4) * V, N = (kSlots + P::T - 1) / P::T;
      C2 zp[N], zm[N];
#pragma unroll
      for (int n = 0; n < N; ++n) {
        int m, v;
        slot_order<V, 4>(idx + n * P::T, m, v);
        if (m >= HP || kx0 + v >= g.nxh) continue;
        zp[n] = ldp(slot(kx0 + v, m, StepA{}, 0));
        zm[n] = self_row(g, kx0 + v) ? zp[n] : ldp(slot(kx0 + v, g.hp + m, StepA{}, 0));
      }
#pragma unroll
      for (int n = 0; n < N; ++n) {
        int m, v;
        slot_order<V, 4>(idx + n * P::T, m, v);
        if (m >= HP || kx0 + v >= g.nxh) continue;
        C2 a, b;
        split_rows(zp[n], zm[n], a, b);
        float4* t = sm + v * PL::VS;
        stp(t + PL::pos(m), a);
        if (m + HP < PL::L) stp(t + PL::pos(m + HP), b);
      }
      __syncthreads();
    }
    if (act_a) {
      C2 x[Q0];
      float4* p = sm + va * PL::VS + j;
      if constexpr (kSame) {
#pragma unroll
        for (int r = 0; r < Q0 / 2; ++r) {
          const C2 zp = ldp(slot(kxa, j, StepA{}, r));
          const C2 zm = self ? zp : ldp(slot(kxa, g.hp + j, StepA{}, r));
          split_rows(zp, zm, x[r], x[r + Q0 / 2]);
        }
      } else {
#pragma unroll
        for (int r = 0; r < Q0; ++r) x[r] = ldp(p + r * PL::S0);
      }
      PDft<Q0, false>::run(x);
#pragma unroll
      for (int r = 0; r < Q0; ++r) stp(p + r * PL::S0, x[r]);
    }
    cp_async_wait_all();
    __syncthreads();
    stage_b<PL, V, false, false>(sm, stw);
    grid_dep_launch_small();
    if (act_c) {
      C2 x[Q2];
      const float4* p = sm + vc * PL::VS + pos_c<PL>(k);
#pragma unroll
      for (int r = 0; r < Q2; ++r) x[r] = ldp(p + r);
      butterfly<Q2, PL::KC, false, false>(x, stw, k);
#pragma unroll
      for (int r = 0; r < Q2; ++r) {
        // lanes E, O -> columns k and k + ny/2
        const float2 w = wny[k + r * PL::KC];
        const float2 o = cmul(make_float2(x[r].re.y, x[r].im.y), w);
        *slot(kxc, k, StepC{}, r) = make_float4(x[r].re.x + o.x, x[r].re.x - o.x, x[r].im.x + o.y,
                                                x[r].im.x - o.y);
      }
    }
  } else {
    C2 x[Q2];
    if (act_c) {
#pragma unroll
      for (int r = 0; r < Q2; ++r) x[r] = ldp(slot(kxc, k, StepC{}, r));
    }
    cp_async_wait_all();
    __syncthreads();  // the twiddles
    if (act_c) {
#pragma unroll
      for (int r = 0; r < Q2; ++r) {
        const float2 w = wny[k + r * PL::KC];
        const float2 e = make_float2(x[r].re.x + x[r].re.y, x[r].im.x + x[r].im.y);
        const float2 o = cmulconj(make_float2(x[r].re.x - x[r].re.y, x[r].im.x - x[r].im.y), w);
        x[r] = {make_float2(e.x, o.x), make_float2(e.y, o.y)};
      }
      butterfly<Q2, PL::KC, true, true>(x, stw, k);
      float4* p = sm + vc * PL::VS + pos_c<PL>(k);
#pragma unroll
      for (int r = 0; r < Q2; ++r) stp(p + r, x[r]);
    }
    __syncthreads();
    stage_b<PL, V, true, true>(sm, stw);
    grid_dep_launch_small();
    if (act_a) {
      C2 y[Q0];
      float4* p = sm + va * PL::VS + j;
#pragma unroll
      for (int r = 0; r < Q0; ++r) y[r] = ldp(p + r * PL::S0);
      PDft<Q0, true>::run(y);
      if constexpr (kSame) {
#pragma unroll
        for (int r = 0; r < Q0 / 2; ++r) {
          C2 zp, zm;
          merge_rows(y[r], y[r + Q0 / 2], self, zp, zm);
          stp(slot(kxa, j, StepA{}, r), zp);
          if (!self) stp(slot(kxa, g.hp + j, StepA{}, r), zm);
        }
      } else {
#pragma unroll
        for (int r = 0; r < Q0; ++r) stp(p + r * PL::S0, y[r]);
      }
    }
    if constexpr (!kSame) {
      __syncthreads();
      constexpr int n = (HP + 3) / 4 * 4 * V;
      for (int i = idx; i < n; i += P::T) {
        int m, v;
        slot_order<V, 4>(i, m, v);
        const int kx = kx0 + v;
        if (m >= HP || kx >= g.nxh) continue;
        const float4* t = sm + v * PL::VS;
        C2 b = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, zp, zm;
        if (m + HP < PL::L) b = ldp(t + PL::pos(m + HP));
        const bool own = self_row(g, kx);
        merge_rows(ldp(t + PL::pos(m)), b, own, zp, zm);
        stp(slot(kx, m, StepA{}, 0), zp);
        if (!own) stp(slot(kx, g.hp + m, StepA{}, 0), zm);
      }
    }
  }
}

// ---------------------------------------------------------------- two slices
// Element accessors of one row for the generic engine: lane e & 1 of slot
// e >> 1.  row: float 0 of the row's slot 0.
__device__ __forceinline__ long long lane_at(const PairGeom& g, int e) {
  const int s = e >> 1;
  return 4 * ((long long)(s >> 2) * g.nxh * 4 + (s & 3)) + (e & 1);
}
__device__ __forceinline__ float2 ld_lane(const PairGeom& g, const float* row, int e) {
  const float* p = row + lane_at(g, e);
  return make_float2(p[0], p[2]);
}
__device__ __forceinline__ void st_lane(const PairGeom& g, float* row, int e, float re, float im) {
  float* p = row + lane_at(g, e);
  p[0] = re;
  p[2] = im;
}

// (lanes y, y + 1 of slice 0; the same of slice 1) <-> (lanes slice 0, slice 1
// of y; the same of y + 1).
__device__ __forceinline__ void swap_lanes(C2& a, C2& b) {
  const C2 u = {make_float2(a.re.x, b.re.x), make_float2(a.im.x, b.im.x)};
  const C2 v = {make_float2(a.re.y, b.re.y), make_float2(a.im.y, b.im.y)};
  a = u;
  b = v;
}

template <class PL, int V>
struct PYZ {
  static constexpr int KC4 = round_up(PL::KC, 4);
  static constexpr int kmax = PL::kmax() > KC4 ? PL::kmax() : KC4;
  static constexpr int T = round_up(V * kmax, 32);
  static constexpr int kTw = PL::L + (PL::L & 1);
  static constexpr size_t kSmem = sizeof(float2) * kTw + sizeof(float4) * V * PL::VS;
};

// The rows are read and written a slot (two of them) at a time, and the tile
// regroups the lanes: a round trip more than an even height on the way in of the
// forward and out of the inverse transform.  Its columns go straight between
// registers and memory: a slot pairs the columns k and k + KC of one stage C
// butterfly (pair_layout.cuh), and the odd one left over of each butterfly goes
// with its neighbour's, by a shuffle.  With slots of neighbouring columns
// (2p, 2p + 1) the forward pass regrouped once more and the inverse read every
// slot twice.
template <class PL, int V, bool INV>
__global__ void __launch_bounds__(PYZ<PL, V>::T, PL::blocks_of(PYZ<PL, V>::T, 28))
k_py_zz(PairGeom g, const float2* __restrict__ tw, float4* S) {
  using P = PYZ<PL, V>;
  constexpr int Q0 = PL::Q0, Q2 = PL::Q2, L = PL::L, H = pair_split(L), T = P::T, KC = PL::KC;
  constexpr int kRows = H / 2;            // slots of a half row
  constexpr int KS = pair_kcs(L, KC), kFull = (Q2 - 1) / 2 * KS;  // slots of two columns of one butterfly
  static_assert(Q2 % 2 == 1, "an odd length");
  extern __shared__ __align__(16) float2 smem[];
  float2* stw = smem;
  float4* sm = reinterpret_cast<float4*>(smem + P::kTw);
  copy_twiddles<P::kTw>(tw, stw);
  cp_async_commit();
  grid_dep_wait();
  // slices z0 and z0 + 1 (the last of an odd count stands alone)
  const int z0 = 2 * blockIdx.y, kx0 = blockIdx.x * V, idx = threadIdx.x;
  const bool two = z0 + 1 < g.nz;
  float4* slice = S + (long long)z0 * g.zstep;
  const long long dz = two ? g.zstep : 0;
  const int half = g.hp * g.nxh;  // slots to the mirrored half
  auto at = [&](int v, int s) { return slice + ((s >> 2) * g.nxh + kx0 + v) * 4 + (s & 3); };
  const int va = idx / PL::KA, j = idx - va * PL::KA;
  float4* pa = sm + va * PL::VS + j;
  // stage C: 4 neighbouring k, then the next kx, then the next 4 k
  int k, vc;
  slot_order<V, 4>(idx, k, vc);
  const bool act_c = k < KC && kx0 + vc < g.nxh;
  // the left over column and its partner's (k = KC, past the end, has none of its own)
  const bool act_l = k <= KC && kx0 + vc < g.nxh, odd = k & 1;
  float4* pc = sm + vc * PL::VS + (k < KC ? pos_c<PL>(k) : 0);
  auto swap = [](float v) { return __shfl_xor_sync(0xffffffffu, v, 1); };
  if (!INV) {
    // all loads of a thread's slots before the first is used
    constexpr int kSlots = round_up(kRows, 4) * V, N = (kSlots + T - 1) / T;
    C2 p0[N], p1[N], m0[N], m1[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      int m, v;
      slot_order<V, 4>(idx + n * T, m, v);
      if (m >= kRows || kx0 + v >= g.nxh) continue;
      const bool self = self_row(g, kx0 + v);
      const float4* src = at(v, m);
      p0[n] = ldp(src);
      p1[n] = ldp(src + dz);
      m0[n] = self ? p0[n] : ldp(src + half);
      m1[n] = self ? p1[n] : ldp(src + half + dz);
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
      int m, v;
      slot_order<V, 4>(idx + n * T, m, v);
      if (m >= kRows || kx0 + v >= g.nxh) continue;
      C2 a0, b0, a1, b1;
      split_rows(p0[n], m0[n], a0, b0);
      split_rows(p1[n], m1[n], a1, b1);
      swap_lanes(a0, a1);
      swap_lanes(b0, b1);
      float4* t = sm + v * PL::VS;
      const int y = 2 * m;
      stp(t + PL::pos(y), a0);
      stp(t + PL::pos(y + 1), a1);
      if (y + H < L) stp(t + PL::pos(y + H), b0);
      if (y + 1 + H < L) stp(t + PL::pos(y + 1 + H), b1);
    }
    cp_async_wait_all();
    __syncthreads();
    if (va < V) {
      C2 x[Q0];
#pragma unroll
      for (int r = 0; r < Q0; ++r) x[r] = ldp(pa + r * PL::S0);
      PDft<Q0, false>::run(x);
#pragma unroll
      for (int r = 0; r < Q0; ++r) stp(pa + r * PL::S0, x[r]);
    }
    __syncthreads();
    stage_b<PL, V, false, false>(sm, stw);
    grid_dep_launch_small();
    C2 x[Q2];
    if (act_c) {
#pragma unroll
      for (int r = 0; r < Q2; ++r) x[r] = ldp(pc + r);
      butterfly<Q2, KC, false, false>(x, stw, k);
#pragma unroll
      for (int r = 0; r + 1 < Q2; r += 2) {
        swap_lanes(x[r], x[r + 1]);
        float4* dst = at(vc, r / 2 * KS + k);
        stp(dst, x[r]);
        if (two) stp(dst + dz, x[r + 1]);
      }
    } else {
      x[Q2 - 1] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    }
    // even k: slice 0 of columns k and k + 1; odd k: slice 1 of k - 1 and k
    const C2 u = x[Q2 - 1];
    const float re = swap(odd ? u.re.x : u.re.y), im = swap(odd ? u.im.x : u.im.y);
    if (act_l && (two || !odd)) {
      float4* dst = at(vc, kFull + (k >> 1));
      stp(odd ? dst + dz : dst, odd ? C2{make_float2(re, u.re.y), make_float2(im, u.im.y)}
                                    : C2{make_float2(u.re.x, re), make_float2(u.im.x, im)});
    }
  } else {
    C2 x[Q2];
    if (act_c) {
#pragma unroll
      for (int r = 0; r + 1 < Q2; r += 2) {
        const float4* src = at(vc, r / 2 * KS + k);
        x[r] = ldp(src);
        x[r + 1] = ldp(src + dz);
      }
    }
    C2 u = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (act_l) u = ldp(at(vc, kFull + (k >> 1)) + (odd ? dz : 0));
    const float re = swap(odd ? u.re.x : u.re.y), im = swap(odd ? u.im.x : u.im.y);
    x[Q2 - 1] = odd ? C2{make_float2(re, u.re.y), make_float2(im, u.im.y)}
                    : C2{make_float2(u.re.x, re), make_float2(u.im.x, im)};
    cp_async_wait_all();
    __syncthreads();
    if (act_c) {
#pragma unroll
      for (int r = 0; r + 1 < Q2; r += 2) swap_lanes(x[r], x[r + 1]);
      butterfly<Q2, KC, true, true>(x, stw, k);
#pragma unroll
      for (int r = 0; r < Q2; ++r) stp(pc + r, x[r]);
    }
    __syncthreads();
    stage_b<PL, V, true, true>(sm, stw);
    grid_dep_launch_small();
    if (va < V) {
      C2 y[Q0];
#pragma unroll
      for (int r = 0; r < Q0; ++r) y[r] = ldp(pa + r * PL::S0);
      PDft<Q0, true>::run(y);
#pragma unroll
      for (int r = 0; r < Q0; ++r) stp(pa + r * PL::S0, y[r]);
    }
    __syncthreads();
    for (int i = idx; i < (kRows + 3) / 4 * 4 * V; i += T) {
      int m, v;
      slot_order<V, 4>(i, m, v);
      if (m >= kRows || kx0 + v >= g.nxh) continue;
      const float4* t = sm + v * PL::VS;
      const int y = 2 * m;
      const C2 zero = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      C2 a0 = ldp(t + PL::pos(y)), a1 = ldp(t + PL::pos(y + 1));
      C2 b0 = y + H < L ? ldp(t + PL::pos(y + H)) : zero;
      C2 b1 = y + 1 + H < L ? ldp(t + PL::pos(y + 1 + H)) : zero;
      swap_lanes(a0, a1);
      swap_lanes(b0, b1);
      const bool self = self_row(g, kx0 + v);
      C2 p0, m0, p1, m1;
      merge_rows(a0, b0, self, p0, m0);
      merge_rows(a1, b1, self, p1, m1);
      float4* dst = at(v, m);
      stp(dst, p0);
      if (!self) stp(dst + half, m0);
      if (two) {
        stp(dst + dz, p1);
        if (!self) stp(dst + half + dz, m1);
      }
    }
  }
}

// ---------------------------------------------------------------- launches
template <class PL, int V>
static int py_eo_go(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st) {
  using P = PYE<PL, V>;
  auto kern = inv ? k_py_eo<PL, V, true> : k_py_eo<PL, V, false>;
  if (int rc = smem_optin(kern, P::kSmem)) return rc;
  CDX_CHECK(launch_pdl(kern, dim3(ceil_div(g.nxh, V), g.nz), dim3(P::T), P::kSmem, st, g, tw,
                       reinterpret_cast<float4*>(S)));
  CDX_LAUNCH_CHECK("k_py_eo");
  return 0;
}

template <class PL, int V>
static int py_zz_go(const PairGeom& g, const float2* tw, float2* S, bool inv, cudaStream_t st) {
  using P = PYZ<PL, V>;
  auto kern = inv ? k_py_zz<PL, V, true> : k_py_zz<PL, V, false>;
  if (int rc = smem_optin(kern, P::kSmem)) return rc;
  CDX_CHECK(launch_pdl(kern, dim3(ceil_div(g.nxh, V), (g.nz + 1) / 2), dim3(P::T), P::kSmem, st, g,
                       tw, reinterpret_cast<float4*>(S)));
  CDX_LAUNCH_CHECK("k_py_zz");
  return 0;
}

}  // namespace cdx
