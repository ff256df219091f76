// Paired transforms: every thread works on two complex vectors at once, held
// lane by lane in 64-bit registers (C2: the real parts of both vectors in one
// float2, the imaginary parts in another), so that each butterfly step is one
// packed FP32 instruction (add/mul/fma.f32x2) for two vectors.  A packed
// instruction takes one issue slot where two scalar ones take two (measured
// on a GB300: 39.5 T lane-operations/s packed against 37.4 T scalar, and with
// three different register operands 26.5 T against 21.7 T); the passes were
// bound by issue slots and by shared-memory wavefronts, and a pair also halves
// the loads, stores, twiddle reads and index arithmetic per vector.
//
// A plan splits L = Q0 Q1 Q2 (Q1 = 1: two radices).  Element e has the digits
// e = a0 Q1 Q2 + a1 Q2 + a2, frequency f = b0 + Q0 b1 + Q0 Q1 b2.  The
// transform runs digit by digit: stage A turns a0 into b0, stage B a1 into b1
// after the twiddle w_{Q0 Q1}^(a1 b0), stage C a2 into b2 after the twiddle
// w_L^(a2 k) with k = b0 + Q0 b1.  Each butterfly writes where it read (digit
// d0 at stride S0, d1 at Q2, d2 at 1), so a stage needs no barrier between
// its reads and its writes, one barrier separates two stages, and the
// transposed transform (C, B, A with the twiddles after the butterflies) goes
// back over the same addresses and the same table.  Stage A's thread holds
// elements j + r L/Q0 and stage C's holds frequencies k + r L/Q2: both read or
// write global memory straight from registers, and what happens between a
// transform and the one that undoes it (the RL ratio, the OTF) happens in
// registers too.
#pragma once

#include "decon_common.cuh"
#include "dft_static.cuh"

namespace cdx {

// Two complex numbers: lane 0 in .x, lane 1 in .y.
struct C2 {
  float2 re, im;
};

__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 relu2(float2 a) {
  return make_float2(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f));  // NaN gives 0, as x > 0 ? x : 0 does
}

__device__ __forceinline__ C2 operator+(C2 a, C2 b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ C2 operator-(C2 a, C2 b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// times -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ C2 rot2(C2 a) {
  return INV ? C2{neg2(a.im), a.re} : C2{a.im, neg2(a.re)};
}
// both lanes times c + i s (CONJ: c - i s)
template <bool CONJ>
__device__ __forceinline__ C2 cmul2(C2 a, float c, float s) {
  const float2 cc = dup2(c), ss = dup2(CONJ ? -s : s);
  return {fma2(neg2(a.im), ss, mul2(a.re, cc)), fma2(a.re, ss, mul2(a.im, cc))};
}
// lane by lane: a times b, or a times conj(b)
template <bool CONJ>
__device__ __forceinline__ C2 cmul2(C2 a, C2 b) {
  if (CONJ) return {fma2(a.im, b.im, mul2(a.re, b.re)), fma2(neg2(a.re), b.im, mul2(a.im, b.re))};
  return {fma2(neg2(a.im), b.im, mul2(a.re, b.re)), fma2(a.re, b.im, mul2(a.im, b.re))};
}

__device__ __forceinline__ C2 ldp(const float4* p) {
  const float4 v = *p;
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float4 pack(C2 x) { return make_float4(x.re.x, x.re.y, x.im.x, x.im.y); }
__device__ __forceinline__ void stp(float4* p, C2 x) { *p = pack(x); }

// x * w_Q^M (its conjugate when INV)
template <int Q, int M, bool INV>
__device__ __forceinline__ C2 twmul2(C2 x) {
  constexpr float c = Tw<Q, M>::re;
  constexpr float s = INV ? -Tw<Q, M>::im : Tw<Q, M>::im;
  if constexpr (s == 0.f && c == 1.f) return x;
  else if constexpr (s == 0.f && c == -1.f) return {neg2(x.re), neg2(x.im)};
  else if constexpr (c == 0.f && s == 1.f) return {neg2(x.im), x.re};
  else if constexpr (c == 0.f && s == -1.f) return {x.im, neg2(x.re)};
  else return cmul2<false>(x, c, s);
}

// ---------------------------------------------------------------- Q-point DFTs
template <int Q, bool INV, class Enable = void>
struct PDft;

template <bool INV>
struct PDft<1, INV> {
  __device__ __forceinline__ static void run(C2*) {}
};
template <bool INV>
struct PDft<2, INV> {
  __device__ __forceinline__ static void run(C2* x) {
    const C2 a = x[0], b = x[1];
    x[0] = a + b;
    x[1] = a - b;
  }
};
template <bool INV>
struct PDft<3, INV> {
  __device__ __forceinline__ static void run(C2* x) {
    // the sine term goes in as one fma per output component
    const C2 s = x[1] + x[2], d = x[1] - x[2];
    const float2 mh = dup2(-0.5f), h = dup2(INV ? -odd_sin<3>(1) : odd_sin<3>(1));
    const C2 a = {fma2(mh, s.re, x[0].re), fma2(mh, s.im, x[0].im)};
    x[0] = x[0] + s;
    x[1] = {fma2(h, d.im, a.re), fma2(neg2(h), d.re, a.im)};
    x[2] = {fma2(neg2(h), d.im, a.re), fma2(h, d.re, a.im)};
  }
};
template <bool INV>
struct PDft<4, INV> {
  __device__ __forceinline__ static void run(C2* x) {
    const C2 a = x[0] + x[2], b = x[0] - x[2];
    const C2 c = x[1] + x[3], d = rot2<INV>(x[1] - x[3]);
    x[0] = a + c;
    x[2] = a - c;
    x[1] = b + d;
    x[3] = b - d;
  }
};
template <bool INV>
struct PDft<8, INV> {
  __device__ __forceinline__ static void run(C2* x) {
    C2 u[4], v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      u[r] = x[r] + x[r + 4];
      v[r] = x[r] - x[r + 4];
    }
    const float2 h = dup2(7.071067812e-01f);
    const C2 r1 = rot2<INV>(v[1]), r3 = rot2<INV>(v[3]);
    // w8 v = h (v + rot v), w8^3 v = h (rot v - v)
    const C2 t1 = v[1] + r1, t3 = r3 - v[3];
    v[1] = {mul2(h, t1.re), mul2(h, t1.im)};
    v[2] = rot2<INV>(v[2]);
    v[3] = {mul2(h, t3.re), mul2(h, t3.im)};
    PDft<4, INV>::run(u);
    PDft<4, INV>::run(v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[2 * q] = u[q];
      x[2 * q + 1] = v[q];
    }
  }
};
// 5 and 7 points by the symmetric/antisymmetric pairing of inputs p and R-p
template <int R, bool INV>
struct PDft<R, INV, std::enable_if_t<R == 5 || R == 7>> {
  __device__ __forceinline__ static void run(C2* x) {
    constexpr int H = (R - 1) / 2;
    C2 s[H + 1], d[H + 1], out[R];
    C2 y0 = x[0];
#pragma unroll
    for (int p = 1; p <= H; ++p) {
      s[p] = x[p] + x[R - p];
      d[p] = x[p] - x[R - p];
      y0 = y0 + s[p];
    }
    out[0] = y0;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      C2 a = x[0], b;
#pragma unroll
      for (int p = 1; p <= H; ++p) {
        const float2 c = dup2(odd_cos<R>((p * q) % R)), sn = dup2(odd_sin<R>((p * q) % R));
        a = {fma2(c, s[p].re, a.re), fma2(c, s[p].im, a.im)};
        if (p == 1)
          b = {mul2(sn, d[p].re), mul2(sn, d[p].im)};
        else
          b = {fma2(sn, d[p].re, b.re), fma2(sn, d[p].im, b.im)};
      }
      const C2 ib = rot2<INV>(b);  // forward: y_q = a - i b, y_{R-q} = a + i b
      out[q] = a + ib;
      out[R - q] = a - ib;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = out[q];
  }
};

constexpr bool pdft_base(int q) { return q <= 5 || q == 7 || q == 8; }
constexpr int pdft_split(int q) {
  // 9 = 3*3, 16 = 4*4; otherwise the largest hand-written factor
  if (q == 9) return 3;
  if (q == 16) return 4;
  constexpr int cands[] = {8, 7, 5, 4, 3, 2};
  for (int c : cands)
    if (q % c == 0 && q / c > 1) return c;
  return q;
}

template <int Q, bool INV>
struct PDft<Q, INV, std::enable_if_t<!pdft_base(Q)>> {
  static constexpr int A = pdft_split(Q);
  static constexpr int B = Q / A;
  __device__ __forceinline__ static void run(C2* x) {
    C2 t[A][B];
    static_for<A>([&](auto n1c) {
      constexpr int n1 = decltype(n1c)::value;
      C2 a[B];
      static_for<B>([&](auto n2c) {
        constexpr int n2 = decltype(n2c)::value;
        a[n2] = x[n1 + A * n2];
      });
      PDft<B, INV>::run(a);
      static_for<B>([&](auto k2c) {
        constexpr int k2 = decltype(k2c)::value;
        t[n1][k2] = twmul2<Q, n1 * k2, INV>(a[k2]);
      });
    });
    static_for<B>([&](auto k2c) {
      constexpr int k2 = decltype(k2c)::value;
      C2 a[A];
      static_for<A>([&](auto n1c) {
        constexpr int n1 = decltype(n1c)::value;
        a[n1] = t[n1][k2];
      });
      PDft<A, INV>::run(a);
      static_for<A>([&](auto k1c) {
        constexpr int k1 = decltype(k1c)::value;
        x[B * k1 + k2] = a[k1];
      });
    });
  }
};

// ---------------------------------------------------------------- plans
// S0: stride of digit d0 in the shared tile (>= Q1 Q2, padded against bank
// conflicts), VS: stride of a vector of the tile.
template <int L_, int Q0_, int Q1_, int Q2_, int S0_, int VS_>
struct PPlan {
  static constexpr int L = L_, Q0 = Q0_, Q1 = Q1_, Q2 = Q2_, S0 = S0_, VS = VS_;
  static constexpr int KA = Q1 * Q2, KB = Q0 * Q2, KC = Q0 * Q1;  // butterflies per vector
  static_assert(Q0 * Q1 * Q2 == L && S0 >= KA && VS >= (Q0 - 1) * S0 + KA, "not a plan of L");
  static constexpr int kmax() {
    const int m = KA > KC ? KA : KC;
    return Q1 > 1 && KB > m ? KB : m;
  }
  static constexpr int qmax() {
    const int m = Q0 > Q2 ? Q0 : Q2;
    return Q1 > m ? Q1 : m;
  }
  // threads of a block of V vectors: one per butterfly of the stage with most
  static constexpr int threads(int V) { return (V * kmax() + 31) / 32 * 32; }
  // blocks per SM to ask for: the packed butterfly holds 4 qmax registers
  static constexpr int blocks_of(int T, int extra) {
    const int b = 65536 / (T * (4 * qmax() + extra));
    const int most = 2048 / T;
    const int m = b < most ? b : most;
    return m < 1 ? 1 : (m > 16 ? 16 : m);
  }
  static constexpr int blocks(int V, int extra) { return blocks_of(threads(V), extra); }
  // element e of a vector
  __device__ __forceinline__ static int pos(int e) {
    return S0 == KA ? e : (e / KA) * S0 + e % KA;
  }
};

// Start copying N float2s (an even number; the tables are padded) of twiddles
// into shared memory; the copy ends with the thread's other async copies.
template <int N>
__device__ __forceinline__ void copy_twiddles(const float2* tw, float2* stw) {
  static_assert(N % 2 == 0, "16-byte copies");
  for (int i = threadIdx.x; i < N / 2; i += blockDim.x) cp_async16(stw + 2 * i, tw + 2 * i);
}

// Blocks per SM: the launch bound, or what the shared memory of an SM (227 KB,
// 1 KB of it kept per block, which covers the kernels' static arrays) holds; 0
// where not even one block fits.
constexpr int resident_blocks(int bound, size_t smem) {
  const int fit = (int)((227u << 10) / (smem + 1024));
  return fit < bound ? fit : bound;
}

// Twiddle factors in the layout of FftDev::tw (stage with span Ns at Ns - 1,
// [r - 1][k]).  AFTER: multiply after the butterfly (the transposed order).
// GTW: the table is in global memory.
template <int Q, int NS, bool INV, bool GTW = false>
__device__ __forceinline__ void twiddle(C2* x, const float2* stw, int k) {
  const float2* tw = stw + (NS - 1) + k;
#pragma unroll
  for (int r = 1; r < Q; ++r) {
    const float2 w = GTW ? __ldg(tw + (r - 1) * NS) : tw[(r - 1) * NS];
    x[r] = cmul2<INV>(x[r], w.x, w.y);
  }
}
template <int Q, int NS, bool INV, bool AFTER, bool GTW = false>
__device__ __forceinline__ void butterfly(C2* x, const float2* stw, int k) {
  if (!AFTER) twiddle<Q, NS, INV, GTW>(x, stw, k);
  PDft<Q, INV>::run(x);
  if (AFTER) twiddle<Q, NS, INV, GTW>(x, stw, k);
}

// Stage B in place on a tile of V vectors, butterfly b of the block per
// thread (vector slowest, then b0, then a2).
// then() runs before the barrier that ends the stage.
template <class PL, int V, bool INV, bool AFTER, class Then>
__device__ __forceinline__ void stage_b(float4* sm, const float2* stw, const Then& then) {
  if constexpr (PL::Q1 > 1) {
    const int idx = threadIdx.x;
    if (idx < V * PL::KB) {
      const int v = idx / PL::KB, w = idx - v * PL::KB;
      const int b0 = w / PL::Q2, a2 = w - b0 * PL::Q2;
      float4* p = sm + v * PL::VS + b0 * PL::S0 + a2;
      C2 x[PL::Q1];
#pragma unroll
      for (int r = 0; r < PL::Q1; ++r) x[r] = ldp(p + r * PL::Q2);
      butterfly<PL::Q1, PL::Q0, INV, AFTER>(x, stw, b0);
#pragma unroll
      for (int r = 0; r < PL::Q1; ++r) stp(p + r * PL::Q2, x[r]);
    }
    then();
    __syncthreads();
  }
}
template <class PL, int V, bool INV, bool AFTER>
__device__ __forceinline__ void stage_b(float4* sm, const float2* stw) {
  stage_b<PL, V, INV, AFTER>(sm, stw, [] {});
}

// The thread's digit-C position k = b0 + Q0 b1 in the tile (vector base).
template <class PL>
__device__ __forceinline__ int pos_c(int k) {
  if constexpr (PL::Q1 == 1) return k * PL::S0;
  const int b1 = k / PL::Q0, b0 = k - b1 * PL::Q0;
  return b0 * PL::S0 + b1 * PL::Q2;
}

}  // namespace cdx
