// z pass on the paired layout: dispatch, and the form on the generic engine for
// depths without a plan.
#include "decon_pz.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

// ---------------------------------------------------------------- generic
// Column v of a tile of W columns: lane v & 1 of the v / 2 th of W / 2
// neighbouring (kx, slot % 4) of a slot block.
struct PairZIO {
  static constexpr bool kSmem = false;
  static constexpr bool kGroup = false;
  float* base;  // float 0 of the tile's first slot at z = 0
  int rowf, nv;  // floats per z, columns inside the block
  __device__ __forceinline__ float2 ld(int v, int e) const {
    if (v >= nv) return make_float2(0.f, 0.f);
    const float* p = base + (long long)e * rowf + 4 * (v >> 1) + (v & 1);
    return make_float2(p[0], p[2]);
  }
  __device__ __forceinline__ void st(int v, int e, float2 x) const {
    if (v >= nv) return;
    float* p = base + (long long)e * rowf + 4 * (v >> 1) + (v & 1);
    p[0] = x.x;
    p[2] = x.y;
  }
};

struct PairOtfStore {
  static constexpr bool kSmem = true;
  static constexpr bool kGroup = false;
  SmemIO io;
  const float4* tz;
  const float* full;  // mode 1: float 0 of the tile's first slot at z = 0
  const int* cir;
  const float* car;
  int nr, rowf, nv, mode, conj;
  __device__ __forceinline__ void st(int v, int e, float2 x) const {
    float2 o = make_float2(0.f, 0.f);
    if (mode == 1) {
      if (v < nv) {
        const float* p = full + (long long)e * rowf + 4 * (v >> 1) + (v & 1);
        o = make_float2(__ldg(p), __ldg(p + 2));
      }
    } else {
      const int ir = cir[v];
      if (ir >= 0) o = otf_lerp(__ldg(tz + (long long)e * nr + ir), car[v]);
    }
    io.st(v, e, conj ? cmulconj(x, o) : cmul(x, o));
  }
};

__global__ void __launch_bounds__(kMaxThreads)
k_pz_gen(PairGeom g, FftDev fz, float4* S, OtfDev otf, int conj, int fwd_only, int W) {
  extern __shared__ __align__(16) float2 smem[];
  const int nz = g.nz;
  const int f0 = blockIdx.x * (W / 2);  // first (kx, slot % 4) of the tile
  float2* stw = smem;
  const SmemIO io{smem + nz, W, 1};
  int* cir = reinterpret_cast<int*>(smem + nz + spad_size(W * nz));
  float* car = reinterpret_cast<float*>(cir + W);
  load_twiddles(fz, stw);
  for (int v = threadIdx.x; v < W; v += blockDim.x) {
    const int f = f0 + (v >> 1), kx = f >> 2, s = blockIdx.y * 4 + (f & 3), y = g.col(s) + (v & 1) * g.col_step(s);
    int ir = -1;
    float ar = 0.f;
    if (kx < g.nxh && s < g.slots && y < g.ny && otf.mode == 0) {
      int i = 0;
      if (otf_radius(otf, kx, y, g.ny, i, ar)) ir = i;
    }
    cir[v] = ir;
    car[v] = ar;
  }
  grid_dep_wait();
  grid_dep_launch();
  __syncthreads();
  const long long at = 4 * ((long long)blockIdx.y * g.nxh * 4 + f0);
  const int nv = min(W, 2 * (4 * g.nxh - f0));
  const PairZIO gio{reinterpret_cast<float*>(S) + at, 4 * g.zstep, nv};
  const float invW = 1.f / (float)W;
  if (fwd_only) {
    GenericRunner::run<false>(fz, W, invW, true, stw, io, gio, gio);
    return;
  }
  const float* full = otf.mode == 1 ? reinterpret_cast<const float*>(otf.full) + at : nullptr;
  const PairOtfStore ost{io, otf.tz, full, cir, car, otf.nr, 4 * g.zstep, nv, otf.mode, conj};
  GenericRunner::run<false>(fz, W, invW, true, stw, io, gio, ost);
  GenericRunner::run<true>(fz, W, invW, true, stw, io, io, gio);
}

// The ratio's mean where the z kernels do not store it themselves: depths without a
// plan and 3D OTFs.
__global__ void __launch_bounds__(32) k_ratio_mean(PairGeom g, const float4* S, OtfDev otf) {
  grid_dep_wait();
  grid_dep_launch();
  store_ratio_mean(otf, reinterpret_cast<const float*>(S), g.nz, 4LL * g.zstep, __ldcg(otf.mean),
                   __ldg(otf.h0));
}

int launch_pz(const PairGeom& g, const FftLen& fz, float2* S, const OtfDev& otf, bool conj,
              cudaStream_t st, bool fwd_only) {
  if (otf.mean_next && (otf.mode == 1 || !fz.d_pair)) {
    CDX_CHECK(launch_pdl(k_ratio_mean, dim3(1), dim3(32), 0, st, g,
                         reinterpret_cast<const float4*>(S), otf));
    CDX_LAUNCH_CHECK("k_ratio_mean");
  }
  if (fz.d_pair) {
    bool done = false;
    const int rc = pzgen(g, fz.d_pair, S, otf, conj, st, fwd_only, &done);
    if (done || rc) return rc;
  }
  // an even number of columns, so that a tile holds whole slots
  int W = (kMaxThreads * kEpt) / g.nz;
  if (W > 16) W = 16;
  W &= ~1;
  if (W < 2) {
    set_error("z pass", "length too long for a column pair");
    return cudaErrorInvalidValue;
  }
  const size_t smem = sizeof(float2) * ((size_t)g.nz + spad_size(W * g.nz) + W);
  if (int rc = smem_optin(k_pz_gen, smem)) return rc;
  CDX_CHECK(launch_pdl(k_pz_gen, dim3(ceil_div(8 * g.nxh, W), ceil_div(g.slots, 4)),
                       dim3(threads_for((long long)W * g.nz)), smem, st, g, fz.dev,
                       reinterpret_cast<float4*>(S), otf, conj ? 1 : 0, fwd_only ? 1 : 0, W));
  CDX_LAUNCH_CHECK("k_pz_gen");
  return 0;
}

}  // namespace cdx
