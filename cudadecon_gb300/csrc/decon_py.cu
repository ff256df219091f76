// y pass on the paired layout: dispatch, and the form on the generic engine for
// heights without a plan.
#include "decon_py.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

// ---------------------------------------------------------------- generic
// Rows r = z nxh + kx, so that neighbouring rows of a tile share their lines.
struct PairRows {
  float* S;
  PairGeom g;
  long long r0, nrows;
  __device__ __forceinline__ bool row(int v, int& kx, float*& p) const {
    const long long r = r0 + v;
    if (r >= nrows) return false;
    const int z = (int)(r / g.nxh);
    kx = (int)(r - (long long)z * g.nxh);
    p = S + 4LL * z * g.zstep + 16LL * kx;
    return true;
  }
  __device__ __forceinline__ long long half() const { return 4LL * (g.hp >> 2) * g.nxh * 4; }
};
struct PairRowSplitLoad {  // row y of the real rows' spectra, times 2
  static constexpr bool kSmem = false;
  static constexpr bool kGroup = false;
  PairRows rows;
  __device__ __forceinline__ float2 ld(int v, int y) const {
    int kx;
    float* row;
    if (!rows.row(v, kx, row)) return make_float2(0.f, 0.f);
    const PairGeom& g = rows.g;
    const bool second = y >= g.H;
    const int e = second ? y - g.H : y;
    const float2 p = ld_lane(g, row, e);
    const float2 m = self_row(g, kx) ? p : ld_lane(g, row + rows.half(), e);
    return second ? make_float2(p.y + m.y, m.x - p.x) : make_float2(p.x + m.x, p.y - m.y);
  }
};
struct PairColIO {  // column ky of the half spectrum
  static constexpr bool kSmem = false;
  static constexpr bool kGroup = false;
  PairRows rows;
  __device__ __forceinline__ float2 ld(int v, int e) const {
    int kx;
    float* row;
    return rows.row(v, kx, row) ? ld_lane(rows.g, row, e) : make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void st(int v, int e, float2 x) const {
    int kx;
    float* row;
    if (rows.row(v, kx, row)) st_lane(rows.g, row, e, x.x, x.y);
  }
};

template <bool INV>
__global__ void __launch_bounds__(kMaxThreads)
k_py_gen(PairGeom g, FftDev fy, float4* S4, int V) {
  extern __shared__ __align__(16) float2 smem[];
  float2* stw = smem;
  const SmemIO io{smem + g.ny, 1, g.ny};
  load_twiddles(fy, stw);
  grid_dep_wait();
  grid_dep_launch();
  __syncthreads();
  const PairRows rows{reinterpret_cast<float*>(S4), g, (long long)blockIdx.x * V,
                      (long long)g.nxh * g.nz};
  const PairColIO cio{rows};
  if (!INV) {
    const PairRowSplitLoad ld{rows};
    GenericRunner::run<false>(fy, V, 1.f, false, stw, io, ld, cio);
  } else {
    GenericRunner::run<true>(fy, V, 1.f, false, stw, io, cio, io);
    for (int i = threadIdx.x; i < V * g.H; i += blockDim.x) {
      const int v = i / g.H, e = i - v * g.H;
      int kx;
      float* row;
      if (!rows.row(v, kx, row)) break;
      const float2 a = io.ld(v, e);
      const float2 b = e + g.H < g.ny ? io.ld(v, e + g.H) : make_float2(0.f, 0.f);
      if (self_row(g, kx)) {
        st_lane(g, row, e, a.x, b.x);
      } else {
        st_lane(g, row, e, a.x - b.y, a.y + b.x);
        st_lane(g, row + rows.half(), e, a.x + b.y, b.x - a.y);
      }
    }
  }
}

template <bool INV>
static int py_gen_go(const PairGeom& g, const FftLen& fy, float2* S, cudaStream_t st) {
  // rows per block: about 2048 elements, fewer where that leaves the chip idle
  // (64 x 2 x 256: 14 us a pass with 1024 rows in each of 9 blocks)
  const long long rows_per_block = (long long)g.nxh * g.nz / (4 * sm_count());
  int V = 2048 / g.ny;
  if (V > rows_per_block) V = (int)rows_per_block;
  if (V < 1) V = 1;
  const size_t smem = sizeof(float2) * ((size_t)g.ny + spad_size(V * g.ny));
  const long long nrows = (long long)g.nxh * g.nz;
  if (int rc = smem_optin(k_py_gen<INV>, smem)) return rc;
  CDX_CHECK(launch_pdl(k_py_gen<INV>, dim3((unsigned)((nrows + V - 1) / V)),
                       dim3(threads_for((long long)V * g.ny)), smem, st, g, fy.dev,
                       reinterpret_cast<float4*>(S), V));
  CDX_LAUNCH_CHECK("k_py_gen");
  return 0;
}

int launch_py(const PairGeom& g, const FftLen& fy, float2* S, bool inverse, cudaStream_t st) {
  if (fy.d_pair) {
    bool done = false;
    const int rc = pygen(g, fy.d_pair, S, inverse, st, &done);
    if (done || rc) return rc;
  }
  return inverse ? py_gen_go<true>(g, fy, S, st) : py_gen_go<false>(g, fy, S, st);
}

}  // namespace cdx
