// Y tiling and maximum-intensity projections of the reference's CLI
// (linearDecon.cpp:497-566 tiling, 1175-1245 stitching, 1434-1473 MaxIntProj).
#include "kernels.h"

namespace cdx {

// Rows yoff .. yoff+tny-1 of a (nx, ny, nz) raw stack, rows past either end
// repeating the nearest edge row (the CLI's get_crop with boundary
// conditions, linearDecon.cpp:548-556), into a (nx, tny, nz) tile.
__global__ void k_tile_rows(const unsigned short* __restrict__ raw, unsigned short* __restrict__ tile,
                            int nx, int ny, int tny, int yoff) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  const int z = blockIdx.z;
  if (x >= nx) return;
  const int ys = min(max(yoff + y, 0), ny - 1);
  tile[((long long)z * tny + y) * nx + x] = raw[((long long)z * ny + ys) * nx + x];
}

int launch_tile_rows(const unsigned short* raw, unsigned short* tile, int nx, int ny, int nz,
                     int tny, int yoff, cudaStream_t st) {
  dim3 grid(ceil_div(nx, 128), tny, nz);
  k_tile_rows<<<grid, 128, 0, st>>>(raw, tile, nx, ny, tny, yoff);
  CDX_LAUNCH_CHECK("k_tile_rows");
  return 0;
}

// Stitch one deconvolved tile (nx, tny, nz) into the output (nx, ny_out, nz) at
// rows y + yoff, with the CLI's rules: zones of a tile near its ends are left
// to the neighbouring tile, a blend zone mixes linearly (BlendTileOverlap),
// and weight marks output voxels already written (linearDecon.cpp:1186-1237).
__global__ void k_stitch(const float* __restrict__ tile, float* out, unsigned char* weight, int nx,
                         int tny, int nz, int ny_out, int yoff, double overlap, int no_zone,
                         int blend_zone, int first, int last, int blend_on) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  const int z = blockIdx.z;
  if (x >= nx || y + yoff >= ny_out) return;
  float blend = 1;
  if (first && y <= overlap)
    blend = 1;
  else if (last && y >= tny - overlap)
    blend = 1;
  else {
    if (y <= no_zone)
      blend = 0;
    else if (y > no_zone && y <= no_zone + blend_zone)
      blend = (double)(y - no_zone) / blend_zone;
    else if (y >= tny - no_zone)
      blend = 0;
    else
      blend = 1;
  }
  const float v = tile[((long long)z * tny + y) * nx + x];
  const long long o = ((long long)z * ny_out + (y + yoff)) * nx + x;
  if (blend_on) {
    const bool w = weight[o] > 0;
    if (blend > 0 && blend < 1 && w)
      out[o] = (float)__dadd_rn((double)__fmul_rn(v, blend),
                                 __dmul_rn((double)out[o], 1.0 - (double)blend));
    else if (blend > 0 && !w)
      out[o] = v;
    else if (blend == 1)
      out[o] = v;
    if (blend > 0) weight[o] = 1;
  } else {
    const bool past_front = (y >= floor((float)overlap / 2.0) || first);
    const bool before_end = (y < floor(tny - (float)overlap / 2.0) || last);
    if (past_front && before_end) out[o] = v;
  }
}

int launch_stitch(const float* tile, float* out, unsigned char* weight, int nx, int tny, int nz,
                  int ny_out, int yoff, double overlap, int no_zone, int blend_zone, bool first,
                  bool last, bool blend, cudaStream_t st) {
  dim3 grid(ceil_div(nx, 128), tny, nz);
  k_stitch<<<grid, 128, 0, st>>>(tile, out, weight, nx, tny, nz, ny_out, yoff, overlap, no_zone,
                                 blend_zone, first ? 1 : 0, last ? 1 : 0, blend ? 1 : 0);
  CDX_LAUNCH_CHECK("k_stitch");
  return 0;
}

// MaxIntProj (linearDecon.cpp:1434-1473): maximum along axis 0 (x), 1 (y) or
// 2 (z), starting from -1e10; outputs (ny, nz), (nx, nz), (nx, ny) images,
// first size fastest.  NaN is never taken (fmaxf returns the other operand, as
// the comparison p > m does).
constexpr int kMipBatch = 8;  // loads in flight per thread
constexpr int kMipCols = 128, kMipSplit = 8;  // axes 1 and 2: columns of a block, its rows at most

// Axis 0: a warp per row, so that its loads are contiguous.  152x256x724: 19 us
// for the call (112 MB, L2-resident in part) against 50 us with a thread per row.
__global__ void __launch_bounds__(256) k_mip_x(const float* __restrict__ in, int nx,
                                               long long rows, float* __restrict__ out) {
  const long long r = blockIdx.x * 8LL + (threadIdx.x >> 5);
  if (r >= rows) return;
  const float* p = in + r * nx;
  float m = -1e10f;
  for (int x0 = threadIdx.x & 31; x0 < nx; x0 += 32 * kMipBatch) {
    float v[kMipBatch];
#pragma unroll
    for (int u = 0; u < kMipBatch; ++u) v[u] = x0 + 32 * u < nx ? __ldg(p + x0 + 32 * u) : -1e10f;
#pragma unroll
    for (int u = 0; u < kMipBatch; ++u) m = fmaxf(m, v[u]);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) out[r] = m;
}

// Axes 1 and 2: the maximum of n values `step` apart for kMipCols neighbouring x and
// one `slow` index (z or y, `slow_step` apart); blockDim.y threads share a column: as
// many as keep all of the grid resident, so that it walks the planes together.
// 152x256x724: 21.9 and 22.6 us (25.4 and 20.1 us with one thread a column and
// no batches; 24.6 us on axis 2 where the grid takes two waves).
__global__ void __launch_bounds__(kMipCols* kMipSplit)
k_mip_col(const float* __restrict__ in, int nx, int n, long long step, long long slow_step,
          float* __restrict__ out) {
  __shared__ float red[kMipSplit][kMipCols];
  const unsigned cols = (nx + kMipCols - 1) / kMipCols, slow = blockIdx.x / cols;
  const int x = (blockIdx.x - slow * cols) * kMipCols + threadIdx.x;
  const int part = threadIdx.y, split = blockDim.y;
  float m = -1e10f;
  if (x < nx) {
    const float* p = in + slow * slow_step + x;
    for (int i0 = part; i0 < n; i0 += split * kMipBatch) {
      float v[kMipBatch];
#pragma unroll
      for (int u = 0; u < kMipBatch; ++u) {
        const int i = i0 + u * split;
        v[u] = i < n ? __ldg(p + i * step) : -1e10f;
      }
#pragma unroll
      for (int u = 0; u < kMipBatch; ++u) m = fmaxf(m, v[u]);
    }
  }
  red[part][threadIdx.x] = m;
  __syncthreads();
  if (part == 0 && x < nx) {
    for (int i = 1; i < split; ++i) m = fmaxf(m, red[i][threadIdx.x]);
    out[(long long)slow * nx + x] = m;
  }
}

int launch_mip(const float* in, int nx, int ny, int nz, int axis, float* out, cudaStream_t st) {
  if (axis < 0 || axis > 2) {
    set_error("mip", "axis must be 0, 1 or 2");
    return cudaErrorInvalidValue;
  }
  if (axis == 0) {
    const long long rows = (long long)ny * nz;
    k_mip_x<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(in, nx, rows, out);
  } else {
    const long long plane = (long long)ny * nx;
    const int n = axis == 1 ? ny : nz, slow = axis == 1 ? nz : ny;
    int split = 1;
    while (split < kMipSplit && (long long)nx * slow * 2 * split <= 2048LL * sm_count()) split *= 2;
    k_mip_col<<<ceil_div(nx, kMipCols) * slow, dim3(kMipCols, split), 0, st>>>(
        in, nx, n, axis == 1 ? nx : plane, axis == 1 ? plane : nx, out);
  }
  CDX_LAUNCH_CHECK("k_mip");
  return 0;
}

}  // namespace cdx
