// Spectrum layout of the paired passes.
//
// Real rows y and y + H (H = ny/2, for ny not divisible by 4 the next multiple
// of 4, so that the halves start on the same alignment) of a slice are
// transformed along x as one complex row Z = row[y] + i row[y + H], and two such
// rows (y = 2m, 2m + 1) form a pair whose lanes a thread transforms together.  The x passes store
// the packed spectrum Z unsplit; the y pass, which reads both Z[kx] and
// Z[-kx] of a row, separates the two real rows' spectra as it loads them (the
// factor 1/2 is folded into the OTF).  For every kx <= nx/2 and z a row of
// 2 hp float4 slots (hp = H/2 rounded up to 4) holds
//   between the x and y passes: slot m < hp      Z[kx]  of pair m,
//                               slot hp + m      Z[-kx] of pair m,
//   after the forward y pass:   the columns ky of the half spectrum, two per
//                               slot: (k, k + ny/2) where the y pass splits
//                               even and odd rows (eo); (k + 2q kc, k + (2q + 1)
//                               kc) of one butterfly of an odd height's plan, its
//                               last kc columns as neighbours (kc); else (2p,
//                               2p + 1).
// A slot holds (re lane 0, re lane 1, im lane 0, im lane 1).  Row 0 and, for
// even nx, row nx/2 are their own mirror image and leave the second half
// unused.
//
// Memory order [z][slot / 4][kx][slot % 4]: the four slots of an x tile's rows
// are contiguous over all kx (nx/2 + 1 runs of 64 bytes back to back), a y tile
// of V neighbouring kx reads runs of 64 V bytes, and 16 neighbouring (kx, slot
// % 4) are a z tile with 256-byte runs.  Stored plane by plane ([kx][z][slot])
// the x passes read scattered 32- or 64-byte runs: x ratio 82 us with 32-byte
// and 73 us with 64-byte runs on the 100 x 256 x 756 grid.
#pragma once

#include "kernels.h"

namespace cdx {

constexpr int kNoColumn = 1 << 24;

struct PairGeom {
  int nx, ny, nz, nxh;
  int H, hp;   // row y shares a complex row with y + H; slots per half row
  int sb;      // blocks of 4 slots per row: hp / 2
  int slots;   // column pairs after the y pass
  int eo;      // 1: columns (k, k + ny/2)
  int kc;      // > 0: columns (k + 2q kc, k + (2q + 1) kc); neither: (2p, 2p + 1)
  int kcs, full;  // slots from one q to the next, slots of such pairs
  int per, last, step;  // other slots: columns per s + last and step further
  float inv_kcs;
  int zstep;   // slots per z: sb * nxh * 4
  int zrows;   // rows of the real arrays per z: ny
  // first column of slot s and how much further the second is; past ny: none.  (The quotient is exact: s + 1/2 lies
  // farther from the multiples of kcs than s < 2^20 rounds.)
  __host__ __device__ int col_step(int s) const { return s < full ? kc : step; }
  __host__ __device__ int col(int s) const {
    if (s >= full) return per * s + last;
    const int q = (int)(((float)s + 0.5f) * inv_kcs), k = s - q * kcs;
    return k < kc ? k + 2 * q * kc : kNoColumn;
  }
  // slot s of row (kx, z)
  __host__ __device__ long long slot(int kx, int z, int s) const {
    return (long long)z * zstep + ((long long)(s >> 2) * nxh + kx) * 4 + (s & 3);
  }
  // float index of the real part of column ky of row (kx, z); the imaginary
  // part is two floats further
  __host__ __device__ long long at(int kx, int z, int ky) const {
    const int h = ny >> 1;
    int s = ky >> 1, lane = ky & 1;
    if (eo) {
      lane = ky >= h;
      s = ky - lane * h;
    } else if (kc) {
      const int r = ky / kc, k = ky - r * kc;
      if (r == ny / kc - 1) {
        lane = k & 1;
        s = full + (k >> 1);
      } else {
        lane = r & 1;
        s = (r >> 1) * kcs + k;
      }
    }
    return 4 * slot(kx, z, s) + lane;
  }
};

// Slots from the first column of a stage C output pair to the next pair's: kc, or
// whole blocks of 4 where the row has room for the slots that leaves empty.
__host__ __device__ inline constexpr int pair_kcs(int ny, int kc) {
  const int up = (kc + 3) / 4 * 4;
  return kc && (ny / kc - 1) / 2 * up + (kc + 1) / 2 <= 2 * pair_half(ny) ? up : kc;
}
// Whether the arrays of an iteration are past what L2 holds of them.  Each pass
// then takes the slices in the order opposite to the one that wrote them, so that
// it finds the last ones still there: x forward up, y forward down, z, y inverse
// up, x ratio down, y forward up, z, y inverse up, x update down.  With every pass
// going up 108x500x980 took 1236 us an iteration against 1202, 96x375x800 657
// against 625 and 100x256x756 352 against 341; below the line it gains nothing
// (64x486x384, 11.9 M voxels: 243 us up, 246 alternating).
inline bool past_l2(const Geom& g) { return g.nvox() >= 12 << 20; }
inline PairGeom pair_geom(const Geom& g) {
  PairGeom p;
  p.nx = g.nx;
  p.ny = g.ny;
  p.nz = g.nz;
  p.nxh = g.nxh;
  p.H = pair_split(g.ny);
  p.hp = pair_half(g.ny);
  p.sb = p.hp / 2;
  p.slots = (g.ny + 1) / 2;
  p.eo = g.eo;
  p.kc = g.kc;
  p.kcs = pair_kcs(g.ny, g.kc);
  p.full = g.kc ? (g.ny / g.kc - 1) / 2 * p.kcs : 0;
  p.per = g.eo ? 1 : 2;
  p.last = g.kc ? g.ny - g.kc - 2 * p.full : 0;
  p.step = g.eo ? g.ny / 2 : 1;
  p.inv_kcs = g.kc ? 1.f / (float)p.kcs : 0.f;
  if (g.kc) p.slots = p.full + (g.kc + 1) / 2;
  p.zstep = p.sb * g.nxh * 4;
  p.zrows = g.ny;
  return p;
}
// The same for a pass that takes the slices from the last to the first: its kernels
// count up from the last slice with the steps turned round, at no cost to them (a
// choice made in the kernel took 1 of 118 us from 100x128x512).  Its arrays start at
// the last slice.
inline PairGeom pair_geom_down(const Geom& g) {
  PairGeom p = pair_geom(g);
  p.zstep = -p.zstep;
  p.zrows = -p.zrows;
  return p;
}
// Last slice of a spectrum, of a real array.
inline float2* last_slice(const PairGeom& up, float2* S) { return S + 2LL * (up.nz - 1) * up.zstep; }
template <class T>
T* last_slice_real(const PairGeom& up, T* x) {
  return x ? x + (long long)(up.nz - 1) * up.ny * up.nx : x;
}

#ifdef __CUDACC__
// Element (kx, z, ky) of a half spectrum in the layout of g.
__device__ __forceinline__ void st_spec(const Geom& g, const PairGeom& pg, float2* S, int kx, int z,
                                        int ky, float2 v) {
  if (g.pair) {
    float* p = reinterpret_cast<float*>(S) + pg.at(kx, z, ky);
    p[0] = v.x;
    p[2] = v.y;
  } else {
    S[(long long)kx * g.plane + (long long)z * g.nyp + ky] = v;
  }
}
#endif

// The paired passes (launchers of kernels.h dispatch to them when g.pair).
int launch_py(const PairGeom& g, const FftLen& fy, float2* S, bool inverse, cudaStream_t st);
int launch_pz(const PairGeom& g, const FftLen& fz, float2* S, const OtfDev& otf, bool conj,
              cudaStream_t st, bool fwd_only);

}  // namespace cdx
