// Shared pieces of the TMA tile-pipeline acoustic PML kernels (forward step
// in acoustic_stream_fwd.cu, fused boundary-saving adjoint step in
// acoustic_stream_bwd.cu).
//
// A persistent CTA walks tiles t = blockIdx.x + k * gridDim.x (shot fastest,
// then 128-column strip, then TZ-row band).  The haloed stencil rows of a
// tile -- (TZ + 2R) x W floats, W = 136 or 144 (see Row<R>) -- arrive in one
// of S shared-memory stages by TMA (cp.async.bulk.tensor); out-of-bounds box
// elements read as zero, which is the zero padding of conv2d(padding=order/2)
// (acoustic.py:71).  Thread 0 re-arms a stage with tile k+S as soon as all
// warps are done with tile k.  The point operands (previous field,
// coefficient planes) are fetched with 16-byte global loads issued before the
// stage wait, so their latency overlaps it; the coefficient planes are shared
// by all shots and stay in L2.  Each warp computes TZ/NW rows with a fully
// unrolled register window along z; lanes own 4 adjacent columns (float4),
// x-neighbours come from the staged row.  Every mbarrier wait is bounded and
// a timeout ends the CTA's loop at the next barrier.
#pragma once
#include <algorithm>

#include "sgb_common.cuh"
#include "acoustic_args.cuh"
#include "tma.cuh"

namespace sgb {

constexpr unsigned FULL = 0xffffffffu;

constexpr int round32(int n) { return (n + 31) / 32 * 32; }

// Width W of a staged stencil row and the offset LO of column x0 in it: the
// box spans columns [x0 - LO, x0 - LO + W).  136 floats (LO = 4) for even
// radii, 144 (LO = 8) for odd radii (keeps 2R rows a multiple of 128 bytes).
template <int R>
struct Row {
  static constexpr int W = (R % 2 == 0) ? TX + 8 : TX + 16;
  static constexpr int LO = (W - TX) / 2;
};

// Tile t -> (shot, strip, band), shot fastest; 32-bit arithmetic.
struct Tile {
  int b, x0, z0;
};
__device__ __forceinline__ Tile tile_geom(int t, int nshots, int ntx, int tz) {
  Tile g;
  g.b = t % nshots;
  const int rest = t / nshots;
  g.x0 = (rest % ntx) * TX;
  g.z0 = (rest / ntx) * tz;
  return g;
}
// The same for the tiles t, t + G, t + 2 G, ... of a CTA without a division per
// tile: (shot, strip, band) advance by those of G, with carries.
struct TileWalk {
  Tile g;      // of the current tile
  Tile d;      // of G
  int nshots, nx;  // carry limits: shots, ntx * TX
  __device__ __forceinline__ TileWalk(int t, int G, int nshots_, int ntx, int tz)
      : g(tile_geom(t, nshots_, ntx, tz)), d(tile_geom(G, nshots_, ntx, tz)), nshots(nshots_), nx(ntx * TX) {}
  __device__ __forceinline__ void next(int tz) {
    g.b += d.b;
    g.x0 += d.x0;
    g.z0 += d.z0;
    if (g.b >= nshots) {
      g.b -= nshots;
      g.x0 += TX;
    }
    if (g.x0 >= nx) {
      g.x0 -= nx;
      g.z0 += tz;
    }
  }
};

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// Value of component (rx & 3) of lane (rx >> 2)'s float4, for every lane.
__device__ __forceinline__ float gather_lane(const float4& v, int rx) {
  const int src = rx >> 2, m = rx & 3;
  const float a = __shfl_sync(FULL, v.x, src), b = __shfl_sync(FULL, v.y, src);
  const float c = __shfl_sync(FULL, v.z, src), d = __shfl_sync(FULL, v.w, src);
  return m == 0 ? a : (m == 1 ? b : (m == 2 ? c : d));
}

// Cross-stencil Laplacian (without 1/h^2) of the 4 columns of a lane at the
// centre row of `win`, x-neighbours from the staged row `srow` (its element
// Row<R>::LO is column x0).  Two columns per instruction: the tile kernels are
// bound by how many instructions their 16 warps per SM issue (427 per 128-point
// row of the 8th-order adjoint, half of the issue slots).  With the division-free
// walk above: 64 shots of 500 x 1100, 160 steps and their adjoint 44.7 -> 42.8 ms.
template <int R>
__device__ __forceinline__ float4 lap_row(const float4 (&win)[2 * R + 1], const float* srow, int lane,
                                          const FdWeights& w) {
  const float4 l = lds4(srow + Row<R>::LO - 4 + 4 * lane);
  const float4 r = lds4(srow + Row<R>::LO + 4 + 4 * lane);
  const float4 c = win[R];
  const float a[12] = {l.x, l.y, l.z, l.w, c.x, c.y, c.z, c.w, r.x, r.y, r.z, r.w};
  float2 o[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // columns 2h, 2h + 1
    const int m = 4 + 2 * h;
    F2 s = mul2(f2(w.c[0], w.c[0]), f2(a[m], a[m + 1]));
#pragma unroll
    for (int j = 1; j <= R; ++j) {
      const float4 &u = win[R + j], &d = win[R - j];
      // odd offsets straddle the register pairs of the loaded quads: scalar sums
      // (written as a pair) cost less than the moves that would pair their operands
      const F2 xs = (j & 1) ? f2(a[m + j] + a[m - j], a[m + 1 + j] + a[m + 1 - j])
                            : add2(f2(a[m + j], a[m + 1 + j]), f2(a[m - j], a[m + 1 - j]));
      const F2 zs = h == 0 ? add2(f2(u.x, u.y), f2(d.x, d.y)) : add2(f2(u.z, u.w), f2(d.z, d.w));
      s = fma2(f2(w.c[j], w.c[j]), add2(xs, zs), s);
    }
    o[h] = unpack(s);
  }
  return make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
}

// Sources of shot b in rows [zlo, zlo + nrow) and columns [x0, x0 + 128):
// one candidate per lane (the first 32 sources of the shot), as a ballot mask
// plus (row offset, column offset, value) in the owning lane.
struct WarpSrc {
  unsigned mask;
  int zl, xl;
  float v;
};
__device__ __forceinline__ WarpSrc warp_sources(int lane, int b, int zlo, int nrow, int x0, const int* src_ptr,
                                                const int* src_z, const int* src_x, const int* src_wrow,
                                                const float* wavelet, int nt, int t, int* status) {
  WarpSrc s{0u, -1, 0, 0.f};
  const int p0 = src_ptr[b], p1 = src_ptr[b + 1];
  const int q = p0 + lane;
  if (q < p1) {
    const int zs = src_z[q] - zlo, xs = src_x[q] - x0;
    if (zs >= 0 && zs < nrow && xs >= 0 && xs < TX) {
      s.zl = zs;
      s.xl = xs;
      s.v = wavelet[(long long)src_wrow[q] * nt + t];
    }
  }
  s.mask = __ballot_sync(FULL, s.zl >= 0);
  if (p1 - p0 > 32 && lane == 0) atomicOr(status, DEV_ERR_CAPACITY);
  return s;
}

// Add (sign = +1) or subtract (-1) the sources of local row i to v.
__device__ __forceinline__ void apply_sources(const WarpSrc& s, int i, int lane, float sign, float4& v) {
  unsigned m = s.mask;
  while (m) {
    const int srcl = __ffs(m) - 1;
    m &= m - 1;
    const int zl = __shfl_sync(FULL, s.zl, srcl), xl = __shfl_sync(FULL, s.xl, srcl);
    const float val = __shfl_sync(FULL, s.v, srcl);
    if (zl == i && (xl >> 2) == lane) set_comp(v, xl & 3, comp(v, xl & 3) + sign * val);
  }
}

// The receivers of shot b in the rows [z0, z0 + TZ) and columns [x0, x0 + TX)
// of a tile: f(row in tile, column in tile, rec_col) for each.  The rows of a
// shot are adjacent in the table, so all NWP warps of the CTA walk the band's
// receivers as one range, eight column loads per lane in flight (the columns
// of a row need not be sorted); the row of a receiver comes from the band's
// row pointers, one per lane.  With the receivers of a row walked by one warp
// and one load in flight, a tile on a row of 1000 receivers took about 10 us.
template <int TZ, int NWP, class F>
__device__ __forceinline__ void tile_receivers(const int* rp, const int* rec_x, const int* rec_col, int lane, int wid,
                                               int x0, int z0, int nz, const F& f) {
  static_assert(TZ <= 32, "one row pointer per lane");
  constexpr int U = 8;
  const int rows = min(TZ, nz - z0);
  const int pv = __ldg(rp + z0 + min(lane, rows - 1));  // first receiver of row `lane`
  const int p1 = __ldg(rp + z0 + rows);
  const int p0 = __shfl_sync(FULL, pv, 0);
  for (int q0 = p0 + wid * 32; q0 < p1; q0 += 32 * NWP * U) {
    int rx[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = q0 + u * 32 * NWP + lane;
      rx[u] = q < p1 ? __ldg(rec_x + q) - x0 : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = q0 + u * 32 * NWP + lane;
      const bool in = rx[u] >= 0 && rx[u] < TX;
      if (!__any_sync(FULL, in)) continue;
      int lr = 0;  // the last row whose first receiver is at or before q
      for (int r = 1; r < rows; ++r) lr += __shfl_sync(FULL, pv, r) <= q ? 1 : 0;
      if (in) f(lr, rx[u], __ldg(rec_col + q));
    }
  }
}

// Brings the table entries that tile_receivers will read first into L1, issued
// before a stage wait so that only the sampling itself follows the tile's stores.
template <int TZ, int NWP>
__device__ __forceinline__ void prefetch_receivers(const int* rp, const int* rec_x, const int* rec_col, int lane,
                                                   int wid, int z0, int nz) {
  const int p0 = __ldg(rp + z0), p1 = __ldg(rp + min(z0 + TZ, nz));
  const int q = p0 + (wid * 32 + lane) * 8;  // 32 bytes of each table per thread
  if (q < p1) {
    asm volatile("prefetch.global.L1 [%0];\n" ::"l"(rec_x + q));
    asm volatile("prefetch.global.L1 [%0];\n" ::"l"(rec_col + q));
  }
}

// This CTA's share of a boundary-ring copy between a field
// [nshots][nz][pitch] and its slots [nshots][ring.size] (slot order of
// Ring::index): scatter = slots -> field, else field -> slots.  Four
// elements per thread and round: their loads are issued together.
__device__ __forceinline__ void ring_copy_share(const Ring& ring, int nshots, int pitch, long long sstride,
                                                float* field, float* slots, bool scatter) {
  const long long n = (long long)nshots * ring.size;
  const long long stride = (long long)gridDim.x * blockDim.x;
  auto cell_ptr = [&](long long i) -> float* {
    const int b = (int)(i / ring.size);
    int z, x;
    ring.cell((int)(i - (long long)b * ring.size), z, x);
    return field + b * sstride + (long long)z * pitch + x;
  };
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    float* f[4];
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) f[q] = cell_ptr(i + q * stride);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = scatter ? slots[i + q * stride] : *f[q];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (scatter)
        *f[q] = v[q];
      else
        slots[i + q * stride] = v[q];
    }
  }
  for (; i < n; i += stride) {
    float* f = cell_ptr(i);
    if (scatter)
      *f = slots[i];
    else
      slots[i] = *f;
  }
}

template <class Kern>
static int resident_blocks(Kern kern, int threads, size_t smem) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, threads, smem) != cudaSuccess || nb < 1) nb = 1;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return nb * (sms > 0 ? sms : 152);
}

// Variant selection shared with the host (acoustic_stream.cu).
extern int g_fwd_cfg, g_bwd_cfg, g_habc_fwd_cfg;

}  // namespace sgb
