// nufft_kernels.cu — the 2D NUFFT pair of the stack-of-spirals path on the device (reference
// `Nufft2`, nufft.rs:125-299): exponential-of-semicircle kernel exp(beta (sqrt(1 - z^2) - 1)),
// beta = 2.30 w, w = ceil(-log10 tol) + 1 clamped to 2..16, oversampling 2, deapodization by the
// kernel's sampled transform.  Type 1 spreads (tiles, in a fixed order), type 2 interpolates; the fine-grid
// FFT is a shared-memory radix-2 kernel (a direct DFT for lengths that are not powers of two).
// Point positions and kernel offsets are formed in FP64 (the kernel is steep: an FP32 position
// would cost ~1e-5 of relative accuracy); the taps and sums are FP32.
//
// Also the spiral forwards (spiral.rs): the exact sum over voxels at each sample and the
// time-segmented combination of L type-2 transforms.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "driver.h"
#include "es_taps.cuh"
#include "host_tables.h"
#include "mrsim_internal.h"
#include "nufft.h"

namespace mrsim {

namespace {

__device__ __forceinline__ int wrap(int m, int n) {
  m %= n;
  return m < 0 ? m + n : m;
}

template <class R>
__device__ __forceinline__ typename Vec2<R>::type mk2(R a, R b);
template <>
__device__ __forceinline__ float2 mk2<float>(float a, float b) {
  return make_float2(a, b);
}
template <>
__device__ __forceinline__ double2 mk2<double>(double a, double b) {
  return make_double2(a, b);
}
// In FP64 as on the host, where 65,536 samples' sines took 2 ms.
__global__ void spiral_stat_kernel(const double* __restrict__ k, int npts, int snx, int sny, double xoff, double yoff,
                                   float2* __restrict__ stat) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npts) return;
  const double ninv = 1.0 / ((double)snx * sny);
  double sn, cs;
  sincos(-kTau * (k[2 * j] * xoff / snx + k[2 * j + 1] * yoff / sny), &sn, &cs);
  stat[j] = make_float2((float)(cs * ninv), (float)(sn * ninv));
}

template <class R>
__global__ void place_kernel(const NufftGridT<R> g, const typename Vec2<R>::type* __restrict__ modes,
                             typename Vec2<R>::type* __restrict__ grid, int batch, size_t mode_stride,
                             size_t grid_stride, const R* __restrict__ scale) {
  using V = typename Vec2<R>::type;
  const int b = blockIdx.y;
  const int nmodes = g.m_out0 * g.m_out1;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nmodes; e += gridDim.x * blockDim.x) {
    const int j0 = e % g.m_out0, j1 = e / g.m_out0;
    const int b0 = wrap(g.m_lo0 + j0, g.nf0), b1 = wrap(g.m_lo1 + j1, g.nf1);
    V v = modes[b * mode_stride + e];
    R s = g.corr0[j0] * g.corr1[j1];
    if (scale) s *= scale[b];
    grid[b * grid_stride + (size_t)b0 + (size_t)g.nf0 * b1] = mk2<R>(v.x * s, v.y * s);
  }
}

template <class R>
__global__ void extract_kernel(const NufftGridT<R> g, const typename Vec2<R>::type* __restrict__ grid,
                               typename Vec2<R>::type* __restrict__ modes, size_t grid_stride, size_t mode_stride) {
  using V = typename Vec2<R>::type;
  const int b = blockIdx.y;
  const int nmodes = g.m_out0 * g.m_out1;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nmodes; e += gridDim.x * blockDim.x) {
    const int j0 = e % g.m_out0, j1 = e / g.m_out0;
    const int b0 = wrap(g.m_lo0 + j0, g.nf0), b1 = wrap(g.m_lo1 + j1, g.nf1);
    const V v = grid[b * grid_stride + (size_t)b0 + (size_t)g.nf0 * b1];
    const R s = g.corr0[j0] * g.corr1[j1];
    modes[b * mode_stride + e] = mk2<R>(v.x * s, v.y * s);
  }
}

// One CTA per line of length n (power of two): stride between elements `es`, between lines
// `ls`; lines = blockIdx.x within batch item blockIdx.y (batch stride `bs`).
template <class V>
__global__ void fft_pow2_kernel(V* __restrict__ data, int n, int logn, size_t es, size_t ls, size_t bs,
                                const V* __restrict__ tw, int sign) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  V* buf = reinterpret_cast<V*>(fft_smem);
  V* base = data + blockIdx.y * bs + blockIdx.x * ls;
  // bit-reversed load
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int r = __brev(i) >> (32 - logn);
    buf[r] = base[(size_t)i * es];
  }
  __syncthreads();
  for (int s = 1; s <= logn; ++s) {
    const int m = 1 << s, h = m >> 1;
    for (int t = threadIdx.x; t < n / 2; t += blockDim.x) {
      const int grp = t / h, pos = t % h;
      const int i0 = grp * m + pos, i1 = i0 + h;
      V w = tw[(size_t)pos * (n / m)];  // e^{-i 2 pi pos / m}
      if (sign > 0) w.y = -w.y;
      const V a = buf[i0], b = buf[i1];
      V bw;
      bw.x = b.x * w.x - b.y * w.y;
      bw.y = b.x * w.y + b.y * w.x;
      V s0, s1;
      s0.x = a.x + bw.x;
      s0.y = a.y + bw.y;
      s1.x = a.x - bw.x;
      s1.y = a.y - bw.y;
      buf[i0] = s0;
      buf[i1] = s1;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) base[(size_t)i * es] = buf[i];
}

// Direct DFT of one line (any n), e^{sign i 2 pi j k / n}.
template <class V>
__global__ void dft_line_kernel(V* __restrict__ data, int n, size_t es, size_t ls, size_t bs, const V* __restrict__ tw,
                                int sign) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  V* buf = reinterpret_cast<V*>(fft_smem);
  V* base = data + blockIdx.y * bs + blockIdx.x * ls;
  for (int i = threadIdx.x; i < n; i += blockDim.x) buf[i] = base[(size_t)i * es];
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    decltype(V().x) ar = 0, ai = 0;
    for (int j = 0; j < n; ++j) {
      V w = tw[((long long)j * k) % n];
      if (sign > 0) w.y = -w.y;
      const V a = buf[j];
      ar = fma(a.x, w.x, fma(-a.y, w.y, ar));
      ai = fma(a.x, w.y, fma(a.y, w.x, ai));
    }
    V o;
    o.x = ar;
    o.y = ai;
    base[(size_t)k * es] = o;  // inputs are in shared memory: no hazard
  }
}

constexpr int kBatchBlock = 4;  // batch items a type-1 or type-2 thread serves with one set of taps

// Type 2: out[j] = sum over the w x w taps of grid, for each point of each batch item; a thread
// serves one point for up to kBatchBlock batch items (blockIdx.y), forming the taps once.  The tap
// loops run to the compile-time bound kWMax (guarded by w), so taps and column indices live in
// registers; a window wraps at most once when the fine grid is at least 2 kWMax wide (else the
// general modulo).
template <class R>
__global__ void __launch_bounds__(128) interp_kernel(const NufftGridT<R> g, const typename Vec2<R>::type* __restrict__ grid,
                                                     const double* __restrict__ u, int npts,
                                                     typename Vec2<R>::type* __restrict__ out, size_t grid_stride,
                                                     size_t out_stride, int batch) {
  using V = typename Vec2<R>::type;
  const int b0 = blockIdx.y * kBatchBlock, nb = min(kBatchBlock, batch - b0);
  const int w = g.w;
  const bool wide = g.nf0 >= 2 * kWMax && g.nf1 >= 2 * kWMax;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < npts; j += gridDim.x * blockDim.x) {
    R k0[kWMax], k1[kWMax];
    const int a0 = es_taps<R>(u[2 * j], g.nf0, w, g.beta, k0);
    const int a1 = es_taps<R>(u[2 * j + 1], g.nf1, w, g.beta, k1);
    int col[kWMax];
#pragma unroll
    for (int i0 = 0; i0 < kWMax; ++i0) {
      int c = a0 + i0;
      if (wide) {
        c = c < 0 ? c + g.nf0 : c;
        c = c >= g.nf0 ? c - g.nf0 : c;
      } else {
        c = wrap(c, g.nf0);
      }
      col[i0] = c;
    }
    R re[kBatchBlock], im[kBatchBlock];
#pragma unroll
    for (int q = 0; q < kBatchBlock; ++q) re[q] = im[q] = 0;
#pragma unroll
    for (int i1 = 0; i1 < kWMax; ++i1) {
      if (i1 >= w) break;
      int c1 = a1 + i1;
      if (wide) {
        c1 = c1 < 0 ? c1 + g.nf1 : c1;
        c1 = c1 >= g.nf1 ? c1 - g.nf1 : c1;
      } else {
        c1 = wrap(c1, g.nf1);
      }
      const V* row = grid + (size_t)g.nf0 * c1;
      R rr[kBatchBlock], ri[kBatchBlock];
#pragma unroll
      for (int q = 0; q < kBatchBlock; ++q) rr[q] = ri[q] = 0;
#pragma unroll
      for (int i0 = 0; i0 < kWMax; ++i0) {
        if (i0 >= w) break;
#pragma unroll
        for (int q = 0; q < kBatchBlock; ++q)
          if (q < nb) {
            const V v = __ldg(row + (size_t)(b0 + q) * grid_stride + col[i0]);
            rr[q] = fma(v.x, k0[i0], rr[q]);
            ri[q] = fma(v.y, k0[i0], ri[q]);
          }
      }
#pragma unroll
      for (int q = 0; q < kBatchBlock; ++q) {
        re[q] = fma(rr[q], k1[i1], re[q]);
        im[q] = fma(ri[q], k1[i1], im[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < kBatchBlock; ++q)
      if (q < nb) out[(size_t)(b0 + q) * out_stride + j] = mk2<R>(re[q], im[q]);
  }
}

// The wrapped offset of cell c from a window start a on a ring of n cells, in [0, n).
__device__ __forceinline__ int ring_offset(int c, int a, int n) {
  int d = c - a;
  while (d < 0) d += n;
  while (d >= n) d -= n;
  return d;
}

// ---- the points of each spread tile ---------------------------------------------------------------
// lo[axis][j]: the ring cell one before the point's window (the window is widened by a cell each side);
// -1 where either coordinate has no position (its taps are zero: it reaches no tile).
__global__ void bins_origin_kernel(const double* __restrict__ u, int npts, int nf0, int nf1, int w, int* __restrict__ lo) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npts) return;
  double p0, p1;
  const int a0 = es_origin(u[2 * j], nf0, 0.5 * w, p0), a1 = es_origin(u[2 * j + 1], nf1, 0.5 * w, p1);
  const bool ok = p0 >= 0.0 && p1 >= 0.0;
  lo[j] = ok ? wrap(a0 - 1, nf0) : -1;
  lo[npts + j] = ok ? wrap(a1 - 1, nf1) : -1;
}

// One block per tile of one axis and parent list (block = parent * tiles + tile): the parent's points
// (p_start / p_pts; NULL: all npts in order) whose `span` cells from lo[j] on meet the tile's, counted
// (count != NULL) or stored from start[block] on, in the parent's order.
constexpr int kBinThreads = 256;
__global__ void __launch_bounds__(kBinThreads) bins_select_kernel(const int* __restrict__ lo, int npts,
                                                                  const int* __restrict__ p_start,
                                                                  const int* __restrict__ p_pts, int tiles, int nf,
                                                                  int span, int* __restrict__ count,
                                                                  const int* __restrict__ start, int* __restrict__ pts) {
  __shared__ int part[kBinThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int parent = blockIdx.x / tiles, t0 = (blockIdx.x % tiles) * kSpreadTile, len = min(kSpreadTile, nf - t0);
  const int b0 = p_start ? p_start[parent] : 0, b1 = p_start ? p_start[parent + 1] : npts;
  int at = count ? 0 : start[blockIdx.x];
  for (int base = b0; base < b1; base += kBinThreads) {
    int j = -1;
    bool hit = false;
    if (base + tid < b1) {
      j = p_pts ? p_pts[base + tid] : base + tid;
      const int l = lo[j];
      int d = t0 - l;  // from the span's first cell to the tile's, and back, around the ring
      int e = -d;
      if (d < 0) d += nf;
      if (e < 0) e += nf;
      hit = l >= 0 && (d < span || e < len);
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) part[warp] = __popc(m);
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kBinThreads / 32; ++w) {
      before += w < warp ? part[w] : 0;
      total += part[w];
    }
    if (hit && !count) pts[at + before + __popc(m & ((1u << lane) - 1u))] = j;
    at += total;
    __syncthreads();
  }
  if (count && tid == 0) count[blockIdx.x] = at;
}

// One block: start[i] = sum of count[0 .. i), start[n] the total.
__global__ void __launch_bounds__(1024) bins_scan_kernel(const int* __restrict__ count, int n, int* __restrict__ start) {
  __shared__ int part[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, per = (n + 1023) / 1024;
  const int i0 = min(n, tid * per), i1 = min(n, i0 + per);
  int v = 0;
  for (int i = i0; i < i1; ++i) v += count[i];
  int x = v;
#pragma unroll
  for (int h = 1; h < 32; h <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, x, h);
    if (lane >= h) x += o;
  }
  if (lane == 31) part[warp] = x;
  __syncthreads();
  x -= v;
  for (int w = 0; w < warp; ++w) x += part[w];
  for (int i = i0; i < i1; ++i) {
    start[i] = x;
    x += count[i];
  }
  if (tid == 1023) start[n] = x;
}

constexpr int kSpreadChunk = 64;  // points whose taps a spread block holds at a time

// Type 1 spreading without atomics: one block per 8 x 8 tile of the fine grid and group of up to
// kBatchBlock batch items (the taps formed once for the group).  The tile's points (nufft_bins2: every
// point whose window can reach the tile, in point order) pass through shared memory in chunks with
// their taps; the block's kSpreadParts parts (a thread per cell each) take every kSpreadParts-th point of
// a chunk, add w_j (k0 k1) (nufft.rs:236-250) to their own sums, and the parts are added in order at
// the end: a tile's points are one serial chain of additions per cell otherwise, and at one item a few
// hundred tiles of 64 threads leave the chip idle (65,536 points on a 128 x 128 fine grid: 0.97 ms
// with one part, 0.38 with four).  The order is fixed, so the grid is the same on every run; a window that
// wraps onto a cell twice (a fine grid narrower than the kernel) adds both taps.
constexpr int kSpreadParts = 4, kCellsPerTile = kSpreadTile * kSpreadTile;
template <class R>
__global__ void __launch_bounds__(kCellsPerTile * kSpreadParts)
    spread_tile_kernel(const NufftGridT<R> g, typename Vec2<R>::type* __restrict__ grid, const double* __restrict__ u,
                       const typename Vec2<R>::type* __restrict__ wts, size_t grid_stride, size_t w_stride,
                       const NufftBins bins, int batch) {
  using V = typename Vec2<R>::type;
  __shared__ R sk0[kSpreadChunk][kWMax], sk1[kSpreadChunk][kWMax];
  __shared__ int sa0[kSpreadChunk], sa1[kSpreadChunk];
  __shared__ V sw[kBatchBlock][kSpreadChunk];
  __shared__ V sums[kSpreadParts - 1][kCellsPerTile];
  const int b0 = blockIdx.y * kBatchBlock, nb = min(kBatchBlock, batch - b0), tile = blockIdx.x;
  const int cell = (int)threadIdx.x % kCellsPerTile, part = (int)threadIdx.x / kCellsPerTile;
  const int c0 = (tile % bins.tiles0) * kSpreadTile + cell % kSpreadTile;
  const int c1 = (tile / bins.tiles0) * kSpreadTile + cell / kSpreadTile;
  const bool mine = c0 < g.nf0 && c1 < g.nf1;
  const int w = g.w;
  R re[kBatchBlock], im[kBatchBlock];
#pragma unroll
  for (int q = 0; q < kBatchBlock; ++q) re[q] = im[q] = 0;
  const int p0 = bins.start[tile], p1 = bins.start[tile + 1];
  for (int base = p0; base < p1; base += kSpreadChunk) {
    const int n = min(kSpreadChunk, p1 - base);
    // the two axes' taps and the weights by different threads
    const int t = (int)threadIdx.x % kSpreadChunk, job = (int)threadIdx.x / kSpreadChunk;
    if (t < n) {
      const int j = bins.pts[base + t];
      if (job == 0) sa0[t] = es_taps<R>(u[2 * j], g.nf0, w, g.beta, sk0[t]);
      if (job == 1) sa1[t] = es_taps<R>(u[2 * j + 1], g.nf1, w, g.beta, sk1[t]);
      if (job == 2) {
#pragma unroll
        for (int q = 0; q < kBatchBlock; ++q)
          if (q < nb) sw[q][t] = wts[(size_t)(b0 + q) * w_stride + j];
      }
    }
    __syncthreads();
    if (mine)
      for (int q = part; q < n; q += kSpreadParts) {
        const int d0 = ring_offset(c0, sa0[q], g.nf0);
        if (d0 >= w) continue;
        const int d1 = ring_offset(c1, sa1[q], g.nf1);
        if (d1 >= w) continue;
        for (int i1 = d1; i1 < w; i1 += g.nf1)
          for (int i0 = d0; i0 < w; i0 += g.nf0) {
            const R v = sk0[q][i0] * sk1[q][i1];
#pragma unroll
            for (int bq = 0; bq < kBatchBlock; ++bq) {
              re[bq] += sw[bq][q].x * v;
              im[bq] += sw[bq][q].y * v;
            }
          }
      }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < kBatchBlock; ++q) {
    if (q >= nb) break;
    if (part > 0) sums[part - 1][cell] = mk2<R>(re[q], im[q]);
    __syncthreads();
    if (part == 0 && mine) {
      for (int o = 0; o < kSpreadParts - 1; ++o) {
        re[q] += sums[o][cell].x;
        im[q] += sums[o][cell].y;
      }
      grid[(size_t)(b0 + q) * grid_stride + (size_t)c0 + (size_t)g.nf0 * c1] = mk2<R>(re[q], im[q]);
    }
    __syncthreads();
  }
}

// The taps and window origins of every point, once for all batch items: [j][kWMax] of each axis, zero from w.
__global__ void spread_taps_kernel(const NufftGridT<double> g, const double* __restrict__ u, int npts,
                                   double* __restrict__ taps, int2* __restrict__ org) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npts) return;
  double k0[kWMax], k1[kWMax];
#pragma unroll
  for (int i = 0; i < kWMax; ++i) k0[i] = k1[i] = 0.0;
  org[j] = make_int2(es_taps<double>(u[2 * j], g.nf0, g.w, g.beta, k0),
                     es_taps<double>(u[2 * j + 1], g.nf1, g.w, g.beta, k1));
  double* t = taps + (size_t)j * 2 * kWMax;
#pragma unroll
  for (int i = 0; i < kWMax; ++i) {
    t[i] = k0[i];
    t[kWMax + i] = k1[i];
  }
}

// The same spread for many items, FP64: a lane is a batch item, a warp holds two rows of the tile for it,
// so a point's taps are broadcasts and its weight is read from shared memory once for 16 cells.  With a
// thread per cell and four items, 58 % of the threads a point visits are outside its window and every
// contribution waits for its own loads: 576 items at 65,536 points on a 128 x 128 fine grid took
// 28.1 ms, here 4.2.  No pipe is full (shared memory 38 %, FP64 27 %, issue 46 % of the cycles, at 26 %
// occupancy): a chunk's loads and its sums alternate at its barriers.  Points are added in their order in
// the tile.
constexpr int kItemLanes = 32, kItemChunk = 32, kPadTaps = 8 + kWMax + 8;
__global__ void __launch_bounds__(128) spread_items_kernel(const NufftGridT<double> g, double2* __restrict__ grid,
                                                           const double* __restrict__ taps, const int2* __restrict__ org,
                                                           const double2* __restrict__ wts, size_t grid_stride,
                                                           size_t w_stride, const NufftBins bins, int batch) {
  __shared__ double sk0[kItemChunk][kPadTaps], sk1[kItemChunk][kPadTaps];  // taps at 8 .. 8 + w, zeros around
  __shared__ double2 sw[kItemChunk][kItemLanes + 1];
  __shared__ int2 so[kItemChunk];  // the tile's first cell within each window (negative before it)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x;
  const int b0 = blockIdx.y * kItemLanes, nb = min(kItemLanes, batch - b0);
  const int x0 = (tile % bins.tiles0) * kSpreadTile, y0 = (tile / bins.tiles0) * kSpreadTile;
  const int w = g.w;
  for (int i = tid; i < kItemChunk * 8; i += 128) {
    const int p = i / 8, x = i % 8;
    sk0[p][x] = sk0[p][8 + kWMax + x] = sk1[p][x] = sk1[p][8 + kWMax + x] = 0.0;
  }
  double re[2][kSpreadTile], im[2][kSpreadTile];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int x = 0; x < kSpreadTile; ++x) re[r][x] = im[r][x] = 0.0;
  const int p0 = bins.start[tile], p1 = bins.start[tile + 1];
  for (int base = p0; base < p1; base += kItemChunk) {
    const int n = min(kItemChunk, p1 - base);
    __syncthreads();
    for (int i = tid; i < n * 2 * kWMax; i += 128) {
      const int p = i / (2 * kWMax), x = i % (2 * kWMax);
      const double t = taps[(size_t)bins.pts[base + p] * (2 * kWMax) + x];
      (x < kWMax ? sk0[p][8 + x] : sk1[p][8 + x - kWMax]) = t;
    }
    const int j = lane < n ? bins.pts[base + lane] : 0;
    if (warp == 0 && lane < n) {
      const int2 o = org[j];
      int d0 = ring_offset(x0, o.x, g.nf0), d1 = ring_offset(y0, o.y, g.nf1);
      d0 = d0 > g.nf0 / 2 ? d0 - g.nf0 : d0;
      d1 = d1 > g.nf1 / 2 ? d1 - g.nf1 : d1;
      so[lane] = make_int2(d0, d1);
    }
    if (lane < n)
      for (int b = warp; b < kItemLanes; b += 4)  // neighbouring lanes take neighbouring points
        sw[lane][b] = b < nb ? wts[(size_t)(b0 + b) * w_stride + j] : make_double2(0.0, 0.0);
    __syncthreads();
    for (int q = 0; q < n; ++q) {
      const int d0 = so[q].x, d1 = so[q].y + 2 * warp;  // of column 0, of this warp's first row
      if (d0 <= -kSpreadTile || d0 >= w || d1 < -1 || d1 >= w) continue;
      const double2 v = sw[q][lane];
      const double ka = sk1[q][8 + d1], kb = sk1[q][9 + d1];
      const double2 va = make_double2(v.x * ka, v.y * ka), vb = make_double2(v.x * kb, v.y * kb);
      const double* k0 = &sk0[q][8 + d0];
#pragma unroll
      for (int x = 0; x < kSpreadTile; ++x) {
        const double k = k0[x];
        re[0][x] += va.x * k;
        im[0][x] += va.y * k;
        re[1][x] += vb.x * k;
        im[1][x] += vb.y * k;
      }
    }
  }
  if (lane >= nb) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int c1 = y0 + 2 * warp + r;
    if (c1 >= g.nf1) continue;
    double2* out = grid + (size_t)(b0 + lane) * grid_stride + (size_t)g.nf0 * c1 + x0;
#pragma unroll
    for (int x = 0; x < kSpreadTile; ++x)
      if (x0 + x < g.nf0) out[x] = make_double2(re[r][x], im[r][x]);
  }
}

// ---- the 1D type-1 NUFFT (`Nufft1`, nufft.rs:25-112), FP64 --------------------------------------
// Spreading without atomics: one block per 256-cell tile of the fine grid and weight vector, one
// thread per cell; the tile's points (nufft_bins1, in point order) pass through shared memory with
// their taps, and each cell adds g += w_j k_i point after point as the reference does
// (nufft.rs:80-97).
__global__ void __launch_bounds__(kSpreadTile1)
    spread1_tile_kernel(const double* __restrict__ pos, const double2* __restrict__ wts, int npos, int nf, int w,
                        double beta, double2* __restrict__ grid, const NufftBins bins) {
  __shared__ double sk[kSpreadChunk][kWMax];
  __shared__ int sm0[kSpreadChunk];
  __shared__ double2 sw[kSpreadChunk];
  const int q = blockIdx.y, tile = blockIdx.x;
  const int c = tile * kSpreadTile1 + (int)threadIdx.x;
  const bool mine = c < nf;
  double re = 0.0, im = 0.0;
  const int p0 = bins.start[tile], p1 = bins.start[tile + 1];
  for (int base = p0; base < p1; base += kSpreadChunk) {
    const int n = min(kSpreadChunk, p1 - base);
    if ((int)threadIdx.x < n) {
      const int t = threadIdx.x, j = bins.pts[base + t];
      sm0[t] = es_taps<double>(pos[j], nf, w, beta, sk[t]);  // fine position 2 pos on nf = 2n cells
      sw[t] = wts[(size_t)q * npos + j];
    }
    __syncthreads();
    if (mine)
      for (int t = 0; t < n; ++t) {
        const int d = ring_offset(c, sm0[t], nf);
        for (int i = d; i < w; i += nf) {
          re += sw[t].x * sk[t][i];
          im += sw[t].y * sk[t][i];
        }
      }
    __syncthreads();
  }
  if (mine) grid[(size_t)q * nf + c] = make_double2(re, im);
}

__global__ void extract1_kernel(const double2* __restrict__ grid, int nf, int k_lo, int n_out,
                                const double* __restrict__ corr, int nw, double2* __restrict__ out) {
  const int q = blockIdx.y;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n_out; j += gridDim.x * blockDim.x) {
    const double2 v = grid[(size_t)q * nf + wrap(k_lo + j, nf)];
    out[(size_t)q * n_out + j] = make_double2(v.x * corr[j], v.y * corr[j]);
  }
}

// ---- spiral forwards ---------------------------------------------------------------------------
// The exact sum (`spiral_kspace_exact`, spiral.rs:107-137): one thread per sample, voxels staged
// in shared memory in tiles; the k.r + f tau phase in FP64 (nonuniform k), reduced to turns.
constexpr int kTileVox = 256;

__global__ void __launch_bounds__(256) spiral_exact_kernel(const SpiralExactArgs a) {
  __shared__ double sx[kTileVox], sy[kTileVox];
  __shared__ float sr[kTileVox], sph[kTileVox], samp[kTileVox];
  __shared__ float sm[kTileVox][4];
  __shared__ float sd[kTileVox][4];
  __shared__ float sla[kTileVox];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const bool ok = j < a.npts;
  double kx = 0, ky = 0;
  float tau = 0.f;
  if (ok) {
    kx = a.k[2 * j] / a.nx;
    ky = a.k[2 * j + 1] / a.ny;
    tau = (float)a.tau_ms[j];
  }
  const double taus = ok ? a.tau_ms[j] / 1000.0 : 0.0;
  float re = 0.f, im = 0.f;
  const int nvox = a.snx * a.sny;
  for (int v0 = 0; v0 < nvox; v0 += kTileVox) {
    __syncthreads();
    for (int t = threadIdx.x; t < kTileVox; t += blockDim.x) {
      const int i = v0 + t;
      if (i < nvox) {
        const int x = i % a.snx, y = i / a.snx;
        sx[t] = ((double)x - a.sxs - a.xoff) / a.ox;
        sy[t] = ((double)y - a.sys - a.yoff) / a.oy;
        sr[t] = a.rate ? a.rate[i] : 0.f;
        sph[t] = a.phase_turns ? a.phase_turns[i] : 0.f;
        samp[t] = a.amp[i];
        sla[t] = a.log_amp ? a.log_amp[i] : 0.f;
        for (int c = 0; c < 4; ++c) {
          sm[t][c] = c < a.ncomp ? a.comp[(size_t)c * nvox + i] : 0.f;
          sd[t][c] = (a.decay && c < a.ncomp) ? a.decay[(size_t)c * nvox + i] : 0.f;
        }
      } else {
        samp[t] = 0.f;
        sla[t] = 0.f;
        for (int c = 0; c < 4; ++c) sm[t][c] = sd[t][c] = 0.f;
        sx[t] = sy[t] = 0.0;
        sr[t] = sph[t] = 0.f;
      }
    }
    __syncthreads();
    if (!ok) continue;
    const int nt = min(kTileVox, nvox - v0);
    for (int t = 0; t < nt; ++t) {
      // w = sum_c m_c exp(ln A - tau d_c) under relaxation, sum_c m_c otherwise (spiral.rs:75-80)
      float w = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c < a.ncomp) {
          const float e = a.relax ? __expf(sla[t] - tau * sd[t][c]) : 1.f;
          w = fmaf(sm[t][c], e, w);
        }
      }
      if (w == 0.f) continue;
      double th = kx * sx[t] + ky * sy[t] + (double)sr[t] * taus;
      th -= rint(th);
      float thf = (float)th + sph[t];
      thf -= rintf(thf);
      float sn, cs;
      sincospif(2.0f * thf, &sn, &cs);
      const float amp = samp[t] * w;
      re = fmaf(amp, cs, re);
      im = fmaf(amp, sn, im);
    }
  }
  if (ok) a.out[j] = make_float2(re * a.inv_nvox, im * a.inv_nvox);
}

// Segment images: img_l(r) = x(r) e^{rate(r) tau_l} for every segment l (spiral.rs:174-201).
__global__ void segment_images_kernel(const float2* __restrict__ x, const float2* __restrict__ rate, int nvox,
                                      const double* __restrict__ tau_l, int L, float2* __restrict__ out) {
  const int l = blockIdx.y;
  const double tl = tau_l[l];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nvox; i += gridDim.x * blockDim.x) {
    const float2 r = rate[i];
    const float mag = __expf(r.x * (float)tl);
    double th = (double)r.y * tl / 6.283185307179586;
    th -= rint(th);
    float sn, cs;
    sincospif(2.0f * (float)th, &sn, &cs);
    const float2 v = x[i];
    const float er = mag * cs, ei = mag * sn;
    out[(size_t)l * nvox + i] = make_float2(v.x * er - v.y * ei, v.x * ei + v.y * er);
  }
}

// out_j = stat_j * sum_l b[tau_idx_j][l] * seg[l][j]
__global__ void segment_combine_kernel(const float2* __restrict__ seg, int npts, int L, const int* __restrict__ tau_idx,
                                       const double* __restrict__ b, const float2* __restrict__ stat,
                                       float2* __restrict__ out, int by_point) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < npts; j += gridDim.x * blockDim.x) {
    const double* bj = b + (size_t)tau_idx[j] * L * 2;
    float re = 0.f, im = 0.f;
    for (int l = 0; l < L; ++l) {
      const float2 v = seg[by_point ? (size_t)j * L + l : (size_t)l * npts + j];
      const float br = (float)bj[2 * l], bi = (float)bj[2 * l + 1];
      re = fmaf(br, v.x, fmaf(-bi, v.y, re));
      im = fmaf(br, v.y, fmaf(bi, v.x, im));
    }
    const float2 s = stat[j];
    out[j] = make_float2(re * s.x - im * s.y, re * s.y + im * s.x);
  }
}

}  // namespace

// ---- launchers ------------------------------------------------------------------------------------
template <class V>
void fft2(V* grid, int n0, int n1, const V* tw0, const V* tw1, int batch, int sign, cudaStream_t st) {
  const size_t gs = (size_t)n0 * n1;
  // rows (axis 0, contiguous), then columns (axis 1, stride n0)
  for (int axis = 0; axis < 2; ++axis) {
    const int n = axis == 0 ? n0 : n1;
    if (n == 1) continue;  // a length-1 transform is the identity
    const int lines = axis == 0 ? n1 : n0;
    const size_t es = axis == 0 ? 1 : (size_t)n0;
    const size_t ls = axis == 0 ? (size_t)n0 : 1;
    const V* tw = axis == 0 ? tw0 : tw1;
    const int threads = std::min(256, std::max(32, n / 2));
    dim3 grid_dim(lines, batch);
    const size_t smem = sizeof(V) * n;  // n <= 16384: at most 256 KiB in FP64, refused above 227 KiB
    if ((n & (n - 1)) == 0) {
      int logn = 0;
      while ((1 << logn) < n) ++logn;
      if (smem > 48 * 1024)
        cudaFuncSetAttribute(fft_pow2_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      fft_pow2_kernel<V><<<grid_dim, threads, smem, st>>>(grid, n, logn, es, ls, gs, tw, sign);
    } else {
      if (smem > 48 * 1024)
        cudaFuncSetAttribute(dft_line_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      dft_line_kernel<V><<<grid_dim, std::min(256, n), smem, st>>>(grid, n, es, ls, gs, tw, sign);
    }
  }
}
template void fft2<float2>(float2*, int, int, const float2*, const float2*, int, int, cudaStream_t);
template void fft2<double2>(double2*, int, int, const double2*, const double2*, int, int, cudaStream_t);

template <class R>
void nufft_type2(const NufftGridT<R>& g, const typename Vec2<R>::type* modes, int batch, size_t mode_stride,
                 const double* u, int npts, typename Vec2<R>::type* out, size_t out_stride,
                 typename Vec2<R>::type* work, int sign, const R* scale, cudaStream_t st) {
  using V = typename Vec2<R>::type;
  const size_t gs = (size_t)g.nf0 * g.nf1;
  cudaMemsetAsync(work, 0, gs * batch * sizeof(V), st);
  dim3 pg((g.m_out0 * g.m_out1 + 255) / 256, batch);
  place_kernel<R><<<pg, 256, 0, st>>>(g, modes, work, batch, mode_stride, gs, scale);
  nufft_fft2(g, work, batch, sign, st);
  dim3 ig(std::max(1, std::min((npts + 127) / 128, 4096)), (batch + kBatchBlock - 1) / kBatchBlock);
  interp_kernel<R><<<ig, 128, 0, st>>>(g, work, u, npts, out, gs, out_stride, batch);
}

template <class R>
void nufft_type1(const NufftGridT<R>& g, const double* u, int npts, const NufftBins& bins,
                 const typename Vec2<R>::type* wts, int batch, size_t w_stride, typename Vec2<R>::type* modes,
                 size_t mode_stride, typename Vec2<R>::type* work, int sign, cudaStream_t st, void* taps) {
  const size_t gs = (size_t)g.nf0 * g.nf1;
  // every cell of every tile is written (zero where no point reaches it)
  bool done = false;
  if constexpr (sizeof(R) == 8) {
    if (taps) {
      double* t = (double*)taps;
      int2* org = (int2*)(t + (size_t)npts * 2 * kWMax);
      spread_taps_kernel<<<(npts + 127) / 128, 128, 0, st>>>(g, u, npts, t, org);
      dim3 ig(bins.tiles0 * bins.tiles1, (batch + kItemLanes - 1) / kItemLanes);
      spread_items_kernel<<<ig, 128, 0, st>>>(g, work, t, org, wts, gs, w_stride, bins, batch);
      done = true;
    }
  }
  if (!done) {
    dim3 sg(bins.tiles0 * bins.tiles1, (batch + kBatchBlock - 1) / kBatchBlock);
    spread_tile_kernel<R><<<sg, kCellsPerTile * kSpreadParts, 0, st>>>(g, work, u, wts, gs, w_stride, bins, batch);
  }
  nufft_fft2(g, work, batch, sign, st);
  dim3 eg((g.m_out0 * g.m_out1 + 255) / 256, batch);
  extract_kernel<R><<<eg, 256, 0, st>>>(g, work, modes, gs, mode_stride);
}

template void nufft_type2<float>(const NufftGridT<float>&, const float2*, int, size_t, const double*, int, float2*,
                                 size_t, float2*, int, const float*, cudaStream_t);
template void nufft_type2<double>(const NufftGridT<double>&, const double2*, int, size_t, const double*, int, double2*,
                                  size_t, double2*, int, const double*, cudaStream_t);
template void nufft_type1<float>(const NufftGridT<float>&, const double*, int, const NufftBins&, const float2*, int,
                                 size_t, float2*, size_t, float2*, int, cudaStream_t, void*);
template void nufft_type1<double>(const NufftGridT<double>&, const double*, int, const NufftBins&, const double2*, int,
                                  size_t, double2*, size_t, double2*, int, cudaStream_t, void*);

// The lists are made on the device, rows of tiles first and each row's tiles from its list (a pass of
// every tile over every point would grow with their product).  On the host, with a ring walk per point
// and axis, twice, they and the voxel and sample tables of the forward were 80 of 204 ms of a volume
// with 65,536 points.
NufftBins nufft_bins2(DevArena& A, DevArena& T, int nf0, int nf1, int w, const double* d_u, int npts,
                      cudaStream_t st) {
  NufftBins b;
  b.tiles0 = (nf0 + kSpreadTile - 1) / kSpreadTile;
  b.tiles1 = (nf1 + kSpreadTile - 1) / kSpreadTile;
  const int nt = b.tiles0 * b.tiles1, span = w + 2;
  // tiles that a span can meet on an axis (one more where the ring's last tile is cut)
  auto most = [&](int nf, int tiles) { return std::min(tiles, (span + 6) / kSpreadTile + (nf % kSpreadTile ? 2 : 1)); };
  const size_t m1 = most(nf1, b.tiles1), m0 = most(nf0, b.tiles0);
  int* lo = (int*)T.alloc((size_t)npts * 2 * 4);
  int* count = (int*)T.alloc((size_t)nt * 4);
  int* rstart = (int*)T.alloc((size_t)(b.tiles1 + 1) * 4);
  int* rpts = (int*)T.alloc(m1 * npts * 4);
  int* start = (int*)A.alloc((size_t)(nt + 1) * 4);
  int* pts = (int*)A.alloc(m0 * m1 * npts * 4);
  bins_origin_kernel<<<(npts + 255) / 256, 256, 0, st>>>(d_u, npts, nf0, nf1, w, lo);
  const int *lo0 = lo, *lo1 = lo + npts, *none = nullptr;
  bins_select_kernel<<<b.tiles1, kBinThreads, 0, st>>>(lo1, npts, none, none, b.tiles1, nf1, span, count, none, nullptr);
  bins_scan_kernel<<<1, 1024, 0, st>>>(count, b.tiles1, rstart);
  bins_select_kernel<<<b.tiles1, kBinThreads, 0, st>>>(lo1, npts, none, none, b.tiles1, nf1, span, nullptr, rstart, rpts);
  bins_select_kernel<<<nt, kBinThreads, 0, st>>>(lo0, npts, rstart, rpts, b.tiles0, nf0, span, count, none, nullptr);
  bins_scan_kernel<<<1, 1024, 0, st>>>(count, nt, start);
  bins_select_kernel<<<nt, kBinThreads, 0, st>>>(lo0, npts, rstart, rpts, b.tiles0, nf0, span, nullptr, start, pts);
  MRSIM_CUDA(cudaGetLastError());
  b.start = start;
  b.pts = pts;
  return b;
}

// From 16 items on a lane per item is the faster (half of a last chunk's lanes may be idle); a fine ring
// of fewer than 64 cells could meet a tile with both ends of a window, which the signed offset excludes.
size_t nufft_spread_taps(const NufftGridT<double>& g, int npts, int batch) {
  if (batch < 16 || npts <= 0 || g.nf0 < 64 || g.nf1 < 64) return 0;
  return (size_t)npts * (2 * kWMax * sizeof(double) + sizeof(int2));
}


void nufft1_run(const Nufft1Grid& g, const double* pos, int npos, const NufftBins& bins, const double2* wts, int nw,
                double2* out, double2* work, cudaStream_t st) {
  // every cell of every tile is written (zero where no source reaches it)
  spread1_tile_kernel<<<dim3(bins.tiles0, nw), kSpreadTile1, 0, st>>>(pos, wts, npos, g.nf, g.w, g.beta, work, bins);
  fft2<double2>(work, g.nf, 1, g.tw, g.tw, nw, 1, st);  // the inverse transform (e^{+i}) of each fine grid
  dim3 eg((g.n_out + 255) / 256, nw);
  extract1_kernel<<<eg, 256, 0, st>>>(work, g.nf, g.k_lo, g.n_out, g.corr, nw, out);
}

void spiral_exact(const SpiralExactArgs& a, cudaStream_t st) {
  spiral_exact_kernel<<<(a.npts + 255) / 256, 256, 0, st>>>(a);
}

void segment_images(const float2* x, const float2* rate, int nvox, const double* tau_l, int L, float2* out,
                    cudaStream_t st) {
  dim3 g((nvox + 255) / 256, L);
  segment_images_kernel<<<g, 256, 0, st>>>(x, rate, nvox, tau_l, L, out);
}

void spiral_stat(const double* k, int npts, int snx, int sny, int ox, int oy, float2* stat, cudaStream_t st) {
  spiral_stat_kernel<<<(npts + 255) / 256, 256, 0, st>>>(k, npts, snx, sny, (ox - 1.0) / 2.0, (oy - 1.0) / 2.0, stat);
}

void segment_combine(const float2* seg, int npts, int L, const int* tau_idx, const double* b, const float2* stat,
                     float2* out, bool by_point, cudaStream_t st) {
  segment_combine_kernel<<<(npts + 255) / 256, 256, 0, st>>>(seg, npts, L, tau_idx, b, stat, out, by_point ? 1 : 0);
}

}  // namespace mrsim
