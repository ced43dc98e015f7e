// nufft_tiled.cu — the type-2 transform of the spiral forwards for a batch of mode grids at one set of
// points (nufft.rs:259-292 with the forwards' width w = 13), FP32.
//
// The general kernels (nufft_kernels.cu) pass every fine grid through memory six times (clear, place,
// two FFT axes) and interpolate with a thread per point, whose 169 taps are scattered loads of one
// batch item each: 0.80 + 0.24 ms per slice of 8 coils x 16 segments at 65,536 points.  Here
//   rows      a warp reads a mode row, deapodizes it and transforms it zero-padded to the fine length;
//             only the mode rows exist between the two passes
//   columns   16 columns at a time through shared memory; the zero rows are never read
//   points    a block holds the fine cells around a tile of window origins for 16 batch items, and each
//             half-warp serves four points of one origin at once with the items on its lanes, so a
//             cell is read once from shared memory for the four and the grid from L2 once per tile.
//             The points are ordered by window origin and their taps formed once per trajectory.
// The taps and each point's sum are the general kernel's, operation for operation.  No pipe is full: at 16
// items FMA 27 % and shared-memory loads 30 % of the elapsed time, at 128 items FMA about 43 % (a fifth of it
// for the empty places of a group); a tile's loads and its sums alternate, at two blocks of 108 registers an
// SM.  Results come out [point][item]: the combination that follows reads an item range of a point in one
// run.  That slice takes 0.24 + 0.06 ms (16 segments of one coil: 134 + 49 us, here 51 + 17 + 22 for the
// order and the taps).
#include <cuda_runtime.h>

#include <algorithm>

#include "driver.h"
#include "es_taps.cuh"
#include "mrsim_internal.h"
#include "nufft.h"
#include "row_fft.h"

namespace mrsim {
namespace {

constexpr int kW = 13;                            // taps per axis
// Window origins of a tile, and the groups of points a block takes at a time.  The wide tile reads each
// grid cell 4.4 times instead of 10 and leaves fewer half-warps without a group; the small one gives a
// batch of one chunk enough blocks.
struct Small {
  static constexpr int kTX = 8, kTY = 4, kGroups = 32;
};
struct Wide {
  static constexpr int kTX = 16, kTY = 8, kGroups = 64;
};
constexpr int kGroup = 4;                         // points of one origin a warp serves together
constexpr int kItems = 16;                        // batch items of a block
constexpr int kTapStride = 28;                    // floats a point: its taps of each axis, two unused

__device__ __forceinline__ int wrap_cell(int m, int n) { return m < 0 ? m + n : (m >= n ? m - n : m); }

// key[j] = tile * kCells + cell of the point's origin; rank[j] its place among the points of that
// origin; taps[j] its taps.
template <class T>
__global__ void points_key_kernel(const double* __restrict__ u, int npts, int nf0, int nf1, float beta, int tiles0,
                                  int* __restrict__ count, int* __restrict__ key, int* __restrict__ rank,
                                  float* __restrict__ taps) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npts) return;
  float k0[kWMax], k1[kWMax];
  const int a0 = wrap_cell(es_taps<float>(u[2 * j], nf0, kW, beta, k0), nf0);
  const int a1 = wrap_cell(es_taps<float>(u[2 * j + 1], nf1, kW, beta, k1), nf1);
  const int k = ((a1 / T::kTY) * tiles0 + a0 / T::kTX) * (T::kTX * T::kTY) + (a1 % T::kTY) * T::kTX + a0 % T::kTX;
  key[j] = k;
  rank[j] = atomicAdd(&count[k], 1);  // (which point gets which place changes no result)
  float* t = taps + (size_t)j * kTapStride;
#pragma unroll
  for (int i = 0; i < kW; ++i) {
    t[i] = k0[i];
    t[kW + i] = k1[i];
  }
}

// One warp per tile: each origin's first group within the tile (ceil(count / kGroup) groups each) and
// the tile's groups.  The scan over the tiles then has only their number to walk: one block over every
// origin took 120 us at 65,536 of them.
template <class T>
__global__ void __launch_bounds__(256) points_tile_kernel(const int* __restrict__ count, int tiles,
                                                          int* __restrict__ local, int* __restrict__ groups) {
  constexpr int kCells = T::kTX * T::kTY;
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= tiles) return;
  int base = 0;
#pragma unroll
  for (int c = lane; c < kCells; c += 32) {
    const int v = (count[t * kCells + c] + kGroup - 1) / kGroup;
    int x = v;
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, x, h);
      if (lane >= h) x += o;
    }
    local[t * kCells + c] = base + x - v;
    base += __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) groups[t] = base;
}

// One block: first group of each tile, and the work items (tile, first group, groups) of up to
// T::kGroups groups.
template <class T>
__global__ void __launch_bounds__(1024) points_scan_kernel(const int* __restrict__ groups, int tiles,
                                                           int* __restrict__ first, int4* __restrict__ items,
                                                           int* __restrict__ n_items) {
  constexpr int kItemGroups = T::kGroups;
  __shared__ int part[2][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, per = (tiles + 1023) / 1024;
  int v[2] = {0, 0};  // groups and items of this thread's tiles
  for (int t = tid * per; t < min(tiles, (tid + 1) * per); ++t) {
    v[0] += groups[t];
    v[1] += (groups[t] + kItemGroups - 1) / kItemGroups;
  }
  int x[2] = {v[0], v[1]};
  for (int q = 0; q < 2; ++q) {
    for (int h = 1; h < 32; h <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, x[q], h);
      if (lane >= h) x[q] += o;
    }
    if (lane == 31) part[q][warp] = x[q];
  }
  __syncthreads();
  for (int q = 0; q < 2; ++q) {
    x[q] -= v[q];
    for (int w = 0; w < warp; ++w) x[q] += part[q][w];
  }
  if (tid == 1023) *n_items = x[1] + v[1];
  for (int t = tid * per; t < min(tiles, (tid + 1) * per); ++t) {
    first[t] = x[0];
    for (int g = 0; g < groups[t]; g += kItemGroups)
      items[x[1]++] = make_int4(t, x[0] + g, min(kItemGroups, groups[t] - g), 0);
    x[0] += groups[t];
  }
}

template <class T>
__global__ void points_place_kernel(const int* __restrict__ key, const int* __restrict__ rank, int npts,
                                    const int* __restrict__ first, const int* __restrict__ local,
                                    int* __restrict__ pts) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npts) return;
  constexpr int kCells = T::kTX * T::kTY;
  const int k = key[j];
  pts[(first[k / kCells] + local[k] + rank[j] / kGroup) * kGroup + rank[j] % kGroup] = j;
}

// One warp per mode row: tmp[b][j1][c0], the zero-padded row transforms (sigma = +1).
template <int E>
__global__ void __launch_bounds__(256) mode_rows_kernel(const NufftGrid g, const float2* __restrict__ modes, int rows,
                                                        float2* __restrict__ tmp) {
  constexpr int N = 32 * E, LE = log2_c(E), NP = N + N / 32;
  constexpr bool P2 = (E & (E - 1)) == 0;
  __shared__ __align__(16) float2 tw[N];
  __shared__ float corr[N];
  __shared__ __align__(16) float2 rb[8][NP];
  for (int i = threadIdx.x; i < N; i += 256) {
    tw[i] = g.tw0[i];
    const int j0 = i - g.m_lo0 < N ? i - g.m_lo0 : i - g.m_lo0 - N;  // mode of fine cell i, if any
    corr[i] = j0 >= 0 && j0 < g.m_out0 ? g.corr0[j0] : 0.f;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* row = rb[warp];
  for (int r = blockIdx.x * 8 + warp; r < rows; r += gridDim.x * 8) {
    const float s1 = g.corr1[r % g.m_out1];
    const float2* m = modes + (size_t)r * g.m_out0;
    float2 b[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int c = lane + 32 * k;
      const int j0 = c - g.m_lo0 < N ? c - g.m_lo0 : c - g.m_lo0 - N;
      float2 v = make_float2(0.f, 0.f);
      if (j0 >= 0 && j0 < g.m_out0) {
        v = m[j0];
        const float s = corr[c] * s1;
        v = make_float2(v.x * s, v.y * s);
      }
      b[P2 ? bitrev_c(k, LE) : k] = v;
    }
    warp_row_fft<E, false>(b, tw, lane);
    const int k2 = (int)(__brev(lane) >> 27);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) {
      const int k = k1 + E * k2;
      row[k + (k >> 5)] = b[k1];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int c = lane + 32 * k;
      tmp[(size_t)r * N + c] = row[c + (c >> 5)];
    }
    __syncwarp();
  }
}

// 16 columns of one item: grid[b][c1][c0] from the mode rows of tmp.
constexpr int kCols = 16;
template <int E>
__global__ void __launch_bounds__(256) mode_cols_kernel(const NufftGrid g, const float2* __restrict__ tmp,
                                                        float2* __restrict__ grid) {
  constexpr int N = 32 * E, LE = log2_c(E), LD = kCols + 1;
  constexpr bool P2 = (E & (E - 1)) == 0;
  extern __shared__ __align__(16) float2 csm[];
  float2* tw = csm;      // [N]
  float2* s = tw + N;    // [N][LD]: the columns' inputs by fine cell, then their transforms
  const int c0 = blockIdx.x * kCols, nf0 = g.nf0, m1 = g.m_out1;
  const float2* src = tmp + (size_t)blockIdx.y * m1 * nf0 + c0;
  for (int i = threadIdx.x; i < N; i += 256) tw[i] = g.tw1[i];
  for (int i = threadIdx.x; i < N * kCols; i += 256) {
    const int c = i / kCols, x = i % kCols;
    const int j1 = c - g.m_lo1 < N ? c - g.m_lo1 : c - g.m_lo1 - N;
    s[c * LD + x] = j1 >= 0 && j1 < m1 ? src[(size_t)j1 * nf0 + x] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k2 = (int)(__brev(lane) >> 27);
  for (int x = warp; x < kCols; x += 8) {
    float2 b[E];
#pragma unroll
    for (int k = 0; k < E; ++k) b[P2 ? bitrev_c(k, LE) : k] = s[(lane + 32 * k) * LD + x];
    warp_row_fft<E, false>(b, tw, lane);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) s[(k1 + E * k2) * LD + x] = b[k1];
  }
  __syncthreads();
  float2* dst = grid + (size_t)blockIdx.y * N * nf0 + c0;
  for (int i = threadIdx.x; i < N * kCols; i += 256) dst[(size_t)(i / kCols) * nf0 + i % kCols] = s[(i / kCols) * LD + i % kCols];
}

template <class T>
constexpr size_t points_smem() {
  return sizeof(float2) * (size_t)(T::kTX + kW - 1) * (T::kTY + kW - 1) * (kItems + 1) +
         sizeof(float4) * 2 * T::kGroups * kW + sizeof(int) * (T::kGroups * (kGroup + 1));
}

// kItems batch items on the lanes of each half-warp.
template <class T>
__global__ void __launch_bounds__(256, 2) points_kernel(const NufftGrid g, const float2* __restrict__ grid,
                                                        const float* __restrict__ taps, const int* __restrict__ key,
                                                        const int4* __restrict__ items, const int* __restrict__ n_items,
                                                        const int* __restrict__ pts, int tiles0, int batch,
                                                        float2* __restrict__ out) {
  constexpr int BI = kItems, LD = BI + 1, LANES = 32 / BI, kItemGroups = T::kGroups;
  constexpr int kRX = T::kTX + kW - 1, kRY = T::kTY + kW - 1;  // fine cells that the tile's windows reach
  extern __shared__ __align__(16) unsigned char psm[];
  float4* k0s = reinterpret_cast<float4*>(psm);        // [group][tap] of the group's four points
  float4* k1s = k0s + kItemGroups * kW;
  float2* cells = reinterpret_cast<float2*>(k1s + kItemGroups * kW);  // [cell][item]
  int* pj = reinterpret_cast<int*>(cells + kRX * kRY * LD);           // [group][point]
  int* at = pj + kItemGroups * kGroup;                                // [group]: its origin's cell
  const int b0 = blockIdx.y * BI, nb = min(BI, batch - b0), tid = threadIdx.x;
  const int nf0 = g.nf0, nf1 = g.nf1;
  const size_t gs = (size_t)nf0 * nf1;
  const int lane = tid & 31, sub = lane / BI, bi = lane % BI;
  const int n = *n_items;
  for (int it = blockIdx.x; it < n; it += gridDim.x) {
    const int4 item = items[it];
    const int ng = item.z, x0 = (item.x % tiles0) * T::kTX, y0 = (item.x / tiles0) * T::kTY;
    __syncthreads();  // every thread is done with the item before
    for (int i = tid; i < kRX * kRY * BI; i += 256) {  // neighbouring threads take neighbouring cells
      const int c = i % (kRX * kRY), b = i / (kRX * kRY);
      const int c0 = wrap_cell(x0 + c % kRX, nf0), c1 = wrap_cell(y0 + c / kRX, nf1);
      cells[c * LD + b] = b < nb ? __ldg(grid + (b0 + b) * gs + (size_t)c1 * nf0 + c0) : make_float2(0.f, 0.f);
    }
    for (int t = tid; t < ng * kGroup; t += 256) {
      const int j = pts[item.y * kGroup + t];
      pj[t] = j;
      if (t % kGroup == 0) {  // a group's first place is never empty
        const int c = key[j] % (T::kTX * T::kTY);
        at[t / kGroup] = (c / T::kTX) * kRX + c % T::kTX;
      }
      float k[kTapStride];
      const float4* src = reinterpret_cast<const float4*>(taps + (size_t)max(j, 0) * kTapStride);
#pragma unroll
      for (int i = 0; i < kTapStride / 4; ++i) {
        const float4 v = j >= 0 ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        k[4 * i] = v.x, k[4 * i + 1] = v.y, k[4 * i + 2] = v.z, k[4 * i + 3] = v.w;
      }
      float* f0 = reinterpret_cast<float*>(k0s + (t / kGroup) * kW) + t % kGroup;
      float* f1 = reinterpret_cast<float*>(k1s + (t / kGroup) * kW) + t % kGroup;
#pragma unroll
      for (int i = 0; i < kW; ++i) {
        f0[kGroup * i] = k[i];
        f1[kGroup * i] = k[kW + i];
      }
    }
    __syncthreads();
    for (int q = (tid >> 5) * LANES + sub; q < ng; q += 8 * LANES) {
      float4 k0[kW];
#pragma unroll
      for (int i = 0; i < kW; ++i) k0[i] = k0s[q * kW + i];
      float re[kGroup], im[kGroup];
#pragma unroll
      for (int p = 0; p < kGroup; ++p) re[p] = im[p] = 0.f;
      const float2* base = cells + at[q] * LD + bi;
#pragma unroll 1
      for (int i1 = 0; i1 < kW; ++i1) {
        float rr[kGroup], ri[kGroup];
#pragma unroll
        for (int p = 0; p < kGroup; ++p) rr[p] = ri[p] = 0.f;
#pragma unroll
        for (int i0 = 0; i0 < kW; ++i0) {
          const float2 v = base[(i1 * kRX + i0) * LD];
          const float k[kGroup] = {k0[i0].x, k0[i0].y, k0[i0].z, k0[i0].w};
#pragma unroll
          for (int p = 0; p < kGroup; ++p) {
            rr[p] = fmaf(v.x, k[p], rr[p]);
            ri[p] = fmaf(v.y, k[p], ri[p]);
          }
        }
        const float4 kk = k1s[q * kW + i1];
        const float k[kGroup] = {kk.x, kk.y, kk.z, kk.w};
#pragma unroll
        for (int p = 0; p < kGroup; ++p) {
          re[p] = fmaf(rr[p], k[p], re[p]);
          im[p] = fmaf(ri[p], k[p], im[p]);
        }
      }
#pragma unroll
      for (int p = 0; p < kGroup; ++p) {
        const int j = pj[q * kGroup + p];
        if (j >= 0 && bi < nb) out[(size_t)j * batch + b0 + bi] = make_float2(re[p], im[p]);
      }
    }
  }
}

template <int E0>
void launch_rows(const NufftGrid& g, const float2* modes, int batch, float2* tmp, cudaStream_t st) {
  const int rows = batch * g.m_out1;
  mode_rows_kernel<E0><<<std::min((rows + 7) / 8, 148 * 8), 256, 0, st>>>(g, modes, rows, tmp);
}
template <int E1>
void launch_cols(const NufftGrid& g, const float2* tmp, int batch, float2* grid, cudaStream_t st) {
  const size_t smem = sizeof(float2) * (size_t)(32 * E1) * (kCols + 2);
  mode_cols_kernel<E1><<<dim3(g.nf0 / kCols, batch), 256, smem, st>>>(g, tmp, grid);
}

}  // namespace

// The forwards' width, and fine lengths that a warp's row transform takes in whole (32 E, E even: E = 6 has
// an instance too); longer or ragged lines keep the general kernels, whose block per line holds any length.
bool nufft_tiled_fits(const NufftGrid& g) {
  return g.w == kW && g.nf0 % 64 == 0 && g.nf1 % 64 == 0 && g.nf0 <= 256 && g.nf1 <= 256;
}

namespace {
template <class T>
NufftPoints make_points(DevArena& A, const NufftGrid& g, const double* d_u, int npts, cudaStream_t st) {
  constexpr int kCells = T::kTX * T::kTY;
  NufftPoints P;
  P.tiles0 = (g.nf0 + T::kTX - 1) / T::kTX;
  const int tiles = P.tiles0 * ((g.nf1 + T::kTY - 1) / T::kTY), nkeys = tiles * kCells;
  // every group holds at least one point; an item is a whole T::kGroups groups or a tile's last
  const size_t max_items = (size_t)tiles + npts / T::kGroups + 1;
  int* count = (int*)A.alloc((size_t)nkeys * 4);
  int* key = (int*)A.alloc((size_t)npts * 4);
  int* rank = (int*)A.alloc((size_t)npts * 4);
  int* local = (int*)A.alloc((size_t)nkeys * 4);
  int* groups = (int*)A.alloc((size_t)tiles * 4);
  int* first = (int*)A.alloc((size_t)tiles * 4);
  int* pts = (int*)A.alloc((size_t)npts * kGroup * 4);
  float* taps = (float*)A.alloc((size_t)npts * kTapStride * 4);
  P.items = (int4*)A.alloc(max_items * sizeof(int4));
  P.n_items = (int*)A.alloc(4);
  P.pts = pts;
  P.key = key;
  P.taps = taps;
  P.max_items = (int)max_items;
  MRSIM_CUDA(cudaMemsetAsync(count, 0, (size_t)nkeys * 4, st));
  MRSIM_CUDA(cudaMemsetAsync(pts, 0xff, (size_t)npts * kGroup * 4, st));
  points_key_kernel<T><<<(npts + 255) / 256, 256, 0, st>>>(d_u, npts, g.nf0, g.nf1, g.beta, P.tiles0, count, key, rank,
                                                           taps);
  points_tile_kernel<T><<<(tiles + 7) / 8, 256, 0, st>>>(count, tiles, local, groups);
  points_scan_kernel<T><<<1, 1024, 0, st>>>(groups, tiles, first, P.items, P.n_items);
  points_place_kernel<T><<<(npts + 255) / 256, 256, 0, st>>>(key, rank, npts, first, local, pts);
  MRSIM_CUDA(cudaGetLastError());
  return P;
}

template <class T>
void launch_points(const NufftGrid& g, const float2* grid, const NufftPoints& P, int batch, float2* out,
                   cudaStream_t st) {
  constexpr size_t smem = points_smem<T>();
  MRSIM_CUDA(cudaFuncSetAttribute(points_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int chunks = (batch + kItems - 1) / kItems;
  const int blocks = std::max(1, std::min(P.max_items, (2 * 148 * 4 + chunks - 1) / chunks));
  points_kernel<T><<<dim3(blocks, chunks), 256, smem, st>>>(g, grid, P.taps, P.key, P.items, P.n_items, P.pts, P.tiles0,
                                                            batch, out);
}
}  // namespace

NufftPoints nufft_points(DevArena& A, const NufftGrid& g, const double* d_u, int npts, int batch, cudaStream_t st) {
  // 65,536 points on a 256 x 256 fine grid: 16 items 51 us with small tiles and 55 with wide ones, 128 items
  // 276 and 244.  The line between is set, not measured: three chunks give the wide tiles' blocks five items each to even
  // out.
  const bool wide = batch > 2 * kItems;
  NufftPoints P = wide ? make_points<Wide>(A, g, d_u, npts, st) : make_points<Small>(A, g, d_u, npts, st);
  P.wide = wide;
  return P;
}

void nufft_type2_tiled(const NufftGrid& g, const float2* modes, int batch, const NufftPoints& P, float2* out,
                       float2* grid, float2* tmp, cudaStream_t st) {
#define MRSIM_NT(F, E, ...)              \
  switch (E) {                           \
    case 2: F<2>(__VA_ARGS__); break;    \
    case 4: F<4>(__VA_ARGS__); break;    \
    case 6: F<6>(__VA_ARGS__); break;    \
    default: F<8>(__VA_ARGS__); break;   \
  }
  MRSIM_NT(launch_rows, g.nf0 / 32, g, modes, batch, tmp, st)
  MRSIM_NT(launch_cols, g.nf1 / 32, g, tmp, batch, grid, st)
#undef MRSIM_NT
  if (P.wide)
    launch_points<Wide>(g, grid, P, batch, out, st);
  else
    launch_points<Small>(g, grid, P, batch, out, st);
  MRSIM_CUDA(cudaGetLastError());
}

}  // namespace mrsim
