// epi_device.h — what the EPI kernels share (epi_ystage.cu, epi_yadjoint.cu, epi_ythin.cu, epi_kernels.cu): packed
// arithmetic, the reduced phase, asynchronous copies, and the shapes of the staged kernels' tiles.
#pragma once

#include <cuda_runtime.h>

#include "mrsim_internal.h"
#include "row_fft.h"

// Template flags select whole code paths (packed or scalar, class or coil accumulators); the paths
// an instance does not take leave loops the front end reports as unreachable.
#pragma nv_diag_suppress 128

namespace mrsim {

namespace {

constexpr float kTwoPiF = 6.28318530717958647692f;

// The reduced phase s + f t in turns (s = static phase + k.r term, |s| <= 1 turn; f the voxel's
// off-resonance in Hz; t = t_hi + t_lo the line time in s, |f t| < 2^22) with one rounding to an
// integer: n = round(s + f t_hi) by adding and subtracting 1.5 * 2^23 (the FMA's rounded value
// serves only to choose n), r = f t_hi - n from one FMA of the exact product (|r| < 2: one rounding
// of at most ulp(1)/2), and
//   theta = (r + s) + f t_lo,   |theta| <= 1/2 + ulps,
// whose last two roundings are at most ulp(1/2)/2 each.
__device__ __forceinline__ float phase_turns(float s, float f, float t_hi, float t_lo) {
  const float nn = __fsub_rn(12582912.0f, __fadd_rn(fmaf(f, t_hi, s), 12582912.0f));  // -n
  return fmaf(f, t_lo, __fadd_rn(fmaf(f, t_hi, nn), s));
}

// Packed FP32 pairs (sm_100 add/sub/mul/fma.rn.f32x2): one instruction for two lanes, each lane
// rounding exactly like the scalar operation, so a packed computation is bitwise the scalar one.
__device__ __forceinline__ unsigned long long pk2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 upk2(unsigned long long r) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
  return d;
}
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pk2(a)), "l"(pk2(b)), "l"(pk2(c)));
  return upk2(d);
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(d);
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(d);
}
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(d);
}
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// The reduced phase s + f t (s = static phase + k.r term, |s| <= 1 turn, t = t_hi + t_lo) on a pair
// of lanes with one rounding to an integer: n = round(s + f t_hi) (the FMA's rounded value serves
// only to choose n), r = f t_hi - n from one FMA of the exact product (|r| < 2: one rounding of
// at most ulp(1)/2), and
//   theta = (r + s) + f t_lo,   |theta| <= 1/2 + ulps,
// whose last two roundings are at most ulp(1/2)/2 each: six packed operations.
__device__ __forceinline__ float2 phase_turns2(float2 s, float2 f, float2 t_hi, float2 t_lo) {
  const float2 M = dup2(12582912.0f);
  const float2 nn = fsub2(M, fadd2(ffma2(f, t_hi, s), M));  // -n
  const float2 r = ffma2(f, t_hi, nn);
  return ffma2(f, t_lo, fadd2(r, s));
}

// The kernels of a step are launched so that one may start while the one before it still runs
// (programmatic dependent launch): its blocks take their place as the last blocks of the one before
// drain, read the tables that no kernel writes, and wait here before they touch anything else.  Every
// kernel of the chain waits, so what a kernel sees after it is what in-order launches give; copies and
// kernels that do not call grid_begin are waited for before a launch starts, as always.  A step of
// one slice is five launches of 3 to 8 us; the overlap takes the launch gaps and table setups out of
// its chain (39.9 -> 21.0 us).  Chained are the y-stages and x-stages of at most kChainTiles tiles and
// the statics of at most 148 units.  Above that the y-stages run instances without the wait (with it a
// 1200-unit step took 1.5 % longer and gained nothing), and the x-stages and statics, whose wait then
// returns at once, plain launches.
// A chained kernel may be resident while an earlier one of its chain still writes (the y-adjoint while
// the statics kernel forms the phase, every link having triggered at its start), so what a kernel of
// the chain writes is not read-only for its lifetime: it is read by plain loads or asynchronous copies,
// never through __ldg, which is for the tables and planes that copies alone write.
constexpr int kChainTiles = 4 * 296;
__device__ __forceinline__ void grid_begin() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void grid_wait() { cudaGridDependencySynchronize(); }

// The k.r phase (K Y mod m2) / m2 in turns of line K (ky - ys) and row Y (2(y - sys) - (oy - 1)),
// m2 = 2 sny: an exact integer index, in 32 bits wherever the product fits.
__device__ __forceinline__ double kr_turns(int K, int Y, int m2) {
  const int r = m2 <= 65536 ? (K * Y) % m2 : (int)(((long long)K * Y) % m2);
  return (double)r / (double)m2;
}

// cp.async helpers (16-byte copies zero-fill the bytes past src_bytes)
__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gmem_src, int src_bytes = 8) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(gmem_src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;\n" ::); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait_n() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(gmem_src), "r"(src_bytes));
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem_src), "r"(src_bytes));
}

constexpr int kT = 4;   // lines per tile of ystage_kernel

// On basis rows every coil's sample is mostly the constant row's sum, so that sum's rounding is nearly
// the same in every coil and does not average out over the coils in the adjoint, as the coils' own sums'
// did.  It is therefore added up in blocks of 16 rows, and those in blocks of 64.  What the adjoint makes
// of the forward's rounding (32 coils, 64 x 64 on 128 x 128, in FP32 on the CPU): one chain of rows 1.4e-7,
// blocks of 32 7.4e-8, of 16 6.3e-8, exact sums 2.8e-8, per-coil sums 1.9e-8, beside 1.8e-7 from the sines in
// all of them; the adjoint's own blocks (adj_blocked) give more back.  The pair against 64 bits, 128 x 128 on
// 256 x 256, 32 coils, k-space and compartment gradients: per-coil sums 2.55e-7 and 4.00e-7, basis rows in
// one chain 2.57e-7 and 4.26e-7, now 2.19e-7 and 3.57e-7.
constexpr int kConstBlock = 16, kConstBlocks = 64;
constexpr int kTY = 4;  // rows per tile of yadjoint_kernel

// ystage_q_kernel: ring stages, and input planes and rows per stage
constexpr int kFwdStages = 3;
__host__ __device__ __forceinline__ constexpr int fwdq_planes(int nc, bool maps) { return maps ? 3 + 3 * nc : 2 + nc; }
__host__ __device__ __forceinline__ constexpr int fwdq_rows(int nc, bool maps) {
  return fwdq_planes(nc, maps) <= 5 ? 8 : fwdq_planes(nc, maps) <= 12 ? 4 : 2;
}

// Lines per h chunk of yadjoint_kernel for `ncoils` coils (16 coil-lines per chunk, at least one line).
__host__ __device__ __forceinline__ int adjoint_chunk_lines(int ncoils) { return ncoils >= 16 ? 1 : 16 / ncoils; }

// yadjoint_q_kernel: ring stages, lines per chunk, floats of a line record
constexpr int kAdjStages = 3;
__host__ __device__ __forceinline__ constexpr int adjq_chunk_lines(int nq) { return nq >= 16 ? 1 : 16 / nq; }
__host__ __device__ __forceinline__ constexpr int adjq_line_floats(int nc, bool maps) {
  return ((maps ? 5 : 4 + 3 * nc) + 3) / 4 * 4;
}
// rows per thread: 4 with class decay and up to 3 compartments, else 2 (registers)
__host__ __device__ __forceinline__ constexpr int adjq_rows(int nc, bool maps) { return !maps && nc <= 3 ? 4 : 2; }
// ... the same with coil-class rows (two rows per thread in 80 registers and three CTAs per SM
// measured 30 % slower than four rows: the per-line loads then serve half the rows)
__host__ __device__ __forceinline__ constexpr int adjq_rows_v(int nc, bool maps, bool virt) {
  return adjq_rows(nc, maps);
}

// Dynamic shared memory of the staged kernels, which hold a table of every row (forward) or line
// (adjoint) of a tile beside their ring, and the most that a block can have beside their static tables
// (4 KB of piece offsets at the most).  A plan whose rows or lines do not fit takes the per-thread-load
// forward and the general adjoint, whose tables are smaller: with three compartments 1,900 lines fit
// (15 echoes of 128 lines) and the general kernel holds 3,100 to 4,200.
constexpr size_t kStagedSmem = 227 * 1024 - 4608;
inline size_t ystage_q_smem(int nc, bool maps, int qg, int max_sny, bool basis) {
  return sizeof(float) * ((size_t)kFwdStages * fwdq_planes(nc, maps) * fwdq_rows(nc, maps) * 128 +
                          (size_t)max_sny * (8 + (qg + 3) / 4 * 4) + (basis ? 2 * 8 * 256 : 0));
}
inline size_t yadjoint_q_smem(int nq, int ty, int nc, bool maps, int max_lines) {
  return sizeof(float2) * (size_t)kAdjStages * adjq_chunk_lines(nq) * nq * 128 +
         sizeof(float) * (size_t)(max_lines + adjq_chunk_lines(nq)) * (2 * ty + adjq_line_floats(nc, maps));
}
// On basis rows the adjoint adds its lines in blocks of 16 too, whose whole sums are in shared memory,
// where they leave two blocks an SM (about 170 lines with gradients of three compartments, 430 without):
// what the forward's rounding costs the pair more than per-coil sums, this one gives back.  The rule is
// a unit's own lines and the built-in rows per thread, so every form and grouping takes the same one.
constexpr int kLineBlock = 32;
constexpr size_t kBlockedSmem = 108 * 1024;
__host__ __device__ __forceinline__ constexpr size_t adj_sum_bytes(int ty, int nc, bool grads) {
  return (size_t)1024 * ty * nc * (grads ? 4 : 2);
}
__host__ __device__ __forceinline__ constexpr bool adj_blocked(int nq, int nc, bool maps, bool grads, int lines) {
  return (size_t)8 * kAdjStages * adjq_chunk_lines(nq) * nq * 128 +
             (size_t)4 * (lines + adjq_chunk_lines(nq)) * (2 * adjq_rows(nc, maps) + adjq_line_floats(nc, maps)) +
             adj_sum_bytes(adjq_rows(nc, maps), nc, grads) <=
         kBlockedSmem;
}

// The thin y kernels (ystage_thin_kernel, yadjoint_thin_kernel), for plans of few tiles: blocks of 32
// columns x 4 G lines (forward) or rows (adjoint), whose 8 warps form the terms of different rows or
// lines side by side and then add them in the same order as the full kernels, operation for operation:
// a slab computed alone has the bits that it has in its series, whichever form each plan takes.
constexpr int kThinCols = 32;
__host__ __device__ __forceinline__ constexpr int thin_rows(int g) { return 32 / g; }  // rows of a forward chunk
constexpr int kThinLines = 16;  // lines of an adjoint chunk
__host__ __device__ __forceinline__ constexpr int thin_stages(int nq) { return nq <= 4 ? 3 : 2; }
inline size_t ystage_thin_smem(int g, int nc, int qg, int max_sny) {
  return sizeof(float) * ((size_t)kFwdStages * fwdq_planes(nc, false) * thin_rows(g) * kThinCols +
                          2 * (size_t)thin_rows(g) * 4 * g * kThinCols + (size_t)max_sny * (4 * g + (qg + 3) / 4 * 4));
}
inline size_t yadjoint_thin_smem(int g, int nq, int nc, int max_lines) {
  return sizeof(float2) * ((size_t)thin_stages(nq) * kThinLines * nq * kThinCols +
                           (size_t)kThinLines * 4 * g * kThinCols) +
         sizeof(float) * (size_t)(max_lines + kThinLines) * (4 * g + adjq_line_floats(nc, false));
}
//
// thin_groups: G for a plan of `tiles` full tiles of `outs` lines or rows by 128 columns, 0 for the full
// kernels.  G = 1 makes eight blocks of a full tile, G = 2 four that read less.  Forward and adjoint of n
// slices of 64 x 64 on 128 x 128 (8 n and 16 n tiles), 8 coils, 3 compartments, in us, G = 1 / 2 / full:
// n = 1: 17 / 20 / 35 and 14 / 18 / 27; 3: 18 / 17 / 40 and 23 / 18 / 41; 6: 28 / 26 / 38 and 37 / 28 / 42;
// 12: 50 / 40 / 59 and 66 / 51 / 47; 24: 85 / 68 / 64 and 120 / 87 / 71; one coil: 14 / 15 / 22 and
// 7 / 8 / 12, n = 8: 23 / 25 / 50 and 17 / 16 / 26, n = 16: 34 / 32 / 52 and 30 / 25 / 28.  So: two blocks
// an SM of G = 1, then a full tile an SM.
inline int thin_groups(long long tiles, int outs) {
  const long long t = tiles * outs / 8;
  return t <= 37 ? 1 : t <= 148 ? 2 : 0;
}

// A launch of 256-thread blocks that may start while the kernel before it still runs (`overlap`); the
// kernel calls grid_begin and grid_wait.
template <class K, class... A>
void launch_chained(K kernel, dim3 blocks, size_t smem, cudaStream_t st, bool overlap, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = blocks;
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  MRSIM_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
}

template <class K>
void set_smem(K kernel, size_t bytes) {
  // past 48 KB of static + dynamic shared memory the launch needs the dynamic opt-in
  // (the whole limit, so that threads launching one kernel with different sizes never lower it
  // between another's opt-in and launch)
  if (bytes <= 40 * 1024) return;  // no kernel here has 8 KB of static shared memory beside dynamic
  cudaFuncAttributes fa;
  MRSIM_CUDA(cudaFuncGetAttributes(&fa, kernel));
  if (bytes + fa.sharedSizeBytes > 48 * 1024)
    MRSIM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    227 * 1024 - (int)fa.sharedSizeBytes));
}

}  // namespace

// The thin kernels' launches of a pass: n tiles (epi_ythin.cu).
void launch_ystage_thin(const EpiPlan* p, int pass, const int4* tiles, int n, cudaStream_t st);
void launch_yadjoint_thin(const EpiPlan* p, int pass, const int4* tiles, int n, cudaStream_t st);

namespace {
// The tiles of units [u0, u1) in a list with per-unit starts `start` (empty: the whole list).
struct TileRange {
  int t0, n;
};
TileRange tile_range(const std::vector<int>& start, int n_tiles, int u0, int u1) {
  if (start.empty() || (u0 == 0 && (u1 < 0 || u1 == (int)start.size() - 1))) return {0, n_tiles};
  if (u1 < 0) u1 = (int)start.size() - 1;
  if (u0 < 0 || u0 > u1 || u1 >= (int)start.size()) fail("unit range outside the plan");
  return {start[u0], start[u1] - start[u0]};
}

}  // namespace

}  // namespace mrsim
