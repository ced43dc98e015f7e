// recon_kernels.cu — the reconstruction of one slice's coils on the device (reference
// `reconstruct_coils_full`, kspace.rs:1301-1378): GRAPPA calibration (FP64 normal equations and
// pivoted Gaussian elimination, `GrappaKernel::fit` kspace.rs:1547-1599 + `solve_hermitian`
// :1457-1491), GRAPPA apply (kspace.rs:1605-1632), the radial window (kspace.rs:1327-1342), the
// centred inverse 2D DFT (`inverse_2d`, kspace.rs:1428-1453) and the Roemer combine
// (kspace.rs:1343-1373).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "hermitian_solve.cuh"
#include "mrsim_internal.h"
#include "recon_kernels.h"
#include "row_fft.h"

namespace mrsim {

namespace {

// The source feature i of GRAPPA at readout kx: lines s0/s1, readout offsets -1/0/+1 (wrapped),
// every coil; layout (line*3 + point)*nc + coil (`grappa_feature`, kspace.rs:1526-1538).
__device__ __forceinline__ float2 feature(const float2* __restrict__ k, int nx, int ny, int nc, int s0, int s1,
                                          int kx, int i) {
  int ci = i % nc;
  int p = i / nc;
  int li = p / 3, ki = p % 3;
  int kxs = kx + ki - 1;
  kxs = kxs < 0 ? kxs + nx : (kxs >= nx ? kxs - nx : kxs);
  int sl = li == 0 ? s0 : s1;
  return k[(size_t)ci * nx * ny + (size_t)sl * nx + kxs];
}

// The normal equations [A^H A | A^H b], FP64 sums over the reference band in the reference's order (band
// line, then readout point): a block of 16 x 16 entries of one system, one thread each.  A chunk of
// readout points' features (16 of the rows, 16 of the columns) is gathered and widened to FP64 once in
// shared memory for all 256 entries; bound by that memory (two 16-byte reads per four FMAs).  30
// systems of 8 coils, 23 band lines x 64 points: 219 us, 614 with a gather per entry and term.
constexpr int kNormTile = 16, kNormChunk = 32;
__global__ void __launch_bounds__(256) grappa_normal_kernel(const GrappaSystem* __restrict__ sys) {
  __shared__ double2 fi_s[kNormChunk][kNormTile], fj_s[kNormChunk][kNormTile];
  const GrappaSystem& S = sys[blockIdx.z];
  const int nf = 6 * S.nc, nc = S.nc, nx = S.nx, ny = S.ny;
  const int cols = nf + nc;
  const int i0 = blockIdx.y * kNormTile, j0 = blockIdx.x * kNormTile;
  if (i0 >= nf || j0 >= cols) return;
  const int ti = threadIdx.x / kNormTile, tj = threadIdx.x % kNormTile;
  double ar = 0.0, ai = 0.0;
  for (int b = S.acs_lo; b < S.acs_hi; ++b) {
    const int s0 = b, s1 = b + S.accel, tgt = b + S.d;
    if (s1 > S.acs_hi || tgt > S.acs_hi || !(S.lines[s0] && S.lines[s1] && S.lines[tgt])) continue;
    for (int k0 = 0; k0 < nx; k0 += kNormChunk) {
      const int nk = min(kNormChunk, nx - k0);
      for (int e = threadIdx.x; e < 2 * kNormTile * kNormChunk; e += 256) {
        // neighbouring threads take neighbouring readout points of one feature
        const int kk = e % kNormChunk, f = e / kNormChunk, side = f / kNormTile, ff = f % kNormTile;
        const int c = (side ? j0 : i0) + ff;
        double2 v = make_double2(0.0, 0.0);
        if (kk < nk && c < (side ? cols : nf)) {
          const float2 x = c < nf ? feature(S.k, nx, ny, nc, s0, s1, k0 + kk, c)
                                  : S.k[(size_t)(c - nf) * nx * ny + (size_t)tgt * nx + k0 + kk];
          v = make_double2((double)x.x, (double)x.y);
        }
        (side ? fj_s : fi_s)[kk][ff] = v;
      }
      __syncthreads();
      for (int kk = 0; kk < nk; ++kk) {
        const double2 a = fi_s[kk][ti], y = fj_s[kk][tj];
        const double xi = -a.y;
        ar += a.x * y.x - xi * y.y;
        ai += a.x * y.y + xi * y.x;
      }
      __syncthreads();
    }
  }
  if (i0 + ti < nf && j0 + tj < cols) S.work[(size_t)(i0 + ti) * cols + j0 + tj] = make_double2(ar, ai);
}

// One CTA per system: scale by the mean diagonal, add the Tikhonov term, then the pivoted
// Gaussian elimination of [H | B] with every right-hand side at once (hermitian_solve.cuh), in shared
// memory where the system fits (16 coils; `shared`): its steps are a chain, and through global memory
// each took 15 us (30 systems of 48 unknowns: 711 us, here 145).
__global__ void __launch_bounds__(256) grappa_solve_kernel(const GrappaSystem* __restrict__ sys, double lambda,
                                                           int shared) {
  extern __shared__ __align__(16) unsigned char gs_smem[];
  const GrappaSystem& S = sys[blockIdx.x];
  const int nf = 6 * S.nc, nc = S.nc;
  const int cols = nf + nc;
  double2* W = shared ? reinterpret_cast<double2*>(gs_smem) : S.work;
  double* scratch = shared ? reinterpret_cast<double*>(W + (size_t)nf * cols) : S.fscratch;
  __shared__ double red_v[256];
  __shared__ int red_i[256];
  __shared__ double s_scale;
  __shared__ int s_zero;
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int i = 0; i < nf; ++i) sum += S.work[(size_t)i * cols + i].x;
    double mean = sum / (double)nf;
    s_zero = !(mean > 0.0);
    s_scale = s_zero ? 0.0 : 1.0 / mean;
  }
  __syncthreads();
  if (s_zero) {
    for (int e = threadIdx.x; e < nc * nf; e += blockDim.x) S.weights[e] = make_float2(0.f, 0.f);
    return;
  }
  const double sc = s_scale;
  for (int e = threadIdx.x; e < nf * cols; e += blockDim.x) {  // (scale, then add: two roundings)
    double2 v = S.work[e];
    v.x = __dmul_rn(v.x, sc);
    v.y = __dmul_rn(v.y, sc);
    if (e / cols == e % cols) v.x = __dadd_rn(v.x, lambda);
    W[e] = v;
  }
  __syncthreads();
  hermitian_solve_block(W, nf, nc, scratch, scratch + nf, scratch + 2 * nf, S.weights, red_v, red_i);
}

// GRAPPA apply: one thread per (missing line, kx) of one (unit, echo) and eight output coils at a time:
// a source sample is read once for the eight, and their weights come from shared memory ([feature][8],
// one offset d at a time).  600 units, 8 coils, 23 lines of 64: 117 us, 697 with a thread per output
// coil.
constexpr int kApplyCoils = 8;
__global__ void __launch_bounds__(256) grappa_apply_kernel(const ReconJob* __restrict__ jobs,
                                                           const int4* __restrict__ fills, int n_fills) {
  extern __shared__ __align__(16) float2 wts[];  // [6 nc][kApplyCoils]
  const ReconJob& J = jobs[blockIdx.y];
  const int nx = J.nx, ny = J.ny, nc = J.nc, nf = 6 * nc;
  const size_t per = (size_t)nx * ny;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int first = blockIdx.x * blockDim.x / nx;
  const int last = min(n_fills - 1, (int)((blockIdx.x + 1) * blockDim.x - 1) / nx);
  if (first >= n_fills) return;
  const bool mine = e < n_fills * nx;
  const int kx = e % nx;
  const int4 fl = fills[min(e / nx, n_fills - 1)];  // ky, d, s0, s1 (by d)
  int kxs[3];
#pragma unroll
  for (int ki = 0; ki < 3; ++ki) {
    const int x = kx + ki - 1;
    kxs[ki] = x < 0 ? x + nx : (x >= nx ? x - nx : x);
  }
  for (int d = fills[first].y; d <= fills[last].y; ++d)
    for (int co0 = 0; co0 < nc; co0 += kApplyCoils) {
      __syncthreads();  // every thread is done with the weights before
      for (int t = threadIdx.x; t < nf * kApplyCoils; t += blockDim.x) {
        const int c = t / nf, f = t % nf;
        wts[f * kApplyCoils + c] =
            co0 + c < nc ? J.grappa_w[((size_t)(d - 1) * nc + co0 + c) * nf + f] : make_float2(0.f, 0.f);
      }
      __syncthreads();
      if (!mine || fl.y != d) continue;
      float vr[kApplyCoils], vi[kApplyCoils];
#pragma unroll
      for (int c = 0; c < kApplyCoils; ++c) vr[c] = vi[c] = 0.f;
#pragma unroll
      for (int li = 0; li < 2; ++li)
#pragma unroll
        for (int ki = 0; ki < 3; ++ki) {
          const float2* src = J.k + (size_t)(li == 0 ? fl.z : fl.w) * nx + kxs[ki];
          const float2* w = wts + (li * 3 + ki) * nc * kApplyCoils;
          for (int ci = 0; ci < nc; ++ci) {
            const float2 x = src[ci * per];
#pragma unroll
            for (int c = 0; c < kApplyCoils; c += 2) {
              const float4 w2 = *reinterpret_cast<const float4*>(w + ci * kApplyCoils + c);
              vr[c] = vr[c] + (w2.x * x.x - w2.y * x.y);
              vi[c] = vi[c] + (w2.x * x.y + w2.y * x.x);
              vr[c + 1] = vr[c + 1] + (w2.z * x.x - w2.w * x.y);
              vi[c + 1] = vi[c + 1] + (w2.z * x.y + w2.w * x.x);
            }
          }
        }
#pragma unroll
      for (int c = 0; c < kApplyCoils; ++c)
        if (co0 + c < nc) J.k[(co0 + c) * per + (size_t)fl.x * nx + kx] = make_float2(vr[c], vi[c]);
    }
}

// Window, inverse DFT and Roemer combine of one (unit, echo): one CTA per block of YB image rows.
// Per coil: h[y][kx] = sum_ky w k[ky][kx] e^{-i2pi (ky-ys)(y-ys)/ny}  (rows y of the block)
//           img[y][x] = sum_kx h[y][kx] e^{-i2pi (kx-xs)(x-xs)/nx}
//           acc[y][x] += s_q(x,y) img[y][x]
// and finally out = acc / max(sum_q s_q^2, 1e-12).  The exponentials come from exact integer
// indices into one table per axis.
__global__ void __launch_bounds__(256) recon_combine_kernel(const ReconJob* __restrict__ jobs, int YB) {
  extern __shared__ float2 sm[];
  const ReconJob& J = jobs[blockIdx.y];
  const int nx = J.nx, ny = J.ny, nc = J.nc;
  const int y0 = blockIdx.x * YB;
  const int ys = ny / 2, xs = nx / 2;
  float2* Ey = sm;              // ny
  float2* Ex = Ey + ny;         // nx
  float2* h = Ex + nx;          // [YB][nx]
  for (int i = threadIdx.x; i < ny; i += blockDim.x) Ey[i] = J.ey_tab[i];
  for (int i = threadIdx.x; i < nx; i += blockDim.x) Ex[i] = J.ex_tab[i];
  const int nout = YB * nx;
  // accumulators: each thread owns outputs o = threadIdx.x + k*blockDim.x
  constexpr int MAXO = 4;  // YB*nx <= 4*256 outputs per CTA (the host picks YB)
  float2 acc[MAXO];
#pragma unroll
  for (int k = 0; k < MAXO; ++k) acc[k] = make_float2(0.f, 0.f);
  __syncthreads();
  for (int q = 0; q < nc; ++q) {
    const float2* kq = J.k + (size_t)q * nx * ny;
    // stage 1
    for (int o = threadIdx.x; o < nout; o += blockDim.x) {
      const int yy = o / nx, kx = o % nx;
      const int y = y0 + yy;
      float hr = 0.f, hi = 0.f;
      if (y < ny) {
        const int yc = y - ys;
        // m = (ky - ys) yc mod ny, stepped: the same table entries without a modulo per term
        const int step = ((yc % ny) + ny) % ny;
        int m = (((-ys * yc) % ny) + ny) % ny;
        for (int ky = 0; ky < ny; ++ky, m = m + step >= ny ? m + step - ny : m + step) {
          float2 v = kq[(size_t)ky * nx + kx];
          if (J.window) {
            float w = J.window[(size_t)ky * nx + kx];
            v.x *= w;
            v.y *= w;
          }
          const float2 t = Ey[m];
          hr = hr + (v.x * t.x - v.y * t.y);
          hi = hi + (v.x * t.y + v.y * t.x);
        }
      }
      h[o] = make_float2(hr, hi);
    }
    __syncthreads();
    // stage 2
#pragma unroll
    for (int k = 0; k < MAXO; ++k) {
      const int o = threadIdx.x + k * blockDim.x;
      if (o >= nout) break;
      const int yy = o / nx, x = o % nx;
      const int y = y0 + yy;
      if (y >= ny) continue;
      const int xc = x - xs;
      float ir = 0.f, ii = 0.f;
      const int step = ((xc % nx) + nx) % nx;
      int m = (((-xs * xc) % nx) + nx) % nx;
      for (int kx = 0; kx < nx; ++kx, m = m + step >= nx ? m + step - nx : m + step) {
        const float2 v = h[yy * nx + kx];
        const float2 t = Ex[m];
        ir = ir + (v.x * t.x - v.y * t.y);
        ii = ii + (v.x * t.y + v.y * t.x);
      }
      if (J.coil_images)
        J.coil_images[(size_t)q * nx * ny + (size_t)y * nx + x] = make_float2(ir, ii);
      const float s = J.sens[(size_t)q * nx * ny + (size_t)y * nx + x];
      acc[k].x = acc[k].x + ir * s;
      acc[k].y = acc[k].y + ii * s;
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < MAXO; ++k) {
    const int o = threadIdx.x + k * blockDim.x;
    if (o >= nout) break;
    const int yy = o / nx, x = o % nx;
    const int y = y0 + yy;
    if (y >= ny) continue;
    const size_t p = (size_t)y * nx + x;
    const float inv = J.inv_ssum[p];
    J.combined[p] = make_float2(acc[k].x * inv, acc[k].y * inv);
  }
}

// The same by FFTs, for matrices of 32 E points per axis (E <= 4): a cluster of S blocks per (unit, echo)
// takes S coils at a time, a block each.  A coil's k-space is windowed and row-transformed by a warp per
// row as it is read and column-transformed in shared memory; then every block adds the coils' images, in
// coil order, to the Roemer sums of its share of the pixels, so the sums are the same for every S.
// With xs = nx/2 and ys = ny/2 multiples of 16 the centred transform is the plain one between sign flips:
// e^{-i2pi (k - s)(x - s)/n} = (-1)^(k + x) e^{-i2pi kx/n}.
// The twiddles carry their rounding along: it is the forward x-transform's too, and would add up with it
// (one slice of 8 coils against 64 bits: direct sums 1.45e-7, FFT with float32 twiddles 1.53e-7, with both
// parts 1.22e-7).
// Bound by shared memory (90 % of its cycles while the blocks run; the 600 units' last wave is short).
// One block a unit fills the chip from 592 units on; fewer units share their coils among up to 8 blocks.  600
// units of 64 x 64 x 8 coils: 241 us, 0.65 TB/s of k-space (as direct sums 2142 us: 64-term sums at 12 %
// of the FMA rate); one slice of 8 coils 16 us; 32 partitions of 32 coils 59 us.
template <int EX, int EY>
struct ReconShape {
  static constexpr int NX = 32 * EX, NY = 32 * EY, LD = NX + 1;
  static constexpr int T = NX * NY >= 8192 ? 512 : 256, NW = T / 32, NP = NX * NY / T;
  // images of a block of a cluster: two where they fit, so that one is read while the next is formed
  static constexpr int NB = NY * LD <= 6 * 1024 ? 2 : 1;
  static constexpr size_t smem(bool multi) { return sizeof(float2) * ((size_t)(multi ? NB : 1) * NY * LD + 2 * NX + 2 * NY); }
};

template <int EX, int EY, int S>
__global__ void __launch_bounds__(ReconShape<EX, EY>::T) recon_fft_kernel(const ReconJob* __restrict__ jobs) {
  using R = ReconShape<EX, EY>;
  constexpr int NX = R::NX, NY = R::NY, LD = R::LD, T = R::T, NW = R::NW, NP = R::NP;
  constexpr int LX = log2_c(EX), LY = log2_c(EY);
  constexpr bool PX = (EX & (EX - 1)) == 0, PY = (EY & (EY - 1)) == 0;
  extern __shared__ __align__(16) float2 sm[];
  constexpr int NB = S > 1 ? R::NB : 1;
  float2* twx = sm;             // e^{-i2pi j/NX}, then what their rounding took
  float2* twy = twx + 2 * NX;
  float2* imgs = twy + 2 * NY;  // [NB][NY][LD]
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int rank = S > 1 ? (int)cl.block_rank() : 0;
  const ReconJob& J = jobs[blockIdx.x / S];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nc = J.nc;
  for (int i = tid; i < 2 * NX; i += T) twx[i] = J.ex_tab[i];
  for (int i = tid; i < 2 * NY; i += T) twy[i] = J.ey_tab[i];
  const float* __restrict__ sens = J.sens;
  float2* const coil_images = J.coil_images;
  constexpr int MP = (NP + S - 1) / S;  // this block's pixels: tid + (first + p) T
  const int first = rank * MP;
  float2 acc[MP];
#pragma unroll
  for (int p = 0; p < MP; ++p) acc[p] = make_float2(0.f, 0.f);
  auto sync = [&] {
    if (S == 1)
      __syncthreads();
    else
      cl.sync();
  };
  __syncthreads();
  const int k2 = (int)(__brev(lane) >> 27);
  for (int q0 = 0; q0 < nc; q0 += S) {
    const int q = q0 + rank;
    float2* img = imgs + (NB == 2 ? (q0 / S & 1) * NY * LD : 0);
    if (q < nc) {  // (the whole block)
      const float2* kq = J.k + (size_t)q * NX * NY;
      for (int ky = warp; ky < NY; ky += NW) {
        float2 b[EX];
#pragma unroll
        for (int m = 0; m < EX; ++m) {
          const int kx = lane + 32 * m;
          float2 v = kq[ky * NX + kx];
          float w = J.window ? J.window[ky * NX + kx] : 1.f;
          w = ((kx + ky) & 1) ? -w : w;
          b[PX ? bitrev_c(m, LX) : m] = make_float2(v.x * w, v.y * w);
        }
        warp_row_fft<EX, true, true>(b, twx, lane);
#pragma unroll
        for (int k1 = 0; k1 < EX; ++k1) img[ky * LD + k1 + EX * k2] = b[k1];
      }
      __syncthreads();
      for (int x = warp; x < NX; x += NW) {
        float2 b[EY];
#pragma unroll
        for (int m = 0; m < EY; ++m) b[PY ? bitrev_c(m, LY) : m] = img[(lane + 32 * m) * LD + x];
        warp_row_fft<EY, true, true>(b, twy, lane);
#pragma unroll
        for (int k1 = 0; k1 < EY; ++k1) img[(k1 + EY * k2) * LD + x] = b[k1];
      }
    }
    sync();  // the round's images are whole
    // (a pixel's images and sensitivities are loaded before they are added: the loads of the round fly)
    const int nq = min(S, nc - q0);
#pragma unroll
    for (int p = 0; p < MP; ++p) {
      if (NP % S != 0 && first + p >= NP) break;
      const int i = tid + (first + p) * T, y = i / NX, x = i % NX;
      float2 v[S];
      float s[S];
#pragma unroll
      for (int r = 0; r < S; ++r)
        if (S == 1 || r < nq) {
          v[r] = (S > 1 ? cl.map_shared_rank(img, r) : img)[y * LD + x];
          s[r] = sens[(size_t)(q0 + r) * NX * NY + i];
        }
#pragma unroll
      for (int r = 0; r < S; ++r)
        if (S == 1 || r < nq) {
          if ((x + y) & 1) v[r] = make_float2(-v[r].x, -v[r].y);
          if (coil_images) coil_images[(size_t)(q0 + r) * NX * NY + i] = v[r];
          acc[p].x = fmaf(s[r], v[r].x, acc[p].x);
          acc[p].y = fmaf(s[r], v[r].y, acc[p].y);
        }
    }
    if (NB == 1) sync();  // every block has read them
  }
  if (NB == 2) sync();  // (no block leaves while another reads its images)
#pragma unroll
  for (int p = 0; p < MP; ++p) {
    if (NP % S != 0 && first + p >= NP) break;
    const int i = tid + (first + p) * T;
    const float inv = J.inv_ssum[i];
    J.combined[i] = make_float2(acc[p].x * inv, acc[p].y * inv);
  }
}

__global__ void window_copy_kernel(const ReconJob* __restrict__ jobs) {
  const ReconJob& J = jobs[blockIdx.y];
  if (!J.reconstructed) return;  // only the captured slices keep their reconstructed k-space
  const int n = J.nc * J.nx * J.ny;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    float2 v = J.k[e];
    if (J.window) {
      const float w = J.window[e % (J.nx * J.ny)];
      v.x *= w;
      v.y *= w;
    }
    J.reconstructed[e] = v;
  }
}

}  // namespace

namespace {
template <int EX, int EY>
void launch_recon_fft(const ReconJob* d_jobs, int n_jobs, int nc, cudaStream_t st) {
  using R = ReconShape<EX, EY>;
  int S = 1;
  while (2 * S <= std::min(8, nc) && (long long)n_jobs * 2 * S <= 592) S *= 2;
  auto k = S == 8   ? recon_fft_kernel<EX, EY, 8>
           : S == 4 ? recon_fft_kernel<EX, EY, 4>
           : S == 2 ? recon_fft_kernel<EX, EY, 2>
                    : recon_fft_kernel<EX, EY, 1>;
  const size_t smem = R::smem(S > 1);
  if (smem > 48 * 1024)
    MRSIM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n_jobs * S));
  cfg.blockDim = dim3(R::T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)S;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  MRSIM_CUDA(cudaLaunchKernelEx(&cfg, k, d_jobs));
}

template <int EX>
void launch_recon_fft_y(int ey, const ReconJob* d_jobs, int n_jobs, int nc, cudaStream_t st) {
  switch (ey) {
    case 1: launch_recon_fft<EX, 1>(d_jobs, n_jobs, nc, st); break;
    case 2: launch_recon_fft<EX, 2>(d_jobs, n_jobs, nc, st); break;
    case 3: launch_recon_fft<EX, 3>(d_jobs, n_jobs, nc, st); break;
    default: launch_recon_fft<EX, 4>(d_jobs, n_jobs, nc, st); break;
  }
}
}  // namespace

void launch_grappa_fit(const GrappaSystem* d_sys, int n_sys, int max_nc, double lambda, cudaStream_t st) {
  if (n_sys <= 0) return;
  const int nf = 6 * max_nc, cols = nf + max_nc;
  const dim3 grid((cols + kNormTile - 1) / kNormTile, (nf + kNormTile - 1) / kNormTile, n_sys);
  grappa_normal_kernel<<<grid, 256, 0, st>>>(d_sys);
  const size_t smem = (size_t)nf * cols * sizeof(double2) + (size_t)(2 * nf + max_nc * 2 * nf) * sizeof(double);
  constexpr size_t kMost = 216 * 1024;  // beside 3 KB of static shared memory
  const bool shared = smem <= kMost;
  if (shared && smem > 40 * 1024)
    MRSIM_CUDA(cudaFuncSetAttribute(grappa_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
  grappa_solve_kernel<<<n_sys, 256, shared ? smem : 0, st>>>(d_sys, lambda, shared ? 1 : 0);
}

void launch_grappa_apply(const ReconJob* d_jobs, int n_jobs, const int4* d_fills, int n_fills, int nx, int nc,
                         cudaStream_t st) {
  if (n_jobs <= 0 || n_fills <= 0) return;
  const dim3 grid(((long long)n_fills * nx + 255) / 256, n_jobs);
  grappa_apply_kernel<<<grid, 256, sizeof(float2) * 6 * nc * kApplyCoils, st>>>(d_jobs, d_fills, n_fills);
}

void launch_recon_combine(const ReconJob* d_jobs, int n_jobs, int nx, int ny, int nc, bool capture_reconstructed,
                          cudaStream_t st) {
  if (n_jobs <= 0) return;
  if (capture_reconstructed) {
    dim3 g(64, n_jobs);
    window_copy_kernel<<<g, 256, 0, st>>>(d_jobs);
  }
  if (nx % 32 == 0 && ny % 32 == 0 && nx <= 128 && ny <= 128) {
    switch (nx / 32) {
      case 1: launch_recon_fft_y<1>(ny / 32, d_jobs, n_jobs, nc, st); break;
      case 2: launch_recon_fft_y<2>(ny / 32, d_jobs, n_jobs, nc, st); break;
      case 3: launch_recon_fft_y<3>(ny / 32, d_jobs, n_jobs, nc, st); break;
      default: launch_recon_fft_y<4>(ny / 32, d_jobs, n_jobs, nc, st); break;
    }
    return;
  }
  const int YB = std::max(1, std::min(8, 1024 / nx));
  dim3 grid((ny + YB - 1) / YB, n_jobs);
  size_t smem = sizeof(float2) * (size_t)(ny + nx + YB * nx);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(recon_combine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  recon_combine_kernel<<<grid, 256, smem, st>>>(d_jobs, YB);
}

}  // namespace mrsim
