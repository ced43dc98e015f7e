// epi_kernels.cu — the exact-DFT EPI forward operator and its adjoint / VJP, FP32, sm_100a.
//
// The forward restates `build_coil_kspace_timed` (reference kspace.rs:607-1042) without its
// spikes and noise.  For each unit (one slice of one volume, every echo's acquired lines) it
// evaluates, exactly (no time segmentation, no NUFFT),
//
//   g_q[j][x] = s * sum_y amp_q(x,y) * W_j(x,y) * e^{i 2pi theta_j(x,y)}          (y-stage)
//   k_q[row_j][kx] = (1/nvox) sum_x g_q[j][x] * E_j(x) * tw_pol(j)(kx, x)           (x-stage)
//
//   theta_j = a(x,y) + f(x,y) * t_j + (ky_j - ys)(y - sys - yoff)/sny + Py(y)*decay_j
//   W_j     = sum_c rel_cj(x,y) m_c(x,y)
//
// `a` is the static phase in turns (object phase, eddy object-phase ramp), `Py*decay` the y part
// of the separable eddy polynomial (kspace.rs:904-925), E_j its x and z parts, and tw the x-stage
// twiddle of the line's readout polarity (`XStage`, kspace.rs:1052-1140).  The k.r phase of the
// y-DFT is an exact integer index (ky-ys)*(2(y-sys)-(oy-1)) mod 2*sny; f*t is split hi+lo
// (two-product) so the phase keeps ~1e-7 turn accuracy before the MUFU sin/cos of the reduced
// argument.  amp_q(x,y) = ex_q(x)*ey_q(y) + off is `coil_sensitivity` (kspace.rs:226-237)
// factored per axis (the Gaussian is separable).
//
// The adjoint is the Hermitian transpose with respect to complex compartment images, plus the
// vector-Jacobian products of L = sum |k - d|^2 with respect to the fieldmap and each
// compartment's R2 = 1/T2 (the reference has no adjoint; the oracle is the FP64 transpose).
//
// Kernels, in the order a step runs them:
//   statics_kernel                     static phase a(x,y) in turns (FP64 per-slice quadratic)
//   ystage_q_kernel / ystage_kernel    y-stage (epi_ystage.cu: staged-input form; per-thread-load fallback);
//                                      with the 8-coil ring it accumulates 5 ey classes + offset,
//                                      with other rings of 6 or more coils the rows of a coil basis
//   xfft_warp_kernel / xfft_kernel /   x-stage: warp-per-row FFT (N = 32..256), shared-memory
//   xgemm_kernel                       radix-2 FFT (other powers of two), DFT GEMM (other widths)
//   yadjoint_q_kernel / yadjoint_kernel  y-adjoint (epi_yadjoint.cu: fixed coil or class count; any
//                                      coil count)
//   ystage_thin_kernel / yadjoint_thin_kernel  both for plans of few tiles (epi_ythin.cu), same bits
// The class-mode and packed (f32x2) paths are exact rearrangements: equal ey rows, and lanes that
// round like the scalar operations.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>

#include <cstring>
#include <map>

#include "epi_device.h"
#include "mrsim_internal.h"
#include "row_fft.h"

namespace mrsim {

namespace {

// ---------------------------------------------------------------------------------------------
// statics: a(x,y) = frac( (phi0 + eddy object phase) / 2pi ) in FP64, stored as f32 turns.
// phi0 = phase0[i] (explicit) or the phase model `PhaseModel::at` (phase.rs:141) sampled by
// `phase_slice` (kspace.rs:1156-1180).
__global__ void statics_kernel(const StaticDesc* descs) {
  grid_begin();
  const StaticDesc& d = descs[blockIdx.y];
  const int n = d.snx * d.sny;
  const double inv_tau = 0.15915494309189533577;
  const int ox = d.snx / d.nx, oy = d.sny / d.ny;
  const int sxs = ox * (d.nx / 2), sys = oy * (d.ny / 2);
  const double xoff = (ox - 1.0) / 2.0, yoff = (oy - 1.0) / 2.0;
  const bool explicit_phase = (d.flags & 1) != 0;
  // Within a slice the phase model is a quadratic in (x, y): with r0 = (x - sx - off)/o,
  // r1 = (y - sy - off)/o and r2 the slice coordinate, background + shot term are
  //   A + B r0 + C r1 + D r0^2 + E r1^2 + F r0 r1
  // and the eddy object-phase ramp is affine in x and y.  Each thread forms the six FP64
  // coefficients once and evaluates its voxels by Horner's rule.
  double c00 = 0, cx = 0, cy = 0, cxx = 0, cyy = 0, cxy = 0;
  {
    const double o = d.o, sx = d.snx / 2.0, sy = d.sny / 2.0, off = (o - 1.0) / 2.0;
    const double r2 = d.z - d.nz_full / 2.0;
    const double* c = d.bg;
    double A = 0, B = 0, C = 0, D = 0, E = 0, F = 0;
    if (!explicit_phase) {
      const double* q = d.shot_q;
      const double* dx = d.shot_dx;
      const double* rot = d.shot_rot;
      A = d.global + c[0] + c[3] * r2 + c[6] * r2 * r2 + q[0] * (dx[0] + rot[1] * r2) +
          q[1] * (dx[1] - rot[0] * r2) + q[2] * dx[2];
      B = c[1] + c[8] * r2 + q[1] * rot[2] - q[2] * rot[1];
      C = c[2] + c[9] * r2 - q[0] * rot[2] + q[2] * rot[0];
      D = c[4];
      E = c[5];
      F = c[7];
    }
    // r0 = a0 + x / o, r1 = b0 + y / o
    const double a0 = -(sx + off) / o, b0 = -(sy + off) / o, io = 1.0 / o;
    c00 = A + B * a0 + C * b0 + D * a0 * a0 + E * b0 * b0 + F * a0 * b0;
    cx = (B + 2.0 * D * a0 + F * b0) * io;
    cy = (C + 2.0 * E * b0 + F * a0) * io;
    cxx = D * io * io;
    cyy = E * io * io;
    cxy = F * io * io;
    if (d.flags & 2) {  // + e0 (x - sxs - xoff)/ox + e1 (y - sys - yoff)/oy + e2 zc
      const double* e = d.eddy_phase_coef;
      c00 += -e[0] * (sxs + xoff) / ox - e[1] * (sys + yoff) / oy + e[2] * d.zc_c;
      cx += e[0] / ox;
      cy += e[1] / oy;
    }
  }
  grid_wait();  // the step before may still read this phase
  const double* __restrict__ phase0 = d.phase0;
  float* __restrict__ out = d.out;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = i % d.snx, y = i / d.snx;
    double p0 = explicit_phase ? phase0[i] : fma(x, fma(cxx, x, fma(cxy, y, cx)), fma(y, fma(cyy, y, cy), c00));
    if (explicit_phase && (d.flags & 2)) p0 += fma(cx, x, fma(cy, y, c00));
    double tt = p0 * inv_tau;
    tt -= rint(tt);
    out[i] = (float)tt;
  }
}

// Chains in which a column's coils are added to the constant basis row (coil q in chain q mod 4), before
// the chains are added.  That row is nearly all of H, and its rounding is common to every voxel of a
// column, which a coil's own was not: H of 32 coils is off by 9.3e-8 in one chain, 7.8e-8 in four (7.9e-8
// by per-coil sums).
constexpr int kCoilChains = 4;

// ---------------------------------------------------------------------------------------------
// x-stage as a register-tiled complex GEMM.  A tile is up to 32 rows (lines of ONE readout polarity
// x coils) by 64 output columns; K runs over the contraction in chunks of 32 staged in shared memory.
//   forward : out[q][row_j][kx] = (1/nvox) sum_x  g[q][j][x] E_j(x)        tw_pol[x][kx]
//   adjoint : h[q][j][x]        = (1/nvox) conj(E_j(x)) sum_kx conj(tw_pol[x][kx]) r[q][row_j][kx]
// Each of 256 threads owns 4 rows x 2 columns.
// nb > 0: g holds the unit's nb basis rows ([r][line][x]).  The forward forms each coil's
// g_q = ex_q sum_r U_qr G_r + off G_last as it stages A; the adjoint's tile holds every coil of its
// lines and writes G_r = s sum_q (ex_q U_qr + off [r = last]) h_q.
template <bool ADJ>
__global__ void __launch_bounds__(256) xgemm_kernel(const UnitDesc* __restrict__ units,
                                                    const XTile* __restrict__ tiles, int nb) {
  __shared__ float2 As[32][33];   // [row][k]
  __shared__ float2 Bs[32][64];   // [k][col]
  __shared__ int lrow[32], lline[32], lq[32];
  __shared__ float ldec[32];
  const XTile& T = tiles[blockIdx.x];
  const UnitDesc& u = units[T.unit];
  const int snx = u.snx, nx = u.nx;
  const int K = ADJ ? nx : snx;       // contraction length
  const int N = ADJ ? snx : nx;       // output columns
  const int nrows = T.nl * T.nq;
  const int ox = snx / nx, sxs = ox * (nx / 2);
  const double xoff = (ox - 1.0) / 2.0;
  const bool eddy = (u.flags & UF_EDDY) != 0;
  if (threadIdx.x < 32) {
    const int r = threadIdx.x;
    if (r < nrows) {
      const int jj = r / T.nq, qq = r % T.nq;
      const LineRec& L = u.lines[T.line[jj]];
      lrow[r] = L.row;
      lline[r] = T.line[jj];
      lq[r] = T.q0 + qq;
      ldec[r] = L.decay;
    } else {
      lrow[r] = 0;
      lline[r] = 0;
      lq[r] = -1;
      ldec[r] = 0.f;
    }
  }
  __syncthreads();
  // the twiddles of this tile's polarity: forward [x][kx], adjoint [kx][x] (transposed table)
  const float2* tw = u.geo.tw + (size_t)(ADJ ? 2 + T.pol : T.pol) * snx * nx;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 8 row groups of 4
  float2 acc[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
  for (int k0 = 0; k0 < K; k0 += 32) {
    // stage A: 32 rows x 32 k
    for (int e = threadIdx.x; e < 32 * 32; e += 256) {
      const int r = e >> 5, kk = e & 31, k = k0 + kk;
      float2 v = make_float2(0.f, 0.f);
      if (lq[r] >= 0 && k < K) {
        if (!ADJ) {
          if (nb > 0) {
            const float* co = u.geo.bco + lq[r] * kBasisPad;
            const float2* G = u.g + (size_t)lline[r] * snx + k;
            const size_t rs = (size_t)u.n_lines * snx;
            float2 t = make_float2(0.f, 0.f), last = t;
            for (int b = 0; b < nb; ++b) {
              last = G[b * rs];
              t = ffma2(dup2(co[b]), last, t);
            }
            v = ffma2(dup2(u.geo.coil_off), last, fmul2(dup2(u.geo.ex[(size_t)lq[r] * snx + k]), t));
          } else {
            v = u.g[((size_t)lq[r] * u.n_lines + lline[r]) * snx + k];
          }
          if (eddy) {
            const double xc = ((double)k - sxs - xoff) / ox;
            double tv = ((double)u.eddy_cx * xc + (double)u.eddy_qx * xc * xc + (double)u.eddy_z) * (double)ldec[r];
            tv -= rint(tv);
            float sn, cs;
            __sincosf(kTwoPiF * (float)tv, &sn, &cs);
            v = make_float2(v.x * cs - v.y * sn, v.x * sn + v.y * cs);
          }
        } else {
          v = u.kspace[((size_t)lq[r] * u.n_rows + lrow[r]) * nx + k];
        }
      }
      As[r][kk] = v;
    }
    // stage B: 32 k x 64 columns
    for (int e = threadIdx.x; e < 32 * 64; e += 256) {
      const int kk = e >> 6, c = e & 63, k = k0 + kk, col = T.col0 + c;
      Bs[kk][c] = (k < K && col < N) ? __ldg(tw + (size_t)k * N + col) : make_float2(0.f, 0.f);
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < 32; ++kk) {
      const float2 b0 = Bs[kk][tx], b1 = Bs[kk][tx + 32];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = As[ty * 4 + i][kk];
        if (!ADJ) {
          acc[i][0].x = fmaf(a.x, b0.x, fmaf(-a.y, b0.y, acc[i][0].x));
          acc[i][0].y = fmaf(a.x, b0.y, fmaf(a.y, b0.x, acc[i][0].y));
          acc[i][1].x = fmaf(a.x, b1.x, fmaf(-a.y, b1.y, acc[i][1].x));
          acc[i][1].y = fmaf(a.x, b1.y, fmaf(a.y, b1.x, acc[i][1].y));
        } else {  // a * conj(b)
          acc[i][0].x = fmaf(a.x, b0.x, fmaf(a.y, b0.y, acc[i][0].x));
          acc[i][0].y = fmaf(a.y, b0.x, fmaf(-a.x, b0.y, acc[i][0].y));
          acc[i][1].x = fmaf(a.x, b1.x, fmaf(a.y, b1.y, acc[i][1].x));
          acc[i][1].y = fmaf(a.y, b1.x, fmaf(-a.x, b1.y, acc[i][1].y));
        }
      }
    }
    __syncthreads();
  }
  const float inv_n = 1.0f / (float)(snx * u.sny);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (lq[r] < 0) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = T.col0 + tx + 32 * h;
      if (col >= N) continue;
      float2 v = make_float2(acc[i][h].x * inv_n, acc[i][h].y * inv_n);
      if (!ADJ) {
        u.kspace[((size_t)lq[r] * u.n_rows + lrow[r]) * nx + col] = v;
      } else {
        if (eddy) {
          const double xc = ((double)col - sxs - xoff) / ox;
          double tv = ((double)u.eddy_cx * xc + (double)u.eddy_qx * xc * xc + (double)u.eddy_z) * (double)ldec[r];
          tv -= rint(tv);
          float sn, cs;
          __sincosf(kTwoPiF * (float)tv, &sn, &cs);
          v = make_float2(v.x * cs + v.y * sn, v.y * cs - v.x * sn);
        }
        if (nb > 0)
          Bs[r][tx + 32 * h] = v;  // every thread left the last k chunk's products at a barrier
        else
          u.g[((size_t)lq[r] * u.n_lines + lline[r]) * snx + col] = v;
      }
    }
  }
  if (ADJ && nb > 0) {
    __syncthreads();
    const float s = u.signal_scale, so = s * u.geo.coil_off;
    for (int e = threadIdx.x; e < T.nl * 64; e += 256) {
      const int jj = e >> 6, c = e & 63, col = T.col0 + c;
      if (col >= N) continue;
      float2 G[kBasisPad - 2], last = make_float2(0.f, 0.f);
#pragma unroll
      for (int b = 0; b < kBasisPad - 2; ++b) G[b] = make_float2(0.f, 0.f);
      float2 chain[kCoilChains];
#pragma unroll
      for (int k = 0; k < kCoilChains; ++k) chain[k] = make_float2(0.f, 0.f);
      auto add = [&](int q, float2& l) {
        const float2 h = Bs[jj * T.nq + q][c];
        const float* co = u.geo.bco + (T.q0 + q) * kBasisPad;
        const float ex = s * u.geo.ex[(size_t)(T.q0 + q) * snx + col];
        const float2 w = fmul2(dup2(ex), h);
        l = ffma2(dup2(fmaf(ex, co[kBasisPad - 1], so)), h, l);
#pragma unroll
        for (int b = 0; b < kBasisPad - 2; ++b)
          if (b < nb - 1) G[b] = ffma2(dup2(co[b]), w, G[b]);
      };
      for (int q = 0; q < T.nq; q += kCoilChains)
#pragma unroll
        for (int k = 0; k < kCoilChains; ++k)
          if (q + k < T.nq) add(q + k, chain[k]);
      last = fadd2(fadd2(chain[0], chain[1]), fadd2(chain[2], chain[3]));
      const size_t base = (size_t)T.line[jj] * snx + col, rs = (size_t)u.n_lines * snx;
#pragma unroll
      for (int b = 0; b < kBasisPad - 2; ++b)
        if (b < nb - 1) u.g[base + b * rs] = G[b];
      u.g[base + (nb - 1) * rs] = last;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// x-stage as per-row FFTs when snx = N is a power of two.  The twiddle of the line's polarity
// factors as tw[x][kx] = premod(x) e^{i2pi K x/N} post(kx), K = kx - xs, since
// (K + gh)(x - c) = K x + gh (x - c) - K c, so
//   forward : out[q][row_j][kx] = (1/nvox) post(kx) FFT+[ g[q][j][x] E_j(x) premod(x) ](K mod N)
//   adjoint : h[q][j][x]        = (1/nvox) conj(E_j(x) premod(x)) FFT-[ r[q][row_j][kx] conj(post(kx)) at K mod N ](x)
// (FFT+- : sum e^{+-i2pi k x/N}).  A CTA of 256 threads transforms up to 2048/N rows of one unit
// ([coil][line] order) in shared memory: radix-2 decimation in time from bit-reversed loads.
// Tile = (unit, first row, rows).
template <bool ADJ>
__global__ void __launch_bounds__(256) xfft_kernel(const UnitDesc* __restrict__ units, const int4* __restrict__ tiles) {
  __shared__ __align__(16) float2 buf[kXfftMaxN];
  __shared__ __align__(16) float2 tws[kXfftMaxN / 2];
  __shared__ int rq[256], rline[256], rrow[256], rpol[256];
  __shared__ float rdec[256];
  const int4 t = tiles[blockIdx.x];
  const UnitDesc& u = units[t.x];
  const int r0 = t.y, nr = t.z;
  const int N = u.snx, nx = u.nx, nl = u.n_lines;
  const int logn = 31 - __clz(N), half = N >> 1;
  const int tid = threadIdx.x;
  const float2* __restrict__ xf = u.geo.xf;
  const float2* __restrict__ premod = xf + half;
  const float2* __restrict__ post = xf + half + 2 * N;
  for (int k = tid; k < half; k += 256) tws[k] = xf[k];
  for (int r = tid; r < nr; r += 256) {
    const int R = r0 + r, q = R / nl, j = R % nl;
    const LineRec& L = u.lines[j];
    rq[r] = q;
    rline[r] = j;
    rrow[r] = L.row;
    rpol[r] = L.pol < 0 ? 1 : 0;
    rdec[r] = L.decay;
  }
  __syncthreads();
  const int ox = N / nx, xs = nx / 2, sxs = ox * xs;
  const double xoff = (ox - 1.0) / 2.0;
  const bool eddy = (u.flags & UF_EDDY) != 0;
  // E_j(x) = e^{i2pi (cx xc + qx xc^2 + z) decay_j}: the x and z parts of the eddy polynomial
  auto eddy_factor = [&](int x, float dec) {
    const double xc = ((double)x - sxs - xoff) / ox;
    double tv = ((double)u.eddy_cx * xc + (double)u.eddy_qx * xc * xc + (double)u.eddy_z) * (double)dec;
    tv -= rint(tv);
    float sn, cs;
    __sincosf(kTwoPiF * (float)tv, &sn, &cs);
    return make_float2(cs, sn);
  };
  const float inv_n = 1.0f / (float)(N * u.sny);
  const int kpos = nx - xs;  // K in [-xs, kpos)
  if (!ADJ) {
    for (int e = tid; e < nr * N; e += 256) {
      const int r = e >> logn, x = e & (N - 1);
      const float2 v = u.g[(size_t)(r0 + r) * N + x];
      float2 m = premod[rpol[r] * N + x];
      if (eddy) m = cmul(m, eddy_factor(x, rdec[r]));
      buf[(r << logn) + (__brev(x) >> (32 - logn))] = cmul(v, m);
    }
  } else {
    for (int e = tid; e < nr * N; e += 256) {
      const int r = e >> logn, k = e & (N - 1);
      const int K = k < kpos ? k : k - N;
      const int kx = K + xs;
      float2 v = make_float2(0.f, 0.f);
      if (kx >= 0 && kx < nx) {
        const float2 p = post[kx];
        v = cmul(u.kspace[((size_t)rq[r] * u.n_rows + rrow[r]) * nx + kx], make_float2(p.x, -p.y));
      }
      buf[(r << logn) + (__brev(k) >> (32 - logn))] = v;
    }
  }
  __syncthreads();
  for (int s = 1; s <= logn; ++s) {
    const int h = 1 << (s - 1);
    for (int b = tid; b < nr * half; b += 256) {
      const int r = b >> (logn - 1), bb = b & (half - 1);
      const int pos = bb & (h - 1), grp = bb >> (s - 1);
      const int i0 = (r << logn) + (grp << s) + pos, i1 = i0 + h;
      float2 w = tws[pos << (logn - s)];  // e^{-i2pi pos / 2h}
      if (!ADJ) w.y = -w.y;
      const float2 a = buf[i0], bw = cmul(buf[i1], w);
      buf[i0] = make_float2(a.x + bw.x, a.y + bw.y);
      buf[i1] = make_float2(a.x - bw.x, a.y - bw.y);
    }
    __syncthreads();
  }
  if (!ADJ) {
    for (int e = tid; e < nr * nx; e += 256) {
      const int r = e / nx, kx = e % nx;
      const int k = (kx - xs) & (N - 1);
      const float2 v = cmul(buf[(r << logn) + k], post[kx]);
      u.kspace[((size_t)rq[r] * u.n_rows + rrow[r]) * nx + kx] = make_float2(v.x * inv_n, v.y * inv_n);
    }
  } else {
    for (int e = tid; e < nr * N; e += 256) {
      const int r = e >> logn, x = e & (N - 1);
      float2 m = premod[rpol[r] * N + x];
      if (eddy) m = cmul(m, eddy_factor(x, rdec[r]));
      const float2 v = cmul(buf[e], make_float2(m.x, -m.y));
      u.g[(size_t)(r0 + r) * N + x] = make_float2(v.x * inv_n, v.y * inv_n);
    }
  }
}

// The same x-stage with one warp per row for N = 32 E (E = 1..8, any E), no block barriers: lane t
// holds x[t + 32 m] (m < E).  With n = t + 32 m and k = k1 + E k2, W = e^{+-i2pi/N}:
//   X[k1 + E k2] = sum_t W^{t k1} [ sum_m x[t + 32 m] W^{32 m k1} ] W^{E t k2}
// so each lane does an E-point DFT of its registers (radix-2, unrolled), the twiddles W^{t k1},
// and the 32-point DFTs over t run as five radix-2 decimation-in-frequency stages of lane
// shuffles, which leave X[k1 + E k2] in lane bitrev5(k2).  A per-warp shared row (padded one
// slot in 32) puts the results back in natural order for coalesced stores.
//
// CLS (8 coils in 5 classes + offset): a tile is (unit, first line, up to 4 lines) x all 8 coils.
// Adjoint: warp w transforms coil w of each line into shared memory, and the CTA then writes the
// 6 class rows G_v = s sum_{q in v} ex_q h_q, G_off = s off sum_q h_q ([v][line][x] in g) that
// the class-mode y-adjoint combines as sum_v ey_v(y) G_v + G_off.  Forward: the CTA stages the
// tile's class rows from the class-mode y-stage and each row loads g_q = ex_q G_cls(q) + G_off.
template <int E, bool ADJ, bool CLS>
__global__ void __launch_bounds__(256, E <= 4 ? 4 : 2) xfft_warp_kernel(const UnitDesc* __restrict__ units,
                                                           const int4* __restrict__ tiles) {
  constexpr int N = 32 * E, LE = log2_c(E);
  constexpr bool P2 = (E & (E - 1)) == 0;  // E a power of two: radix-2 register DFT, else direct
  constexpr int NP = N + N / 32;  // padded row
  constexpr int RT = 32;          // rows per tile
  static_assert(!CLS || E <= 4, "coil classes: rows of at most 128 points");
  __shared__ __align__(16) float2 hsm[CLS ? 4 * 8 * N : 1];  // [line][coil][x]
  __shared__ int cls_s[8];
  __shared__ __align__(16) float2 tw[N];        // e^{-i2pi j/N}
  __shared__ __align__(16) float2 pm[2 * N];    // premodulation per polarity
  __shared__ __align__(16) float2 pt[N];        // post-twiddle per kx (nx <= N)
  __shared__ __align__(16) float2 rb[8][NP];
  __shared__ int rq[RT], rrow[RT], rpol[RT];
  __shared__ float rdec[RT];
  const int4 t = tiles[blockIdx.x];
  const UnitDesc& u = units[t.x];
  const int r0 = t.y, nr = CLS ? 8 * t.z : t.z;  // CLS: first line, lines
  const int nx = u.nx, nl = u.n_lines, n_rows = u.n_rows;
  // the unit's buffers, read once: the row loop's warp barriers order memory, so the fields would
  // otherwise be loaded again for every row
  float2* const ksp = u.kspace;
  float2* const gbuf = u.g;
  // forward: the 8 coils' ex rows ([q][x]) after the class rows of at most 4 lines (24 N float2)
  float* exs = CLS ? reinterpret_cast<float*>(hsm + 24 * N) : nullptr;
  grid_begin();
  // a small launch fills its tables while the kernel before it ends; a larger one issues its row copies
  // first, which then fly while the tables fill
  const bool fill = ADJ || gridDim.x <= kChainTiles;
  if (!fill) grid_wait();
  // forward: the tile's class rows, [line][v][x], as 16-byte asynchronous copies (N is even and the
  // rows of g start on 16-byte boundaries)
  auto stage_rows = [&] {
    constexpr int HN = N / 2;
    const float4* g4 = reinterpret_cast<const float4*>(gbuf);
    float4* h4 = reinterpret_cast<float4*>(hsm);
    for (int e = threadIdx.x; e < (nr >> 3) * 6 * HN; e += 256) {
      const int jl = e / (6 * HN), v = (e / HN) % 6, x2 = e % HN;
      cp_async16(h4 + e, g4 + ((size_t)v * nl + r0 + jl) * HN + x2, 16);
    }
    cp_async_commit();
  };
  if (CLS && !ADJ && !fill) stage_rows();
  if (CLS && !ADJ)
    for (int e = threadIdx.x; e < 8 * N; e += 256) exs[e] = u.geo.ex[e];
  const float2* __restrict__ xf = u.geo.xf;
  for (int k = threadIdx.x; k < N / 2; k += 256) {
    const float2 w = xf[k];
    tw[k] = w;
    tw[k + N / 2] = make_float2(-w.x, -w.y);
  }
  // the output side's table carries the 1/(N sny) scale: the post-twiddle in the forward, the
  // premodulation in the adjoint
  const float inv_n = 1.0f / (float)(N * u.sny);
  for (int k = threadIdx.x; k < 2 * N; k += 256) {
    const float2 v = xf[N / 2 + k];
    pm[k] = ADJ ? make_float2(v.x * inv_n, v.y * inv_n) : v;
  }
  for (int k = threadIdx.x; k < nx; k += 256) {
    const float2 v = xf[N / 2 + 2 * N + k];
    pt[k] = ADJ ? v : make_float2(v.x * inv_n, v.y * inv_n);
  }
  if (CLS && threadIdx.x < 8) cls_s[threadIdx.x] = u.geo.cls[threadIdx.x];
  for (int r = threadIdx.x; r < nr; r += 256) {
    const int R = CLS ? (r & 7) * nl + r0 + (r >> 3) : r0 + r;  // CLS: row r = (line r / 8, coil r % 8)
    const LineRec& L = u.lines[R % nl];
    rq[r] = R / nl;
    rrow[r] = L.row;
    rpol[r] = L.pol < 0 ? 1 : 0;
    rdec[r] = L.decay;
  }
  if (fill) grid_wait();
  if (CLS && !ADJ && fill) stage_rows();
  if (CLS && !ADJ) cp_async_wait0();
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ox = N / nx, xs = nx / 2, sxs = ox * xs;
  const double xoff = (ox - 1.0) / 2.0;
  const bool eddy = (u.flags & UF_EDDY) != 0;
  const int kpos = nx - xs;
  float2* row = rb[warp];
  // premodulation of the line's polarity times E_j(x) = e^{i2pi (cx xc + qx xc^2 + z) decay_j}
  auto modulation = [&](int pol, float dec, int x) {
    float2 md = pm[pol * N + x];
    if (eddy) {
      const double xc = ((double)x - sxs - xoff) / ox;
      double tv = ((double)u.eddy_cx * xc + (double)u.eddy_qx * xc * xc + (double)u.eddy_z) * (double)dec;
      tv -= rint(tv);
      float sn, cs;
      __sincosf(kTwoPiF * (float)tv, &sn, &cs);
      md = cmul(md, make_float2(cs, sn));
    }
    return md;
  };
  // adjoint: the k-space samples of the warp's next row are loaded while the current row transforms
  // (zero outside the acquired kx)
  float2 pre[ADJ ? E : 1];
  auto fetch = [&](int r) {
    const float2* kr = ksp + ((size_t)rq[r] * n_rows + rrow[r]) * nx;
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int n = lane + 32 * m;
      const int kx = (n < kpos ? n : n - N) + xs;
      pre[ADJ ? m : 0] = kx >= 0 && kx < nx ? kr[kx] : make_float2(0.f, 0.f);
    }
  };
  if (ADJ && warp < nr) fetch(warp);
  for (int r = warp; r < nr; r += 8) {
    const int R = CLS ? (r & 7) * nl + r0 + (r >> 3) : r0 + r, q = rq[r], orow = rrow[r], pol = rpol[r];
    const float dec = rdec[r];
    float2 b[E];
    if (!ADJ && CLS) {
      const int jl = r >> 3, c = cls_s[q];
      const float2* cr = hsm + (jl * 6) * N;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int x = lane + 32 * m;
        const float ex = exs[q * N + x];
        const float2 gv = cr[c * N + x], go = cr[5 * N + x];
        b[P2 ? bitrev_c(m, LE) : m] = cmul(make_float2(fmaf(ex, gv.x, go.x), fmaf(ex, gv.y, go.y)), modulation(pol, dec, x));
      }
    } else if (!ADJ) {
      const float2* gr = gbuf + (size_t)R * N;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int x = lane + 32 * m;
        b[P2 ? bitrev_c(m, LE) : m] = cmul(gr[x], modulation(pol, dec, x));
      }
    } else {
      float2 cur[E];
#pragma unroll
      for (int m = 0; m < E; ++m) cur[m] = pre[ADJ ? m : 0];
      if (r + 8 < nr) fetch(r + 8);
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int n = lane + 32 * m;
        const int kx = (n < kpos ? n : n - N) + xs;
        float2 v = make_float2(0.f, 0.f);
        if (kx >= 0 && kx < nx) {
          const float2 p = pt[kx];
          v = cmul(cur[m], make_float2(p.x, -p.y));
        }
        b[P2 ? bitrev_c(m, LE) : m] = v;
      }
    }
    warp_row_fft<E, ADJ>(b, tw, lane);
    const int k2 = __brev(lane) >> 27;
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) {
      const int k = k1 + E * k2;
      row[k + (k >> 5)] = b[k1];
    }
    __syncwarp();
    if (!ADJ) {
      float2* out = ksp + ((size_t)q * n_rows + orow) * nx;
      for (int kx = lane; kx < nx; kx += 32) {
        const int k = ((kx - xs) % N + N) % N;
        out[kx] = cmul(row[k + (k >> 5)], pt[kx]);
      }
    } else {
      float2* gr = CLS ? hsm + ((r >> 3) * 8 + (r & 7)) * N : gbuf + (size_t)R * N;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int x = lane + 32 * m;
        const float2 md = modulation(pol, dec, x);
        gr[x] = cmul(row[x + (x >> 5)], make_float2(md.x, -md.y));
      }
    }
    __syncwarp();
  }
  if (CLS && ADJ) {
    __syncthreads();
    const float s = u.signal_scale, so = s * u.geo.coil_off;
    float* sex = reinterpret_cast<float*>(&rb[0][0]);  // s ex_q(x), [q][x], in the free reorder rows
    for (int e = threadIdx.x; e < 8 * N; e += 256) sex[e] = s * u.geo.ex[e];
    __syncthreads();
    const int nj = nr >> 3;
    for (int e = threadIdx.x; e < nj * N; e += 256) {
      const int jl = e / N, x = e % N;
      float2 G[6];
#pragma unroll
      for (int v = 0; v < 6; ++v) G[v] = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float2 h = hsm[(jl * 8 + q) * N + x];
        const float ex = sex[q * N + x];
        const int c = cls_s[q];
#pragma unroll
        for (int v = 0; v < 5; ++v)
          if (c == v) {
            G[v].x = fmaf(ex, h.x, G[v].x);
            G[v].y = fmaf(ex, h.y, G[v].y);
          }
        G[5].x += h.x;
        G[5].y += h.y;
      }
      G[5] = make_float2(so * G[5].x, so * G[5].y);
#pragma unroll
      for (int v = 0; v < 6; ++v) gbuf[((size_t)v * nl + r0 + jl) * N + x] = G[v];
    }
  }
}

// The same x-stage on the rows of a coil basis (nb of them, at most 7), for any coil count: a tile is
// (unit, first line, lines) x every coil.  Forward: the tile's basis rows G_r ([r][line][x] in g, the
// y-stage's) are staged once, and each coil's row is formed as the warp loads it,
//   g_q(x) = ex_q(x) sum_r U_qr G_r(x) + off G_last(x);
// adjoint: the coils' rows h_q pass through shared memory, at most 32 at a time, and the CTA writes
//   G_r(x) = s sum_q (ex_q(x) U_qr + off [r = last]) h_q(x).
// Against one row per coil the forward reads and the adjoint writes nb rows in place of ncoils, and
// both y-stages run on nb rows.  The coil sums cost 2 (nb + 1) FMAs per row element, about what the
// row's transform costs, and stay small beside the y-stages (each element serves sny voxels).
constexpr int kBasisRows = 32;  // coil rows the adjoint holds at a time
__host__ __device__ constexpr int basis_lines(int ncoils) { return ncoils >= kBasisRows ? 1 : kBasisRows / ncoils; }
// float2 of dynamic shared memory: tables, reorder rows, then the staged basis or coil rows
__host__ __device__ constexpr size_t basis_smem(int E, int staged_rows) {
  return (size_t)(32 * E) * 4 + 8 * (size_t)(33 * E) + (size_t)staged_rows * 32 * E;
}

template <int E, bool ADJ>
__global__ void __launch_bounds__(256, E > 4 ? 2 : ADJ ? 3 : 4) xfft_basis_kernel(const UnitDesc* __restrict__ units,
                                                            const int4* __restrict__ tiles, int nb) {
  constexpr int N = 32 * E, LE = log2_c(E);
  constexpr bool P2 = (E & (E - 1)) == 0;
  constexpr int NP = N + N / 32;
  extern __shared__ __align__(16) float2 bsm[];
  float2* tw = bsm;           // e^{-i2pi j/N}
  float2* pm = tw + N;        // premodulation per polarity
  float2* pt = pm + 2 * N;    // post-twiddle per kx (nx <= N)
  float2* rb = pt + N;        // [8][NP]
  float2* st = rb + 8 * NP;   // forward: basis rows [line][r][x]; adjoint: coil rows [line][coil][x]
  __shared__ __align__(16) float co[kMaxCoils * kBasisPad];  // (read as float4)
  __shared__ int lrow[kBasisRows], lpol[kBasisRows];
  __shared__ float ldec[kBasisRows];
  const int4 t = tiles[blockIdx.x];
  const UnitDesc& u = units[t.x];
  const int j0 = t.y, nj = t.z;
  const int nx = u.nx, nl = u.n_lines, n_rows = u.n_rows, nc = u.ncoils;
  float2* const ksp = u.kspace;
  float2* const gbuf = u.g;
  const float* __restrict__ exg = u.geo.ex;
  auto stage_rows = [&] {
    constexpr int HN = N / 2;
    const float4* g4 = reinterpret_cast<const float4*>(gbuf);
    float4* h4 = reinterpret_cast<float4*>(st);
    for (int e = threadIdx.x; e < nj * nb * HN; e += 256) {
      const int jl = e / (nb * HN), r = (e / HN) % nb, x2 = e % HN;
      cp_async16(h4 + e, g4 + ((size_t)r * nl + j0 + jl) * HN + x2, 16);
    }
    cp_async_commit();
  };
  grid_begin();
  const bool fill = ADJ || gridDim.x <= kChainTiles;
  if (!fill) grid_wait();
  if (!ADJ && !fill) stage_rows();
  const float2* __restrict__ xf = u.geo.xf;
  for (int k = threadIdx.x; k < N / 2; k += 256) {
    const float2 w = xf[k];
    tw[k] = w;
    tw[k + N / 2] = make_float2(-w.x, -w.y);
  }
  const float inv_n = 1.0f / (float)(N * u.sny);
  for (int k = threadIdx.x; k < 2 * N; k += 256) {
    const float2 v = xf[N / 2 + k];
    pm[k] = ADJ ? make_float2(v.x * inv_n, v.y * inv_n) : v;
  }
  for (int k = threadIdx.x; k < nx; k += 256) {
    const float2 v = xf[N / 2 + 2 * N + k];
    pt[k] = ADJ ? v : make_float2(v.x * inv_n, v.y * inv_n);
  }
  for (int k = threadIdx.x; k < nc * kBasisPad; k += 256) co[k] = u.geo.bco[k];
  if (threadIdx.x < nj) {
    const LineRec& L = u.lines[j0 + threadIdx.x];
    lrow[threadIdx.x] = L.row;
    lpol[threadIdx.x] = L.pol < 0 ? 1 : 0;
    ldec[threadIdx.x] = L.decay;
  }
  if (fill) grid_wait();
  if (!ADJ && fill) stage_rows();
  if (!ADJ) cp_async_wait0();
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ox = N / nx, xs = nx / 2, sxs = ox * xs;
  const double xoff = (ox - 1.0) / 2.0;
  const bool eddy = (u.flags & UF_EDDY) != 0;
  const int kpos = nx - xs;
  const float off = u.geo.coil_off;
  float2* row = rb + warp * NP;
  auto modulation = [&](int pol, float dec, int x) {  // as xfft_warp_kernel's
    float2 md = pm[pol * N + x];
    if (eddy) {
      const double xc = ((double)x - sxs - xoff) / ox;
      double tv = ((double)u.eddy_cx * xc + (double)u.eddy_qx * xc * xc + (double)u.eddy_z) * (double)dec;
      tv -= rint(tv);
      float sn, cs;
      __sincosf(kTwoPiF * (float)tv, &sn, &cs);
      md = cmul(md, make_float2(cs, sn));
    }
    return md;
  };
  for (int q0 = 0; q0 < nc; q0 += ADJ ? kBasisRows : nc) {
    const int nq = ADJ ? min(kBasisRows, nc - q0) : nc;
    const int nr = nj * nq;
    // adjoint: the next row's k-space samples are loaded while the current one transforms
    float2 pre[ADJ ? E : 1];
    auto fetch = [&](int r) {
      const float2* kr = ksp + ((size_t)(q0 + r % nq) * n_rows + lrow[r / nq]) * nx;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int n = lane + 32 * m;
        const int kx = (n < kpos ? n : n - N) + xs;
        pre[ADJ ? m : 0] = kx >= 0 && kx < nx ? kr[kx] : make_float2(0.f, 0.f);
      }
    };
    if (ADJ && warp < nr) fetch(warp);
    for (int r = warp; r < nr; r += 8) {
      const int jl = r / nq, q = q0 + r % nq, pol = lpol[jl];
      const float dec = ldec[jl];
      float2 b[E];
      if (!ADJ) {
        const float4 c0 = *reinterpret_cast<const float4*>(co + q * kBasisPad);
        const float4 c1 = *reinterpret_cast<const float4*>(co + q * kBasisPad + 4);
        const float cf[kBasisPad] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const float2* cr = st + jl * nb * N;
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int x = lane + 32 * m;
          const float ex = __ldg(exg + q * N + x);
          float2 a = fmul2(dup2(cf[0]), cr[x]), last = make_float2(0.f, 0.f);
#pragma unroll
          for (int v = 1; v < kBasisPad - 1; ++v)
            if (v < nb) {
              last = cr[v * N + x];
              a = ffma2(dup2(cf[v]), last, a);
            }
          const float2 g = ffma2(dup2(off), last, fmul2(dup2(ex), a));
          b[P2 ? bitrev_c(m, LE) : m] = cmul(g, modulation(pol, dec, x));
        }
      } else {
        float2 cur[E];
#pragma unroll
        for (int m = 0; m < E; ++m) cur[m] = pre[ADJ ? m : 0];
        if (r + 8 < nr) fetch(r + 8);
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int n = lane + 32 * m;
          const int kx = (n < kpos ? n : n - N) + xs;
          float2 v = make_float2(0.f, 0.f);
          if (kx >= 0 && kx < nx) {
            const float2 p = pt[kx];
            v = cmul(cur[m], make_float2(p.x, -p.y));
          }
          b[P2 ? bitrev_c(m, LE) : m] = v;
        }
      }
      warp_row_fft<E, ADJ>(b, tw, lane);
      const int k2 = __brev(lane) >> 27;
#pragma unroll
      for (int k1 = 0; k1 < E; ++k1) {
        const int k = k1 + E * k2;
        row[k + (k >> 5)] = b[k1];
      }
      __syncwarp();
      if (!ADJ) {
        float2* out = ksp + ((size_t)q * n_rows + lrow[jl]) * nx;
        for (int kx = lane; kx < nx; kx += 32) {
          const int k = kx >= xs ? kx - xs : kx - xs + N;
          out[kx] = cmul(row[k + (k >> 5)], pt[kx]);
        }
      } else {
        float2* gr = st + (size_t)r * N;
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int x = lane + 32 * m;
          const float2 md = modulation(pol, dec, x);
          gr[x] = cmul(row[x + (x >> 5)], make_float2(md.x, -md.y));
        }
      }
      __syncwarp();
    }
    if (ADJ) {
      __syncthreads();
      const float s = u.signal_scale, so = s * off;
      for (int e = threadIdx.x; e < nj * N; e += 256) {
        const int jl = e / N, x = e % N;
        const size_t base = (size_t)(j0 + jl) * N + x, rs = (size_t)nl * N;
        float2 G[kBasisPad - 2], last = q0 > 0 ? gbuf[base + (nb - 1) * rs] : make_float2(0.f, 0.f);
#pragma unroll
        for (int v = 0; v < kBasisPad - 2; ++v)  // past the first 32 coils: on from this thread's own sums
          G[v] = q0 > 0 && v < nb - 1 ? gbuf[base + v * rs] : make_float2(0.f, 0.f);
        const float2* hr = st + (size_t)jl * nq * N + x;
        float2 chain[kCoilChains];
#pragma unroll
        for (int k = 0; k < kCoilChains; ++k) chain[k] = make_float2(0.f, 0.f);
        auto add = [&](int q, float2& l) {
          const float2 h = hr[q * N];
          const float4 c0 = *reinterpret_cast<const float4*>(co + (q0 + q) * kBasisPad);
          const float4 c1 = *reinterpret_cast<const float4*>(co + (q0 + q) * kBasisPad + 4);
          const float cf[kBasisPad] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
          const float ex = s * __ldg(exg + (q0 + q) * N + x);
          const float2 w = fmul2(dup2(ex), h);
          l = ffma2(dup2(fmaf(ex, cf[kBasisPad - 1], so)), h, l);
#pragma unroll
          for (int v = 0; v < kBasisPad - 2; ++v) G[v] = ffma2(dup2(cf[v]), w, G[v]);
        };
        int q = 0;
        for (; q + kCoilChains <= nq; q += kCoilChains)
#pragma unroll
          for (int k = 0; k < kCoilChains; ++k) add(q + k, chain[k]);
#pragma unroll
        for (int k = 0; k < kCoilChains - 1; ++k)
          if (q + k < nq) add(q + k, chain[k]);
        last = fadd2(last, fadd2(fadd2(chain[0], chain[1]), fadd2(chain[2], chain[3])));
#pragma unroll
        for (int v = 0; v < kBasisPad - 2; ++v)
          if (v < nb - 1) gbuf[base + v * rs] = G[v];
        gbuf[base + (nb - 1) * rs] = last;
      }
      __syncthreads();  // before the next coils' rows overwrite these
    }
  }
}

}  // namespace

// ---- plans and launchers ----------------------------------------------------------------------
void append_xtiles(std::vector<XTile>& out, const UnitDesc& u, int unit_index, const LineRec* lines, int dir) {
  const int nl = u.n_lines, nc = u.ncoils;
  const int N = dir == 0 ? u.nx : u.snx;
  const int nq = std::min(nc, 32);
  const int lines_per_tile = std::max(1, 32 / nq);
  for (int pol = 0; pol < 2; ++pol) {
    std::vector<int> group;
    for (int l = 0; l < nl; ++l)
      if ((lines[l].pol < 0 ? 1 : 0) == pol) group.push_back(l);
    for (size_t g0 = 0; g0 < group.size(); g0 += lines_per_tile)
      for (int q0 = 0; q0 < nc; q0 += nq)
        for (int c0 = 0; c0 < N; c0 += 64) {
          XTile t;
          std::memset(&t, 0, sizeof t);
          t.unit = unit_index;
          t.q0 = q0;
          t.nq = std::min(nq, nc - q0);
          t.nl = (int)std::min<size_t>(lines_per_tile, group.size() - g0);
          t.col0 = c0;
          t.pol = pol;
          for (int k = 0; k < t.nl; ++k) t.line[k] = group[g0 + k];
          out.push_back(t);
        }
  }
}

EpiPlan::~EpiPlan() {
  for (void* p : allocs) {
    if (pool_stream)
      cudaFreeAsync(p, pool_stream);
    else
      cudaFree(p);
  }
}

namespace {
// A plan's arrays, gathered on the host and sent up as one allocation and one copy.
struct PlanArrays {
  std::vector<char> blob;
  std::vector<std::pair<void**, size_t>> slots;
  template <class T>
  void add(T** slot, const void* src, size_t bytes) {
    *slot = nullptr;
    if (bytes == 0) return;
    const size_t at = blob.size();
    blob.resize(at + (bytes + 255) / 256 * 256);
    std::memcpy(blob.data() + at, src, bytes);
    slots.emplace_back((void**)slot, at);
  }
  void send(EpiPlan* p, mrsim_context* ctx) {
    if (blob.empty()) return;
    void* d = nullptr;
    p->allocs.reserve(1);
    if (ctx) {
      MRSIM_CUDA(cudaMallocFromPoolAsync(&d, blob.size(), ctx->pool, ctx->stream));
      p->pool_stream = ctx->stream;
      p->allocs.push_back(d);
      MRSIM_CUDA(cudaMemcpyAsync(d, blob.data(), blob.size(), cudaMemcpyHostToDevice, ctx->stream));
    } else {
      MRSIM_CUDA(cudaMalloc(&d, blob.size()));
      p->allocs.push_back(d);
      MRSIM_CUDA(cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice));
      MRSIM_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // the plan runs on streams that do not wait for this one
    }
    for (auto& s : slots) *s.first = (char*)d + s.second;
  }
};
}  // namespace

EpiPlan* epi_plan_create(const UnitDesc* hu, int n, const StaticDesc* hs, int ns, const EpiPlanOptions* opt,
                         mrsim_context* ctx, const HostLines* lines) {
  EpiPlan* p = new EpiPlan();
  PlanArrays arrays;
  try {
    if (opt) p->opt = *opt;
    p->n_units = n;
    p->host_units.assign(hu, hu + n);
    p->host_statics.assign(hs, hs + ns);
    p->n_statics = ns;
    arrays.add(&p->d_statics, hs, sizeof(StaticDesc) * ns);
    for (int i = 0; i < ns; ++i) p->max_static_n = std::max(p->max_static_n, hs[i].snx * hs[i].sny);
    int max_coils = 0;
    for (int i = 0; i < n; ++i) {
      max_coils = std::max(max_coils, hu[i].ncoils);
      p->max_sny = std::max(p->max_sny, hu[i].sny);
      p->max_snx = std::max(p->max_snx, hu[i].snx);
      p->max_nx = std::max(p->max_nx, hu[i].nx);
      p->max_lines = std::max(p->max_lines, hu[i].n_lines);
      if (hu[i].ncomp > kMaxComp) fail("a unit has more than 8 compartments");
      if (hu[i].ncoils > kMaxCoils) fail("more than 64 coils");
    }
    p->max_coils = max_coils;
    for (int i = 0; i < n; ++i)
      p->max_hchunk = std::max(p->max_hchunk, adjoint_chunk_lines(hu[i].ncoils) * hu[i].ncoils);
    int max_comp = 0;
    for (int i = 0; i < n; ++i) max_comp = std::max(max_comp, hu[i].ncomp);
    p->nc = max_comp <= 1 ? 1 : max_comp <= 2 ? 2 : max_comp <= 3 ? 3 : max_comp <= 4 ? 4 : 8;
    p->qg = max_coils <= 1 ? 1 : max_coils <= 2 ? 2 : max_coils <= 4 ? 4 : 8;
    // x-stage as per-row FFTs when every unit has a power-of-two snx with FFT tables
    p->xfft = n > 0 && !p->opt.dft_x;
    for (int i = 0; i < n; ++i) {
      const int N = hu[i].snx;
      const bool pow2 = N >= 8 && N <= kXfftMaxN && (N & (N - 1)) == 0, warp = N % 32 == 0 && N <= 256;
      if (hu[i].geo.xf == nullptr || !(pow2 || warp) || hu[i].nx > N) p->xfft = false;
    }
    if (p->xfft) {
      const int N0 = hu[0].snx;
      p->xfft_e = (N0 % 32 == 0 && N0 <= 256) ? N0 / 32 : 0;
      bool all_warp = true;
      for (int i = 0; i < n; ++i) {
        if (hu[i].snx != N0) p->xfft_e = 0;
        all_warp = all_warp && hu[i].snx % 32 == 0 && hu[i].snx <= 256;
      }
      // every row a warp width but not one width (a batch of 128, 192 and 256): the warp FFT once
      // per width over that width's tiles
      if (p->xfft_e == 0 && all_warp) p->xfft_e = -1;
      // otherwise the shared-memory radix-2 FFT serves, which needs every row length to be a power
      // of two; failing that, the DFT GEMM
      if (p->xfft_e == 0)
        for (int i = 0; i < n; ++i) {
          const int N = hu[i].snx;
          if (!(N >= 8 && N <= kXfftMaxN && (N & (N - 1)) == 0)) p->xfft = false;
        }
    }
    for (int i = 0; i < n; ++i) p->adj_narrow = p->adj_narrow || (hu[i].snx & 1) || ((uintptr_t)hu[i].g & 15);
    auto has_maps = [&](bool maps) {
      for (int i = 0; i < n; ++i)
        if (((hu[i].flags & UF_MAPS) != 0) == maps) return true;
      return false;
    };
    // rows per thread of the fixed-count y-adjoint: the built-in choice, or 2 where 4 would be (the tunable)
    auto adj_ty = [&](bool maps, bool rows, bool basis) {
      const int ty = adjq_rows_v(p->nc, maps, rows);
      return p->opt.adj_rows == 2 && ty == 4 && !(basis && p->adj_narrow) ? 2 : ty;
    };
    auto adj_fits = [&](int nq, bool rows, bool basis) {  // on nq coils or rows, for every kind of unit here
      for (bool maps : {false, true})
        if (has_maps(maps) &&
            yadjoint_q_smem(nq, adj_ty(maps, rows, basis), p->nc, maps, p->max_lines) > kStagedSmem)
          return false;
      return true;
    };
    auto fwd_fits = [&](bool maps, bool basis) {
      return ystage_q_smem(p->nc, maps, p->qg, p->max_sny, basis) <= kStagedSmem;
    };
    // The coil basis (coil_basis, driver.cpp) where every unit has one of the same row count: rings of
    // 6, 7 and 9 or more coils, and of 8 where the class rows have no x-stage (rows past 128 points,
    // the DFT GEMM).  Its 4 to 7 rows replace the coils in both y-stages, whose work per voxel and
    // line is the phase plus two FMAs per row: one series of 32 coils (128 x 128 on 256 x 256, 120
    // units) takes 4.3 ms against 19.3 ms with 32 rows.  The kernels with eight compartments, or four
    // with voxel maps, have no registers for it; the x-stages that expand the rows are the warp FFT
    // and, with every coil in one tile (32), the DFT GEMM.
    {
      const bool gemm = !p->xfft, warp = p->xfft && p->xfft_e != 0;
      const bool cls8 = p->xfft && p->xfft_e >= 1 && p->xfft_e <= 4;
      int nb = n > 0 && !p->opt.no_classes && !p->opt.no_basis && (gemm || warp) && p->nc <= 4 ? hu[0].geo.nbas : 0;
      bool all8 = true, any_maps = false;
      for (int i = 0; i < n && nb; ++i) {
        const UnitDesc& u = hu[i];
        all8 = all8 && u.ncoils == 8;
        any_maps = any_maps || (u.flags & UF_MAPS) != 0;
        if (u.geo.nbas != nb || (gemm && u.ncoils > 32) || (warp && ((uintptr_t)u.g & 15)) ||
            (long long)u.ncoils * u.n_lines * u.snx >= (1LL << 31))
          nb = 0;
      }
      if ((all8 && cls8) || (any_maps && p->nc > 3)) nb = 0;
      if (nb && !(adj_fits(nb, true, true) && (!has_maps(false) || fwd_fits(false, true)) && (!any_maps || fwd_fits(true, true))))
        nb = 0;
      p->basis_nb = nb;
    }
    {  // the kernels read the rows a y-stage runs on as geo.ncls rows of geo.eyc and a constant one
      std::vector<UnitDesc> du(hu, hu + n);
      if (p->basis_nb)
        for (UnitDesc& u : du) {
          u.geo.ncls = u.geo.nbas - 1;
          u.geo.eyc = u.geo.bas;
        }
      arrays.add(&p->d_units, du.data(), sizeof(UnitDesc) * n);
    }
    // the staged-input forward serves a pass when every unit has snx % 4 == 0 and 16-byte aligned
    // input planes (cooperative 16-byte copies), and on basis rows also when not (4-byte copies; 12
    // coils, voxel maps, rows of 150: 0.44 ms against 0.87 ms with the per-thread loads)
    auto al16 = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
    for (int pass = 0; pass < 2; ++pass) {
      bool ok = true, wide = true;
      for (int i = 0; i < n; ++i) {
        const UnitDesc& u = hu[i];
        if (((u.flags & UF_MAPS) != 0) != (pass == 1)) continue;
        wide = wide && (u.snx % 4) == 0 && al16(u.phase) && al16(u.fmap) && al16(u.comp) && al16(u.t2map) &&
             al16(u.timap) && al16(u.log_amp) && (u.ncomp <= 1 || u.comp_stride % 4 == 0) &&
             (u.ncomp <= 1 || (u.map_stride % 4) == 0);
      }
      // eight coils with voxel maps (four or more compartments) or eight compartments take more
      // registers than the 256-thread CTA leaves: those shapes keep the per-thread-load kernel
      if (p->qg == 8 && (p->nc == 8 || (pass == 1 && p->nc >= 4))) ok = false;
      if (!wide && !p->basis_nb) ok = false;
      if (!fwd_fits(pass == 1, p->basis_nb > 0)) ok = false;
      p->fwdq[pass] = ok;
      p->fwd_narrow[pass] = !wide;
      // coil classes: every unit with the same 8 coils in 5 classes (the ring) -> 6 accumulators
      bool cl = ok && n > 0 && p->qg == 8 && (pass == 0 || p->nc <= 3);
      for (int i = 0; i < n && cl; ++i) {
        const UnitDesc& u = hu[i];
        if (((u.flags & UF_MAPS) != 0) != (pass == 1)) continue;
        cl = u.ncoils == 8 && u.geo.ncls == 5 && u.geo.coil_off != 0.f && u.geo.cls && u.geo.eyc;
      }
      p->fwd_nv[pass] = p->basis_nb ? p->basis_nb : (cl && !p->opt.no_classes) ? 6 : 0;
    }
    // coil classes through the forward x-stage: every unit's y-stage runs in class mode and the
    // rows have at most 128 points
    {
      bool fc = p->xfft && p->xfft_e >= 1 && p->xfft_e <= 4 && n > 0;
      for (int pass = 0; pass < 2 && fc; ++pass) {
        bool any = false;
        for (int i = 0; i < n && !any; ++i) any = ((hu[i].flags & UF_MAPS) != 0) == (pass == 1);
        if (any && p->fwd_nv[pass] != 6) fc = false;
      }
      p->fwd_cls = fc || p->basis_nb > 0;
    }
    for (int pass = 0; pass < 2; ++pass) {
      auto make_tiles = [&](int lines, int cols) {
        std::vector<int4> t;
        p->y_start[pass].assign(n + 1, 0);
        for (int i = 0; i < n; ++i) {
          p->y_start[pass][i] = (int)t.size();
          if (((hu[i].flags & UF_MAPS) != 0) != (pass == 1)) continue;
          for (int l = 0; l < hu[i].n_lines; l += lines)
            for (int x0 = 0; x0 < hu[i].snx; x0 += cols)
              for (int q0 = 0; q0 < (p->basis_nb ? 1 : hu[i].ncoils); q0 += p->qg) t.push_back(make_int4(i, l, x0, q0));
        }
        p->y_start[pass][n] = (int)t.size();
        return t;
      };
      std::vector<int4> tiles = make_tiles(p->fwdq[pass] ? 8 : kT, 128);
      const bool small = p->fwdq[pass] && pass == 0 && !p->fwd_narrow[pass] && (int)tiles.size() <= kChainTiles;
      p->fwd_chain[pass] = small;
      // (not where the full kernel expands classes to coils)
      if (small && !(p->fwd_nv[pass] && !p->fwd_cls)) {
        const int g = thin_groups((long long)tiles.size(), 8);
        if (g && ystage_thin_smem(g, p->nc, p->qg, p->max_sny) <= kStagedSmem) {
          p->fwd_thin[pass] = g;
          tiles = make_tiles(4 * g, kThinCols);
        }
      }
      p->n_ytiles[pass] = (int)tiles.size();
      arrays.add(&p->d_ytiles[pass], tiles.data(), sizeof(int4) * tiles.size());
    }
    // x-stage tiles of 32 rows, or where those would not fill the chip (two blocks per SM) of one line of
    // every coil, or one row per warp
    long long x_rows = 0;
    for (int i = 0; i < n; ++i) x_rows += (long long)hu[i].ncoils * hu[i].n_lines;
    const bool few = x_rows < 296 * 32;
    if (p->xfft && p->basis_nb) {
      // tiles of a few lines x every coil: by unit, or with mixed widths ordered by width
      std::vector<int4> ct;
      auto unit_tiles = [&](int i) {
        const int step = few ? 1 : basis_lines(hu[i].ncoils);
        p->basis_rows = std::max(p->basis_rows, step * std::min(hu[i].ncoils, kBasisRows));
        p->basis_lines = std::max(p->basis_lines, step);
        for (int j0 = 0; j0 < hu[i].n_lines; j0 += step)
          ct.push_back(make_int4(i, j0, std::min(step, hu[i].n_lines - j0), 0));
      };
      if (p->xfft_e > 0) p->c_start.assign(n + 1, 0);
      for (int E = 1; E <= 8; ++E) {
        p->ce_first[E] = (int)ct.size();
        for (int i = 0; i < n; ++i) {
          if (hu[i].snx != 32 * E) continue;
          if (p->xfft_e > 0) p->c_start[i] = (int)ct.size();
          unit_tiles(i);
        }
        p->ce_count[E] = (int)ct.size() - p->ce_first[E];
      }
      if (p->xfft_e > 0) p->c_start[n] = (int)ct.size();
      p->n_ctiles = (int)ct.size();
      arrays.add(&p->d_ctiles, ct.data(), sizeof(int4) * ct.size());
    } else if (p->xfft && p->xfft_e < 0) {
      // one list ordered by width, no per-unit ranges (such a plan runs whole)
      std::vector<int4> ft;
      for (int E = 1; E <= 8; ++E) {
        p->fe_first[E] = (int)ft.size();
        for (int i = 0; i < n; ++i) {
          if (hu[i].snx != 32 * E) continue;
          const int rows = hu[i].ncoils * hu[i].n_lines;
          for (int r0 = 0; r0 < rows; r0 += 32) ft.push_back(make_int4(i, r0, std::min(32, rows - r0), 0));
        }
        p->fe_count[E] = (int)ft.size() - p->fe_first[E];
      }
      p->f_start.clear();
      p->n_ftiles = (int)ft.size();
      arrays.add(&p->d_ftiles, ft.data(), sizeof(int4) * ft.size());
    } else if (p->xfft) {
      std::vector<int4> ft;
      p->f_start.assign(n + 1, 0);
      for (int i = 0; i < n; ++i) {
        p->f_start[i] = (int)ft.size();
        const int rows = hu[i].ncoils * hu[i].n_lines;
        const int per = p->xfft_e ? (few ? 8 : 32) : std::min(256, kXfftMaxN / hu[i].snx);
        for (int r0 = 0; r0 < rows; r0 += per) ft.push_back(make_int4(i, r0, std::min(per, rows - r0), 0));
      }
      p->f_start[n] = (int)ft.size();
      p->n_ftiles = (int)ft.size();
      arrays.add(&p->d_ftiles, ft.data(), sizeof(int4) * ft.size());
    }
    // x-stage GEMM tiles, from host copies of the line tables (one readback per table that has none)
    std::map<const LineRec*, std::vector<LineRec>> read;
    HostLines known = lines ? *lines : HostLines();
    for (int dir = 0; dir < 2 && !p->xfft; ++dir) {
      std::vector<XTile> xt;
      p->g_start[dir].assign(n + 1, 0);
      for (int i = 0; i < n; ++i) {
        p->g_start[dir][i] = (int)xt.size();
        const int nl = hu[i].n_lines;
        if (nl == 0) continue;
        const LineRec*& table = known[hu[i].lines];
        if (!table) {
          if (!ctx) fail("a plan needs its units' line tables");
          std::vector<LineRec>& L = read[hu[i].lines];
          L.resize(nl);
          MRSIM_CUDA(cudaMemcpyAsync(L.data(), hu[i].lines, sizeof(LineRec) * nl, cudaMemcpyDeviceToHost, ctx->stream));
          MRSIM_CUDA(cudaStreamSynchronize(ctx->stream));
          table = L.data();
        }
        append_xtiles(xt, hu[i], i, table, dir);
      }
      p->g_start[dir][n] = (int)xt.size();
      p->n_gtiles[dir] = (int)xt.size();
      arrays.add(&p->d_gtiles[dir], xt.data(), sizeof(XTile) * xt.size());
    }
    // the fixed-coil-count y-adjoint serves a pass when every unit has the same coil count (1, 2,
    // 4 or 8), an even snx and 16-byte aligned h rows (cooperative 16-byte copies), and on basis rows
    // any of them (8-byte copies where some row is not so)
    int nq_all = n > 0 ? hu[0].ncoils : 0;
    for (int i = 0; i < n; ++i)
      if (hu[i].ncoils != nq_all || (long long)hu[i].ncoils * hu[i].n_lines * hu[i].snx >= (1LL << 31)) nq_all = 0;
    if (p->adj_narrow) nq_all = 0;
    if (nq_all != 1 && nq_all != 2 && nq_all != 4 && nq_all != 8) nq_all = 0;
    const bool coil_rows_fit = nq_all == 0 || adj_fits(nq_all, false, false);
    // coil classes in the adjoint: every unit has the 8-coil ring (5 classes + offset), rows of
    // at most 128 points in the warp FFT, and the fixed-count y-adjoint for its shape
    {
      bool cl = n > 0 && p->xfft && p->xfft_e >= 1 && p->xfft_e <= 4 && p->nc <= 4 && nq_all == 8;
      for (int i = 0; i < n && cl; ++i) {
        const UnitDesc& u = hu[i];
        cl = u.ncoils == 8 && u.geo.ncls == 5 && u.geo.coil_off != 0.f && u.geo.cls && u.geo.eyc;
      }
      if (cl && !adj_fits(6, true, false)) cl = false;
      p->adj_cls = (cl && !p->opt.no_classes) || p->basis_nb > 0;
      if (!coil_rows_fit) nq_all = 0;
    }
    for (int pass = 0; pass < 4; ++pass) {
      bool maps = pass & 1, grads = pass & 2;
      p->adjq[pass] = p->basis_nb ? p->basis_nb : p->adj_cls ? 6 : (maps && p->nc == 8) ? 0 : nq_all;
      const int ty = adj_ty(maps, p->adj_cls, p->basis_nb > 0);
      p->adj_ty[pass] = ty;
      auto make_tiles = [&](int rows, int cols) {
        std::vector<int4> t;
        p->a_start[pass].assign(n + 1, 0);
        for (int i = 0; i < n; ++i) {
          p->a_start[pass][i] = (int)t.size();
          bool um = (hu[i].flags & UF_MAPS) != 0;
          bool ug = (hu[i].flags & (UF_WANT_FMAP_GRAD | UF_WANT_R2_GRAD)) != 0;
          if (um != maps || ug != grads) continue;
          for (int y0 = 0; y0 < hu[i].sny; y0 += rows)
            for (int x0 = 0; x0 < hu[i].snx; x0 += cols) t.push_back(make_int4(i, y0, x0, 0));
        }
        p->a_start[pass][n] = (int)t.size();
        return t;
      };
      const int full = p->adjq[pass] ? 2 * ty : kTY;
      std::vector<int4> yt = make_tiles(full, 128);
      const bool small = p->adjq[pass] && !maps && !p->adj_narrow && ty == adjq_rows_v(p->nc, maps, p->adj_cls) &&
                         (int)yt.size() <= kChainTiles;
      p->adj_chain[pass] = small;
      if (small) {
        const int g = thin_groups((long long)yt.size(), full);
        if (g && yadjoint_thin_smem(g, p->adjq[pass], p->nc, p->max_lines) <= kStagedSmem) {
          p->adj_thin[pass] = g;
          yt = make_tiles(4 * g, kThinCols);
        }
      }
      p->n_atiles[pass] = (int)yt.size();
      arrays.add(&p->d_atiles[pass], yt.data(), sizeof(int4) * yt.size());
    }
    if (!p->basis_nb && (p->adj_cls || p->fwd_cls)) {  // the class x-stage tiles: 4 lines x the 8 coils
      std::vector<int4> ct;
      p->c_start.assign(n + 1, 0);
      for (int i = 0; i < n; ++i) {
        p->c_start[i] = (int)ct.size();
        for (int j0 = 0, step = few ? 1 : 4; j0 < hu[i].n_lines; j0 += step)
          ct.push_back(make_int4(i, j0, std::min(step, hu[i].n_lines - j0), 0));
      }
      p->c_start[n] = (int)ct.size();
      p->n_ctiles = (int)ct.size();
      arrays.add(&p->d_ctiles, ct.data(), sizeof(int4) * ct.size());
    }
    arrays.send(p, ctx);
  } catch (...) {
    delete p;
    throw;
  }
  return p;
}

void epi_plan_statics(const EpiPlan* p, cudaStream_t st, int u0, int u1) {
  if (u1 < 0) u1 = p->n_statics;
  if (u0 < 0 || u0 > u1 || u1 > p->n_statics) fail("unit range outside the plan");
  if (u1 == u0) return;
  // a few voxels per thread: eight blocks per unit, or more where the units are few
  const int per_unit = std::max(8, 592 / (u1 - u0));
  launch_chained(statics_kernel, dim3(std::min(per_unit, (p->max_static_n + 255) / 256), u1 - u0), 0, st,
                 u1 - u0 <= 148, (const StaticDesc*)(p->d_statics + u0));
}

void epi_plan_forward(const EpiPlan* p, cudaStream_t st, int u0, int u1) {
  epi_plan_forward_ystage(p, st, u0, u1);
  epi_plan_forward_xstage(p, st, u0, u1);
}

void epi_plan_adjoint(const EpiPlan* p, cudaStream_t st, int u0, int u1) {
  epi_plan_adjoint_xstage(p, st, u0, u1);
  epi_plan_adjoint_ystage(p, st, u0, u1);
}

namespace {
void launch_xstage(const EpiPlan* p, cudaStream_t st, int u0, int u1, bool adj) {
  if (p->basis_nb && p->xfft) {
    if (p->xfft_e < 0 && !(u0 == 0 && (u1 < 0 || u1 == p->n_units)))
      fail("a plan of mixed row widths runs its units whole");
    const TileRange R = tile_range(p->c_start, p->n_ctiles, u0, u1);
    for (int E = 1; E <= 8; ++E) {
      if (p->ce_count[E] == 0) continue;
      // one width: the tiles of the unit range; mixed widths: the width's whole list
      const int first = p->xfft_e > 0 ? R.t0 : p->ce_first[E], count = p->xfft_e > 0 ? R.n : p->ce_count[E];
      if (count == 0) continue;
      const int4* tiles = p->d_ctiles + first;
      const size_t sm = sizeof(float2) * basis_smem(E, adj ? p->basis_rows : p->basis_lines * p->basis_nb);
#define MRSIM_XB(EV, ADJ)                                                                 \
  case EV: {                                                                              \
    auto k = xfft_basis_kernel<EV, ADJ>;                                                  \
    set_smem(k, sm);                                                                      \
    launch_chained(k, dim3((unsigned)count), sm, st, count <= kChainTiles, p->d_units, tiles, p->basis_nb);  \
    break;                                                                                \
  }
#define MRSIM_XBA(ADJ) MRSIM_XB(1, ADJ) MRSIM_XB(2, ADJ) MRSIM_XB(3, ADJ) MRSIM_XB(4, ADJ) \
  MRSIM_XB(5, ADJ) MRSIM_XB(6, ADJ) MRSIM_XB(7, ADJ) MRSIM_XB(8, ADJ)
      if (adj) {
        switch (E) { MRSIM_XBA(true) }
      } else {
        switch (E) { MRSIM_XBA(false) }
      }
#undef MRSIM_XBA
#undef MRSIM_XB
      MRSIM_CUDA(cudaGetLastError());
    }
    return;
  }
  if (!p->basis_nb && ((adj && p->adj_cls) || (!adj && p->fwd_cls))) {
    const TileRange R = tile_range(p->c_start, p->n_ctiles, u0, u1);
    if (R.n == 0) return;
    const int4* tiles = p->d_ctiles + R.t0;
    const unsigned g = (unsigned)R.n;
#define MRSIM_XC(ADJ)                                                                             \
  switch (p->xfft_e) {                                                                            \
    case 1: launch_chained(xfft_warp_kernel<1, ADJ, true>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;          \
    case 2: launch_chained(xfft_warp_kernel<2, ADJ, true>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;          \
    case 3: launch_chained(xfft_warp_kernel<3, ADJ, true>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;          \
    default: launch_chained(xfft_warp_kernel<4, ADJ, true>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
  }
    if (adj) {
      MRSIM_XC(true)
    } else {
      MRSIM_XC(false)
    }
#undef MRSIM_XC
    MRSIM_CUDA(cudaGetLastError());
    return;
  }
  if (p->xfft && p->xfft_e < 0) {
    if (!(u0 == 0 && (u1 < 0 || u1 == p->n_units))) fail("a plan of mixed row widths runs its units whole");
    for (int E = 1; E <= 8; ++E) {
      if (p->fe_count[E] == 0) continue;
      const int4* tiles = p->d_ftiles + p->fe_first[E];
      const unsigned g = (unsigned)p->fe_count[E];
#define MRSIM_XE(ADJ)                                                                               \
  switch (E) {                                                                                      \
    case 1: launch_chained(xfft_warp_kernel<1, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    case 2: launch_chained(xfft_warp_kernel<2, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    case 3: launch_chained(xfft_warp_kernel<3, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    case 4: launch_chained(xfft_warp_kernel<4, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    case 5: launch_chained(xfft_warp_kernel<5, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    case 6: launch_chained(xfft_warp_kernel<6, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    case 7: launch_chained(xfft_warp_kernel<7, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;           \
    default: launch_chained(xfft_warp_kernel<8, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;          \
  }
      if (adj) {
        MRSIM_XE(true)
      } else {
        MRSIM_XE(false)
      }
#undef MRSIM_XE
      MRSIM_CUDA(cudaGetLastError());
    }
    return;
  }
  if (p->xfft) {
    const TileRange R = tile_range(p->f_start, p->n_ftiles, u0, u1);
    if (R.n == 0) return;
    const int4* tiles = p->d_ftiles + R.t0;
    const unsigned g = (unsigned)R.n;
#define MRSIM_XF(ADJ)                                                                             \
  switch (p->xfft_e) {                                                                            \
    case 1: launch_chained(xfft_warp_kernel<1, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 2: launch_chained(xfft_warp_kernel<2, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 3: launch_chained(xfft_warp_kernel<3, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 4: launch_chained(xfft_warp_kernel<4, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 5: launch_chained(xfft_warp_kernel<5, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 6: launch_chained(xfft_warp_kernel<6, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 7: launch_chained(xfft_warp_kernel<7, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    case 8: launch_chained(xfft_warp_kernel<8, ADJ, false>, dim3(g), 0, st, g <= kChainTiles, p->d_units, tiles); break;         \
    default: xfft_kernel<ADJ><<<g, 256, 0, st>>>(p->d_units, tiles);                              \
  }
    if (adj) {
      MRSIM_XF(true)
    } else {
      MRSIM_XF(false)
    }
#undef MRSIM_XF
    MRSIM_CUDA(cudaGetLastError());
    return;
  }
  const int dir = adj ? 1 : 0;
  const TileRange R = tile_range(p->g_start[dir], p->n_gtiles[dir], u0, u1);
  if (R.n == 0) return;
  const XTile* tiles = (const XTile*)p->d_gtiles[dir] + R.t0;
  if (adj)
    xgemm_kernel<true><<<(unsigned)R.n, 256, 0, st>>>(p->d_units, tiles, p->basis_nb);
  else
    xgemm_kernel<false><<<(unsigned)R.n, 256, 0, st>>>(p->d_units, tiles, p->basis_nb);
  MRSIM_CUDA(cudaGetLastError());
}
}  // namespace

void epi_plan_forward_xstage(const EpiPlan* p, cudaStream_t st, int u0, int u1) { launch_xstage(p, st, u0, u1, false); }

void epi_plan_adjoint_xstage(const EpiPlan* p, cudaStream_t st, int u0, int u1) { launch_xstage(p, st, u0, u1, true); }

}  // namespace mrsim
