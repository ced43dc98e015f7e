// hermitian_solve.cuh — one CTA solves a dense complex system [H | B] in place (n x (n + nrhs),
// row-major, FP64) by Gaussian elimination with partial pivoting, every right-hand side at once
// (`solve_hermitian`, kspace.rs:1455-1491).  The pivots depend on H alone, so each column of B
// goes through the reference's sequence of operations for that right-hand side; the products and
// sums use the non-contracting FP64 intrinsics, so every value rounds as the reference's separate
// multiply and add do, whatever contraction the including file is compiled with.
#pragma once

#include <cuda_runtime.h>

namespace mrsim {

struct HsCd {
  double re, im;
};
__device__ __forceinline__ HsCd hs_mul(HsCd a, HsCd b) {
  return {__dsub_rn(__dmul_rn(a.re, b.re), __dmul_rn(a.im, b.im)),
          __dadd_rn(__dmul_rn(a.re, b.im), __dmul_rn(a.im, b.re))};
}
__device__ __forceinline__ double hs_abs(double2 h) {
  return __dsqrt_rn(__dadd_rn(__dmul_rn(h.x, h.x), __dmul_rn(h.y, h.y)));
}
__device__ __forceinline__ HsCd hs_recip(HsCd d) {
  const double m2 = __dadd_rn(__dmul_rn(d.re, d.re), __dmul_rn(d.im, d.im));
  if (m2 < 1e-18) return {0.0, 0.0};
  return {__ddiv_rn(d.re, m2), __ddiv_rn(-d.im, m2)};
}

// W: [n][n + nrhs] in global memory; fre/fim: n doubles each; xs: nrhs * 2n doubles (solution
// scratch); out: [nrhs][n] complex f32.  red_v / red_i: shared arrays of an
// entry per warp.  W and the scratch may be in shared memory.  blockDim.x is a multiple of 32.  Every
// thread of the block calls it.
__device__ inline void hermitian_solve_block(double2* W, int n, int nrhs, double* fre, double* fim, double* xs,
                                             float2* out, double* red_v, int* red_i) {
  const int cols = n + nrhs;
  for (int col = 0; col < n; ++col) {
    // pivot: the first row of largest |h[r][col]| among r >= col (the reference keeps `col`
    // unless a later row is strictly larger)
    double best = -1.0;
    int bi = col;
    for (int r = col + (int)threadIdx.x; r < n; r += blockDim.x) {
      const double m = hs_abs(W[(size_t)r * cols + col]);
      if (m > best) {
        best = m;
        bi = r;
      }
    }
    // (largest value, then lowest row, in any order of comparison)
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
      const double o = __shfl_xor_sync(0xffffffffu, best, h);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, h);
      if (o > best || (o == best && oi < bi)) {
        best = o;
        bi = oi;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      red_v[threadIdx.x >> 5] = best;
      red_i[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double b = red_v[0];
      int p = red_i[0];
      for (int t = 1; t < (int)blockDim.x / 32; ++t)
        if (red_v[t] > b || (red_v[t] == b && red_i[t] < p)) {
          b = red_v[t];
          p = red_i[t];
        }
      if (!(b > hs_abs(W[(size_t)col * cols + col]))) p = col;
      red_i[0] = p;
    }
    __syncthreads();
    const int piv = red_i[0];
    if (piv != col)
      for (int c = threadIdx.x; c < cols; c += blockDim.x) {
        const double2 a = W[(size_t)col * cols + c];
        W[(size_t)col * cols + c] = W[(size_t)piv * cols + c];
        W[(size_t)piv * cols + c] = a;
      }
    __syncthreads();
    const double2 dd = W[(size_t)col * cols + col];
    const HsCd dinv = hs_recip({dd.x, dd.y});
    for (int r = col + 1 + (int)threadIdx.x; r < n; r += blockDim.x) {
      const double2 h = W[(size_t)r * cols + col];
      const HsCd f = hs_mul({h.x, h.y}, dinv);
      fre[r] = f.re;
      fim[r] = f.im;
    }
    __syncthreads();
    // a warp per row, lanes along it
    for (int r = col + 1 + (int)(threadIdx.x >> 5); r < n; r += blockDim.x >> 5) {
      const HsCd f = {fre[r], fim[r]};
      for (int c = col + (int)(threadIdx.x & 31); c < cols; c += 32) {
        const double2 p = W[(size_t)col * cols + c];
        const HsCd s = hs_mul(f, {p.x, p.y});
        double2 h = W[(size_t)r * cols + c];
        h.x = __dsub_rn(h.x, s.re);
        h.y = __dsub_rn(h.y, s.im);
        W[(size_t)r * cols + c] = h;
      }
    }
    __syncthreads();
  }
  // back substitution, one warp per right-hand side: the lanes form 32 products at a time, and every
  // lane subtracts them in the reference's order (column by column)
  const int lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < nrhs; q += blockDim.x >> 5) {
    double* xre = xs + (size_t)q * 2 * n;
    double* xim = xre + n;
    for (int col = n - 1; col >= 0; --col) {
      const double2 b = W[(size_t)col * cols + n + q];
      HsCd s = {b.x, b.y};
      for (int c0 = col + 1; c0 < n; c0 += 32) {
        HsCd t = {0.0, 0.0};
        if (c0 + lane < n) {
          const double2 h = W[(size_t)col * cols + c0 + lane];
          t = hs_mul({h.x, h.y}, {xre[c0 + lane], xim[c0 + lane]});
        }
        const int m = n - c0 < 32 ? n - c0 : 32;
        for (int l = 0; l < m; ++l) {
          s.re = __dsub_rn(s.re, __shfl_sync(0xffffffffu, t.re, l));
          s.im = __dsub_rn(s.im, __shfl_sync(0xffffffffu, t.im, l));
        }
      }
      const double2 d = W[(size_t)col * cols + col];
      const HsCd x = hs_mul(s, hs_recip({d.x, d.y}));
      if (lane == 0) {
        xre[col] = x.re;
        xim[col] = x.im;
      }
      __syncwarp();
    }
    for (int f = lane; f < n; f += 32) out[(size_t)q * n + f] = make_float2((float)xre[f], (float)xim[f]);
  }
}

}  // namespace mrsim
