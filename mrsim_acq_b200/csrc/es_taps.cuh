// es_taps.cuh — the exponential-of-semicircle taps of a NUFFT point (`nufft.rs:48-108`).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace mrsim {
namespace {

__device__ __forceinline__ float es_exp(float x) { return __expf(x); }
__device__ __forceinline__ double es_exp(double x) { return exp(x); }

constexpr int kWMax = 16;

// First fine cell of coordinate u (period n) on a fine grid of nf = 2n cells, and its fine position p.
// A coordinate with no position on the ring (p is NaN: u, or 2u, is not finite) starts at cell 0, so
// that every cell formed from the origin is one of the grid's; es_taps gives it taps of zero.
__device__ __forceinline__ int es_origin(double u, int nf, double half, double& p) {
  p = fmod(2.0 * u, (double)nf);
  if (p < 0.0) p += nf;
  return p >= 0.0 ? (int)floor(p - half) + 1 : 0;
}

// First fine cell and the w taps of coordinate u (all zero where u has no position).
template <class R>
__device__ __forceinline__ int es_taps(double u, int nf, int w, R beta, R* k) {
  const double half = 0.5 * w;
  double p;
  const int m0 = es_origin(u, nf, half, p);
  const R ih = (R)(1.0 / half);
#pragma unroll
  for (int i = 0; i < kWMax; ++i) {
    if (i >= w) break;
    const R z = (R)((double)(m0 + i) - p) * ih;
    k[i] = fabs(z) < (R)1 ? es_exp(beta * (sqrt((R)1 - z * z) - (R)1)) : (R)0;
  }
  return m0;
}

}  // namespace
}  // namespace mrsim
