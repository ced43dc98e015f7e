// row_fft.h — the transform of a row of N = 32 E points by one warp, in registers.
#pragma once

#include <cuda_runtime.h>

// Template flags select whole code paths; the paths an instance does not take leave loops the front end
// reports as unreachable.
#pragma nv_diag_suppress 128

namespace mrsim {

namespace {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

__host__ __device__ constexpr int bitrev_c(int v, int bits) {
  int r = 0;
  for (int b = 0; b < bits; ++b) r |= ((v >> b) & 1) << (bits - 1 - b);
  return r;
}
__host__ __device__ constexpr int log2_c(int v) { return v <= 1 ? 0 : 1 + log2_c(v / 2); }

// The transform of one row held by a warp: in, b[bitrev(m)] (E a power of two; else b[m]) is
// x[lane + 32 m]; out, b[k1] is X[k1 + E bitrev5(lane)].  tw: e^{-i2pi j/N} in shared memory; LOW: tw[N + j]
// is what rounding took from tw[j], and the products take both.
template <int E, bool ADJ, bool LOW = false>
__device__ __forceinline__ void warp_row_fft(float2 (&b)[E], const float2* tw, int lane) {
  constexpr int N = 32 * E;
  constexpr bool P2 = (E & (E - 1)) == 0;
  // v (w + l)
  auto cmul2 = [](float2 v, float2 w, float2 l) {
    const float2 c = make_float2(fmaf(v.x, l.x, -v.y * l.y), fmaf(v.x, l.y, v.y * l.x));
    return make_float2(fmaf(v.x, w.x, fmaf(-v.y, w.y, c.x)), fmaf(v.x, w.y, fmaf(v.y, w.x, c.y)));
  };
  // W(j) = e^{sigma i2pi j/N}: sigma = +1 forward, -1 adjoint
  auto W = [&](int j) {
    const float2 w = tw[j];
    return ADJ ? w : make_float2(w.x, -w.y);
  };
  auto times = [&](float2 v, int j) { return LOW ? cmul2(v, W(j), W(N + j)) : cmul(v, W(j)); };
  // E-point DFT of the registers: decimation in time from bit-reversed order, or for E not a
  // power of two the direct sum Y[k1] = sum_m b[m] W^{32 (m k1 mod E)}
  if (!P2) {
    float2 y[E];
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) {
      y[k1] = b[0];
#pragma unroll
      for (int m = 1; m < E; ++m) {
        const float2 v = (m * k1) % E == 0 ? b[m] : times(b[m], 32 * ((m * k1) % E));
        y[k1] = make_float2(y[k1].x + v.x, y[k1].y + v.y);
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) b[k1] = y[k1];
  }
#pragma unroll
  for (int len = 2; len <= (P2 ? E : 1); len <<= 1) {
#pragma unroll
    for (int i = 0; i < E; i += len) {
#pragma unroll
      for (int p = 0; p < len / 2; ++p) {
        float2 v = b[i + p + len / 2];
        const int j = p * (E / len) * 32;
        if (4 * j == N)  // W(N/4) = sigma i exactly
          v = ADJ ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
        else if (p != 0)
          v = times(v, j);
        const float2 a = b[i + p];
        b[i + p] = make_float2(a.x + v.x, a.y + v.y);
        b[i + p + len / 2] = make_float2(a.x - v.x, a.y - v.y);
      }
    }
  }
#pragma unroll
  for (int k1 = 1; k1 < E; ++k1) b[k1] = times(b[k1], lane * k1);
  // 32-point DFTs across the lanes: radix-2 decimation in frequency.  The last two stages'
  // twiddles are exact: 1 at h = 1, and 1 or W(N/4) = sigma i (a swap and a sign) at h = 2.
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
    const float sg = up ? -1.f : 1.f;
    const float2 w = h >= 4 && up ? W((lane & (h - 1)) * (N / (2 * h))) : make_float2(1.f, 0.f);
    const float2 l = LOW && h >= 4 && up ? W(N + (lane & (h - 1)) * (N / (2 * h))) : make_float2(0.f, 0.f);
    const bool quarter = h == 2 && up && (lane & 1);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) {
      const float ox_ = __shfl_xor_sync(0xffffffffu, b[k1].x, h);
      const float oy_ = __shfl_xor_sync(0xffffffffu, b[k1].y, h);
      const float2 v = make_float2(fmaf(sg, b[k1].x, ox_), fmaf(sg, b[k1].y, oy_));
      if (h >= 4)
        b[k1] = LOW ? cmul2(v, w, l) : cmul(v, w);
      else if (h == 2)  // times sigma i: -i for the adjoint (e^{-i pi/2}), +i for the forward
        b[k1] = quarter ? (ADJ ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x)) : v;
      else
        b[k1] = v;
    }
  }
}

}  // namespace

}  // namespace mrsim
