// spiral_iter.cu — the iterations of the spiral reconstruction (grid_recon.rs:178-275) as one launch:
// the Chebyshev semi-iteration of a batch of images, and the power iteration for lambda_hi, FP64.
//
// Each step applies Q A^H W A Q, the Toeplitz convolution of spiral_recon.cu, to an n x n image.  As
// separate kernels a step is 18 launches that pass a 2n x 2n grid through memory a dozen times (FFT
// lines of 8 warps, five launches per projection), and the power iteration's up to 1000 steps wait
// for the host in each: 385 of the 605 ms of a 64 x 64 x 48 stack-of-spirals volume.  Here an image
// stays in shared memory for all its steps.  Of the padded grid only the n rows that are ever nonzero
// exist, as rows of 2n spectrum values, so a step is
//   R   row:     inverse FFT_n of the projected result, the update, zero-padded FFT_2n
//   C   column:  zero-padded FFT_2n down the n rows, times the circulant's transform, inverse FFT_2n
//   R'  row:     inverse FFT_2n, crop, FFT_n
//   C'  column:  FFT_n, the band, inverse FFT_n
// with a barrier after each.  A warp transforms a line in registers (E points a lane, then radix-2
// stages by shuffle); spectra keep the order the transform leaves them in (slot lane + 32 k1 holds
// frequency k1 + E bitrev5(lane)), the tables are permuted to it once, and the inverse undoes the
// forward's steps, so no line is ever reordered.  Rows are padded by one value: lanes that read a
// column of 16-byte values then meet no bank twice.  Q is applied to the first vector only: every
// later one is a combination of projected ones.
//
// A cluster of C blocks holds one image, n / C rows each; column lines cross the blocks through
// distributed shared memory.  C = 1 holds n <= 64 (198 KB with the direction's rows) and fills the
// chip from the batch; 96 and 128 need 2 and 4.  The power iteration has one image, so it takes 8
// blocks: its steps are a chain, and eight SMs shorten each.  Bound by shared memory (96 % of its cycles
// while the blocks run, FP64 pipe 25 to 40 %; about 2.2 MFLOP a step at n = 64) and, in the power
// iteration, by the latency of its exchanges (no pipe above 2 %).  Measured at n = 64: 576 images x 80
// steps 14.8 ms (6.8 of about 37 TFLOP/s, 0.18; before 125 ms of kernels), 1000 power steps 9.5 ms
// (before 1000 x 19 launches and a host wait each, about 200 ms).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "driver.h"
#include "mrsim_internal.h"
#include "spiral_recon.h"

namespace mrsim {
namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 zmulc(double2 a, double2 b) {  // a conj(b)
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 shflx(double2 v, int h) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, h), __shfl_xor_sync(0xffffffffu, v.y, h));
}

// E-point DFT of a lane's registers, natural order in and out; W(j) = w^{j}, w = e^{-+i2pi/E}
template <int E, bool INV>
__device__ __forceinline__ void lane_dft(double2 (&b)[E], const double2* tw, int step) {
  if (E == 1) return;
  if (E == 2) {
    const double2 a = b[0], c = b[E - 1];
    b[0] = make_double2(a.x + c.x, a.y + c.y);
    b[E - 1] = make_double2(a.x - c.x, a.y - c.y);
    return;
  }
  if (E == 4) {
    const double2 s0 = make_double2(b[0].x + b[E / 2].x, b[0].y + b[E / 2].y);
    const double2 d0 = make_double2(b[0].x - b[E / 2].x, b[0].y - b[E / 2].y);
    const double2 s1 = make_double2(b[1 % E].x + b[E - 1].x, b[1 % E].y + b[E - 1].y);
    const double2 d1 = make_double2(b[1 % E].x - b[E - 1].x, b[1 % E].y - b[E - 1].y);
    const double2 r1 = INV ? make_double2(-d1.y, d1.x) : make_double2(d1.y, -d1.x);  // +-i d1
    b[0] = make_double2(s0.x + s1.x, s0.y + s1.y);
    b[1 % E] = make_double2(d0.x + r1.x, d0.y + r1.y);
    b[E / 2] = make_double2(s0.x - s1.x, s0.y - s1.y);
    b[E - 1] = make_double2(d0.x - r1.x, d0.y - r1.y);
    return;
  }
  double2 y[E];
#pragma unroll
  for (int k = 0; k < E; ++k) {
    y[k] = b[0];
#pragma unroll
    for (int m = 1; m < E; ++m) {
      const int j = (m * k) % E;
      const double2 v = j == 0 ? b[m] : INV ? zmulc(b[m], tw[j * step]) : zmul(b[m], tw[j * step]);
      y[k] = make_double2(y[k].x + v.x, y[k].y + v.y);
    }
  }
#pragma unroll
  for (int k = 0; k < E; ++k) b[k] = y[k];
}

// Forward: b[m] = x[lane + 32 m] becomes b[k1] = X[k1 + E bitrev5(lane)] (N = 32 E, e^{-i}).  tw holds
// e^{-i2pi j / (N scale)}.
template <int E>
__device__ __forceinline__ void line_fft(double2 (&b)[E], const double2* tw, int scale, int lane) {
  constexpr int N = 32 * E;
  lane_dft<E, false>(b, tw, 32 * scale);
#pragma unroll
  for (int k1 = 1; k1 < E; ++k1) b[k1] = zmul(b[k1], tw[lane * k1 * scale]);
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
    const double sg = up ? -1.0 : 1.0;
    const double2 w = h > 1 && up ? tw[(lane & (h - 1)) * (N / (2 * h)) * scale] : make_double2(1.0, 0.0);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) {
      const double2 o = shflx(b[k1], h);
      const double2 v = make_double2(fma(sg, b[k1].x, o.x), fma(sg, b[k1].y, o.y));
      b[k1] = h > 1 ? zmul(v, w) : v;
    }
  }
}

// The inverse (unnormalised, e^{+i}) from that order: the forward's steps undone in reverse.
template <int E>
__device__ __forceinline__ void line_ifft(double2 (&b)[E], const double2* tw, int scale, int lane) {
  constexpr int N = 32 * E;
#pragma unroll
  for (int h = 1; h <= 16; h <<= 1) {
    const bool up = (lane & h) != 0;
    const double sg = up ? -1.0 : 1.0;
    const double2 w = h > 1 && up ? tw[(lane & (h - 1)) * (N / (2 * h)) * scale] : make_double2(1.0, 0.0);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) {
      const double2 v = h > 1 ? zmulc(b[k1], w) : b[k1];
      const double2 o = shflx(v, h);
      b[k1] = make_double2(fma(sg, v.x, o.x), fma(sg, v.y, o.y));
    }
  }
#pragma unroll
  for (int k1 = 1; k1 < E; ++k1) b[k1] = zmulc(b[k1], tw[lane * k1 * scale]);
  lane_dft<E, true>(b, tw, 32 * scale);
}

// One image's grid in a cluster of C blocks of T threads.
template <int EN, int C, int T>
struct Grid {
  static constexpr int E2 = 2 * EN, N = 32 * EN, N2 = 2 * N, RP = N / C, LD = N2 + 1, NW = T / 32;
  double2* rows;        // [RP][LD]
  const double2* tw;    // e^{-i2pi j / N2}, j < N2
  const double2* tfp;   // [slot][k1 * 32 + lane]: the circulant's transform, permuted, over N2^2
  const unsigned char* keep;  // [slot][k1 * 32 + lane] of N, or NULL without a band
  int rank, lane, warp;

  __device__ __forceinline__ void sync() const {
    if (C == 1)
      __syncthreads();
    else
      cg::this_cluster().sync();
  }
  // the row y of the image, wherever it lives
  __device__ __forceinline__ double2* row(int y) const {
    if (C == 1) return rows + y * LD;
    return cg::this_cluster().map_shared_rank(rows, y / RP) + (y % RP) * LD;
  }
  // local row yl <- zero-padded FFT_2n of a row held as d[m] = x[lane + 32 m]
  __device__ __forceinline__ void put_padded(int yl, const double2 (&d)[EN]) const {
    double2 b[E2];
#pragma unroll
    for (int m = 0; m < E2; ++m) b[m] = m < EN ? d[m % EN] : make_double2(0.0, 0.0);
    line_fft<E2>(b, tw, 1, lane);
#pragma unroll
    for (int k = 0; k < E2; ++k) rows[yl * LD + lane + 32 * k] = b[k];
  }
  // C: every column of the padded grid
  __device__ __forceinline__ void convolve() const {
    for (int c = rank * NW + warp; c < N2; c += C * NW) {
      double2 b[E2];
#pragma unroll
      for (int m = 0; m < E2; ++m) b[m] = m < EN ? row(lane + 32 * m)[c] : make_double2(0.0, 0.0);
      double2 t[E2];
#pragma unroll
      for (int k = 0; k < E2; ++k) t[k] = __ldg(tfp + (size_t)c * N2 + 32 * k + lane);
      line_fft<E2>(b, tw, 1, lane);
#pragma unroll
      for (int k = 0; k < E2; ++k) b[k] = zmul(b[k], t[k]);
      line_ifft<E2>(b, tw, 1, lane);
#pragma unroll
      for (int m = 0; m < EN; ++m) row(lane + 32 * m)[c] = b[m];
    }
  }
  // R' of a local row without its last step: the cropped row
  __device__ __forceinline__ void crop(int yl, double2 (&d)[EN]) const {
    double2 b[E2];
#pragma unroll
    for (int k = 0; k < E2; ++k) b[k] = rows[yl * LD + lane + 32 * k];
    line_ifft<E2>(b, tw, 1, lane);
#pragma unroll
    for (int m = 0; m < EN; ++m) d[m] = b[m];
  }
  __device__ __forceinline__ void put_spectrum(int yl, double2 (&d)[EN]) const {
    line_fft<EN>(d, tw, 2, lane);
#pragma unroll
    for (int k = 0; k < EN; ++k) rows[yl * LD + lane + 32 * k] = d[k];
  }
  // C': every column of the row spectra
  __device__ __forceinline__ void mask() const {
    constexpr double s = 1.0 / ((double)N * (double)N);
    for (int c = rank * NW + warp; c < N; c += C * NW) {
      double2 b[EN];
#pragma unroll
      for (int m = 0; m < EN; ++m) b[m] = row(lane + 32 * m)[c];
      line_fft<EN>(b, tw, 2, lane);
#pragma unroll
      for (int k = 0; k < EN; ++k) {
        const double f = keep[c * N + 32 * k + lane] ? s : 0.0;
        b[k] = make_double2(b[k].x * f, b[k].y * f);
      }
      line_ifft<EN>(b, tw, 2, lane);
#pragma unroll
      for (int m = 0; m < EN; ++m) row(lane + 32 * m)[c] = b[m];
    }
  }
  __device__ __forceinline__ void take(int yl, double2 (&d)[EN]) const {
#pragma unroll
    for (int k = 0; k < EN; ++k) d[k] = rows[yl * LD + lane + 32 * k];
    line_ifft<EN>(d, tw, 2, lane);
  }
  // one application of the convolution and the band up to the row step R; without a band the
  // cropped rows stay in place of the row spectra, to be read back by take_plain
  __device__ __forceinline__ void apply() const {
    convolve();
    sync();
    for (int yl = warp; yl < RP; yl += NW) {
      double2 d[EN];
      crop(yl, d);
      if (keep) {
        put_spectrum(yl, d);
      } else {
#pragma unroll
        for (int m = 0; m < EN; ++m) rows[yl * LD + lane + 32 * m] = d[m];
      }
    }
    if (keep) {
      sync();
      mask();
      sync();
    } else {
      __syncwarp();
    }
  }
  __device__ __forceinline__ void result(int yl, double2 (&d)[EN]) const {
    if (keep) {
      take(yl, d);
    } else {
#pragma unroll
      for (int m = 0; m < EN; ++m) d[m] = rows[yl * LD + lane + 32 * m];
    }
  }
  // Q of rows held by `get` (a local row to registers), left where result() reads it
  template <class F>
  __device__ __forceinline__ void project(F get) const {
    for (int yl = warp; yl < RP; yl += NW) {
      double2 d[EN];
      get(yl, d);
      if (keep) {
        put_spectrum(yl, d);
      } else {
#pragma unroll
        for (int m = 0; m < EN; ++m) rows[yl * LD + lane + 32 * m] = d[m];
      }
    }
    if (keep) {
      sync();
      mask();
      sync();
    } else {
      __syncwarp();
    }
  }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) v += __shfl_xor_sync(0xffffffffu, v, h);
  return v;
}

struct IterArgs {
  const double2* tfp;
  const unsigned char* keep;
  const double2* tw;
  double2* x;      // chebyshev: [batch][n n] solutions
  double2* r;      // chebyshev: right-hand sides in, residuals out; power: the start vector
  double* out;     // chebyshev: [batch][2] |r|^2 at the start and the end; power: lambda, iterations
  double theta, delta;
  int iterations;
  double tol;
};

constexpr int kIterThreads = 512;   // Chebyshev: 16 warps, four lines each at n = 64
constexpr int kPowerBlocks = 8, kPowerThreads = 256;

// The Chebyshev semi-iteration (grid_recon.rs:238-275): r = Q r, x = 0, dir = r / theta; then
// x += dir; r -= N dir; dir = rho1 rho dir + (2 rho1 / delta) r.
template <int EN, int C>
__global__ void __launch_bounds__(kIterThreads, 1) chebyshev_kernel(const IterArgs a) {
  using G = Grid<EN, C, kIterThreads>;
  constexpr int N = G::N, RP = G::RP, NW = G::NW;
  extern __shared__ __align__(16) double2 ism[];
  __shared__ double part[C * NW];
  G g;
  g.rank = C == 1 ? 0 : (int)cg::this_cluster().block_rank();
  g.lane = threadIdx.x & 31;
  g.warp = threadIdx.x >> 5;
  g.rows = ism;
  double2* dir = ism + RP * G::LD;   // [RP][N]
  double2* tw = dir + RP * N;
  g.tw = tw;
  g.tfp = a.tfp;
  g.keep = a.keep;
  for (int i = threadIdx.x; i < G::N2; i += kIterThreads) tw[i] = a.tw[i];
  const int b = blockIdx.x / C;
  const size_t base = (size_t)b * N * N + (size_t)g.rank * RP * N;
  double2* const x = a.x + base;
  double2* const r = a.r + base;
  __syncthreads();
  // sum over the image of each thread's part, in a fixed order, by every block
  auto image_sum = [&](double v) {
    v = warp_sum(v);
    g.sync();
    if (g.lane == 0)
      for (int q = 0; q < C; ++q) {
        double* p = C == 1 ? part : cg::this_cluster().map_shared_rank(part, q);
        p[g.rank * NW + g.warp] = v;
      }
    g.sync();
    double s = 0.0;
    for (int i = 0; i < C * NW; ++i) s += part[i];
    return s;
  };
  g.project([&](int yl, double2 (&d)[EN]) {
#pragma unroll
    for (int m = 0; m < EN; ++m) d[m] = r[yl * N + g.lane + 32 * m];
  });
  double ss = 0.0;
  for (int yl = g.warp; yl < RP; yl += NW) {
    double2 d[EN];
    g.result(yl, d);
#pragma unroll
    for (int m = 0; m < EN; ++m) {
      const int i = yl * N + g.lane + 32 * m;
      r[i] = d[m];
      x[i] = make_double2(0.0, 0.0);
      ss = fma(d[m].x, d[m].x, fma(d[m].y, d[m].y, ss));
      d[m] = make_double2(d[m].x * (1.0 / a.theta), d[m].y * (1.0 / a.theta));
      dir[i] = d[m];
    }
    g.put_padded(yl, d);
  }
  const double r0 = image_sum(ss);  // its barriers also publish the padded rows
  const double sigma1 = a.theta / a.delta;
  double rho = 1.0 / sigma1;
  ss = a.iterations > 0 ? 0.0 : ss;
  for (int it = 0; it < a.iterations; ++it) {
    g.apply();
    const double rho1 = 1.0 / (2.0 * sigma1 - rho), c1 = rho1 * rho, c2 = 2.0 * rho1 / a.delta;
    rho = rho1;
    const bool last = it + 1 == a.iterations;
    for (int yl = g.warp; yl < RP; yl += NW) {
      double2 rv[EN], xv[EN], dv[EN], nd[EN];
#pragma unroll
      for (int m = 0; m < EN; ++m) {
        const int i = yl * N + g.lane + 32 * m;
        rv[m] = r[i];
        xv[m] = x[i];
        dv[m] = dir[i];
      }
      g.result(yl, nd);
#pragma unroll
      for (int m = 0; m < EN; ++m) {
        const int i = yl * N + g.lane + 32 * m;
        x[i] = make_double2(xv[m].x + dv[m].x, xv[m].y + dv[m].y);
        rv[m] = make_double2(rv[m].x - nd[m].x, rv[m].y - nd[m].y);
        r[i] = rv[m];
        if (last) ss = fma(rv[m].x, rv[m].x, fma(rv[m].y, rv[m].y, ss));
        dv[m] = make_double2(dv[m].x * c1 + rv[m].x * c2, dv[m].y * c1 + rv[m].y * c2);
        dir[i] = dv[m];
      }
      if (!last) g.put_padded(yl, dv);
    }
    g.sync();
  }
  const double rn = image_sum(ss);
  if (g.rank == 0 && threadIdx.x == 0) {
    a.out[2 * b] = r0;
    a.out[2 * b + 1] = rn;
  }
  if (C > 1) g.sync();  // no block leaves while another may still read its shared memory
}

// The power iteration (grid_recon.rs:178-197): lambda = |N v| / |v| until it changes by at most tol of
// itself, at most `iterations` times.  The vector is kept at the scale the estimate of the step
// before gives it (any scale has the same quotient), so its norm is summed beside the row step and
// read after that step's barrier.
template <int EN>
__global__ void __launch_bounds__(kPowerThreads, 1) power_kernel(const IterArgs a) {
  constexpr int C = kPowerBlocks;
  using G = Grid<EN, C, kPowerThreads>;
  constexpr int N = G::N, RP = G::RP, NW = G::NW;
  extern __shared__ __align__(16) double2 ism[];
  __shared__ double part[2][C * NW];
  G g;
  g.rank = (int)cg::this_cluster().block_rank();
  g.lane = threadIdx.x & 31;
  g.warp = threadIdx.x >> 5;
  g.rows = ism;
  double2* tw = ism + RP * G::LD;
  g.tw = tw;
  g.tfp = a.tfp;
  g.keep = a.keep;
  for (int i = threadIdx.x; i < G::N2; i += kPowerThreads) tw[i] = a.tw[i];
  const double2* v0 = a.r + (size_t)g.rank * RP * N;
  g.sync();
  auto publish = [&](double v, int par) {
    v = warp_sum(v);
    if (g.lane < C) cg::this_cluster().map_shared_rank(&part[par][0], g.lane)[g.rank * NW + g.warp] = v;
  };
  auto total = [&](int par) { return warp_sum(part[par][g.lane] + part[par][g.lane + 32]); };
  static_assert(C * NW == 64, "two partial sums a lane");
  double ss = 0.0;
  g.project([&](int yl, double2 (&d)[EN]) {
#pragma unroll
    for (int m = 0; m < EN; ++m) {
      d[m] = v0[yl * N + g.lane + 32 * m];
      ss = fma(d[m].x, d[m].x, fma(d[m].y, d[m].y, ss));
    }
  });
  publish(ss, 1);
  for (int yl = g.warp; yl < RP; yl += NW) {
    double2 d[EN];
    g.result(yl, d);
    g.put_padded(yl, d);
  }
  g.sync();
  double norm = sqrt(total(1)), scale = 1.0, lam = 0.0;
  int it = 0;
  while (it < a.iterations) {
    g.apply();
    ss = 0.0;
    for (int yl = g.warp; yl < RP; yl += NW) {
      double2 d[EN];
      g.result(yl, d);
#pragma unroll
      for (int m = 0; m < EN; ++m) {
        ss = fma(d[m].x, d[m].x, fma(d[m].y, d[m].y, ss));
        d[m] = make_double2(d[m].x * scale, d[m].y * scale);
      }
      g.put_padded(yl, d);
    }
    publish(ss, it & 1);
    g.sync();
    const double nu = sqrt(total(it & 1)), next = nu / norm;
    const bool done = fabs(next - lam) <= a.tol * next;
    lam = next;
    norm = nu * scale;
    scale = 1.0 / next;
    ++it;
    if (done) break;
  }
  if (g.rank == 0 && threadIdx.x == 0) {
    a.out[0] = lam;
    a.out[1] = (double)it;
  }
  g.sync();
}

// the circulant's transform and the band in the order the line transforms leave spectra in
__global__ void permute_tables_kernel(const double2* __restrict__ tf, const unsigned char* __restrict__ keep, int en,
                                      double2* __restrict__ tfp, unsigned char* __restrict__ keepp) {
  const int e2 = 2 * en, n = 32 * en, n2 = 2 * n;
  const double s = 1.0 / ((double)n2 * (double)n2);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n2 * n2; i += gridDim.x * blockDim.x) {
    const int c = i / n2, k = i % n2;
    const int kx = (c >> 5) + e2 * (int)(__brev(c & 31) >> 27), ky = (k >> 5) + e2 * (int)(__brev(k & 31) >> 27);
    const double2 v = tf[kx + (size_t)n2 * ky];
    tfp[i] = make_double2(v.x * s, v.y * s);
  }
  if (keep)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * n; i += gridDim.x * blockDim.x) {
      const int c = i / n, k = i % n;
      const int kx = (c >> 5) + en * (int)(__brev(c & 31) >> 27), ky = (k >> 5) + en * (int)(__brev(k & 31) >> 27);
      keepp[i] = keep[kx + n * ky];
    }
}

template <class K>
void launch_cluster(K kernel, int blocks, int cluster, int threads, size_t smem, const IterArgs& a, cudaStream_t st) {
  MRSIM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  MRSIM_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
}

template <int EN, int C>
void run_chebyshev(int batch, const IterArgs& a, cudaStream_t st) {
  using G = Grid<EN, C, kIterThreads>;
  const size_t smem = sizeof(double2) * ((size_t)G::RP * G::LD + (size_t)G::RP * G::N + G::N2);
  static_assert(sizeof(double2) * ((size_t)G::RP * (G::LD + G::N) + G::N2) + 8 * C * G::NW <= 227 * 1024,
                "an image's rows must fit the cluster");
  launch_cluster(chebyshev_kernel<EN, C>, batch * C, C, kIterThreads, smem, a, st);
}

template <int EN>
void run_power(const IterArgs& a, cudaStream_t st) {
  using G = Grid<EN, kPowerBlocks, kPowerThreads>;
  const size_t smem = sizeof(double2) * ((size_t)G::RP * G::LD + G::N2);
  launch_cluster(power_kernel<EN>, kPowerBlocks, kPowerBlocks, kPowerThreads, smem, a, st);
}

}  // namespace

bool spiral_iter_fits(int n) { return n == 32 || n == 64 || n == 96 || n == 128; }

void spiral_iter_tables(const double2* tf, const unsigned char* keep, int n, double2* tfp, unsigned char* keepp,
                        cudaStream_t st) {
  permute_tables_kernel<<<148, 256, 0, st>>>(tf, keep, n / 32, tfp, keepp);
  MRSIM_CUDA(cudaGetLastError());
}

void spiral_chebyshev(int n, int batch, const double2* tfp, const unsigned char* keepp, const double2* tw2, double2* r,
                      double2* x, double* norms, double theta, double delta, int iterations, cudaStream_t st) {
  IterArgs a{};
  a.tfp = tfp;
  a.keep = keepp;
  a.tw = tw2;
  a.x = x;
  a.r = r;
  a.out = norms;
  a.theta = theta;
  a.delta = delta;
  a.iterations = iterations;
  switch (n) {
    case 32: run_chebyshev<1, 1>(batch, a, st); break;
    case 64: run_chebyshev<2, 1>(batch, a, st); break;
    case 96: run_chebyshev<3, 2>(batch, a, st); break;
    default: run_chebyshev<4, 4>(batch, a, st); break;
  }
}

void spiral_power(int n, const double2* tfp, const unsigned char* keepp, const double2* tw2, double2* v0, double* out,
                  int iterations, double tol, cudaStream_t st) {
  IterArgs a{};
  a.tfp = tfp;
  a.keep = keepp;
  a.tw = tw2;
  a.r = v0;
  a.out = out;
  a.iterations = iterations;
  a.tol = tol;
  switch (n) {
    case 32: run_power<1>(a, st); break;
    case 64: run_power<2>(a, st); break;
    case 96: run_power<3>(a, st); break;
    default: run_power<4>(a, st); break;
  }
}

}  // namespace mrsim
