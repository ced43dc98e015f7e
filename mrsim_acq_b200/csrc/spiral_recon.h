// spiral_recon.h — the device spiral reconstruction (see spiral_recon.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "driver.h"
#include "mrsim_internal.h"
#include "nufft.h"

namespace mrsim {

// grid_recon.rs:36-50
constexpr int kDcfIterations = 10;
constexpr int kLsIterations = 80;
constexpr double kLsKappa = 100.0;
constexpr int kPowerIterations = 1000;
constexpr double kPowerTol = 1e-10;
constexpr double kLambdaMargin = 1.1;

// The iterations as one launch each, for n = 32, 64, 96, 128 (spiral_iter.cu): tables permuted from
// the circulant's transform and the band (NULL: none); norms [batch][2] = |r|^2 before and after; out
// = lambda and the iterations taken.
bool spiral_iter_fits(int n);
void spiral_iter_tables(const double2* tf, const unsigned char* keep, int n, double2* tfp, unsigned char* keepp,
                        cudaStream_t st);
void spiral_chebyshev(int n, int batch, const double2* tfp, const unsigned char* keepp, const double2* tw2, double2* r,
                      double2* x, double* norms, double theta, double delta, int iterations, cudaStream_t st);
void spiral_power(int n, const double2* tfp, const unsigned char* keepp, const double2* tw2, double2* v0, double* out,
                  int iterations, double tol, cudaStream_t st);

struct SpiralRecon {
  mrsim_context* ctx;
  int n, npts, iterations;
  double kappa;
  bool band;
  double lambda_hi = 0.0;
  int power_iterations = 0;
  DevArena A;
  NufftGridT<double> g{};
  NufftBins bins_k;  // the trajectory's spread bins on g
  const double2* tw_n = nullptr;
  const double2* tw_2n = nullptr;
  double* d_k = nullptr;
  double* d_w = nullptr;    // normalized density weights
  double* d_win = nullptr;  // window per sample
  unsigned char* d_keep = nullptr;
  double2* d_tf = nullptr;  // transform of the Toeplitz kernel's circulant, 2n x 2n
  double2* d_tfp = nullptr;  // where spiral_iter_fits(n): it and the band in the iterations' order
  unsigned char* d_keepp = nullptr;
  std::vector<double> w_host, k_host;

  struct Scratch {
    double2* pad;
    double2* tmp;
  };

  // `SpiralRecon::with_params` (grid_recon.rs:152-198); the window is win_acq's.  call_scoped: it ends
  // with the call that made it, so its memory comes from the context's pool.
  SpiralRecon(mrsim_context* ctx, const double* k, int npts, int n, const mrsim_acquisition& win_acq,
              int iterations, double kappa, bool band_limited, bool call_scoped = false);
  // Images per pass through the Chebyshev iteration.  As one launch, four waves of 148 blocks, where a
  // pass's samples, fine grids and images stay below 8 GB; else 256: the launches per step fill the
  // chip with fewer, and their padded grids (128 n^2 bytes an image) are 34 GB for 256 at n = 1024.
  int max_batch() const {
    const size_t per = ((size_t)npts + (size_t)g.nf0 * g.nf1 + (size_t)n * n) * 16;
    return d_tfp && 592 * per <= ((size_t)8 << 30) ? 592 : 256;
  }
  Scratch scratch(DevArena& T, int batch) const;
  void project(double2* x, int batch, cudaStream_t st) const;
  void normal(const double2* x, double2* out, int batch, const Scratch& s, cudaStream_t st) const;
  void sumsq(const double2* v, int batch, double* out, cudaStream_t st) const;
  // device buffers: data [batch][npts], images [batch][n*n]
  void gridding(const double2* d_data, int batch, double2* d_out);
  void images(const double2* d_data, int batch, double2* d_x);
  void rings(const double2* d_coil, int n_part, int ncoils, int ring, const double* zsens, double2* d_out);
};

}  // namespace mrsim
