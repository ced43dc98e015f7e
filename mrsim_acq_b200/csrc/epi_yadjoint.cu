// epi_yadjoint.cu — the y-stage of the EPI adjoint (see epi_kernels.cu) and its launcher.
#include "epi_device.h"

namespace mrsim {

namespace {

// ---------------------------------------------------------------------------------------------
// y-adjoint: per voxel, over every line j and coil q:
//   H_j = s * sum_q (ex_q ey_q + off) h_q[j][x];   Z_j = conj(e^{i2pi theta_j}) H_j
//   comp_grad_c = sum_j rel_cj Z_j                          (A^H r, complex)
//   fmap_grad   = 4 pi sum_c m_c Im(sum_j t_j rel_cj Z_j)   (dL/dfmap, L = sum |r|^2)
//   r2_grad_c   = -2 m_c Re(sum_j trf_j rel_cj Z_j)         (dL/dR2_c)
// A CTA of 128 threads covers 128 columns x TY rows (one column each).  The line table sits in
// shared memory; h arrives by cp.async in double-buffered chunks of JC lines x every coil.

template <int TY, int NC, bool MAPS, bool GRADS>
__global__ void __launch_bounds__(128) yadjoint_kernel(const UnitDesc* __restrict__ units,
                                                       const int4* __restrict__ tiles) {
  extern __shared__ __align__(16) float smem[];
  static_assert(TY == 4, "the row tables are read as float4");
  constexpr int ROWS = TY;
  const int4 tl = tiles[blockIdx.x];  // unit, y0, x0
  const UnitDesc& u = units[tl.x];
  const int snx = u.snx, sny = u.sny, ncomp = u.ncomp, nlines = u.n_lines, ncoils = u.ncoils;
  const int y0 = tl.y;
  const int JC = adjoint_chunk_lines(ncoils);
  // shared layout: h buffers (2 x JC x ncoils x 128 float2), then floats
  float2* hbuf = reinterpret_cast<float2*>(smem);
  float* Bt = reinterpret_cast<float*>(hbuf + 2 * JC * ncoils * 128);  // [nlines][ROWS]
  float* Ey = Bt + nlines * ROWS;                                        // [ncoils][ROWS]
  float* Ex = Ey + ncoils * ROWS;                                        // [ncoils][128], scale folded
  float* Lt = Ex + ncoils * 128;                                         // [nlines][LF] line table
  constexpr int LF = 5 + NC;  // t_hi, t_lo, trf, inhom, t_phase, rel[NC]
  const int ys = u.ny / 2;
  const int oy = sny / u.ny;
  const int sys = oy * ys;
  const int col = threadIdx.x;
  const int x = tl.z + col;
  const bool xok = x < snx;
  const float2* __restrict__ hcol = u.g + (xok ? x : 0);
  const size_t qstride = (size_t)nlines * snx;
  // the first h chunk is in flight while the tables fill
  auto issue_chunk = [&](int c, int buf) {
    const int j0 = c * JC;
    for (int jj = 0; jj < JC; ++jj) {
      const int j = j0 + jj;
      if (j >= nlines) break;
      for (int q = 0; q < ncoils; ++q)
        cp_async8(hbuf + ((size_t)(buf * JC + jj) * ncoils + q) * 128 + col, hcol + q * qstride + (size_t)j * snx);
    }
    cp_async_commit();
  };
  const int nchunks = (nlines + JC - 1) / JC;
  if (nchunks > 0) issue_chunk(0, 0);
  for (int idx = threadIdx.x; idx < nlines * ROWS; idx += blockDim.x) {
    const int j = idx / ROWS, r = idx % ROWS;
    const int y = y0 + r;
    float v = 0.f;
    if (y < sny) {
      const LineRec& L = u.lines[j];
      double tv = kr_turns(L.ky - ys, 2 * (y - sys) - (oy - 1), 2 * sny);
      if (u.flags & UF_EDDY) {
        const double yc = ((double)y - sys - (oy - 1) / 2.0) / oy;
        tv += ((double)u.eddy_cy * yc + (double)u.eddy_qy * yc * yc) * (double)L.decay;
      }
      tv -= rint(tv);
      v = (float)tv;
    }
    Bt[idx] = v;
  }
  for (int idx = threadIdx.x; idx < ncoils * ROWS; idx += blockDim.x) {
    const int q = idx / ROWS, r = idx % ROWS;
    const int y = y0 + r;
    Ey[idx] = y < sny ? u.geo.ey[(size_t)q * sny + y] : 0.f;
  }
  for (int idx = threadIdx.x; idx < ncoils * 128; idx += blockDim.x) {
    const int q = idx / 128, c = idx % 128;
    const int xx = tl.z + c;
    Ex[idx] = xx < snx ? u.signal_scale * u.geo.ex[(size_t)q * snx + xx] : 0.f;
  }
  for (int j = threadIdx.x; j < nlines; j += blockDim.x) {
    const LineRec& L = u.lines[j];
    float* e = Lt + j * LF;
    e[0] = L.t_hi;
    e[1] = L.t_lo;
    e[2] = L.trf_ms;
    e[3] = L.inhom_ms;
    e[4] = L.t_hi + L.t_lo;
#pragma unroll
    for (int c = 0; c < NC; ++c) e[5 + c] = L.rel[c];
  }
  __syncthreads();
  const bool active = xok && y0 < sny;
  const bool distort = (u.flags & UF_DISTORT) != 0;
  float a[TY], f[TY], r2[TY][MAPS ? NC : 1], r2i[TY][MAPS ? NC : 1], la[TY];
#pragma unroll
  for (int ty = 0; ty < TY; ++ty) {
    const int y = min(y0 + ty, sny - 1);
    const int i = (xok ? x : 0) + snx * y;
    a[ty] = u.phase ? __ldg(u.phase + i) : 0.f;
    f[ty] = distort ? __ldg(u.fmap + i) : 0.f;
    la[ty] = (MAPS && u.log_amp) ? __ldg(u.log_amp + i) : 0.f;
    if (MAPS) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        r2[ty][MAPS ? c : 0] = r2i[ty][MAPS ? c : 0] = 0.f;
        if (c < ncomp) {
          const float t2 = u.t2map ? __ldg(u.t2map + (size_t)c * u.map_stride + i) : u.t2u[c];
          const float ti = u.timap ? __ldg(u.timap + (size_t)c * u.map_stride + i) : u.tiu[c];
          r2[ty][MAPS ? c : 0] = 1.0f / t2;
          r2i[ty][MAPS ? c : 0] = 1.0f / ti;
        }
      }
    }
  }
  float2 cg[TY][NC];
  float Uy[TY][GRADS ? NC : 1], Vx[TY][GRADS ? NC : 1];
#pragma unroll
  for (int ty = 0; ty < TY; ++ty)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      cg[ty][c] = make_float2(0.f, 0.f);
      if (GRADS) Uy[ty][GRADS ? c : 0] = Vx[ty][GRADS ? c : 0] = 0.f;
    }
  const float soff = u.signal_scale * u.geo.coil_off;
  for (int c = 0; c < nchunks; ++c) {
    const int buf = c & 1;
    if (c + 1 < nchunks) {
      issue_chunk(c + 1, buf ^ 1);
      cp_async_wait1();
    } else {
      cp_async_wait0();
    }
    // each thread reads back only its own column, which it copied itself: no barrier needed
    const int j0 = c * JC;
    const int jn = min(JC, nlines - j0);
    for (int jj = 0; jj < jn; ++jj) {
      const int j = j0 + jj;
      const float* e = Lt + j * LF;
      const float thi = e[0], tlo = e[1], trf = e[2], tinh = e[3], tph = e[4];
      // (Re, Im) pairs in packed f32x2 arithmetic: each lane rounds as the scalar product, sum and
      // fused multiply-add do, so the sums are bitwise the scalar ones in half the issue slots
      float2 H[TY];
      float2 hs = make_float2(0.f, 0.f);
#pragma unroll
      for (int ty = 0; ty < TY; ++ty) H[ty] = make_float2(0.f, 0.f);
      const float2* hb = hbuf + (size_t)(buf * JC + jj) * ncoils * 128 + col;
#pragma unroll 4
      for (int q = 0; q < ncoils; ++q) {
        const float2 h = hb[q * 128];
        const float ex = Ex[q * 128 + col];
        hs = fadd2(hs, h);
        const float2 uu = fmul2(dup2(ex), h);
        const float4 e4 = *reinterpret_cast<const float4*>(Ey + q * ROWS);
        const float ey[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
        for (int ty = 0; ty < TY; ++ty) H[ty] = ffma2(dup2(ey[ty]), uu, H[ty]);
      }
      const float hsr = hs.x, hsi = hs.y;
      const float4 b4 = *reinterpret_cast<const float4*>(Bt + j * ROWS);
      const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int ty = 0; ty < TY; ++ty) {
        const float hr = fmaf(soff, hsr, H[ty].x), hi = fmaf(soff, hsi, H[ty].y);
        const float th = phase_turns(a[ty] + bt[ty], f[ty], thi, tlo);
        float sn, cs;
        __sincosf(kTwoPiF * th, &sn, &cs);
        const float zr = fmaf(cs, hr, sn * hi);  // Z = conj(P) * H
        const float zi = fmaf(cs, hi, -sn * hr);
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          if (cc < ncomp) {
            float r;
            if (MAPS)
              r = __expf(la[ty] - trf * r2[ty][MAPS ? cc : 0] - tinh * r2i[ty][MAPS ? cc : 0]);
            else
              r = e[5 + cc];
            cg[ty][cc].x = fmaf(r, zr, cg[ty][cc].x);
            cg[ty][cc].y = fmaf(r, zi, cg[ty][cc].y);
            if (GRADS) {
              Uy[ty][GRADS ? cc : 0] = fmaf(r * tph, zi, Uy[ty][GRADS ? cc : 0]);
              Vx[ty][GRADS ? cc : 0] = fmaf(r * trf, zr, Vx[ty][GRADS ? cc : 0]);
            }
          }
        }
      }
    }
  }
  if (!active) return;
  const size_t plane = (size_t)snx * sny;
#pragma unroll
  for (int ty = 0; ty < TY; ++ty) {
    const int y = y0 + ty;
    if (y >= sny) break;
    const size_t i = (size_t)x + (size_t)snx * y;
    float fg = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if (c >= ncomp) break;
      u.comp_grad[c * plane + i] = cg[ty][c];
      if (GRADS) {
        const float m = __ldg(u.comp + (size_t)c * u.comp_stride + i);
        fg = fmaf(m, Uy[ty][GRADS ? c : 0], fg);
        if (u.r2_grad) u.r2_grad[c * plane + i] = -2.0f * m * Vx[ty][GRADS ? c : 0];
      }
    }
    if (GRADS && u.fmap_grad) u.fmap_grad[i] = distort ? 4.0f * 3.14159265358979f * fg : 0.f;
  }
}

// ---------------------------------------------------------------------------------------------
// y-adjoint for a compile-time coil count NQ (every unit of the plan has NQ coils, an even snx and
// 16-byte aligned h rows).  Same sums as yadjoint_kernel, reorganised so the per-(line, voxel)
// work is the coil combination and the phase:
//   * a CTA of 256 threads covers 128 columns x 2*TY rows (two groups of TY rows, one column each;
//     TY = 4 with class decay, 2 with voxel maps, whose rates take the registers);
//   * amp_q(x, y) = s * (ex_q(x) ey_q(y) + off) of the thread's TY rows sits in registers, so the
//     coil combination is 2 FMAs per (coil, row) from one shared load of h per coil;
//   * h arrives through a 3-stage ring of JC-line chunks (every coil, 128 columns) filled by
//     cooperative 16-byte cp.async, one barrier per chunk;
//   * the line table carries rel_cj, rel_cj * t_j and rel_cj * trf_j (class decay), so every
//     accumulator update is one FMA.


// VIRT = 1: the h rows are the NQ = classes + 1 class rows of the class-mode x-adjoint (scale, ex and
// the coil offset already applied), so amp_v(y) = ey_v(y) for the classes and 1 for the offset row;
// VIRT = 2: the NQ basis rows of the basis x-adjoint (the unit's eyc holds the coil basis); the constant
// row, which carries most of H, is added last, so that one sum alone rounds at its size.
// NARROW: odd rows (or g off a 16-byte boundary), so the ring fills by 8-byte copies.
// CHAIN: a small launch, chained to the kernel before it.
template <int NQ, int TY, int NC, bool MAPS, bool GRADS, int VIRT, bool NARROW, bool CHAIN>
__global__ void __launch_bounds__(256, (VIRT && !MAPS && TY == 2) ? 3 : 2) yadjoint_q_kernel(const UnitDesc* __restrict__ units,
                                                            const int4* __restrict__ tiles) {
  extern __shared__ __align__(16) float smem[];
  static_assert(TY == 2 || TY == 4, "the row phases are read as one float2 / float4");
  constexpr int ROWS = 2 * TY;
  constexpr int JC = adjq_chunk_lines(NQ);
  constexpr int LF = adjq_line_floats(NC, MAPS);
  constexpr int STAGE = JC * NQ * 128;        // float2 per stage
  constexpr int PIECES = JC * NQ * 64;        // 16-byte pieces per stage
  constexpr int PPT = (PIECES + 255) / 256;   // pieces per thread
  if (CHAIN) grid_begin();
  const int4 tl = tiles[blockIdx.x];  // unit, y0, x0
  const UnitDesc& u = units[tl.x];
  const int snx = u.snx, sny = u.sny, ncomp = u.ncomp, nlines = u.n_lines;
  const int y0 = tl.y, x0 = tl.z;
  float2* hbuf = reinterpret_cast<float2*>(smem);
  float* Bt = reinterpret_cast<float*>(hbuf + kAdjStages * STAGE);  // [nlines][ROWS]
  // the line tables cover whole chunks (zero entries past nlines), so the packed path runs every
  // line of a chunk without a branch
  const int nlp = (nlines + JC - 1) / JC * JC;
  float* Lt = Bt + nlp * ROWS;                                       // [nlp][LF]
  const int tid = threadIdx.x;
  const int col = tid & 127, rg = tid >> 7;
  const int x = x0 + col;
  const bool xok = x < snx;
  const int nchunks = (nlines + JC - 1) / JC;

  // This thread's 16-byte pieces k = tid + 256 i of a chunk: row r = k / 64 = (line jj, coil q),
  // column pair 2 (k % 64); the destination is float2 2k of the stage.  The source offset of
  // each piece for the chunk's first line (or -1 past snx) sits in a per-thread shared table, so
  // a chunk costs one shared load, a compare and a select per piece.  (The plan keeps
  // NQ * lines * snx below 2^31.)
  __shared__ int ptab[PPT * 256];
  const float2* __restrict__ gsrc = u.g;
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    const int k = tid + 256 * i;
    if (PIECES % 256 == 0 || k < PIECES) {
      const int r = k >> 6, xx = x0 + (k & 63) * 2;
      ptab[i * 256 + tid] = xx < snx ? ((r % NQ) * nlines + r / NQ) * snx + xx : -1;
    }
  }
  auto issue_chunk = [&](int c, int stage) {
    if (NARROW && c < nchunks) {
      float2* dst = hbuf + stage * STAGE;
      for (int k = tid; k < STAGE; k += 256) {
        const int r = k >> 7, xx = x0 + (k & 127), j = c * JC + r / NQ;
        const bool ok = xx < snx && j < nlines;
        cp_async8(dst + k, gsrc + (ok ? ((size_t)(r % NQ) * nlines + j) * snx + xx : 0), ok ? 8 : 0);
      }
    } else if (c < nchunks) {
      const int rem = nlines - c * JC, jo = c * JC * snx;
      float2* dst = hbuf + stage * STAGE;
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int k = tid + 256 * i;
        if (PIECES % 256 == 0 || k < PIECES) {
          const int o = ptab[i * 256 + tid];
          const bool ok = o >= 0 && ((tid >> 6) + 4 * i) / NQ < rem;
          cp_async16(dst + 2 * k, gsrc + (ok ? o + jo : 0), ok ? 16 : 0);
        }
      }
    }
    cp_async_commit();
  };
  if (!CHAIN) {  // (as in the forward: a small launch fills its tables first)
#pragma unroll
    for (int c = 0; c < kAdjStages - 1; ++c) issue_chunk(c, c);
  }

  const int ys = u.ny / 2;
  const int oy = sny / u.ny;
  const int sys = oy * ys;
  for (int idx = tid; idx < nlp * ROWS; idx += 256) {
    const int j = idx / ROWS, r = idx % ROWS;
    const int y = y0 + r;
    float v = 0.f;
    if (y < sny && j < nlines) {
      const LineRec& L = u.lines[j];
      double tv = kr_turns(L.ky - ys, 2 * (y - sys) - (oy - 1), 2 * sny);
      if (u.flags & UF_EDDY) {
        const double yc = ((double)y - sys - (oy - 1) / 2.0) / oy;
        tv += ((double)u.eddy_cy * yc + (double)u.eddy_qy * yc * yc) * (double)L.decay;
      }
      tv -= rint(tv);
      v = (float)tv;
    }
    Bt[idx] = v;
  }
  for (int j = tid; j < nlp; j += 256) {
    float* e = Lt + j * LF;
    if (j >= nlines) {
#pragma unroll
      for (int k = 0; k < LF; ++k) e[k] = 0.f;
      continue;
    }
    const LineRec& L = u.lines[j];
    const float tph = L.t_hi + L.t_lo;
    e[0] = L.t_hi;
    e[1] = L.t_lo;
    e[2] = L.trf_ms;
    e[3] = L.inhom_ms;
    if (MAPS) {
      e[4] = tph;
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) {  // zero weights past ncomp: those accumulators stay 0
        const float r = c < ncomp ? L.rel[c] : 0.f;
        e[4 + c] = r;
        e[4 + NC + c] = r * tph;
        e[4 + 2 * NC + c] = r * L.trf_ms;
      }
    }
  }

  if (CHAIN) {
    grid_wait();
#pragma unroll
    for (int c = 0; c < kAdjStages - 1; ++c) issue_chunk(c, c);
  }
  // per-thread constants of its 4 rows
  const bool distort = (u.flags & UF_DISTORT) != 0;
  const int xs_ = xok ? x : 0;
  const float s = u.signal_scale, off = u.geo.coil_off;
  float amp[TY][NQ];
  float a[TY], f[TY];
  float r2[TY][MAPS ? NC : 1], r2i[TY][MAPS ? NC : 1], la[TY];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const float ex = VIRT ? 0.f : u.geo.ex[(size_t)q * snx + xs_];
#pragma unroll
    for (int ty = 0; ty < TY; ++ty) {
      const int y = min(y0 + rg * TY + ty, sny - 1);
      if (VIRT)
        amp[ty][q] = q < NQ - 1 ? u.geo.eyc[(size_t)q * sny + y] : 1.f;
      else
        amp[ty][q] = s * fmaf(ex, u.geo.ey[(size_t)q * sny + y], off);
    }
  }
#pragma unroll
  for (int ty = 0; ty < TY; ++ty) {
    const int y = min(y0 + rg * TY + ty, sny - 1);
    const int i = xs_ + snx * y;
    a[ty] = !u.phase ? 0.f : CHAIN ? u.phase[i] : __ldg(u.phase + i);  // (see grid_wait)
    f[ty] = distort ? __ldg(u.fmap + i) : 0.f;
    la[ty] = (MAPS && u.log_amp) ? __ldg(u.log_amp + i) : 0.f;
    if (MAPS) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        r2[ty][MAPS ? c : 0] = r2i[ty][MAPS ? c : 0] = 0.f;
        if (c < ncomp) {
          const float t2 = u.t2map ? __ldg(u.t2map + (size_t)c * u.map_stride + i) : u.t2u[c];
          const float ti = u.timap ? __ldg(u.timap + (size_t)c * u.map_stride + i) : u.tiu[c];
          r2[ty][MAPS ? c : 0] = 1.0f / t2;
          r2i[ty][MAPS ? c : 0] = 1.0f / ti;
        }
      }
    }
  }
  // PK (class rows, class decay, 4 rows): rows (0, 1) and (2, 3) run as packed f32x2 pairs, with
  // accumulators pcx/pcy/puy/pvx[pair][c] holding the two rows' Re/Im comp sums, t- and trf-sums
  constexpr bool PK = VIRT && !MAPS;
  constexpr int NPR = PK ? TY / 2 : 1;  // row pairs
  float2 pcx[NPR][NC], pcy[NPR][NC], puy[NPR][NC], pvx[NPR][NC];
  if (PK) {
#pragma unroll
    for (int pp = 0; pp < NPR; ++pp)
#pragma unroll
      for (int c = 0; c < NC; ++c) pcx[pp][c] = pcy[pp][c] = puy[pp][c] = pvx[pp][c] = make_float2(0.f, 0.f);
  }
  float2 cg[TY][NC];
  float Uy[TY][GRADS ? NC : 1], Vx[TY][GRADS ? NC : 1];
#pragma unroll
  for (int ty = 0; ty < TY; ++ty)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      cg[ty][c] = make_float2(0.f, 0.f);
      if (GRADS) Uy[ty][GRADS ? c : 0] = Vx[ty][GRADS ? c : 0] = 0.f;
    }

  // basis rows: the sums of whole blocks of kLineBlock lines, [sum][thread], and their additions
  static_assert(kLineBlock % JC == 0, "whole chunks in a block");
  float2* const whole = reinterpret_cast<float2*>(Lt + (size_t)nlp * LF) + tid;
  const bool blocked = VIRT == 2 && adj_blocked(NQ, NC, MAPS, GRADS, nlines);
  auto each_sum = [&](auto f) {  // f(sum, its place)
    int k = 0;
    if (PK) {
#pragma unroll
      for (int pp = 0; pp < NPR; ++pp)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          f(pcx[pp][c], whole[256 * k++]);
          f(pcy[pp][c], whole[256 * k++]);
          if (GRADS) {
            f(puy[pp][c], whole[256 * k++]);
            f(pvx[pp][c], whole[256 * k++]);
          }
        }
    } else {
#pragma unroll
      for (int ty = 0; ty < TY; ++ty)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          f(cg[ty][c], whole[256 * k++]);
          if (GRADS) {
            float2 t = make_float2(Uy[ty][GRADS ? c : 0], Vx[ty][GRADS ? c : 0]);
            f(t, whole[256 * k++]);
            Uy[ty][GRADS ? c : 0] = t.x;
            Vx[ty][GRADS ? c : 0] = t.y;
          }
        }
    }
  };
  if (VIRT == 2 && blocked) each_sum([](float2& acc, float2& w) { w = acc; });  // (zeros)

  int s_use = 0, s_issue = kAdjStages - 1;  // stages of chunk c and of chunk c + stages - 1
  auto add_chunk = [&](int c) {
    cp_async_wait_n<kAdjStages - 2>();
    __syncthreads();  // chunk c landed for every thread; every thread is done with chunk c - 1
    issue_chunk(c + kAdjStages - 1, s_issue);
    s_issue = s_issue + 1 == kAdjStages ? 0 : s_issue + 1;
    const float2* hs = hbuf + s_use * STAGE + col;
    s_use = s_use + 1 == kAdjStages ? 0 : s_use + 1;
    const int j0 = c * JC;
#pragma unroll
    for (int jj = 0; jj < JC; ++jj) {
      const int j = j0 + jj;
      if (!PK && j >= nlines) break;  // (the packed path reads the zero entries instead)
      const float* e = Lt + j * LF;
      const float4 e0 = *reinterpret_cast<const float4*>(e);
      const float thi = e0.x, tlo = e0.y, trf = e0.z, tinh = e0.w;
      if (PK) {
        float2 Hx[NPR], Hy[NPR];  // [pair] = rows (2p, 2p + 1); starts from the offset row (amplitude 1)
        if (VIRT == 1) {
          const float2 h = hs[(jj * NQ + NQ - 1) * 128];
#pragma unroll
          for (int pp = 0; pp < NPR; ++pp) {
            Hx[pp] = dup2(h.x);
            Hy[pp] = dup2(h.y);
          }
        }
#pragma unroll
        for (int q = 0; q < NQ - 1; ++q) {
          const float2 h = hs[(jj * NQ + q) * 128];
          const float2 hx = dup2(h.x), hy = dup2(h.y);
#pragma unroll
          for (int pp = 0; pp < NPR; ++pp) {
            const float2 am = make_float2(amp[2 * pp][q], amp[(2 * pp + 1) % TY][q]);
            Hx[pp] = VIRT == 2 && q == 0 ? fmul2(am, hx) : ffma2(am, hx, Hx[pp]);
            Hy[pp] = VIRT == 2 && q == 0 ? fmul2(am, hy) : ffma2(am, hy, Hy[pp]);
          }
        }
        if (VIRT == 2) {
          const float2 h = hs[(jj * NQ + NQ - 1) * 128];
#pragma unroll
          for (int pp = 0; pp < NPR; ++pp) {
            Hx[pp] = fadd2(Hx[pp], dup2(h.x));
            Hy[pp] = fadd2(Hy[pp], dup2(h.y));
          }
        }
        float2 btp[NPR];
        if (TY == 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(Bt + j * ROWS + rg * TY);
          btp[0] = make_float2(b4.x, b4.y);
          btp[NPR - 1] = make_float2(b4.z, b4.w);
        } else {
          btp[0] = *reinterpret_cast<const float2*>(Bt + j * ROWS + rg * TY);
        }
        const float2 thi2 = dup2(thi), tlo2 = dup2(tlo);
#pragma unroll
        for (int pp = 0; pp < NPR; ++pp) {
          const int t0 = 2 * pp, t1 = (2 * pp + 1) % TY;
          const float2 bt2 = btp[pp];
          float2 th = phase_turns2(fadd2(make_float2(a[t0], a[t1]), bt2), make_float2(f[t0], f[t1]), thi2, tlo2);
          th = fmul2(dup2(kTwoPiF), th);
          float s0, c0, s1, c1;
          __sincosf(th.x, &s0, &c0);
          __sincosf(th.y, &s1, &c1);
          const float2 cs2 = make_float2(c0, c1), sn2 = make_float2(s0, s1);
          const float2 zr = ffma2(cs2, Hx[pp], fmul2(sn2, Hy[pp]));  // Z = conj(P) H per row
          const float2 zi = ffma2(cs2, Hy[pp], fsub2(dup2(0.f), fmul2(sn2, Hx[pp])));
#pragma unroll
          for (int cc = 0; cc < NC; ++cc) {
            const float2 r = dup2(e[4 + cc]);
            pcx[PK ? pp : 0][cc] = ffma2(r, zr, pcx[PK ? pp : 0][cc]);
            pcy[PK ? pp : 0][cc] = ffma2(r, zi, pcy[PK ? pp : 0][cc]);
            if (GRADS) {
              puy[PK ? pp : 0][cc] = ffma2(dup2(e[4 + NC + cc]), zi, puy[PK ? pp : 0][cc]);
              pvx[PK ? pp : 0][cc] = ffma2(dup2(e[4 + 2 * NC + cc]), zr, pvx[PK ? pp : 0][cc]);
            }
          }
        }
        continue;
      }
      float2 H[TY];
      {
        const float2 h = hs[jj * NQ * 128];
#pragma unroll
        for (int ty = 0; ty < TY; ++ty) H[ty] = make_float2(amp[ty][0] * h.x, amp[ty][0] * h.y);
      }
#pragma unroll
      for (int q = 1; q < NQ; ++q) {
        const float2 h = hs[(jj * NQ + q) * 128];
#pragma unroll
        for (int ty = 0; ty < TY; ++ty) {
          H[ty].x = fmaf(amp[ty][q], h.x, H[ty].x);
          H[ty].y = fmaf(amp[ty][q], h.y, H[ty].y);
        }
      }
      float bt[TY];
      if (TY == 4) {
        const float4 b4 = *reinterpret_cast<const float4*>(Bt + j * ROWS + rg * TY);
        bt[0] = b4.x, bt[1] = b4.y, bt[TY > 2 ? 2 : 0] = b4.z, bt[TY > 3 ? 3 : 0] = b4.w;
      } else {
        const float2 b2 = *reinterpret_cast<const float2*>(Bt + j * ROWS + rg * TY);
        bt[0] = b2.x, bt[1] = b2.y;
      }
      const float tph = MAPS ? e[4] : 0.f;
#pragma unroll
      for (int ty = 0; ty < TY; ++ty) {
        const float th = phase_turns(a[ty] + bt[ty], f[ty], thi, tlo);
        float sn, cs;
        __sincosf(kTwoPiF * th, &sn, &cs);
        const float zr = fmaf(cs, H[ty].x, sn * H[ty].y);  // Z = conj(P) * H
        const float zi = fmaf(cs, H[ty].y, -sn * H[ty].x);
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          if (!MAPS || cc < ncomp) {
            float r, rt, rf;
            if (MAPS) {
              r = __expf(la[ty] - trf * r2[ty][MAPS ? cc : 0] - tinh * r2i[ty][MAPS ? cc : 0]);
              rt = r * tph;
              rf = r * trf;
            } else {
              r = e[4 + cc];
              rt = e[4 + NC + cc];
              rf = e[4 + 2 * NC + cc];
            }
            cg[ty][cc].x = fmaf(r, zr, cg[ty][cc].x);
            cg[ty][cc].y = fmaf(r, zi, cg[ty][cc].y);
            if (GRADS) {
              Uy[ty][GRADS ? cc : 0] = fmaf(rt, zi, Uy[ty][GRADS ? cc : 0]);
              Vx[ty][GRADS ? cc : 0] = fmaf(rf, zr, Vx[ty][GRADS ? cc : 0]);
            }
          }
        }
      }
    }
  };
  if (VIRT == 2 && blocked) {
    for (int c0 = 0; c0 < nchunks; c0 += kLineBlock / JC) {
      const int c1 = min(nchunks, c0 + kLineBlock / JC);
      for (int c = c0; c < c1; ++c) add_chunk(c);
      if (c1 < nchunks)
        each_sum([](float2& acc, float2& w) {
          w = fadd2(w, acc);
          acc = make_float2(0.f, 0.f);
        });
    }
  } else {
    for (int c = 0; c < nchunks; ++c) add_chunk(c);
  }
  cp_async_wait0();
  if (!xok) return;
  if (VIRT == 2 && blocked) each_sum([](float2& acc, float2& w) { acc = fadd2(w, acc); });
  if (PK) {
#pragma unroll
    for (int ty = 0; ty < TY; ++ty)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int pp = PK ? (ty >> 1) % NPR : 0;
        const bool hi = ty & 1;
        cg[ty][c] = make_float2(hi ? pcx[pp][c].y : pcx[pp][c].x, hi ? pcy[pp][c].y : pcy[pp][c].x);
        if (GRADS) {
          Uy[ty][GRADS ? c : 0] = hi ? puy[pp][c].y : puy[pp][c].x;
          Vx[ty][GRADS ? c : 0] = hi ? pvx[pp][c].y : pvx[pp][c].x;
        }
      }
  }
  const size_t plane = (size_t)snx * sny;
#pragma unroll
  for (int ty = 0; ty < TY; ++ty) {
    const int y = y0 + rg * TY + ty;
    if (y >= sny) break;
    const size_t i = (size_t)x + (size_t)snx * y;
    float fg = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if (c >= ncomp) break;
      u.comp_grad[c * plane + i] = cg[ty][c];
      if (GRADS) {
        const float m = __ldg(u.comp + (size_t)c * u.comp_stride + i);
        fg = fmaf(m, Uy[ty][GRADS ? c : 0], fg);
        if (u.r2_grad) u.r2_grad[c * plane + i] = -2.0f * m * Vx[ty][GRADS ? c : 0];
      }
    }
    if (GRADS && u.fmap_grad) u.fmap_grad[i] = distort ? 4.0f * 3.14159265358979f * fg : 0.f;
  }
}

}  // namespace

void epi_plan_adjoint_ystage(const EpiPlan* p, cudaStream_t st, int u0, int u1) {
  for (int pass = 0; pass < 4; ++pass) {
    const TileRange R = tile_range(p->a_start[pass], p->n_atiles[pass], u0, u1);
    if (R.n == 0) continue;
    const int4* tiles = p->d_atiles[pass] + R.t0;
    const bool maps = pass & 1, grads = (pass & 2) != 0;
    const int NCv = p->nc;
    if (p->adj_thin[pass]) {
      launch_yadjoint_thin(p, pass, tiles, R.n, st);
      continue;
    }
    if (p->adjq[pass]) {
      const int NQv = p->adjq[pass];
      const int TYv = p->adj_ty[pass];
      size_t smq = yadjoint_q_smem(NQv, TYv, NCv, maps, p->max_lines);
      if (p->basis_nb) smq = std::max(smq, std::min(smq + adj_sum_bytes(TYv, NCv, grads), kBlockedSmem));
      bool launched = false;
      const int virt = p->basis_nb ? 2 : p->adj_cls ? 1 : 0;
      const bool chain = p->adj_chain[pass];
      // the built-in rows per thread, and 2 rows where the built-in choice is 4
#define MRSIM_AQW(NQV, NCV, M, G, V, W)                                                 \
  if (NQv == NQV && NCv == NCV && maps == M && grads == G && virt == V && p->adj_narrow == W) { \
    if (TYv == adjq_rows_v(NCV, M, V) && !M && !W && chain) {                         \
      auto k = yadjoint_q_kernel<NQV, adjq_rows_v(NCV, M, V), NCV, M, G, V, W, !M && !W>;   \
      set_smem(k, smq);                                                                 \
      launch_chained(k, dim3((unsigned)R.n), smq, st, true, p->d_units, tiles);         \
      launched = true;                                                                  \
    } else if (TYv == adjq_rows_v(NCV, M, V)) {                                         \
      auto k = yadjoint_q_kernel<NQV, adjq_rows_v(NCV, M, V), NCV, M, G, V, W, false>;  \
      set_smem(k, smq);                                                                 \
      k<<<(unsigned)R.n, 256, smq, st>>>(p->d_units, tiles);                            \
      launched = true;                                                                  \
    } else if (!W && adjq_rows_v(NCV, M, V) == 4 && TYv == 2) {                         \
      auto k = yadjoint_q_kernel<NQV, 2, NCV, M, G, V, false, false>;                   \
      set_smem(k, smq);                                                                 \
      k<<<(unsigned)R.n, 256, smq, st>>>(p->d_units, tiles);                            \
      launched = true;                                                                  \
    }                                                                                   \
  }
#define MRSIM_AQV(NQV, NCV, M, G, V) MRSIM_AQW(NQV, NCV, M, G, V, false)
#define MRSIM_AQ(NQV, NCV, M, G) MRSIM_AQV(NQV, NCV, M, G, 0)
#define MRSIM_AQC(NCV, M, G) MRSIM_AQ(1, NCV, M, G) MRSIM_AQ(2, NCV, M, G) MRSIM_AQ(4, NCV, M, G) MRSIM_AQ(8, NCV, M, G)
#define MRSIM_AQN(M, G) MRSIM_AQC(1, M, G) MRSIM_AQC(2, M, G) MRSIM_AQC(3, M, G) MRSIM_AQC(4, M, G)
#define MRSIM_AQK(M, G) MRSIM_AQL(4, M, G) MRSIM_AQL(6, M, G) MRSIM_AQL(7, M, G) \
  MRSIM_AQV(6, 1, M, G, 1) MRSIM_AQV(6, 2, M, G, 1) MRSIM_AQV(6, 3, M, G, 1) MRSIM_AQV(6, 4, M, G, 1)
#define MRSIM_AQB(NQV, NCV, M, G) MRSIM_AQV(NQV, NCV, M, G, 2) MRSIM_AQW(NQV, NCV, M, G, 2, true)
#define MRSIM_AQL(NQV, M, G) MRSIM_AQB(NQV, 1, M, G) MRSIM_AQB(NQV, 2, M, G) MRSIM_AQB(NQV, 3, M, G) MRSIM_AQB(NQV, 4, M, G)
      MRSIM_AQN(false, false) MRSIM_AQN(true, false) MRSIM_AQN(false, true) MRSIM_AQN(true, true)
      MRSIM_AQC(8, false, false) MRSIM_AQC(8, false, true)
      MRSIM_AQK(false, false) MRSIM_AQK(true, false) MRSIM_AQK(false, true) MRSIM_AQK(true, true)
#undef MRSIM_AQK
#undef MRSIM_AQL
#undef MRSIM_AQB
#undef MRSIM_AQN
#undef MRSIM_AQC
#undef MRSIM_AQ
#undef MRSIM_AQV
#undef MRSIM_AQW
      if (!launched) fail("no adjoint kernel instance for this unit shape");
      MRSIM_CUDA(cudaGetLastError());
      continue;
    }
    size_t sm = sizeof(float2) * (size_t)2 * p->max_hchunk * 128 +
                sizeof(float) * ((size_t)kTY * (p->max_lines + p->max_coils) + 128 * (size_t)p->max_coils +
                                 (size_t)p->max_lines * (5 + NCv));
    bool launched = false;
#define MRSIM_A(NCV, M, G)                                                              \
  if (NCv == NCV && maps == M && grads == G) {                                          \
    auto k = yadjoint_kernel<kTY, NCV, M, G>;                                           \
    set_smem(k, sm);                                                                    \
    k<<<(unsigned)R.n, 128, sm, st>>>(p->d_units, tiles);                               \
    launched = true;                                                                    \
  }
#define MRSIM_AN(M, G) MRSIM_A(1, M, G) MRSIM_A(2, M, G) MRSIM_A(3, M, G) MRSIM_A(4, M, G) MRSIM_A(8, M, G)
    MRSIM_AN(false, false) MRSIM_AN(true, false) MRSIM_AN(false, true) MRSIM_AN(true, true)
#undef MRSIM_AN
#undef MRSIM_A
    if (!launched) fail("no adjoint kernel instance for this unit shape");
    MRSIM_CUDA(cudaGetLastError());
  }
}

}  // namespace mrsim
