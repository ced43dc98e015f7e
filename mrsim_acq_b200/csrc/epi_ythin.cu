// epi_ythin.cu — the y-stages of the EPI forward and adjoint for plans of few tiles (see epi_device.h).
#include "epi_device.h"

namespace mrsim {

namespace {

// The same sums for a plan of few tiles (thin_groups), without voxel maps and from 16-byte aligned rows:
// 32 columns x 4 G lines a block.  A warp has four of the lines and every (8 / G)-th row of a chunk: it
// forms their terms W P into shared memory; then each warp adds the chunk's terms of one line, in row
// order, to every coil or row (G = 1: to half of them).  The chain of a tile is thus its additions, not
// its rows' phases.
// One slice of one coil (64 lines on 128 x 128) is 8 tiles of the full kernel, 23 us; here 64 blocks.
// Bound by latency: two to four warps a scheduler, whose phases, exchange and additions alternate (4 slices
// of 8 coils: FMA pipe 20 %, shared memory 57 % of the cycles).
template <int G, int QG, int NV, int NC>
__global__ void __launch_bounds__(256, 2) ystage_thin_kernel(const UnitDesc* __restrict__ units,
                                                             const int4* __restrict__ tiles, int cls_rows) {
  constexpr int NA = NV ? NV : QG, QGP = (NA + 3) / 4 * 4, TL = 4 * G, CW = kThinCols, P = 8 / G;
  constexpr int CS = 2 / G, NO = (NA + CS - 1) / CS;  // warps per line of the additions, outputs of each
  constexpr int NPL = fwdq_planes(NC, false), RC = thin_rows(G);
  constexpr int STAGE = NPL * RC * CW, PIECES = STAGE / 4, PPT = (PIECES + 255) / 256;
  extern __shared__ __align__(16) float smem[];
  float* ring = smem;                                                    // [stage][plane][RC][CW]
  float2* terms = reinterpret_cast<float2*>(ring + kFwdStages * STAGE);   // [RC][TL][CW]
  grid_begin();
  const int4 tl = tiles[blockIdx.x];  // unit, line0, x0, q0
  const UnitDesc& u = units[tl.x];
  const int snx = u.snx, sny = u.sny, ncomp = u.ncomp, x0 = tl.z;
  float* Ey = reinterpret_cast<float*>(terms + RC * TL * CW);             // [sny][QGP]
  float* Bt = Ey + sny * QGP;                                            // [sny][TL]
  __shared__ const float* plane_s[NPL];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < NPL)
    plane_s[tid] = tid == 0          ? u.phase
                   : tid == 1        ? ((u.flags & UF_DISTORT) ? u.fmap : nullptr)
                   : tid - 2 < ncomp ? u.comp + (size_t)(tid - 2) * u.comp_stride
                                     : nullptr;
  const int nl = min(TL, u.n_lines - tl.y);
  const int ys = u.ny / 2, oy = sny / u.ny, sys = oy * ys;
  for (int idx = tid; idx < sny * TL; idx += 256) {
    const int y = idx / TL, j = idx % TL;
    float v = 0.f;
    if (j < nl) {
      const LineRec& L = u.lines[tl.y + j];
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
  for (int idx = tid; idx < QGP * sny; idx += 256) {
    const int y = idx / QGP, qq = idx % QGP;
    if (NV) {
      const int nc = u.geo.ncls;
      Ey[idx] = qq < nc ? u.geo.eyc[(size_t)qq * sny + y] : (qq == nc ? 1.f : 0.f);
    } else {
      const int q = tl.w + qq;
      Ey[idx] = (qq < QG && q < u.ncoils) ? u.geo.ey[(size_t)q * sny + y] : 0.f;
    }
  }
  // the lines whose terms this warp forms, and the line and outputs that it adds
  const int part = warp % P, jb = warp / P * 4, jl = warp / CS, o0 = warp % CS;
  float thi[4], tlo[4], rel[4][NC];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool have = jb + j < nl;
    const LineRec& L = u.lines[tl.y + (have ? jb + j : 0)];
    thi[j] = have ? L.t_hi : 0.f;
    tlo[j] = have ? L.t_lo : 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) rel[j][c] = have && c < ncomp ? L.rel[c] : 0.f;
  }
  const int x = x0 + lane;
  const bool xok = x < snx;
  const float off = u.geo.coil_off;
  float exq[NV ? 1 : NO];
  if (!NV) {
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      const int q = tl.w + o0 + o * CS;
      exq[NV ? 0 : o] = xok && q < u.ncoils ? u.geo.ex[(size_t)q * snx + x] : 0.f;
    }
  }
  const int nch = (sny + RC - 1) / RC;
  auto issue_rows = [&](int c) {
    if (c < nch) {
      float* dst = ring + (c % kFwdStages) * STAGE;
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int k = tid + 256 * i;
        if (PIECES % 256 == 0 || k < PIECES) {
          // absent planes, and rows or columns past the plane, zero-fill
          const float* base = plane_s[k / (RC * CW / 4)];
          const int y = c * RC + k / (CW / 4) % RC, xx = x0 + k % (CW / 4) * 4;
          const bool ok = base != nullptr && y < sny && xx < snx;
          cp_async16(dst + 4 * k, ok ? base + (size_t)y * snx + xx : (const float*)u.g, ok ? 16 : 0);
        }
      }
    }
    cp_async_commit();
  };
  __syncthreads();
  grid_wait();
#pragma unroll
  for (int c = 0; c < kFwdStages - 1; ++c) issue_rows(c);
  // block, blocks: the constant row's whole blocks of kConstBlock and of kConstBlocks rows
  float2 acc[NO], block = make_float2(0.f, 0.f), blocks = block;
#pragma unroll
  for (int o = 0; o < NO; ++o) acc[o] = make_float2(0.f, 0.f);
  const bool blocked = NV == 4 || NV == 7 || (NV && cls_rows == 2);  // (six rows may be class rows)
  for (int c = 0; c < nch; ++c) {
    cp_async_wait_n<kFwdStages - 2>();
    __syncthreads();  // rows of chunk c landed; every warp is done with chunk c - 1 and its terms
    issue_rows(c + kFwdStages - 1);
    const float* S = ring + (c % kFwdStages) * STAGE + lane;
#pragma unroll
    for (int i = 0; i < RC / P; ++i) {
      const int r = part + i * P;  // (a row past the last has zero planes; its terms are not added)
      const float4 b4 = *reinterpret_cast<const float4*>(Bt + min(c * RC + r, sny - 1) * TL + jb);
      const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
      const float2 a2 = dup2(S[r * CW]), f2 = dup2(S[(RC + r) * CW]);
      float m[NC];
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) m[cc] = S[((2 + cc) * RC + r) * CW];
      float2* w = terms + (r * TL + jb) * CW + lane;
#pragma unroll
      for (int jp = 0; jp < 4; jp += 2) {
        float2 th = phase_turns2(fadd2(a2, make_float2(bt[jp], bt[jp + 1])), f2, make_float2(thi[jp], thi[jp + 1]),
                                 make_float2(tlo[jp], tlo[jp + 1]));
        th = fmul2(dup2(kTwoPiF), th);
        float s0, c0, s1, c1;
        __sincosf(th.x, &s0, &c0);
        __sincosf(th.y, &s1, &c1);
        float2 W = fmul2(make_float2(rel[jp][0], rel[jp + 1][0]), dup2(m[0]));
#pragma unroll
        for (int cc = 1; cc < NC; ++cc) W = ffma2(make_float2(rel[jp][cc], rel[jp + 1][cc]), dup2(m[cc]), W);
        w[jp * CW] = fmul2(dup2(W.x), make_float2(c0, s0));
        w[(jp + 1) * CW] = fmul2(dup2(W.y), make_float2(c1, s1));
      }
    }
    __syncthreads();
    const float* e = Ey + c * RC * QGP + o0;
    const float2* w = terms + jl * CW + lane;
    const int rn = min(RC, sny - c * RC);
    auto add_row = [&](int r) {
      const float2 t = w[r * TL * CW];
#pragma unroll
      for (int o = 0; o < NO; ++o) {
        const int qq = o0 + o * CS;
        if (NV && qq == NA - 1)
          acc[o] = fadd2(acc[o], t);  // the offset or constant row is all ones
        else if (NA % CS == 0 || qq < NA)
          acc[o] = ffma2(dup2(NV ? e[r * QGP + o * CS] : fmaf(exq[NV ? 0 : o], e[r * QGP + o * CS], off)), t, acc[o]);
      }
    };
    for (int r = 0; r < rn; r += kConstBlock) {
      if (blocked)
#pragma unroll
        for (int o = 0; o < NO; ++o)
          if (o0 + o * CS == NA - 1) {
            block = fadd2(block, acc[o]);
            acc[o] = make_float2(0.f, 0.f);
            if ((c * RC + r) % kConstBlocks == 0) {
              blocks = fadd2(blocks, block);
              block = make_float2(0.f, 0.f);
            }
          }
      if (r + kConstBlock <= rn) {
#pragma unroll
        for (int k = 0; k < kConstBlock; ++k) add_row(r + k);
      } else {
        for (int k = r; k < rn; ++k) add_row(k);
      }
    }
  }
  cp_async_wait0();
  if (!xok || jl >= nl) return;
  const float s = u.signal_scale;
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int qq = o0 + o * CS, q = NV ? qq : tl.w + qq;
    if (qq >= NA || (!NV && q >= u.ncoils)) break;
    const float sv = NV && qq == NA - 1 && cls_rows == 1 ? s * off : s;
    const float2 t = blocked && qq == NA - 1 ? fadd2(blocks, fadd2(block, acc[o])) : acc[o];
    u.g[((size_t)q * u.n_lines + tl.y + jl) * snx + x] = make_float2(sv * t.x, sv * t.y);
  }
}

// The same sums for a plan of few tiles (thin_groups), without voxel maps and from 16-byte aligned rows
// of h: 32 columns x 4 G rows a block.  A warp has four of the rows and every (8 / G)-th line of a chunk:
// it forms their Z into shared memory; then each warp adds the chunk's lines of one row, in order, to the
// row's sums (G = 1: to the compartment gradients, or to the t- and trf-weighted sums).
// That slice is 16 tiles of the full kernel, 12 us with its x-stage; here 128 blocks, 7 us.
template <int G, int NQ, int NC, bool GRADS, int VIRT>
__global__ void __launch_bounds__(256, 2) yadjoint_thin_kernel(const UnitDesc* __restrict__ units,
                                                               const int4* __restrict__ tiles) {
  constexpr int CW = kThinCols, JL = kThinLines, NST = thin_stages(NQ), LF = adjq_line_floats(NC, false);
  constexpr int ROWS = 4 * G, P = 8 / G, CS = 2 / G;
  constexpr int STAGE = JL * NQ * CW, PIECES = STAGE / 2, PPT = PIECES / 256;
  static_assert(PIECES % 256 == 0 && JL % P == 0, "whole copies per thread, whole shares of a chunk");
  extern __shared__ __align__(16) float smem[];
  float2* ring = reinterpret_cast<float2*>(smem);  // [stage][line][coil or row][CW]
  float2* terms = ring + NST * STAGE;              // [JL][row][CW]
  grid_begin();
  const int4 tl = tiles[blockIdx.x];  // unit, y0, x0
  const UnitDesc& u = units[tl.x];
  const int snx = u.snx, sny = u.sny, ncomp = u.ncomp, nlines = u.n_lines, y0 = tl.y, x0 = tl.z;
  const int nchunks = (nlines + JL - 1) / JL, nlp = nchunks * JL;  // (zero entries past nlines)
  float* Lt = reinterpret_cast<float*>(terms + JL * ROWS * CW);  // [nlp][LF]
  float* Bt = Lt + nlp * LF;                                     // [nlp][ROWS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ys = u.ny / 2, oy = sny / u.ny, sys = oy * ys;
  for (int idx = tid; idx < nlp * ROWS; idx += 256) {
    const int j = idx / ROWS, y = y0 + idx % ROWS;
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
#pragma unroll
    for (int k = 0; k < LF; ++k) e[k] = 0.f;
    if (j >= nlines) continue;
    const LineRec& L = u.lines[j];
    const float tph = L.t_hi + L.t_lo;
    e[0] = L.t_hi;
    e[1] = L.t_lo;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float r = c < ncomp ? L.rel[c] : 0.f;
      e[4 + c] = r;
      e[4 + NC + c] = r * tph;
      e[4 + 2 * NC + c] = r * L.trf_ms;
    }
  }
  // the rows whose Z this warp forms, and the row and sums that it adds
  const int part = warp % P, rb = warp / P * 4, row = warp / CS, half = warp % CS;
  const int x = x0 + lane;
  const bool xok = x < snx;
  const int xs_ = xok ? x : 0;
  const float s = u.signal_scale, off = u.geo.coil_off;
  float amp[4][NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const float ex = VIRT ? 0.f : u.geo.ex[(size_t)q * snx + xs_];
#pragma unroll
    for (int ty = 0; ty < 4; ++ty) {
      const int y = min(y0 + rb + ty, sny - 1);
      if (VIRT)
        amp[ty][q] = q < NQ - 1 ? u.geo.eyc[(size_t)q * sny + y] : 1.f;
      else
        amp[ty][q] = s * fmaf(ex, u.geo.ey[(size_t)q * sny + y], off);
    }
  }
  auto issue_chunk = [&](int c) {
    if (c < nchunks) {
      float2* dst = ring + (c % NST) * STAGE;
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int k = tid + 256 * i, r = k / (CW / 2), xx = x0 + k % (CW / 2) * 2, j = c * JL + r / NQ;
        const bool in = xx < snx && j < nlines;
        cp_async16(dst + 2 * k, u.g + (in ? ((size_t)(r % NQ) * nlines + j) * snx + xx : 0), in ? 16 : 0);
      }
    }
    cp_async_commit();
  };
  grid_wait();
#pragma unroll
  for (int c = 0; c < NST - 1; ++c) issue_chunk(c);
  const bool distort = (u.flags & UF_DISTORT) != 0;
  float a[4], f[4];
#pragma unroll
  for (int ty = 0; ty < 4; ++ty) {
    const size_t i = (size_t)xs_ + (size_t)snx * min(y0 + rb + ty, sny - 1);
    a[ty] = u.phase ? u.phase[i] : 0.f;  // (see grid_wait)
    f[ty] = distort ? __ldg(u.fmap + i) : 0.f;
  }
  float2 cg[NC];
  float Uy[GRADS ? NC : 1], Vx[GRADS ? NC : 1];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    cg[c] = make_float2(0.f, 0.f);
    if (GRADS) Uy[GRADS ? c : 0] = Vx[GRADS ? c : 0] = 0.f;
  }
  // basis rows: the sums of whole blocks of kLineBlock lines (adj_blocked)
  static_assert(kLineBlock % JL == 0, "whole chunks in a block");
  const bool blocked = VIRT == 2 && adj_blocked(NQ, NC, false, GRADS, nlines);
  float2 wcg[NC];
  float wUy[GRADS ? NC : 1], wVx[GRADS ? NC : 1];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    wcg[c] = make_float2(0.f, 0.f);
    if (GRADS) wUy[GRADS ? c : 0] = wVx[GRADS ? c : 0] = 0.f;
  }
  auto fold = [&] {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      wcg[c] = fadd2(wcg[c], cg[c]);
      cg[c] = make_float2(0.f, 0.f);
      if (GRADS) {
        wUy[GRADS ? c : 0] += Uy[GRADS ? c : 0];
        wVx[GRADS ? c : 0] += Vx[GRADS ? c : 0];
        Uy[GRADS ? c : 0] = Vx[GRADS ? c : 0] = 0.f;
      }
    }
  };
  for (int c = 0; c < nchunks; ++c) {
    cp_async_wait_n<NST - 2>();
    __syncthreads();  // chunk c landed; every warp is done with chunk c - 1 and its terms
    issue_chunk(c + NST - 1);
    const float2* hs = ring + (c % NST) * STAGE + lane;
#pragma unroll
    for (int i = 0; i < JL / P; ++i) {
      const int jj = part + i * P, j = c * JL + jj;
      const float2 t = *reinterpret_cast<const float2*>(Lt + j * LF);
      const float4 b4 = *reinterpret_cast<const float4*>(Bt + j * ROWS + rb);
      const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
      float2 H[4];
      if (VIRT == 1) {  // as the full kernel: from the offset row (amplitude 1) on
        const float2 h = hs[(jj * NQ + NQ - 1) * CW];
#pragma unroll
        for (int ty = 0; ty < 4; ++ty) H[ty] = h;
      } else {
        const float2 h = hs[jj * NQ * CW];
#pragma unroll
        for (int ty = 0; ty < 4; ++ty) H[ty] = fmul2(dup2(amp[ty][0]), h);
      }
#pragma unroll
      for (int q = VIRT == 1 ? 0 : 1; q < (VIRT ? NQ - 1 : NQ); ++q) {
        const float2 h = hs[(jj * NQ + q) * CW];
#pragma unroll
        for (int ty = 0; ty < 4; ++ty) H[ty] = ffma2(dup2(amp[ty][q]), h, H[ty]);
      }
      if (VIRT == 2) {  // the constant row last
        const float2 h = hs[(jj * NQ + NQ - 1) * CW];
#pragma unroll
        for (int ty = 0; ty < 4; ++ty) H[ty] = fadd2(H[ty], h);
      }
#pragma unroll
      for (int tp = 0; tp < 4; tp += 2) {
        float2 th = phase_turns2(fadd2(make_float2(a[tp], a[tp + 1]), make_float2(bt[tp], bt[tp + 1])),
                                 make_float2(f[tp], f[tp + 1]), dup2(t.x), dup2(t.y));
        th = fmul2(dup2(kTwoPiF), th);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          float sn, cs;
          __sincosf(k ? th.y : th.x, &sn, &cs);
          const float2 h = H[tp + k];
          terms[(jj * ROWS + rb + tp + k) * CW + lane] = make_float2(fmaf(cs, h.x, sn * h.y), fmaf(cs, h.y, -sn * h.x));
        }
      }
    }
    __syncthreads();
    const float2* z = terms + row * CW + lane;
    const float* e = Lt + c * JL * LF + 4;
    if (blocked && c * JL % kLineBlock == 0) fold();
    if (half == 0) {
#pragma unroll
      for (int jj = 0; jj < JL; ++jj) {
        const float2 v = z[jj * ROWS * CW];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) cg[cc] = ffma2(dup2(e[jj * LF + cc]), v, cg[cc]);
      }
    }
    if (GRADS && half == CS - 1) {
#pragma unroll
      for (int jj = 0; jj < JL; ++jj) {
        const float2 v = z[jj * ROWS * CW];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          Uy[GRADS ? cc : 0] = fmaf(e[jj * LF + NC + cc], v.y, Uy[GRADS ? cc : 0]);
          Vx[GRADS ? cc : 0] = fmaf(e[jj * LF + 2 * NC + cc], v.x, Vx[GRADS ? cc : 0]);
        }
      }
    }
  }
  cp_async_wait0();
  if (!xok || y0 + row >= sny) return;
  if (blocked) {
    fold();
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      cg[c] = wcg[c];
      if (GRADS) {
        Uy[GRADS ? c : 0] = wUy[GRADS ? c : 0];
        Vx[GRADS ? c : 0] = wVx[GRADS ? c : 0];
      }
    }
  }
  const size_t plane = (size_t)snx * sny, i = (size_t)x + (size_t)snx * (y0 + row);
  float fg = 0.f;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (c >= ncomp) break;
    if (half == 0) u.comp_grad[c * plane + i] = cg[c];
    if (GRADS && half == CS - 1) {
      const float m = __ldg(u.comp + (size_t)c * u.comp_stride + i);
      fg = fmaf(m, Uy[GRADS ? c : 0], fg);
      if (u.r2_grad) u.r2_grad[c * plane + i] = -2.0f * m * Vx[GRADS ? c : 0];
    }
  }
  if (GRADS && half == CS - 1 && u.fmap_grad) u.fmap_grad[i] = distort ? 4.0f * 3.14159265358979f * fg : 0.f;
}

}  // namespace

void launch_ystage_thin(const EpiPlan* p, int pass, const int4* tiles, int n, cudaStream_t st) {
  const int G = p->fwd_thin[pass], QG = p->qg, NVv = p->fwd_nv[pass], NCv = p->nc, kind = p->basis_nb ? 2 : p->fwd_cls ? 1 : 0;
  const size_t sm = ystage_thin_smem(G, NCv, QG, p->max_sny);
  bool launched = false;
#define MRSIM_YT(QGV, NVV, NCV)                                                                          \
  if (QG == QGV && NVv == NVV && NCv == NCV) {                                                           \
    auto k = G == 1 ? ystage_thin_kernel<1, QGV, NVV, NCV> : ystage_thin_kernel<2, QGV, NVV, NCV>;       \
    set_smem(k, sm);                                                                                     \
    launch_chained(k, dim3((unsigned)n), sm, st, true, p->d_units, tiles, kind);                         \
    launched = true;                                                                                     \
  }
#define MRSIM_YTQ(NCV) MRSIM_YT(1, 0, NCV) MRSIM_YT(2, 0, NCV) MRSIM_YT(4, 0, NCV) MRSIM_YT(8, 0, NCV)
#define MRSIM_YTV(NVV) MRSIM_YT(8, NVV, 1) MRSIM_YT(8, NVV, 2) MRSIM_YT(8, NVV, 3) MRSIM_YT(8, NVV, 4)
  MRSIM_YTQ(1) MRSIM_YTQ(2) MRSIM_YTQ(3) MRSIM_YTQ(4) MRSIM_YTQ(8)
  MRSIM_YTV(4) MRSIM_YTV(6) MRSIM_YTV(7)
#undef MRSIM_YTV
#undef MRSIM_YTQ
#undef MRSIM_YT
  if (!launched) fail("no forward kernel instance for this unit shape");
  MRSIM_CUDA(cudaGetLastError());
}

void launch_yadjoint_thin(const EpiPlan* p, int pass, const int4* tiles, int n, cudaStream_t st) {
  const int G = p->adj_thin[pass], NQv = p->adjq[pass], NCv = p->nc;
  const bool grads = (pass & 2) != 0;
  const int virt = p->basis_nb ? 2 : p->adj_cls ? 1 : 0;
  const size_t sm = yadjoint_thin_smem(G, NQv, NCv, p->max_lines);
  bool launched = false;
#define MRSIM_AT(NQV, NCV, GR, V)                                                                        \
  if (NQv == NQV && NCv == NCV && grads == GR && virt == V) {                                            \
    auto k = G == 1 ? yadjoint_thin_kernel<1, NQV, NCV, GR, V> : yadjoint_thin_kernel<2, NQV, NCV, GR, V>;  \
    set_smem(k, sm);                                                                                     \
    launch_chained(k, dim3((unsigned)n), sm, st, true, p->d_units, tiles);                               \
    launched = true;                                                                                     \
  }
#define MRSIM_ATC(NCV, GR) MRSIM_AT(1, NCV, GR, 0) MRSIM_AT(2, NCV, GR, 0) MRSIM_AT(4, NCV, GR, 0) MRSIM_AT(8, NCV, GR, 0)
#define MRSIM_ATV(NCV, GR) MRSIM_AT(6, NCV, GR, 1) MRSIM_AT(4, NCV, GR, 2) MRSIM_AT(6, NCV, GR, 2) MRSIM_AT(7, NCV, GR, 2)
#define MRSIM_ATN(GR) MRSIM_ATC(1, GR) MRSIM_ATC(2, GR) MRSIM_ATC(3, GR) MRSIM_ATC(4, GR) MRSIM_ATC(8, GR) \
  MRSIM_ATV(1, GR) MRSIM_ATV(2, GR) MRSIM_ATV(3, GR) MRSIM_ATV(4, GR)
  MRSIM_ATN(false) MRSIM_ATN(true)
#undef MRSIM_ATN
#undef MRSIM_ATV
#undef MRSIM_ATC
#undef MRSIM_AT
  if (!launched) fail("no adjoint kernel instance for this unit shape");
  MRSIM_CUDA(cudaGetLastError());
}

}  // namespace mrsim
