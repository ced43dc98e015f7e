// epi_ystage.cu — the y-stage of the EPI forward (see epi_kernels.cu) and its launcher.
#include "epi_device.h"

namespace mrsim {

namespace {

// ---------------------------------------------------------------------------------------------
// y-stage of the forward.  One CTA = (unit, T lines, 128 columns, QG coils); one thread per
// column x accumulates T*QG complex sums over every sim row y.
struct Tile {
  int unit, line0, x0, q0;
};

template <int T, int QG, int NC, bool MAPS>
__global__ void __launch_bounds__(128, 4) ystage_kernel(const UnitDesc* __restrict__ units,
                                                        const Tile* __restrict__ tiles) {
  // A CTA of 128 threads: one column each, T lines x QG coils per thread.
  constexpr int LG = 1;
  constexpr int TL = LG * T;  // lines per CTA
  static_assert(T == 4, "the phase table is read as float4");
  extern __shared__ __align__(16) float smem[];
  const Tile tl = tiles[blockIdx.x];
  const UnitDesc& u = units[tl.unit];
  const int snx = u.snx, sny = u.sny;
  const int ncomp = u.ncomp;
  float* Bt = smem;                 // [sny][TL] phase terms per (row, line)
  float* Ey = smem + sny * TL;      // [sny][QGP] (QGP = QG rounded up to 4)
  constexpr int QGP = (QG + 3) / 4 * 4;
  __shared__ float rel_s[TL][kMaxComp];
  __shared__ float tinh_s[TL], trf_s[TL];
  __shared__ float thi_s[TL], tlo_s[TL];

  const int nl = min(TL, u.n_lines - tl.line0);
  const int ys = u.ny / 2;
  const int oy = sny / u.ny;
  const int sys = oy * ys;
  for (int idx = threadIdx.x; idx < sny * TL; idx += blockDim.x) {
    const int y = idx / TL, j = idx % TL;
    float v = 0.f;
    if (j < nl) {
      const LineRec& L = u.lines[tl.line0 + j];
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
  for (int idx = threadIdx.x; idx < QGP * sny; idx += blockDim.x) {
    const int y = idx / QGP, qq = idx % QGP;
    const int q = tl.q0 + qq;
    Ey[idx] = (qq < QG && q < u.ncoils) ? u.geo.ey[(size_t)q * sny + y] : 0.f;
  }
  if (threadIdx.x < TL) {
    const int j = threadIdx.x;
    if (j < nl) {
      const LineRec& L = u.lines[tl.line0 + j];
      thi_s[j] = L.t_hi;
      tlo_s[j] = L.t_lo;
      tinh_s[j] = L.inhom_ms;
      trf_s[j] = L.trf_ms;
      for (int c = 0; c < kMaxComp; ++c) rel_s[j][c] = L.rel[c];
    } else {
      thi_s[j] = tlo_s[j] = tinh_s[j] = trf_s[j] = 0.f;
      for (int c = 0; c < kMaxComp; ++c) rel_s[j][c] = 0.f;
    }
  }
  __syncthreads();

  const int col = threadIdx.x & 127, lg = threadIdx.x >> 7;
  const int jb = lg * T;  // this thread's first line within the CTA
  const int x = tl.x0 + col;
  const bool xok = x < snx;
  const int xs_ = xok ? x : 0;
  float exq[QG];
  const float off = u.geo.coil_off;
#pragma unroll
  for (int qq = 0; qq < QG; ++qq) {
    const int q = tl.q0 + qq;
    exq[qq] = (xok && q < u.ncoils) ? u.geo.ex[(size_t)q * snx + x] : 0.f;
  }
  float thi[T], tlo[T], relr[T][NC];
#pragma unroll
  for (int j = 0; j < T; ++j) {
    thi[j] = thi_s[jb + j];
    tlo[j] = tlo_s[jb + j];
#pragma unroll
    for (int c = 0; c < NC; ++c) relr[j][c] = rel_s[jb + j][c];
  }
  float2 acc[T][QG];
#pragma unroll
  for (int j = 0; j < T; ++j)
#pragma unroll
    for (int qq = 0; qq < QG; ++qq) acc[j][qq] = make_float2(0.f, 0.f);

  const bool distort = (u.flags & UF_DISTORT) != 0;
  const float* __restrict__ comp = u.comp;
  const float* __restrict__ fmap = u.fmap;
  const float* __restrict__ phase = u.phase;
  // row y's inputs, prefetched one row ahead
  float na = 0.f, nf = 0.f, nm[NC];
  {
    const int i = xs_;
    na = phase ? __ldg(phase + i) : 0.f;
    nf = distort ? __ldg(fmap + i) : 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) nm[c] = c < ncomp ? __ldg(comp + (size_t)c * u.comp_stride + i) : 0.f;
  }
  for (int y = 0; y < sny; ++y) {
    const int i = xs_ + snx * y;
    const float a = na, f = nf;
    float m[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) m[c] = nm[c];
    if (y + 1 < sny) {
      const int i1 = i + snx;
      na = phase ? __ldg(phase + i1) : 0.f;
      nf = distort ? __ldg(fmap + i1) : 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) nm[c] = c < ncomp ? __ldg(comp + (size_t)c * u.comp_stride + i1) : 0.f;
    }
    float r2[MAPS ? NC : 1], r2i[MAPS ? NC : 1];
    float la = 0.f;
    if (MAPS) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        r2[MAPS ? c : 0] = r2i[MAPS ? c : 0] = 0.f;
        if (c < ncomp) {
          const float t2 = u.t2map ? __ldg(u.t2map + (size_t)c * u.map_stride + i) : u.t2u[c];
          const float ti = u.timap ? __ldg(u.timap + (size_t)c * u.map_stride + i) : u.tiu[c];
          r2[MAPS ? c : 0] = 1.0f / t2;
          r2i[MAPS ? c : 0] = 1.0f / ti;
        }
      }
      if (u.log_amp) la = __ldg(u.log_amp + i);
    }
    float amp[QG];
#pragma unroll
    for (int q4 = 0; q4 < QGP; q4 += 4) {
      const float4 e4 = *reinterpret_cast<const float4*>(Ey + y * QGP + q4);
      const float ev[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (q4 + k < QG) amp[q4 + k] = fmaf(exq[q4 + k], ev[k], off);
    }
    const float4 b4 = *reinterpret_cast<const float4*>(Bt + y * TL + jb);
    const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
    for (int j = 0; j < T; ++j) {
      const float th = phase_turns(a + bt[j], f, thi[j], tlo[j]);
      float sn, cs;
      __sincosf(kTwoPiF * th, &sn, &cs);
      float W = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (c < ncomp) {
          float r;
          if (MAPS)
            r = __expf(la - trf_s[jb + j] * r2[MAPS ? c : 0] - tinh_s[jb + j] * r2i[MAPS ? c : 0]);
          else
            r = relr[j][c];
          W = fmaf(r, m[c], W);
        }
      }
      const float wr = W * cs, wi = W * sn;
#pragma unroll
      for (int qq = 0; qq < QG; ++qq) {
        acc[j][qq].x = fmaf(amp[qq], wr, acc[j][qq].x);
        acc[j][qq].y = fmaf(amp[qq], wi, acc[j][qq].y);
      }
    }
  }
  if (!xok) return;
  const float s = u.signal_scale;
#pragma unroll
  for (int qq = 0; qq < QG; ++qq) {
    const int q = tl.q0 + qq;
    if (q >= u.ncoils) break;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      if (jb + j < nl)
        u.g[((size_t)q * u.n_lines + tl.line0 + jb + j) * snx + x] = make_float2(acc[j][qq].x * s, acc[j][qq].y * s);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// y-stage of the forward with the per-row inputs staged in shared memory (every unit of the plan
// has snx % 4 == 0 and 16-byte aligned input planes).  Same sums as ystage_kernel:
//   * a CTA of 256 threads covers 128 columns x 8 lines (two groups of 4 lines, one column each)
//     x QG coils, so each row's inputs serve 8 lines;
//   * the inputs of RC rows (static phase, fieldmap, compartments, and with voxel maps T2, T2',
//     log amplitude) arrive through a 3-stage ring filled by cooperative 16-byte cp.async, one
//     barrier per RC rows, in place of per-thread global loads one row ahead.
// NV > 0: the tile holds every coil of the unit and accumulates coil classes instead of coils
// (NV = classes + 1 for the coil offset): acc_v += ey_v(y) W P, acc_off += W P, and the epilogue
// expands g_q = s (ex_q acc_cls(q) + off acc_off).
// cls_rows (with NV): 1 writes the class rows G_v = s T_v and G_off = s off T_off ([v][line][x],
// the layout the class-mode x-stage expands) instead of the coil rows; 2 writes basis rows (the
// unit's eyc holds the coil basis, whose last row is constant), G_v = s T_v for every row.
// NARROW: some plane or row is not on a 16-byte boundary, so the ring fills by 4-byte copies.
// CHAIN: a small launch, chained to the kernel before it.
template <int QG, int NV, int NC, bool MAPS, bool NARROW, bool CHAIN>
__global__ void __launch_bounds__(256, 2) ystage_q_kernel(const UnitDesc* __restrict__ units,
                                                          const Tile* __restrict__ tiles, int cls_rows) {
  constexpr int T = 4, TL = 8;
  constexpr int NA = NV ? NV : QG;             // accumulators per line
  constexpr int NPL = fwdq_planes(NC, MAPS);
  constexpr int RC = fwdq_rows(NC, MAPS);
  static_assert(kConstBlock % RC == 0, "whole chunks in a block");
  constexpr int STAGE = NPL * RC * 128;        // floats per stage
  constexpr int PIECES = NPL * RC * 32;        // 16-byte pieces per stage
  constexpr int PPT = (PIECES + 255) / 256;
  constexpr int QGP = (NA + 3) / 4 * 4;
  // plane order: 0 static phase, 1 fieldmap, 2.. compartments, then T2, T2' maps and log amplitude
  constexpr int P_COMP = 2, P_T2 = 2 + NC, P_TI = 2 + 2 * NC, P_LA = 2 + 3 * NC;
  extern __shared__ __align__(16) float smem[];
  float* ring = smem;                           // [stage][plane][RC][128]
  float* Bt = ring + kFwdStages * STAGE;        // [sny][TL]
  if (CHAIN) grid_begin();
  const Tile tl = tiles[blockIdx.x];
  const UnitDesc& u = units[tl.unit];
  const int snx = u.snx, sny = u.sny, ncomp = u.ncomp;
  float* Ey = Bt + sny * TL;                    // [sny][QGP]: ey per coil, or per class and 1
  // basis rows: the constant row's whole blocks, of kConstBlock and of kConstBlocks rows, [line][thread]
  float2* const whole = reinterpret_cast<float2*>(Ey + sny * QGP);
  const bool blocked = NV == 4 || NV == 7 || (NV && cls_rows == 2);  // (six rows may be class rows)
  __shared__ const float* plane_s[NPL];
  __shared__ float rel_s[TL][kMaxComp];
  __shared__ float tinh_s[TL], trf_s[TL], thi_s[TL], tlo_s[TL];
  const int tid = threadIdx.x;
  const bool distort = (u.flags & UF_DISTORT) != 0;
  if (tid < NPL) {
    const float* pp = nullptr;
    const int k = tid;
    if (k == 0) pp = u.phase;
    else if (k == 1) pp = distort ? u.fmap : nullptr;
    else if (k < P_T2) pp = (k - P_COMP) < ncomp ? u.comp + (size_t)(k - P_COMP) * u.comp_stride : nullptr;
    else if (k < P_TI) pp = ((k - P_T2) < ncomp && u.t2map) ? u.t2map + (size_t)(k - P_T2) * u.map_stride : nullptr;
    else if (k < P_LA) pp = ((k - P_TI) < ncomp && u.timap) ? u.timap + (size_t)(k - P_TI) * u.map_stride : nullptr;
    else pp = u.log_amp;
    plane_s[k] = pp;
  }
  __syncthreads();
  const int x0 = tl.x0;
  const int nch = (sny + RC - 1) / RC;
  auto issue_rows = [&](int c) {
    if (NARROW && c < nch) {
      float* dst = ring + (c % kFwdStages) * STAGE;
      for (int k = tid; k < STAGE; k += 256) {
        const int pl = k / (RC * 128), r = (k / 128) % RC, xx = x0 + (k & 127), y = c * RC + r;
        const float* base = plane_s[pl];
        const bool ok = base != nullptr && y < sny && xx < snx;
        cp_async4(dst + k, ok ? base + (size_t)y * snx + xx : (const float*)u.g, ok ? 4 : 0);
      }
    } else if (c < nch) {
      float* dst = ring + (c % kFwdStages) * STAGE;
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int k = tid + 256 * i;
        if (PIECES % 256 == 0 || k < PIECES) {
          const int pl = k / (RC * 32), rem = k % (RC * 32);
          const int r = rem >> 5, c4 = (rem & 31) * 4;
          // absent planes (no static phase, no distortion, compartments past ncomp) and rows
          // or columns past the plane zero-fill: the row loop reads every plane unconditionally
          const float* base = plane_s[pl];
          const int y = c * RC + r, xx = x0 + c4;
          const bool ok = base != nullptr && y < sny && xx < snx;
          cp_async16(dst + (pl * RC + r) * 128 + c4, ok ? base + (size_t)y * snx + xx : (const float*)u.g, ok ? 16 : 0);
        }
      }
    }
    cp_async_commit();
  };
  // the first rows fly while the tables fill; a small launch fills its tables while the kernel before
  // it still runs instead
  if (!CHAIN) {
#pragma unroll
    for (int c = 0; c < kFwdStages - 1; ++c) issue_rows(c);
  }

  const int nl = min(TL, u.n_lines - tl.line0);
  const int ys = u.ny / 2;
  const int oy = sny / u.ny;
  const int sys = oy * ys;
  for (int idx = tid; idx < sny * TL; idx += 256) {
    const int y = idx / TL, j = idx % TL;
    float v = 0.f;
    if (j < nl) {
      const LineRec& L = u.lines[tl.line0 + j];
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
      const int q = tl.q0 + qq;
      Ey[idx] = (qq < QG && q < u.ncoils) ? u.geo.ey[(size_t)q * sny + y] : 0.f;
    }
  }
  if (tid < TL) {
    const int j = tid;
    if (j < nl) {
      const LineRec& L = u.lines[tl.line0 + j];
      thi_s[j] = L.t_hi;
      tlo_s[j] = L.t_lo;
      tinh_s[j] = L.inhom_ms;
      trf_s[j] = L.trf_ms;
      for (int c = 0; c < kMaxComp; ++c) rel_s[j][c] = c < ncomp ? L.rel[c] : 0.f;
    } else {
      thi_s[j] = tlo_s[j] = tinh_s[j] = trf_s[j] = 0.f;
      for (int c = 0; c < kMaxComp; ++c) rel_s[j][c] = 0.f;
    }
  }
  if (CHAIN) {
    grid_wait();
#pragma unroll
    for (int c = 0; c < kFwdStages - 1; ++c) issue_rows(c);
  }
  __syncthreads();

  const int col = tid & 127, lg = tid >> 7;
  const int jb = lg * T;
  const int x = x0 + col;
  const bool xok = x < snx;
  const float off = u.geo.coil_off;
  float exq[NV ? 1 : QG];
  if (!NV) {
#pragma unroll
    for (int qq = 0; qq < QG; ++qq) {
      const int q = tl.q0 + qq;
      exq[NV ? 0 : qq] = (xok && q < u.ncoils) ? u.geo.ex[(size_t)q * snx + x] : 0.f;
    }
  }
  float thi[T], tlo[T], relr[T][MAPS ? 1 : NC], trf[MAPS ? T : 1], tinh[MAPS ? T : 1];
#pragma unroll
  for (int j = 0; j < T; ++j) {
    thi[j] = thi_s[jb + j];
    tlo[j] = tlo_s[jb + j];
    if (MAPS) {
      trf[MAPS ? j : 0] = trf_s[jb + j];
      tinh[MAPS ? j : 0] = tinh_s[jb + j];
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) relr[j][MAPS ? 0 : c] = rel_s[jb + j][c];
    }
  }
  const bool has_t2 = MAPS && plane_s[P_T2] != nullptr, has_ti = MAPS && plane_s[P_TI] != nullptr;
  const bool has_la = MAPS && plane_s[P_LA] != nullptr;
  float2 acc[T][NA];
#pragma unroll
  for (int j = 0; j < T; ++j)
#pragma unroll
    for (int qq = 0; qq < NA; ++qq) acc[j][qq] = make_float2(0.f, 0.f);
  if (blocked)
#pragma unroll
    for (int j = 0; j < 2 * T; ++j) whole[j * 256 + tid] = make_float2(0.f, 0.f);

  for (int c = 0; c < nch; ++c) {
    cp_async_wait_n<kFwdStages - 2>();
    __syncthreads();  // rows of chunk c landed; every thread is done with chunk c - 1
    if (blocked && c * RC % kConstBlock == 0)
#pragma unroll
      for (int j = 0; j < T; ++j) {
        float2 b = fadd2(whole[j * 256 + tid], acc[j][NA - 1]);
        acc[j][NA - 1] = make_float2(0.f, 0.f);
        if (c * RC % kConstBlocks == 0) {
          whole[(T + j) * 256 + tid] = fadd2(whole[(T + j) * 256 + tid], b);
          b = make_float2(0.f, 0.f);
        }
        whole[j * 256 + tid] = b;
      }
    issue_rows(c + kFwdStages - 1);
    const float* S = ring + (c % kFwdStages) * STAGE + col;
    const int rn = min(RC, sny - c * RC);
    for (int r = 0; r < rn; ++r) {
      const int y = c * RC + r;
      const float a = S[(0 * RC + r) * 128];
      const float f = S[(1 * RC + r) * 128];
      float m[NC];
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) m[cc] = S[((P_COMP + cc) * RC + r) * 128];
      float r2[MAPS ? NC : 1], r2i[MAPS ? NC : 1];
      float la = 0.f;
      if (MAPS) {
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          r2[MAPS ? cc : 0] = r2i[MAPS ? cc : 0] = 0.f;
          if (cc < ncomp) {
            const float t2 = has_t2 ? S[((P_T2 + cc) * RC + r) * 128] : u.t2u[cc];
            const float ti = has_ti ? S[((P_TI + cc) * RC + r) * 128] : u.tiu[cc];
            r2[MAPS ? cc : 0] = 1.0f / t2;
            r2i[MAPS ? cc : 0] = 1.0f / ti;
          }
        }
        if (has_la) la = S[(P_LA * RC + r) * 128];
      }
      float amp[NA];
#pragma unroll
      for (int q4 = 0; q4 < QGP; q4 += 4) {
        const float4 e4 = *reinterpret_cast<const float4*>(Ey + y * QGP + q4);
        const float ev[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (q4 + k < NA) amp[q4 + k] = NV ? ev[k] : fmaf(exq[NV ? 0 : q4 + k], ev[k], off);
      }
      const float4 b4 = *reinterpret_cast<const float4*>(Bt + y * TL + jb);
      const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
      if (NV && !MAPS) {
        // lines (0, 1) and (2, 3) as packed pairs: the same arithmetic, two lanes per instruction
        const float2 a2 = dup2(a), f2 = dup2(f);
#pragma unroll
        for (int jp = 0; jp < T; jp += 2) {
          float2 th = phase_turns2(fadd2(a2, make_float2(bt[jp], bt[jp + 1])), f2,
                                   make_float2(thi[jp], thi[jp + 1]), make_float2(tlo[jp], tlo[jp + 1]));
          th = fmul2(dup2(kTwoPiF), th);
          float s0, c0, s1, c1;
          __sincosf(th.x, &s0, &c0);
          __sincosf(th.y, &s1, &c1);
          float2 W = fmul2(make_float2(relr[jp][MAPS ? 0 : 0], relr[jp + 1][MAPS ? 0 : 0]), dup2(m[0]));
#pragma unroll
          for (int cc = 1; cc < NC; ++cc)
            W = ffma2(make_float2(relr[jp][MAPS ? 0 : cc], relr[jp + 1][MAPS ? 0 : cc]), dup2(m[cc]), W);
          const float2 w0 = fmul2(dup2(W.x), make_float2(c0, s0)), w1 = fmul2(dup2(W.y), make_float2(c1, s1));
#pragma unroll
          for (int qq = 0; qq < NA - 1; ++qq) {
            acc[jp][qq] = ffma2(dup2(amp[qq]), w0, acc[jp][qq]);
            acc[jp + 1][qq] = ffma2(dup2(amp[qq]), w1, acc[jp + 1][qq]);
          }
          acc[jp][NA - 1] = fadd2(acc[jp][NA - 1], w0);
          acc[jp + 1][NA - 1] = fadd2(acc[jp + 1][NA - 1], w1);
        }
        continue;
      }
#pragma unroll
      for (int j = 0; j < T; ++j) {
        const float th = phase_turns(a + bt[j], f, thi[j], tlo[j]);
        float sn, cs;
        __sincosf(kTwoPiF * th, &sn, &cs);
        float W = 0.f;
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
          if (!MAPS || cc < ncomp) {  // class decay: rel and m are 0 past ncomp
            float rr;
            if (MAPS)
              rr = __expf(la - trf[MAPS ? j : 0] * r2[MAPS ? cc : 0] - tinh[MAPS ? j : 0] * r2i[MAPS ? cc : 0]);
            else
              rr = relr[j][MAPS ? 0 : cc];
            W = fmaf(rr, m[cc], W);
          }
        }
        const float wr = W * cs, wi = W * sn;
#pragma unroll
        for (int qq = 0; qq < NA; ++qq) {
          if (NV && qq == NA - 1) {  // the coil-offset row is all ones
            acc[j][qq].x += wr;
            acc[j][qq].y += wi;
          } else if (NV) {
            acc[j][qq] = ffma2(make_float2(amp[qq], amp[qq]), make_float2(wr, wi), acc[j][qq]);
          } else {
            acc[j][qq].x = fmaf(amp[qq], wr, acc[j][qq].x);
            acc[j][qq].y = fmaf(amp[qq], wi, acc[j][qq].y);
          }
        }
      }
    }
  }
  cp_async_wait0();
  if (!xok) return;
  if (blocked)
#pragma unroll
    for (int j = 0; j < T; ++j)
      acc[j][NA - 1] = fadd2(whole[(T + j) * 256 + tid], fadd2(whole[j * 256 + tid], acc[j][NA - 1]));
  const float s = u.signal_scale;
  if (NV && cls_rows) {
#pragma unroll
    for (int j = 0; j < T; ++j) {
      if (jb + j >= nl) break;
#pragma unroll
      for (int v = 0; v < NA; ++v) {
        const float sv = v == NA - 1 && cls_rows == 1 ? s * off : s;
        u.g[((size_t)v * u.n_lines + tl.line0 + jb + j) * snx + x] = make_float2(sv * acc[j][v].x, sv * acc[j][v].y);
      }
    }
    return;
  }
  if (NV) {
    // expand the classes to the unit's coils (all in this tile)
    for (int q = 0; q < u.ncoils; ++q) {
      const int cl = u.geo.cls[q];
      const float e = s * u.geo.ex[(size_t)q * snx + x], o = s * off;
#pragma unroll
      for (int j = 0; j < T; ++j) {
        float2 v = acc[j][0];
#pragma unroll
        for (int k = 1; k < NA - 1; ++k)
          if (cl == k) v = acc[j][k];
        if (jb + j < nl)
          u.g[((size_t)q * u.n_lines + tl.line0 + jb + j) * snx + x] =
              make_float2(fmaf(e, v.x, o * acc[j][NA - 1].x), fmaf(e, v.y, o * acc[j][NA - 1].y));
      }
    }
    return;
  }
#pragma unroll
  for (int qq = 0; qq < QG; ++qq) {
    const int q = tl.q0 + qq;
    if (q >= u.ncoils) break;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      if (jb + j < nl)
        u.g[((size_t)q * u.n_lines + tl.line0 + jb + j) * snx + x] = make_float2(acc[j][qq].x * s, acc[j][qq].y * s);
    }
  }
}

}  // namespace

void epi_plan_forward_ystage(const EpiPlan* p, cudaStream_t st, int u0, int u1) {
  for (int pass = 0; pass < 2; ++pass) {
    const TileRange R = tile_range(p->y_start[pass], p->n_ytiles[pass], u0, u1);
    if (R.n == 0) continue;
    const Tile* tiles = (const Tile*)p->d_ytiles[pass] + R.t0;
    const bool maps = pass == 1;
    const int QG = p->qg, NCv = p->nc;
    if (p->fwd_thin[pass]) {
      launch_ystage_thin(p, pass, p->d_ytiles[pass] + R.t0, R.n, st);
      continue;
    }
    if (p->fwdq[pass]) {
      const size_t smq = ystage_q_smem(NCv, maps, QG, p->max_sny, p->basis_nb > 0);
      bool launched = false;
      const int NVv = p->fwd_nv[pass];
      const bool narrow = p->fwd_narrow[pass];
      const bool chain = p->fwd_chain[pass];
      const int rows_kind = p->basis_nb ? 2 : p->fwd_cls ? 1 : 0;
#define MRSIM_YFW(QGV, NVV, NCV, M, W)                                                  \
  if (QG == QGV && NVv == NVV && NCv == NCV && maps == M && narrow == W) {              \
    if (!M && !W && chain) {                                                          \
      auto k = ystage_q_kernel<QGV, NVV, NCV, M, W, !M && !W>;                          \
      set_smem(k, smq);                                                                 \
      launch_chained(k, dim3((unsigned)R.n), smq, st, true, p->d_units, tiles, rows_kind);  \
    } else {                                                                            \
      auto k = ystage_q_kernel<QGV, NVV, NCV, M, W, false>;                             \
      set_smem(k, smq);                                                                 \
      k<<<(unsigned)R.n, 256, smq, st>>>(p->d_units, tiles, rows_kind);                 \
    }                                                                                   \
    launched = true;                                                                    \
  }
#define MRSIM_YF(QGV, NVV, NCV, M) MRSIM_YFW(QGV, NVV, NCV, M, false)
#define MRSIM_YFB(NVV) MRSIM_YFW(8, NVV, 1, false, true) MRSIM_YFW(8, NVV, 2, false, true) \
  MRSIM_YFW(8, NVV, 3, false, true) MRSIM_YFW(8, NVV, 4, false, true) MRSIM_YFW(8, NVV, 1, true, true) \
  MRSIM_YFW(8, NVV, 2, true, true) MRSIM_YFW(8, NVV, 3, true, true)
      MRSIM_YFB(4) MRSIM_YFB(6) MRSIM_YFB(7)
#define MRSIM_YFQ(NCV, M) MRSIM_YF(1, 0, NCV, M) MRSIM_YF(2, 0, NCV, M) MRSIM_YF(4, 0, NCV, M) MRSIM_YF(8, 0, NCV, M)
#define MRSIM_YFN(M) MRSIM_YFQ(1, M) MRSIM_YFQ(2, M) MRSIM_YFQ(3, M) MRSIM_YFQ(4, M) MRSIM_YFQ(8, M)
      MRSIM_YFN(false) MRSIM_YFN(true)
      MRSIM_YF(8, 6, 1, false) MRSIM_YF(8, 6, 2, false) MRSIM_YF(8, 6, 3, false) MRSIM_YF(8, 6, 4, false)
      MRSIM_YF(8, 6, 1, true) MRSIM_YF(8, 6, 2, true) MRSIM_YF(8, 6, 3, true)
      MRSIM_YF(8, 4, 1, false) MRSIM_YF(8, 4, 2, false) MRSIM_YF(8, 4, 3, false) MRSIM_YF(8, 4, 4, false)
      MRSIM_YF(8, 4, 1, true) MRSIM_YF(8, 4, 2, true) MRSIM_YF(8, 4, 3, true)
      MRSIM_YF(8, 7, 1, false) MRSIM_YF(8, 7, 2, false) MRSIM_YF(8, 7, 3, false) MRSIM_YF(8, 7, 4, false)
      MRSIM_YF(8, 7, 1, true) MRSIM_YF(8, 7, 2, true) MRSIM_YF(8, 7, 3, true)
#undef MRSIM_YFN
#undef MRSIM_YFQ
#undef MRSIM_YF
#undef MRSIM_YFB
#undef MRSIM_YFW
      if (!launched) fail("no forward kernel instance for this unit shape");
      MRSIM_CUDA(cudaGetLastError());
      continue;
    }
    const size_t sm = sizeof(float) * (size_t)p->max_sny * (kT + (QG + 3) / 4 * 4);
    bool launched = false;
#define MRSIM_Y(QGV, NCV, M)                                                            \
  if (QG == QGV && NCv == NCV && maps == M) {                                           \
    auto k = ystage_kernel<kT, QGV, NCV, M>;                                            \
    set_smem(k, sm);                                                                    \
    k<<<(unsigned)R.n, 128, sm, st>>>(p->d_units, tiles);                               \
    launched = true;                                                                    \
  }
#define MRSIM_YQ(NCV, M) MRSIM_Y(1, NCV, M) MRSIM_Y(2, NCV, M) MRSIM_Y(4, NCV, M) MRSIM_Y(8, NCV, M)
#define MRSIM_YN(M) MRSIM_YQ(1, M) MRSIM_YQ(2, M) MRSIM_YQ(3, M) MRSIM_YQ(4, M) MRSIM_YQ(8, M)
    MRSIM_YN(false) MRSIM_YN(true)
#undef MRSIM_YN
#undef MRSIM_YQ
#undef MRSIM_Y
    if (!launched) fail("no forward kernel instance for this unit shape");
    MRSIM_CUDA(cudaGetLastError());
  }
}

}  // namespace mrsim
