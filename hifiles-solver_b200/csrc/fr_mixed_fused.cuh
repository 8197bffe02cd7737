// fr_mixed_fused.cuh -- kernels of the fused RK stage for dense-operator
// element types (fr_mixed_fused.cu has the design notes and the host side):
// shared-memory plans, the FP64 tensor-core product units, the gradient,
// update and trace kernels, and the table of launch shapes.  Included by
// fr_mixed_fused.cu (3-D element types) and fr_mixed_fused_2d.cu (2-D), so
// the two sets of template instances build in parallel.
#pragma once

#include <cuda_runtime.h>

#include "fr_update.cuh"
#include "fr_physics.cuh"

namespace frb_mixed {
using namespace frb;

constexpr int kMixedEPB = 8;   // elements per block: 8 x (D + 2) columns fill whole 8-column tiles
constexpr int kMixedNT = 256;  // threads per block

__host__ __device__ constexpr int c4(int x) { return (x + 3) / 4 * 4; }
__host__ __device__ constexpr int c8(int x) { return (x + 7) / 8 * 8; }
__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
// smallest leading dimension >= x that is 4 or 12 mod 16
__host__ __device__ constexpr int bank_ld(int x) { return (x % 16 == 4 || x % 16 == 12) ? x : bank_ld(x + 1); }
// column tiles per warp unit: all of them up to 6, else a divisor
__host__ __device__ constexpr int tiles_per_unit(int ntl)
{
  return ntl <= 6 ? ntl : (ntl % 5 == 0 ? 5 : (ntl % 4 == 0 ? 4 : (ntl % 3 == 0 ? 3 : 4)));
}

// Shared-memory plan and product shapes of one element type (doubles).
constexpr size_t kMixedSmemMax = 227 * 1024;  // dynamic shared memory of one block
__host__ __device__ constexpr int r2(int x) { return (x + 1) / 2 * 2; }  // 16-byte region starts

template <int D, int NU, int NF, int EPB, int MINB = 1>
struct MPlan {
  static constexpr int F = D + 2, DD = D * D, EU = EPB * NU, EF = EPB * NF;
  static constexpr int N = EPB * F, NP = c8(N);          // (element, field) columns
  static constexpr int NG = N * D, NGP = c8(NG);         // (element, field, dimension) columns
  static constexpr int ldU = bank_ld(c4(NU));
  static constexpr int ldF = bank_ld(c8(NF));
  static constexpr int ldG = bank_ld(cmax(c8(D * NU), (D - 1) * NU + c4(NU)));
  static constexpr int ldT = bank_ld(c4(D * NU));
  static constexpr int MT_U = c8(NU) / 8, MT_F = c8(NF) / 8, MT_G = c8(D * NU) / 8;
  static constexpr int KS_U = c4(NU) / 4, KS_F = c4(NF) / 4, KS_T = c4(D * NU) / 4;
  static constexpr int NTL = NP / 8, NTLG = NGP / 8;
  static constexpr int TN = tiles_per_unit(NTL), TNG = tiles_per_unit(NTLG);
  // kernel A: the matrices U | own traces | gradient | X (delta, then the
  // gradient at the flux points, then the transformed flux); then what else the
  // load phase stages: left normals [D][EF], detJ [EU], JGinv [EPB][DD NU] (when
  // it fits)
  static constexpr int oU = 0, oUF = oU + NP * ldU, oG = oUF + NP * ldF, oX = oG + NP * ldG;
  static constexpr int nX = cmax(cmax(NP * ldF, NGP * ldF), NP * ldT);
  static constexpr int oNL = oX + r2(nX), oDJ = oNL + r2(D * EF), oJG = oDJ + r2(EU);
  // JGinv is staged when MINB blocks with it fit in an SM's shared memory
  // (228 KB, 1 KB reserved per block), else read through the L1 cache
  static constexpr bool SJ = (size_t)MINB * (sizeof(double) * (size_t)(oJG + r2(DD * EU)) + 1024) <= 228 * 1024 &&
                             sizeof(double) * (size_t)(oJG + r2(DD * EU)) <= kMixedSmemMax;
  static constexpr int nA = oJG + (SJ ? r2(DD * EU) : 0);
  // kernel B: the jump norm_tconf - norm_tdisf | the new state [NP][ldU] |
  // div_tdisf, RK register (then |div/detJ| for residual norms), state [F][EU] |
  // detJ [EU]
  static constexpr int oJ = 0, oUn = r2(NP * ldF), oDV = oUn + r2(NP * ldU), oRG = oDV + r2(F * EU);
  static constexpr int oUO = oRG + r2(F * EU), oDJb = oUO + r2(F * EU), nB = oDJb + r2(EU);
  // trace kernel: the state
  static constexpr int nC = NP * ldU;
  static_assert(ldT >= c4(D * NU) && ldG >= c8(D * NU) && ldF >= c8(NF) && ldU >= c4(NU), "plan");
};

struct MixedType {
  int NU, NF;
  long long E, off;  // elements; first flux point in the flux-point space
  const double *A45u, *A45f, *A6, *A1, *A2, *A3, *A0;  // operators in fragment order
  const double *JG, *detj;
  double *U, *REG, *DIV, *ND, *DV;
  double* partial;  // non-null on a stage whose residual norms are wanted: [block][F]
};

struct MixedFpts {
  long long NT;  // flux points over all types
  const int* mate;
  const int* side;  // bit 0 left side, bits 2.. boundary type
  const double* nL;   // [D][NT]
  const double* tdA;  // [NT]
  double* VF;         // [F-1][NT]
  double* BV;         // [boundary points][F]
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b)
{
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// One warp unit of C = A1 B1 (+ A2 B2): rows 8 mt .. 8 mt + 7 (u / NB) and TN
// column tiles from TN (u % NB).  A in fragment order, B's column n starts at
// b(n) (rows contiguous); epi(row, n, C[row][n], C[row][n + 1]) for n even.
template <int NTL, int TN, int KS1, int KS2, class B1, class B2, class Epi>
__device__ __forceinline__ void mma_unit(int u, const double* __restrict__ A1, B1 b1, const double* __restrict__ A2,
                                         B2 b2, Epi epi)
{
  constexpr int NB = (NTL + TN - 1) / TN;
  const int lane = threadIdx.x & 31, mt = u / NB, nt0 = (u - mt * NB) * TN;
  double acc[TN][2];
  const double* p1[TN];
  const double* p2[TN];
#pragma unroll
  for (int j = 0; j < TN; j++) {
    acc[j][0] = 0.0;
    acc[j][1] = 0.0;
    const int n = (nt0 + j < NTL ? nt0 + j : nt0) * 8 + (lane >> 2);
    p1[j] = b1(n) + (lane & 3);
    p2[j] = KS2 > 0 ? b2(n) + (lane & 3) : p1[j];
  }
  // operator fragments are fetched CH k-steps ahead of their MMAs, so their
  // read-only-cache latency is paid once per CH steps
  constexpr int CH = 8;
  const double* a1 = A1 + (size_t)mt * KS1 * 32 + lane;
#pragma unroll
  for (int k0 = 0; k0 < KS1; k0 += CH) {
    double af[CH];
#pragma unroll
    for (int i = 0; i < CH; i++) af[i] = k0 + i < KS1 ? __ldg(a1 + (k0 + i) * 32) : 0.0;
#pragma unroll
    for (int i = 0; i < CH; i++)
      if (k0 + i < KS1)
#pragma unroll
        for (int j = 0; j < TN; j++)
          if (nt0 + j < NTL) dmma(acc[j], af[i], p1[j][(k0 + i) * 4]);
  }
  if constexpr (KS2 > 0) {
    const double* a2 = A2 + (size_t)mt * KS2 * 32 + lane;
#pragma unroll
    for (int k0 = 0; k0 < KS2; k0 += CH) {
      double af[CH];
#pragma unroll
      for (int i = 0; i < CH; i++) af[i] = k0 + i < KS2 ? __ldg(a2 + (k0 + i) * 32) : 0.0;
#pragma unroll
      for (int i = 0; i < CH; i++)
        if (k0 + i < KS2)
#pragma unroll
          for (int j = 0; j < TN; j++)
            if (nt0 + j < NTL) dmma(acc[j], af[i], p2[j][(k0 + i) * 4]);
    }
  }
#pragma unroll
  for (int j = 0; j < TN; j++)
    if (nt0 + j < NTL) epi(mt * 8 + (lane >> 2), (nt0 + j) * 8 + 2 * (lane & 3), acc[j][0], acc[j][1]);
}

template <int NTL, int TN>
__host__ __device__ constexpr int units(int mt)
{
  return mt * ((NTL + TN - 1) / TN);
}

// zero rows r0 .. r1 - 1 of the first ncol columns of a column-major matrix:
// the padding rows a product reads (times the operator's zero columns), which
// must hold finite values
template <int R0, int R1, int LD, int NCOL, int NTH>
__device__ __forceinline__ void zero_pad_rows(double* a)
{
  constexpr int W = R1 - R0;
  if constexpr (W > 0)
    for (int i = threadIdx.x; i < NCOL * W; i += NTH) a[(i / W) * LD + R0 + i % W] = 0.0;
}

// the block's state into columns (element, field) of sU (rows = solution points)
template <int F, int NU, int EPB, int ldU, int NTH>
__device__ __forceinline__ void load_state(double* sU, const double* __restrict__ U, long long e0, long long E,
                                           int nval)
{
  const int nuv = nval * NU;
  const size_t NUE = (size_t)NU * E;
  for (int r = threadIdx.x; r < nuv; r += NTH) {
    const int el = r / NU, p = r - el * NU;
    double* dst = sU + el * F * ldU + p;
    const double* src = U + (size_t)NU * e0 + r;
#pragma unroll
    for (int k = 0; k < F; k++) cp_async<8>(dst + k * ldU, src + NUE * k);
  }
}

// ------------------------------------------------------------------ kernel A
// A load phase issues the block's global reads together: state, own traces,
// normals and metrics into shared memory, wiring and the neighbours' traces into
// the registers of the threads that use them (blocks of more than four flux
// points per thread read those where they use them, and boundary points their
// place in the boundary list); otherwise the compute phases only write.
template <int D, int NU, int NF, int EPB, int NTH, int MINB>
__global__ void __launch_bounds__(NTH, MINB) mixed_grad_kernel(MixedType t, MixedFpts m,
                                                               const double* __restrict__ UFc, PhysT<double> ph)
{
  using Q = MPlan<D, NU, NF, EPB, MINB>;
  constexpr int F = D + 2, NW = NTH / 32, DD = D * D, EF = Q::EF;
  extern __shared__ __align__(16) double msm[];
  double* sU = msm + Q::oU;
  double* sUF = msm + Q::oUF;
  double* sG = msm + Q::oG;
  double* sX = msm + Q::oX;
  double* sNL = msm + Q::oNL;
  double* sDJ = msm + Q::oDJ;
  double* sJG = msm + Q::oJG;
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long E = t.E, NT = m.NT, e0 = (long long)blockIdx.x * EPB;
  const int nval = (int)(E - e0 < EPB ? E - e0 : EPB), nuv = nval * NU, nfv = nval * NF;
  const long long gb = t.off + (long long)NF * e0;

  // load phase: asynchronous copies (cp.async), many in flight per thread, of
  // everything at known addresses; the neighbours' traces go straight to the
  // registers of the threads that use them (up to four flux points per thread:
  // first every mate, then every trace, so two round trips and no barrier; a
  // boundary point reads its own, unused).  The matrices are not cleared: only the
  // padding rows the products read are zeroed (U and delta here, the flux before
  // its products); every other padding entry only reaches outputs that are not
  // written.
  constexpr int IT = (EF + NTH - 1) / NTH;
  constexpr bool PRE = IT <= 4;
  int mtr[PRE ? IT : 1], sdr[PRE ? IT : 1];
  if constexpr (PRE) {
#pragma unroll
    for (int it = 0; it < IT; it++) {
      const int r = tid + it * NTH;
      const long long g = gb + (r < nfv ? r : 0);
      mtr[it] = m.mate[g];
      sdr[it] = m.side[g];
    }
  }
  zero_pad_rows<NU, c4(NU), Q::ldU, Q::NP, NTH>(sU);
  zero_pad_rows<NF, c4(NF), Q::ldF, Q::NP, NTH>(sX);  // delta's padding rows
  load_state<F, NU, EPB, Q::ldU, NTH>(sU, t.U, e0, E, nval);
  for (int r = tid; r < nfv; r += NTH) {
    const int el = r / NF, f = r - el * NF;
    const long long g = gb + r;
    double* dst = sUF + el * F * Q::ldF + f;
#pragma unroll
    for (int k = 0; k < F; k++) cp_async<8>(dst + k * Q::ldF, UFc + g + NT * k);
#pragma unroll
    for (int d = 0; d < D; d++) cp_async<8>(&sNL[d * EF + r], m.nL + g + NT * d);
  }
  for (int i = tid; i < nuv; i += NTH) {
    cp_async<8>(&sDJ[i], t.detj + (size_t)NU * e0 + i);
    if constexpr (Q::SJ)
#pragma unroll
      for (int q = 0; q < DD; q++) cp_async<8>(&sJG[i + q * nuv], t.JG + (size_t)DD * NU * e0 + i + q * nuv);
  }
  double unr[PRE ? IT : 1][F];
  auto gather = [&](int r, int mt, double (&un)[F]) {
    const long long h = mt < 0 ? gb + (r < nfv ? r : 0) : (long long)mt;
#pragma unroll
    for (int k = 0; k < F; k++) un[k] = UFc[h + NT * k];
  };
  if constexpr (PRE) {
#pragma unroll
    for (int it = 0; it < IT; it++) gather(tid + it * NTH, mtr[it], unr[it]);
  }
  cp_async_wait_all();
  __syncthreads();
  auto jg = [&](int i) { return Q::SJ ? sJG + DD * i : t.JG + (size_t)DD * ((size_t)NU * e0 + i); };

  // LDG common solution at the own flux points: delta = u_c - u_own into X
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = tid + it * NTH;
    if (i >= nfv) continue;
    const int el = i / NF, f = i - el * NF, pi = PRE ? it : 0;
    if constexpr (!PRE) {
      mtr[0] = m.mate[gb + i];
      sdr[0] = m.side[gb + i];
      gather(i, mtr[0], unr[0]);
    }
    const int sd = sdr[pi];
    double n[D], uo[F];
#pragma unroll
    for (int d = 0; d < D; d++) n[d] = sNL[d * EF + i];
#pragma unroll
    for (int k = 0; k < F; k++) uo[k] = sUF[(el * F + k) * Q::ldF + f];
    double* dx = sX + (el * F) * Q::ldF + f;
    if (sd >> 2) {
      BdyPoint<D, double> q;
#pragma unroll
      for (int k = 0; k < F; k++) q.u[k] = uo[k];
#pragma unroll
      for (int d = 0; d < D; d++) q.n[d] = n[d];
      ldg_boundary<D, double>(ph, sd >> 2, q, dx, sUF + (el * F) * Q::ldF + f, Q::ldF);
    } else {
      const bool left = sd & 1;
      const double pen = ldg_beta<D, double>(ph.pen_fact, n);
#pragma unroll
      for (int k = 0; k < F; k++) {
        const double un = unr[pi][k];
        const double ul = left ? uo[k] : un, ur = left ? un : uo[k];
        const double uc = 0.5 * (ul + ur) - pen * (ul - ur);
        dx[k * Q::ldF] = uc - uo[k];
      }
    }
  }
  __syncthreads();

  // reference-space gradient: rows (d, point) of sG
  {
    auto bu = [&](int n) { return sU + n * Q::ldU; };
    auto bd = [&](int n) { return sX + n * Q::ldF; };
    auto epi = [&](int r, int n, double v0, double v1) {
      sG[n * Q::ldG + r] = v0;
      sG[(n + 1) * Q::ldG + r] = v1;
    };
    for (int u = warp; u < units<Q::NTL, Q::TN>(Q::MT_G); u += NW)
      mma_unit<Q::NTL, Q::TN, Q::KS_U, Q::KS_F>(u, t.A45u, bu, t.A45f, bd, epi);
  }
  __syncthreads();

  // physical gradient in place (transform_grad_disu_upts: JGinv / detJ)
  for (int i = tid; i < nuv; i += NTH) {
    const int el = i / NU, p = i - el * NU;
    const double inv = 1.0 / sDJ[i];
    const double* G = jg(i);
    double Gm[D][D];
#pragma unroll
    for (int r = 0; r < D; r++)
#pragma unroll
      for (int c = 0; c < D; c++) Gm[r][c] = G[r + D * c] * inv;
#pragma unroll
    for (int k = 0; k < F; k++) {
      double* s = sG + (el * F + k) * Q::ldG + p;
      double gr[D];
#pragma unroll
      for (int r = 0; r < D; r++) gr[r] = s[r * NU];
#pragma unroll
      for (int c = 0; c < D; c++) {
        double acc = 0.0;
#pragma unroll
        for (int r = 0; r < D; r++) acc = fma(gr[r], Gm[r][c], acc);
        s[c * NU] = acc;
      }
    }
  }
  __syncthreads();

  // gradient at the flux points: column d N + (element, field) of X for
  // dimension d (dimension-major, so the 8 columns of a fragment load are
  // consecutive columns of sG and hit distinct banks)
  {
    auto bg = [&](int n) {
      const int c = n < Q::NG ? n : Q::NG - 1, d = c / Q::N;
      return sG + (c - d * Q::N) * Q::ldG + d * NU;
    };
    auto epi = [&](int r, int n, double v0, double v1) {
      sX[n * Q::ldF + r] = v0;
      sX[(n + 1) * Q::ldF + r] = v1;
    };
    for (int u = warp; u < units<Q::NTLG, Q::TNG>(Q::MT_F); u += NW)
      mma_unit<Q::NTLG, Q::TNG, Q::KS_U, 0>(u, t.A6, bg, t.A6, bg, epi);
  }
  __syncthreads();

  // viscous normal projections (interior points) and boundary viscous fluxes
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = tid + it * NTH;
    if (i >= nfv) continue;
    const int el = i / NF, f = i - el * NF;
    const long long g = gb + i;
    const int sd = PRE ? sdr[PRE ? it : 0] : m.side[g];
    double n[D], uo[F], gf[F][D];
#pragma unroll
    for (int d = 0; d < D; d++) n[d] = sNL[d * EF + i];
#pragma unroll
    for (int k = 0; k < F; k++) {
      uo[k] = sUF[(el * F + k) * Q::ldF + f];
#pragma unroll
      for (int c = 0; c < D; c++) gf[k][c] = sX[(c * Q::N + el * F + k) * Q::ldF + f];
    }
    if (sd >> 2) {
      BdyPoint<D, double> q;
#pragma unroll
      for (int k = 0; k < F; k++) {
        q.u[k] = uo[k];
#pragma unroll
        for (int c = 0; c < D; c++) q.g[k][c] = gf[k][c];
      }
#pragma unroll
      for (int d = 0; d < D; d++) q.n[d] = n[d];
      vis_boundary<D, double, false>(ph, sd >> 2, q, m.BV + (size_t)(-1 - (long long)m.mate[g]) * F);
    } else {
      double pr[F - 1];
      vis_flux_proj<D, double>(ph, uo, gf, n, pr);
#pragma unroll
      for (int k = 0; k < F - 1; k++) m.VF[g + NT * k] = pr[k];
    }
  }
  __syncthreads();

  zero_pad_rows<D * NU, c4(D * NU), Q::ldT, Q::NP, NTH>(sX);  // the flux's padding rows
  // transformed flux at the solution points (evaluate_invFlux, then
  // evaluate_viscFlux adding to it): rows (d, point) of X.  The viscous flux
  // takes one reciprocal of rho (vis_flux_fast): its terms are ~1/Re of the
  // inviscid flux they are added to, so its ulp-level differences from the
  // reference's divisions stay far below the rounding of the sum.
  for (int i = tid; i < nuv; i += NTH) {
    const int el = i / NU, p = i - el * NU;
    const double* G = jg(i);
    double q[F], tf[F][D];
    {
      double fi[F][D];
#pragma unroll
      for (int k = 0; k < F; k++) q[k] = sU[(el * F + k) * Q::ldU + p];
      inv_flux<D, double>(ph, q, fi);
#pragma unroll
      for (int k = 0; k < F; k++)
#pragma unroll
        for (int l = 0; l < D; l++) {
          double acc = 0.0;
#pragma unroll
          for (int mm = 0; mm < D; mm++) acc = fma(G[l + D * mm], fi[k][mm], acc);
          tf[k][l] = acc;
        }
    }
    {
      double gq[F][D], fv[F][D];
#pragma unroll
      for (int k = 0; k < F; k++)
#pragma unroll
        for (int c = 0; c < D; c++) gq[k][c] = sG[(el * F + k) * Q::ldG + c * NU + p];
      vis_flux_fast<D, double>(ph, q, gq, fv);
#pragma unroll
      for (int k = 0; k < F; k++)
#pragma unroll
        for (int l = 0; l < D; l++) {
          double acc = tf[k][l];
#pragma unroll
          for (int mm = 0; mm < D; mm++) acc = fma(G[l + D * mm], fv[k][mm], acc);
          sX[(el * F + k) * Q::ldT + l * NU + p] = acc;
        }
    }
  }
  __syncthreads();

  // norm_tdisf = sum_d opp_1[d] f_d and div_tdisf = sum_d opp_2[d] f_d
  {
    auto bt = [&](int n) { return sX + n * Q::ldT; };
    const size_t NFE = (size_t)NF * E, NUE = (size_t)NU * E;
    auto put = [&](double* out, int rows, size_t stride, int r, int n, double v) {
      const int el = n / F, k = n - el * F;
      if (r < rows && el < nval) out[r + (size_t)rows * (e0 + el) + stride * k] = v;
    };
    auto epi_nd = [&](int r, int n, double v0, double v1) {
      put(t.ND, NF, NFE, r, n, v0);
      put(t.ND, NF, NFE, r, n + 1, v1);
    };
    auto epi_dv = [&](int r, int n, double v0, double v1) {
      put(t.DV, NU, NUE, r, n, v0);
      put(t.DV, NU, NUE, r, n + 1, v1);
    };
    constexpr int U1 = units<Q::NTL, Q::TN>(Q::MT_F), U2 = units<Q::NTL, Q::TN>(Q::MT_U);
    for (int u = warp; u < U1 + U2; u += NW) {
      if (u < U1) mma_unit<Q::NTL, Q::TN, Q::KS_T, 0>(u, t.A1, bt, t.A1, bt, epi_nd);
      else mma_unit<Q::NTL, Q::TN, Q::KS_T, 0>(u - U1, t.A2, bt, t.A2, bt, epi_dv);
    }
  }
}

// ------------------------------------------------------ kernel A, Euler form
// The inviscid stage needs no gradient: the transformed inviscid flux at the
// solution points (evaluate_invFlux), then norm_tdisf = sum_d opp_1[d] f_d
// and div_tdisf = sum_d opp_2[d] f_d.  JGinv is read through the L1 cache.
template <int D, int NU, int NF, int EPB>
struct MPlanInv {
  using Q = MPlan<D, NU, NF, EPB>;
  static constexpr int oU = 0, oT = Q::NP * Q::ldU, nI = oT + Q::NP * Q::ldT;
};

template <int D, int NU, int NF, int EPB, int NTH, int MINB>
__global__ void __launch_bounds__(NTH, MINB) mixed_inv_kernel(MixedType t, MixedFpts m,
                                                              const double* __restrict__ UFc, PhysT<double> ph)
{
  using Q = MPlan<D, NU, NF, EPB>;
  using I = MPlanInv<D, NU, NF, EPB>;
  constexpr int F = D + 2, NW = NTH / 32, DD = D * D;
  extern __shared__ __align__(16) double msm[];
  double* sU = msm + I::oU;
  double* sT = msm + I::oT;
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long E = t.E, e0 = (long long)blockIdx.x * EPB;
  const int nval = (int)(E - e0 < EPB ? E - e0 : EPB), nuv = nval * NU;
  (void)m;
  (void)UFc;
  zero_pad_rows<NU, c4(NU), Q::ldU, Q::NP, NTH>(sU);
  zero_pad_rows<D * NU, c4(D * NU), Q::ldT, Q::NP, NTH>(sT);
  load_state<F, NU, EPB, Q::ldU, NTH>(sU, t.U, e0, E, nval);
  cp_async_wait_all();
  __syncthreads();
  for (int i = tid; i < nuv; i += NTH) {
    const int el = i / NU, p = i - el * NU;
    const double* G = t.JG + (size_t)DD * ((size_t)NU * e0 + i);
    double q[F], fi[F][D];
#pragma unroll
    for (int k = 0; k < F; k++) q[k] = sU[(el * F + k) * Q::ldU + p];
    inv_flux<D, double>(ph, q, fi);
#pragma unroll
    for (int k = 0; k < F; k++)
#pragma unroll
      for (int l = 0; l < D; l++) {
        double acc = 0.0;
#pragma unroll
        for (int mm = 0; mm < D; mm++) acc = fma(G[l + D * mm], fi[k][mm], acc);
        sT[(el * F + k) * Q::ldT + l * NU + p] = acc;
      }
  }
  __syncthreads();
  auto bt = [&](int n) { return sT + n * Q::ldT; };
  const size_t NFE = (size_t)NF * E, NUE = (size_t)NU * E;
  auto put = [&](double* out, int rows, size_t stride, int r, int n, double v) {
    const int el = n / F, k = n - el * F;
    if (r < rows && el < nval) out[r + (size_t)rows * (e0 + el) + stride * k] = v;
  };
  auto epi_nd = [&](int r, int n, double v0, double v1) {
    put(t.ND, NF, NFE, r, n, v0);
    put(t.ND, NF, NFE, r, n + 1, v1);
  };
  auto epi_dv = [&](int r, int n, double v0, double v1) {
    put(t.DV, NU, NUE, r, n, v0);
    put(t.DV, NU, NUE, r, n + 1, v1);
  };
  constexpr int U1 = units<Q::NTL, Q::TN>(Q::MT_F), U2 = units<Q::NTL, Q::TN>(Q::MT_U);
  for (int u = warp; u < U1 + U2; u += NW) {
    if (u < U1) mma_unit<Q::NTL, Q::TN, Q::KS_T, 0>(u, t.A1, bt, t.A1, bt, epi_nd);
    else mma_unit<Q::NTL, Q::TN, Q::KS_T, 0>(u - U1, t.A2, bt, t.A2, bt, epi_dv);
  }
}

// ------------------------------------------------------------------ kernel B
// MODE 1: RK45 stage update (rk_a, rk_b, dt) and the new traces into UFn;
// MODE 0: div_tconf_upts into t.DIV only.  A flux point's inputs (own and
// neighbour's trace and projections, normal flux, normal, dA) are each used
// once, by its own thread: they go to registers, the neighbour's as soon as the
// mate has arrived; what the product's epilogue needs (divergence, register,
// state, detJ) is copied to shared memory meanwhile.  Staging all of it in
// shared memory took two rounds of copies with a barrier each and twice the
// shared memory per element.
template <int D, int VISC>
struct FptRegs {
  static constexpr int F = D + 2;
  int mt, sd;
  double uo[F], un[F], nd[F], vo[VISC ? F - 1 : 1], vn[VISC ? F - 1 : 1], n[D], tl;
};

template <int D, int NU, int NF, int EPB, int NTH, int MINB, int MODE, int VISC = 1, int RIEMANN = 0>
__global__ void __launch_bounds__(NTH, MINB) mixed_update_kernel(MixedType t, MixedFpts m,
                                                                 const double* __restrict__ UFc,
                                                                 double* __restrict__ UFn, PhysT<double> ph,
                                                                 double rk_a, double rk_b, double dt)
{
  using Q = MPlan<D, NU, NF, EPB>;
  constexpr int F = D + 2, NW = NTH / 32, EU = Q::EU, EF = Q::EF, IT = (EF + NTH - 1) / NTH;
  extern __shared__ __align__(16) double msm[];
  double* sJ = msm + Q::oJ;
  double* sUn = msm + Q::oUn;
  double* sDV = msm + Q::oDV;
  double* sRG = msm + Q::oRG;
  double* sRes = sRG;  // |div/detJ| [F][EU] for residual norms: each entry by the thread that read the register
  double* sUO = msm + Q::oUO;
  double* sDJ = msm + Q::oDJb;
  const int tid = threadIdx.x, warp = tid >> 5;
  const long long E = t.E, NT = m.NT, e0 = (long long)blockIdx.x * EPB;
  const int nval = (int)(E - e0 < EPB ? E - e0 : EPB), nuv = nval * NU, nfv = nval * NF;
  const long long gb = t.off + (long long)NF * e0;
  const size_t NFE = (size_t)NF * E, NUE = (size_t)NU * E;

  auto load = [&](int r, FptRegs<D, VISC>& q) {
    const long long g = gb + r;
    q.mt = m.mate[g];
    q.sd = m.side[g];
    const double* nd = t.ND + (size_t)NF * e0 + r;
#pragma unroll
    for (int k = 0; k < F; k++) {
      q.uo[k] = UFc[g + NT * k];
      q.nd[k] = nd[NFE * k];
    }
    if constexpr (VISC != 0) {
#pragma unroll
      for (int k = 0; k < F - 1; k++) q.vo[k] = m.VF[g + NT * k];
    }
#pragma unroll
    for (int d = 0; d < D; d++) q.n[d] = m.nL[g + NT * d];
    q.tl = m.tdA[g];
    // the neighbour's values (a boundary point reads its own, unused), no branch between the loads
    const long long h = q.mt < 0 ? g : (long long)q.mt;
#pragma unroll
    for (int k = 0; k < F; k++) q.un[k] = UFc[h + NT * k];
    if constexpr (VISC != 0) {
#pragma unroll
      for (int k = 0; k < F - 1; k++) q.vn[k] = m.VF[h + NT * k];
    }
  };
  for (int r = tid; r < nuv; r += NTH) {
    const size_t ix = (size_t)NU * e0 + r;
#pragma unroll
    for (int k = 0; k < F; k++) {
      cp_async<8>(&sDV[k * EU + r], t.DV + ix + NUE * k);
      if (MODE == 1) {
        cp_async<8>(&sRG[k * EU + r], t.REG + ix + NUE * k);
        cp_async<8>(&sUO[k * EU + r], t.U + ix + NUE * k);
      }
    }
    if (MODE == 1) cp_async<8>(&sDJ[r], t.detj + ix);
  }
  zero_pad_rows<NF, c4(NF), Q::ldF, Q::NP, NTH>(sJ);

  // common normal fluxes times the own tdA, minus norm_tdisf
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = tid + it * NTH;
    if (i >= nfv) continue;
    FptRegs<D, VISC> q;
    load(i, q);
    const int el = i / NF, f = i - el * NF;
    double c[F];
    if (q.sd >> 2) {
      FUBdy<D, double> b;
#pragma unroll
      for (int k = 0; k < F; k++) {
        b.ul[k] = q.uo[k];
        b.bv[k] = VISC ? m.BV[(size_t)(-1 - (long long)q.mt) * F + k] : 0.0;
      }
#pragma unroll
      for (int d = 0; d < D; d++) b.n[d] = q.n[d];
      b.tl = q.tl;
      fu_boundary<D, VISC, double, RIEMANN>(ph, q.sd >> 2, b, c, 1);
    } else {
      const bool left = q.sd & 1;
      double ul[F], ur[F], fn[F];
#pragma unroll
      for (int k = 0; k < F; k++) {
        ul[k] = left ? q.uo[k] : q.un[k];
        ur[k] = left ? q.un[k] : q.uo[k];
      }
      if constexpr (RIEMANN == 2 && D == 2) roe<double>(ph, ul, ur, q.n, fn);
      else rusanov<D, double>(ph, ul, ur, q.n, fn);
#pragma unroll
      for (int k = 0; k < F; k++) c[k] = left ? fn[k] * q.tl : -fn[k] * q.tl;
      if constexpr (VISC != 0) {
        double nn = q.n[0] * q.n[0];
#pragma unroll
        for (int d = 1; d < D; d++) nn = fma(q.n[d], q.n[d], nn);
        const double pen = ldg_beta<D, double>(ph.pen_fact, q.n);
#pragma unroll
        for (int k = 0; k < F; k++) {
          const double ao = k ? q.vo[k ? k - 1 : 0] : 0.0, an = k ? q.vn[k ? k - 1 : 0] : 0.0;
          const double fv = ldg_normal<double>(left ? ao : an, left ? an : ao, ul[k], ur[k], pen, ph.tau, nn);
          c[k] = left ? c[k] + fv * q.tl : c[k] + (-fv) * q.tl;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < F; k++) sJ[(el * F + k) * Q::ldF + f] = c[k] - q.nd[k];
  }
  cp_async_wait_all();
  __syncthreads();

  // div_tconf = div_tdisf + opp_3 jump, then the RK45 update
  // (RK45_update_kernel: rhs = -div / detJ)
  {
    // padding rows of the new state, read (times zero) by the trace product
    if constexpr (MODE == 1) zero_pad_rows<NU, c4(NU), Q::ldU, Q::NP, NTH>(sUn);
    auto bj = [&](int n) { return sJ + n * Q::ldF; };
    auto one = [&](int r, int n, double v) {
      const int el = n / F, k = n - el * F;
      if (r >= NU || el >= nval) return;
      const int li = k * EU + el * NU + r;
      const size_t ix = (size_t)NU * e0 + (size_t)el * NU + r + NUE * k;
      const double div = v + sDV[li];
      if (MODE == 0) {
        t.DIV[ix] = div;
      } else {
        const double rhs = -div / sDJ[el * NU + r];
        const double res = fma(rk_a, sRG[li], dt * rhs);
        // |div/detJ| of compute_res_upts (src/eles.cpp:6086-6115; no sources here)
        if (t.partial) sRes[li] = fabs(rhs);
        t.REG[ix] = res;
        const double un = fma(rk_b, res, sUO[li]);
        t.U[ix] = un;
        sUn[n * Q::ldU + r] = un;
      }
    };
    auto epi = [&](int r, int n, double v0, double v1) {
      one(r, n, v0);
      one(r, n + 1, v1);
    };
    for (int u = warp; u < units<Q::NTL, Q::TN>(Q::MT_U); u += NW)
      mma_unit<Q::NTL, Q::TN, Q::KS_F, 0>(u, t.A3, bj, t.A3, bj, epi);
  }
  if constexpr (MODE == 1) {
    __syncthreads();
    if (t.partial) {
      // the block's L1 residual sum of each field: one warp per field, lanes
      // over the block's points and a fixed tree (one thread per field walking
      // the points was a chain of EPB x NU dependent additions)
      for (int k = warp; k < F; k += NW) {
        double bs = 0.0;
        for (int i = tid & 31; i < nuv; i += 32) bs += sRes[k * EU + i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) bs += __shfl_down_sync(0xffffffffu, bs, o);
        if ((tid & 31) == 0) t.partial[(size_t)blockIdx.x * F + k] = bs;
      }
    }
    auto bu = [&](int n) { return sUn + n * Q::ldU; };
    auto one = [&](int r, int n, double v) {
      const int el = n / F, k = n - el * F;
      if (r < NF && el < nval) UFn[gb + r + (long long)NF * el + NT * k] = v;
    };
    auto epi = [&](int r, int n, double v0, double v1) {
      one(r, n, v0);
      one(r, n + 1, v1);
    };
    for (int u = warp; u < units<Q::NTL, Q::TN>(Q::MT_F); u += NW)
      mma_unit<Q::NTL, Q::TN, Q::KS_U, 0>(u, t.A0, bu, t.A0, bu, epi);
  }
}

// ------------------------------------------------------------ trace kernel
// UFn = opp_0 U (extrapolate_solution) with the update kernel's product, so
// the traces match the ones the update kernel writes bit for bit.
template <int D, int NU, int NF, int EPB, int NTH>
__global__ void __launch_bounds__(NTH) mixed_trace_kernel(MixedType t, long long NT, double* __restrict__ UFn)
{
  using Q = MPlan<D, NU, NF, EPB>;
  constexpr int F = D + 2, NW = NTH / 32;
  extern __shared__ __align__(16) double msm[];
  const int warp = threadIdx.x >> 5;
  const long long E = t.E, e0 = (long long)blockIdx.x * EPB;
  const int nval = (int)(E - e0 < EPB ? E - e0 : EPB);
  const long long gb = t.off + (long long)NF * e0;
  zero_pad_rows<NU, c4(NU), Q::ldU, Q::NP, NTH>(msm);
  load_state<F, NU, EPB, Q::ldU, NTH>(msm, t.U, e0, E, nval);
  cp_async_wait_all();
  __syncthreads();
  auto bu = [&](int n) { return msm + n * Q::ldU; };
  auto one = [&](int r, int n, double v) {
    const int el = n / F, k = n - el * F;
    if (r < NF && el < nval) UFn[gb + r + (long long)NF * el + NT * k] = v;
  };
  auto epi = [&](int r, int n, double v0, double v1) {
    one(r, n, v0);
    one(r, n + 1, v1);
  };
  for (int u = warp; u < units<Q::NTL, Q::TN>(Q::MT_F); u += NW)
    mma_unit<Q::NTL, Q::TN, Q::KS_U, 0>(u, t.A0, bu, t.A0, bu, epi);
}

// ------------------------------------------------------------ dispatch
// Launch shapes: elements per block, threads per block, blocks per SM the
// registers are capped for.  Gradient and update kernels pick theirs
// independently (fr_mixed_stage_autotune); the products give the same bits
// in every shape, since each output is the same chain of k-steps.
struct MixedShape {
  int epb, nth, minb;
};
constexpr MixedShape kGradShapes[] = {{8, 256, 1}, {4, 128, 3}, {4, 160, 3}, {4, 128, 4}, {8, 256, 2}};
constexpr MixedShape kUpdShapes[] = {{8, 256, 2}, {4, 160, 3}, {4, 128, 4}};
constexpr int kNGrad = sizeof(kGradShapes) / sizeof(kGradShapes[0]);
constexpr int kNUpd = sizeof(kUpdShapes) / sizeof(kUpdShapes[0]);
// Elements per block of a type with NF flux points: the shape's, or filled as
// many (in fours, whole column tiles) as give each flux point a thread.  Types
// with few points would leave most of a block idle otherwise: triangles of
// P = 2 had 36 flux points on 128 threads (update kernel of 17280: 26.5 us).
__host__ __device__ constexpr int shape_epb(MixedShape s, int nf, bool fill)
{
  return fill ? cmax(s.epb, s.nth / nf / 4 * 4) : s.epb;
}

using GradFn = void (*)(MixedType, MixedFpts, const double*, PhysT<double>);
using UpdFn = void (*)(MixedType, MixedFpts, const double*, double*, PhysT<double>, double, double, double);
using TraceFn = void (*)(MixedType, long long, double*);

// Physics forms: 0 Navier-Stokes (Rusanov + LDG), 1 Euler with Rusanov,
// 2 Euler with Roe (2-D).  The Euler forms have one launch shape, slot 1 of
// either list: the flux kernel of 4 elements x 128 threads, and the update
// kernel of 4 x 160, or of 4 x 128 where blocks are not filled.
constexpr int kNForms = 3;

struct MixedKernels {
  int D, NU, NF;
  // elements per block of each launch shape, threads per block of the update kernels
  int epb_a[kNForms][kNGrad], epb_b[kNForms][kNUpd], epb_c, nth_b[kNForms][kNUpd];
  GradFn grad[kNForms][kNGrad];
  size_t smem_a[kNForms][kNGrad];
  UpdFn upd0[kNForms][kNUpd], upd1[kNForms][kNUpd];
  size_t smem_b[kNForms][kNUpd];
  TraceFn trace;
  size_t smem_c;
};

template <int D, int NU, int NF, bool FILL, int V>
void fill_grad(MixedKernels& k)
{
  constexpr MixedShape g = kGradShapes[V];
  constexpr int epb = shape_epb(g, NF, FILL);
  k.epb_a[0][V] = epb;
  k.smem_a[0][V] = sizeof(double) * MPlan<D, NU, NF, epb, g.minb>::nA;
  k.grad[0][V] = k.smem_a[0][V] <= kMixedSmemMax ? mixed_grad_kernel<D, NU, NF, epb, g.nth, g.minb> : nullptr;
}

template <int D, int NU, int NF, bool FILL, int V>
void fill_upd(MixedKernels& k)
{
  constexpr MixedShape u = kUpdShapes[V];
  constexpr int epb = shape_epb(u, NF, FILL);
  k.epb_b[0][V] = epb;
  k.nth_b[0][V] = u.nth;
  k.smem_b[0][V] = sizeof(double) * MPlan<D, NU, NF, epb>::nB;
  const bool fits = k.smem_b[0][V] <= kMixedSmemMax;
  k.upd0[0][V] = fits ? mixed_update_kernel<D, NU, NF, epb, u.nth, u.minb, 0> : nullptr;
  k.upd1[0][V] = fits ? mixed_update_kernel<D, NU, NF, epb, u.nth, u.minb, 1> : nullptr;
}

template <int D, int NU, int NF, bool FILL>
void fill_euler(MixedKernels& k)
{
  constexpr MixedShape g = kGradShapes[1], u = kUpdShapes[FILL ? 1 : 2];
  constexpr int ge = shape_epb(g, NF, FILL), ue = shape_epb(u, NF, FILL);
  const size_t sa = sizeof(double) * MPlanInv<D, NU, NF, ge>::nI, sb = sizeof(double) * MPlan<D, NU, NF, ue>::nB;
  const bool fa = sa <= kMixedSmemMax, fb = sb <= kMixedSmemMax;
  for (int f = 1; f < kNForms; f++) {
    k.epb_a[f][1] = ge;
    k.epb_b[f][1] = ue;
    k.nth_b[f][1] = u.nth;
    k.smem_a[f][1] = sa;
    k.smem_b[f][1] = sb;
    k.grad[f][1] = fa ? mixed_inv_kernel<D, NU, NF, ge, g.nth, g.minb> : nullptr;
  }
  k.upd0[1][1] = fb ? mixed_update_kernel<D, NU, NF, ue, u.nth, u.minb, 0, 0, 0> : nullptr;
  k.upd1[1][1] = fb ? mixed_update_kernel<D, NU, NF, ue, u.nth, u.minb, 1, 0, 0> : nullptr;
  if constexpr (D == 2) {
    k.upd0[2][1] = fb ? mixed_update_kernel<D, NU, NF, ue, u.nth, u.minb, 0, 0, 2> : nullptr;
    k.upd1[2][1] = fb ? mixed_update_kernel<D, NU, NF, ue, u.nth, u.minb, 1, 0, 2> : nullptr;
  }
}

// Without FILL, the shapes that a stage starts with (gradient 3, update 1, and
// the Euler forms) keep their own number of elements; the others are filled
// all the same, so that every shape is there for meshes of any size.
template <int D, int NU, int NF, bool FILL>
MixedKernels mixed_kernels()
{
  MixedKernels k{};
  k.D = D;
  k.NU = NU;
  k.NF = NF;
  fill_grad<D, NU, NF, true, 0>(k);
  fill_grad<D, NU, NF, true, 1>(k);
  fill_grad<D, NU, NF, true, 2>(k);
  fill_grad<D, NU, NF, FILL, 3>(k);
  fill_grad<D, NU, NF, true, 4>(k);
  fill_upd<D, NU, NF, true, 0>(k);
  fill_upd<D, NU, NF, FILL, 1>(k);
  fill_upd<D, NU, NF, true, 2>(k);
  static_assert(kNGrad == 5 && kNUpd == 3, "one fill per shape");
  fill_euler<D, NU, NF, FILL>(k);
  constexpr int te = shape_epb(MixedShape{kMixedEPB, kMixedNT, 1}, NF, true);
  k.epb_c = te;
  k.trace = mixed_trace_kernel<D, NU, NF, te, kMixedNT>;
  k.smem_c = sizeof(double) * MPlan<D, NU, NF, te>::nC;
  return k;
}


// The kernels of a type of E elements, for physics form pf.  Filling the blocks
// pays where they would otherwise come in more than one wave; a mesh whose
// blocks of 4 elements are all resident at once is bound by the latency of one
// block, which grows with its elements.  Blocks of 4 elements resident per SM:
// three of the viscous update kernel, five of the Euler one, four with the Roe
// flux; where filling only doubles the elements, a second wave of Euler blocks
// is no slower either.  A stage, us, blocks of 4 elements / filled: triangles of
// P = 3 Navier-Stokes, 1404: 12.6 / 14.7, 2520: 18.7 / 16.7, 8448: 34.7 / 28.9;
// Euler 1984: 10.5 / 12.6, 2960: 10.5 / 13.6, 6048: 16.7 / 14.6; P = 2 Roe 1404:
// 10.5 / 12.6, 2520: 14.6 / 12.6; quads of P = 3 Euler, 5850: 16.7 / 18.7, 8188:
// 20.8 / 19.1.
template <int D, int NU, int NF>
MixedKernels mixed_kernels_for(long long E, int pf)
{
  constexpr bool doubles = shape_epb(kUpdShapes[1], NF, true) <= 2 * kUpdShapes[1].epb;
  const int per_sm = pf == 0 ? 3 : (pf == 2 ? 4 : (doubles ? 10 : 5));
  return E > 4LL * 148 * per_sm ? mixed_kernels<D, NU, NF, true>() : mixed_kernels<D, NU, NF, false>();
}

// the kernels of the 2-D element types of orders 2 and 3 (fr_mixed_fused_2d.cu)
bool find_kernels_2d(int NU, int NF, long long E, int pf, MixedKernels* out);
// the kernels of orders 1 and 4 (fr_mixed_fused_p14.cu)
bool find_kernels_p14(int D, int NU, int NF, long long E, int pf, MixedKernels* out);

}  // namespace frb_mixed
