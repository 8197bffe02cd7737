// fr_update.cuh -- the last part of an RK stage, one element-blocked kernel:
// norm_tconf - norm_tdisf, the VCJH correction (calculate_corrected_divergence,
// src/eles.cpp:1594-1661) and the RK45 stage update (eles::AdvanceSolution,
// src/eles.cpp:1155-1178) with the next stage's flux-point traces, or the
// residual alone.  Two forms:
//   FUSED 1  the common interface fluxes of the element's own flux points are
//            formed here (int_inters::calculate_common_invFlux,
//            src/int_inters.cpp:225-354, calculate_common_viscFlux,
//            src/int_inters.cpp:359-470; boundary points as
//            bdy_inters::evaluate_boundaryConditions_invFlux,
//            src/bdy_inters.cpp:245-389).  Both elements of an interface
//            evaluate its flux, each for its own flux point, from the same two
//            traces, the same left normal and their own dA, so the two copies
//            are the ones a separate interface pass writes for the two sides.
//            The own trace is interpolated from the state held here (the
//            arithmetic that produced the stored traces, so the values agree
//            bit for bit).
//   FUSED 0  fr_face_kernel has written them to CF.
// Bound: HBM (hex P = 3 FP64: 30.6 kB per element and stage).  A flux-point
// thread's own inputs (neighbour trace and projections, own projections,
// normals, dA, normal flux) are each used once by that thread, so they go to
// registers, all loads in flight at once; what a solution point needs (state,
// register, divergence, inverse Jacobian) is copied to shared memory by
// cp.async, the state in a padded order for the line reads of the traces.  The
// bulk-copy version of this kernel (about a hundred copies per element issued
// by two warps, every input through shared memory, 4.2 k warp instructions per
// element) was bound by instruction issue.  32^3, a stage: 222 us against
// 229 in FP64, 156 against 172 in FP32.
#pragma once

#include <cuda_runtime.h>

#include "fr_fused.cuh"

namespace frb {

// Whether a stage's update kernel forms the interface fluxes itself: quads, and
// hexes of odd order.  Hexes of orders 2 and 4 run fr_face_kernel first, which
// forms each interface's flux once instead of from both sides.  A stage with it
// / without it (best update tile of each), us: 64000 hexes P = 2 573 / 610, FP32
// 411 / 435; 18000 walled, WALE 261 / 273; 13824 hexes P = 4 405 / 441, FP32 298
// / 312; 4845 P = 4 149 / 161; Euler the same within 2 %.  Meshes that do not
// fill the GPU would do better without (512 hexes P = 2 12.8 / 11.1, 150 of P = 4
// 14.0 / 13.2); an order has one form, whatever the mesh.
template <int DIM, int P>
__host__ __device__ constexpr bool update_fused()
{
  return DIM == 2 || P % 2 == 1;
}

__device__ __forceinline__ void cp_async_wait_but1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// Shared-memory plan (byte offsets): state [F][element][PtMap::N] (FP64), RK
// register, 1/detJ (MODE 1), norm_tconf - norm_tdisf [F][element][NF],
// divergence (viscous), transformed flux and JGinv (inviscid), opp_3 factors
// (and, inviscid, the derivative rows) that threads index with their own point,
// norm partials.
template <int DIM, int P, int EPB, int NT, int VISC, int MODE, typename TC>
struct UpdPlan {
  using S = Shape<DIM, P>;
  __host__ __device__ static constexpr size_t r16(size_t b) { return (b + 15) / 16 * 16; }
  static constexpr size_t NW = EPB * (size_t)PtMap<DIM, P, double>::N, NWT = EPB * (size_t)PtMap<DIM, P, TC>::N;
  static constexpr size_t bU = r16(8 * S::F * NW);
  static constexpr size_t bREG = MODE == 1 ? r16(8 * (size_t)EPB * S::F * S::NU) : 0;
  static constexpr size_t bIDJ = MODE == 1 ? r16(8 * (size_t)EPB * S::NU) : 0;
  static constexpr size_t bC = r16(sizeof(TC) * EPB * S::F * S::NF);
  static constexpr size_t bDV = VISC ? r16(sizeof(TC) * EPB * S::F * S::NU) : 0;
  static constexpr size_t bFL = VISC ? 0 : r16(sizeof(TC) * DIM * S::F * NWT);
  static constexpr size_t bJ = VISC ? 0 : r16(sizeof(TC) * EPB * DIM * DIM * S::NU);
  static constexpr size_t bG = r16(sizeof(TC) * (2 * (P + 1) + (VISC ? 0 : (P + 1) * (P + 1))));
  static constexpr size_t bRED = MODE == 1 ? r16(sizeof(double) * (NT / 32) * S::F) : 0;
  static constexpr size_t oU = 0, oREG = oU + bU, oIDJ = oREG + bREG, oC = oIDJ + bIDJ, oDV = oC + bC,
                          oFL = oDV + bDV, oJ = oFL + bFL, oG = oJ + bJ, oRED = oG + bG, total = oRED + bRED;
};

template <int DIM, int P, int EPB, int NT, int VISC, int MODE, typename TC>
__host__ __device__ constexpr size_t update_smem_bytes()
{
  return UpdPlan<DIM, P, EPB, NT, VISC, MODE, TC>::total;
}

// Common normal flux (times the own dA) of a boundary flux point:
// bdy_inters::evaluate_boundaryConditions_invFlux (src/bdy_inters.cpp:245-389):
// ghost state, then the central flux of the two states
// (convective_flux_boundary, src/inters.cpp:368-387), Roe in 2-D with
// RIEMANN 2, the own flux for slip_wall_dual (right_flux,
// src/inters.cpp:299-308); plus the viscous part from the gradient kernel.
template <int DIM, typename TC>
struct FUBdy {
  TC ul[DIM + 2], n[DIM], tl, bv[DIM + 2];
};
template <int DIM, int VISC, typename TC, int RIEMANN>
__device__ __noinline__ void fu_boundary(PhysT<TC> ph, int type, FUBdy<DIM, TC> q, TC* c, int cst)
{
  constexpr int F = DIM + 2, D = DIM;
  TC ug[F], fn[F];
  bc_ghost<D, TC>(ph, type, q.ul, q.n, ug);
  TC fl[F][D], fr[F][D];
  inv_flux<D, TC>(ph, q.ul, fl);
  inv_flux<D, TC>(ph, ug, fr);
  if (type == 16) {
    for (int k = 0; k < F; k++) {
      TC s = fl[k][0] * q.n[0];
      for (int l = 1; l < D; l++) s = s + fl[k][l] * q.n[l];
      fn[k] = s;
    }
  } else if (RIEMANN == 2 && DIM == 2) {
    roe<TC>(ph, q.ul, ug, q.n, fn);
  } else {
    for (int k = 0; k < F; k++) {
      TC s = fl[k][0] * q.n[0], r = fr[k][0] * q.n[0];
      for (int l = 1; l < D; l++) { s = s + fl[k][l] * q.n[l]; r = r + fr[k][l] * q.n[l]; }
      fn[k] = TC(0.5) * (s + r);
    }
  }
  for (int k = 0; k < F; k++) {
    TC v = fn[k] * q.tl;
    if (VISC) v = v + q.bv[k] * q.tl;
    c[k * cst] = v;
  }
}

// What a flux-point thread loads: the neighbour's and the own viscous
// projections, the neighbour's trace, the left normal, the own dA and the
// normal flux (FUSED 1), or the common flux and the normal flux (FUSED 0).
template <int D, int VISC, int FUSED, typename TC>
struct FptIn {
  static constexpr int F = D + 2;
  int mt;
  unsigned char sd;
  TC un[FUSED ? F : 1], vn[FUSED && VISC ? F - 1 : 1], vo[FUSED && VISC ? F - 1 : 1], n[FUSED ? D : 1], tl;
  TC nd[VISC ? F : 1], cf[FUSED ? 1 : F];
};

// idetj holds 1/detJ at the solution points (the update multiplies by it).
// BV is the viscous normal flux of boundary points from the gradient kernel
// (side bits 2.. hold the boundary type there, and mate = -1 - the point's
// place in the boundary list).  MINB: CTAs per SM the registers are capped
// for.  VEC = 0: inputs only 8-byte aligned.  The body serves element block
// blk (fr_update_kernel: blockIdx.x; merged batch launches: their share of
// the grid).
template <int DIM, int P, int EPB, int NT, int VISC, int MODE, typename TC, int FUSED, int RIEMANN = 0, int VEC = 1>
__device__ __forceinline__ void
fr_update_body(long long blk, double* __restrict__ U, double* __restrict__ REG, TC* __restrict__ UFn,
               const TC* __restrict__ UF, const TC* __restrict__ CF, const int* __restrict__ mate,
               const unsigned char* __restrict__ side, const TC* __restrict__ VF, const TC* __restrict__ ND,
               const TC* __restrict__ DV, const TC* __restrict__ JG, const TC* __restrict__ nL,
               const TC* __restrict__ tdA, const double* __restrict__ idetj, const TC* __restrict__ BV,
               double* __restrict__ DIV, double* __restrict__ partial, long long E, const Line<TC>& L,
               const PhysT<TC>& ph, double rk_a, double rk_b, double dt, int first_stage)
{
  using S = Shape<DIM, P>;
  using MU = PtMap<DIM, P, double>;
  using MT = PtMap<DIM, P, TC>;
  using Q = UpdPlan<DIM, P, EPB, NT, VISC, MODE, TC>;
  constexpr int N1 = P + 1, NU = S::NU, NF = S::NF, F = S::F, D = DIM, DD = DIM * DIM;
  constexpr int NW = (int)Q::NW, NWT = (int)Q::NWT;
  constexpr int IF = Items<NT, EPB * NF>::N, IU = Items<NT, EPB * NU>::N;
  extern __shared__ __align__(16) unsigned char fr_smem[];
  double* sU = reinterpret_cast<double*>(fr_smem + Q::oU);
  double* sREG = reinterpret_cast<double*>(fr_smem + Q::oREG);
  double* sIDJ = reinterpret_cast<double*>(fr_smem + Q::oIDJ);
  TC* sC = reinterpret_cast<TC*>(fr_smem + Q::oC);
  TC* sDV = reinterpret_cast<TC*>(fr_smem + Q::oDV);
  TC* sFl = reinterpret_cast<TC*>(fr_smem + Q::oFL);
  TC* sJ = reinterpret_cast<TC*>(fr_smem + Q::oJ);
  TC* sg = reinterpret_cast<TC*>(fr_smem + Q::oG);   // gL (negated), gR, derivative rows (inviscid)
  auto sRed = reinterpret_cast<double (*)[F]>(fr_smem + Q::oRED);
  const int tid = threadIdx.x;
  const long long e0 = blk * EPB;
  const int nval = (int)(E - e0 < EPB ? E - e0 : EPB), nuv = nval * NU;
  const long long NFE = (long long)NF * E;
  const bool want_reg = MODE == 1 && !first_stage;

  // --- asynchronous copies: the state (and JGinv) first, then what the
  // solution points need
  {
    constexpr int V8 = (VEC && NU % 2 == 0) ? 2 : 1, R = EPB * NU / V8;
    for (int w = tid; w < F * R; w += NT) {
      const int k = w / R, r = (w - k * R) * V8;
      if (r < nuv) cp_async<8 * V8>(sU + k * NW + MU::run(r), U + (size_t)NU * (e0 + E * k) + r);
    }
    if constexpr (!VISC) {
      constexpr int VJ = (VEC && (EPB * DD * NU * sizeof(TC)) % 16 == 0) ? 16 / sizeof(TC) : 1;
      cp_run<VJ, NT>(sJ, JG + (size_t)DD * NU * e0, DD * nuv);
    }
    cp_async_commit();
    constexpr int VT = (VEC && (NU * sizeof(TC)) % 16 == 0) ? 16 / sizeof(TC) : 1, RT = EPB * NU / VT;
    if (want_reg)
      for (int w = tid; w < F * R; w += NT) {
        const int k = w / R, r = (w - k * R) * V8;
        if (r < nuv) cp_async<8 * V8>(sREG + k * EPB * NU + r, REG + (size_t)NU * (e0 + E * k) + r);
      }
    if constexpr (VISC != 0)
      for (int w = tid; w < F * RT; w += NT) {
        const int k = w / RT, r = (w - k * RT) * VT;
        if (r < nuv) cp_async<(int)sizeof(TC) * VT>(sDV + k * EPB * NU + r, DV + (size_t)NU * (e0 + E * k) + r);
      }
    if (MODE == 1) cp_run<V8, NT>(sIDJ, idetj + (size_t)NU * e0, nuv);
    cp_async_commit();
  }
  if (tid < N1) {
    sg[tid] = -L.gL[tid];
    sg[N1 + tid] = L.gR[tid];
  }
  if constexpr (!VISC)
    for (int i = tid; i < N1 * N1; i += NT) sg[2 * N1 + i] = L.D[i / N1][i % N1];

  // --- a flux-point thread's inputs
  auto load = [&](int w, FptIn<D, VISC, FUSED, TC>& in) {
    const int el = w / NF, f = w - el * NF;
    const long long own = f + NF * (e0 + el);
    if constexpr (FUSED != 0) {
      in.mt = mate[own];
      in.sd = side[own];
      in.tl = tdA[own];
#pragma unroll
      for (int d = 0; d < D; d++) in.n[d] = nL[own + NFE * d];
      if constexpr (VISC != 0)
#pragma unroll
        for (int k = 0; k < F - 1; k++) in.vo[k] = VF[own + NFE * k];
    } else {
#pragma unroll
      for (int k = 0; k < F; k++) in.cf[k] = CF[own + NFE * k];
    }
    if constexpr (VISC != 0)
#pragma unroll
      for (int k = 0; k < F; k++) in.nd[k] = ND[own + NFE * k];
    if constexpr (FUSED != 0) {
      // without a branch between the loads; a boundary point takes the viscous
      // normal flux of the gradient kernel for `un` (its own trace, unused, on
      // the Euler path) and its own projections, unused, for `vn`
      const bool bd = in.mt < 0;
      const long long mo = bd ? own : (long long)in.mt;
      const TC* pu = UF + mo;
      long long st = NFE;
      if (VISC && bd) {
        pu = BV + (-1 - (long long)in.mt) * F;
        st = 1;
      }
#pragma unroll
      for (int k = 0; k < F; k++) in.un[k] = pu[st * k];
      if constexpr (VISC != 0)
#pragma unroll
        for (int k = 0; k < F - 1; k++) in.vn[k] = VF[mo + NFE * k];
    }
  };
  FptIn<D, VISC, FUSED, TC> in0;
  if constexpr (IF == 1)
    if (tid < nval * NF) load(tid, in0);
  cp_async_wait_but1();
  __syncthreads();

  // --- Euler path: transformed inviscid flux at the solution points
  // (evaluate_invFlux, src/eles.cpp:1331-1418)
  if constexpr (!VISC) {
#pragma unroll
    for (int it = 0; it < IU; it++) {
      const int w = tid + it * NT, el = w / NU, u = w - el * NU;
      if (w >= nuv) continue;
      int a, b, c;
      upt_abc<DIM, P>(u, a, b, c);
      TC g[DD], qv[F], fi[F][D];
#pragma unroll
      for (int q = 0; q < DD; q++) g[q] = sJ[DD * w + q];
#pragma unroll
      for (int k = 0; k < F; k++) qv[k] = (TC)sU[k * NW + el * MU::N + MU::slot(a, b, c)];
      inv_flux<D, TC>(ph, qv, fi);
#pragma unroll
      for (int l = 0; l < D; l++)
#pragma unroll
        for (int k = 0; k < F; k++) {
          TC acc = g[l] * fi[k][0];
#pragma unroll
          for (int m = 1; m < D; m++) acc = acc + g[l + D * m] * fi[k][m];
          sFl[(l * F + k) * NWT + el * MT::N + MT::slot(a, b, c)] = acc;
        }
    }
    __syncthreads();
  }

  // the line through a flux point: first point, axis, end
  struct FLine { int a, b, c, ax; bool plus; };
  auto fline = [&](int f) {
    FLine q;
    int u0, st;
    fpt_line<DIM, P>(f, u0, st, q.ax, q.plus);
    upt_abc<DIM, P>(u0, q.a, q.b, q.c);
    return q;
  };
  auto trace = [&](const double* s, int st, bool plus) {
    // the opp_0 row of f in column order, (((0 + t0) + t1) + ...)
    TC acc = TC(0);
#pragma unroll
    for (int m = 0; m <= P; m++) acc = acc + (TC)s[m * st] * (plus ? L.Lp[m] : L.Lm[m]);
    return acc;
  };

  // --- common fluxes at the own flux points, minus the discontinuous normal flux
#pragma unroll
  for (int it = 0; it < IF; it++) {
    const int w = tid + it * NT, el = w / NF, f = w - el * NF;
    if (w >= nval * NF) continue;
    if constexpr (IF > 1) load(w, in0);
    const FptIn<D, VISC, FUSED, TC>& in = in0;
    TC c[F];
    FLine ln;
    if (FUSED || !VISC) ln = fline(f);
    if constexpr (FUSED != 0) {
      const double* su = sU + el * MU::N + MU::slot(ln.a, ln.b, ln.c);
      const int st = ln.ax == 0 ? 1 : (ln.ax == 1 ? MU::S1 : MU::S2);
      TC uo[F];
#pragma unroll
      for (int k = 0; k < F; k++) uo[k] = trace(su + k * NW, st, ln.plus);
      if (in.sd >> 2) {
        FUBdy<DIM, TC> q;
#pragma unroll
        for (int k = 0; k < F; k++) {
          q.ul[k] = uo[k];
          q.bv[k] = in.un[k];
        }
#pragma unroll
        for (int d = 0; d < D; d++) q.n[d] = in.n[d];
        q.tl = in.tl;
        fu_boundary<DIM, VISC, TC, RIEMANN>(ph, in.sd >> 2, q, c, 1);
      } else {
        const bool left = in.sd & 1;
        TC ul[F], ur[F], fn[F];
#pragma unroll
        for (int k = 0; k < F; k++) {
          ul[k] = left ? uo[k] : in.un[k];
          ur[k] = left ? in.un[k] : uo[k];
        }
        if constexpr (RIEMANN == 2 && DIM == 2) roe<TC>(ph, ul, ur, in.n, fn);
        else rusanov<D, TC>(ph, ul, ur, in.n, fn);
        const TC ts = left ? in.tl : -in.tl;   // the right side's flux points the other way
#pragma unroll
        for (int k = 0; k < F; k++) c[k] = fn[k] * ts;
        if constexpr (VISC != 0) {
          TC nn = in.n[0] * in.n[0];
#pragma unroll
          for (int d = 1; d < D; d++) nn = fr_fma(in.n[d], in.n[d], nn);
          const TC pen = (in.sd & 2) ? -ph.pen_fact : ph.pen_fact;
          // every field, density included, takes the tau (u_l - u_r) penalty;
          // the density's viscous projections are zero
#pragma unroll
          for (int k = 0; k < F; k++) {
            const TC ao = k ? in.vo[k ? k - 1 : 0] : TC(0), an = k ? in.vn[k ? k - 1 : 0] : TC(0);
            const TC fv = ldg_normal<TC>(left ? ao : an, left ? an : ao, ul[k], ur[k], pen, ph.tau, nn);
            c[k] = c[k] + fv * ts;
          }
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < F; k++) c[k] = in.cf[k];
    }
    if constexpr (VISC != 0) {
#pragma unroll
      for (int k = 0; k < F; k++) sC[(k * EPB + el) * NF + f] = c[k] - in.nd[k];   // daxpy(-1, norm_tdisf, norm_tconf)
    } else {
      // norm_tdisf from the transformed flux (extrapolate_totalFlux), then norm_tconf - norm_tdisf
      const TC* sf = sFl + ln.ax * F * NWT + el * MT::N + MT::slot(ln.a, ln.b, ln.c);
      const int st = ln.ax == 0 ? 1 : (ln.ax == 1 ? MT::S1 : MT::S2);
#pragma unroll
      for (int k = 0; k < F; k++) {
        TC v = TC(0);
#pragma unroll
        for (int m = 0; m <= P; m++) v = v + sf[k * NWT + m * st] * (ln.plus ? L.Lp[m] : L.Lm[m]);
        sC[(k * EPB + el) * NF + f] = c[k] - (ln.plus ? v : -v);
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();

  // --- correction and update at the solution points
  double red[F];
#pragma unroll
  for (int k = 0; k < F; k++) red[k] = 0.0;
#pragma unroll
  for (int it = 0; it < IU; it++) {
    const int w = tid + it * NT, el = w / NU, u = w - el * NU;
    if (w >= nuv) continue;
    int abc[3];
    upt_abc<DIM, P>(u, abc[0], abc[1], abc[2]);
    const int su = MU::slot(abc[0], abc[1], abc[2]);
    // opp_3 row of u: one column per face, in flux-point order (the same for every field)
    int qf[S::NFACE];
    TC cf[S::NFACE];
#pragma unroll
    for (int fc = 0; fc < S::NFACE; fc++) {
      int al;
      qf[fc] = face_fpt<DIM, P>(fc, abc[0], abc[1], abc[2], al);
      cf[fc] = sg[(face_plus<DIM>(fc) ? N1 : 0) + al];
    }
    const double idj = MODE == 1 ? sIDJ[w] : 1.0;
#pragma unroll
    for (int k = 0; k < F; k++) {
      const size_t gi = (size_t)NU * (e0 + E * k) + w;
      TC acc;
      if constexpr (VISC != 0) {
        acc = sDV[k * EPB * NU + w];
      } else {
        acc = TC(0);
#pragma unroll
        for (int d = 0; d < D; d++) {
          const TC* s = sFl + (d * F + k) * NWT + el * MT::N +
                        MT::slot(d == 0 ? 0 : abc[0], d == 1 ? 0 : abc[1], d == 2 ? 0 : abc[2]);
#pragma unroll
          for (int m = 0; m <= P; m++) acc = acc + s[m * MT::stride(d)] * sg[2 * N1 + N1 * abc[d] + m];
        }
      }
      const TC* cc = sC + (k * EPB + el) * NF;
#pragma unroll
      for (int fc = 0; fc < S::NFACE; fc++) acc = acc + cc[qf[fc]] * cf[fc];
      const double R = (double)acc;
      if (MODE == 0) {
        DIV[gi] = R;
      } else {
        const double rhs = -R * idj;
        const double res = first_stage ? dt * rhs : rk_a * sREG[k * EPB * NU + w] + dt * rhs;
        REG[gi] = res;
        double* us = sU + k * NW + el * MU::N + su;
        const double un = *us + rk_b * res;
        U[gi] = un;
        *us = un;
        red[k] += fabs(rhs);
      }
    }
  }
  if constexpr (MODE == 1) {
    if (partial) {
      // deterministic per-block partial sums of |div/detjac| (CalcNormResidual)
      const int lane = tid & 31, wid = tid >> 5;
#pragma unroll
      for (int k = 0; k < F; k++) {
        double v = red[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sRed[wid][k] = v;
      }
    }
    __syncthreads();
    if (partial && tid < F) {
      double v = 0.0;
      for (int i = 0; i < NT / 32; i++) v += sRed[i][tid];
      partial[(size_t)blk * F + tid] = v;
    }
    // traces of the updated state for the next stage
#pragma unroll
    for (int it = 0; it < IF; it++) {
      const int w = tid + it * NT, el = w / NF, f = w - el * NF;
      if (w >= nval * NF) continue;
      const FLine ln = fline(f);
      const double* su = sU + el * MU::N + MU::slot(ln.a, ln.b, ln.c);
      const int st = ln.ax == 0 ? 1 : (ln.ax == 1 ? MU::S1 : MU::S2);
#pragma unroll
      for (int k = 0; k < F; k++) UFn[f + NF * (e0 + el) + NFE * k] = trace(su + k * NW, st, ln.plus);
    }
  }
}

template <int DIM, int P, int EPB, int NT, int VISC, int MODE, typename TC, int FUSED, int RIEMANN = 0, int MINB = 1,
          int VEC = 1>
__global__ void __launch_bounds__(NT, MINB)
fr_update_kernel(double* __restrict__ U, double* __restrict__ REG, TC* __restrict__ UFn, const TC* __restrict__ UF,
                 const TC* __restrict__ CF, const int* __restrict__ mate, const unsigned char* __restrict__ side,
                 const TC* __restrict__ VF, const TC* __restrict__ ND, const TC* __restrict__ DV,
                 const TC* __restrict__ JG, const TC* __restrict__ nL, const TC* __restrict__ tdA,
                 const double* __restrict__ idetj, const TC* __restrict__ BV, double* __restrict__ DIV,
                 double* __restrict__ partial, long long E, Line<TC> L, PhysT<TC> ph, double rk_a, double rk_b,
                 double dt, int first_stage)
{
  fr_update_body<DIM, P, EPB, NT, VISC, MODE, TC, FUSED, RIEMANN, VEC>(blockIdx.x, U, REG, UFn, UF, CF, mate, side, VF,
                                                                       ND, DV, JG, nL, tdA, idetj, BV, DIV, partial,
                                                                       E, L, ph, rk_a, rk_b, dt, first_stage);
}

}  // namespace frb
