// fr_fused.cuh -- fused, sum-factorised FR stage kernels for tensor-product
// elements (quadrilaterals D=2, hexahedra D=3) on sm_100a.
//
// One RK stage of the reference (CalcResidual, src/solver.cpp:65-225, then
// eles::AdvanceSolution, src/eles.cpp:1091-1188) runs as
//   viscous :  fr_grad_kernel -> [fr_face_kernel ->] fr_update_kernel
//   inviscid:                    [fr_face_kernel ->] fr_update_kernel
// with the interface kernel folded into the update where that is the faster
// form (fr_update.cuh).  The element kernels are element-blocked: a CTA owns
// EPB elements, stages their solution in shared memory, and applies the
// reference's operators as 1-D line contractions (every dense operator opp_0..opp_6 of a Gauss-point tensor
// element has exactly one non-trivial factor per line, so the contraction
// reproduces the dense product term by term).  Elements exchange data only
// through flux-point traces in HBM:
//   UF  (n_fpts, n_eles, F)      solution at the flux points, double-buffered
//                                across stages (written by the stage update)
//   VF  (n_fpts, n_eles, F-1)    own viscous flux at the flux points projected
//                                on the interface's left normal (viscous path)
//   ND  (n_fpts, n_eles, F)      normal discontinuous flux (norm_tdisf_fpts)
//   DV  (n_upts, n_eles, F)      divergence of the discontinuous flux
//   CF  (n_fpts, n_eles, F)      common normal flux times tdA (norm_tconf_fpts)
// mate[i] is the flat index (fpt + n_fpts*ele) of the matching point across
// the interface; side[i] bit 0 = this side is the left one, bit 1 = the LDG
// penalty sign is negative.  Both sides evaluate the common flux with the
// left/right roles and the left normal nL, so the two copies are identical.
#pragma once

#include <cuda_runtime.h>

#include "fr_physics.cuh"

namespace frb {

constexpr int kMaxN1 = 6;   // P <= 5 in the fused kernels

template <typename T>
struct Line {               // 1-D operator pieces (see Line1D in fr_host.hpp)
  T Lm[kMaxN1], Lp[kMaxN1], D[kMaxN1][kMaxN1], gL[kMaxN1], gR[kMaxN1], w[kMaxN1];
};

template <int DIM, int P>
struct Shape {
  static constexpr int N1 = P + 1;
  static constexpr int NU = DIM == 2 ? N1 * N1 : N1 * N1 * N1;
  static constexpr int NFPF = DIM == 2 ? N1 : N1 * N1;
  static constexpr int NFACE = 2 * DIM;
  static constexpr int NF = NFACE * NFPF;
  static constexpr int F = DIM + 2;
};

// Line through flux point f: first solution point, stride along the line,
// axis, and whether the face is at the +1 end.  Reference orderings:
// quads src/eles_quads.cpp:259-300, hexes src/eles_hexas.cpp:262-324.
template <int DIM, int P>
__device__ __forceinline__ void fpt_line(int f, int& u0, int& stride, int& axis, bool& plus)
{
  constexpr int N1 = P + 1;
  if (DIM == 2) {
    int fc = f / N1, j = f - fc * N1;
    switch (fc) {
      case 0: u0 = j; stride = N1; axis = 1; plus = false; break;
      case 1: u0 = N1 * j; stride = 1; axis = 0; plus = true; break;
      case 2: u0 = P - j; stride = N1; axis = 1; plus = true; break;
      default: u0 = N1 * (P - j); stride = 1; axis = 0; plus = false; break;
    }
  } else {
    constexpr int N2 = N1 * N1;
    int fc = f / N2, r = f - fc * N2, j = r / N1, k = r - j * N1;
    switch (fc) {
      case 0: u0 = (P - k) + N1 * j; stride = N2; axis = 2; plus = false; break;
      case 1: u0 = k + N2 * j; stride = N1; axis = 1; plus = false; break;
      case 2: u0 = N1 * k + N2 * j; stride = 1; axis = 0; plus = true; break;
      case 3: u0 = (P - k) + N2 * j; stride = N1; axis = 1; plus = true; break;
      case 4: u0 = N1 * (P - k) + N2 * j; stride = 1; axis = 0; plus = false; break;
      default: u0 = k + N1 * j; stride = N2; axis = 2; plus = true; break;
    }
  }
}

// Flux point of face fc on the line through solution point (a, b, c), and the
// index of that point along the face normal.
template <int DIM, int P>
__device__ __forceinline__ int face_fpt(int fc, int a, int b, int c, int& along)
{
  constexpr int N1 = P + 1;
  if (DIM == 2) {
    switch (fc) {
      case 0: along = b; return a;
      case 1: along = a; return N1 + b;
      case 2: along = b; return 2 * N1 + (P - a);
      default: along = a; return 3 * N1 + (P - b);
    }
  }
  constexpr int N2 = N1 * N1;
  switch (fc) {
    case 0: along = c; return (P - a) + N1 * b;
    case 1: along = b; return N2 + a + N1 * c;
    case 2: along = a; return 2 * N2 + b + N1 * c;
    case 3: along = b; return 3 * N2 + (P - a) + N1 * c;
    case 4: along = a; return 4 * N2 + (P - b) + N1 * c;
    default: along = c; return 5 * N2 + a + N1 * b;
  }
}

// end of face fc (reference normals: quads f0 -y, f1 +x, f2 +y, f3 -x;
// hexes f0 -z, f1 -y, f2 +x, f3 +y, f4 -x, f5 +z)
template <int DIM>
__device__ __forceinline__ bool face_plus(int fc)
{
  if (DIM == 2) return fc == 1 || fc == 2;
  return fc == 2 || fc == 3 || fc == 5;
}

// Value at flux point f of a field stored point-major (s[u * sst]): the
// reference's opp_0 row of f applied in column order, (((0 + t0) + t1) + ...).
template <int DIM, int P, typename T, typename S>
__device__ __forceinline__ T line_interp(const Line<T>& L, const S* s, int sst, int f)
{
  int u0, st, ax; bool plus;
  fpt_line<DIM, P>(f, u0, st, ax, plus);
  T acc = T(0);
#pragma unroll
  for (int m = 0; m <= P; m++) acc = acc + (T)s[(u0 + m * st) * sst] * (plus ? L.Lp[m] : L.Lm[m]);
  return acc;
}

template <int DIM, int P>
__device__ __forceinline__ void upt_abc(int u, int& a, int& b, int& c)
{
  constexpr int N1 = P + 1;
  if (DIM == 2) { b = u / N1; a = u - b * N1; c = 0; }
  else { c = u / (N1 * N1); int r = u - c * N1 * N1; b = r / N1; a = r - b * N1; }
}

// Faces at the two ends of the lines along axis d (minus end, plus end).
template <int DIM>
__host__ __device__ constexpr int line_face(int d, int plus)
{
  return DIM == 2 ? (d == 0 ? (plus ? 1 : 3) : (plus ? 2 : 0))
                  : (d == 0 ? (plus ? 2 : 4) : (d == 1 ? (plus ? 3 : 1) : (plus ? 5 : 0)));
}

// Shared-memory order of a field's solution points: point (a, b, c) of an
// element at a + S1 b + S2 c, N words per element.  Hexahedra of P = 3 pad
// the z-planes of 16 points (18 doubles, 20 floats): lines along x are then
// read as whole 16-byte vectors without bank conflicts, lines along z too,
// lines along y with 2-way conflicts in FP64 and none in FP32 (unpadded: 4-way
// along y).  The other point counts are free of conflicts, or 2-way, as they are.
template <int DIM, int P, typename TC>
struct PtMap {
  static constexpr int N1 = P + 1;
  static constexpr int S1 = N1;
  static constexpr int S2 = DIM == 3 ? (N1 == 4 ? (sizeof(TC) == 8 ? 18 : 20) : N1 * N1) : 0;
  static constexpr int N = DIM == 3 ? S2 * N1 : N1 * N1;
  static constexpr int PLANE = DIM == 3 ? N1 * N1 : N1 * N1;   // points per unpadded run
  __device__ static __forceinline__ int slot(int a, int b, int c) { return a + S1 * b + S2 * c; }
  __host__ __device__ static constexpr int stride(int d) { return d == 0 ? 1 : (d == 1 ? S1 : S2); }
  // slot of the first point of line (j0, j1) along axis d, whose points are (., j0, j1), (j0, ., j1), (j0, j1, .)
  __device__ static __forceinline__ int line(int d, int j0, int j1)
  {
    return d == 0 ? S1 * j0 + S2 * j1 : (d == 1 ? j0 + S2 * j1 : j0 + S1 * j1);
  }
  // slot of point r of a run of whole elements
  __device__ static __forceinline__ int run(int r)
  {
    if constexpr (DIM == 3 && S2 != N1 * N1) return (r / PLANE) * S2 + r % PLANE;
    else return r;
  }
};

template <int NT, int ITEMS>
struct Items {
  static constexpr int N = (ITEMS + NT - 1) / NT;
};

// ---------------------------------------------------------------------------
// Initial flux-point traces from the state (used once after the state is set).
template <int DIM, int P, typename TC>
__global__ void fr_trace_kernel(const double* __restrict__ U, TC* __restrict__ UF, long long E, Line<TC> L,
                                double* __restrict__ Uout = nullptr)
{
  using S = Shape<DIM, P>;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // with Uout, U is a staged state that the same pass copies into place
  // (the grid then covers max(NF, NU) points per element)
  if (Uout && i < E * S::NU)
#pragma unroll
    for (int k = 0; k < S::F; k++) Uout[i + (size_t)S::NU * E * k] = U[i + (size_t)S::NU * E * k];
  if (i >= E * S::NF) return;
  long long e = i / S::NF;
  int f = (int)(i - e * S::NF);
#pragma unroll
  for (int k = 0; k < S::F; k++) {
    const double* ue = U + (size_t)S::NU * (e + E * k);
    UF[f + (size_t)S::NF * (e + E * k)] = line_interp<DIM, P, TC, double>(L, ue, 1, f);
  }
}

// ---------------------------------------------------------------------------
// Asynchronous global -> shared copies (cp.async, sm_80 and later; no
// multicast).  Each thread copies its own elements; cp_async_wait_all plus a
// block barrier makes them visible to the block.
template <int N>
__device__ __forceinline__ void cp_async(void* dst, const void* src)
{
  static_assert(N == 4 || N == 8 || N == 16, "cp.async copies 4, 8 or 16 bytes");
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(src), "n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// N contiguous shared values, 16 bytes per load where N allows (s 16-byte aligned)
template <int N, typename T>
__device__ __forceinline__ void lds_line(const T* s, T (&v)[N])
{
  if constexpr (sizeof(T) == 8 && N % 2 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const double2 q = *reinterpret_cast<const double2*>(s + i);
      v[i] = q.x; v[i + 1] = q.y;
    }
  } else if constexpr (sizeof(T) == 4 && N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 q = *reinterpret_cast<const float4*>(s + i);
      v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = s[i];
  }
}

template <int N, typename T>
__device__ __forceinline__ void sts_line(T* s, const T (&v)[N])
{
  if constexpr (sizeof(T) == 8 && N % 2 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 2) *reinterpret_cast<double2*>(s + i) = make_double2(v[i], v[i + 1]);
  } else if constexpr (sizeof(T) == 4 && N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(s + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) s[i] = v[i];
  }
}

// N values of a line of stride ST (16-byte accesses along x where the rows allow)
template <int N, int ST, typename T>
__device__ __forceinline__ void lds_strided(const T* s, T (&v)[N])
{
  if constexpr (ST == 1) lds_line<N, T>(s, v);
  else {
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = s[i * ST];
  }
}
template <int N, int ST, typename T>
__device__ __forceinline__ void sts_strided(T* s, const T (&v)[N])
{
  if constexpr (ST == 1) sts_line<N, T>(s, v);
  else {
#pragma unroll
    for (int i = 0; i < N; i++) s[i * ST] = v[i];
  }
}

// Contiguous run of n values to shared memory, V values per copy and the
// remainder one by one (dst and src 16-byte aligned where V > 1).
template <int V, int NT, typename T>
__device__ __forceinline__ void cp_run(T* dst, const T* src, int n)
{
  for (int i = threadIdx.x; i < n / V; i += NT) cp_async<(int)sizeof(T) * V>(dst + i * V, src + i * V);
  if constexpr (V > 1)
    for (int i = n / V * V + threadIdx.x; i < n; i += NT) cp_async<(int)sizeof(T)>(dst + i, src + i);
}

// Boundary points of the gradient kernel, out of line so that the hot loop
// bodies stay compact (most meshes have few or no boundary points).  The
// inputs travel by value, so no array of the calling thread has its address
// taken.
template <int D, typename TC>
struct BdyPoint {
  TC u[D + 2], n[D], g[D + 2][D], fv[D + 2][D];
};

// LDG common solution of a boundary point: ghost state from the boundary
// condition, then ldg_solution with flux_spec 1 or 2, u_c = (u_r + u_l)/2
// (bdy_inters::evaluate_boundaryConditions_invFlux, src/bdy_inters.cpp:245-389);
// writes delta = u_c - u_own and u_own at stride st.
template <int D, typename TC>
__device__ __noinline__ void ldg_boundary(PhysT<TC> ph, int type, BdyPoint<D, TC> q, TC* dx, TC* uf, int st)
{
  constexpr int F = D + 2;
  TC ug[F];
  bc_ghost<D, TC>(ph, type, q.u, q.n, ug);
  for (int k = 0; k < F; k++) {
    TC uc = TC(0.5) * (ug[k] + q.u[k]);
    dx[k * st] = uc - q.u[k];
    uf[k * st] = q.u[k];
  }
}

// Viscous normal flux of a boundary point, bdy_inters::evaluate_boundaryConditions_viscFlux
// (src/bdy_inters.cpp:905-1057): own flux q.fv (flux_spec 1) or the ghost
// side's with the adiabatic-wall energy gradient (flux_spec 2, types 12 and
// 14), plus tau n (u_l - u_r), on the normal.  q.g is the own gradient; with
// HAVE_FV = false the own flux is evaluated here from q.u and q.g.
template <int D, typename TC, bool HAVE_FV = true>
__device__ __noinline__ void vis_boundary(PhysT<TC> ph, int type, BdyPoint<D, TC> q, TC* bv)
{
  constexpr int F = D + 2;
  if (!HAVE_FV) vis_flux_fast<D, TC>(ph, q.u, q.g, q.fv);
  TC ug[F];
  bc_ghost<D, TC>(ph, type, q.u, q.n, ug);
  if (type == 12 || type == 14) {
    bc_vis_gradient<D, TC>(ph, q.u, ug, q.g);
    vis_flux_fast<D, TC>(ph, ug, q.g, q.fv);
  }
  for (int k = 0; k < F; k++) {
    TC fnk = (q.fv[k][0] + ph.tau * q.n[0] * (q.u[k] - ug[k])) * q.n[0];
    for (int d = 1; d < D; d++) fnk = fnk + (q.fv[k][d] + ph.tau * q.n[d] * (q.u[k] - ug[k])) * q.n[d];
    bv[k] = fnk;
  }
}

// Shared-memory plan of fr_grad_kernel, in words of TC; "per point" arrays are
// [component][element][PtMap::N]:
//   oF0  state [F], then (each point's own thread overwrites it) the
//        transformed flux along axis 0, then the running divergence
//   oF1  transformed flux along axes 1 .. D-1
//   oM   JGinv (the reference's order, element after element), then detJ
//   oG   reference gradient, then in place the physical gradient [F*D]
//   oUf  own solution at the flux points [F][element][NF]
//   oS   transformed SGS flux [(F-1)*D] (LES only)
//   oMlp the learned closure's parameters (LES 2 only)
// Region sizes are rounded up to 4 words: every region starts on 16 bytes.
template <int DIM, int P, int EPB, typename TC>
struct GradPlan {
  using S = Shape<DIM, P>;
  __host__ __device__ static constexpr int r4(int n) { return (n + 3) / 4 * 4; }
  static constexpr int NW = EPB * PtMap<DIM, P, TC>::N;
  static constexpr int oF0 = 0, oF1 = oF0 + r4(S::F * NW), oM = oF1 + r4((DIM - 1) * S::F * NW);
  static constexpr int oDJ = oM + r4(EPB * DIM * DIM * S::NU), oG = oDJ + r4(EPB * S::NU);
  static constexpr int oUf = oG + r4(S::F * DIM * NW), oS = oUf + r4(S::F * EPB * S::NF);
  __host__ __device__ static constexpr int size(int les) { return oS + (les ? r4((S::F - 1) * DIM * NW) : 0); }
  static constexpr int oMlp = (int)sizeof(TC) * size(1);   // in bytes
};

template <int DIM, int P, int EPB, typename TC, int LES = 0>
__host__ __device__ constexpr size_t grad_smem_bytes()
{
  return sizeof(TC) * GradPlan<DIM, P, EPB, TC>::size(LES) + (LES == 2 ? kMlpSmem : 0);
}

// Viscous stage, part 1 (per element):
//   LDG common solution at every own flux point (the delta_disu_fpts of
//   int_inters::calculate_common_invFlux, src/int_inters.cpp:331-350)
//   -> corrected reference gradient (calculate_gradient + correct_gradient,
//   src/eles.cpp:1667-1968) -> physical gradient
//   -> total discontinuous flux at the solution points (evaluate_invFlux +
//   evaluate_viscFlux) -> its divergence DV (calculate_divergence) and its
//   normal component at the flux points ND (extrapolate_totalFlux)
//   -> viscous flux at the own flux points from the extrapolated state and
//   gradient (what calculate_common_viscFlux evaluates for this side), kept
//   only as its projection on the interface's left normal: VF (F-1 values,
//   the mass component is zero).
// With LES = 1 the eddy-viscosity SGS flux (Smagorinsky, WALE), with LES = 2 the
// learned closure's, joins the viscous flux at the solution points (evaluate_viscFlux, src/eles.cpp:2369-2380); its transformed
// components (sgsf_upts, src/eles.cpp:2382-2409) are extrapolated to the flux
// points (evaluate_sgsFlux, src/eles.cpp:3294-3368) and added there to the
// physical viscous flux before the projection, as calculate_common_viscFlux
// adds sgsf_fpts (src/int_inters.cpp:415-427).
//
// Work split.  The line contractions (traces, reference gradient, divergence,
// normal flux) are one (field, element, line) task per thread and axis: the
// line's values are read once, its operator rows are compile-time entries of
// the constant bank, and the element's fields fill F warps or more; the
// pointwise fluxes are one solution point or flux point per thread, taking the
// gradient one column at a time, so that a point nearly fits 96 registers (FP64
// P = 3: 40 bytes of spill stores; 224 at 80, none at 128 or in FP32; a line's
// two flux points per thread, and whole gradients, filled 128).  Bound: FP64
// issue, 60 k FP64 instructions per hex P = 3 element (948 cycles of an SM).
// One output per thread instead, each reading its line and its operator row
// from shared memory behind run-time index arithmetic, took 5.5 k warp
// instructions per element of which a third were FP64.  A stage's gradient
// kernel, us: 32^3 P = 3 FP64 325 -> 285, FP32 258 -> 213; 4845 hexes P = 4 169
// -> 93; 18000 hexes P = 2 with WALE 225 -> 193; 13031 quads P = 4 57 -> 42.
// The neighbours' traces go to registers (two dependent loads, issued before
// the wait for the staged state); state, JGinv and detJ reach shared memory
// through cp.async.  VEC = 0 keeps every global read element-sized (inputs
// only 8-byte aligned); PERS = 1 makes the blocks persistent: they walk over
// element blocks blk0, blk0 + bstride, ...; MINB is the CTAs per SM the
// registers are sized for.
// Outputs VF (n_fpts, n_eles, F-1), ND (n_fpts, n_eles, F), DV (n_upts, n_eles, F),
// BV (n_boundary_points, F) the viscous normal flux at boundary points (side
// bits 2.. hold the boundary type, mate = -1 - position in the boundary
// list; with BV null the mesh has no boundary points and those bits are
// ignored), and, when GRAD is not null, the corrected physical gradient
// grad_disu_upts (n_upts, n_eles, F, D).
// The body serves element block blk0 (and, with PERS, blk0 + k bstride);
// fr_grad_kernel runs it for blockIdx.x, merged batch launches for their
// share of the grid.
template <int DIM, int P, int EPB, int NT, typename TC, int LES = 0, int VEC = 1, int PERS = 0>
__device__ __forceinline__ void
fr_grad_body(long long blk0, long long bstride, const double* __restrict__ U, const TC* __restrict__ UF,
             const int* __restrict__ mate, const unsigned char* __restrict__ side, const TC* __restrict__ JG,
             const TC* __restrict__ detj, const TC* __restrict__ nL, TC* __restrict__ VF, TC* __restrict__ ND,
             TC* __restrict__ DV, long long E, const Line<TC>& L, const PhysT<TC>& ph, TC* __restrict__ GRAD,
             TC* __restrict__ BV)
{
  using S = Shape<DIM, P>;
  using G = GradPlan<DIM, P, EPB, TC>;
  using M = PtMap<DIM, P, TC>;
  constexpr int N1 = P + 1, NU = S::NU, NF = S::NF, F = S::F, D = DIM, DD = DIM * DIM, NW = G::NW;
  constexpr int NLN = NU / N1;                      // lines per axis
  constexpr int LT = F * EPB * NLN;                 // (field, element, line) tasks per axis
  constexpr int IU = Items<NT, EPB * NU>::N, IF = Items<NT, EPB * NF>::N;
  static_assert(NT >= LT, "one line task per thread");
  extern __shared__ __align__(16) unsigned char fr_smem[];
  TC* sm = reinterpret_cast<TC*>(fr_smem);
  TC* sF0 = sm + G::oF0;
  TC* sJ = sm + G::oM;
  TC* sDJ = sm + G::oDJ;
  TC* sG = sm + G::oG;
  TC* sUf = sm + G::oUf;
  TC* sS = sm + G::oS;
  auto flux = [&](int l, int k, int el) { return sm + (l == 0 ? G::oF0 : G::oF1 + (l - 1) * F * NW) + k * NW + el * M::N; };
  auto grad = [&](int k, int d, int el) { return sG + (k + F * d) * NW + el * M::N; };
  const int tid = threadIdx.x;
  const long long NFE = (long long)NF * E;
  // the closure's parameters, waited for with the state
  if constexpr (LES == 2) cp_run<4, NT>(reinterpret_cast<float*>(fr_smem + G::oMlp), ph.mlp, kMlpN);
  // the thread's line task
  const int k = tid / (EPB * NLN), kr = tid - k * (EPB * NLN), el = kr / NLN, j = kr - el * NLN;
  const int j0 = DIM == 3 ? j % N1 : j, j1 = DIM == 3 ? j / N1 : 0;
  auto end_fpt = [&](int d, int e, int q0, int q1) {
    int al;
    return face_fpt<DIM, P>(line_face<DIM>(d, e), d == 0 ? 0 : q0, d == 0 ? q0 : (d == 1 ? 0 : q1), d == 2 ? 0 : q1, al);
  };

  for (long long blk = blk0;; blk += bstride) {
  const long long e0 = blk * EPB;
  const int nval = (int)(E - e0 < EPB ? E - e0 : EPB);
  const bool line = tid < LT && el < nval;

  // --- inputs: state, metrics (cp.async); the neighbours' traces at both ends
  // of the thread's lines (boundary points, mate < 0, have none)
  {
    constexpr int VU = (VEC && sizeof(TC) == 8 && NU % 2 == 0) ? 2 : 1;
    constexpr int R = EPB * NU / VU, IS = Items<NT, F * R>::N;
    double tmp[sizeof(TC) == 8 ? 1 : IS];   // FP32: every load in flight before the first is rounded
#pragma unroll
    for (int it = 0; it < IS; it++) {
      const int w = tid + it * NT, kk = w / R, r = (w - kk * R) * VU;
      const bool ok = w < F * R && r < nval * NU;
      const double* src = U + (size_t)NU * (e0 + E * kk) + r;
      if constexpr (sizeof(TC) == 8) {
        if (ok) cp_async<8 * VU>(sF0 + kk * NW + M::run(r), src);
      } else {
        tmp[it] = ok ? *src : 1.0;
      }
    }
    if constexpr (sizeof(TC) != 8)
#pragma unroll
      for (int it = 0; it < IS; it++) {
        const int w = tid + it * NT, kk = w / R, r = w - kk * R;
        if (w < F * R && r < nval * NU) sF0[kk * NW + M::run(r)] = (TC)tmp[it];
      }
    constexpr int VJ = (VEC && (EPB * DD * NU * sizeof(TC)) % 16 == 0) ? 16 / sizeof(TC) : 1;
    constexpr int VD = (VEC && (EPB * NU * sizeof(TC)) % 16 == 0) ? 16 / sizeof(TC) : 1;
    cp_run<VJ, NT>(sJ, JG + (size_t)DD * NU * e0, nval * DD * NU);
    cp_run<VD, NT>(sDJ, detj + (size_t)NU * e0, nval * NU);
    cp_async_commit();
  }
  // two rounds of loads, each without a branch between them (one round trip
  // per flux point otherwise): the wiring, then the traces; a boundary point
  // reads its own trace, which is not used
  TC un[D][2];
  unsigned char sd[D][2];
  {
    int mt[D][2];
    const unsigned ob = line ? NF * el : 0;   // block-local: one base per array for the whole block
#pragma unroll
    for (int d = 0; d < D; d++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const unsigned own = ob + end_fpt(d, e, j0, j1);
        mt[d][e] = (mate + NF * e0)[own];
        sd[d][e] = (side + NF * e0)[own];
        if (mt[d][e] < 0) mt[d][e] = (int)(NF * e0 + own);
      }
    const TC* uk = UF + (line ? NFE * k : 0);
#pragma unroll
    for (int d = 0; d < D; d++)
#pragma unroll
      for (int e = 0; e < 2; e++) un[d][e] = uk[mt[d][e]];
  }
  cp_async_wait_all();
  __syncthreads();

  // --- lines: own traces, LDG common solution u_c = (uL+uR)/2 - beta (uL-uR),
  // delta = u_c - u_own, corrected reference gradient along the line (FMAs: it
  // only feeds the viscous flux)
  if (line) {
#pragma unroll
    for (int d = 0; d < D; d++) {
      const int base = M::line(d, j0, j1);
      TC v[N1], dl[2];
      if (d == 0) lds_strided<N1, M::stride(0)>(sF0 + k * NW + el * M::N + base, v);
      else if (d == 1) lds_strided<N1, M::stride(1)>(sF0 + k * NW + el * M::N + base, v);
      else lds_strided<N1, M::stride(2)>(sF0 + k * NW + el * M::N + base, v);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int f = end_fpt(d, e, j0, j1);
        // the reference's opp_0 row of f in column order, (((0 + t0) + t1) + ...)
        TC uo = TC(0);
#pragma unroll
        for (int m = 0; m <= P; m++) uo = uo + v[m] * (e ? L.Lp[m] : L.Lm[m]);
        sUf[(k * EPB + el) * NF + f] = uo;
        if (BV && (sd[d][e] >> 2)) {
          BdyPoint<D, TC> q;
          TC dx[F], uf[F];
#pragma unroll
          for (int kk = 0; kk < F; kk++) {
            TC t = TC(0);
#pragma unroll
            for (int m = 0; m <= P; m++)
              t = t + sF0[kk * NW + el * M::N + base + m * M::stride(d)] * (e ? L.Lp[m] : L.Lm[m]);
            q.u[kk] = t;
          }
          const size_t own = f + (size_t)NF * (e0 + el);
#pragma unroll
          for (int dd = 0; dd < D; dd++) q.n[dd] = nL[own + NFE * dd];
          ldg_boundary<D, TC>(ph, sd[d][e] >> 2, q, dx, uf, 1);
          dl[e] = dx[k];
          continue;
        }
        // the jump u_l - u_r changes its sign with the side (bit 0: left), as
        // the penalty does with bit 1
        const int sb = sd[d][e] & 3;
        const TC pen = (sb == 1 || sb == 2) ? ph.pen_fact : -ph.pen_fact;
        dl[e] = (TC(0.5) * (uo + un[d][e]) - pen * (uo - un[d][e])) - uo;
      }
      TC g[N1];
#pragma unroll
      for (int i = 0; i < N1; i++) {
        TC acc = v[0] * L.D[i][0];
#pragma unroll
        for (int m = 1; m <= P; m++) acc = fr_fma(v[m], L.D[i][m], acc);
        acc = fr_fma(dl[0], L.gL[i], acc);
        g[i] = fr_fma(dl[1], L.gR[i], acc);
      }
      if (d == 0) sts_strided<N1, M::stride(0)>(grad(k, d, el) + base, g);
      else if (d == 1) sts_strided<N1, M::stride(1)>(grad(k, d, el) + base, g);
      else sts_strided<N1, M::stride(2)>(grad(k, d, el) + base, g);
    }
  }
  __syncthreads();

  // --- points: physical gradient and total flux
#pragma unroll
  for (int it = 0; it < IU; it++) {
    const int w = tid + it * NT, pe = w / NU, u = w - pe * NU;
    if (w >= EPB * NU || pe >= nval) continue;
    int a, b, c;
    upt_abc<DIM, P>(u, a, b, c);
    const int su = M::slot(a, b, c);
    TC gr[F][D], q[F];
#pragma unroll
    for (int kk = 0; kk < F; kk++) {
#pragma unroll
      for (int d = 0; d < D; d++) gr[kk][d] = grad(kk, d, pe)[su];
      q[kk] = sF0[kk * NW + pe * M::N + su];
    }
    const TC* gj = sJ + DD * w;
    const TC dj = sDJ[w];
    // physical gradient: d/dx_c = sum_r (JGinv(r,c)/detJ) d/dr
    // (src/eles.cpp:1822-1878), one column at a time into the viscous flux
    const TC inv = fr_rcp(dj);
    VisState<D, TC> vs;
    vis_begin<D, TC>(ph, q, vs);
    TC gp[LES ? F : 1][D];
#pragma unroll
    for (int cc = 0; cc < D; cc++) {
      const TC m0 = gj[0 + D * cc] * inv, m1 = gj[1 + D * cc] * inv, m2 = D == 3 ? gj[2 + D * cc] * inv : TC(0);
      TC col[F];
#pragma unroll
      for (int kk = 0; kk < F; kk++) {
        TC acc = fr_fma(gr[kk][1], m1, gr[kk][0] * m0);
        if (D == 3) acc = fr_fma(gr[kk][D - 1], m2, acc);
        col[kk] = acc;
        if constexpr (LES != 0) gp[kk][cc] = acc;
        grad(kk, cc, pe)[su] = acc;
        if (GRAD) GRAD[u + (size_t)NU * (e0 + pe + E * (kk + (long long)F * cc))] = acc;
      }
      vis_column<D, TC>(vs, cc, col);
    }
    TC fi[F][D], fv[F][D], g[DD];
    inv_flux<D, TC>(ph, q, fi);
    vis_flux_end<D, TC>(vs, fv);
#pragma unroll
    for (int m = 0; m < DD; m++) g[m] = gj[m];
    if constexpr (LES != 0) {
      TC fs[F][D];
      if constexpr (LES == 2) sgs_flux_learned<D, TC>(G::oMlp, ph.gamma, q, gp, dj, TC(P + 1), ph.filter_ratio, fs);
      else sgs_flux<D, TC>(ph, q, gp, dj, TC(P + 1), fs);
#pragma unroll
      for (int kk = 1; kk < F; kk++)
#pragma unroll
        for (int l = 0; l < D; l++) {
          TC t = g[l] * fs[kk][0];
#pragma unroll
          for (int m = 1; m < D; m++) t = t + g[l + D * m] * fs[kk][m];
          sS[((kk - 1) + (F - 1) * l) * NW + pe * M::N + su] = t;
          fv[kk][l] = fv[kk][l] + fs[kk][l];
        }
    }
#pragma unroll
    for (int kk = 0; kk < F; kk++)
#pragma unroll
      for (int l = 0; l < D; l++) {
        // inviscid part in the reference's rounding, viscous part added term by
        // term (the density has none)
        TC acc = g[l] * fi[kk][0];
#pragma unroll
        for (int m = 1; m < D; m++) acc = acc + g[l + D * m] * fi[kk][m];
        if (kk > 0) {
#pragma unroll
          for (int m = 0; m < D; m++) acc = fr_fma(g[l + D * m], fv[kk][m], acc);
        }
        flux(l, kk, pe)[su] = acc;
      }
  }
  __syncthreads();

  // the left normal of the thread's flux point, in flight during the divergence
  const int qe = tid / NF, qf = tid - qe * NF;
  const bool qlive = tid < EPB * NF && qe < nval;
  TC nrm[D];
  if constexpr (IF == 1) {
    if (qlive) {
#pragma unroll
      for (int d = 0; d < D; d++) nrm[d] = (nL + NF * e0 + NFE * d)[(unsigned)tid];
    }
  }

  // --- lines: divergence of the total discontinuous flux (the reference's
  // sum_d opp_2[d] row, axes in order: the running sum is kept in place of
  // the flux along axis 0) and the discontinuous normal flux at both ends
  // (opp_1 rows in column order).  A warp that holds whole elements of one
  // field needs no block barrier between the axes.
  constexpr bool WSYNC = 32 % NLN == 0 && (EPB * NLN) % 32 == 0;
#pragma unroll
  for (int d = 0; d < D; d++) {
    if (line) {
      const int base = M::line(d, j0, j1);
      const size_t oe = (size_t)NF * (e0 + el) + NFE * k;
      TC v[N1], acc[N1];
      TC* run = sF0 + k * NW + el * M::N + base;
      if (d == 0) lds_strided<N1, M::stride(0)>(run, v);
      else if (d == 1) lds_strided<N1, M::stride(1)>(flux(d, k, el) + base, v);
      else lds_strided<N1, M::stride(2)>(flux(d, k, el) + base, v);
      TC vm = TC(0), vp = TC(0);
#pragma unroll
      for (int m = 0; m <= P; m++) {
        vm = vm + v[m] * L.Lm[m];
        vp = vp + v[m] * L.Lp[m];
      }
      ND[oe + end_fpt(d, 0, j0, j1)] = -vm;
      ND[oe + end_fpt(d, 1, j0, j1)] = vp;
      if (d == 1) lds_strided<N1, M::stride(1)>(run, acc);
      if (d == 2) lds_strided<N1, M::stride(2)>(run, acc);
#pragma unroll
      for (int i = 0; i < N1; i++) {
        TC t = d == 0 ? TC(0) : acc[i];
#pragma unroll
        for (int m = 0; m <= P; m++) t = t + v[m] * L.D[i][m];
        acc[i] = t;
      }
      if (d == D - 1) {
        TC* out = DV + (size_t)NU * (e0 + el + E * k) + j0 + (DIM == 3 ? N1 * j1 : 0);
#pragma unroll
        for (int i = 0; i < N1; i++) out[i * (DIM == 3 ? N1 * N1 : N1)] = acc[i];
      } else if (d == 0) sts_strided<N1, M::stride(0)>(run, acc);
      else sts_strided<N1, M::stride(1)>(run, acc);
    }
    if (d < D - 1) {
      if constexpr (WSYNC) __syncwarp();
      else __syncthreads();
    }
  }

  // --- flux points: the own corrected gradient (and SGS flux) extrapolated
  // along the line through the point (opp_6 rows in column order with FMAs), one
  // column at a time into the own viscous flux, projected on the left normal
  // (VF, or BV at a boundary point).
#pragma unroll
  for (int it = 0; it < IF; it++) {
    const int w = tid + it * NT, pe = it ? w / NF : qe, f = it ? w - pe * NF : qf;
    if (w >= EPB * NF || pe >= nval) continue;
    const long long own = f + NF * (e0 + pe);
    int u0, ust, ax, a, b, c;
    bool plus;
    fpt_line<DIM, P>(f, u0, ust, ax, plus);
    upt_abc<DIM, P>(u0, a, b, c);
    const int base = M::slot(a, b, c) + pe * M::N, st = ax == 0 ? 1 : (ax == 1 ? M::S1 : M::S2);
    TC uf[F], n[D], Lc[N1];
#pragma unroll
    for (int m = 0; m <= P; m++) Lc[m] = plus ? L.Lp[m] : L.Lm[m];
#pragma unroll
    for (int kk = 0; kk < F; kk++) uf[kk] = sUf[(kk * EPB + pe) * NF + f];
#pragma unroll
    for (int d = 0; d < D; d++) n[d] = IF == 1 ? nrm[d] : nL[own + NFE * d];
    auto extrap = [&](const TC* s) {
      TC acc = s[0] * Lc[0];
#pragma unroll
      for (int m = 1; m <= P; m++) acc = fr_fma(s[m * st], Lc[m], acc);
      return acc;
    };
    const int btype = BV ? side[own] >> 2 : 0;
    if (btype) {
      BdyPoint<D, TC> q;
#pragma unroll
      for (int kk = 0; kk < F; kk++) {
        q.u[kk] = uf[kk];
#pragma unroll
        for (int d = 0; d < D; d++) q.g[kk][d] = extrap(sG + (kk + F * d) * NW + base);
      }
#pragma unroll
      for (int d = 0; d < D; d++) q.n[d] = n[d];
      TC* out = &BV[(-1 - (long long)mate[own]) * F];
      if constexpr (LES == 0) {
        vis_boundary<D, TC, false>(ph, btype, q, out);
      } else {
        vis_flux_fast<D, TC>(ph, q.u, q.g, q.fv);
#pragma unroll
        for (int kk = 1; kk < F; kk++)
#pragma unroll
          for (int d = 0; d < D; d++) q.fv[kk][d] = q.fv[kk][d] + extrap(sS + ((kk - 1) + (F - 1) * d) * NW + base);
        vis_boundary<D, TC>(ph, btype, q, out);
      }
      continue;
    }
    VisState<D, TC> vs;
    vis_begin<D, TC>(ph, uf, vs);
#pragma unroll
    for (int d = 0; d < D; d++) {
      TC col[F];
#pragma unroll
      for (int kk = 0; kk < F; kk++) col[kk] = extrap(sG + (kk + F * d) * NW + base);
      vis_column<D, TC>(vs, d, col);
    }
    if constexpr (LES == 0) {
      // the projection is accumulated as the flux is formed (no full flux held)
      TC pr[F - 1];
      vis_proj_end<D, TC>(vs, n, pr);
#pragma unroll
      for (int kk = 1; kk < F; kk++) (VF + NF * e0 + NFE * (kk - 1))[(unsigned)w] = pr[kk - 1];
    } else {
      TC fv[F][D];
      vis_flux_end<D, TC>(vs, fv);
#pragma unroll
      for (int kk = 1; kk < F; kk++) {
#pragma unroll
        for (int d = 0; d < D; d++) fv[kk][d] = fv[kk][d] + extrap(sS + ((kk - 1) + (F - 1) * d) * NW + base);
        VF[own + NFE * (kk - 1)] = project<D, TC>(fv, kk, n);
      }
    }
  }
  if (!PERS || (blk + bstride) * EPB >= E) break;
  __syncthreads();   // this block's arrays have been read
  }
}

template <int DIM, int P, int EPB, int NT, typename TC, int LES = 0, int MINB = 1, int VEC = 1, int PERS = 0>
__global__ void __launch_bounds__(NT, MINB)
fr_grad_kernel(const double* __restrict__ U, const TC* __restrict__ UF, const int* __restrict__ mate,
               const unsigned char* __restrict__ side, const TC* __restrict__ JG, const TC* __restrict__ detj,
               const TC* __restrict__ nL, TC* __restrict__ VF, TC* __restrict__ ND, TC* __restrict__ DV,
               long long E, Line<TC> L, PhysT<TC> ph, TC* __restrict__ GRAD, TC* __restrict__ BV)
{
  fr_grad_body<DIM, P, EPB, NT, TC, LES, VEC, PERS>(blockIdx.x, gridDim.x, U, UF, mate, side, JG, detj, nL, VF, ND,
                                                     DV, E, L, ph, GRAD, BV);
}

// Boundary point j of the interface kernel (flat own index bf[j], type
// bt[j]), out of line so that the interior path keeps few registers.
template <int DIM, int VISC, typename TC>
__device__ __noinline__ void face_boundary(PhysT<TC> ph, long long j, const TC* __restrict__ UF,
                                           const TC* __restrict__ nL, const TC* __restrict__ tdA, TC* __restrict__ CF,
                                           long long NFE, const int* __restrict__ bf,
                                           const unsigned char* __restrict__ bt, const TC* __restrict__ BV)
{
  constexpr int F = DIM + 2, D = DIM;
  const long long a = bf[j];
  const int type = bt[j];
  TC ul[F], ug[F], n[D], fn[F];
#pragma unroll
  for (int k = 0; k < F; k++) ul[k] = UF[a + NFE * k];
#pragma unroll
  for (int d = 0; d < D; d++) n[d] = nL[a + NFE * d];
  bc_ghost<D, TC>(ph, type, ul, n, ug);
  TC fl[F][D], fr[F][D];
  inv_flux<D, TC>(ph, ul, fl);
  inv_flux<D, TC>(ph, ug, fr);
  if (type == 16) {
#pragma unroll
    for (int k = 0; k < F; k++) {
      TC s = fl[k][0] * n[0];
#pragma unroll
      for (int l = 1; l < D; l++) s = s + fl[k][l] * n[l];
      fn[k] = s;
    }
  } else {
#pragma unroll
    for (int k = 0; k < F; k++) {
      TC s = fl[k][0] * n[0], q = fr[k][0] * n[0];
#pragma unroll
      for (int l = 1; l < D; l++) { s = s + fl[k][l] * n[l]; q = q + fr[k][l] * n[l]; }
      fn[k] = TC(0.5) * (s + q);
    }
  }
  const TC tl = tdA[a];
#pragma unroll
  for (int k = 0; k < F; k++) {
    TC c = fn[k] * tl;
    if (VISC) c = c + BV[j * F + k] * tl;
    CF[a + NFE * k] = c;
  }
}

// ---------------------------------------------------------------------------
// Common interface fluxes, once per interface flux point (one thread each):
// int_inters::calculate_common_invFlux (Rusanov, src/int_inters.cpp:225-354)
// and, viscous, calculate_common_viscFlux (LDG from the two sides' normal
// projections VF, src/int_inters.cpp:359-470).  Writes norm_tconf_fpts of
// both sides: +f_n tdA_l on the left, -f_n tdA_r on the right.
// face[i] = (left flat index, right flat index) of interface point i;
// fsign[i] != 0 when the LDG penalty sign is negative there.
// Threads past nint take the boundary points: ghost state, inviscid common
// flux of bdy_inters::evaluate_boundaryConditions_invFlux (central flux of the
// two states, convective_flux_boundary, src/inters.cpp:368-387; the own flux
// for slip_wall_dual, right_flux, src/inters.cpp:299-308), plus the viscous part
// BV from the gradient kernel.
// Blocks of exactly 128 threads (one shared staging column per thread); the
// body serves block blk (fr_face_kernel: blockIdx.x; merged batch launches:
// their share of the grid).
template <int DIM, int VISC, typename TC>
__device__ __forceinline__ void
fr_face_body(long long blk, const int2* __restrict__ face, const unsigned char* __restrict__ fsign, long long nint,
             const TC* __restrict__ UF, const TC* __restrict__ VF, const TC* __restrict__ nL,
             const TC* __restrict__ tdA, TC* __restrict__ CF, long long NFE, const PhysT<TC>& ph, long long nbdy,
             const int* __restrict__ bf, const unsigned char* __restrict__ bt, const TC* __restrict__ BV)
{
  constexpr int F = DIM + 2, D = DIM;
  long long i = blk * 128 + threadIdx.x;
  if (i >= nint) {
    if (i - nint < nbdy) face_boundary<DIM, VISC, TC>(ph, i - nint, UF, nL, tdA, CF, NFE, bf, bt, BV);
    return;
  }
  // FP64: the point's inputs reach shared memory through cp.async (one
  // column per thread, field-major: no bank conflicts, no barrier), so they
  // are all in flight at once without holding registers; FP32 reads them
  // directly
  constexpr bool STAGE = sizeof(TC) == 8;
  constexpr int NV = 2 * F + D + 2 + (VISC ? 2 * (F - 1) : 0);
  __shared__ TC sv[STAGE ? NV : 1][STAGE ? 128 : 1];
  const int t = threadIdx.x;
  const int2 lr = face[i];
  const long long a = lr.x, b = lr.y;
  auto in = [&](int j, const TC* src) -> TC { return STAGE ? sv[j][t] : *src; };
  if constexpr (STAGE) {
    int j = 0;
#pragma unroll
    for (int k = 0; k < F; k++) cp_async<sizeof(TC)>(&sv[j++][t], UF + a + NFE * k);
#pragma unroll
    for (int k = 0; k < F; k++) cp_async<sizeof(TC)>(&sv[j++][t], UF + b + NFE * k);
#pragma unroll
    for (int d = 0; d < D; d++) cp_async<sizeof(TC)>(&sv[j++][t], nL + a + NFE * d);
    cp_async<sizeof(TC)>(&sv[j++][t], tdA + a);
    cp_async<sizeof(TC)>(&sv[j++][t], tdA + b);
    if (VISC) {
#pragma unroll
      for (int k = 1; k < F; k++) cp_async<sizeof(TC)>(&sv[j++][t], VF + a + NFE * (k - 1));
#pragma unroll
      for (int k = 1; k < F; k++) cp_async<sizeof(TC)>(&sv[j++][t], VF + b + NFE * (k - 1));
    }
    cp_async_commit();
    cp_async_wait_all();
  }
  TC ul[F], ur[F], n[D];
#pragma unroll
  for (int k = 0; k < F; k++) { ul[k] = in(k, UF + a + NFE * k); ur[k] = in(F + k, UF + b + NFE * k); }
#pragma unroll
  for (int d = 0; d < D; d++) n[d] = in(2 * F + d, nL + a + NFE * d);
  const TC tl = in(2 * F + D, tdA + a), tr = in(2 * F + D + 1, tdA + b);
  TC fn[F];
  rusanov<D, TC>(ph, ul, ur, n, fn);
  TC cl[F], cr[F];
#pragma unroll
  for (int k = 0; k < F; k++) { cl[k] = fn[k] * tl; cr[k] = -fn[k] * tr; }
  if (VISC) {
    TC nn = n[0] * n[0];
#pragma unroll
    for (int d = 1; d < D; d++) nn = fr_fma(n[d], n[d], nn);
    const TC pen = fsign[i] ? -ph.pen_fact : ph.pen_fact;
#pragma unroll
    for (int k = 0; k < F; k++) {
      TC al = k ? in(2 * F + D + 2 + (k - 1), VF + a + NFE * (k - 1)) : TC(0);
      TC ar = k ? in(2 * F + D + 2 + (F - 1) + (k - 1), VF + b + NFE * (k - 1)) : TC(0);
      TC fv = ldg_normal<TC>(al, ar, ul[k], ur[k], pen, ph.tau, nn);
      cl[k] = cl[k] + fv * tl;
      cr[k] = cr[k] + (-fv) * tr;
    }
  }
#pragma unroll
  for (int k = 0; k < F; k++) { CF[a + NFE * k] = cl[k]; CF[b + NFE * k] = cr[k]; }
}

template <int DIM, int VISC, typename TC>
__global__ void __launch_bounds__(128)
fr_face_kernel(const int2* __restrict__ face, const unsigned char* __restrict__ fsign, long long nint,
               const TC* __restrict__ UF, const TC* __restrict__ VF, const TC* __restrict__ nL,
               const TC* __restrict__ tdA, TC* __restrict__ CF, long long NFE, PhysT<TC> ph,
               long long nbdy = 0, const int* __restrict__ bf = nullptr, const unsigned char* __restrict__ bt = nullptr,
               const TC* __restrict__ BV = nullptr)
{
  fr_face_body<DIM, VISC, TC>(blockIdx.x, face, fsign, nint, UF, VF, nL, tdA, CF, NFE, ph, nbdy, bf, bt, BV);
}

// Block partial sums -> norms: one CTA of 256 threads per field; thread t
// sums partials t, t+256, ... in order, then a fixed shared-memory tree.  The
// order depends only on the number of partials, so results are reproducible.
static __global__ void __launch_bounds__(256)
fr_norm_finalize(const double* __restrict__ partial, int nblk, int F, double inv_n, double* __restrict__ out)
{
  __shared__ double s[256];
  const int k = blockIdx.x;
  double acc = 0.0;
  for (int b = threadIdx.x; b < nblk; b += 256) acc += partial[(size_t)b * F + k];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[k] = s[0] * inv_n;
}

}  // namespace frb
