// fr_diag.cu -- integral diagnostics on the device: the quantities of
// eles::CalcIntegralQuantities (src/eles.cpp:6503-6641) -- kinetic energy,
// enstrophy (the reference's "vorticity": rho |w|^2 / 2), pressure
// dilatation, strain colon product and its deviatoric form -- on the
// reference's volume cubature: the state and its corrected gradient are
// interpolated to each cubature point with the dense nodal-basis rows
// opp_volume_cubpts (column order, as the reference's loop), the quantities
// are formed with the reference's expressions, and weight x detJ at the
// cubature point integrates them.  One thread per (element, cubature point);
// per-block partial sums, added by fr_diag_finalize in a fixed order, so the
// result does not depend on scheduling.
#include <cuda_runtime.h>

namespace frb {

constexpr int kDiagQ = 5;

// Shared-memory order of an element's data: per solution point its C values
// (state, then with NQ 5 the gradient), padded to an even stride so that a
// thread reads two per load.
template <int D, int NQ>
struct DiagPlan {
  static constexpr int F = D + 2, C = NQ > 1 ? F * (D + 1) : F, LD = (C + 1) / 2 * 2 + (NQ > 1 ? 2 : 0);
};
constexpr int kDiagThreads = 128;
constexpr size_t kDiagSmemCap = 90 * 1024;   // two or more blocks per SM

// elements per block: one thread per cubature point as far as shared memory allows
template <int D, int NQ>
int diag_epb(int nu, int nc)
{
  const size_t per = sizeof(double) * (size_t)nu * DiagPlan<D, NQ>::LD;
  const int by_points = nc < kDiagThreads ? kDiagThreads / nc : 1;
  const int by_smem = (int)(kDiagSmemCap / per);
  const int e = by_points < by_smem ? by_points : by_smem;
  return e < 1 ? 1 : e;
}

// NQ 5: all five quantities (G, the corrected gradient (nu, E, F, D), is
// read); NQ 1: the kinetic energy alone (G unused).  Bound: the interpolation,
// nu x C multiply-adds per cubature point (hex P = 3: 34.6 k per element, FP64
// pipe).  A block stages its elements' state and gradient in shared memory
// once (coalesced), and a thread carries all C values of its cubature point
// through one pass over the solution points: per point one operator entry
// from the L1 cache and C / 2 16-byte shared loads (broadcasts within an
// element) feed C FMAs.  Reading state and gradient per cubature point from
// global memory took 430 us (five quantities, 24^3 hexes of P = 3) where this
// takes 44.
template <int D, typename TG, int NQ>
__global__ void __launch_bounds__(kDiagThreads)
fr_diag_kernel(const double* __restrict__ U, const TG* __restrict__ G, const double* __restrict__ opp,
               const double* __restrict__ W, const double* __restrict__ detj, long long E, int nu, int nc,
               double gamma, int epb, double* __restrict__ partial)
{
  using Q = DiagPlan<D, NQ>;
  constexpr int F = D + 2, C = Q::C, LD = Q::LD;
  extern __shared__ __align__(16) double diag_smem[];
  __shared__ double red[NQ][kDiagThreads / 32];
  double acc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) acc[q] = 0.0;
  for (long long e0 = (long long)blockIdx.x * epb; e0 < E; e0 += (long long)gridDim.x * epb) {
    const int nval = (int)(E - e0 < epb ? E - e0 : epb), run = nval * nu;
    __syncthreads();   // the elements before have been read
    for (int r = threadIdx.x; r < run; r += kDiagThreads) {
      double* dst = diag_smem + (size_t)r * LD;
      const size_t src = (size_t)nu * e0 + r, st = (size_t)nu * E;
#pragma unroll
      for (int m = 0; m < F; m++) dst[m] = U[src + st * m];
      if constexpr (NQ > 1) {
#pragma unroll
        for (int m = 0; m < F * D; m++) dst[F + m] = (double)G[src + st * m];
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nval * nc; i += kDiagThreads) {
    const int el = i / nc, j = i - el * nc;
    const long long e = e0 + el;
    double v[(C + 1) / 2 * 2];
#pragma unroll
    for (int m = 0; m < (C + 1) / 2 * 2; m++) v[m] = 0.0;
    const double* row = diag_smem + (size_t)el * nu * LD;
#pragma unroll 2
    for (int k = 0; k < nu; k++) {
      const double o = __ldg(opp + j + (size_t)nc * k);
#pragma unroll
      for (int m = 0; m < C; m += 2) {
        const double2 x = *reinterpret_cast<const double2*>(row + k * LD + m);
        v[m] = fma(o, x.x, v[m]);
        if (m + 1 < C) v[m + 1] = fma(o, x.y, v[m + 1]);
      }
    }
    double u[F], g[F][D];
#pragma unroll
    for (int m = 0; m < F; m++) {
      u[m] = v[m];
      if constexpr (NQ > 1) {
#pragma unroll
        for (int n = 0; n < D; n++) g[m][n] = v[F + m + F * n];
      }
    }
    const double wj = W[j], dj = detj[j + (size_t)nc * e];
    const double irho = 1. / u[0];
    double tke = 0.0;
#pragma unroll
    for (int n = 1; n < F - 1; n++) tke += 0.5 * u[n] * u[n];
    acc[0] += irho * tke * wj * dj;
    if (NQ > 1) {
      const double dudx = irho * (g[1][0] - u[1] * irho * g[0][0]);
      const double dudy = irho * (g[1][1] - u[1] * irho * g[0][1]);
      const double dvdx = irho * (g[2][0] - u[2] * irho * g[0][0]);
      const double dvdy = irho * (g[2][1] - u[2] * irho * g[0][1]);
      double dudz = 0, dvdz = 0, dwdx = 0, dwdy = 0, dwdz = 0;
      if (D == 3) {
        dudz = irho * (g[1][D - 1] - u[1] * irho * g[0][D - 1]);
        dvdz = irho * (g[2][D - 1] - u[2] * irho * g[0][D - 1]);
        dwdx = irho * (g[D][0] - u[D] * irho * g[0][0]);
        dwdy = irho * (g[D][1] - u[D] * irho * g[0][1]);
        dwdz = irho * (g[D][D - 1] - u[D] * irho * g[0][D - 1]);
      }
      // vorticity: rho |w|^2 / 2
      const double wz = dvdx - dudy;
      double vort = wz * wz;
      if (D == 3) {
        const double wx = dwdy - dvdz, wy = dudz - dwdx;
        vort += wx * wx + wy * wy;
      }
      vort *= 0.5 / irho;
      // pressure dilatation
      const double pressure = (gamma - 1.0) * (u[F - 1] - irho * tke);
      const double pd = D == 2 ? pressure * (dudx + dvdy) : pressure * (dudx + dvdy + dwdz);
      // strain-rate colon products
      double S[3][3];
      S[0][0] = dudx;
      S[0][1] = (dudy + dvdx) / 2.0;
      S[1][0] = S[0][1];
      S[1][1] = dvdy;
      double diag = (S[0][0] + S[1][1]) / 3.0;
      if (D == 3) {
        S[0][2] = (dudz + dwdx) / 2.0;
        S[1][2] = (dvdz + dwdy) / 2.0;
        S[2][0] = S[0][2];
        S[2][1] = S[1][2];
        S[2][2] = dwdz;
        diag += S[2][2] / 3.0;
      }
      double sc = 0.0, dsc = 0.0;
#pragma unroll
      for (int a = 0; a < D; a++)
#pragma unroll
        for (int b = 0; b < D; b++) sc += S[a][b] * S[a][b];
#pragma unroll
      for (int a = 0; a < D; a++) S[a][a] -= diag;
#pragma unroll
      for (int a = 0; a < D; a++)
#pragma unroll
        for (int b = 0; b < D; b++) dsc += S[a][b] * S[a][b];
      acc[1] += vort * wj * dj;
      acc[2 % NQ] += pd * wj * dj;
      acc[3 % NQ] += sc * wj * dj;
      acc[4 % NQ] += dsc * wj * dj;
    }
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[q][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double v = 0.0;
    for (int w = 0; w < kDiagThreads / 32; w++) v += red[threadIdx.x][w];
    partial[(size_t)blockIdx.x * NQ + threadIdx.x] = v;
  }
}

// block partials -> quantities: one warp per quantity, strided sums and a
// fixed tree
__global__ void fr_diag_finalize(const double* __restrict__ partial, int nblk, int nq, double* __restrict__ out)
{
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = 0.0;
#pragma unroll 4
  for (int b = lane; b < nblk; b += 32) v += partial[(size_t)b * nq + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) out[q] = v;
}

namespace {

template <int D, typename TG, int NQ>
cudaError_t diag_launch(const double* U, const TG* G, const double* opp, const double* W, const double* detj,
                        long long E, int nu, int nc, double gamma, double* partial, int nblk, double* out,
                        cudaStream_t st)
{
  const int epb = diag_epb<D, NQ>(nu, nc);
  const size_t sm = sizeof(double) * (size_t)epb * nu * DiagPlan<D, NQ>::LD;
  if (cudaError_t e = cudaFuncSetAttribute(fr_diag_kernel<D, TG, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sm))
    return e;
  const long long groups = (E + epb - 1) / epb;
  const int grid = (int)(groups < nblk ? groups : nblk);
  fr_diag_kernel<D, TG, NQ><<<grid, kDiagThreads, sm, st>>>(U, G, opp, W, detj, E, nu, nc, gamma, epb, partial);
  fr_diag_finalize<<<1, 32 * NQ, 0, st>>>(partial, grid, NQ, out);
  return cudaGetLastError();
}

}  // namespace

// G null: the kinetic energy alone (out[0]); otherwise all five quantities.
// nblk: the most partials that `partial` holds (5 values each).
cudaError_t launch_diagnostics(int dims, int tc_size, const double* U, const void* G, const double* opp,
                               const double* W, const double* detj, long long E, int nu, int nc, double gamma,
                               double* partial, int nblk, double* out, cudaStream_t st)
{
#define FR_DIAG(D_, T_, NQ_) \
  return diag_launch<D_, T_, NQ_>(U, (const T_*)G, opp, W, detj, E, nu, nc, gamma, partial, nblk, out, st)
  if (!G) {
    if (dims == 2) FR_DIAG(2, double, 1);
    FR_DIAG(3, double, 1);
  }
  if (dims == 2 && tc_size == 8) FR_DIAG(2, double, kDiagQ);
  if (dims == 2) FR_DIAG(2, float, kDiagQ);
  if (tc_size == 8) FR_DIAG(3, double, kDiagQ);
  FR_DIAG(3, float, kDiagQ);
#undef FR_DIAG
}

}  // namespace frb
