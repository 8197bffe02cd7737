// fr_diag.cu -- integral diagnostics on the device: the quantities of
// eles::CalcIntegralQuantities (src/eles.cpp:6503-6641) -- kinetic energy,
// enstrophy (the reference's "vorticity": rho |w|^2 / 2), pressure
// dilatation, strain colon product and its deviatoric form -- on the
// reference's volume cubature: the state and its corrected gradient are
// interpolated to each cubature point with the dense nodal-basis rows
// opp_volume_cubpts (column order, as the reference's loop), the quantities
// are formed with the reference's expressions, and weight x detJ at the
// cubature point integrates them.  Per-block partial sums, added by
// fr_diag_finalize in a fixed order, so the result does not depend on
// scheduling.
#include <cuda_runtime.h>

namespace frb {

constexpr int kDiagQ = 5;

// Values per point: the state, then with NQ 5 the gradient.
template <int D, int NQ>
struct DiagPlan {
  static constexpr int F = D + 2, C = NQ > 1 ? F * (D + 1) : F;
};
constexpr int kDiagThreads = 128, kDiagWarps = kDiagThreads / 32;
constexpr int kDiagRows = 32, kDiagLdv = kDiagRows + 4;   // cubature points per pass, and their stride
constexpr int kDiagTN = 5;                                // 8-column tiles per warp unit

// smallest leading dimension >= ceil4(nu) that is 4 or 12 mod 16
__host__ __device__ inline int diag_ld(int nu)
{
  int x = (nu + 3) / 4 * 4;
  while (x % 16 != 4 && x % 16 != 12) x++;
  return x;
}
inline size_t diag_smem(int nu, int cols)
{
  return sizeof(double) * (size_t)((cols + 7) / 8 * 8) * (diag_ld(nu) + kDiagLdv);
}

// largest dynamic shared memory of a block: the device's 227 KB less the
// kernel's own norm partials
constexpr int kDiagSmemMax = 226 * 1024;

// elements per block: columns for whole units of tiles, within 100 KB
template <int D, int NQ>
int diag_epb(int nu)
{
  int e = NQ > 1 && D == 3 ? 4 : 8;
  while (e > 1 && diag_smem(nu, e * DiagPlan<D, NQ>::C) > 100 * 1024) e /= 2;
  return e;
}

// NQ 5: all five quantities (G, the corrected gradient (nu, E, F, D), is
// read); NQ 1: the kinetic energy alone (G unused).  Bound: the interpolation,
// nu x C multiply-adds per cubature point (hex P = 3: 34.6 k per element, FP64
// rate).  It is a product of the operator rows with the block's columns
// (element, value), on the FP64 tensor cores (m8n8k4, the columns as they lie
// in global memory): one 8-byte shared load feeds 256 multiply-adds, where a
// thread per cubature point spends a broadcast 16-byte load per two, and was
// bound by those (five quantities of 24^3 hexes of P = 3: 141 us, now 86; reading
// state and gradient from global memory per point took 430).  32 cubature points a
// pass; a thread then forms the quantities of one point.  blockIdx.x walks over
// groups of epb elements, blockIdx.y over the passes.
template <int D, typename TG, int NQ>
__global__ void __launch_bounds__(kDiagThreads, 5)
fr_diag_kernel(const double* __restrict__ U, const TG* __restrict__ G, const double* __restrict__ opp,
               const double* __restrict__ W, const double* __restrict__ detj, long long E, int nu, int nc,
               double gamma, int epb, int ldk, double* __restrict__ partial)
{
  constexpr int F = D + 2, C = DiagPlan<D, NQ>::C;
  extern __shared__ __align__(16) double diag_smem_buf[];
  __shared__ double red[NQ][kDiagWarps];
  const int ncol = epb * C, NTL = (ncol + 7) / 8, KS = (nu + 3) / 4;
  double* sB = diag_smem_buf;               // [column][ldk]
  double* sV = sB + (size_t)NTL * 8 * ldk;  // [column][kDiagLdv]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t4 = lane & 3;
  double acc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) acc[q] = 0.0;
  // padding rows and columns hold zeros, or an earlier element's values
  for (int i = tid; i < NTL * 8 * ldk; i += kDiagThreads) sB[i] = 0.0;
  for (long long e0 = (long long)blockIdx.x * epb; e0 < E; e0 += (long long)gridDim.x * epb) {
    const int nval = (int)(E - e0 < epb ? E - e0 : epb), run = nval * nu;
    __syncthreads();   // the elements before have been read
    for (int r = tid; r < run; r += kDiagThreads) {
      const int el = r / nu;
      double* dst = sB + (size_t)el * C * ldk + (r - el * nu);
      const size_t src = (size_t)nu * e0 + r, st = (size_t)nu * E;
#pragma unroll
      for (int m = 0; m < F; m++) dst[m * ldk] = U[src + st * m];
      if constexpr (NQ > 1) {
#pragma unroll
        for (int m = 0; m < F * D; m++) dst[(F + m) * ldk] = (double)G[src + st * m];
      }
    }
    __syncthreads();
    for (int j0 = kDiagRows * blockIdx.y; j0 < nc; j0 += kDiagRows * gridDim.y) {
      const int rows = nc - j0 < kDiagRows ? nc - j0 : kDiagRows;
      const int MT = (rows + 7) / 8, NB = (NTL + kDiagTN - 1) / kDiagTN;
      for (int u = warp; u < MT * NB; u += kDiagWarps) {
        const int mt = u / NB, nt0 = (u - mt * NB) * kDiagTN, r = j0 + mt * 8 + g8;
        double c[kDiagTN][2];
        const double* bp[kDiagTN];
#pragma unroll
        for (int j = 0; j < kDiagTN; j++) {
          c[j][0] = c[j][1] = 0.0;
          bp[j] = sB + (size_t)((nt0 + j < NTL ? nt0 + j : nt0) * 8 + g8) * ldk + t4;
        }
        for (int k0 = 0; k0 < KS; k0 += 8) {
          double a[8];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int k = (k0 + i) * 4 + t4;
            a[i] = (r < nc && k < nu) ? __ldg(opp + r + (size_t)nc * k) : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 8; i++)
            if (k0 + i < KS)
#pragma unroll
              for (int j = 0; j < kDiagTN; j++)
                asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                    : "+d"(c[j][0]), "+d"(c[j][1])
                    : "d"(a[i]), "d"(bp[j][(k0 + i) * 4]));
        }
#pragma unroll
        for (int j = 0; j < kDiagTN; j++)
          if (nt0 + j < NTL) {
            double* v = sV + (size_t)((nt0 + j) * 8 + 2 * t4) * kDiagLdv + mt * 8 + g8;
            v[0] = c[j][0];
            v[kDiagLdv] = c[j][1];
          }
      }
      __syncthreads();
      for (int i = tid; i < nval * rows; i += kDiagThreads) {
        const int el = i / rows, jj = i - el * rows, j = j0 + jj;
        const long long e = e0 + el;
        const double* v = sV + (size_t)el * C * kDiagLdv + jj;
        double u[F], g[F][D];
#pragma unroll
        for (int m = 0; m < F; m++) {
          u[m] = v[m * kDiagLdv];
          if constexpr (NQ > 1) {
#pragma unroll
            for (int n = 0; n < D; n++) g[m][n] = v[(F + m + F * n) * kDiagLdv];
          }
        }
        const double wj = W[j], dj = detj[j + (size_t)nc * e];
        const double irho = 1. / u[0];
        double tke = 0.0;
#pragma unroll
        for (int n = 1; n < F - 1; n++) tke += 0.5 * u[n] * u[n];
        acc[0] += irho * tke * wj * dj;
        if constexpr (NQ > 1) {
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
      __syncthreads();   // the values have been read
    }
  }
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[q][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double v = 0.0;
    for (int w = 0; w < kDiagWarps; w++) v += red[threadIdx.x][w];
    partial[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * NQ + threadIdx.x] = v;
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
  const int epb = diag_epb<D, NQ>(nu);
  const size_t sm = diag_smem(nu, epb * DiagPlan<D, NQ>::C);
  // the limit belongs to the kernel, not to the call: every call sets the same
  // one, so that it is there on each device and calls of other orders from
  // other threads never lower it
  if (cudaError_t e = cudaFuncSetAttribute(fr_diag_kernel<D, TG, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kDiagSmemMax))
    return e;
  const long long groups = (E + epb - 1) / epb;
  // one block per group of elements over all its passes; a mesh of few groups
  // spreads the passes of a large rule over more blocks (kinetic energy of 27
  // hexes of P = 3 with 729 points: 80 us with 4 blocks of 23 passes, 32 now)
  const int gx = (int)(groups < nblk ? groups : nblk), passes = (nc + kDiagRows - 1) / kDiagRows;
  const int gy = passes < nblk / gx ? passes : nblk / gx;
  fr_diag_kernel<D, TG, NQ><<<dim3(gx, gy), kDiagThreads, sm, st>>>(U, G, opp, W, detj, E, nu, nc, gamma, epb,
                                                                    diag_ld(nu), partial);
  fr_diag_finalize<<<1, 32 * NQ, 0, st>>>(partial, gx * gy, NQ, out);
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
