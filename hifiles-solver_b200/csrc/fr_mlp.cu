// fr_mlp.cu -- training and standalone inference of the learned SGS closure
// (parameter layout and the per-point model in fr_mlp.cuh), and the kernel
// that evaluates the closure's inputs from a solver's state and gradient.
//
// Training step on a batch of N samples (x_n, c*_n, weight s_n; s_n = 1 when
// no weights are given):
//   loss = (1/N) sum_n s_n (c(x_n) - c*_n)^2
// fr_mlp_loss_grad_kernel: persistent CTAs, each over tiles of 128 samples
// (tile = CTA, CTA + grid, ...); the three 64 x 64 products of a sample
// (forward, weight gradient, input gradient) are register-tiled FP32 products
// over shared memory, and a CTA keeps its gradient in registers over all its
// tiles -> one partial gradient per CTA.  fr_mlp_reduce_kernel sums the
// partials in a fixed order; the number of CTAs depends on the batch alone, so
// a gradient is the same bit for bit on every run and every GPU.
// fr_mlp_adam_kernel applies Adam.
#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "fr_b200.h"
#include "fr_launch.hpp"
#include "fr_mlp.cuh"

namespace frb {

extern thread_local std::string g_err;

namespace {

constexpr int kTile = 128;
constexpr int kLd = kTile + 4;   // row stride of the sample-minor arrays: 8 rows at one sample fall in 8 bank groups
// Shared memory of fr_mlp_loss_grad_kernel (floats): W2 transposed [i][j] and
// as it is [j][i], h1 and h2 (then their loss derivatives) [unit][sample], x
// [6][sample], partial outputs per warp [8][sample], d loss / d o [sample].
constexpr int kGradThreads = 256, kGradWarps = kGradThreads / 32;
constexpr int kSmW2T = 0, kSmW2 = kSmW2T + kMlpH * kMlpH, kSmH1 = kSmW2 + kMlpH * kMlpH, kSmH2 = kSmH1 + kMlpH * kLd,
              kSmX = kSmH2 + kMlpH * kLd, kSmO = kSmX + kMlpIn * kLd, kSmDo = kSmO + kGradWarps * kTile,
              kSmEnd = kSmDo + kTile;
constexpr size_t kGradSmem = sizeof(float) * kSmEnd;
// Most CTAs of the loss gradient: two for each of a B200's 148 SMs (104 KB of
// shared memory each).  A constant and not a query, since the number of partial
// sums decides the last bits of a gradient.
constexpr int kGradCtas = 296;

fr_status mlp_fail(fr_status s, const std::string& m)
{
  g_err = m;
  return s;
}

__global__ void __launch_bounds__(256) fr_mlp_forward_kernel(const float* __restrict__ w, const float* __restrict__ X,
                                                             long long n, float* __restrict__ out)
{
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float x[kMlpIn];
#pragma unroll
  for (int k = 0; k < kMlpIn; k++) x[k] = X[i * kMlpIn + k];
  out[i] = mlp_eval(w, x);
}

// acc[r][c] += w[r] v.c for 8 weights (two broadcast quads) and 4 samples
__device__ __forceinline__ void mlp_fma_8x4(float (&acc)[8][4], const float* w8, const float* v4)
{
  const float4 wa = *reinterpret_cast<const float4*>(w8), wb = *reinterpret_cast<const float4*>(w8 + 4);
  const float4 v = *reinterpret_cast<const float4*>(v4);
  const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
  for (int r = 0; r < 8; r++) {
    acc[r][0] = fmaf(w[r], v.x, acc[r][0]);
    acc[r][1] = fmaf(w[r], v.y, acc[r][1]);
    acc[r][2] = fmaf(w[r], v.z, acc[r][2]);
    acc[r][3] = fmaf(w[r], v.w, acc[r][3]);
  }
}

// Bound: FP32 FMA issue, 13.6 k multiply-adds a sample (24 us of FP32 peak for
// 65536 samples).  A product over [unit][sample] arrays gives each warp 8
// units and all 128 samples, 4 per lane: 8 x 4 register tile, so 3 16-byte
// shared loads (2 of them broadcasts) feed 32 FMAs; the weight gradient takes
// a 4 x 4 tile per thread with K = the samples, 8 loads per 64 FMAs.  Both
// leave the FMA pipe ahead of the shared-memory pipe; one output per thread
// with two loads per FMA was bound by the latter, and left 512 partials to add
// (a step with its reduction and Adam, 65536 samples: 240 us, now 76).
__global__ void __launch_bounds__(kGradThreads, 2) fr_mlp_loss_grad_kernel(const float* __restrict__ w,
                                                                           const float* __restrict__ X,
                                                                           const float* __restrict__ Y,
                                                                           const float* __restrict__ SW, long long n,
                                                                           float inv_n, float* __restrict__ partial)
{
  extern __shared__ __align__(16) float mlp_smem[];
  float* sW2T = mlp_smem + kSmW2T;
  float* sW2 = mlp_smem + kSmW2;
  float* sH1 = mlp_smem + kSmH1;   // h1, then d loss / d a1
  float* sH2 = mlp_smem + kSmH2;   // d loss / d a2
  float* sX = mlp_smem + kSmX;
  float* sO = mlp_smem + kSmO;
  float* sDo = mlp_smem + kSmDo;
  const int t = threadIdx.x, lane = t & 31, wp = t >> 5, s4 = 4 * lane, u0 = 8 * wp;
  for (int e = t; e < kMlpH * kMlpH; e += kGradThreads) {
    const float v = w[kMlpW2 + e];
    sW2[e] = v;
    sW2T[(e % kMlpH) * kMlpH + e / kMlpH] = v;
  }
  // weight-gradient tile: rows j0 + 8 q of d a2, rows i0 + 4 p of h1
  const int j0 = (lane & 7) + 32 * (wp & 1), i0 = (lane >> 3) + 16 * (wp >> 1);
  // first-layer gradient: unit t / 4, quarter t % 4 of the samples
  const int iu = t >> 2, qu = t & 3;
  float gW2[4][4], gW1[kMlpIn], gB1 = 0.f, gW3[8], gB2[8], gB3 = 0.f, gL = 0.f;
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int p = 0; p < 4; p++) gW2[q][p] = 0.f;
#pragma unroll
  for (int k = 0; k < kMlpIn; k++) gW1[k] = 0.f;
#pragma unroll
  for (int r = 0; r < 8; r++) gW3[r] = gB2[r] = 0.f;

  const long long ntile = (n + kTile - 1) / kTile;
  for (long long tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const long long b0 = tile * kTile;
    const int live = (int)(n - b0 < kTile ? n - b0 : kTile);
    __syncthreads();   // the tile before has been read
    for (int e = t; e < kMlpIn * kTile; e += kGradThreads) {
      const int sm = e / kMlpIn, k = e - sm * kMlpIn;
      sX[k * kLd + sm] = sm < live ? (X[b0 * kMlpIn + e] - w[kMlpXm + k]) * w[kMlpXs + k] : 0.f;
    }
    __syncthreads();
    // ---- layer 1: units u0 .. u0 + 7, samples s4 .. s4 + 3
    {
      float4 x[kMlpIn];
#pragma unroll
      for (int k = 0; k < kMlpIn; k++) x[k] = *reinterpret_cast<const float4*>(sX + k * kLd + s4);
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const float b = __ldg(w + kMlpB1 + u0 + r);
        float4 a = make_float4(b, b, b, b);
#pragma unroll
        for (int k = 0; k < kMlpIn; k++) {
          const float c = __ldg(w + kMlpW1 + (u0 + r) * kMlpIn + k);
          a.x = fmaf(c, x[k].x, a.x);
          a.y = fmaf(c, x[k].y, a.y);
          a.z = fmaf(c, x[k].z, a.z);
          a.w = fmaf(c, x[k].w, a.w);
        }
        *reinterpret_cast<float4*>(sH1 + (u0 + r) * kLd + s4) =
            make_float4(tanhf(a.x), tanhf(a.y), tanhf(a.z), tanhf(a.w));
      }
    }
    __syncthreads();
    // ---- layer 2 and this warp's share of the output
    float h2[8][4];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) h2[r][c] = __ldg(w + kMlpB2 + u0 + r);
#pragma unroll 4
    for (int i = 0; i < kMlpH; i++) mlp_fma_8x4(h2, sW2T + i * kMlpH + u0, sH1 + i * kLd + s4);
    {
      float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const float w3 = __ldg(w + kMlpW3 + u0 + r);
#pragma unroll
        for (int c = 0; c < 4; c++) {
          h2[r][c] = tanhf(h2[r][c]);
          o[c] = fmaf(w3, h2[r][c], o[c]);
        }
      }
      *reinterpret_cast<float4*>(sO + wp * kTile + s4) = make_float4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
    if (t < kTile) {
      float o = w[kMlpB3];
#pragma unroll
      for (int q = 0; q < kGradWarps; q++) o += sO[q * kTile + t];
      const bool lv = t < live;
      const float r = lv ? mlp_softplus(o) - Y[b0 + t] : 0.f;
      const float sw = (lv && SW) ? SW[b0 + t] : 1.f;
      const float sig = 1.f / (1.f + expf(-o));
      const float d = 2.f * sw * r * sig * inv_n;   // d loss / d o
      sDo[t] = d;
      gB3 += d;
      gL = fmaf(sw * r, r, gL);
    }
    __syncthreads();
    // ---- output layer's gradient and d loss / d a2 = do w3_j (1 - h2_j^2)
    {
      const float4 d4 = *reinterpret_cast<const float4*>(sDo + s4);
      const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const float w3 = __ldg(w + kMlpW3 + u0 + r);
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const float h = h2[r][c];
          gW3[r] = fmaf(d[c], h, gW3[r]);
          h2[r][c] = d[c] * w3 * (1.f - h * h);
          gB2[r] += h2[r][c];
        }
        *reinterpret_cast<float4*>(sH2 + (u0 + r) * kLd + s4) = make_float4(h2[r][0], h2[r][1], h2[r][2], h2[r][3]);
      }
    }
    __syncthreads();
    // ---- dW2[j][i] += sum_s da2_j h1_i
#pragma unroll 2
    for (int s = 0; s < kTile; s += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; q++) a[q] = *reinterpret_cast<const float4*>(sH2 + (j0 + 8 * q) * kLd + s);
#pragma unroll
      for (int p = 0; p < 4; p++) b[p] = *reinterpret_cast<const float4*>(sH1 + (i0 + 4 * p) * kLd + s);
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int p = 0; p < 4; p++)
          gW2[q][p] = fmaf(a[q].w, b[p].w, fmaf(a[q].z, b[p].z, fmaf(a[q].y, b[p].y, fmaf(a[q].x, b[p].x, gW2[q][p]))));
    }
    // ---- d loss / d a1_i = (sum_j W2[j][i] da2_j) (1 - h1_i^2), in place
    float da[8][4];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) da[r][c] = 0.f;
#pragma unroll 4
    for (int j = 0; j < kMlpH; j++) mlp_fma_8x4(da, sW2 + j * kMlpH + u0, sH2 + j * kLd + s4);
    __syncthreads();   // every thread has read h1 for dW2
#pragma unroll
    for (int r = 0; r < 8; r++) {
      float4* q = reinterpret_cast<float4*>(sH1 + (u0 + r) * kLd + s4);
      const float4 h = *q;
      *q = make_float4(da[r][0] * (1.f - h.x * h.x), da[r][1] * (1.f - h.y * h.y), da[r][2] * (1.f - h.z * h.z),
                       da[r][3] * (1.f - h.w * h.w));
    }
    __syncthreads();
    // ---- dW1[i][k] += sum_s da1_i x_k, db1_i += sum_s da1_i over a quarter of the samples
#pragma unroll 2
    for (int s = 4 * qu; s < kTile; s += 16) {
      const float4 a = *reinterpret_cast<const float4*>(sH1 + iu * kLd + s);
      gB1 += (a.x + a.y) + (a.z + a.w);
#pragma unroll
      for (int k = 0; k < kMlpIn; k++) {
        const float4 x = *reinterpret_cast<const float4*>(sX + k * kLd + s);
        gW1[k] = fmaf(a.w, x.w, fmaf(a.z, x.z, fmaf(a.y, x.y, fmaf(a.x, x.x, gW1[k]))));
      }
    }
  }
  // ---- this CTA's partial gradient and loss
  float* P = partial + (size_t)blockIdx.x * (kMlpTrain + 1);
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int p = 0; p < 4; p++) P[kMlpW2 + (j0 + 8 * q) * kMlpH + i0 + 4 * p] = gW2[q][p];
#pragma unroll
  for (int k = 0; k < kMlpIn; k++) {
    gW1[k] += __shfl_xor_sync(0xffffffffu, gW1[k], 1);
    gW1[k] += __shfl_xor_sync(0xffffffffu, gW1[k], 2);
    if (qu == 0) P[kMlpW1 + iu * kMlpIn + k] = gW1[k];
  }
  gB1 += __shfl_xor_sync(0xffffffffu, gB1, 1);
  gB1 += __shfl_xor_sync(0xffffffffu, gB1, 2);
  if (qu == 0) P[kMlpB1 + iu] = gB1;
#pragma unroll
  for (int r = 0; r < 8; r++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      gW3[r] += __shfl_xor_sync(0xffffffffu, gW3[r], o);
      gB2[r] += __shfl_xor_sync(0xffffffffu, gB2[r], o);
    }
    if (lane == 0) {
      P[kMlpW3 + u0 + r] = gW3[r];
      P[kMlpB2 + u0 + r] = gB2[r];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gB3 += __shfl_xor_sync(0xffffffffu, gB3, o);
    gL += __shfl_xor_sync(0xffffffffu, gL, o);
  }
  __syncthreads();
  if (lane == 0) {   // zero in the warps without samples of their own
    sO[wp] = gB3;
    sO[kGradWarps + wp] = gL;
  }
  __syncthreads();
  if (t == 0) {
    float b3 = 0.f, l = 0.f;
    for (int q = 0; q < kGradWarps; q++) {
      b3 += sO[q];
      l += sO[kGradWarps + q];
    }
    P[kMlpB3] = b3;
    P[kMlpTrain] = l;
  }
}

// grad[p] = sum over CTAs of partial[b][p]; loss = sum of the per-CTA squared
// residuals / n.  A block takes 32 parameters: 8 rows of threads over the
// partials (coalesced 128-byte reads), then the rows in order.
constexpr int kRedRows = 8;
__global__ void __launch_bounds__(32 * kRedRows) fr_mlp_reduce_kernel(const float* __restrict__ partial, int nblk,
                                                                      float inv_n, float* __restrict__ grad,
                                                                      float* __restrict__ loss)
{
  __shared__ float s[kRedRows][32];
  const int c = threadIdx.x & 31, r = threadIdx.x >> 5, p = blockIdx.x * 32 + c;
  float acc = 0.f;
  if (p <= kMlpTrain) {
#pragma unroll 4
    for (int b = r; b < nblk; b += kRedRows) acc += partial[(size_t)b * (kMlpTrain + 1) + p];
  }
  s[r][c] = acc;
  __syncthreads();
  if (r > 0 || p > kMlpTrain) return;
  acc = 0.f;
#pragma unroll
  for (int q = 0; q < kRedRows; q++) acc += s[q][c];
  if (p < kMlpTrain) grad[p] = acc;
  else if (loss) *loss = acc * inv_n;
}

__global__ void fr_mlp_adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                                   float* __restrict__ v, float lr, float b1, float b2, float eps, float c1,
                                   float c2)
{
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kMlpTrain) return;
  const float gp = g[p];
  const float mp = b1 * m[p] + (1.f - b1) * gp;
  const float vp = b2 * v[p] + (1.f - b2) * gp * gp;
  m[p] = mp;
  v[p] = vp;
  w[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

template <int D, typename TC>
__global__ void fr_sgs_inputs_kernel(const double* __restrict__ U, const TC* __restrict__ G,
                                     const double* __restrict__ detj, long long npts, int nu, long long E, double n1,
                                     double filter_ratio, float* __restrict__ X)
{
  constexpr int F = D + 2;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npts) return;
  double q[F], g[F][D];
#pragma unroll
  for (int k = 0; k < F; k++) {
    q[k] = U[i + npts * k];
#pragma unroll
    for (int d = 0; d < D; d++) g[k][d] = (double)G[i + npts * (k + (long long)F * d)];
  }
  float x[kMlpIn];
  double delta, S[D][D], smag, de[D];
  sgs_learned_inputs<D, double>(q, g, detj[i], n1, filter_ratio, x, delta, S, smag, de);
#pragma unroll
  for (int k = 0; k < kMlpIn; k++) X[i * kMlpIn + k] = x[k];
  (void)nu; (void)E;
}

}  // namespace

// Host launcher used by fr_solver_sgs_features (fr_solver.cu).
cudaError_t launch_sgs_inputs(int dims, int tc_size, const double* U, const void* G, const double* detj, long long npts,
                              int nu, long long E, int order, double filter_ratio, float* X, cudaStream_t st)
{
  unsigned g = (unsigned)((npts + 255) / 256);
  if (dims == 2 && tc_size == 8)
    fr_sgs_inputs_kernel<2, double><<<g, 256, 0, st>>>(U, (const double*)G, detj, npts, nu, E, order + 1.0,
                                                       filter_ratio, X);
  else if (dims == 2)
    fr_sgs_inputs_kernel<2, float><<<g, 256, 0, st>>>(U, (const float*)G, detj, npts, nu, E, order + 1.0,
                                                      filter_ratio, X);
  else if (tc_size == 8)
    fr_sgs_inputs_kernel<3, double><<<g, 256, 0, st>>>(U, (const double*)G, detj, npts, nu, E, order + 1.0,
                                                       filter_ratio, X);
  else
    fr_sgs_inputs_kernel<3, float><<<g, 256, 0, st>>>(U, (const float*)G, detj, npts, nu, E, order + 1.0,
                                                      filter_ratio, X);
  return cudaGetLastError();
}

// Parameters of a closure that is switched off: zero weights, unit input
// scaling and b3 = -20, so c = softplus(-20) ~ 2e-9.
void mlp_default_params(float* w)
{
  for (int p = 0; p < kMlpN; p++) w[p] = 0.f;
  w[kMlpB3] = -20.f;
  for (int k = 0; k < kMlpIn; k++) w[kMlpXs + k] = 1.f;
}

}  // namespace frb

using namespace frb;

int fr_mlp_n_params(void) { return kMlpN; }
int fr_mlp_n_trained(void) { return kMlpTrain; }

long long fr_mlp_scratch_floats(long long n) { return ((n + kTile - 1) / kTile) * (long long)(kMlpTrain + 1); }

fr_status fr_mlp_forward(const float* w, const float* x, long long n, float* out, void* stream)
{
  if (!w || (n > 0 && (!x || !out)) || n < 0) return mlp_fail(FR_ERR_ARG, "bad argument");
  if (n == 0) return FR_OK;
  fr_mlp_forward_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(w, x, n, out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FR_OK : mlp_fail(FR_ERR_CUDA, cudaGetErrorString(e));
}

fr_status fr_mlp_loss_grad(const float* w, const float* x, const float* y, const float* sw, long long n, float* grad,
                           float* loss, float* scratch, long long scratch_floats, void* stream)
{
  if (!w || !x || !y || !grad || !scratch || n <= 0) return mlp_fail(FR_ERR_ARG, "bad argument");
  if (scratch_floats < fr_mlp_scratch_floats(n))
    return mlp_fail(FR_ERR_ARG, "scratch smaller than fr_mlp_scratch_floats(n)");
  const long long nblk = (n + kTile - 1) / kTile;
  if (nblk > 0x7fffffffLL) return mlp_fail(FR_ERR_ARG, "batch too large");
  cudaStream_t st = (cudaStream_t)stream;
  const float inv_n = (float)(1.0 / (double)n);
  static SmemLimit limit;
  limit((const void*)fr_mlp_loss_grad_kernel, kGradSmem);
  const int grid = (int)(nblk < kGradCtas ? nblk : kGradCtas);
  fr_mlp_loss_grad_kernel<<<grid, kGradThreads, kGradSmem, st>>>(w, x, y, sw, n, inv_n, scratch);
  fr_mlp_reduce_kernel<<<(kMlpTrain + 1 + 31) / 32, 32 * kRedRows, 0, st>>>(scratch, grid, inv_n, grad, loss);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FR_OK : mlp_fail(FR_ERR_CUDA, cudaGetErrorString(e));
}

fr_status fr_mlp_adam(float* w, const float* grad, float* m, float* v, int step, float lr, void* stream)
{
  if (!w || !grad || !m || !v || step < 1 || !(lr > 0.f)) return mlp_fail(FR_ERR_ARG, "bad argument");
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = (float)(1.0 - std::pow(0.9, step)), c2 = (float)(1.0 - std::pow(0.999, step));
  fr_mlp_adam_kernel<<<(kMlpTrain + 255) / 256, 256, 0, (cudaStream_t)stream>>>(w, grad, m, v, lr, b1, b2, eps, c1,
                                                                                 c2);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FR_OK : mlp_fail(FR_ERR_CUDA, cudaGetErrorString(e));
}
