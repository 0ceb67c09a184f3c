// Learned scattering surrogate: training data, training, packing, evaluation.
//
// * Training data: FP64 Gauss-Mehler (Gauss-Chebyshev) quadrature of the classical
//   scattering integral of the universal (ZBL) potential,
//       theta = pi - 2 beta Int_0^1 du / g(u),   g(u)^2 = 1 - Phi(r0/u) u / (r0 eps) - beta^2 u^2,
//   beta = b / r0, r0 the distance of closest approach (safeguarded Newton to 1e-14),
//   and of Biersack's time integral
//       tau = sqrt(r0^2 - b^2) - r0 Int_0^1 [1/g(u) - 1/sqrt(1 - beta^2 u^2)] du / u^2,
//   both with the weight 1/sqrt(1 - u^2) absorbed: the integrands are evaluated as
//   F(u) = sqrt(1 - u^2) / g(u) at the positive Chebyshev nodes u_j = cos((2j-1) pi / 2N).
//   Samples are log-uniform in eps over [1e-4, 1e4] and area-weighted in b over
//   [0, 12] (b = 12 sqrt(U)), drawn from Philox.  The sin^2(theta/2) target is the
//   quadrature's or, on request, the FP64 magic formula's at the same samples
//   (scatter64: the reference's Newton solve and magic formula, trim.C:180-271).
// * Training: the project's own FP32 kernels, two a step: forward and backward pass
//   (the blocks' weight gradients added in block order, so that a run repeats bit for
//   bit) and Adam.  The last epochs are quantisation-aware:
//   the two hidden 64x64 layers see BF16-rounded weights and inputs in the forward
//   pass, as in inference.
// * Inference: mtg_surrogate.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "mytrim_gpu.h"
#include "mtg_collide64.cuh"
#include "mtg_common.cuh"
#include "mtg_kernels.h"
#include "mtg_scatter32.cuh"
#include "mtg_surrogate.cuh"

namespace mtg
{

constexpr int QN = 256; // Gauss-Chebyshev nodes (QN / 2 evaluations per integral)
// per node u: 1 / u, u, u^2, sqrt(1 - u^2) and sqrt(1 - u^2) / u^2
struct QuadNode
{
  double inv_u, u, u2, s, s_u2;
};
__constant__ QuadNode c_nodes[QN / 2];

// universal screening function (trim.C:196-203)
__host__ __device__ __forceinline__ double
screening(double r)
{
  return 0.18175 * exp64(-3.1998 * r) + 0.50986 * exp64(-0.94229 * r) + 0.28022 * exp64(-0.4029 * r) +
         0.028171 * exp64(-0.20162 * r);
}

// phi(r) as a polynomial of degree 7 on each 128th of an octave from 2^-6 to 2^8: 128
// nodes a sample, on a unit that runs FP64 at 2 lanes per SM and clock, where the four
// exponentials take 63 operations and this 9.  It is good to 1.5e-15 up
// to r = 128 and to 4e-15 above, as the exponentials of rounded products are.  Below 2^-6
// the exponentials stand, from 2^8 on the last one of them (the others are below 1e-20 of
// it).  131,072 targets of the training set 6.0 -> 1.7 ms.
constexpr int PHI_OCT = 14, PHI_LO = -6, PHI_BITS = 7, PHI_N = 8;
static __device__ double g_phi[(PHI_OCT << PHI_BITS) * PHI_N];

// phi(r) outside the table
__device__ __forceinline__ double
phi_outside(double r)
{
  return r < 1.0 ? screening(r) : 0.028171 * exp64(-0.20162 * r);
}

// t in [-1, 1) and the first coefficient of r's piece; NULL outside the table
__device__ __forceinline__ const double *
phi_piece(double r, double & t)
{
  const long long bits = __double_as_longlong(r);
  const int k = int(bits >> (52 - PHI_BITS)) - ((1023 + PHI_LO) << PHI_BITS);
  if (k < 0 || k >= PHI_OCT << PHI_BITS)
    return nullptr;
  const long long frac = (bits << PHI_BITS) & 0x000fffffffffffffll;
  t = fma(2.0, __longlong_as_double(0x3ff0000000000000ll | frac), -3.0);
  return g_phi + k * PHI_N;
}

// far: whether phi counts beyond the table
__device__ __forceinline__ double
phi_table(double r, bool far)
{
  double t;
  const double * c = phi_piece(r, t);
  if (!c)
    return far || r < 1.0 ? phi_outside(r) : 0.0;
  double v = c[PHI_N - 1];
#pragma unroll
  for (int i = PHI_N - 2; i >= 0; --i)
    v = fma(v, t, c[i]);
  return v;
}

// phi and its derivative, the latter for Newton steps only
__device__ __forceinline__ void
phi_slope(double r, double & phi, double & dphi)
{
  double t;
  const double * c = phi_piece(r, t);
  if (!c)
  {
    phi = phi_outside(r);
    dphi = r < 1.0 ? -1.0 : -0.20162 * phi; // below 2^-6 within a factor of 1.3, for Newton steps
    return;
  }
  double v = c[PHI_N - 1], d = 0.0;
#pragma unroll
  for (int i = PHI_N - 2; i >= 0; --i)
  {
    d = fma(d, t, v);
    v = fma(v, t, c[i]);
  }
  phi = v;
  // dt / dr = 2 / h, h the width of a piece of r's octave
  const int e = int((__double_as_longlong(r) >> 52) & 0x7ff) - 1023;
  dphi = d * __longlong_as_double((long long)(1023 + 1 + PHI_BITS - e) << 52);
}

// distance of closest approach: root of f(r) = 1 - Phi(r)/(r eps) - b^2/r^2
__device__ double
closest_approach(double eps, double b)
{
  const double ie = 1.0 / eps;
  double hi = 0.5 * (ie + sqrt(ie * ie + 4.0 * b * b)) * (1.0 + 1e-12) + 1e-300;
  double lo = b > 0.0 ? b : hi * 1e-9;
  double r = 0.5 * (lo + hi);
  for (int it = 0; it < 200; ++it)
  {
    double phi, dphi;
    phi_slope(r, phi, dphi);
    const double ir = 1.0 / r;
    const double p = phi * ie * ir, q = b * b * ir * ir;
    const double f = 1.0 - p - q;
    if (f > 0.0)
      hi = r;
    else
      lo = r;
    const double fp = (p + 2.0 * q) * ir - dphi * ie * ir;
    double rn = r - f / fp;
    if (!(rn > lo && rn < hi))
      rn = 0.5 * (lo + hi);
    if (fabs(rn - r) <= 1e-14 * r)
    {
      r = rn;
      break;
    }
    r = rn;
  }
  return r;
}

// theta (as sin^2(theta / 2)) and tau by quadrature
__device__ void
scatter_quadrature(double eps, double b, double & s2, double & tau)
{
  const double r0 = closest_approach(eps, b);
  const double beta = b / r0;
  const double beta2 = beta * beta;
  const double ie = 1.0 / (r0 * eps);
  // from r = 256 on phi u / (r0 eps) = phi / (r eps) is below 5e-27 / eps: less than half
  // an ulp of h2 below, which r0 <= 64 keeps above 0.9 there
  const bool far = !(eps >= 1e-9 && r0 <= 64.0);
  double I = 0.0, J = 0.0;
#pragma unroll 2
  for (int j = 0; j < QN / 2; ++j)
  {
    const QuadNode & n = c_nodes[j];
    const double h2 = fma(-beta2, n.u2, 1.0);                           // 1 - beta^2 u^2
    const double g2 = fma(-phi_table(r0 * n.inv_u, far), n.u * ie, h2);
    const double ig = rsqrt(g2);
    I = fma(n.s, ig, I);
    J = fma(n.s_u2, ig - rsqrt(h2), J);
  }
  const double w = 3.14159265358979323846 / QN;
  const double theta = 3.14159265358979323846 - 2.0 * beta * w * I;
  const double sh = sin(0.5 * theta);
  s2 = sh * sh;
  tau = sqrt(fmax(r0 * r0 - b * b, 0.0)) - r0 * w * J;
}

__global__ void
quadrature_kernel(const double * eps, const double * b, long long n, double * s2, double * tau)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  double s, t;
  scatter_quadrature(eps[i], b[i], s, t);
  s2[i] = s;
  if (tau)
    tau[i] = t;
}

// normalised network inputs / targets for one sample
__host__ __device__ __forceinline__ double
baseline_ln_s2(double eps, double b)
{
  const double w = 2.0 * eps * b;
  return -log(1.0 + w * w * exp(2.0 * double(SG_D4) * b));
}

__global__ void
make_training_data(long long n, uint32_t k0, uint32_t k1, uint32_t offset, int target, float * x, float * y,
                   float * wts)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const U4 d = philox(U4{uint32_t(i), uint32_t(i >> 32), offset, 0x5347u}, k0, k1);
  const double le = -4.0 + 8.0 * (u53(d.x, d.y) - 0.5 / 9007199254740992.0);
  const double b = 12.0 * sqrt(u53(d.z, d.w) - 0.5 / 9007199254740992.0);
  const double eps = exp64(le * 2.302585092994046);
  double s2, tau;
  scatter_quadrature(eps, b, s2, tau);
  if (target == MTG_SURROGATE_TARGET_MAGIC)
  {
    double ct, st;
    int niter;
    scatter64(eps, b, s2, ct, st, niter, 0);
  }
  x[2 * i] = float(le * 0.25);
  x[2 * i + 1] = float(b / 6.0 - 1.0);
  y[2 * i] = float((log(fmax(s2, 1e-300)) - baseline_ln_s2(eps, b)) / SG_Y0);
  y[2 * i + 1] = float(tau / SG_Y1);
  // energy-transfer weight of the sample's sin^2(theta/2) error: the energy given to
  // the recoil is proportional to s2, and so is theta^2 at small angles (the angular
  // diffusion); a floor keeps every sample in the fit
  if (wts)
    wts[i] = float(s2 + SG_WEIGHT_FLOOR);
}

__global__ void
scale_weights(float * w, long long n, float f)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    w[i] *= f;
}

// ------------------------------------------------------------------ training
// Parameter vector layout: W1[64][2] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] W4[2][64] b4[2]
struct Offsets
{
  int w1, b1, w2, b2, w3, b3, w4, b4;
};
constexpr Offsets OFF{0, 128, 192, 4288, 4352, 8448, 8512, 8640};
static_assert(OFF.b4 + 2 == SG_NPARAM, "parameter layout");

__device__ __forceinline__ float
bf16_round(float v)
{
  return __bfloat162float(__float2bfloat16_rn(v));
}

// ---- one training step
//
// A batch step is 25,000 multiply-adds a sample (forward, data gradients, weight
// gradients) on weights that fit a corner of shared memory, so the whole step is one
// kernel: a block takes up to 64 samples at a time through all layers and back without leaving the SM,
// and keeps the weight gradients of its samples in registers (4 x 4 of each 64 x 64
// layer per thread) until it has done all its tiles.  A second kernel adds the blocks'
// gradients in block order (at most one block per SM) and takes the Adam step.  Layer by
// layer through global memory, with a thread per output, a step of 16,384 samples took
// 0.68 ms (64 steps with their 131,072 samples' targets 50.6 ms, now 5.0; a pass takes 41 us,
// its multiply-adds 10.4 at the issue rate); it is FP32 throughout, each sum in the same
// order as then but for the weight gradients' grouping by block.
//
// The 64 x 64 products read their operands from rows of 68 floats: a warp's 16-byte reads
// along a row, and of one column of 16 rows, then fall on different banks.
constexpr int TLD = 68;
template <int TS> // samples per tile, a multiple of 4 up to 64
struct TrainSmem
{
  float w1[SG_H * 2], b1[SG_H], b2[SG_H], b3[SG_H], w4[2 * SG_H], b4[2], pad[2];
  float w2[SG_H][TLD], w3[SG_H][TLD]; // [out][in]
  float h[3][TS][TLD];                // layer outputs
  float d[3][TS][TLD];                // silu'(z), then the gradient of z
  float x[TS][2], y[TS][2], wt[TS], dO[TS][2];
  float red[4][SG_H];
};

// z -> silu(z), silu'(z)
__device__ __forceinline__ void
silu_pair(float z, float & h, float & dh)
{
  const float s = 1.0f / (1.0f + expf(-z));
  h = z * s;
  dh = s * (1.0f + z * (1.0f - s));
}

// h_out = silu(h_in W^T + b) and its derivative, for the tile's TS x 64 outputs; thread
// (ts, tn) does samples 4 ts .. 4 ts + 3 and outputs tn, tn + 16, tn + 32, tn + 48
template <int TS>
__device__ __forceinline__ void
tile_forward(const float (*in)[TLD], const float (*w)[TLD], const float * bias, float (*out)[TLD], float (*der)[TLD],
             bool round_out)
{
  const int ts = threadIdx.x >> 4, tn = threadIdx.x & 15;
  if (4 * ts >= TS)
    return;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      acc[i][j] = bias[tn + 16 * j];
#pragma unroll 4
  for (int k = 0; k < SG_H; k += 4)
  {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      a[i] = *reinterpret_cast<const float4 *>(&in[4 * ts + i][k]);
      b[i] = *reinterpret_cast<const float4 *>(&w[tn + 16 * i][k]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
        acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
        acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      float h, dh;
      silu_pair(acc[i][j], h, dh);
      out[4 * ts + i][tn + 16 * j] = round_out ? bf16_round(h) : h;
      der[4 * ts + i][tn + 16 * j] = dh;
    }
}

// der = (dz W) * der: the gradient of the layer below's pre-activations; thread (ts, tk)
// does samples 4 ts .. 4 ts + 3 and inputs 4 tk .. 4 tk + 3
template <int TS>
__device__ __forceinline__ void
tile_backward(const float (*dz)[TLD], const float (*w)[TLD], float (*der)[TLD])
{
  const int ts = threadIdx.x >> 4, k0 = 4 * (threadIdx.x & 15);
  if (4 * ts >= TS)
    return;
  float acc[4][4] = {};
#pragma unroll 4
  for (int n = 0; n < SG_H; n += 4)
  {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      a[i] = *reinterpret_cast<const float4 *>(&dz[4 * ts + i][n]);
      b[i] = *reinterpret_cast<const float4 *>(&w[n + i][k0]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      const float an[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
      for (int q = 0; q < 4; ++q)
      {
        acc[i][0] = fmaf(an[q], b[q].x, acc[i][0]);
        acc[i][1] = fmaf(an[q], b[q].y, acc[i][1]);
        acc[i][2] = fmaf(an[q], b[q].z, acc[i][2]);
        acc[i][3] = fmaf(an[q], b[q].w, acc[i][3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
  {
    float4 * o = reinterpret_cast<float4 *>(&der[4 * ts + i][k0]);
    const float4 s = *o;
    *o = make_float4(acc[i][0] * s.x, acc[i][1] * s.y, acc[i][2] * s.z, acc[i][3] * s.w);
  }
}

// g += dz^T h over the tile: outputs 4 (t / 16) .. + 3, inputs 4 (t % 16) .. + 3
template <int TS>
__device__ __forceinline__ void
tile_weights(const float (*dz)[TLD], const float (*h)[TLD], float (&g)[4][4])
{
  const int n0 = 4 * (threadIdx.x >> 4), k0 = 4 * (threadIdx.x & 15);
#pragma unroll 8
  for (int s = 0; s < TS; ++s)
  {
    const float4 a = *reinterpret_cast<const float4 *>(&dz[s][n0]);
    const float4 b = *reinterpret_cast<const float4 *>(&h[s][k0]);
    const float an[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      g[i][0] = fmaf(an[i], b.x, g[i][0]);
      g[i][1] = fmaf(an[i], b.y, g[i][1]);
      g[i][2] = fmaf(an[i], b.z, g[i][2]);
      g[i][3] = fmaf(an[i], b.w, g[i][3]);
    }
  }
}

// Forward and backward pass of the batch rows (*step * B + i) % n of a training set
// (step NULL: row i), block b on tiles b, b + gridDim.x, ...: the block's gradients
// into P[b][SG_NPARAM], its loss into lossp[b].  `wts`: the samples' weights of output 0
// (NULL: 1); output 1 is weighted by w1.  quant: the hidden layers' weights and inputs
// are rounded to BF16.
template <int TS>
__global__ void __launch_bounds__(256, 1)
train_pass_kernel(const float * xs, const float * ys, const float * wts, long long n, long long B, const int * step,
                  const float * params, int quant, float w1, float * P, float * lossp)
{
  extern __shared__ __align__(16) unsigned char train_smem[];
  TrainSmem<TS> & m = *reinterpret_cast<TrainSmem<TS> *>(train_smem);
  const int t = threadIdx.x;
  for (int i = t; i < SG_H * SG_H; i += 256)
  {
    const float a = params[OFF.w2 + i], b = params[OFF.w3 + i];
    m.w2[i >> 6][i & 63] = quant ? bf16_round(a) : a;
    m.w3[i >> 6][i & 63] = quant ? bf16_round(b) : b;
  }
  if (t < 128)
  {
    m.w1[t] = params[OFF.w1 + t];
    m.w4[t] = params[OFF.w4 + t];
  }
  if (t < 64)
  {
    m.b1[t] = params[OFF.b1 + t];
    m.b2[t] = params[OFF.b2 + t];
    m.b3[t] = params[OFF.b3 + t];
  }
  if (t < 2)
    m.b4[t] = params[OFF.b4 + t];

  float g2[4][4] = {}, g3[4][4] = {};
  float gb1 = 0.0f, gb2 = 0.0f, gb3 = 0.0f; // output t % 64, a quarter of the tile's samples
  float g1 = 0.0f, g4 = 0.0f, gb4 = 0.0f;   // threads below 128 (gb4: 2)
  float loss = 0.0f;
  const long long first = step ? (long long)*step * B : 0;
  for (long long at = (long long)blockIdx.x * TS; at < B; at += (long long)gridDim.x * TS)
  {
    __syncthreads(); // the weights are in place; the last tile is done
    const int rows = int(B - at < TS ? B - at : TS);
    if (t < TS)
    {
      // rows past the batch's end hold zeros and get zero gradients
      const long long src = t < rows ? (first + at + t) % n : 0;
      m.x[t][0] = t < rows ? xs[2 * src] : 0.0f;
      m.x[t][1] = t < rows ? xs[2 * src + 1] : 0.0f;
      m.y[t][0] = t < rows ? ys[2 * src] : 0.0f;
      m.y[t][1] = t < rows ? ys[2 * src + 1] : 0.0f;
      m.wt[t] = t < rows && wts ? wts[src] : 1.0f;
    }
    __syncthreads();
    for (int i = t; i < TS * SG_H; i += 256)
    {
      const int s = i >> 6, j = i & 63;
      const float z = fmaf(m.x[s][1], m.w1[2 * j + 1], fmaf(m.x[s][0], m.w1[2 * j], m.b1[j]));
      float h, dh;
      silu_pair(z, h, dh);
      m.h[0][s][j] = quant ? bf16_round(h) : h;
      m.d[0][s][j] = dh;
    }
    __syncthreads();
    tile_forward<TS>(m.h[0], m.w2, m.b2, m.h[1], m.d[1], quant != 0);
    __syncthreads();
    tile_forward<TS>(m.h[1], m.w3, m.b3, m.h[2], m.d[2], false);
    __syncthreads();
    if (t < 2 * TS)
    {
      // output layer, loss and its gradient 2 w (o - y) / B
      const int s = t >> 1, c = t & 1;
      float o = m.b4[c];
#pragma unroll 4
      for (int k = 0; k < SG_H; k += 4)
      {
        const float4 a = *reinterpret_cast<const float4 *>(&m.h[2][s][k]);
        const float4 b = *reinterpret_cast<const float4 *>(&m.w4[c * SG_H + k]);
        o = fmaf(a.x, b.x, o);
        o = fmaf(a.y, b.y, o);
        o = fmaf(a.z, b.z, o);
        o = fmaf(a.w, b.w, o);
      }
      const float wc = c ? w1 : m.wt[s];
      const float e = s < rows ? o - m.y[s][c] : 0.0f;
      m.dO[s][c] = 2.0f * wc * e / float(B);
      loss += wc * e * e;
    }
    __syncthreads();
    if (t < 2 * SG_H)
    {
      const int c = t >> 6, k = t & 63;
      for (int s = 0; s < TS; ++s)
        g4 = fmaf(m.dO[s][c], m.h[2][s][k], g4);
    }
    else if (t < 2 * SG_H + 2)
      for (int s = 0; s < TS; ++s)
        gb4 += m.dO[s][t - 2 * SG_H];
    for (int i = t; i < TS * SG_H; i += 256)
    {
      const int s = i >> 6, k = i & 63;
      const float g = fmaf(m.dO[s][1], m.w4[SG_H + k], m.dO[s][0] * m.w4[k]);
      m.d[2][s][k] = g * m.d[2][s][k];
    }
    __syncthreads();
    tile_weights<TS>(m.d[2], m.h[1], g3);
    tile_backward<TS>(m.d[2], m.w3, m.d[1]);
    __syncthreads();
    tile_weights<TS>(m.d[1], m.h[0], g2);
    tile_backward<TS>(m.d[1], m.w2, m.d[0]);
    __syncthreads();
    if (t < 2 * SG_H)
      for (int s = 0; s < TS; ++s)
        g1 = fmaf(m.d[0][s][t >> 1], m.x[s][t & 1], g1);
    for (int s = TS / 4 * (t >> 6); s < TS / 4 * (t >> 6) + TS / 4; ++s)
    {
      gb1 += m.d[0][s][t & 63];
      gb2 += m.d[1][s][t & 63];
      gb3 += m.d[2][s][t & 63];
    }
  }
  float * out = P + (long long)blockIdx.x * SG_NPARAM;
  const int n0 = 4 * (t >> 4), k0 = 4 * (t & 15);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      out[OFF.w2 + (n0 + i) * SG_H + k0 + j] = g2[i][j];
      out[OFF.w3 + (n0 + i) * SG_H + k0 + j] = g3[i][j];
    }
  if (t < 2 * SG_H)
  {
    out[OFF.w1 + t] = g1;
    out[OFF.w4 + t] = g4;
  }
  else if (t < 2 * SG_H + 2)
    out[OFF.b4 + t - 2 * SG_H] = gb4;
  const float gb[3] = {gb1, gb2, gb3};
  const int off[3] = {OFF.b1, OFF.b2, OFF.b3};
  for (int l = 0; l < 3; ++l)
  {
    __syncthreads();
    m.red[t >> 6][t & 63] = gb[l];
    __syncthreads();
    if (t < SG_H)
      out[off[l] + t] = ((m.red[0][t] + m.red[1][t]) + m.red[2][t]) + m.red[3][t];
  }
  __syncthreads();
  float * red = &m.red[0][0];
  red[t] = loss;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1)
  {
    if (t < w)
      red[t] += red[t + w];
    __syncthreads();
  }
  if (t == 0)
    lossp[blockIdx.x] = red[0];
}

// Gradient of parameter i: the blocks' gradients added in block order within each of
// four quarters of the blocks, one per group of 128 threads, then the quarters (a thread
// per parameter waited on 152 loads: 15.6 us a step, now 9.9).
constexpr int GSLICES = 4;
__device__ __forceinline__ float
sum_blocks(const float * P, int parts, int i)
{
  __shared__ float part[GSLICES][128];
  const int q = threadIdx.x >> 7;
  float g = 0.0f;
  if (i < SG_NPARAM)
  {
    const int p1 = parts * (q + 1) / GSLICES;
#pragma unroll 8
    for (int p = parts * q / GSLICES; p < p1; ++p)
      g += P[(long long)p * SG_NPARAM + i];
  }
  part[q][threadIdx.x & 127] = g;
  __syncthreads();
  const int t = threadIdx.x & 127;
  return ((part[0][t] + part[1][t]) + part[2][t]) + part[3][t];
}

__global__ void __launch_bounds__(128 * GSLICES)
gradient_sum_kernel(const float * P, int parts, float * g)
{
  const int i = blockIdx.x * 128 + (threadIdx.x & 127);
  const float s = sum_blocks(P, parts, i);
  if (threadIdx.x < 128 && i < SG_NPARAM)
    g[i] = s;
}

// gradient sum and Adam step; the last block to finish counts the step
__global__ void __launch_bounds__(128 * GSLICES)
adam_step(float * w, const float * P, int parts, float * m, float * v, int * step, unsigned int * done, float lr,
          float b1, float b2, float eps_adam, float lr_final_frac, int total_steps)
{
  const int i = blockIdx.x * 128 + (threadIdx.x & 127);
  const int t = *step + 1;
  const float gi = sum_blocks(P, parts, i);
  if (threadIdx.x < 128 && i < SG_NPARAM)
  {
    // cosine decay from lr to lr * lr_final_frac
    const float prog = fminf(1.0f, float(t) / float(total_steps));
    const float lrt = lr * (lr_final_frac + (1.0f - lr_final_frac) * 0.5f * (1.0f + cosf(3.14159265f * prog)));
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.0f - powf(b1, float(t)));
    const float vh = vi / (1.0f - powf(b2, float(t)));
    w[i] -= lrt * mh / (sqrtf(vh) + eps_adam);
  }
  // every thread of the block has read the step (sum_blocks has synchronised it)
  if (threadIdx.x == 0 && atomicAdd(done, 1u) == gridDim.x - 1)
  {
    *done = 0u;
    *step = t;
  }
}

// flat parameters -> inference layout
__global__ void
pack_net(const float * w, SurrogateNet * net)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 128)
    net->w1[i / 2][i % 2] = w[OFF.w1 + i];
  if (i < 64)
  {
    net->b1[i] = w[OFF.b1 + i];
    net->b2[i] = w[OFF.b2 + i];
    net->b3[i] = w[OFF.b3 + i];
    net->w4[0][i] = w[OFF.w4 + i];
    net->w4[1][i] = w[OFF.w4 + 64 + i];
  }
  if (i < 2)
    net->b4[i] = w[OFF.b4 + i];
  if (i < 64 * SG_LD)
  {
    const int r = i / SG_LD, c = i % SG_LD;
    net->w2[r][c] = __float2bfloat16_rn(c < 64 ? w[OFF.w2 + r * 64 + c] : 0.0f);
    net->w3[r][c] = __float2bfloat16_rn(c < 64 ? w[OFF.w3 + r * 64 + c] : 0.0f);
  }
}

// surrogate evaluation for the scatter service (whole warps; tail lanes use dummy input)
__global__ void
surrogate_eval_kernel(const SurrogateNet * gnet, const double * eps, const double * b, long long n, double * s2,
                      int fallback_exact)
{
  __shared__ SurrogateNet net;
  for (int i = threadIdx.x; i < int(sizeof(SurrogateNet) / 4); i += blockDim.x)
    reinterpret_cast<float *>(&net)[i] = reinterpret_cast<const float *>(gnet)[i];
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const float e = i < n ? float(eps[i]) : 1.0f;
  const float bb = i < n ? float(b[i]) : 1.0f;
  const bool in = surrogate_in_domain(e, bb);
  const float o0 = surrogate_eval_warp(&net, in && i < n, surrogate_x1(in ? e : 1.0f), surrogate_x2(in ? bb : 1.0f));
  if (i >= n)
    return;
  float s, c;
  if (in)
    surrogate_s2_from(e, bb, o0, s, c);
  else
  {
    // outside the trained domain the exact FP32 path applies, as in the engine
    int it;
    scatter32(e, bb, s, c, it);
  }
  s2[i] = double(s);
}

} // namespace mtg

// ------------------------------------------------------------------ host side
namespace mtg
{

// the quadrature's nodes and the pieces of phi, made once per process
struct QuadTables
{
  QuadNode nodes[QN / 2];
  std::vector<double> phi;
};

// phi(r) with the rounding of each exponent's product made good (host)
static double
screening_exact(double r)
{
  const double c[4] = {0.18175, 0.50986, 0.28022, 0.028171}, d[4] = {3.1998, 0.94229, 0.4029, 0.20162};
  double phi = 0.0;
  for (int i = 0; i < 4; ++i)
  {
    const double x = -d[i] * r, e = exp64(x);
    phi += c[i] * fma(e, fma(-d[i], r, -x), e);
  }
  return phi;
}

static const QuadTables &
quad_tables()
{
  static QuadTables q;
  static std::once_flag once;
  std::call_once(once, [] {
    const double pi = 3.14159265358979323846;
    for (int j = 1; j <= QN / 2; ++j)
    {
      const double u = std::cos((2.0 * j - 1.0) * pi / (2.0 * QN));
      const double s = std::sqrt(1.0 - u * u);
      q.nodes[j - 1] = QuadNode{1.0 / u, u, u * u, s, s / (u * u)};
    }
    // each piece: the interpolant at its PHI_N Chebyshev points, as a Chebyshev series
    // c_0 / 2 + sum c_k T_k(t), then in powers of t
    q.phi.resize(size_t(PHI_OCT << PHI_BITS) * PHI_N);
    double T[PHI_N][PHI_N] = {}; // T_k's coefficients
    T[0][0] = T[1][1] = 1.0;
    for (int k = 2; k < PHI_N; ++k)
      for (int i = 0; i < PHI_N; ++i)
        T[k][i] = (i > 0 ? 2.0 * T[k - 1][i - 1] : 0.0) - T[k - 2][i];
    for (int p = 0; p < PHI_OCT << PHI_BITS; ++p)
    {
      const double a = std::ldexp(1.0 + double(p & ((1 << PHI_BITS) - 1)) / (1 << PHI_BITS), PHI_LO + (p >> PHI_BITS));
      const double h = std::ldexp(1.0, PHI_LO + (p >> PHI_BITS) - PHI_BITS);
      double y[PHI_N];
      for (int m = 0; m < PHI_N; ++m)
        y[m] = screening_exact(a + 0.5 * h * (std::cos((2 * m + 1) * pi / (2 * PHI_N)) + 1.0));
      for (int k = 0; k < PHI_N; ++k)
      {
        double c = 0.0;
        for (int m = 0; m < PHI_N; ++m)
          c += y[m] * std::cos(k * (2 * m + 1) * pi / (2 * PHI_N));
        c *= (k > 0 ? 2.0 : 1.0) / PHI_N;
        for (int i = 0; i < PHI_N; ++i)
          q.phi[size_t(p) * PHI_N + i] += c * T[k][i];
      }
    }
  });
  return q;
}

// onto the current device, for every context that integrates (before its first use): a
// flag for the process would leave a second device, or one that was reset, with zeros.
// Contexts that share a device write the same bytes.
cudaError_t
upload_quadrature()
{
  const QuadTables & q = quad_tables();
  const cudaError_t e = cudaMemcpyToSymbol(c_nodes, q.nodes, sizeof q.nodes);
  return e != cudaSuccess ? e : cudaMemcpyToSymbol(g_phi, q.phi.data(), sizeof(double) * q.phi.size());
}

cudaError_t
launch_quadrature(const double * eps, const double * b, long long n, double * s2, double * tau, cudaStream_t st)
{
  if (n > 0)
    quadrature_kernel<<<(unsigned int)((n + 127) / 128), 128, 0, st>>>(eps, b, n, s2, tau);
  return cudaGetLastError();
}

cudaError_t
launch_surrogate_eval(const void * net, const double * eps, const double * b, long long n, double * s2,
                      cudaStream_t st)
{
  if (n > 0)
    surrogate_eval_kernel<<<(unsigned int)((n + 127) / 128), 128, 0, st>>>(
        reinterpret_cast<const SurrogateNet *>(net), eps, b, n, s2, 0);
  return cudaGetLastError();
}

cudaError_t
launch_pack_net(const float * params, void * net, cudaStream_t st)
{
  pack_net<<<(64 * SG_LD + 127) / 128, 128, 0, st>>>(params, reinterpret_cast<SurrogateNet *>(net));
  return cudaGetLastError();
}

size_t
surrogate_net_bytes()
{
  return sizeof(SurrogateNet);
}

// A training pass's tile and blocks: one block per SM of the current device at most, and
// the tile whose busiest block is done first.  A tile of TS samples takes a time like
// TS + TILE_FIXED: measured 15, 14 and 8.5 us for 64, 56 and 28 (the threads of the 64 x 64
// products that a small tile leaves idle take as long as the others, and so do the
// barriers).  us per step, Adam's included, by batch, for tiles of 64, 56 and 28:
//     4096  28.9  30.7  28.0      12000  47.7  45.4  44.7      26000  62.7  71.7  76.9
//     8192  31.1  33.0  36.1      16384  48.4  46.3  53.0      29185  75.9  72.1  77.9
//     9000  31.2  45.2  43.5      20000  61.6  59.5  61.5      32768  77.1  72.3  86.4
//    10007  47.0  45.4  44.5      25536  62.9  59.5  70.0      65536 120.8 125.6 152.4
// (by samples alone 20,000 and 29,185 went to 28.)
constexpr int TILE_FIXED = 19;
struct TrainShape
{
  void (*kernel)(const float *, const float *, const float *, long long, long long, const int *, const float *, int,
                 float, float *, float *) = nullptr;
  int blocks = 0;
  size_t smem = 0;
};

template <int TS>
static void
try_tile(long long B, int sms, long long & best, TrainShape & t)
{
  const long long tiles = (B + TS - 1) / TS;
  const long long time = (tiles + sms - 1) / sms * (TS + TILE_FIXED);
  if (t.kernel && time >= best)
    return;
  best = time;
  t.kernel = train_pass_kernel<TS>;
  t.blocks = int(std::min<long long>(tiles, sms));
  t.smem = sizeof(TrainSmem<TS>);
}

static cudaError_t
train_shape(long long B, TrainShape & t)
{
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  e = e ? e : cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e)
    return e;
  sms = std::max(sms, 1);
  long long best = 0;
  try_tile<64>(B, sms, best, t);
  try_tile<56>(B, sms, best, t);
  try_tile<28>(B, sms, best, t);
  return cudaFuncSetAttribute(t.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(t.smem));
}

// device memory cut from one allocation, freed with it
struct Arena
{
  unsigned char * base = nullptr;
  size_t size = 0;
  ~Arena()
  {
    if (base)
      cudaFree(base);
  }
  // bytes of an array, kept 256-byte aligned
  size_t add(size_t bytes)
  {
    const size_t at = size;
    size += (bytes + 255) / 256 * 256;
    return at;
  }
  cudaError_t alloc() { return cudaMalloc(&base, size); }
  float * at(size_t o) { return reinterpret_cast<float *>(base + o); }
};

constexpr unsigned int PARAM_BLOCKS = (SG_NPARAM + 127) / 128;

// ---- exported to the C ABI layer (mtg_api.cu)

cudaError_t
surrogate_gradients(const float * params_h, const float * x_h, const float * y_h, long long n, float w_tau,
                    float * loss_h, float * grads_h)
{
  TrainShape shape;
  cudaError_t e = train_shape(n, shape);
  if (e)
    return e;
  const int blocks = shape.blocks;
  const size_t B = size_t(n);
  Arena a;
  const size_t ow = a.add(4 * SG_NPARAM), og = a.add(4 * SG_NPARAM), ox = a.add(8 * B), oy = a.add(8 * B),
               oP = a.add(4 * size_t(SG_NPARAM) * blocks), ol = a.add(4 * size_t(blocks));
  if ((e = a.alloc()) != cudaSuccess)
    return e;
  e = cudaMemcpy(a.at(ow), params_h, SG_NPARAM * 4, cudaMemcpyHostToDevice);
  e = e ? e : cudaMemcpy(a.at(ox), x_h, 8 * B, cudaMemcpyHostToDevice);
  e = e ? e : cudaMemcpy(a.at(oy), y_h, 8 * B, cudaMemcpyHostToDevice);
  if (e)
    return e;
  shape.kernel<<<blocks, 256, shape.smem>>>(a.at(ox), a.at(oy), nullptr, n, n, nullptr, a.at(ow), 0, w_tau, a.at(oP),
                                            a.at(ol));
  gradient_sum_kernel<<<PARAM_BLOCKS, 128 * GSLICES>>>(a.at(oP), blocks, a.at(og));
  e = cudaGetLastError();
  e = e ? e : cudaMemcpy(grads_h, a.at(og), SG_NPARAM * 4, cudaMemcpyDeviceToHost);
  std::vector<float> lp(static_cast<size_t>(blocks));
  e = e ? e : cudaMemcpy(lp.data(), a.at(ol), 4 * lp.size(), cudaMemcpyDeviceToHost);
  if (!e)
  {
    double s = 0.0;
    for (float v : lp)
      s += v;
    *loss_h = float(s / double(n));
  }
  return e;
}

// Train from scratch.  params_out: SG_NPARAM floats; net_out: device SurrogateNet.
cudaError_t
surrogate_train(long long n_train, int batch, int epochs, int qat_epochs, float lr, unsigned long long seed,
                float w_tau, int target, int weighting, float * params_dev, void * net_dev, double * final_loss,
                double * train_seconds)
{
  TrainShape shape;
  cudaError_t e = train_shape(batch, shape);
  if (e)
    return e;
  const int blocks = shape.blocks;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0);
  const size_t n = size_t(n_train);
  Arena a;
  const size_t ox = a.add(8 * n), oy = a.add(8 * n), owt = a.add(weighting ? 4 * n : 0), om = a.add(4 * SG_NPARAM),
               ov = a.add(4 * SG_NPARAM), ostep = a.add(8), oP = a.add(4 * size_t(SG_NPARAM) * blocks),
               ol = a.add(4 * size_t(blocks));
  e = a.alloc();
  std::vector<float> w0(SG_NPARAM, 0.0f);
  const long long steps_per_epoch = std::max<long long>(1, n_train / batch);
  const int total = int(steps_per_epoch * epochs);
  if (!e)
  {
    float *x = a.at(ox), *y = a.at(oy), *wts = weighting ? a.at(owt) : nullptr, *m = a.at(om), *v = a.at(ov);
    int * step = reinterpret_cast<int *>(a.at(ostep)); // and the finished blocks of a step
    const uint32_t k0 = uint32_t(seed), k1 = uint32_t(seed >> 32) ^ 0x53474E4Eu;
    make_training_data<<<(unsigned int)((n_train + 127) / 128), 128>>>(n_train, k0, k1, 0u, target, x, y, wts);
    // initial weights: uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) from a host LCG
    uint64_t st = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto uni = [&]() {
      st = st * 6364136223846793005ull + 1442695040888963407ull;
      return float((st >> 11) * (1.0 / 9007199254740992.0)) * 2.0f - 1.0f;
    };
    for (int i = 0; i < 128; ++i)
      w0[OFF.w1 + i] = uni() * 1.2f;
    for (int i = 0; i < 4096; ++i)
      w0[OFF.w2 + i] = uni() * 0.3f;
    for (int i = 0; i < 4096; ++i)
      w0[OFF.w3 + i] = uni() * 0.3f;
    for (int i = 0; i < 128; ++i)
      w0[OFF.w4 + i] = uni() * 0.2f;
    if (wts)
    {
      // normalise the weights to mean 1 over the training set
      std::vector<float> hw(n);
      e = cudaMemcpy(hw.data(), wts, 4 * n, cudaMemcpyDeviceToHost);
      double sum = 0.0;
      for (float w : hw)
        sum += double(w);
      if (!e && sum > 0.0)
        scale_weights<<<(unsigned int)((n_train + 255) / 256), 256>>>(wts, n_train, float(double(n_train) / sum));
    }
    e = e ? e : cudaMemcpy(params_dev, w0.data(), 4 * SG_NPARAM, cudaMemcpyHostToDevice);
    e = e ? e : cudaMemset(a.base + om, 0, oP - om); // Adam's moments and the step count
    for (int it = 0; it < total && !e; ++it)
    {
      const int quant = it >= int(steps_per_epoch * (epochs - qat_epochs));
      shape.kernel<<<blocks, 256, shape.smem>>>(x, y, wts, n_train, batch, step, params_dev, quant, w_tau, a.at(oP),
                                                a.at(ol));
      adam_step<<<PARAM_BLOCKS, 128 * GSLICES>>>(params_dev, a.at(oP), blocks, m, v, step,
                                       reinterpret_cast<unsigned int *>(step) + 1, lr, 0.9f, 0.999f, 1e-8f, 0.02f,
                                       total);
      e = cudaGetLastError();
    }
  }
  if (!e)
  {
    std::vector<float> lp(static_cast<size_t>(blocks));
    e = cudaMemcpy(lp.data(), a.at(ol), 4 * lp.size(), cudaMemcpyDeviceToHost);
    double sum = 0.0;
    for (float val : lp)
      sum += val;
    *final_loss = sum / double(batch);
  }
  e = e ? e : launch_pack_net(params_dev, net_dev, nullptr);
  e = e ? e : cudaDeviceSynchronize();
  cudaEventRecord(e1);
  cudaEventSynchronize(e1);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, e0, e1);
  *train_seconds = ms / 1e3;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return e;
}

cudaError_t
upload_newton_guess32_surrogate(const float * table)
{
  return upload_newton_guess32_here(table);
}

} // namespace mtg
