// FP32 cascade path: the same collision loop as the FP64 plain path
// (TrimBase::trim, trim.C:74-424) in single precision, with three changes of
// evaluation that keep FP32 accurate and fast:
//   * electronic stopping and the maximum impact parameter of the free flight are
//     read from a per-(species, material) table of (S(E), p_max(E)) pairs, uniform
//     in ln E with 2048 points and filled by the FP64 code, instead of
//     re-evaluating ~11 transcendentals per element (S) and a chain of two square
//     roots, a power and two divisions (p_max) per collision;
//   * the Newton solve for the distance of closest approach iterates on
//     d = r - b (the same Newton steps as trim.C:192-233 written in a variable
//     that does not cancel), and sin^2(theta/2) is formed as (1 - co)(1 + co)
//     with 1 - co = d (1 - A F / (F + 1)) / (r + roc), algebraically equal to
//     1 - co^2 of trim.C:266-269 without its cancellation at small angles; the
//     solve starts from a tabulated first guess (mtg_newton_guess.h), so one
//     step nearly always meets the reference's stopping test;
//   * the random azimuth is drawn directly (uniform angle around the flight
//     direction) instead of by unit-ball rejection; the two give the same
//     distribution, and the direct draw has no data-dependent loop.
// Energies are kept as a float pair (value + rounding remainder) so that
// the small per-collision losses are not rounded away, and the lane tallies use
// Kahan-compensated sums; FP64 instructions stay out of the collision loop.
#include <mutex>
#include <vector>

#include "mtg_cascade32.cuh"
#include "mtg_collide64.cuh"

namespace mtg
{

// calls f with the kernel of a feature level; the surrogate engine runs the cluster-only
// levels in the geometry variants
template <bool SG, bool ONE, bool PACED, class F>
static cudaError_t
with_kernel(int level, F f)
{
  switch (level)
  {
    case LVL_LEAN: return f(cascade32_kernel<LVL_LEAN, SG, ONE, PACED>);
    case LVL_MID: return f(cascade32_kernel<LVL_MID, SG, ONE, PACED>);
    case LVL_EVENTS: return f(cascade32_kernel<LVL_EVENTS, SG, ONE, PACED>);
    case LVL_GEO: return f(cascade32_kernel<LVL_GEO, SG, ONE, PACED>);
    case LVL_CLU: return f(cascade32_kernel<SG ? LVL_GEO : LVL_CLU, SG, ONE, PACED>);
    case LVL_CLU_EV: return f(cascade32_kernel<SG ? LVL_FULL : LVL_CLU_EV, SG, ONE, PACED>);
    default: return f(cascade32_kernel<LVL_FULL, SG, ONE, PACED>);
  }
}

// paced: only in the plain engine's runs of one simulation (EngineParams::take_mask)
template <class F>
static cudaError_t
with_kernel(int level, int surrogate, int one, int paced, F f)
{
  if (surrogate)
    return one ? with_kernel<true, true, false>(level, f) : with_kernel<true, false, false>(level, f);
  if (paced)
    return with_kernel<false, true, true>(level, f);
  return one ? with_kernel<false, true, false>(level, f) : with_kernel<false, false, false>(level, f);
}

cudaError_t
launch_cascade32(const EngineParams & prm, const Fp32Tables & t, int grid, int block, size_t smem, cudaStream_t st,
                 int surrogate)
{
  Tables32 tabs;
  tabs.mats = reinterpret_cast<const Mat32 *>(t.mats32);
  tabs.cold = reinterpret_cast<const MatCold32 *>(t.cold32);
  tabs.sims = reinterpret_cast<const Sim32 *>(t.sims32);
  tabs.stop = reinterpret_cast<const float2 *>(t.stop);
  tabs.lnE_min = t.lnE_min;
  tabs.inv_dlnE = t.inv_dlnE;
  tabs.cw = t.cw;
  tabs.tau = t.tau;
  tabs.flscale = t.flscale;
  tabs.net = reinterpret_cast<const SurrogateNet *>(t.mlp);
  One32 one;
  if (prm.stage_tables)
  {
    one.sim = *t.one_sim;
    one.desc = *t.one_desc;
  }
  else
    memset(&one, 0, sizeof one);
  return with_kernel(prm.level, surrogate, prm.stage_tables, prm.take_mask != 0u, [&](auto * kernel) {
    kernel<<<grid, block, smem, st>>>(prm, tabs, one);
    return cudaGetLastError();
  });
}

// residency of the variant of feature level `level` (KernelLevel), with the
// shared-memory opt-in it needs
cudaError_t
occupancy32(int block, size_t smem, int * blocks_per_sm, int surrogate, int level, int one)
{
  auto query = [&](auto * kernel) {
    if (smem > 48 * 1024)
    {
      const cudaError_t e = allow_shared_memory(kernel);
      if (e != cudaSuccess)
        return e;
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, block, smem);
  };
  if (one && !surrogate)
  {
    const cudaError_t e = with_kernel(level, 0, 1, 1, query);
    if (e != cudaSuccess)
      return e;
  }
  return with_kernel(level, surrogate, one, 0, query);
}

// bytes the stacks and overflow lists hold per recoil: the larger of the two layouts
size_t
record_size32()
{
  return sizeof(Rec32Tag);
}

size_t
cold_slot_bytes32()
{
  return sizeof(LaneCold<AccKahan32>);
}

// ---- scattering service (FP32 exact)
__global__ void
scatter32_kernel(const double * eps, const double * b, long long n, double * s2, int potential)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const float e = float(eps[i]), bb = float(b[i]);
  float s, c;
  int it;
  scatter32(e, bb, s, c, it, potential);
  s2[i] = double(s);
}

cudaError_t
launch_scatter32(const double * eps, const double * b, long long n, double * s2, int potential, cudaStream_t st)
{
  const int block = 256;
  if (n > 0)
    scatter32_kernel<<<(unsigned int)((n + block - 1) / block), block, 0, st>>>(eps, b, n, s2, potential);
  return cudaGetLastError();
}

// ---- first-guess table of the FP32 Newton solve
// phi(r) of the universal (pot 0) or Moliere (1) potential in FP64 (trim.C:197-213),
// with the project's exp64 so that the table has the same bits on every host
static double
screening_phi64(int pot, double r)
{
  if (pot == 1)
    return 0.35 * exp64(-0.3 * r) + 0.55 * exp64(-1.2 * r) + 0.1 * exp64(-6.0 * r);
  return 0.18175 * exp64(-3.1998 * r) + 0.50986 * exp64(-0.94229 * r) + 0.28022 * exp64(-0.4029 * r) +
         0.028171 * exp64(-0.20162 * r);
}

const float *
newton_guess_table32()
{
  // f(r) = b^2 / r + phi(r) / eps - r falls strictly with r, f(b) = phi(b) / eps > 0
  // and f(b + 2 / eps) < 0 because phi <= 1.000001: 72 halvings of that bracket
  // (at most 2^19 wide) leave the root to 1e-16, far below float resolution of d
  static std::vector<float> table;
  static std::once_flag once;
  std::call_once(once, [] {
    table.resize(NG_CELLS);
    for (int pot = 0; pot < NG_POT; ++pot)
      for (int i = 0; i < NG_U; ++i)
      {
        const double eps = exp64((NG_U0 + i * NG_DU) * 0.69314718055994531);
        for (int j = 0; j < NG_B; ++j)
        {
          const double b = j * NG_DB;
          double lo = b, hi = b + 2.0 / eps;
          for (int it = 0; it < 72; ++it)
          {
            const double m = 0.5 * (lo + hi);
            const double f = b * b / m + screening_phi64(pot, m) / eps - m;
            (f > 0.0 ? lo : hi) = m;
          }
          const double d = 0.5 * (lo + hi) - b;
          table[(size_t(pot) * NG_U + i) * NG_B + j] = float(log64(d) * 1.4426950408889634);
        }
      }
  });
  return table.data();
}

cudaError_t
upload_newton_guess32()
{
  return upload_newton_guess32_here(newton_guess_table32());
}

// ---- stopping through the FP32 table (one (species, material) row)
__global__ void
stopping32_kernel(const float * row, float lnE_min, float inv_d, const double * E, long long n, double * out)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
  {
    float S = 0.0f, pmax = 0.0f;
    stop_lookup(reinterpret_cast<const float2 *>(row), lnE_min, inv_d, float(E[i]), S, pmax);
    out[i] = double(S);
  }
}

cudaError_t
launch_stopping32(const float * row, float lnE_min, float inv_d, const double * E, long long n, double * out,
                  cudaStream_t st)
{
  const int block = 256;
  if (n > 0)
    stopping32_kernel<<<(unsigned int)((n + block - 1) / block), block, 0, st>>>(row, lnE_min, inv_d, E, n, out);
  return cudaGetLastError();
}

} // namespace mtg
