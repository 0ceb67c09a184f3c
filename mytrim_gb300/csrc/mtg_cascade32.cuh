// The single-precision cascade kernel: the warp-cooperative scheme of mtg_engine.cuh
// (a member per lane, one collision per loop iteration, a LIFO recoil stack per warp)
// laid out for a machine whose bound is issue slots.
//
// At the benchmark workloads every warp iteration holds some 4 lanes that displace a
// recoil and 4 whose member comes to rest, out of 32: code that belongs to one of those
// events runs nearly every iteration for an eighth of the lanes.  So an iteration does
// as little as it can for them, and the rest waits until it can be done for more lanes:
//   * a displaced recoil is written to the stack as the collision leaves it: momentum
//     not normalised, the sum that its path key is mixed from, and a bit that says
//     whether it left a vacancy; the lane that starts it normalises, mixes and counts;
//   * a lane whose member came to rest keeps it until the warp refills (refill_min idle
//     lanes, 8 by default) and does the tallies of the rest then;
//   * the lanes hand their energy sums to the FP64 arrays on the same iterations, every
//     64 (a branch that is uniform over the warp).
// A recoil is 48 bytes (64 with the event log), moved in 16-byte pieces.  Runs of a
// single simulation (ONE) read its constants as kernel parameters and its material rows
// with shared-memory addresses; other runs through pointers.  Together, against the
// kernel that did each event's work in its own iteration and kept every table behind a
// generic pointer (end-to-end times, same trajectories): Ag 200 keV into Si 295 -> 259 ms
// (500,000 primaries), B 10 keV into SiO2/Si 30.1 -> 25.9 ms (10^6), Cu 100 keV 4.43 ->
// 3.91 ms (10^4), Xe into UO2 with bubbles 27.7 -> 23.5 ms (10^5), Au 1 MeV with voxels
// 52.6 -> 39.1 ms (10^4), As 50 keV with the event log 35.6 -> 27.4 ms (70,000).
#pragma once

#include "mtg_common.cuh"
#include "mtg_engine.cuh"
#include "mtg_geometry.cuh"
#include "mtg_kernels.h"
#include "mtg_scatter32.cuh"
#include "mtg_surrogate.cuh"

namespace mtg
{

struct P32
{
  float x, y, z;
  float dx, dy, dz;
  float E, El; // energy as value + remainder
  uint64_t key;
  uint32_t meta; // generation << 7 | species (a simulation has at most 33)
  uint32_t prim;
  int sim;
  int tag; // IonBase::_tag: cluster index where a followed recoil was created, else -1
};
constexpr uint32_t META_SPECIES = 0x3fu, META_VACANCY = 0x40u;
constexpr int META_GEN = 7;

__device__ __forceinline__ int
member_gen(const P32 & p)
{
  return int(p.meta >> META_GEN);
}
__device__ __forceinline__ int
member_species(const P32 & p)
{
  return int(p.meta & META_SPECIES);
}

// a recoil on the stack or in the overflow lists: position and energy; momentum and
// primary; the unmixed path key, meta (with META_VACANCY) and simulation
struct alignas(16) Rec32
{
  float4 a, b;
  uint4 c;
};
// with the event log: the tag too
struct alignas(16) Rec32Tag
{
  float4 a, b;
  uint4 c, d;
};

__device__ __forceinline__ float
record_energy(const Rec32 & r)
{
  return r.a.w;
}
__device__ __forceinline__ float
record_energy(const Rec32Tag & r)
{
  return r.a.w;
}

struct Tables32
{
  const Mat32 * mats;
  const MatCold32 * cold; // the rest of the same rows, in global memory
  const Sim32 * sims;
  const float2 * stop; // (S, p_max) pairs, STOP_N per row
  float lnE_min, inv_dlnE;
  float cw, tau, flscale; // run-wide settings: first-flight cap, tau, 1 / length scale
  const SurrogateNet * net;
};

// the target element of a collision as the tallies and the event log see it
struct Target32
{
  int Z2;
  float m2, Elbind, Edisp, maz, mam;
};

// constants of the simulation of a single-simulation run
struct One32
{
  Sim32 sim;
  SimDesc desc;
};

// what a collision leaves of its target atom
struct Recoil32
{
  float x, y, z, E;
  float dx, dy, dz; // momentum, not normalised
  uint32_t gen;
  int tag;
};

// E -= d for |d| <= E, keeping the rounding remainder: FastTwoSum twice (Dekker 1971;
// with the larger term first it gives TwoSum's remainder in half its operations, 2.7 %
// of the kernel's time on Ag into Si)
__device__ __forceinline__ void
ff_sub(float & hi, float & lo, float d)
{
  const float s = hi - d;
  const float err = (hi - s) - d;
  const float l = lo + err;
  const float h = s + l;
  lo = l - (h - s);
  hi = h;
}

// S(E) and p_max(E) from one row of the table; false below its first point, where
// S scales as sqrt(E) from there and p_max is left to the formula
__device__ __forceinline__ bool
stop_lookup(const float2 * row, float lnE_min, float inv_d, float E, float & S, float & pmax)
{
  const float u = (__logf(E) - lnE_min) * inv_d;
  if (!(u > 0.0f))
  {
    S = row[0].x * sqrtf(E * float(1.0 / STOP_EMIN));
    return false;
  }
  const int i = min(int(u), STOP_N - 2);
  const float f = u - float(i);
  const float2 a = row[i], b = row[i + 1];
  S = fmaf(f, b.x - a.x, a.x);
  pmax = fmaf(f, b.y - a.y, a.y);
  return true;
}

// what the first half of a collision hands to the scattering and the second half
struct PhaseA32
{
  int mat, nn;   // material row (from the simulation's first) and target element
  float two_m1;
  float4 el;     // Elbind, disp_thresh, Edisp, recoil
  float eps, b;  // reduced energy and impact parameter
  float ec, my;
  float ls, dee; // flight length and electronic loss
  uint32_t azimuth;
  bool gone;     // outside the sample: no collision, the member is dropped
  int tag;       // the material's _tag: the cluster index inside a cluster, else -1
};

// flight, target atom and electronic loss (trim.C:80-170)
template <bool EXT, bool ONE>
__device__ __forceinline__ PhaseA32
phase_a32(P32 & p, uint32_t ic, const Sim32 & sim, const Mat32 * mats, const Tables32 & t, uint32_t k0, uint32_t k1)
{
  PhaseA32 a;
  // n_layers, n_mat, mat_base in one read where they are not parameters: a warp's lanes
  // follow members of many simulations then, and each of these reads is a gather.  With
  // Sim32's fields read in 16-byte pieces the batch of 4096 simulations (2 x 10^5 primaries)
  // takes 204 ms, 213 field by field.
  const int4 sh = ONE ? make_int4(sim.n_layers, sim.n_mat, 0, 0) : *reinterpret_cast<const int4 *>(&sim.n_layers);
  mats += sh.z;
  // material lookup: SampleLayers (sample_layers.C:27-43) or sampleClusters
  // (sample_clusters.C:42-53)
  int k = 0;
  a.gone = false;
  a.tag = -1;
  if (EXT && sim.geometry == 1)
  {
    const float pos[3] = {p.x, p.y, p.z};
    const int l = cluster_lookup<float>(pos, sim.w, sim.bc, sim.kn, sim.kd, sim.cmr, sim.cl, sim.cl_next,
                                        sim.cl_head, sim.n_clusters, sim.cl_mask, sim.mn, sim.inv_mcell);
    a.gone = l == -2; // no material: the member is dropped (trim.C:81-83)
    k = l >= 0 ? 1 : 0;
    a.tag = l >= 0 ? l : -1; // sampleClusters::lookupMaterial sets material[1]->_tag = l
  }
  else
    while (k < sh.x - 1 && !(p.x < sim.layer_end[k])) // layer k is of material k
      ++k;
  a.mat = int(p.meta & META_SPECIES) * sh.y + k;
  const Mat32 & mc = mats[a.mat];
  const float4 head = *reinterpret_cast<const float4 *>(&mc); // inv_pi_arho, two_m1, row, nel
  a.two_m1 = head.y;
  const int nel = __float_as_int(head.w);

  // normalise direction; here and below each sum of two products says which of them is
  // rounded first, so that the kernel's variants follow the same trajectories bit for bit
  {
    const float s = rsqrtf(fmaf(p.dz, p.dz, fmaf(p.dy, p.dy, p.dx * p.dx)));
    p.dx *= s;
    p.dy *= s;
    p.dz *= s;
  }
  const float E = p.E;

  // electronic stopping (material.C:114-121) and maximum impact parameter
  // (trim.C:88-94) from the table; the formula below its first point
  float S, pmax;
  if (!stop_lookup(t.stop + size_t(__float_as_uint(head.z)) * STOP_N, t.lnE_min, t.inv_dlnE, E, S, pmax))
  {
    const float eeg = sqrtf(E * mc.f * mc.epsdg);
    pmax = mc.a / (eeg + sqrtf(eeg) + 0.125f * __expf(0.1f * __logf(eeg)));
  }
  // free flight (trim.C:88-94); the first one's draw comes from the key's bits
  float ls = head.x / (pmax * pmax);
  if (ic == 1)
    ls = key_u24f(p.key) * fminf(ls, t.cw);
  a.ls = ls;

  // impact parameter and azimuth from one Philox2x32-10 block per collision; the
  // target atom of a multi-element material from a second block whose counter is
  // the member key with its top bit flipped
  const U2 d = draw_pair(p.key, ic, k0, k1);
  a.azimuth = d.y;
  const float pimp = pmax * sqrtf(u24f(d.x));
  int nn = 0;
  if (nel > 1)
  {
    float hh = u24f(draw_pair(p.key ^ 0x8000000000000000ull, ic, k0, k1).x);
    for (; nn < nel - 1; ++nn)
    {
      hh -= mc.t[nn];
      if (hh <= 0.0f)
        break;
    }
  }
  a.nn = nn;
  const float4 e = reinterpret_cast<const float4 *>(mc.el + nn)[0]; // fi, inv_ai, ec, my
  a.el = reinterpret_cast<const float4 *>(mc.el + nn)[1];
  a.eps = e.x * E;
  a.b = pimp * e.y;
  a.ec = e.z;
  a.my = e.w;

  // electronic loss
  a.dee = ls * S;
  return a;
}

// The energy transfer and everything after it (trim.C:275-411).  Returns the collision
// flags; `state` is what the member came to rest as (ST_MOVING while it has not).  A
// displaced recoil to follow (CF_PUSH) is left in `rec`; its vacancy or replacement is
// counted by the lane that starts it (LaneSink::displaced), `vac` says which it is.
template <bool ONE, class Sink>
__device__ __forceinline__ int
phase_b32(P32 & p, const PhaseA32 & a, const Sim32 & sim, const Tables32 & t, const MatCold32 * cold, float s2,
          float c2, Recoil32 & rec, bool & vac, int & state, Sink & sink)
{
  const MatCold32 & mc = cold[a.mat];
  auto target = [&]() {
    return Target32{mc.Z2[a.nn], mc.m2[a.nn], a.el.x, a.el.z, mc.maz, mc.mam};
  };
  const float E = p.E;
  const float ls = a.ls;
  float dee = a.dee;

  // energy transfer, electronic loss, momenta (trim.C:275-296)
  float den = a.ec * s2 * E;
  {
    float h = p.E, l = p.El;
    ff_sub(h, l, dee);
    const bool all = dee >= E;
    dee = all ? E + p.El : dee;
    p.E = all ? 0.0f : h;
    p.El = all ? 0.0f : l;
  }
  sink.eel(dee, p.x, p.y, p.z);
  const float p1 = sqrtf(a.two_m1 * p.E);
  {
    float h = p.E, l = p.El;
    ff_sub(h, l, den);
    const bool all = den >= p.E;
    den = all ? p.E + p.El : den;
    p.E = all ? 0.0f : h;
    p.El = all ? 0.0f : l;
  }
  const float p2 = sqrtf(a.two_m1 * p.E);

  // recoil at the pre-flight position (trim.C:306-318)
  rec.x = p.x;
  rec.y = p.y;
  rec.z = p.z;
  rec.gen = (p.meta >> META_GEN) + 1u;
  const float fl = (ls - t.tau) * t.flscale;
  p.x = fmaf(p.dx, fl, p.x);
  p.y = fmaf(p.dy, fl, p.y);
  p.z = fmaf(p.dz, fl, p.z);
  const float ox = p.dx, oy = p.dy, oz = p.dz;
  rec.E = den - a.el.x;
  rec.tag = -1; // a new IonBase (ion.C:26)

  // azimuth around the flight direction: orthonormal basis by Duff et al.,
  // "Building an Orthonormal Basis, Revisited" (JCGT 2017)
  const float sgn = copysignf(1.0f, p.dz);
  const float ia = -1.0f / (sgn + p.dz);
  const float bxy = p.dx * p.dy * ia;
  const float ux = 1.0f + sgn * p.dx * p.dx * ia, uy = sgn * bxy, uz = -sgn * p.dx;
  const float vx = bxy, vy = sgn + p.dy * p.dy * ia, vz = -p.dy;
  float sphi, cphi;
  __sincosf(6.283185307179586f * u24f(a.azimuth), &sphi, &cphi);
  const float px = cphi * ux + sphi * vx;
  const float py = cphi * uy + sphi * vy;
  const float pz = cphi * uz + sphi * vz;

  // new direction: cos(psi), sin(psi) of psi = atan2(st, ct + my) (trim.C:336-341)
  const float ct = c2 - s2;
  const float st = 2.0f * sqrtf(s2 * c2);
  const float cy = ct + a.my;
  const float ih = rsqrtf(fmaf(st, st, cy * cy));
  const float cpsi = cy * ih, spsi = st * ih;
  p.dx = p.dx * cpsi + px * spsi;
  p.dy = p.dy * cpsi + py * spsi;
  p.dz = p.dz * cpsi + pz * spsi;
  rec.dx = fmaf(ox, p1, -(p.dx * p2));
  rec.dy = fmaf(oy, p1, -(p.dy * p2));
  rec.dz = fmaf(oz, p1, -(p.dz * p2));

  state = ST_MOVING;
  // CUT boundaries (trim.C:344-352)
  if (!ONE || sim.any_cut)
  {
    bool out;
    if constexpr (ONE)
      out = p.x > sim.cut_hi[0] || p.x < sim.cut_lo[0] || p.y > sim.cut_hi[1] || p.y < sim.cut_lo[1] ||
            p.z > sim.cut_hi[2] || p.z < sim.cut_lo[2];
    else
    {
      const float4 c = *reinterpret_cast<const float4 *>(sim.cut_lo);
      const float2 d = *reinterpret_cast<const float2 *>(sim.cut_hi + 1);
      out = p.x > c.w || p.x < c.x || p.y > d.x || p.y < c.y || p.z > d.y || p.z < c.z;
    }
    if (out)
    {
      sink.lost(p.E + p.El + den, p, mc.Z1, mc.m1);
      return CF_DONE;
    }
  }

  // fate of recoil and projectile (trim.C:357-411)
  int flags = 0;
  float2 fate; // Ef, follow_gen
  if constexpr (!ONE)
    fate = *reinterpret_cast<const float2 *>(&sim.Ef);
  const bool displaced = rec.E > a.el.y;
  vac = p.E > a.el.z;
  sink.enuc(displaced ? a.el.x : den, rec.x, rec.y, rec.z);
  if (displaced)
  {
    const bool follow = int(rec.gen) < (ONE ? sim.follow_gen : __float_as_int(fate.y));
    if constexpr (Sink::EV)
    {
      const Target32 el = target();
      sink.history(p, mc.Z1, mc.m1);
      sink.branch(rec, el, p.key);
      if (follow)
        rec.tag = a.tag; // trim.C:365, after followRecoil's output
      if (vac)
        sink.vacancy_event(rec, el, rec.E, p.key);
      else
        sink.replacement_event(rec, el, rec.E, p.key);
    }
    if (follow)
    {
      sink.member_vacancy(vac);
      flags |= CF_PUSH;
    }
    else
    {
      sink.unfollowed(rec.E);
      if (vac)
        sink.vacancy(rec, target(), rec.E);
      else
        sink.replacement(rec);
      sink.count_bins();
    }
    if (!vac)
      state = __float_as_int(a.el.w) >> 8; // ST_REPLACEMENT, or ST_SUBSTITUTIONAL in another element's place
  }
  else
  {
    if constexpr (Sink::EV)
      sink.dissipate(rec, rec.E, target(), p.key);
    if (p.E < (ONE ? sim.Ef : fate.x))
      state = ST_INTERSTITIAL;
  }
  if (state != ST_MOVING)
  {
    p.E += p.El;
    p.El = 0.0f;
    flags |= CF_DONE;
  }
  else if (!(p.E == p.E))
  {
    sink.numeric();
    flags |= CF_DONE;
  }
  return flags;
}

// resident 128-thread blocks per SM the register budget of each feature level is cut
// for: lean, mid and events 8 (64 registers; 7 measured 1.4 % slower on Ag into Si, 9
// 0.2 % faster there and 10 % slower on the 4096-simulation batch), the others 7 (72; 6
// measured 4.5 % slower on Xe into UO2 with bubbles); the surrogate's tensor-core
// fragments need 128 registers (5 blocks 18 % slower, 3 blocks 8 %)
template <int LVL, bool SURROGATE>
struct Blocks32
{
  static constexpr int value =
      SURROGATE ? 4 : LVL == LVL_LEAN || LVL == LVL_MID || LVL == LVL_EVENTS ? 8 : 7;
};

template <int LVL, bool SURROGATE, bool ONE, bool PACED = false>
__global__ void __launch_bounds__(128, Blocks32<LVL, SURROGATE>::value)
cascade32_kernel(const __grid_constant__ EngineParams prm, const __grid_constant__ Tables32 tabs,
                 const __grid_constant__ One32 one)
{
  constexpr bool MID = LVL >= LVL_MID;
  constexpr bool EXT = level_clusters(LVL);   // the cluster geometry
  constexpr bool POT = level_potentials(LVL); // the Moliere and C-Kr potentials
  using Sink = LaneSink<Sink32, LVL>;
  using Rec = std::conditional_t<Sink::EV, Rec32Tag, Rec32>;
  extern __shared__ __align__(16) unsigned char smem[];
  // recoils sent between warps: with the network only (Ag into Si, 50,000 primaries: 113 ->
  // 99 ms; the exact kernels gain up to 7 % of some runs and lose up to 8 % of others)
  constexpr bool SHARE = SURROGATE;
  if constexpr (SHARE)
    RecoilPool<Rec>::start(prm.pool);

  // per-block vacancy / replacement counters, material rows and the network
  unsigned int * s_hist = reinterpret_cast<unsigned int *>(smem + prm.hist_smem_offset);
  for (int i = threadIdx.x; i < prm.hist_smem_bins; i += blockDim.x)
    s_hist[i] = 0u;
  if (ONE)
    for (int i = threadIdx.x; i < int(sizeof(Mat32) / 16) * prm.n_stage_mats; i += blockDim.x)
      reinterpret_cast<uint4 *>(smem)[i] = reinterpret_cast<const uint4 *>(tabs.mats)[i];
  const SurrogateNet * net = nullptr;
  if (SURROGATE)
  {
    net = reinterpret_cast<const SurrogateNet *>(smem + (ONE ? sizeof(Mat32) * prm.n_stage_mats : 0));
    for (int i = threadIdx.x; i < int(sizeof(SurrogateNet) / 4); i += blockDim.x)
      reinterpret_cast<float *>(const_cast<SurrogateNet *>(net))[i] = reinterpret_cast<const float *>(tabs.net)[i];
  }
  __syncthreads();

  const unsigned int FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned int lt = lanemask_lt();
  const long long warp_id = (long long)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  Rec * stack = reinterpret_cast<Rec *>(prm.stacks) + warp_id * prm.stack_cap;
  long long n_work = prm.total_primaries;
  // members per refill: the launch's choice for fresh primaries; for the records of
  // a drain pass, a quarter of a warp's fair share (at most one per lane)
  int max_take = prm.max_take;
  if (prm.in_records)
  {
    const long long c = (long long)*prm.in_count;
    n_work = c < prm.in_cap ? c : prm.in_cap;
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long share = n_work / (nwarps * 4);
    max_take = share < 1 ? 1 : (share > 32 ? 32 : int(share));
  }

  int top = 0;
  bool work_done = false; // no more primaries / input records for this warp
  bool live = false;
  int fin = -1; // state of a member whose end the lane has yet to tally (ST_MOVING: dropped or lost)
  P32 p;
  p.sim = 0;
  p.tag = -1;
  uint32_t ic = 0;
  const Sim32 * psim = tabs.sims; // the member's simulation, where there are several
  int cur_sim = ONE ? 0 : -1;

  Sink sink;
  sink.cold = reinterpret_cast<LaneCold<AccKahan32> *>(smem + prm.cold_offset) + threadIdx.x;
  sink.cold->vcell = -1;
  sink.cold->vacc = 0.0f;
  sink.cold->evac_bin = -1;
  sink.cold->ev_next = sink.cold->ev_end = 0;
  sink.prm = &prm;
  sink.s_hist = s_hist;
  sink.sim = ONE ? &one.desc : nullptr;
  sink.isim = 0;
  sink.gprim = -1;
  sink.range_mode = ONE ? one.desc.range_mode : 0;
  sink.vox = ONE && MID && prm.voxels != nullptr && one.desc.voxel_n[0] > 0;
  sink.dep_in = false;
  sink.vac_bin = sink.repl_bin = -1;
  sink.reset_prim();
  sink.reset_sim();
  sink.reset_member();

  [[maybe_unused]] RecoilPool<Rec> pool;
  [[maybe_unused]] bool give = false;
  unsigned int steps = 0;
  [[maybe_unused]] unsigned int take_mask = 2u * prm.take_mask + 1u; // halved at the first refill
again:
  while (true)
  {
    ++steps;
    // ---- when refill_min lanes are idle: the ends of their members, then recoils from
    // the warp's stack, then new work (an idle warp always gets here: refill_min <= 32)
    const unsigned int idle = __ballot_sync(FULL, !live);
    const int nidle = __popc(idle);
    if (nidle >= prm.refill_min)
    {
      __syncwarp(); // the recoils other lanes pushed
      const int rank = __popc(idle & lt);
      const int npop = nidle < top ? nidle : top;
      // PACED: a warp that has members takes new work in every (take_mask + 1)th iteration
      // only; where it runs out in between, its cascades are smaller than was thought
      if (PACED && idle == FULL)
        take_mask >>= 1;
      const int need = PACED && (steps & take_mask) && idle != FULL ? 0 : min(nidle - npop, max_take);
      long long base = 0;
      if (need > 0 && !work_done)
      {
        unsigned long long b = 0;
        const int leader = __ffs(idle) - 1;
        if (lane == leader)
          b = atomicAdd(prm.next_primary, (unsigned long long)need);
        base = (long long)__shfl_sync(FULL, b, leader);
      }
      const long long avail = work_done ? 0 : n_work - base; // > 0 only with need > 0, or unused
      if (!live)
      {
        if (fin >= 0)
        {
          // the end of the lane's last member
          sink.a_coll += ic;
          if (fin != ST_MOVING)
          {
            const Sim32 & sim = ONE ? one.sim : *psim;
            const MatCold32 & mc = tabs.cold[(ONE ? 0 : sim.mat_base) + int(p.meta & META_SPECIES) * sim.n_mat];
            sink.stop(fin, p, mc.Z1, mc.m1);
          }
          if (MID && prm.records)
            sink.record(p, ic);
          fin = -1;
        }
        const Rec * src = nullptr;
        bool start = rank < npop;
        const int r = rank - npop;
        if (start)
          src = stack + (top - 1 - rank);
        else if (r < need && r < avail)
        {
          start = true;
          if (prm.in_records)
            src = reinterpret_cast<const Rec *>(prm.in_records) + (base + r);
        }
        if (start)
        {
          uint32_t meta;
          if (src)
          {
            const float4 a = src->a, b = src->b;
            const uint4 c = src->c;
            p.x = a.x;
            p.y = a.y;
            p.z = a.z;
            p.E = a.w;
            const float s = rsqrtf(fmaf(b.z, b.z, fmaf(b.x, b.x, b.y * b.y)));
            p.dx = b.x * s;
            p.dy = b.y * s;
            p.dz = b.z * s;
            p.prim = __float_as_uint(b.w);
            p.El = 0.0f;
            p.key = mix64(uint64_t(c.y) << 32 | c.x);
            meta = c.z;
            p.meta = meta & ~META_VACANCY;
            if (!ONE)
              p.sim = int(c.w);
            if constexpr (Sink::EV)
              p.tag = int(src->d.x);
          }
          else
          {
            long long g = base + r, first = 0;
            const int s = !ONE && prm.n_sims > 1 ? find_sim(prm, g, first) : 0;
            const SimDesc & d = ONE ? one.desc : prm.sims[s];
            g += d.prim_begin - first;
            p.x = float(d.pos[0]);
            p.y = float(d.pos[1]);
            p.z = float(d.pos[2]);
            p.dx = float(d.dir[0]);
            p.dy = float(d.dir[1]);
            p.dz = float(d.dir[2]);
            p.E = float(d.E0);
            p.El = float(d.E0 - double(p.E));
            p.key = root_key(d.sim_key, uint64_t(g - d.prim_begin + d.key_offset));
            p.prim = uint32_t(g);
            meta = p.meta = 0u;
            if (!ONE)
              p.sim = s;
            p.tag = -1;
          }
          if (!ONE && p.sim != cur_sim)
          {
            sink.flush_prim();
            sink.flush_sim(cur_sim);
            cur_sim = p.sim;
            sink.sim = prm.sims + cur_sim;
            sink.isim = cur_sim;
            sink.range_mode = sink.sim->range_mode;
            sink.vox = MID && prm.voxels != nullptr && sink.sim->voxel_n[0] > 0;
            sink.gprim = -1;
            psim = tabs.sims + cur_sim;
          }
          if ((long long)p.prim != sink.gprim)
          {
            sink.flush_prim();
            sink.gprim = (long long)p.prim;
            if (sink.n_newton > 0x40000000u)
              sink.flush_sim(cur_sim);
          }
          if (src)
            sink.displaced((meta & META_VACANCY) != 0, p.x, p.E);
          if constexpr (Sink::EV)
          {
            // IonMDTag: the demo programs' MD-gap mark, taken when the member starts
            // (apps/mytrim_solid.C:156-159); a spawned recoil's _md is 0 (ion.C:88-93)
            const Sim32 & sim = ONE ? one.sim : *psim;
            const MatCold32 & mc = tabs.cold[(ONE ? 0 : sim.mat_base) + int(p.meta & META_SPECIES) * sim.n_mat];
            const SimDesc & d = *sink.sim;
            sink.cold->m_md = (d.md_Z != 0 && mc.Z1 == d.md_Z && p.E > d.md_Emin_f && p.E < d.md_Emax_f) ? 1 : 0;
          }
          sink.reset_member();
          ++sink.cold->n_members;
          ic = 0;
          live = true;
        }
      }
      top -= npop;
      if (avail <= need)
        work_done = true;
      __syncwarp(); // popped before another lane pushes into the same place
      if (__ballot_sync(FULL, live) == 0)
        break;
    }

    // ---- one collision per live lane
    const Sim32 & sim = ONE ? one.sim : *psim;
    Recoil32 rec;
    bool vac = false;
    int flags = 0, niter = 0;
    PhaseA32 a;
    float s2, c2;
    if (live)
    {
      ++ic;
      a = phase_a32<EXT, ONE>(p, ic, sim, ONE ? reinterpret_cast<const Mat32 *>(smem) : tabs.mats, tabs, prm.k0,
                              prm.k1);
    }
    if constexpr (SURROGATE)
    {
      // warp-collective: the lanes whose collision is in the network's domain are
      // evaluated together, the others (no member, or the exact fallback) only take
      // part in the shuffles; the network is trained on the universal potential only
      const bool nn = live && !a.gone && (!POT || sim.potential == 0) && surrogate_in_domain(a.eps, a.b);
      const float o0 = surrogate_eval_warp(net, nn, nn ? surrogate_x1(a.eps) : 0.0f, nn ? surrogate_x2(a.b) : 0.0f);
      if (live && !a.gone)
      {
        if (nn)
          surrogate_s2_from(a.eps, a.b, o0, s2, c2);
        else
        {
          sink.fallback();
          scatter32(a.eps, a.b, s2, c2, niter, POT ? sim.potential : 0);
        }
      }
    }
    if (live)
    {
      int state = ST_MOVING;
      if (EXT && a.gone)
      {
        --sink.a_coll; // dropped without a collision (no checkPKAState), which its record counts
        flags = CF_DONE;
      }
      else
      {
        if constexpr (!SURROGATE)
          scatter32(a.eps, a.b, s2, c2, niter, POT ? sim.potential : 0);
        sink.newton(niter);
        flags = phase_b32<ONE>(p, a, sim, tabs, tabs.cold + (ONE ? 0 : sim.mat_base), s2, c2, rec, vac, state, sink);
        if (!(flags & CF_DONE) && ic >= prm.max_collisions)
        {
          atomicOr(prm.error_flags, ERRB_BUDGET);
          flags |= CF_DONE;
        }
      }
      if (flags & CF_DONE)
      {
        live = false;
        fin = state;
      }
    }

    // ---- push displaced recoils onto the warp stack
    const bool push = (flags & CF_PUSH) != 0;
    const unsigned int pm = __ballot_sync(FULL, push);
    if (pm)
    {
      if (push)
      {
        const uint64_t key = p.key + 0x9E3779B97F4A7C15ull * uint64_t(ic); // child_key before its mixer
        const uint32_t meta = rec.gen << META_GEN | (vac ? META_VACANCY : 0u) | (__float_as_uint(a.el.w) & 0xffu);
        Rec q;
        q.a = make_float4(rec.x, rec.y, rec.z, rec.E);
        q.b = make_float4(rec.dx, rec.dy, rec.dz, __uint_as_float(p.prim));
        q.c = make_uint4(uint32_t(key), uint32_t(key >> 32), meta, uint32_t(p.sim));
        if constexpr (Sink::EV)
          q.d = make_uint4(uint32_t(rec.tag), 0u, 0u, 0u);
        const int slot = top + __popc(pm & lt);
        if (slot < prm.stack_cap)
          stack[slot] = q;
        else
        {
          const unsigned long long o = atomicAdd(prm.overflow_count, 1ull);
          if ((long long)o < prm.overflow_cap)
            reinterpret_cast<Rec *>(prm.overflow)[o] = q;
          else
            atomicOr(prm.error_flags, ERRB_QUEUE_FULL);
        }
      }
      top = min(top + __popc(pm), prm.stack_cap);
    }
    if ((steps & 63u) == 0u)
      sink.hand_over();
    if constexpr (SHARE)
      if (((steps + (unsigned int)warp_id) & 7u) == 0u && pool.wanted(prm, top))
      {
        give = true;
        break;
      }
  }
  if constexpr (SHARE)
  {
    // outside the loop, so that its code stays together (inside it 104 ms)
    if (give)
    {
      give = false;
      top = pool.send(prm, stack, top, lane);
      goto again;
    }
    if ((top = pool.wait(prm, (unsigned int)warp_id, stack, lane)) != 0)
    {
      --steps; // the pass that found no work
      goto again;
    }
  }
  sink.flush_prim();
  sink.flush_sim(cur_sim);
  sink.flush_voxel();
  sink.flush_events();
  if (prm.hist_smem_bins)
  {
    // every warp of the block has left its loop: add the block's counts
    __syncthreads();
    for (int i = threadIdx.x; i < prm.hist_smem_bins; i += blockDim.x)
      if (s_hist[i])
        atomicAdd(prm.hist + prm.hist_smem_base + i, (unsigned long long)s_hist[i]);
  }
  if (lane == 0)
    atomicAdd(prm.warp_steps, (unsigned long long)(steps - 1)); // the last pass finds no work
}

} // namespace mtg
