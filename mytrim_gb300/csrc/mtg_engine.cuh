// Persistent, warp-cooperative cascade kernel.
//
// The reference follows one cascade with a host FIFO: pop a member, run
// TrimBase::trim on it until it stops, push every recoil it displaces
// (apps/runmytrim.C:71-93, trim.C:369).  Here every lane of a warp holds one
// cascade member in registers and the 32 lanes advance one collision per loop
// iteration.  Each warp owns a LIFO recoil stack in HBM:
//   * a lane whose member came to rest pops the next recoil from its warp's
//     stack (warp-synchronous ballot + prefix count, no atomics);
//   * with the stack empty, idle lanes take fresh primaries from one global
//     counter (one atomicAdd per warp refill);
//   * recoils are pushed with a ballot + prefix count; a full stack spills into
//     a global overflow list that a follow-up launch drains.
// In the FP64 and surrogate kernels a busy warp sends recoils to warps that have run
// out (RecoilPool); the only wait in them is an idle warp's, for 20 ms of sleep and, for
// recoils already on their way to it, another 20 at most.  Every loop is bounded
// (collisions per member, Newton iterations, rejection passes).  The single-precision
// kernel is in mtg_cascade32.cuh; it shares the tallies and parameters.
//
// Random numbers are keyed by the member's path key and collision index, so the
// result does not depend on which lane or warp ran which member.
//
// Tallies: per-lane accumulators flushed to per-primary arrays when a lane
// switches primary (vacancies, collisions, electronic and nuclear energy), the
// primary's stopping point written once, depth histograms through per-lane
// atomics, per-simulation counters flushed once per lane.
#pragma once

#include <type_traits>

#include "mtg_tables.h"
#include "mtg_common.cuh"

namespace mtg
{

struct PrimaryTallies
{
  unsigned long long * vac;  // vacancies (KP count in range mode)
  unsigned long long * coll; // collisions
  double * eel;              // electronic loss [eV]
  double * enuc;             // nuclear (phonon) deposit [eV]
  double * fx;               // stopping point of the primary (generation 0)
  double * fy;
  double * fz;
  int * fstate;              // final state of the primary, 0 if lost / not stopped
};

struct MemberRecord
{
  uint64_t key;
  int sim, species, gen, state;
  unsigned int ncoll, nvac;
  double E, x, y, z, eel;
};

struct EngineParams
{
  const SimDesc * sims;
  int n_sims;
  // the order in which the simulations' primaries are started: simulation order[i] has
  // the work indexes from order_end[i - 1] to order_end[i]
  const int * order;
  const long long * order_end;
  const SpeciesConst * species;
  const MatConst * mats;
  int stage_tables;               // stage species+mats of simulation 0 into shared memory
  int n_stage_species, n_stage_mats;
  long long total_primaries;
  unsigned long long * next_primary;
  // drain mode: members read from `in_records` (count in device memory) instead
  // of fresh primaries
  const void * in_records;
  const unsigned long long * in_count;
  long long in_cap;
  // per-warp stacks and overflow list
  void * stacks;
  int stack_cap;
  void * overflow;
  unsigned long long * overflow_count;
  long long overflow_cap;
  // tallies
  PrimaryTallies prim;
  SimTotals * totals;
  unsigned long long * hist; // all histograms, per-simulation bases in SimDesc
  double * voxels;           // energy-deposition voxels of all simulations (may be NULL):
                             // FP64 sums in global memory (L2 atomics), fed by each lane's
                             // short FP32 run of deposits into one cell
  unsigned int * error_flags;
  uint32_t k0, k1;
  unsigned int max_collisions; // per member
  int max_take;                // fresh primaries one warp takes per refill (load balance)
  unsigned int take_mask;      // iterations between two refills with new work, less one (2^k - 1);
                               // 0: no pace (FP32 engine)
  int refill_min;              // idle lanes a warp waits for before refilling them
  int cold_offset;             // byte offset of the per-thread LaneCold slots in dynamic shared memory
  // optional per-member records (replay checks)
  MemberRecord * records;
  unsigned long long * n_records;
  long long records_cap;
  // optional event log (mask bit k selects EventKind k; 0 = off)
  EventRec * events;
  unsigned long long * n_events;       // slots reserved
  unsigned long long * n_event_unused; // reserved slots that no event filled
  long long events_cap;
  int event_chunk;                     // slots a lane reserves at a time (1, 8 or 16)
  unsigned int event_mask;
  int any_evac; // some simulation keeps a vacancy-energy histogram
  int level;    // KernelLevel of the launched variant
  unsigned long long * warp_steps; // loop iterations of all warps (lane occupancy = collisions / 32 steps)
  // single-simulation runs with few depth bins count vacancies and replacements in
  // a per-block shared-memory histogram (hist_smem_bins counters from byte offset
  // hist_smem_offset), added to the global one when the block ends; 0 = global atomics
  int hist_smem_bins;
  int hist_smem_offset;
  long long hist_smem_base; // global index of shared bin 0
  // recoils that busy warps give to idle ones (RecoilPool): counts, ring, a mailbox and
  // 32 records per warp; what a launch's ring entries are told by; the least energy sent
  struct PoolControl * pool;
  unsigned long long * pool_ring;
  unsigned int * pool_box;
  void * pool_recs;
  unsigned int pool_nonce;
  float share_min; // eV
  int share_after; // and only while more warps than this wait
};

// Recoils that busy warps give to idle ones.
//
// A warp owns the cascades it started, and at the end of a run, or in a run of fewer
// primaries than warps, most warps have none left while a few still have hundreds of
// recoils on their stacks.  An idle warp enters its number in a ring and watches its own
// mailbox; a busy warp looks every eighth iteration (FP64: every fourth) how many wait (at
// the count it loaded the time before, so that it does not wait for it) and, while any do,
// sends one of them the older half of its stack, 32 recoils at most, if they hold enough
// energy to be worth the move (share_min): a mailbox per warp, because a common list of
// chunks that all idle warps watched was slower by a factor of a hundred than no sharing
// at all.
//
// The notes are single releasing stores: a fence (__threadfence) also empties the SM's L1,
// from which all its warps read their tables, and is left to the receipt of a letter.
//
// Nothing here depends on another warp's progress but the last step of a letter, between
// a sender's claim of a mailbox and its note that the recoils are in it.  An idle warp
// leaves when all others that have started are idle or gone, or after PATIENCE ns; it gives
// up its mailbox first, by a compare-and-swap that fails if a sender has claimed it.  Then
// it waits for that letter, PATIENCE ns more at most (ERRB_LOST_LETTER: the run is made
// again).  (A grid need not be resident as a whole: another stream's kernel may hold a
// part of the SMs.  An idle warp finds all work taken, by warps that have started, so those
// that have not bring none.)
//
// FP64 kernel, Ag 200 keV into Si: 64 primaries 55 -> 42 ms, 1000 107 -> 87 ms, 2000
// 153 -> 139 ms.  With the network, 50,000 Ag 113 -> 100 ms.  The exact FP32 kernel goes
// without: a warp's iteration takes it 2 us instead of 30 and more, a letter 7; 10^4 Au
// 1 MeV with voxels gained 8 % and Xe into bubbles 6, 10^4 Cu 100 keV lost 14 %, 10^6 B 7
// and the 4096-simulation batch 12.
struct PoolControl
{
  unsigned int hungry; // warps waiting
  int active;          // warps that have started and neither wait nor left
  unsigned int pad0[30];
  int avail; // entries of the ring that no sender has taken
  unsigned int pad1[31];
  unsigned int head;
  unsigned int pad2[31];
  unsigned int tail;
  unsigned int pad3[31];
};

template <class Rec>
struct RecoilPool
{
  static constexpr int NO_SHARING = 0x7fffffff; // EngineParams::share_after
  static constexpr unsigned int PATIENCE = 20000000u;
  static constexpr unsigned int WAITING = 1u, CLAIMED = 2u, LEFT = 3u, FULL = 0x100u; // mailbox states; FULL + records
  static constexpr int RING_BITS = 14; // more entries than the GPU holds warps
  static constexpr unsigned int RING = 1u << RING_BITS;

  int avail = 0; // as last looked at

  static __device__ __forceinline__ unsigned int tag(const EngineParams & prm, unsigned int ticket)
  {
    return (prm.pool_nonce << 10) ^ (ticket >> RING_BITS);
  }

  // a block's first step, before it takes work; a call, because inlined it moves the hot
  // loop's registers (50,000 Ag with the network 100.9 -> 102.3 ms)
  static __device__ __noinline__ void start(PoolControl * ctl)
  {
    if (threadIdx.x == 0)
      atomicAdd(&ctl->active, int(blockDim.x >> 5));
  }

  // an idle warp waits for recoils (all lanes) and puts them on its empty stack; their
  // number, 0: none will come
  static __device__ __forceinline__ int wait(const EngineParams & prm, unsigned int warp, Rec * stack, int lane)
  {
    if (prm.share_after == NO_SHARING)
      return 0;
    unsigned int k = 0;
    if (lane == 0)
    {
      PoolControl * ctl = prm.pool;
      unsigned int * box = prm.pool_box + warp;
      const volatile unsigned int * vbox = box;
      *reinterpret_cast<volatile unsigned int *>(box) = WAITING;
      atomicAdd(&ctl->hungry, 1u);
      atomicSub(&ctl->active, 1);
      const unsigned int t = atomicAdd(&ctl->tail, 1u);
      asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(prm.pool_ring + (t & (RING - 1))),
                   "l"((unsigned long long)tag(prm, t) << 32 | (warp + 1u))
                   : "memory");
      int before;
      asm volatile("atom.add.release.gpu.global.s32 %0, [%1], 1;" : "=r"(before) : "l"(&ctl->avail) : "memory");
      unsigned int slept = 0, limit = PATIENCE;
      bool claimed = false;
      for (int i = 0; i < (1 << 20); ++i)
      {
        const unsigned int f = *vbox;
        if (f >= FULL)
        {
          k = f - FULL;
          break;
        }
        unsigned int ns = 200u;
        if (!claimed)
        {
          unsigned int hungry;
          int active;
          asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(hungry), "=r"(active) : "l"(ctl) : "memory");
          if (active <= 0 || slept >= limit)
          {
            if (atomicCAS(box, WAITING, LEFT) == WAITING)
              break;
            claimed = true; // a sender is about to fill it
            limit = slept + PATIENCE;
          }
          ns = min(max(500u, hungry * 2u), 10000u);
        }
        else if (slept >= limit)
          break;
        __nanosleep(ns);
        slept += ns;
      }
      if (k == 0u)
      {
        if (claimed)
          atomicOr(prm.error_flags, ERRB_LOST_LETTER);
      }
      else
      {
        atomicAdd(&ctl->active, 1);
        __threadfence(); // the letter's recoils after its note
      }
      atomicSub(&ctl->hungry, 1u);
    }
    k = __shfl_sync(0xffffffffu, k, 0);
    __syncwarp();
    if (lane < int(k))
    {
      // past L1, which may hold what the mailbox held before
      using Unit = std::conditional_t<sizeof(Rec) % 16 == 0, uint4, uint2>;
      const Unit * from =
          reinterpret_cast<const Unit *>(reinterpret_cast<const Rec *>(prm.pool_recs) + (warp * 32 + lane));
#pragma unroll
      for (int i = 0; i < int(sizeof(Rec) / sizeof(Unit)); ++i)
        reinterpret_cast<Unit *>(stack + lane)[i] = __ldcg(from + i);
    }
    __syncwarp();
    return int(k);
  }

  // a busy warp's look at who waits: whether to send recoils to one of them
  __device__ __forceinline__ bool wanted(const EngineParams & prm, int top)
  {
    // lane 0's value for all: the lanes need not have loaded the same one
    const bool give = top > 0 && __shfl_sync(0xffffffffu, avail, 0) > prm.share_after;
    asm volatile("ld.volatile.global.b32 %0, [%1];" : "=r"(avail) : "l"(&prm.pool->avail));
    return give;
  }
  // the stack's new top
  static __device__ __forceinline__ int send(const EngineParams & prm, Rec * stack, int top, int lane)
  {
    __syncwarp();
    const int k = min(32, (top + 1) / 2); // the oldest k go
    const int m = min(k, top - k);        // the newest m take their places
    float e = lane < k ? record_energy(stack[lane]) : 0.0f;
    for (int w = 16; w > 0; w >>= 1)
      e += __shfl_xor_sync(0xffffffffu, e, w);
    int to = -1;
    if (lane == 0 && e >= prm.share_min)
    {
      PoolControl * ctl = prm.pool;
      for (int i = 0; i < 4 && to < 0; ++i)
      {
        if (atomicSub(&ctl->avail, 1) <= 0)
        {
          atomicAdd(&ctl->avail, 1);
          break;
        }
        const unsigned int t = atomicAdd(&ctl->head, 1u);
        const volatile unsigned long long * slot = prm.pool_ring + (t & (RING - 1));
        for (int j = 0; j < 64 && to < 0; ++j)
        {
          const unsigned long long q = *slot;
          if ((unsigned int)(q >> 32) == tag(prm, t))
            to = int((unsigned int)q) - 1;
        }
        if (to >= int(gridDim.x * (blockDim.x >> 5)) || (to >= 0 && atomicCAS(prm.pool_box + to, WAITING, CLAIMED) != WAITING))
          to = -1;
      }
    }
    to = __shfl_sync(0xffffffffu, to, 0);
    if (to < 0)
      return top;
    if (lane < k)
      reinterpret_cast<Rec *>(prm.pool_recs)[to * 32 + lane] = stack[lane];
    __syncwarp();
    if (lane == 0)
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(prm.pool_box + to), "r"(FULL + (unsigned int)k)
                   : "memory");
    if (lane < m)
      stack[lane] = stack[top - m + lane];
    __syncwarp();
    return top - k;
  }
};

// largest vacancy + replacement histogram counted in shared memory (u32 counters)
constexpr int HIST_SMEM_MAX = 2048;

__device__ __forceinline__ unsigned int
lanemask_lt()
{
  unsigned int m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// the simulation of work index g; `first`: its first work index
__device__ __forceinline__ int
find_sim(const EngineParams & prm, long long g, long long & first)
{
  const long long * ends = prm.order_end;
  const int n = prm.n_sims;
  int lo = 0, hi = n - 1;
  while (lo < hi)
  {
    const int mid = (lo + hi) >> 1;
    if (g < ends[mid])
      hi = mid;
    else
      lo = mid + 1;
  }
  first = lo > 0 ? ends[lo - 1] : 0;
  return prm.order[lo];
}

// Plain FP64 accumulator (FP64 engine)
struct AccF64
{
  double s;
  __device__ void reset() { s = 0.0; }
  __device__ void add(double x) { s += x; }
  __device__ double value() const { return s; }
  __device__ bool nonzero() const { return s != 0.0; }
  __device__ void atomic_add_to(double * dst) const { atomicAdd(dst, s); }
};

// float -> double by exponent rebias on the bit pattern (no FP64 instruction; the
// FP32 engine flushes denormals, so a zero exponent means zero)
__device__ __forceinline__ double
widen_f32(float f)
{
  const uint32_t u = __float_as_uint(f);
  const uint32_t e = (u >> 23) & 0xffu;
  if (e == 0u)
    return 0.0;
  const unsigned long long bits = ((unsigned long long)(u >> 31) << 63) | ((unsigned long long)(e + 896u) << 52) |
                                  ((unsigned long long)(u & 0x7fffffu) << 29);
  return __longlong_as_double((long long)bits);
}

// Plain FP32 accumulator for the per-collision energy sums of the FP32 engine;
// the engine hands it to the FP64 per-primary arrays every 64 iterations
// (LaneSink::hand_over), so each float sum stays short and accurate to ~1e-7
struct AccF32
{
  float s;
  __device__ void reset() { s = 0.0f; }
  __device__ void add(float x) { s += x; }
  __device__ double value() const { return double(s); }
  __device__ bool nonzero() const { return s != 0.0f; }
  __device__ void atomic_add_to(double * dst) const { atomicAdd(dst, widen_f32(s)); }
};

// Kahan-compensated FP32 accumulator (FP32 engine, long-lived rare sums): keeps
// FP64 work out of the engine.  The error of a compensated sum is bounded by about
// 2u sum|x_i| (u = 2^-24, so ~1.2e-7 of the summed magnitudes) independent of the
// number of terms, where a plain FP32 sum grows as n u sum|x_i|.
struct AccKahan32
{
  float s, c;
  __device__ void reset() { s = c = 0.0f; }
  __device__ void add(float x)
  {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ double value() const { return double(s) - double(c); }
  __device__ bool nonzero() const { return s != 0.0f; }
  // add the sum to a double in global memory without FP64 instructions
  __device__ void atomic_add_to(double * dst) const
  {
    atomicAdd(dst, widen_f32(s));
    if (c != 0.0f)
      atomicAdd(dst, widen_f32(-c));
  }
};

// Rarely-updated tally state of one lane, kept in a per-thread slot of shared
// memory instead of registers (the collision loop needs its registers).
template <class Acc>
struct LaneCold
{
  unsigned int n_rest[4]; // members come to rest, by state; each replacement or substitution is one replacement event
  unsigned int n_lost, n_members, n_passes, n_fallbacks, n_sput, n_back;
  unsigned int m_vac;
  int m_state;
  unsigned int n_dropped; // depth-histogram events beyond the last bin
  Acc e_lost, e_unf, e_sput, m_eel;
  long long vcell; // pending voxel deposit: cell and value
  float vacc;
  int m_md;        // IonMDTag::_md of the lane's member (event-logging levels)
  int evac_bin;    // vacancy-energy bin of the current collision (-1 = none)
  unsigned int ev_next, ev_end; // the lane's reserved event-log slots [ev_next, ev_end)
};

// Kernel feature levels.  Code for a feature a run does not use still costs the
// collision loop (instruction fetch, registers), so the cascade kernel comes in
// up to seven variants and each run takes the smallest that has what it needs:
//   LVL_LEAN    layered samples, universal potential, TrimVacCount tallies (depth,
//               range and lateral histograms), CUT boundaries and sputter counting;
//   LVL_MID     + member records, deposition voxels, the vacancy-energy histogram,
//               TrimRange / TrimPrimaries tally modes;
//   LVL_EVENTS  LVL_MID + the event log (no cluster geometry, universal potential);
//   LVL_GEO     LVL_MID + the cluster geometry, the Moliere and C-Kr potentials;
//   LVL_FULL    LVL_GEO + the event log;
//   LVL_CLU     LVL_MID + the cluster geometry, universal potential only (the plain
//               FP32 engine; the others run LVL_GEO);
//   LVL_CLU_EV  LVL_CLU + the event log (the others run LVL_FULL).
enum KernelLevel : int
{
  LVL_LEAN = 0,
  LVL_MID = 1,
  LVL_EVENTS = 2,
  LVL_GEO = 3,
  LVL_FULL = 4,
  LVL_CLU = 5,
  LVL_CLU_EV = 6,
  LVL_COUNT = 7
};

// the level's cluster geometry, its non-universal potentials, its event log
MTG_HD constexpr bool
level_clusters(int lvl)
{
  return lvl == LVL_GEO || lvl == LVL_FULL || lvl == LVL_CLU || lvl == LVL_CLU_EV;
}
MTG_HD constexpr bool
level_potentials(int lvl)
{
  return lvl == LVL_GEO || lvl == LVL_FULL;
}
MTG_HD constexpr bool
level_events(int lvl)
{
  return lvl == LVL_EVENTS || lvl == LVL_FULL || lvl == LVL_CLU_EV;
}

// the single-precision kernel's tallies (mtg_cascade32.cuh)
struct Sink32
{
  using Acc = AccKahan32;
  using AccHot = AccF32;
  using Real = float;
};

// generation and species of a member (a kernel that packs them overloads these)
template <class P>
__device__ __forceinline__ int
member_gen(const P & p)
{
  return p.gen;
}
template <class P>
__device__ __forceinline__ int
member_species(const P & p)
{
  return p.species;
}

// Device tally sink for one lane of a kernel of level LVL.
template <class Pol, int LVL>
struct LaneSink
{
  static constexpr bool EV = level_events(LVL); // feeds the event log
  static constexpr bool MID = LVL >= LVL_MID;
  using Acc = typename Pol::Acc;       // rare sums (kept in shared memory)
  using AccHot = typename Pol::AccHot; // per-collision sums (registers)
  using Real = typename Pol::Real;
  LaneCold<Acc> * cold;
  const EngineParams * prm;
  unsigned int * s_hist; // the block's vacancy and replacement counters (prm->hist_smem_bins of them)
  const SimDesc * sim;
  int isim;            // its index
  long long gprim;     // global primary index of the current member
  int range_mode;
  // per-primary accumulators
  unsigned int a_vac, a_coll;
  AccHot a_eel, a_enuc;
  // per-simulation Newton-iteration count (every collision), the rest in `cold`
  unsigned int n_newton;
  bool vox;  // this simulation tallies energy deposition in voxels
  bool dep_in; // the last deposit's point lies in the voxel box (its cell is pending)
  // events of the current collision, aggregated per warp after it
  int vac_bin, repl_bin;

  __device__ void reset_sim()
  {
    LaneCold<Acc> & c = *cold;
    c.n_rest[ST_REPLACEMENT] = c.n_rest[ST_SUBSTITUTIONAL] = c.n_rest[ST_INTERSTITIAL] = 0;
    c.n_lost = c.n_members = c.n_passes = c.n_fallbacks = 0;
    c.n_sput = c.n_back = c.n_dropped = 0;
    n_newton = 0;
    c.e_lost.reset();
    c.e_unf.reset();
    c.e_sput.reset();
  }
  // when the lane leaves the kernel: its reserved slots that no event filled are
  // marked unused (the host skips them) and counted
  __device__ void flush_events()
  {
    if constexpr (EV)
    {
      LaneCold<Acc> & c = *cold;
      if (c.ev_end > c.ev_next)
      {
        atomicAdd(prm->n_event_unused, (unsigned long long)(c.ev_end - c.ev_next));
        for (unsigned int s = c.ev_next; s < c.ev_end && (long long)s < prm->events_cap; ++s)
          prm->events[s].kind = EV_UNUSED;
      }
      c.ev_next = c.ev_end = 0;
    }
  }
  // per-member summaries feed the optional member records only
  __device__ void reset_member()
  {
    if (!MID || !prm->records)
      return;
    cold->m_vac = 0;
    cold->m_state = 0;
    cold->m_eel.reset();
  }
  __device__ void reset_prim()
  {
    a_vac = a_coll = 0;
    a_eel.reset();
    a_enuc.reset();
  }

  // ---- event log (opt-in): one entry per selected hook call
  __device__ void event(int kind, Real x, Real y, Real z, Real E, int Z, Real m, int gen, int state, Real aux,
                        uint64_t key, int tag, int md = 0)
  {
    if (!(prm->event_mask & (1u << kind)))
      return;
    // a lane takes its slots event_chunk at a time: the atomic that reserves them
    // returns through L2, and the lane waits for it before writing the record
    LaneCold<Acc> & c = *cold;
    if (c.ev_next == c.ev_end)
    {
      // slot indexes fit 32 bits: a log of 2^32 88-byte records exceeds the device
      // memory; the reservation saturates there once a full log keeps reserving
      const unsigned long long base = atomicAdd(prm->n_events, (unsigned long long)prm->event_chunk);
      c.ev_next = base < 0xfffffff0ull ? (unsigned int)base : 0xfffffff0u;
      c.ev_end = c.ev_next + (unsigned int)prm->event_chunk;
    }
    const unsigned int slot = c.ev_next++;
    if ((long long)slot >= prm->events_cap)
    {
      atomicOr(prm->error_flags, ERRB_EVENTS_FULL);
      return;
    }
    EventRec & r = prm->events[slot];
    r.x = double(x);
    r.y = double(y);
    r.z = double(z);
    r.E = double(E);
    r.aux = double(aux);
    r.key = key;
    r.primary = gprim - sim->prim_begin + sim->key_offset;
    r.sim = isim;
    r.kind = kind;
    r.Z = Z;
    r.m = double(m);
    r.gen = gen;
    r.state = state;
    r.tag = tag;
    r.md = md;
  }
  // TrimHistory::followRecoil (trim.h:146-150): the moving atom's position (after
  // its flight, trim.C:310) at each displaced recoil
  template <class P>
  __device__ void history(const P & p, int Z1, Real m1)
  {
    if constexpr (EV)
      event(EV_HISTORY, Real(p.x), Real(p.y), Real(p.z), Real(p.E), Z1, m1, member_gen(p), 0, Real(0), p.key,
            p.tag, cold->m_md);
  }
  // followRecoil (trim.C:362): a displaced recoil, followed or not
  template <class R, class E>
  __device__ void branch(const R & rec, const E & el, uint64_t key)
  {
    if constexpr (EV)
      event(EV_BRANCH, Real(rec.x), Real(rec.y), Real(rec.z), Real(rec.E), el.Z2, Real(el.m2), rec.gen, 0,
            Real(el.Elbind), key, rec.tag);
  }
  // dissipateRecoilEnergy (trim.C:397-401): a recoil below the displacement energy
  template <class R, class E>
  __device__ void dissipate(const R & rec, Real Erec, const E & el, uint64_t key)
  {
    if constexpr (EV)
      event(EV_DISSIPATE, Real(rec.x), Real(rec.y), Real(rec.z), Erec, el.Z2, Real(el.m2), rec.gen, 0,
            Real(el.Elbind), key, rec.tag);
  }

  // ---- events raised by the collision code (the reference's hooks, trim.h:72-84)
  // energy-deposition voxel tally (extension): one float atomic per deposit
  __device__ void deposit(Real x, Real y, Real z, Real e)
  {
    if (!MID || !vox)
      return;
    const int ix = int(floorf(float(x - Real(sim->voxel_origin[0])) * sim->voxel_inv_cell[0]));
    const int iy = int(floorf(float(y - Real(sim->voxel_origin[1])) * sim->voxel_inv_cell[1]));
    const int iz = int(floorf(float(z - Real(sim->voxel_origin[2])) * sim->voxel_inv_cell[2]));
    dep_in = false;
    if (ix < 0 || iy < 0 || iz < 0 || ix >= sim->voxel_n[0] || iy >= sim->voxel_n[1] || iz >= sim->voxel_n[2])
      return;
    dep_in = true;
    const long long cell = sim->voxel_base + ((long long)iz * sim->voxel_n[1] + iy) * sim->voxel_n[0] + ix;
    LaneCold<Acc> & c = *cold;
    if (cell == c.vcell)
    {
      c.vacc += float(e);
      return;
    }
    flush_voxel();
    c.vcell = cell;
    c.vacc = float(e);
  }
  __device__ void flush_voxel()
  {
    if constexpr (!MID)
      return;
    LaneCold<Acc> & c = *cold;
    // the lane's run of deposits into one cell is short (FP32 is exact enough for
    // it); the cell's sum over the whole run takes up to ~1e8 of them, which FP32
    // would round away once the sum passes 2^24 deposits' worth, so it is kept in
    // FP64 (the float is widened on its bit pattern, no FP64 instruction here)
    if (c.vcell >= 0)
      atomicAdd(prm->voxels + c.vcell, widen_f32(c.vacc));
    c.vcell = -1;
    c.vacc = 0.0f;
  }

  // electronic loss d over the flight path that starts at (x, y, z)
  __device__ void eel(Real d, Real x, Real y, Real z)
  {
    a_eel.add(d);
    if (MID && prm->records)
      cold->m_eel.add(d);
    deposit(x, y, z, d);
  }
  __device__ void newton(int n) { n_newton += (unsigned int)n; }
  __device__ void passes(int n) { cold->n_passes += (unsigned int)n; }
  __device__ void fallback() { ++cold->n_fallbacks; }
  __device__ void numeric() { atomicOr(prm->error_flags, ERRB_NUMERIC); }
  // nuclear (phonon) deposit e at (x, y, z)
  // The collision code deposits a collision's nuclear loss where it deposited the
  // electronic loss just before (the flight's starting point, which is the recoil's
  // position, trim.C:306-318), so the pending voxel cell is already the right one:
  // the same sum as a full deposit, without recomputing the cell.
  __device__ void enuc(Real e, Real /*x*/, Real /*y*/, Real /*z*/)
  {
    a_enuc.add(e);
    if (MID && vox && dep_in)
      cold->vacc += float(e);
  }
  __device__ void unfollowed(Real e) { cold->e_unf.add(e); }
  // the member left the sample carrying `e` (its own energy plus the recoil dropped
  // with it, trim.C:357); through the entrance surface a recoil counts as sputtered
  // when E cos^2 > E_surf, a primary as backscattered
  template <class P>
  __device__ void lost(Real e, const P & p, int Z1, Real m1)
  {
    LaneCold<Acc> & c = *cold;
    if constexpr (EV)
      event(EV_LOST, Real(p.x), Real(p.y), Real(p.z), Real(p.E), Z1, m1, member_gen(p), ST_LOST, e - Real(p.E),
            p.key, p.tag, cold->m_md);
    ++c.n_lost;
    c.e_lost.add(e);
    if (MID && prm->records)
      c.m_state = ST_LOST;
    if (p.x < Real(0) && sim->bc[0] == 2)
    {
      if (member_gen(p) == 0)
        ++c.n_back;
      else if (sim->surface_binding > 0.0f && Real(p.E) * p.dx * p.dx > Real(sim->surface_binding))
      {
        ++c.n_sput;
        c.e_sput.add(Real(p.E));
      }
    }
  }

  template <class R, class E>
  __device__ void vacancy_event(const R & rec, const E & el, Real Erec, uint64_t key)
  {
    if constexpr (EV)
      event(EV_VACANCY, Real(rec.x), Real(rec.y), Real(rec.z), Erec, el.Z2, Real(el.m2), rec.gen, 0,
            Real(el.Elbind), key, rec.tag);
  }
  template <class R, class E>
  __device__ void replacement_event(const R & rec, const E & el, Real Erec, uint64_t key)
  {
    if constexpr (EV)
      event(EV_REPLACEMENT, Real(rec.x), Real(rec.y), Real(rec.z), Erec, el.Z2, Real(el.m2), rec.gen, 0,
            Real(el.Elbind), key, rec.tag);
  }
  // vacancies by the member that makes them, for the member records
  __device__ void member_vacancy(unsigned int add)
  {
    if (MID && prm->records)
      cold->m_vac += add;
  }
  // a displaced recoil as its followed member starts (single-precision kernel): the
  // vacancy or the replacement that the collision left behind
  __device__ void displaced(bool vac, Real x, Real Erec)
  {
    if (vac)
    {
      ++a_vac;
      if (MID && range_mode)
        return;
      vacancy_bins(x, Erec);
    }
    else
      replacement_bin(x);
    count_bins();
  }
  // the depth histograms' counts of the vacancy or replacement just binned
  __device__ void count_bins()
  {
    const int hb = vac_bin >= 0 ? vac_bin : repl_bin;
    if (hb >= 0)
    {
      if (prm->hist_smem_bins)
        atomicAdd(s_hist + (hb - prm->hist_smem_base), 1u);
      else
        atomicAdd(prm->hist + hb, 1ull);
    }
    vac_bin = repl_bin = -1;
    if (MID && prm->any_evac)
    {
      if (cold->evac_bin >= 0)
        atomicAdd(prm->hist + cold->evac_bin, 1ull);
      cold->evac_bin = -1;
    }
  }
  __device__ void vacancy_bins(Real x, Real Erec)
  {
    const int b = depth_bin(x, inv_vac_bin(), sim->hist_vac_n);
    if (b >= 0)
    {
      vac_bin = int(sim->hist_vac_base) + b;
      if (MID && prm->any_evac && sim->hist_evac_rows > 0)
      {
        // TrimVacEnergyCount::vacancyCreation (apps/src/TrimVacEnergyCount.C:32-53):
        // row int(ln E) of the recoil energy, negative rows in row 0
        int row = int(loge(Erec));
        row = row < 0 ? 0 : row;
        if (row < sim->hist_evac_rows)
          cold->evac_bin = int(sim->hist_evac_base) + row * sim->hist_vac_n + b;
        else
          ++cold->n_dropped;
      }
    }
    else if (b == BIN_BEYOND)
      ++cold->n_dropped;
  }
  __device__ void replacement_bin(Real x)
  {
    const int b = depth_bin(x, inv_vac_bin(), sim->hist_vac_n);
    if (b >= 0)
      repl_bin = int(sim->hist_vac_base + sim->hist_vac_n) + b;
    else if (b == BIN_BEYOND)
      ++cold->n_dropped;
  }

  // vacancyCreation's tally (its event: vacancy_event)
  template <class R, class E>
  __device__ void vacancy(const R & rec, const E & el, Real Erec)
  {
    if (MID && range_mode == 2)
    {
      // TrimPrimaries::vacancyCreation (trim.C:446-464): one vacancy per displaced
      // recoil and, for a recoil of the cutoff generation (not followed), the
      // modified Kinchin-Pease count with the material's mean Z and mass
      unsigned int add = 1;
      if (rec.gen == sim->kp_gen)
      {
        const Real az = Real(el.maz), am = Real(el.mam), Er = Erec;
        const Real ed = Real(0.0115) * powr(az, Real(-7.0 / 3.0)) * Er;
        const Real g = Real(3.4008) * powr(ed, Real(1.0 / 6.0)) + Real(0.40244) * powr(ed, Real(3.0 / 4.0)) + ed;
        const Real kd = Real(0.1337) * powr(az, Real(2.0 / 3.0)) / sqrt(am);
        const Real Ev = Er / (Real(1) + kd * g);
        add += (unsigned int)(int(Real(0.8) * Ev / (Real(2) * Real(el.Edisp))));
      }
      a_vac += add;
      member_vacancy(add);
      return;
    }
    if (MID && range_mode)
    {
      // TrimRange::vacancyCreation (apps/src/TrimRange.C:32-47): Kinchin-Pease
      // count of the displaced recoil, each increment truncated like the
      // reference's int accumulator
      const Real Z = Real(el.Z2), m = Real(el.m2), Er = Erec;
      const Real Ed = Real(el.Edisp);
      const Real ed = Real(0.0115) * powr(Z, Real(-7.0 / 3.0)) * Er;
      const Real kd = Real(0.1337) * powr(Z, Real(2.0 / 3.0)) / sqrt(m);
      const Real g = Real(3.4008) * powr(ed, Real(1.0 / 6.0)) + Real(0.40244) * powr(ed, Real(3.0 / 4.0)) + ed;
      const Real Ev = Er / (Real(1) + kd * g);
      unsigned int add = 0;
      if (Ev < Ed)
        add = 0;
      else if (Ev >= Ed / Real(0.4))
        add = (unsigned int)(Ev * Real(0.4) / Ed);
      else
        add = 1;
      a_vac += add;
      member_vacancy(add);
      return;
    }
    ++a_vac;
    member_vacancy(1u);
    vacancy_bins(Real(rec.x), Erec);
  }
  // replacementCollision's tally
  template <class R>
  __device__ void replacement(const R & rec)
  {
    replacement_bin(Real(rec.x));
  }
  // event and tally
  template <class R, class E>
  __device__ void vacancy(const R & rec, const E & el, Real Erec, uint64_t key)
  {
    vacancy_event(rec, el, Erec, key);
    vacancy(rec, el, Erec);
  }
  template <class R, class E>
  __device__ void replacement(const R & rec, const E & el, Real Erec, uint64_t key)
  {
    replacement_event(rec, el, Erec, key);
    replacement(rec);
  }
  template <class P>
  __device__ void stop(int state, const P & p, int Z1, Real m1)
  {
    if constexpr (EV)
      event(EV_REST, Real(p.x), Real(p.y), Real(p.z), Real(p.E), Z1, m1, member_gen(p), state, Real(0), p.key,
            p.tag, cold->m_md);
    if (MID && prm->records)
      cold->m_state = state;
    a_enuc.add(Real(p.E));
    deposit(Real(p.x), Real(p.y), Real(p.z), Real(p.E));
    ++cold->n_rest[state];
    if (member_gen(p) == 0)
    {
      prm->prim.fx[gprim] = double(p.x);
      prm->prim.fy[gprim] = double(p.y);
      prm->prim.fz[gprim] = double(p.z);
      prm->prim.fstate[gprim] = state;
      const int b = depth_bin(Real(p.x), inv_range_bin(), sim->hist_range_n);
      if (b >= 0)
        atomicAdd(prm->hist + sim->hist_range_base + b, 1ull);
      if (sim->hist_lat_n > 0)
      {
        const float qy = (float(p.y) - sim->lat_y0) * sim->inv_hist_lat_bin;
        const float qz = (float(p.z) - sim->lat_z0) * sim->inv_hist_lat_bin;
        const int n = sim->hist_lat_n;
        if (qy >= 0.0f && qz >= 0.0f && qy < float(n) && qz < float(n))
          atomicAdd(prm->hist + sim->hist_lat_base + (long long)int(qz) * n + int(qy), 1ull);
      }
    }
  }

  // truncation toward zero like int(x) in the reference (TrimVacCount.C:36-39),
  // in the engine's own precision; BIN_BEYOND past the last bin, -1 before the
  // first (where the reference drops the event too) or without a histogram
  static constexpr int BIN_BEYOND = -2;
  static __device__ int depth_bin(Real x, Real inv_bin, int n)
  {
    const Real q = x * inv_bin;
    if (n <= 0 || !(q > Real(-1)))
      return -1;
    if (q >= Real(n))
      return BIN_BEYOND;
    return int(q);
  }
  static __device__ Real loge(Real x)
  {
    if constexpr (sizeof(Real) == sizeof(float))
      return __logf(x);
    else
      return log64(x);
  }
  __device__ Real inv_vac_bin() const
  {
    if constexpr (sizeof(Real) == sizeof(float))
      return sim->inv_hist_vac_bin_f;
    else
      return sim->inv_hist_vac_bin;
  }
  __device__ Real inv_range_bin() const
  {
    if constexpr (sizeof(Real) == sizeof(float))
      return sim->inv_hist_range_bin_f;
    else
      return sim->inv_hist_range_bin;
  }
  static __device__ Real powr(Real x, Real y)
  {
    if constexpr (sizeof(Real) == sizeof(float))
      return __powf(x, y);
    else
      return pow64(x, y);
  }

  // hand the energy sums to the per-primary arrays: the single-precision kernel does it
  // on every 64th iteration, so that its sums stay short
  __device__ void hand_over()
  {
    if (a_eel.nonzero())
      a_eel.atomic_add_to(prm->prim.eel + gprim);
    if (a_enuc.nonzero())
      a_enuc.atomic_add_to(prm->prim.enuc + gprim);
    a_eel.reset();
    a_enuc.reset();
  }
  // the record of a member that has ended (records runs)
  template <class P>
  __device__ void record(const P & p, unsigned int ncoll)
  {
    const unsigned long long slot = atomicAdd(prm->n_records, 1ull);
    if ((long long)slot >= prm->records_cap)
      return;
    MemberRecord m;
    m.key = p.key;
    m.sim = p.sim;
    m.species = member_species(p);
    m.gen = member_gen(p);
    m.state = cold->m_state;
    m.ncoll = ncoll;
    m.nvac = cold->m_vac;
    m.E = double(p.E);
    m.x = double(p.x);
    m.y = double(p.y);
    m.z = double(p.z);
    m.eel = cold->m_eel.value();
    prm->records[slot] = m;
  }

  __device__ void flush_prim()
  {
    if (gprim < 0)
      return;
    if (a_vac)
      atomicAdd(prm->prim.vac + gprim, (unsigned long long)a_vac);
    if (a_coll)
      atomicAdd(prm->prim.coll + gprim, (unsigned long long)a_coll);
    if (a_eel.nonzero())
      a_eel.atomic_add_to(prm->prim.eel + gprim);
    if (a_enuc.nonzero())
      a_enuc.atomic_add_to(prm->prim.enuc + gprim);
    reset_prim();
  }
  __device__ void flush_sim(int s)
  {
    if (s < 0)
      return;
    SimTotals * t = prm->totals + s;
    const LaneCold<Acc> & c = *cold;
    using ull = unsigned long long;
    if (c.n_members)
      atomicAdd(&t->members, ull(c.n_members));
    if (const unsigned int n = c.n_rest[ST_REPLACEMENT] + c.n_rest[ST_SUBSTITUTIONAL])
      atomicAdd(&t->replacements, ull(n));
    if (c.n_rest[ST_INTERSTITIAL])
      atomicAdd(&t->interstitials, ull(c.n_rest[ST_INTERSTITIAL]));
    if (c.n_rest[ST_SUBSTITUTIONAL])
      atomicAdd(&t->substitutionals, ull(c.n_rest[ST_SUBSTITUTIONAL]));
    if (c.n_lost)
      atomicAdd(&t->lost, ull(c.n_lost));
    if (n_newton)
      atomicAdd(&t->newton_iters, ull(n_newton));
    if (c.n_passes)
      atomicAdd(&t->rejection_passes, ull(c.n_passes));
    if (c.n_fallbacks)
      atomicAdd(&t->fallbacks, ull(c.n_fallbacks));
    if (c.e_lost.nonzero())
      c.e_lost.atomic_add_to(&t->Elost);
    if (c.e_unf.nonzero())
      c.e_unf.atomic_add_to(&t->Eunfollowed);
    if (c.n_sput)
      atomicAdd(&t->sputtered, ull(c.n_sput));
    if (c.n_back)
      atomicAdd(&t->backscattered, ull(c.n_back));
    if (c.e_sput.nonzero())
      c.e_sput.atomic_add_to(&t->Esputtered);
    if (c.n_dropped)
      atomicAdd(&t->hist_dropped, ull(c.n_dropped));
    reset_sim();
  }
};

// LVL: the feature level (KernelLevel); the collision code knows the cluster
// geometry at LVL_GEO, LVL_FULL, LVL_CLU and LVL_CLU_EV, the non-universal
// potentials at LVL_GEO and LVL_FULL
template <class Pol, int LVL>
__global__ void __launch_bounds__(128, Pol::min_blocks(LVL))
cascade_kernel(const EngineParams prm, const typename Pol::Tables tabs)
{
  constexpr bool MID = LVL >= LVL_MID;
  constexpr bool EXT = level_clusters(LVL);   // the cluster geometry
  constexpr bool POT = level_potentials(LVL); // the Moliere and C-Kr potentials
  using Particle = typename Pol::Particle;
  extern __shared__ __align__(16) unsigned char smem[];
  if (prm.in_records && *prm.in_count == 0)
    return; // a drain pass with nothing to drain
  RecoilPool<Particle>::start(prm.pool);

  // stage the tables of a single-simulation run in shared memory
  // per-block vacancy / replacement counters (zeroed before the staging barrier)
  unsigned int * s_hist = reinterpret_cast<unsigned int *>(smem + prm.hist_smem_offset);
  for (int i = threadIdx.x; i < prm.hist_smem_bins; i += blockDim.x)
    s_hist[i] = 0u;
  if (prm.hist_smem_bins)
    __syncthreads();
  const typename Pol::Tables tab = Pol::stage(prm, tabs, smem);

  const unsigned int FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned int lt = lanemask_lt();
  const long long warp_id = (long long)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  Particle * stack = reinterpret_cast<Particle *>(prm.stacks) + warp_id * prm.stack_cap;
  Particle * overflow = reinterpret_cast<Particle *>(prm.overflow);
  const Particle * in_records = reinterpret_cast<const Particle *>(prm.in_records);
  long long n_work = prm.total_primaries;
  if (prm.in_records)
  {
    const long long c = (long long)*prm.in_count;
    n_work = c < prm.in_cap ? c : prm.in_cap;
  }

  RecoilPool<Particle> pool;
  int top = 0;
  bool work_done = false; // no more primaries / input records for this warp
  // members per refill: the launch's choice for fresh primaries; for the records of
  // a drain pass, a quarter of a warp's fair share (at most one per lane)
  int max_take = prm.max_take;
  if (prm.in_records)
  {
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long share = n_work / (nwarps * 4);
    max_take = share < 1 ? 1 : (share > 32 ? 32 : int(share));
  }
  bool live = false;
  Particle p;
  uint32_t ic = 0;
  typename Pol::Real r1 = 0;
  int cur_sim = -1;
  const SimDesc * sim = nullptr;
  typename Pol::MemberCtx mctx;

  LaneSink<Pol, LVL> sink;
  sink.cold = reinterpret_cast<LaneCold<typename Pol::Acc> *>(smem + prm.cold_offset) + threadIdx.x;
  sink.cold->vcell = -1;
  sink.cold->vacc = 0.0f;
  sink.cold->evac_bin = -1;
  sink.cold->ev_next = sink.cold->ev_end = 0;
  sink.prm = &prm;
  sink.s_hist = s_hist;
  sink.vac_bin = sink.repl_bin = -1;
  sink.sim = nullptr;
  sink.gprim = -1;
  sink.range_mode = 0;
  sink.vox = false;
  sink.dep_in = false;
  sink.reset_prim();
  sink.reset_sim();
  sink.reset_member();

  auto start_member = [&](const Particle & q) {
    p = q;
    ic = 0;
    if (p.sim != cur_sim)
    {
      sink.flush_prim();
      sink.flush_sim(cur_sim);
      cur_sim = p.sim;
      sim = prm.sims + cur_sim;
      sink.sim = sim;
      sink.isim = cur_sim;
      sink.range_mode = sim->range_mode;
      sink.vox = MID && prm.voxels != nullptr && sim->voxel_n[0] > 0;
      sink.gprim = -1;
    }
    if ((long long)p.prim != sink.gprim)
    {
      sink.flush_prim();
      sink.gprim = (long long)p.prim;
      if (sink.n_newton > 0x40000000u || sink.cold->n_passes > 0x40000000u)
        sink.flush_sim(cur_sim);
    }
    Pol::begin_member(mctx, prm, tab, *sim, p);
    if constexpr (LaneSink<Pol, LVL>::EV)
    {
      // IonMDTag: the demo programs' MD-gap mark, taken when the member starts
      // (apps/mytrim_solid.C:156-159); a spawned recoil's _md is 0 (ion.C:88-93)
      const bool gap = double(p.E) > sim->md_Emin && double(p.E) < sim->md_Emax;
      sink.cold->m_md = (sim->md_Z != 0 && mctx.sc->Z1 == sim->md_Z && gap) ? 1 : 0;
    }
    r1 = Pol::first_draw(p.key, prm.k0, prm.k1);
    sink.reset_member();
    ++sink.cold->n_members;
  };

  unsigned int steps = 0;
  while (true)
  {
    ++steps;
    // ---- refill idle lanes: recoils from the warp stack first, then new work
    // idle lanes wait until refill_min (at most 32) of them need a member, so that
    // the member-start code below runs for several lanes at once: without waiting
    // it runs in nearly every iteration, for about four lanes of the 32
    const unsigned int idle = __ballot_sync(FULL, !live);
    if (idle && __popc(idle) >= prm.refill_min)
    {
      __syncwarp(); // the recoils other lanes pushed
      const int nidle = __popc(idle);
      const int rank = __popc(idle & lt);
      const int npop = nidle < top ? nidle : top;
      if (!live && rank < npop)
      {
        start_member(stack[top - 1 - rank]);
        live = true;
      }
      top -= npop;
      int need = nidle - npop;
      if (need > max_take)
        need = max_take;
      if (need > 0 && !work_done)
      {
        unsigned long long base = 0;
        const int leader = __ffs(idle) - 1;
        if (lane == leader)
          base = atomicAdd(prm.next_primary, (unsigned long long)need);
        base = __shfl_sync(FULL, base, leader);
        const long long avail = n_work - (long long)base;
        if (avail <= need)
          work_done = true;
        const int r = rank - npop;
        if (!live && r >= 0 && r < need && r < avail)
        {
          const long long g = (long long)base + r;
          if (prm.in_records)
            start_member(in_records[g]);
          else
          {
            long long first = 0;
            const int s = prm.n_sims > 1 ? find_sim(prm, g, first) : 0;
            start_member(Pol::make_primary(prm.sims[s], s, prm.sims[s].prim_begin + (g - first)));
          }
          live = true;
        }
      }
      __syncwarp(); // popped before another lane pushes into the same place
    }
    if (__ballot_sync(FULL, live) == 0)
    {
      // nothing left: recoils of a busier warp, or the end
      top = pool.wait(prm, (unsigned int)warp_id, stack, lane);
      if (top == 0)
        break;
      continue;
    }

    // ---- one collision per live lane
    Particle rec;
    int flags = 0;
    if (live)
    {
      ++ic;
      ++sink.a_coll;
    }
    // every lane takes part (a policy may evaluate warp-collective code); lanes
    // without a member do no work and get no flags
    flags = Pol::template collide<EXT, POT>(live, p, ic, r1, mctx, prm.k0, prm.k1, rec, sink);
    if (live)
    {
      if (flags & CF_VOID)
        --sink.a_coll; // the member left without a collision (no checkPKAState)
      if (!(flags & CF_DONE) && ic >= prm.max_collisions)
      {
        atomicOr(prm.error_flags, ERRB_BUDGET);
        flags |= CF_DONE;
      }
      if (flags & CF_DONE)
      {
        live = false;
        if (MID && prm.records)
          sink.record(p, ic);
      }
      if (flags & CF_PUSH)
      {
        rec.sim = p.sim;
        rec.prim = p.prim;
      }
    }
    // depth histograms: a collision makes a vacancy or a replacement, never both;
    // about one lane in ten has an event, so each adds its own count (aggregating
    // lanes with __match_any_sync cost more than it saved)
    sink.count_bins();

    // ---- push displaced recoils onto the warp stack
    const bool push = (flags & CF_PUSH) != 0;
    const unsigned int pm = __ballot_sync(FULL, push);
    if (pm)
    {
      if (push)
      {
        const int slot = top + __popc(pm & lt);
        if (slot < prm.stack_cap)
          stack[slot] = rec;
        else
        {
          const unsigned long long o = atomicAdd(prm.overflow_count, 1ull);
          if ((long long)o < prm.overflow_cap)
            overflow[o] = rec;
          else
            atomicOr(prm.error_flags, ERRB_QUEUE_FULL);
        }
      }
      top += __popc(pm);
      if (top > prm.stack_cap)
        top = prm.stack_cap;
    }
    if (((steps + (unsigned int)warp_id) & 3u) == 0u && pool.wanted(prm, top))
      top = pool.send(prm, stack, top, lane);
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
  {
    atomicAdd(prm.warp_steps, (unsigned long long)(steps - 1)); // the last pass finds no work
  }
}

} // namespace mtg
