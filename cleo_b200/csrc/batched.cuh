// batched.cuh — the batched microphysics of one SDM step (exec_mode CLEO_EXEC_BATCHED).
//
// Same results as k_micro (one CTA per gridbox), scheduled for B200 occupancy:
//   k_b_qcond      warp per 1 to 32 gridboxes (seq_per): qcond from the moved superdroplets (after the sort),
//                  their condensate masses added in order (warp_batch_sums)
//   k_b_thermo     thread per gridbox: psat, supersaturation, diffusion factor, the droplets'
//                  Kohler factors that depend on temperature alone
//   k_cond_a       thread per superdroplet: the mandatory two Newton iterations of every
//                  implicit-Euler solve; solves needing more (sub-stepping, or a restart after two
//                  unconverged iterations) are appended to a list keyed by their cost
//   k_cond_place   that list by cost class
//   k_mlp_tc       with nr_seed = CLEO_NRSEED_MLP only: the surrogate's Newton seeds for the
//                  listed solves (the ones the reference guess did not settle in two iterations)
//   k_cond_b       thread per listed solve, neighbouring lanes of similar cost, from the seed
//                  where its residual beats the reference guess's
//   k_b_commit     warp per 2 to 32 gridboxes: the condensed mass of each one's superdroplets
//                  added in their order, their Newton iterations, and the state update
//   k_b_commit_big the same, a warp each: large gridboxes, or all of a small domain's
//   k_b_classify   gridboxes into size buckets (warp-aggregated atomics); the warp kernel's
//                  buckets as records {gridbox, start, count, RNG slot}
//   k_b_perm       thread per gridbox of the warp kernel's buckets: the Fisher-Yates shuffle
//   k_b_small      persistent, warp per gridbox (n <= small_max <= 128; 64- and 128-slot
//                  variants): collisions in registers + per-warp shared memory
//   k_b_cta<false> persistent, CTA per gridbox (small_max < n <= medium_max <= 1024): the same
//                  with shared-memory staging
//   k_b_cta<true>  CTA per gridbox (n > medium_max) with global scratch
// small_max, the pass-A block size, the resident-CTA targets (register budgets) of pass A and of
// the warp kernel's 64-slot variant are chosen by the autotuner (results do not depend on them).
// Every per-gridbox sum of doubles adds its terms in the superdroplets' order, as the reference's
// sequential loop does (warp_batch_sums): condensed mass per droplet goes through a scratch array and is
// summed per gridbox after the solves, so budgets and states are the sequential loop's doubles
// whatever the schedule.
#pragma once

#include "pair_bound.h"

namespace {

using mlp::fence_async_smem;
using mlp::mbar_init;
using mlp::mbar_wait_bounded;
using mlp::MBAR_TRIES;
using mlp::smem_u32;

__device__ __forceinline__ uint32_t warp_sum_u(uint32_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  return __shfl_sync(0xFFFFFFFFu, v, 0);
}

// warp-aggregated append of `want` lanes to a list counter; returns this lane's slot
__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool want) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (m) {
    const int leader = __ffs(m) - 1;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
  }
  return base + __popc(m & ((1u << lane) - 1u));
}

// ---- sums over gridboxes in the superdroplets' order, a warp per 32 consecutive gridboxes ----
// Consecutive gridboxes' ranges follow each other, so a batch of up to 32 gridboxes is one
// contiguous range [gstart[g0], gstart[g0 + nb]). The warp reads it coalesced, SEQ_WIN elements
// at a time, into its shared buffers (term(k) -> dbuf, iters(k) -> ubuf), and lane j adds the
// terms of gridbox g0 + j's valid superdroplets [gstart, gstart + gcount) one after another: the
// reference's sequential loop (seq_sum's order). Each window starts at the first element a lane
// still has to add, so ranges no lane adds are not read, and is loaded into registers while the
// window before it is being added. On smaller domains a warp takes fewer gridboxes (seq_per), down
// to one: a window's additions are a chain, and 32 gridboxes a warp left two warps a scheduler on
// 50 thousand gridboxes (a mass-moment call 59 us, now 45; 4096 gridboxes' commit 25 us, now 8).
// With skip_big, a gridbox of more than
// SEQ_BIG superdroplets is left out (its lane adds nothing): warp_seq_sums sums it with a warp of
// its own, so that one long sequential sum does not hold up its batch and large gridboxes are
// summed in parallel.
constexpr uint32_t SEQ_WIN = 256;
constexpr int SEQ_THREADS = 256;
constexpr uint32_t SEQ_BIG = 128;
template <class Term, class Iters>
__device__ __forceinline__ void warp_batch_sums(const DevCtx& c, uint32_t g0, uint32_t nb,
                                                double* dbuf, uint32_t* ubuf, Term term,
                                                Iters iters, double& sum,
                                                unsigned long long& its, bool skip_big,
                                                double init = 0.0) {
  constexpr int PER = SEQ_WIN / 32;  // elements of a window per lane
  constexpr uint32_t NONE = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const uint32_t hi = c.gstart[g0 + nb];
  const bool own = (uint32_t)lane < nb;
  const uint32_t s = own ? c.gstart[g0 + lane] : hi;
  uint32_t e = own ? s + c.gcount[g0 + lane] : hi;
  if (skip_big && e - s > SEQ_BIG) e = s;
  double acc = init;
  unsigned long long it = 0;
  uint32_t cur = s;  // this lane's next element to add
  // the window [w0, w0 + SEQ_WIN) clipped to hi, loaded into registers a window ahead
  double pv[PER];
  uint32_t pu[PER];
  const auto load = [&](uint32_t w0) {
    const uint32_t w1 = hi - w0 < SEQ_WIN ? hi : w0 + SEQ_WIN;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const uint32_t k = w0 + 32 * q + lane;
      pv[q] = k < w1 ? term(k) : 0.0;
      pu[q] = k < w1 ? iters(k) : 0u;
    }
  };
  uint32_t w0 = __reduce_min_sync(0xFFFFFFFFu, cur < e ? cur : NONE);
  if (w0 != NONE) load(w0);
  while (w0 != NONE) {
    const uint32_t w1 = hi - w0 < SEQ_WIN ? hi : w0 + SEQ_WIN;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      dbuf[32 * q + lane] = pv[q];
      ubuf[32 * q + lane] = pu[q];
    }
    __syncwarp();
    const uint32_t b = e < w1 ? e : w1;
    const uint32_t next = cur < b ? b : cur;  // the cursor after this window
    const uint32_t nw0 = __reduce_min_sync(0xFFFFFFFFu, next < e ? next : NONE);
    if (nw0 != NONE) load(nw0);  // in flight while this window is added
    for (uint32_t k = cur; k < b; ++k) {
      acc += dbuf[k - w0];
      it += ubuf[k - w0];
    }
    cur = next;
    __syncwarp();
    w0 = nw0;
  }
  sum = acc;
  its = it;
}
// the same sequential sums for one gridbox's range [s, e) by a whole warp: up to SEQ_GROUP chunks
// of 32 terms loaded at once, each chunk's terms broadcast one by one and added in order by every
// lane. Two sums (qcond's condensate masses qm, when given, and the condensed masses dm) are
// independent chains and run interleaved; the iterations (integers, any order) are added per lane,
// then across the warp.
constexpr int SEQ_GROUP = 8;
__device__ __forceinline__ void warp_seq_sums(uint32_t s, uint32_t e, const double* qm,
                                              const double* dm, const uint32_t* its_in,
                                              double& qsum, double& dsum,
                                              unsigned long long& its) {
  const uint32_t lane = threadIdx.x & 31;
  double aq = 0.0, ad = 0.0;
  unsigned long long it = 0;
  for (uint32_t k0 = s; k0 < e; k0 += 32 * SEQ_GROUP) {
    double vq[SEQ_GROUP], vd[SEQ_GROUP];
#pragma unroll
    for (int q = 0; q < SEQ_GROUP; ++q) {
      const uint32_t k = k0 + 32 * q + lane;
      const bool in = k < e;
      vq[q] = in && qm ? qm[k] : 0.0;
      vd[q] = in ? dm[k] : 0.0;
      it += in ? its_in[k] : 0u;
    }
#pragma unroll
    for (int q = 0; q < SEQ_GROUP; ++q) {
      const uint32_t c0 = k0 + 32 * q;
      if (c0 >= e) break;  // uniform across the warp
      const uint32_t m = e - c0 < 32 ? e - c0 : 32;
#pragma unroll
      for (uint32_t j = 0; j < 32; ++j) {
        const double tq = __shfl_sync(0xFFFFFFFFu, vq[q], j);
        const double td = __shfl_sync(0xFFFFFFFFu, vd[q], j);
        if (j < m) {
          aq += tq;
          ad += td;
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) it += __shfl_down_sync(0xFFFFFFFFu, it, o);
  qsum = aq;
  dsum = ad;
  its = __shfl_sync(0xFFFFFFFFu, it, 0);
}

// ---- effect_on_hydrometeor_states (movesupersindomain.hpp:95-136) ----
// qcond of gridbox g from the sum m of its superdroplets' condensate masses x xi (summed in their
// order, by k_b_qcond or by the first condensation commit after motion)
__device__ __forceinline__ void set_qcond(const DevCtx& c, uint32_t g, double m) {
  const double R0cubed_VOL0 = R0 * R0 * R0 / VOL0;
  const double rho_cond = m / c.volume[g] * R0cubed_VOL0;
  c.qcond[g] = rho_cond / dry_air_density(c.press[g], c.temp[g], c.qvap[g]);
}
// per: gridboxes of a warp (seq_per)
__global__ void __launch_bounds__(SEQ_THREADS) k_b_qcond(const __grid_constant__ DevCtx c,
                                                         uint32_t per) {
  __shared__ double dbuf[SEQ_THREADS / 32][SEQ_WIN];
  __shared__ uint32_t ubuf[SEQ_THREADS / 32][SEQ_WIN];
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t g0 = warp * per; g0 < c.ngbxs; g0 += nwarps * per) {
    const uint32_t nb = c.ngbxs - g0 < per ? c.ngbxs - g0 : per;
    double m;
    unsigned long long unused;
    warp_batch_sums(
        c, g0, nb, dbuf[wib], ubuf[wib],
        [&](uint32_t i) {
          const uint32_t g = c.sd.gbx[i];
          return g < c.ngbxs ? condensate_mass(c.sd.r[i], c.sd.msol[i], Where{c.err, g, i}) *
                                   (double)c.sd.xi[i]
                             : 0.0;
        },
        [](uint32_t) { return 0u; }, m, unused, false);
    if ((uint32_t)lane < nb) set_qcond(c, g0 + lane, m);
  }
}

// ---- per-gridbox thermodynamics of superdroplets_change (condensation.cpp:43-59) ----
// (every gridbox, empty ones too: the reference evaluates psat for each, and its check of the
// temperature with it)
// With `first` (an SDM step that begins with condensation) it also does k_b_reset's part.
__global__ void k_b_thermo(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b,
                           int first) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid < COST_CLASSES + COST_CURSORS) b.ccnt[tid] = 0;
  if (first && tid < 8) b.ctr[1 + tid] = 0;  // bucket counts and heads
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < c.ngbxs; g += gridDim.x * blockDim.x) {
    if (g == 0) b.ctr[0] = b.ctr[10] = 0;  // deferred solves, big gridboxes
    if (first) b.slot[g] = 0;
    const Where w{c.err, g, c.gstart[g]};
    const double temp = c.temp[g];
    const double psat = saturation_pressure(temp, w);
    b.th_s[g] = supersaturation_ratio(c.press[g], c.qvap[g], psat);
    b.th_ff[g] = diffusion_factor(c.press[g], temp, psat);
    const double akoh = kohler_a(temp);  // the droplets' factors that depend on akoh alone
    b.th_ak[g] = akoh;
    b.th_a3[g] = activation_a3(akoh);
    b.th_u3[g] = unique_a3(akoh);
  }
}

// the surrogate's IO for the batched schedule: row j is the j-th of pass A's solves by class,
// whose first b.ccnt[0] entries are the direct solves that two iterations did not settle (key 0;
// the sub-stepping solves after them cannot use a seed); the seed r^2 goes to b.dm of that
// droplet, which pass B reads (and then overwrites with the droplet's condensed mass)
struct SdmListSeedIO {
  const uint32_t* gbx;
  const double *r, *msol, *temp, *press, *s_ratio;
  double delt;
  const uint32_t* list;
  const uint32_t* count;
  double* seed;
  __device__ __forceinline__ uint32_t rows(uint32_t n) const {
    const uint32_t c = *count;
    return c < n ? c : n;
  }
  __device__ __forceinline__ void features(uint32_t j, float x[mlp::NIN]) const {
    const uint32_t i = list[j];
    const uint32_t g = gbx[i];
    mlp::raw_features(r[i], msol[i], temp[g], press[g], s_ratio[g], delt, x);
  }
  __device__ __forceinline__ void store(uint32_t j, float t) const {
    const uint32_t i = list[j];
    seed[i] = mlp::seed_from(r[i], t);
  }
};

// cost class of a deferred solve of `delt / mindelt` sub-steps: 1 + a quarter-octave of their number,
// read off the leading bits of the single-precision value; class 0 is the restarts of direct solves
__device__ __forceinline__ uint32_t cost_class(double delt, double mindelt) {
  const double ns = ceil(delt / mindelt);
  const float f = ns >= 1.0 ? (ns <= 65535.0 ? (float)ns : 65536.0f) : 1.0f;
  return 1u + ((__float_as_uint(f) >> 21) - (127u << 2));  // 1 .. 65
}
// Class of the restart that continues from zres (resume_restart): class 0, or LONG_RESTART, which is
// counted in class 0 and placed behind its others. Where the solute term governs g, an iterate below
// the root grows by 5/3 an iteration (g / (z g') is -2/3 there), and two iterations from a droplet's
// own size can end at the floor of 1e-8, some 30 iterations below. So the logarithm of r^2 / zres
// tells their number: 1 to 9 more up to 2^4, 22 to 37 from 2^14, little between. All in one class, a
// warp's lanes were at work in 12 of 32 of its iterations where a fifth of the restarts are long
// (k_cond_b 764 us for 2.9 M solves, now 541). The exponent and leading bits are the logarithm
// within 0.09; five classes by it were no better, and their counting cost k_cond_a 9%.
__device__ __forceinline__ uint32_t restart_class(double r, double zres) {
  const int hr = __double2hiint(r), lg = (hr - (1023 << 20)) + (hr - __double2hiint(zres));
  return zres > 0.0 && lg >= (4 << 20) ? LONG_RESTART : 0u;
}
// the appended solves counted per class, a block's in shared memory first; every thread of the block
// calls these. The restarts, most of the solves at a tight tolerance, are counted a warp at a time in
// a register (one shared atomic each ran 32 in a row: 50 us of 275 for 5 M superdroplets).
__device__ __forceinline__ void class_count_begin(uint32_t* cnt) {
  for (uint32_t i = threadIdx.x; i < COST_CLASSES; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
}
__device__ __forceinline__ void class_count(uint32_t* cnt, uint32_t& restarts, bool defer,
                                            uint32_t cls) {
  const bool restart = cls == 0u || cls == LONG_RESTART;
  restarts += __popc(__ballot_sync(0xFFFFFFFFu, defer && restart));
  if (defer && !restart) atomicAdd(&cnt[cls], 1u);
}
__device__ __forceinline__ void class_count_end(uint32_t* cnt, uint32_t restarts,
                                                uint32_t* total) {
  if ((threadIdx.x & 31) == 0 && restarts) atomicAdd(&cnt[0], restarts);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < COST_CLASSES; i += blockDim.x)
    if (cnt[i]) atomicAdd(&total[i], cnt[i]);
}
// The deferred solves by class, restarts first (the long ones fill their part from its end). Only
// neighbouring lanes' costs matter to pass B (and the restarts' place to the surrogate), not the
// order within a class, so blocks of PLACE_ITEMS solves take their shares of each class with one
// atomic: one launch where a radix sort of the 16-bit costs took eleven, which returned at once or
// not (about 16 us of a step), and 7 us where it sorted 400 thousand in 30.
constexpr uint32_t PLACE_ITEMS = 1024;
__global__ void __launch_bounds__(256)
k_cond_place(const uint32_t* __restrict__ n_ptr, const uint32_t* __restrict__ lkeys,
             const uint32_t* __restrict__ lvals, uint32_t* __restrict__ ccnt,
             uint32_t* __restrict__ order) {
  __shared__ uint32_t cnt[COST_CURSORS], start[COST_CURSORS], total[COST_CLASSES];
  const uint32_t nl = *n_ptr;
  constexpr uint32_t PER = PLACE_ITEMS / 256;
  if (threadIdx.x < COST_CLASSES) total[threadIdx.x] = ccnt[threadIdx.x];
  for (uint32_t i0 = blockIdx.x * PLACE_ITEMS; i0 < nl; i0 += gridDim.x * PLACE_ITEMS) {
    if (threadIdx.x < COST_CURSORS) cnt[threadIdx.x] = 0;
    __syncthreads();
    uint32_t cls[PER], val[PER], rank[PER];
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
      const uint32_t i = i0 + q * 256 + threadIdx.x;
      cls[q] = i < nl ? lkeys[i] : COST_CURSORS;
      val[q] = i < nl ? lvals[i] : 0u;
    }
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {  // one shared atomic per class a warp meets
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, cls[q]);
      const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
      uint32_t base = 0;
      if (lane == leader && cls[q] < COST_CURSORS)
        base = atomicAdd(&cnt[cls[q]], (uint32_t)__popc(peers));
      rank[q] = __shfl_sync(0xFFFFFFFFu, base, leader) + __popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (threadIdx.x < COST_CURSORS) {
      const uint32_t m = cnt[threadIdx.x];
      uint32_t s = m ? atomicAdd(&ccnt[COST_CLASSES + threadIdx.x], m) : 0u;
      if (threadIdx.x == LONG_RESTART)
        s = total[0] - s - m;
      else
        for (uint32_t k = 0; k < threadIdx.x; ++k) s += total[k];
      start[threadIdx.x] = s;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q)
      if (cls[q] < COST_CURSORS) order[start[cls[q]] + rank[q]] = val[q];
    __syncthreads();
  }
}

// ---- pass A: superdrop_mass_change (condensation.cpp:98-112) up to two Newton iterations ----
// Bound by issue (930 instructions a warp of droplets, 400 of them FP64) and by the loads at the head
// of each solve; the gridbox index, behind which the gridbox's values wait, is loaded a slot ahead.
// 226 us for 5 M superdroplets at 4 CTAs per SM, 276 at 3. (Copying the next slot's eight values
// ahead into shared memory as well was slower, 281 us: a warp's copies of one gridbox's value are
// 32 separate ones.)
template <int MINB>
__global__ void __launch_bounds__(256, MINB)
k_cond_a(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b) {
  const cleo_b200_params& p = c.p;
  const uint32_t n = c.counters[0];
  const NewtonCfg cfg{p.maxniters, p.rtol, p.atol};
  __shared__ uint32_t cnt[COST_CLASSES];
  class_count_begin(cnt);
  uint32_t restarts = 0;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x;
  uint32_t g_next = i0 + threadIdx.x < n ? c.sd.gbx[i0 + threadIdx.x] : OOB;
  for (; i0 < n; i0 += step) {
    const uint32_t i = (uint32_t)i0 + threadIdx.x;
    const uint32_t g = g_next;
    g_next = i0 + step + threadIdx.x < n ? c.sd.gbx[i0 + step + threadIdx.x] : OOB;
    bool defer = false;
    uint32_t key = 0;
    if (g < c.ngbxs) {
      const Where w{c.err, g, i};
      const double r = c.sd.r[i], msol = c.sd.msol[i];
      // the condensate mass qcond sums (k_b_qcond's term), for the commit to add in order
      if (b.qm) b.qm[i] = condensate_mass(r, msol, w) * (double)c.sd.xi[i];
      const double ffactor_fv = b.th_ff[g] / ventilation_factor(r);
      const OdeConsts o = ode_consts(b.th_s[g], b.th_ak[g], kohler_b(msol), ffactor_fv);
      const double z0 = initialguess_a3(o, r, b.th_a3[g]);
      // ucrit1 || ucrit2, the critical timestep only evaluated when ucrit1 fails
      const bool ucrit1 = first_unique_a3(o, r, z0, b.th_u3[g]);
      double crit = 0.0;
      uint32_t ni = 0;
      if (ucrit1 || below_critical_timestep(o, p.cond_delt, crit)) {
        double radius, zres;
        if (!two_iterations(cfg, o, p.cond_delt, r, z0, ni, radius, zres)) {
          defer = true;  // restart from z0 until converged (impliciteuler.cpp:136-140)
          key = restart_class(r, zres);
          b.zres[i] = zres;
          b.ffv[i] = ffactor_fv;
        } else {
          const double rnew = max_dryradius(radius, msol);  // change_radius
          b.dm[i] = (condensate_mass(rnew, msol, w) - condensate_mass(r, msol, w)) *
                    (double)c.sd.xi[i];
          b.its[i] = ni;
          c.sd.r[i] = rnew;
        }
      } else {
        defer = true;
        key = cost_class(p.cond_delt, fmax(crit, p.cond_minsubdelt));
        b.ffv[i] = ffactor_fv;  // pass B's sub-stepping solve starts from it
      }
    }
    const uint32_t pos = warp_append(&b.ctr[0], defer);
    if (defer) {
      b.lkeys[pos] = key;
      b.lvals[pos] = i;
    }
    class_count(cnt, restarts, defer, key);
  }
  class_count_end(cnt, restarts, b.ccnt);
}

// ---- pass B: the deferred solves, in order of cost ----
template <int MINB>
__global__ void __launch_bounds__(256, MINB)
k_cond_b(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b) {
  const cleo_b200_params& p = c.p;
  const uint32_t nl = b.ctr[0], restarts = b.ccnt[0];
  const NewtonCfg cfg{p.maxniters, p.rtol, p.atol};
  for (uint32_t jr = blockIdx.x * blockDim.x + threadIdx.x; jr < nl;
       jr += gridDim.x * blockDim.x) {
    // the list is sorted by ascending cost: the most expensive solves start first, so that the
    // longest sub-stepping ones do not run alone at the end
    const uint32_t j = nl - 1 - jr;
    const uint32_t i = b.order[j];
    const uint32_t g = c.sd.gbx[i];
    const Where w{c.err, g, i};
    const double r = c.sd.r[i], msol = c.sd.msol[i];
    const double akoh = b.th_ak[g], bkoh = kohler_b(msol);
    uint32_t ni = 0;
    const double seed = p.nr_seed == CLEO_NRSEED_MLP ? b.dm[i] : 0.0;
    double newr;
    if (j < restarts && cfg.maxniters >= 2) {
      // a direct solve whose two iterations in pass A did not converge: the restart continues
      // from them (resume_restart), unless the surrogate's seed converges first
      const OdeConsts o = ode_consts(b.th_s[g], akoh, bkoh, b.ffv[i]);  // pass A's th_ff / ventilation
      ni = 2;
      double rsqrd = 0.0;
      bool done = false;
      if (seed_ok(seed)) {
        const double z0 = initialguess_a3(o, r, b.th_a3[g]);
        const bool ucrit1 = first_unique_a3(o, r, z0, b.th_u3[g]);
        bool tried;
        done = integrate_seeded(cfg, o, p.cond_delt, r, z0, seed, ni, rsqrd, tried) &&
               seeded_root_ok(o, ucrit1, rsqrd);
      }
      if (!done) {
        const int code = resume_restart(cfg, o, p.cond_delt, r, b.zres[i], ni, rsqrd);
        if (code) w.fail(code);
      }
      newr = sqrt(rsqrd);
    } else {
      // (b.ffv: pass A's th_ff / ventilation_factor(r), what solve_condensation computes first)
      newr = solve_condensation_fv(cfg, p.cond_delt, p.cond_minsubdelt, b.th_s[g], akoh, bkoh,
                                   b.ffv[i], r, seed, ni, w);
    }
    const double rnew = max_dryradius(newr, msol);
    b.dm[i] = (condensate_mass(rnew, msol, w) - condensate_mass(r, msol, w)) * (double)c.sd.xi[i];
    b.its[i] = ni;
    c.sd.r[i] = rnew;
  }
}

// ---- size buckets of the gridboxes that hold superdroplets ----
__global__ void k_b_classify(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b) {
  const uint32_t ng = c.ngbxs;
  for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < ng; g0 += gridDim.x * blockDim.x) {
    const uint32_t g = g0 + threadIdx.x;
    const uint32_t n = g < ng ? c.gcount[g] : 0u;
    // buckets: warp kernel's 64-slot variant, its 128-slot variant (65 .. small_max), CTA per
    // gridbox in shared memory, CTA per gridbox with global scratch
    const uint32_t lo = b.small_max < SMALL_MAX ? b.small_max : SMALL_MAX;
    const int bk = (n == 0) ? -1
                 : (n <= lo ? 0 : (n <= b.small_max ? 1 : (n <= b.medium_max ? 2 : 3)));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t pos = warp_append(&b.ctr[1 + q], bk == q);
      if (bk == q) {
        b.bucket[(size_t)q * ng + pos] = g;
        // the warp kernel reads its gridboxes' ranges and RNG slots with the list entry
        if (q < 2) b.brec[(size_t)q * ng + pos] = make_uint4(g, c.gstart[g], n, b.slot[g]);
      }
    }
  }
}

// reduction of the condensed mass and iterations of one gridbox + state update and budgets
// (effect_on_thermodynamic_state, condensation.cpp:72-80 and :126-138; monitor, condensation.hpp:149)
__device__ __forceinline__ void cond_commit(const DevCtx& c, uint32_t g, double totmass,
                                            unsigned long long totits) {
  if (c.p.do_alter_thermo) {
    const double R0cubed_VOL0 = R0 * R0 * R0 / VOL0;
    const double totrho = totmass / c.volume[g] * R0cubed_VOL0;
    const double rho_dry = dry_air_density(c.press[g], c.temp[g], c.qvap[g]);
    const double dq = totrho / rho_dry;
    c.qvap[g] -= dq;
    c.qcond[g] += dq;
    c.temp[g] += (Latent_v / moist_specifc_heat(c.qvap[g], c.qcond[g])) * dq;
  }
  c.cond_mass[g] += totmass;
  c.nr_iters[g] += totits;
}

// ---- the gridboxes' share of a condensation sub-step after its solves ----
// The condensed mass of each gridbox's superdroplets added in their order (warp_batch_sums, the
// reference's sequential reduction, condensation.cpp:29-35), their Newton iterations, then the
// state update (cond_commit). Empty gridboxes commit a zero change, as the reference's do.
// Gridboxes of more than SEQ_BIG superdroplets are listed for k_b_commit_big instead.
__global__ void __launch_bounds__(SEQ_THREADS) k_b_commit(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, uint32_t per) {
  __shared__ double dbuf[SEQ_THREADS / 32][SEQ_WIN];
  __shared__ uint32_t ubuf[SEQ_THREADS / 32][SEQ_WIN];
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t g0 = warp * per; g0 < c.ngbxs; g0 += nwarps * per) {
    const uint32_t nb = c.ngbxs - g0 < per ? c.ngbxs - g0 : per;
    const bool own = (uint32_t)lane < nb;
    const bool big = own && c.gcount[g0 + lane] > SEQ_BIG;
    const uint32_t pos = warp_append(&b.ctr[10], big);
    if (big) b.big[pos] = g0 + lane;
    double m;
    unsigned long long it;
    if (b.qm) {  // qcond from the moved superdroplets first (k_b_qcond's sums, from pass A)
      warp_batch_sums(
          c, g0, nb, dbuf[wib], ubuf[wib], [&](uint32_t i) { return b.qm[i]; },
          [](uint32_t) { return 0u; }, m, it, true);
      if (own && !big) set_qcond(c, g0 + lane, m);
    }
    // (positions past a gridbox's valid superdroplets are loaded but not added)
    warp_batch_sums(
        c, g0, nb, dbuf[wib], ubuf[wib], [&](uint32_t i) { return b.dm[i]; },
        [&](uint32_t i) { return b.its[i]; }, m, it, true);
    if (own && !big) cond_commit(c, g0 + lane, m, it);
  }
}
// the listed gridboxes of more than SEQ_BIG superdroplets, or all of a domain with few (`all`; then
// k_b_commit is not launched), a warp each (the same sums and updates as k_b_commit's lanes make)
__global__ void __launch_bounds__(SEQ_THREADS) k_b_commit_big(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, int all) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t nbig = all ? c.ngbxs : b.ctr[10];
  for (uint32_t j = warp; j < nbig; j += nwarps) {
    const uint32_t g = all ? j : b.big[j];
    const uint32_t s = c.gstart[g], e = s + c.gcount[g];
    double mq, md;
    unsigned long long it;
    warp_seq_sums(s, e, b.qm, b.dm, b.its, mq, md, it);
    if ((threadIdx.x & 31) == 0) {
      if (b.qm) set_qcond(c, g, mq);  // qcond from the moved superdroplets first
      cond_commit(c, g, md, it);
    }
  }
}

// One pair (2jj, 2jj+1) of the shuffled gridbox, collisions.hpp:140-158, on the drops at indexes
// a and bb of the staged arrays. Few pairs collide in a step: a collision needs prob >= 1 or
// phi_coll < prob (coalescence_gamma's and breakup's own tests), so a pair whose first random
// number is above an upper bound of its probability, below 1, is left as it is without
// evaluating the probability. The bound is single precision (pair_bound.h); it replaces three FP64
// divisions, and two correctly rounded powers per pair (Simmel's velocities, a kernel over all
// superdroplets and 16 bytes of traffic for each before).
static __device__ __noinline__ uint32_t collide_pair_exact(const cleo_b200_params& p,
                                                           unsigned long long* sx, double* sr,
                                                           double* sm, uint32_t a, uint32_t bb,
                                                           double scale_p, double VOLUME,
                                                           uint64_t key, uint64_t slot_coll,
                                                           const Where& w) {
  const bool swap = sx[a] < sx[bb];  // d1 is the droplet of larger xi
  const uint32_t i1 = swap ? bb : a, i2 = swap ? a : bb;
  Drop d1{sx[i1], sr[i1], sm[i1]};
  Drop d2{sx[i2], sr[i2], sm[i2]};
  const double tv1 = pair_tv(p, d1.r), tv2 = pair_tv(p, d2.r);
  const double prob = scale_p * (double)d1.xi * pair_prob_tv(p, d1.r, d2.r, tv1, tv2, VOLUME);
  const double phi_coll = cleo_rng_to_unit(cleo_rng_u64(key, slot_coll));
  const double phi_out = cleo_rng_to_unit(cleo_rng_u64(key, slot_coll + 1));
  // the pair's terminal velocities are the flag's too when both are Simmel's (pair_tv)
  const bool tv_known = p.coll_prob == CLEO_PROB_LONG && p.flag_tv == CLEO_TV_SIMMEL;
  const uint32_t nn = enact_collision(p, d1, d2, prob, phi_coll, phi_out, w, tv_known, tv1, tv2);
  sx[i1] = d1.xi;
  sr[i1] = d1.r;
  sm[i1] = d1.msol;
  sx[i2] = d2.xi;
  sr[i2] = d2.r;
  sm[i2] = d2.msol;
  return nn;
}
__device__ __forceinline__ uint32_t collide_pair(const cleo_b200_params& p, unsigned long long* sx,
                                                 double* sr, double* sm, uint32_t a, uint32_t bb,
                                                 uint32_t n, float coef, double VOLUME,
                                                 uint64_t key, uint64_t slot_pairs, uint32_t jj,
                                                 const Where& w) {
  const unsigned long long xa = sx[a], xb = sx[bb];
  const uint64_t u = cleo_rng_u64(key, slot_pairs + 2ull * jj);
  if (pair_apart(p, coef, (float)sr[a], (float)sr[bb], pair_xi(xa, xb), pair_phi(u))) return 0;
  const uint32_t npairs = n / 2;
  const double scale_p = (double)n * ((double)n - 1.0) / (2.0 * (double)npairs);
  return collide_pair_exact(p, sx, sr, sm, a, bb, scale_p, VOLUME, key, slot_pairs + 2ull * jj, w);
}

// Fisher-Yates (shuffle.hpp:80-87) applies swap(p[i], p[J[i]]) for i = n-1 down to 1 to the
// identity. The element that ends at position k started at the position reached from k by
// applying the transpositions (s, J[s]) for s = 1, 2, ..., n-1 (the swaps in reverse order), so
// every thread can find the origin of its own positions without the sequential loop.
template <class JT>
__device__ __forceinline__ uint32_t fy_origin(const JT* J, uint32_t n, uint32_t k) {
  uint32_t pos = k;
  for (uint32_t s = 1; s < n; ++s) {
    const uint32_t j = J[s];
    pos = (pos == s) ? j : ((pos == j) ? s : pos);
  }
  return pos;
}

// ---- small gridboxes: persistent, one warp per gridbox ----
// CAP (64 or 128) is the number of per-warp slots; every lane holds CAP / 32 of them.
// Radius, solute mass and multiplicity of each gridbox are staged in shared memory by bulk
// copies (TMA, cp.async.bulk) into one of two buffers per warp: the next gridbox's copies are
// in flight while the current one is processed. A copy starts at the even element at or below
// the gridbox's first superdroplet (16-byte alignment) and covers an even number of elements, so
// it may read one element past the range (the SoA arrays carry two elements of padding).

// The 64-slot variant stages all seven 8-byte fields (r, msol, xi, coordinates, id), so its
// write-back reads shared memory instead of gathering the coordinates and ids from global memory
// in shuffled order; the 128-slot variant stages r, msol and xi (seven fields of 128 slots would
// leave room for fewer CTAs per SM than its registers allow).
template <int CAP>
struct SmallLayout {
  static constexpr bool ALL = CAP <= 64;
  static constexpr uint32_t NF = ALL ? 7 : 3;  // staged fields per buffer
  static constexpr uint32_t BUF = CAP + 2;  // elements per staged field
  static constexpr uint32_t FIELD = BUF * 8;
  static constexpr uint32_t OFF_BAR = 2 * NF * FIELD;
  static constexpr uint32_t WARP_BYTES = OFF_BAR + 16;
  static constexpr uint32_t BYTES = WARP_BYTES * B_WARPS;
  static_assert(FIELD % 16 == 0 && WARP_BYTES % 16 == 0, "bulk-copy buffers must be aligned");
};

// ---- the shuffles of the warp kernel's gridboxes, a thread each ----
// Fisher-Yates as the reference runs it (shuffle.hpp:80-87): swap(p[i], p[J[i]]) for i = n-1 down
// to 1, the draws in that order. A thread's permutation is bytes in words of its own bank (word w
// of lane l at [w][l]), so no two lanes' swaps conflict. Bound by instruction issue, some 60 for a
// draw and its swap with the lanes of a warp at their own lengths: 15 us for 4.6 M superdroplets,
// where building and walking the swaps' chains inside the warp kernel, a dependent lookup after
// another, took about a third of its 170 us. Word w of item it goes to
// perm[((it / 32) words + w) 32 + it % 32]: written coalesced, and read by the eight consecutive
// items that a CTA of the warp kernel holds from the same sectors.
__global__ void __launch_bounds__(B_THREADS)
k_b_perm(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, int nq) {
  __shared__ uint32_t sp[B_WARPS][WARP_MAX / 4][32];
  const uint32_t t_sdm = *b.tsdm;
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t warp = blockIdx.x * B_WARPS + wib, nwarps = gridDim.x * B_WARPS;
  uint32_t(*W)[32] = sp[wib];
  uint8_t* B = reinterpret_cast<uint8_t*>(&W[0][lane]);
  const auto at = [](uint32_t i) { return (i >> 2) * 128 + (i & 3); };
  for (int q = 0; q < nq; ++q) {
    const uint32_t count = b.ctr[1 + q];
    const uint4* list = b.brec + (size_t)q * c.ngbxs;
    const uint32_t words = (q == 0 ? SMALL_MAX : WARP_MAX) / 4;
    uint32_t* out = b.perm[q];
    for (uint32_t it0 = warp * 32; it0 < count; it0 += nwarps * 32) {
      const uint32_t it = it0 + lane;
      if (it >= count) continue;
      const uint4 rec = list[it];
      const uint32_t n = rec.z, nw = (n + 3) / 4;
      for (uint32_t w = 0; w < nw; ++w) W[w][lane] = 0x03020100u + 0x04040404u * w;
      // draw slot + k for i = n-1-k (cleo_rng_u64's counter advanced by one each)
      uint64_t z = cleo_rng_key(c.p.seed, t_sdm, rec.x) + ((uint64_t)rec.w + 1u) * CLEO_RNG_GOLDEN;
      for (uint32_t i = n - 1; i > 0; --i) {
        const uint64_t u = cleo_mix64(z);
        z += CLEO_RNG_GOLDEN;
        // cleo_rng_range(u, 0, i + 1) for i + 1 below 2^32
        const uint64_t m = i + 1;
        const uint32_t j =
            (uint32_t)(((u >> 32) * m + (((u & 0xFFFFFFFFull) * m) >> 32)) >> 32);
        const uint32_t oi = at(i), oj = at(j);
        const uint8_t t = B[oi];
        B[oi] = B[oj];
        B[oj] = t;
      }
      uint32_t* o = out + (size_t)(it >> 5) * words * 32 + lane;
      for (uint32_t w = 0; w < nw; ++w) o[w * 32] = W[w][lane];
    }
  }
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

template <int MINB, int CAP>
__global__ void __launch_bounds__(B_THREADS, MINB)
k_b_small(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, int q) {
  using L = SmallLayout<CAP>;
  constexpr int H = CAP / 32;
  constexpr uint32_t WORDS = CAP / 4;  // words of a gridbox's permutation (bytes)
  static_assert(CAP % 32 == 0 && CAP <= 128, "a word of the permutation per lane");
  const uint32_t t_sdm = *b.tsdm;
  const float bound_kernel = pair_bound_kernel(c.p);
  extern __shared__ __align__(16) unsigned char smem_small[];
  const cleo_b200_params& p = c.p;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  unsigned char* wsm = smem_small + wib * L::WARP_BYTES;
  uint64_t* bar = reinterpret_cast<uint64_t*>(wsm + L::OFF_BAR);
  const auto field = [&](int buf, int f) { return wsm + (buf * L::NF + f) * L::FIELD; };
  const uint32_t count = b.ctr[1 + q];
  const uint4* list = b.brec + (size_t)q * c.ngbxs;  // {gridbox, start, count, RNG slot}
  // stage a gridbox's fields into buffer buf (lane 0)
  const auto stage = [&](int buf, const uint4& rec) {
    const uint32_t base = rec.y, n = rec.z;
    const uint32_t a0 = base & ~1u;
    const uint32_t bytes = ((n + (base & 1u) + 1u) & ~1u) * 8u;
    fence_async_smem();  // earlier generic accesses of the buffer precede the async writes
    mbar_expect_tx(&bar[buf], L::NF * bytes);
    bulk_g2s(field(buf, 0), c.sd.r + a0, bytes, &bar[buf]);
    bulk_g2s(field(buf, 1), c.sd.msol + a0, bytes, &bar[buf]);
    bulk_g2s(field(buf, 2), c.sd.xi + a0, bytes, &bar[buf]);
    if constexpr (L::ALL) {
      bulk_g2s(field(buf, 3), c.sd.c3 + a0, bytes, &bar[buf]);
      bulk_g2s(field(buf, 4), c.sd.c1 + a0, bytes, &bar[buf]);
      bulk_g2s(field(buf, 5), c.sd.c2 + a0, bytes, &bar[buf]);
      bulk_g2s(field(buf, 6), c.sd.id + a0, bytes, &bar[buf]);
    }
  };
  // static assignment (item = warp + k * warps): no shared counter; a gridbox's list record is
  // loaded two gridboxes ahead and its copies are issued one gridbox ahead
  const uint32_t nwarps = gridDim.x * B_WARPS;
  uint32_t item = blockIdx.x * B_WARPS + wib;
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  uint4 rec_next = item < count ? list[item] : none;
  uint4 rec_after = item + nwarps < count ? list[item + nwarps] : none;
  // the item's permutation, a word per lane, loaded a gridbox ahead (k_b_perm)
  const uint32_t* perm = b.perm[q];
  const auto perm_word = [&](uint32_t it) {
    return (uint32_t)lane < WORDS ? perm[((size_t)(it >> 5) * WORDS + lane) * 32 + (it & 31)] : 0u;
  };
  uint32_t word_next = item < count ? perm_word(item) : 0u;
  uint32_t parity = 0;  // bit k: the phase of bar[k] to wait for
  int cur = 0;
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    if (item < count) stage(0, rec_next);
  }
  __syncwarp();
  for (; item < count; item += nwarps) {
    const uint4 rec = rec_next;
    const uint32_t g = rec.x, base = rec.y, n = rec.z;
    const bool has_next = item + nwarps < count;
    const uint32_t word = word_next;
    if (has_next) word_next = perm_word(item + nwarps);
    rec_next = rec_after;
    rec_after = item + 2 * nwarps < count ? list[item + 2 * nwarps] : none;
    // the next gridbox's copies go out before this one's wait
    if (has_next && lane == 0) stage(cur ^ 1, rec_next);
    const double VOLUME = c.volume[g] * VOL0;  // issued before the wait
    if (!mbar_wait_bounded(&bar[cur], (parity >> cur) & 1u, MBAR_TRIES)) {
      // the step fails with CLEO_ERR_TIMEOUT; before the warp leaves, the copies still in flight
      // into either buffer get a bounded wait to land
      if (lane == 0) Where{c.err, g, base}.fail(CLEO_ERR_TIMEOUT);
      mbar_wait_bounded(&bar[cur], (parity >> cur) & 1u, MBAR_TRIES);
      if (has_next) mbar_wait_bounded(&bar[cur ^ 1], (parity >> (cur ^ 1)) & 1u, MBAR_TRIES);
      return;
    }
    parity ^= 1u << cur;
    const uint32_t off = base & 1u;
    double* s_r = reinterpret_cast<double*>(field(cur, 0)) + off;
    double* s_m = reinterpret_cast<double*>(field(cur, 1)) + off;
    unsigned long long* s_x = reinterpret_cast<unsigned long long*>(field(cur, 2)) + off;
    const uint64_t key = cleo_rng_key(p.seed, t_sdm, g);
    const uint64_t slot_pairs = (uint64_t)rec.w + (n - 1);
    const uint32_t npairs = n / 2;
    const float coef = pair_bound_coef(bound_kernel, n, VOLUME);
    uint32_t nnull = 0;
    for (uint32_t j0 = 0; j0 < npairs; j0 += 32) {  // positions 2jj, 2jj + 1: word jj / 2
      const uint32_t jj = j0 + lane;
      const uint32_t pw = __shfl_sync(0xFFFFFFFFu, word, (jj >> 1) & 31) >> (16 * (jj & 1));
      if (jj < npairs) {
        const uint32_t a = pw & 0xFFu, bb = (pw >> 8) & 0xFFu;
        const Where w{c.err, g, (uint64_t)base + 2 * jj};
        nnull += collide_pair(p, s_x, s_r, s_m, a, bb, n, coef, VOLUME, key, slot_pairs, jj, w);
      }
    }
    __syncwarp();
    const uint32_t totnull = warp_sum_u(nnull);
    const uint32_t nvalid = n - totnull;
    // destinations: valid superdroplets in shuffled order, then the nulls (collisions.hpp:240-248)
    uint32_t src[H], dst[H];
    double c3v[L::ALL ? 1 : H], c1v[L::ALL ? 1 : H], c2v[L::ALL ? 1 : H];
    unsigned long long idv[L::ALL ? 1 : H];
    uint32_t cval = 0, cnull = 0;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      if (32u * h >= n) break;  // uniform across the warp
      const uint32_t k = lane + 32 * h;
      const bool act = k < n;
      const uint32_t pw = __shfl_sync(0xFFFFFFFFu, word, (k >> 2) & 31);
      src[h] = act ? (pw >> (8 * (k & 3))) & 0xFFu : 0;
      const bool valid = act && s_x[src[h]] != 0;
      const unsigned mv = __ballot_sync(0xFFFFFFFFu, valid);
      const unsigned mn = __ballot_sync(0xFFFFFFFFu, act && !valid);
      const unsigned lt = (1u << lane) - 1u;
      dst[h] = valid ? cval + __popc(mv & lt) : nvalid + cnull + __popc(mn & lt);
      cval += __popc(mv);
      cnull += __popc(mn);
      if constexpr (!L::ALL) {
        if (act) {
          const uint32_t s = base + src[h];
          c3v[h] = c.sd.c3[s];
          c1v[h] = c.sd.c1[s];
          c2v[h] = c.sd.c2[s];
          idv[h] = c.sd.id[s];
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const uint32_t k = lane + 32 * h;
      if (k < n) {
        const uint32_t o = base + dst[h];
        c.sd.r[o] = s_r[src[h]];
        c.sd.msol[o] = s_m[src[h]];
        c.sd.xi[o] = s_x[src[h]];
        if (dst[h] >= nvalid) c.sd.gbx[o] = OOB;  // the range's indexes are g already
        if constexpr (L::ALL) {
          c.sd.c3[o] = reinterpret_cast<const double*>(field(cur, 3))[off + src[h]];
          c.sd.c1[o] = reinterpret_cast<const double*>(field(cur, 4))[off + src[h]];
          c.sd.c2[o] = reinterpret_cast<const double*>(field(cur, 5))[off + src[h]];
          c.sd.id[o] = reinterpret_cast<const unsigned long long*>(field(cur, 6))[off + src[h]];
        } else {
          c.sd.c3[o] = c3v[h];
          c.sd.c1[o] = c1v[h];
          c.sd.c2[o] = c2v[h];
          c.sd.id[o] = idv[h];
        }
      }
    }
    __syncwarp();  // every lane is done with buffer cur before it is staged into again
    if (lane == 0) {
      c.gcount[g] = nvalid;
      b.slot[g] = (uint32_t)(slot_pairs + 2ull * npairs);
    }
    cur ^= 1;
  }
}

// Origins of the shuffled positions of a gridbox of n (2 .. CHAIN_MAX) superdroplets for a whole
// CTA, by the chains the warp kernel follows (see k_b_small): FIRST[v] = the first swap index s
// with J[s] = v, NEXT[s] = the next swap index after s with the same J value. The pairs
// (J[s], s), s = 1 .. n-1, are ordered by a bitonic sort of the 32-bit keys J[s] << 16 | s in
// shared memory (`keys`, a power of two >= n - 1 entries), so that equal values lie together in
// increasing s; FIRST and NEXT (n entries each, any memory) are read off the sorted keys, and
// each thread then walks the chains of its positions (about ln n lookups each). P receives the
// origins, as fy_origin computes them. Ends with a barrier.
constexpr uint32_t CHAIN_MAX = 16384;  // keys of up to 16384 swaps: 64 KB of shared memory
// the keys, FIRST and NEXT of up to CHAIN_MAX swaps in shared memory (192 KB): the chain walks'
// dependent lookups stay on chip
constexpr uint32_t LARGE_SMEM = CHAIN_MAX * 4 * 3;
constexpr uint32_t LARGE_THREADS = 1024;  // a gridbox of thousands: four times B_THREADS
__device__ void cta_fy_origins(const uint32_t* J, uint32_t n, uint32_t* keys, uint32_t* FIRST,
                               uint32_t* NEXT, uint32_t* P) {
  constexpr uint32_t NONE = 0xFFFFFFFFu;
  const uint32_t tid = threadIdx.x, nt = blockDim.x;
  const uint32_t m = n - 1;  // swaps s = 1 .. n-1
  uint32_t mp = 1;
  while (mp < m) mp <<= 1;
  for (uint32_t i = tid; i < mp; i += nt) keys[i] = i < m ? (J[i + 1] << 16) | (i + 1) : NONE;
  for (uint32_t v = tid; v < n; v += nt) FIRST[v] = NEXT[v] = NONE;
  __syncthreads();
  for (uint32_t k = 2; k <= mp; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = tid; i < mp; i += nt) {
        const uint32_t l = i ^ j;
        if (l > i) {
          const uint32_t a = keys[i], bk = keys[l];
          if ((a > bk) == ((i & k) == 0)) {
            keys[i] = bk;
            keys[l] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = tid; i < m; i += nt) {
    const uint32_t v = keys[i] >> 16, sidx = keys[i] & 0xFFFFu;
    if (i == 0 || (keys[i - 1] >> 16) != v) FIRST[v] = sidx;
    if (i + 1 < m && (keys[i + 1] >> 16) == v) NEXT[sidx] = keys[i + 1] & 0xFFFFu;
  }
  __syncthreads();
  for (uint32_t k = tid; k < n; k += nt) {
    uint32_t cur = k == 0 ? 0u : J[k];
    uint32_t nx = k == 0 ? FIRST[0] : NEXT[k];
    while (nx != NONE) {  // strictly increasing, so at most n hops
      cur = nx;
      nx = FIRST[cur];
    }
    P[k] = cur;
  }
  __syncthreads();
}

// ---- medium and large gridboxes: one CTA per gridbox ----
// medium: staged in shared memory with the non-staged fields permuted through registers;
// large: staged in global scratch arrays, the shuffle's chain tables in LARGE_SMEM of shared memory.
template <bool LARGE>
__global__ void __launch_bounds__(LARGE ? LARGE_THREADS : B_THREADS)
k_b_cta(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b) {
  const uint32_t t_sdm = *b.tsdm;
  const float bound_kernel = pair_bound_kernel(c.p);
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t shw[40];
  __shared__ uint32_t s_item;
  __shared__ uint64_t s_bar;  // completion of the medium path's bulk copies
  constexpr uint32_t PT = MEDIUM_MAX / B_THREADS;  // superdroplets per thread (medium)
  constexpr uint32_t NT = LARGE ? LARGE_THREADS : B_THREADS;  // threads of the block
  constexpr uint32_t MBUF = MEDIUM_MAX + 2;        // staged elements per field (medium)
  const cleo_b200_params& p = c.p;
  const int tid = threadIdx.x;
  const uint32_t q_idx = LARGE ? 3 : 2;
  const uint32_t count = b.ctr[1 + q_idx];
  const uint32_t* list = b.bucket + (size_t)q_idx * c.ngbxs;
  uint32_t bar_parity = 0;
  if (!LARGE) {
    if (tid == 0) mbar_init(&s_bar, 1);
    __syncthreads();
  }
  while (true) {
    if (tid == 0) s_item = atomicAdd(&b.ctr[5 + q_idx], 1u);
    __syncthreads();
    const uint32_t item = s_item;
    __syncthreads();
    if (item >= count) break;
    const uint32_t g = list[item];
    const uint32_t base = c.gstart[g];
    const uint32_t n = c.gcount[g];
    const uint64_t key = cleo_rng_key(p.seed, t_sdm, g);
    const uint64_t slot = b.slot[g];
    // medium: r, msol, xi staged in shared memory by bulk copies (TMA) from the even element at
    // or below the gridbox's first superdroplet (16-byte alignment; the SoA arrays' padding
    // covers the element a copy may read past the range); large: global scratch
    const uint32_t off = base & 1u;
    double* Sr = LARGE ? c.scr_r + base : reinterpret_cast<double*>(smem) + off;
    double* Sm = LARGE ? c.scr_m + base : reinterpret_cast<double*>(smem) + MBUF + off;
    unsigned long long* Sx = LARGE ? c.scr_x + base
                                   : reinterpret_cast<unsigned long long*>(smem) + 2 * MBUF + off;
    uint32_t* P = LARGE ? c.scr_p + base : reinterpret_cast<uint32_t*>(smem + 24 * MBUF);
    uint32_t* J = LARGE ? c.scr_j + base
                        : reinterpret_cast<uint32_t*>(smem + 24 * MBUF + 4 * MEDIUM_MAX);
    if (!LARGE) {
      if (tid == 0) {  // the previous gridbox's accesses ended at the barriers above
        const uint32_t bytes = ((n + off + 1u) & ~1u) * 8u;
        const uint32_t a0 = base & ~1u;
        fence_async_smem();
        mbar_expect_tx(&s_bar, 3u * bytes);
        bulk_g2s(smem, c.sd.r + a0, bytes, &s_bar);
        bulk_g2s(smem + 8 * MBUF, c.sd.msol + a0, bytes, &s_bar);
        bulk_g2s(smem + 16 * MBUF, c.sd.xi + a0, bytes, &s_bar);
      }
      // every thread waits with a bound; the outcome is agreed by the whole block
      const bool ok = __syncthreads_and(mbar_wait_bounded(&s_bar, bar_parity, MBAR_TRIES) ? 1 : 0);
      if (!ok) {
        if (tid == 0) Where{c.err, g, base}.fail(CLEO_ERR_TIMEOUT);
        mbar_wait_bounded(&s_bar, bar_parity, MBAR_TRIES);  // let the copies in flight land
        return;
      }
      bar_parity ^= 1u;
    }
    for (uint32_t k = tid; k < n; k += NT) {
      if (LARGE) {
        Sr[k] = c.sd.r[base + k];
        Sm[k] = c.sd.msol[base + k];
        Sx[k] = c.sd.xi[base + k];
      }
      if (k >= 1) J[k] = (uint32_t)cleo_rng_range(cleo_rng_u64(key, slot + (n - 1 - k)), 0, (uint64_t)k + 1);
    }
    __syncthreads();
    if (n <= FY_PARALLEL_MAX) {  // every thread traces its own positions
      for (uint32_t k = tid; k < n; k += NT) P[k] = fy_origin(J, n, k);
    } else if (LARGE && n <= CHAIN_MAX) {  // chains, as in the warp kernel (keys in smem)
      cta_fy_origins(J, n, reinterpret_cast<uint32_t*>(smem),
                     reinterpret_cast<uint32_t*>(smem) + CHAIN_MAX,
                     reinterpret_cast<uint32_t*>(smem) + 2 * CHAIN_MAX, P);
    } else {
      for (uint32_t k = tid; k < n; k += NT) P[k] = k;
      __syncthreads();
      if (tid == 0) {
        for (uint32_t it = n > 0 ? n - 1 : 0; it > 0; --it) {
          const uint32_t j = J[it];
          const uint32_t t = P[it];
          P[it] = P[j];
          P[j] = t;
        }
      }
    }
    __syncthreads();
    const uint64_t slot_pairs = slot + (n >= 1 ? n - 1 : 0);
    const uint32_t npairs = n / 2;
    const double VOLUME = c.volume[g] * VOL0;
    const float coef = pair_bound_coef(bound_kernel, n, VOLUME);
    uint32_t nnull = 0;
    for (uint32_t jj = tid; jj < npairs; jj += NT) {
      const uint32_t a = P[2 * jj], bb = P[2 * jj + 1];
      const Where w{c.err, g, (uint64_t)base + 2 * jj};
      nnull += collide_pair(p, Sx, Sr, Sm, a, bb, n, coef, VOLUME, key, slot_pairs, jj, w);
    }
    const uint32_t totnull = block_sum(nnull, shw);
    const uint32_t nvalid = n - totnull;
    uint32_t cval = 0, cnull = 0;
    // destination of shuffled position k; J becomes the inverse map q -> source
    for (uint32_t k0 = 0; k0 < n; k0 += NT) {
      const uint32_t k = k0 + tid;
      const bool act = k < n;
      const uint32_t src = act ? P[k] : 0;
      const bool valid = act && Sx[src] != 0;
      uint32_t tv, tn;
      const uint32_t ev = block_excl_scan(valid ? 1u : 0u, shw, tv);
      const uint32_t en = block_excl_scan((act && !valid) ? 1u : 0u, shw, tn);
      if (act) J[valid ? (cval + ev) : (nvalid + cnull + en)] = src;
      cval += tv;
      cnull += tn;
    }
    __syncthreads();
    if (LARGE) {
      for (uint32_t q = tid; q < n; q += NT) {
        const uint32_t s = base + J[q], o = base + q;
        c.scr_c3[o] = c.sd.c3[s];
        c.scr_c1[o] = c.sd.c1[s];
        c.scr_c2[o] = c.sd.c2[s];
        c.scr_id[o] = c.sd.id[s];
      }
      __syncthreads();
      for (uint32_t q = tid; q < n; q += NT) {
        const uint32_t o = base + q;
        const uint32_t src = J[q];
        c.sd.r[o] = Sr[src];
        c.sd.msol[o] = Sm[src];
        c.sd.xi[o] = Sx[src];
        if (q >= nvalid) c.sd.gbx[o] = OOB;
        c.sd.c3[o] = c.scr_c3[o];
        c.sd.c1[o] = c.scr_c1[o];
        c.sd.c2[o] = c.scr_c2[o];
        c.sd.id[o] = c.scr_id[o];
      }
    } else {
      double c3v[PT], c1v[PT], c2v[PT];
      unsigned long long idv[PT];
#pragma unroll
      for (uint32_t h = 0; h < PT; ++h) {
        const uint32_t q = tid + h * B_THREADS;
        if (q < n) {
          const uint32_t s = base + J[q];
          c3v[h] = c.sd.c3[s];
          c1v[h] = c.sd.c1[s];
          c2v[h] = c.sd.c2[s];
          idv[h] = c.sd.id[s];
        }
      }
      __syncthreads();
#pragma unroll
      for (uint32_t h = 0; h < PT; ++h) {
        const uint32_t q = tid + h * B_THREADS;
        if (q < n) {
          const uint32_t o = base + q;
          const uint32_t src = J[q];
          c.sd.r[o] = Sr[src];
          c.sd.msol[o] = Sm[src];
          c.sd.xi[o] = Sx[src];
          if (q >= nvalid) c.sd.gbx[o] = OOB;
          c.sd.c3[o] = c3v[h];
          c.sd.c1[o] = c1v[h];
          c.sd.c2[o] = c2v[h];
          c.sd.id[o] = idv[h];
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      c.gcount[g] = nvalid;
      b.slot[g] = (uint32_t)(slot_pairs + 2ull * npairs);
    }
  }
}

// reset of the per-gridbox slot offsets at the start of an SDM step and of the bucket counters
// the device copy of the SDM step time: set before a step whose time the device does not hold,
// advanced by the last kernel of every step (so one captured step graph serves every step)
__global__ void k_b_set_t(BatchScratch b, uint32_t t) { *b.tsdm = t; }
// the SDM step's end: its start time advanced; with zero_slot0 (a one-gridbox domain, whose step
// has no per-gridbox reset) the gridbox's RNG slot is reset for the next step here
__global__ void k_b_advance_t(BatchScratch b, uint32_t dt, int zero_slot0) {
  *b.tsdm += dt;
  if (zero_slot0) b.slot[0] = 0;
}

__global__ void k_b_reset(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, int slots) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (slots)
    for (uint32_t g = i; g < c.ngbxs; g += gridDim.x * blockDim.x) b.slot[g] = 0;
  if (i < 8) b.ctr[1 + i] = 0;  // bucket counts and heads
}

}  // namespace
