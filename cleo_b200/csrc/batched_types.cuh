// batched_types.cuh — sizes and scratch of the batched microphysics schedule (batched.cuh).
#pragma once

#include <cstdint>

namespace {

constexpr uint32_t SMALL_MAX = 64;   // largest gridbox of the warp kernel's 64-slot variant
constexpr uint32_t WARP_MAX = 128;   // and of its 128-slot variant (the default limit)
constexpr uint32_t MEDIUM_MAX = 1024;
// r, msol, xi (each with two elements of slack for the bulk copies' alignment), P, J
constexpr uint32_t MEDIUM_SMEM = 24 * (MEDIUM_MAX + 2) + 8 * MEDIUM_MAX;
constexpr uint32_t FY_PARALLEL_MAX = 256;  // gridboxes up to this size shuffle in parallel
constexpr int B_THREADS = 256;
constexpr uint32_t COST_CLASSES = 66;  // restarts, 64 quarter-octaves of sub-steps, those at 2^16
constexpr uint32_t LONG_RESTART = COST_CLASSES;  // restarts of many iterations, counted in class 0
constexpr uint32_t COST_CURSORS = COST_CLASSES + 1;
constexpr int B_WARPS = B_THREADS / 32;

struct BatchScratch {
  double* th_s;      // per gridbox supersaturation ratio
  double* th_ff;     // per gridbox diffusion factor
  double* th_ak;     // per gridbox Kohler factor akoh (kohler_a)
  double* th_a3;     // per gridbox activation_a3(akoh)
  double* th_u3;     // per gridbox unique_a3(akoh)
  double* dm;        // per superdroplet condensed mass x xi
  uint32_t* its;     // per superdroplet Newton iterations
  double* qm;        // per superdroplet condensate mass x xi before the solves, when the first
                     // condensation sub-step after motion also gives qcond (else null)
  double* zres;      // per deferred direct solve: pass A's iterate that pass B resumes from
  double* ffv;       // per deferred solve: pass A's diffusion factor over the ventilation factor
  uint32_t* lkeys;   // cost classes of deferred solves (restart_class, cost_class)
  uint32_t* lvals;   // positions of deferred solves
  uint32_t* ccnt;    // [COST_CLASSES] solves per class, then [COST_CURSORS] k_cond_place's cursors
  uint32_t* order;   // the deferred solves by class
  uint32_t* bucket;  // [4][ngbxs] gridbox lists per size bucket
  uint4* brec;       // [2][ngbxs] the warp kernel's buckets as {gridbox, start, count, RNG slot}
  uint32_t* perm[2];  // the shuffles of those buckets' gridboxes (k_b_perm): 16 and 32 words each
  uint32_t* slot;    // per gridbox RNG slot offset within the SDM step
  uint32_t* ctr;     // [0] deferred solves, [1..4] bucket counts, [5..8] bucket heads,
                     // [10] big gridboxes (commit)
  uint32_t* big;     // gridboxes whose condensation commit takes a warp each (k_b_commit_big)
  uint32_t* tsdm;    // the SDM step's start time (keys the injected random numbers)
  uint32_t small_max;   // gridboxes with 1..small_max superdroplets: warp kernel (<= WARP_MAX)
  uint32_t medium_max;  // small_max..medium_max: CTA kernel in shared memory (<= MEDIUM_MAX)
};

// scratch of the one-gridbox collision path (onebox.cuh)
constexpr uint32_t OB_NONE = 0xFFFFFFFFu;

struct OneBox {
  uint32_t* J;      // swap draws, index s (1 .. n-1)
  uint32_t* head;   // per value: its list of swap indexes; all empty between steps
  uint32_t* next;   // per swap index
  uint32_t* P;      // origin of shuffled position k
  uint32_t* vflag;  // 1 for a valid superdroplet at shuffled position q, scanned; n + 1 entries
  uint32_t* tsums;  // the scan's tile totals
  // these three 0 between steps:
  uint32_t* nnull;  // nulls made by this sub-step's collisions
  uint32_t* ninv;   // superdroplets left with multiplicity 0 (the flags' zeros)
  uint32_t* done;   // finished blocks of k_ob_gather
};

}  // namespace
