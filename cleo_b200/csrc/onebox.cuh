// onebox.cuh — collisions of a domain of one gridbox (the box model) across the whole GPU.
//
// A box model puts all its superdroplets (thousands) in one gridbox, so the per-gridbox kernels
// of batched.cuh run it on one CTA. Here each phase of the gridbox's collision step is a kernel
// over all its superdroplets or pairs, with the same results (collisions.hpp:140-248):
//   k_ob_draw    thread per swap index s >= 1: J[s], the Fisher-Yates draw (shuffle.hpp:80-87), and
//                s pushed onto the list of its value: HEAD[J[s]] = s, NEXT[s] = the one before
//   k_ob_chains  thread per value: its list put in ascending order, so that HEAD[v] is the first
//                swap index with J = v and NEXT[s] the next one after s with the same value (a list
//                of one, the usual case, is in order already)
//                (k_ob_front does these two and the walks in one block's shared memory for stores
//                of up to OB_FRONT_MAX slots)
//   k_ob_pairs   thread per pair (2jj, 2jj+1) of the shuffled order: the origins P of its two
//                positions (the end of the chain J[k] -> NEXT[k] -> HEAD[.] -> ..., 0 ->
//                HEAD[0] -> ... for k = 0), collide_pair on those superdroplets in place (pairs
//                are disjoint), nulls counted, then the two valid flags in shuffled order (its
//                own pair's collision is the only one that touches them); the thread after the
//                last pair takes an odd last position and the flags' end entry
//   (exclusive scan of the flags, where any is zero: three launches on large stores, inside
//   k_ob_gather on the others)
//   k_ob_gather  thread per destination: valid superdroplets in shuffled order, then the nulls, into
//                the other buffer (which the host then makes the current one); it empties the lists
//                for the next step, and its last block sets the count and RNG slot, and the time
//                after a step's last sub-step
// The host takes this path for domains of one gridbox; every array is sized by the store's slots.
// The step is a chain of short kernels, bound by their number and each one's latency. With a counting
// sort of the swap indexes in place of the lists (counts, scan, placement), a scratch copy of the
// records and a tail kernel it took 6 launches and 35 us on 8192 superdroplets, 15 and 70 us on
// 131072; now 3 and 28, 7 and 55.
#pragma once

namespace {

__global__ void k_ob_draw(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b,
                          OneBox o) {
  const uint32_t n = c.gcount[0];
  const uint64_t key = cleo_rng_key(c.p.seed, *b.tsdm, 0);
  const uint64_t slot = b.slot[0];
  for (uint32_t s = 1 + blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const uint32_t j =
        (uint32_t)cleo_rng_range(cleo_rng_u64(key, slot + (n - 1 - s)), 0, (uint64_t)s + 1);
    o.J[s] = j;
    o.next[s] = atomicExch(&o.head[j], s);
  }
}
__global__ void k_ob_chains(const __grid_constant__ DevCtx c, OneBox o) {
  constexpr uint32_t MAX = 24;  // longer lists (values near 0 of large stores) are relinked in place
  const uint32_t n = c.gcount[0];
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    uint32_t s = o.head[v];
    if (s == OB_NONE) continue;
    uint32_t nx = o.next[s];
    if (nx == OB_NONE) continue;
    uint32_t list[MAX], k = 0;
    while (s != OB_NONE && k < MAX) {  // insertion sort as they come
      uint32_t i = k++;
      while (i > 0 && list[i - 1] > s) {
        list[i] = list[i - 1];
        --i;
      }
      list[i] = s;
      s = o.next[s];
    }
    o.head[v] = list[0];
    for (uint32_t i = 0; i < k; ++i) o.next[list[i]] = i + 1 < k ? list[i + 1] : OB_NONE;
    while (s != OB_NONE) {  // the rest, each linked into its place
      nx = o.next[s];
      uint32_t prev = OB_NONE, at = o.head[v];
      while (at != OB_NONE && at < s) {
        prev = at;
        at = o.next[at];
      }
      o.next[s] = at;
      if (prev == OB_NONE)
        o.head[v] = s;
      else
        o.next[prev] = s;
      s = nx;
    }
  }
}
// The front of the step (k_ob_draw, k_ob_chains and the chain walks: the same values) in one block
// for a store of up to OB_FRONT_MAX slots, the tables in shared memory: HEAD as 32-bit words, J and
// NEXT as 16-bit indexes. The origins P go to global memory, so k_ob_pairs reads them instead of
// walking the chains in global memory.
constexpr uint32_t OB_FRONT_THREADS = 1024;
// One block's time grows with the store, the separate kernels' hardly (a step of 8000, 12000, 15900,
// 20000 and 27900 superdroplets: 28.8, 32.2, 36.8, 38.8 and 47.2 us by the one, 33.0, 34.7, 36.8,
// 36.7 and 37.8 by the others), so the line lies where they meet.
constexpr uint32_t OB_FRONT_MAX = 16000;
constexpr size_t ob_front_smem(uint32_t slots) { return (size_t)slots * 8 + 16; }
__global__ void __launch_bounds__(OB_FRONT_THREADS)
k_ob_front(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, OneBox o) {
  extern __shared__ __align__(16) unsigned char ob_smem[];
  constexpr uint32_t NONE = 0xFFFFu;  // no index: n <= OB_FRONT_MAX < 2^16 - 1
  const uint32_t n = c.gcount[0];
  uint32_t* head = reinterpret_cast<uint32_t*>(ob_smem);
  uint16_t* J = reinterpret_cast<uint16_t*>(head + n);
  uint16_t* nxt = J + n;
  const uint32_t t = threadIdx.x;
  for (uint32_t v = t; v < n; v += OB_FRONT_THREADS) head[v] = NONE;
  __syncthreads();
  const uint64_t key = cleo_rng_key(c.p.seed, *b.tsdm, 0);
  const uint64_t slot = b.slot[0];
#pragma unroll 4
  for (uint32_t s = 1 + t; s < n; s += OB_FRONT_THREADS) {
    const uint32_t j =
        (uint32_t)cleo_rng_range(cleo_rng_u64(key, slot + (n - 1 - s)), 0, (uint64_t)s + 1);
    J[s] = (uint16_t)j;
    nxt[s] = (uint16_t)atomicExch(&head[j], s);
  }
  __syncthreads();
  for (uint32_t v = t; v < n; v += OB_FRONT_THREADS) {  // lists of two or more into order
    uint32_t s = head[v];
    if (s == NONE || nxt[s] == NONE) continue;
    uint32_t first = s;
    s = nxt[s];
    nxt[first] = (uint16_t)NONE;
    while (s != NONE) {
      const uint32_t rest = nxt[s];
      if (s < first) {
        nxt[s] = (uint16_t)first;
        first = s;
      } else {
        uint32_t p = first, q = nxt[p];
        while (q != NONE && q < s) {
          p = q;
          q = nxt[p];
        }
        nxt[s] = (uint16_t)q;
        nxt[p] = (uint16_t)s;
      }
      s = rest;
    }
    head[v] = first;
  }
  __syncthreads();
  // the chain walks (ob_origin's), four positions a thread side by side: strictly increasing, so
  // at most n hops
  constexpr uint32_t WIDE = 4;
  for (uint32_t k0 = t; k0 < n; k0 += WIDE * OB_FRONT_THREADS) {
    uint32_t cur[WIDE], nx[WIDE];
    bool more = false;
#pragma unroll
    for (uint32_t q = 0; q < WIDE; ++q) {
      const uint32_t k = k0 + q * OB_FRONT_THREADS;
      cur[q] = k > 0 && k < n ? (uint32_t)J[k] : 0u;
      nx[q] = k < n ? (k == 0 ? head[0] : (uint32_t)nxt[k]) : NONE;
      more |= nx[q] != NONE;
    }
    while (more) {
      more = false;
#pragma unroll
      for (uint32_t q = 0; q < WIDE; ++q) {
        if (nx[q] != NONE) {
          cur[q] = nx[q];
          nx[q] = head[cur[q]];
          more |= nx[q] != NONE;
        }
      }
    }
#pragma unroll
    for (uint32_t q = 0; q < WIDE; ++q) {
      const uint32_t k = k0 + q * OB_FRONT_THREADS;
      if (k < n) o.P[k] = cur[q];
    }
  }
}
// the origin of shuffled position k (what fy_origin computes), by the chains
__device__ __forceinline__ uint32_t ob_origin(const OneBox& o, uint32_t k) {
  uint32_t cur = k == 0 ? 0u : o.J[k];
  uint32_t nx = k == 0 ? o.head[0] : o.next[k];
  while (nx != OB_NONE) {  // strictly increasing, so at most n hops
    cur = nx;
    nx = o.head[cur];
  }
  return cur;
}
// walked: the origins P are in global memory already (k_ob_front), else found here by the chains
__global__ void k_ob_pairs(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b,
                           OneBox o, int walked) {
  const uint32_t n = c.gcount[0], base = c.gstart[0];
  const uint32_t npairs = n / 2;
  const uint64_t key = cleo_rng_key(c.p.seed, *b.tsdm, 0);
  const uint64_t slot_pairs = (uint64_t)b.slot[0] + (n >= 1 ? n - 1 : 0);
  const double VOLUME = c.volume[0] * VOL0;
  const float coef = pair_bound_coef(pair_bound_kernel(c.p), n, VOLUME);
  uint32_t nnull = 0, ninv = 0;
  for (uint32_t jj = blockIdx.x * blockDim.x + threadIdx.x; jj <= npairs;
       jj += gridDim.x * blockDim.x) {
    if (jj < npairs) {
      uint32_t a, bb;
      if (walked) {
        a = o.P[2 * jj];
        bb = o.P[2 * jj + 1];
      } else {
        a = ob_origin(o, 2 * jj);
        bb = ob_origin(o, 2 * jj + 1);
        o.P[2 * jj] = a;
        o.P[2 * jj + 1] = bb;
      }
      const Where w{c.err, 0u, (uint64_t)base + 2 * jj};
      nnull += collide_pair(c.p, c.sd.xi + base, c.sd.r + base, c.sd.msol + base, a, bb, n, coef,
                            VOLUME, key, slot_pairs, jj, w);
      const uint32_t fa = c.sd.xi[base + a] != 0 ? 1u : 0u;
      const uint32_t fb = c.sd.xi[base + bb] != 0 ? 1u : 0u;
      o.vflag[2 * jj] = fa;
      o.vflag[2 * jj + 1] = fb;
      ninv += 2u - fa - fb;
    } else {  // an odd last position (no pair) and the flags' end entry
      if (n & 1u) {
        const uint32_t p = walked ? o.P[n - 1] : ob_origin(o, n - 1);
        o.P[n - 1] = p;
        const uint32_t f = c.sd.xi[base + p] != 0 ? 1u : 0u;
        o.vflag[n - 1] = f;
        ninv += 1u - f;
      }
      o.vflag[n] = 0u;
    }
  }
  if (nnull) atomicAdd(o.nnull, nnull);
  if (ninv) atomicAdd(o.ninv, ninv);
}
// The records into the other buffer: valid superdroplets in shuffled order first, then the nulls
// (collisions.hpp:240-248), the slots outside the gridbox's superdroplets as they are. scanned: the
// flags have been scanned; else, where any is zero, the block counts the ones before its positions
// itself. The lists are emptied for the next step. The last block sets the gridbox's count and RNG
// slot; after the step's last sub-step (dt > 0) it advances the time and starts the next step's slot.
constexpr int OB_THREADS = 256;
__global__ void __launch_bounds__(OB_THREADS)
k_ob_gather(const __grid_constant__ DevCtx c, const __grid_constant__ BatchScratch b, OneBox o,
            Fields dst, int scanned, uint32_t dt) {
  __shared__ uint32_t wsum[OB_THREADS / 32];
  const uint32_t n = c.gcount[0], base = c.gstart[0], nslots = c.counters[0];
  const uint32_t nvalid = n - *o.nnull;
  const uint32_t ninv = *o.ninv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t i0 = blockIdx.x * OB_THREADS; i0 < nslots; i0 += gridDim.x * OB_THREADS) {
    const uint32_t i = i0 + threadIdx.x;
    const bool mine = i >= base && i - base < n;  // a shuffled position of the gridbox
    const uint32_t q = i - base;
    // valid ones before shuffled position q (q itself when all are valid)
    uint32_t before = q;
    if (ninv && scanned) {
      if (mine) before = o.vflag[q];
    } else if (ninv) {  // (uniform across the block)
      const uint32_t q0 = i0 > base ? min(i0 - base, n) : 0u;
      uint32_t x = 0;
      for (uint32_t k = threadIdx.x; k < q0; k += OB_THREADS) x += o.vflag[k];
      const uint32_t f = mine ? o.vflag[q] : 0u;
      const uint32_t own = __popc(__ballot_sync(0xFFFFFFFFu, f != 0) & ((1u << lane) - 1u));
      const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, x);           // before the block
      const uint32_t here = __popc(__ballot_sync(0xFFFFFFFFu, f != 0));  // in this warp
      if (lane == 0) wsum[warp] = all;
      __syncthreads();
      uint32_t s = 0;
      for (int w = 0; w < OB_THREADS / 32; ++w) s += wsum[w];
      __syncthreads();
      if (lane == 0) wsum[warp] = here;
      __syncthreads();
      for (int w = 0; w < warp; ++w) s += wsum[w];
      before = s + own;
      __syncthreads();
    }
    if (i >= nslots) continue;
    if (!mine) {
      copy_rec(c.sd, i, dst, i);
      continue;
    }
    o.head[q] = OB_NONE;
    const uint32_t src = base + o.P[q];
    const bool valid = !ninv || c.sd.xi[src] != 0;
    const uint32_t d = base + (valid ? before : nvalid + (q - before));
    dst.r[d] = c.sd.r[src];
    dst.msol[d] = c.sd.msol[src];
    dst.xi[d] = c.sd.xi[src];
    dst.c3[d] = c.sd.c3[src];
    dst.c1[d] = c.sd.c1[src];
    dst.c2[d] = c.sd.c2[src];
    dst.id[d] = c.sd.id[src];
    dst.gbx[d] = valid ? 0u : OOB;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(o.done, 1u) == gridDim.x - 1) {
      *o.done = 0;
      *o.nnull = 0;
      *o.ninv = 0;
      c.gcount[0] = nvalid;
      b.slot[0] = dt ? 0u : (uint32_t)((uint64_t)b.slot[0] + (n >= 1 ? n - 1 : 0) + 2ull * (n / 2));
      *b.tsdm += dt;
    }
  }
}

}  // namespace
