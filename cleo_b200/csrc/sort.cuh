// sort.cuh — stable counting sort of superdroplets by gridbox index on the GPU.
//
// Replaces SortSupersBySdgbxindex (libs/gridboxes/sortsupers.hpp:93-226): the reference builds a
// histogram of sdgbxindex (out-of-domain keys share the last bucket), an exclusive scan and a
// scatter with atomic_fetch_add, which is stable only on the Serial backend. Here the scatter is
// made stable on the GPU by a least-significant-digit radix sort of (key, position) pairs with
// 8-bit digits: per digit pass, every tile of 4096 keys counts its digits (upsweep), the table of
// tile counts is scanned, and each tile ranks its keys stably with warp match/ballot (downsweep).
// No block waits on another block. A pass is two launches for up to RS_SELF_TILES tiles (each
// downsweep block adds the table up itself), three while the scan's tile totals are few enough for
// a block to add up (RS_RAW_SUMS), else four: on small sorts a launch costs as much as its work
// (about 1.2 us in a graph beside 2 us of run time; 5 launches a pass before).
#pragma once

#include <cstdint>

namespace cleo {

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// (A block that adds the table up itself reads 1 KB a tile: two passes over 64 tiles 60 us against 63,
// over 98 tiles 66 against 62.)
constexpr uint32_t RS_SELF_TILES = 64;
constexpr uint32_t RS_RAW_SUMS = 64;

// per-tile digit counts: hist[d * ntiles + tile], or hist[tile * 256 + d] for SELF. With small_n
// > 0 the pass does nothing for n <= small_n (k_rs_small sorts those in one block). Keys above
// `cap` count as cap.
template <bool SELF>
__global__ void __launch_bounds__(RS_THREADS)
k_rs_upsweep(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ n_ptr, uint32_t n_val,
             int shift, uint32_t* __restrict__ hist, uint32_t ntiles, uint32_t small_n,
             uint32_t cap) {
  __shared__ uint32_t cnt[256];
  const uint32_t n = n_ptr ? *n_ptr : n_val;
  if (small_n > 0 && n <= small_n) return;
  for (int i = threadIdx.x; i < 256; i += RS_THREADS) cnt[i] = 0;
  __syncthreads();
  const uint32_t tile = blockIdx.x;
  const uint64_t base = (uint64_t)tile * RS_TILE;
  // all loads first; then one shared atomic per digit a warp meets: the keys are nearly sorted, so
  // a warp's are mostly one digit, and 32 atomics on it would run one after another
  uint32_t dg[RS_ITEMS];
#pragma unroll
  for (int k = 0; k < RS_ITEMS; ++k) {
    const uint64_t idx = base + (uint64_t)k * RS_THREADS + threadIdx.x;
    dg[k] = idx < n ? (min(keys[idx], cap) >> shift) & 255u : 256u;
  }
#pragma unroll
  for (int k = 0; k < RS_ITEMS; ++k) {
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, dg[k]);
    if (dg[k] < 256u && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
      atomicAdd(&cnt[dg[k]], (uint32_t)__popc(peers));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += RS_THREADS)
    hist[SELF ? (uint64_t)tile * 256 + i : (uint64_t)i * ntiles + tile] = cnt[i];
}

// stable scatter of one digit pass. offs: the counts (SELF), or their scan within scan tiles, with
// the scan tiles' totals in tsums, exclusively scanned or (raw_sums) as they are. vin may be null:
// a value is then its position.
template <bool SELF>
__global__ void __launch_bounds__(RS_THREADS)
k_rs_downsweep(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
               const uint32_t* __restrict__ n_ptr, uint32_t n_val, int shift,
               const uint32_t* __restrict__ offs,
               uint32_t ntiles, const uint32_t* __restrict__ tsums, uint32_t raw_sums,
               uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t small_n,
               uint32_t cap) {
  __shared__ uint32_t wcount[RS_WARPS][256];
  __shared__ uint32_t dbase[256];
  __shared__ uint32_t pre[RS_RAW_SUMS];
  const uint32_t n = n_ptr ? *n_ptr : n_val;
  const uint32_t tile = blockIdx.x;
  const uint64_t base = (uint64_t)tile * RS_TILE;
  if (base >= n || (small_n > 0 && n <= small_n)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // warp w owns the contiguous chunk [w*32*ITEMS, (w+1)*32*ITEMS) of the tile, read in rounds of
  // 32 consecutive keys: rank order = array order. Few tiles (SELF) load them all first, ahead of
  // the table: there a block's own latency counts, 16 loads one behind another's ranking else (16
  // tiles, caches cold: 14.8 us a pass, now 9.5). Many tiles load them round by round: all first
  // takes more than 80 registers and was slower (80 us a pass for 50 on 6.6 M keys).
  uint32_t kk[RS_ITEMS], vv[RS_ITEMS], rk[RS_ITEMS];
  const uint64_t own = base + (uint64_t)warp * 32 * RS_ITEMS + lane;
  if constexpr (SELF) {
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
      const uint64_t idx = own + (uint64_t)j * 32;
      kk[j] = idx < n ? min(kin[idx], cap) : 0u;
      vv[j] = idx < n ? (vin ? vin[idx] : (uint32_t)idx) : 0u;
    }
  }
  for (int i = threadIdx.x; i < RS_WARPS * 256; i += RS_THREADS) (&wcount[0][0])[i] = 0;
  if constexpr (SELF) {
    // digit d = thread: the tiles' counts of it before this one, and in all
    const uint32_t d = threadIdx.x;
    uint32_t before = 0, total = 0;
#pragma unroll 8
    for (uint32_t t = 0; t < ntiles; ++t) {
      const uint32_t c = offs[t * 256 + d];
      before += t < tile ? c : 0u;
      total += c;
    }
    uint32_t x = total;  // exclusive scan of the digits' totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) pre[warp] = x;
    __syncthreads();
    uint32_t w0 = 0;
    for (int w = 0; w < warp; ++w) w0 += pre[w];
    dbase[d] = w0 + x - total + before;
  } else {
    if (raw_sums > 0) {
      if (warp == 0) {  // up to 64 totals: two a lane
        const uint32_t i = 2 * lane;
        const uint32_t a = i < raw_sums ? tsums[i] : 0u;
        const uint32_t b = i + 1 < raw_sums ? tsums[i + 1] : 0u;
        uint32_t x = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
          if (lane >= o) x += y;
        }
        pre[i] = x - a - b;
        pre[i + 1] = x - b;
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < 256; i += RS_THREADS) {
      const uint64_t e = (uint64_t)i * ntiles + tile;
      dbase[i] = offs[e] + (raw_sums > 0 ? pre[e / SCAN_TILE] : tsums[e / SCAN_TILE]);
    }
  }
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const uint64_t idx = own + (uint64_t)j * 32;
    const bool valid = idx < n;
    if constexpr (!SELF) {
      kk[j] = valid ? min(kin[idx], cap) : 0u;
      vv[j] = valid ? (vin ? vin[idx] : (uint32_t)idx) : 0u;
    }
    const uint32_t d = valid ? ((kk[j] >> shift) & 255u) : 256u;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
    const int leader = __ffs(peers) - 1;
    uint32_t prev = 0;
    if (valid) prev = wcount[warp][d];
    __syncwarp();
    if (valid && lane == leader) wcount[warp][d] = prev + __popc(peers);
    __syncwarp();
    rk[j] = valid ? (prev + __popc(peers & lt)) : 0xFFFFFFFFu;
  }
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += RS_THREADS) {
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      const uint32_t c = wcount[w][d];
      wcount[w][d] = s;
      s += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    if (rk[j] != 0xFFFFFFFFu) {
      const uint32_t d = (kk[j] >> shift) & 255u;
      const uint32_t pos = dbase[d] + wcount[warp][d] + rk[j];
      kout[pos] = kk[j];
      vout[pos] = vv[j];
    }
  }
}

// The same stable LSD sort in one block of RS_SMALL_THREADS, for counts (on the device) up to
// RS_SMALL_MAX: `bits` key bits in 8-bit passes between (k0, v0) and (k1, v1), leaving the result
// where the multi-tile passes would (in (k0, v0) after an even number of passes). Returns at once
// for larger n, which the multi-tile passes sort. The first pass's values may be positions (v_first
// null), its keys capped.
constexpr int RS_SMALL_THREADS = 1024;
constexpr int RS_SMALL_WARPS = RS_SMALL_THREADS / 32;
constexpr uint32_t RS_SMALL_MAX = (uint32_t)RS_SMALL_THREADS * RS_ITEMS;  // 16384
__global__ void __launch_bounds__(RS_SMALL_THREADS)
k_rs_small(const uint32_t* k_first, const uint32_t* v_first, uint32_t* k0, uint32_t* v0,
           uint32_t* k1, uint32_t* v1, uint32_t* v_last, const uint32_t* __restrict__ n_ptr,
           uint32_t n_val, uint32_t bits, uint32_t cap) {
  __shared__ uint32_t wcount[RS_SMALL_WARPS][256];
  __shared__ uint32_t dbase[256];
  __shared__ uint32_t wsum[8];
  const uint32_t n = n_ptr ? *n_ptr : n_val;
  if (n > RS_SMALL_MAX) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t d = threadIdx.x;  // digit of the threads below 256
  uint32_t* K[2] = {k0, k1};
  uint32_t* V[2] = {v0, v1};
  int cur = 0;
  for (uint32_t shift = 0; shift < bits; shift += 8) {
    const uint32_t* kin = shift == 0 ? k_first : K[cur];
    const uint32_t* vin = shift == 0 ? v_first : V[cur];
    for (int i = threadIdx.x; i < RS_SMALL_WARPS * 256; i += RS_SMALL_THREADS)
      (&wcount[0][0])[i] = 0;
    __syncthreads();
    uint32_t kk[RS_ITEMS], vv[RS_ITEMS], rk[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {  // array order = rank order, as in k_rs_downsweep
      const uint32_t idx = (uint32_t)warp * 32 * RS_ITEMS + (uint32_t)j * 32 + lane;
      const bool valid = idx < n;
      kk[j] = valid ? min(kin[idx], cap) : 0u;
      vv[j] = valid ? (vin ? vin[idx] : idx) : 0u;
      rk[j] = 0xFFFFFFFFu;
    }
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
      const uint32_t first = (uint32_t)warp * 32 * RS_ITEMS + (uint32_t)j * 32;
      if (first >= n) continue;  // whole warp
      const bool valid = first + lane < n;
      const uint32_t dg = valid ? ((kk[j] >> shift) & 255u) : 256u;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, dg);
      const int leader = __ffs(peers) - 1;
      uint32_t prev = 0;
      if (valid) prev = wcount[warp][dg];
      __syncwarp();
      if (valid && lane == leader) wcount[warp][dg] = prev + __popc(peers);
      __syncwarp();
      if (valid) rk[j] = prev + __popc(peers & lt);
    }
    __syncthreads();
    // the per-warp offsets of a digit, then the exclusive scan of the digits' totals over the first
    // 8 warps
    uint32_t tot = 0, x = 0;
    if (d < 256) {
#pragma unroll 8
      for (int w = 0; w < RS_SMALL_WARPS; ++w) {
        const uint32_t c = wcount[w][d];
        wcount[w][d] = tot;
        tot += c;
      }
      x = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) wsum[warp] = x;
    }
    __syncthreads();
    if (d < 256) {
      uint32_t before = 0;
      for (int w = 0; w < warp; ++w) before += wsum[w];
      dbase[d] = before + x - tot;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
      if (rk[j] != 0xFFFFFFFFu) {
        const uint32_t dg = (kk[j] >> shift) & 255u;
        const uint32_t pos = dbase[dg] + wcount[warp][dg] + rk[j];
        K[1 - cur][pos] = kk[j];
        (v_last && shift + 8 >= bits ? v_last : V[1 - cur])[pos] = vv[j];
      }
    }
    __syncthreads();  // this pass's writes before the next pass reads them
    cur ^= 1;
  }
}

// ---- exclusive scan of u32 (reduce-then-scan over tiles of SCAN_TILE) ----
// The scan kernels take an optional gate: with gate set they do nothing while *gate <= gate_max
// (the digit tables of a multi-tile radix pass that k_rs_small replaces).
__device__ __forceinline__ uint32_t block_exclusive_scan_1024(uint32_t v, uint32_t* wsum,
                                                              uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = (lane < (int)(blockDim.x >> 5)) ? wsum[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
      if (lane >= o) s += y;
    }
    wsum[lane] = s;  // inclusive over warps
  }
  __syncthreads();
  total = wsum[(blockDim.x >> 5) - 1];
  const uint32_t before = warp > 0 ? wsum[warp - 1] : 0u;
  __syncthreads();
  return before + x - v;
}

// phase 1: scan each tile, write the tile's total
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_tiles(const uint32_t* in, uint32_t* out, uint64_t n,  // in == out: scanned in place
             uint32_t* __restrict__ tile_sums, const uint32_t* gate = nullptr,
             uint32_t gate_max = 0) {
  __shared__ uint32_t wsum[32];
  if (gate && *gate <= gate_max) return;
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
  uint32_t v[SCAN_ITEMS], s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0u;
    s += v[k];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan_1024(s, wsum, total);
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// phase 2: one block scans the tile totals (exclusive, in place); *grand gets the total
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_sums(uint32_t* __restrict__ sums, uint32_t nsums, uint32_t* __restrict__ grand,
            const uint32_t* gate = nullptr, uint32_t gate_max = 0) {
  __shared__ uint32_t wsum[32];
  if (gate && *gate <= gate_max) return;
  uint32_t carry = 0;
  for (uint32_t start = 0; start < nsums; start += SCAN_THREADS) {
    const uint32_t i = start + threadIdx.x;
    const uint32_t v = i < nsums ? sums[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan_1024(v, wsum, total);
    if (i < nsums) sums[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0 && grand) *grand = carry;
}

// phase 3: add the scanned tile totals
__global__ void k_scan_add(uint32_t* __restrict__ out, uint64_t n,
                           const uint32_t* __restrict__ tile_sums, const uint32_t* gate = nullptr,
                           uint32_t gate_max = 0) {
  if (gate && *gate <= gate_max) return;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += tile_sums[i / SCAN_TILE];
}

// The count of pairs is *n_ptr on the device, or n_val where n_ptr is null; k_rs_small and
// radix_passes write the last pass's values to v_last where it is given.
// Stable radix sort of (key, value) pairs over `bits` key bits
// (8-bit passes), for up to nt tiles: reads (k_first, v_first) (v_first null: positions; keys
// capped), then uses the buffers (k0, v0) and (k1, v1) in turn, the first pass writing (k1, v1).
// Returns 0 if the result is in (k0, v0), else 1. hist: 256 nt words; tsums: their scan's tile
// totals. With small_n the passes do nothing for counts up to it. Adds its launches to *launches.
inline int radix_passes(cudaStream_t s, const uint32_t* k_first, const uint32_t* v_first,
                        uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1,
                        uint32_t* v_last, const uint32_t* n_ptr, uint32_t n_val, uint32_t bits,
                        uint32_t* hist, uint32_t* tsums,
                        uint32_t nt, uint32_t small_n, uint32_t cap,
                        unsigned long long* launches) {
  const uint64_t nh = (uint64_t)256 * nt;
  const uint32_t nscan = (uint32_t)((nh + SCAN_TILE - 1) / SCAN_TILE);
  uint32_t* K[2] = {k0, k1};
  uint32_t* V[2] = {v0, v1};
  int cur = 0;
  for (uint32_t shift = 0; shift < bits; shift += 8) {
    const uint32_t* kin = shift == 0 ? k_first : K[cur];
    const uint32_t* vin = shift == 0 ? v_first : V[cur];
    uint32_t* vout = v_last && shift + 8 >= bits ? v_last : V[1 - cur];
    if (nt <= RS_SELF_TILES) {
      k_rs_upsweep<true><<<nt, RS_THREADS, 0, s>>>(kin, n_ptr, n_val, (int)shift, hist, nt, small_n,
                                                      cap);
      k_rs_downsweep<true><<<nt, RS_THREADS, 0, s>>>(kin, vin, n_ptr, n_val, (int)shift, hist, nt, tsums,
                                                     0, K[1 - cur], vout, small_n, cap);
      *launches += 2;
    } else {
      const bool raw = nscan <= RS_RAW_SUMS;
      k_rs_upsweep<false><<<nt, RS_THREADS, 0, s>>>(kin, n_ptr, n_val, (int)shift, hist, nt, small_n,
                                                      cap);
      k_scan_tiles<<<nscan, SCAN_THREADS, 0, s>>>(hist, hist, nh, tsums, n_ptr, small_n);
      if (!raw) k_scan_sums<<<1, SCAN_THREADS, 0, s>>>(tsums, nscan, nullptr, n_ptr, small_n);
      k_rs_downsweep<false><<<nt, RS_THREADS, 0, s>>>(kin, vin, n_ptr, n_val, (int)shift, hist, nt, tsums,
                                                      raw ? nscan : 0, K[1 - cur], vout,
                                                      small_n, cap);
      *launches += raw ? 3 : 4;
    }
    cur = 1 - cur;
  }
  return cur;
}

}  // namespace cleo
