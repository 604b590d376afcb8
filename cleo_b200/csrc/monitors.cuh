// monitors.cuh — SDMMonitor members: per-gridbox sums in the superdroplets' order.
//
// A warp takes up to 32 consecutive gridboxes (seq_per): it reads their contiguous range coalesced,
// a window at a time, forms every superdroplet's terms once, and lane j adds gridbox g0 + j's from shared memory
// one after another, as the reference's loops do. A thread per gridbox reading its own range, for
// all droplets and again for raindrops, took 147 us a call on 50 thousand gridboxes of 38 (twice a
// step), now 45.
#pragma once

namespace {

// calculate_massmoments / calculate_rainmassmoments (massmoments_observer.cpp:38-113): the terms
// of all droplets and of raindrops (radius >= 40 um), then fetch_delta_massmoments
// (monitor_massmoments_change.hpp:99-121); which = 0 after microphysics, 1 after motion;
// begin != 0: before_timestepping (moments become the baseline)
// A window of 512 superdroplets holds some 13 gridboxes of 38, whose lanes add side by side. A
// droplet that is not rain adds xi m 0, which is 0 unless the product is not finite: those are
// marked, so a term and a multiplicity are 16 bytes and a bit.
constexpr int MON_THREADS = 128;
constexpr uint32_t MON_WIN = 512;
struct __align__(16) MonTerm {
  float t1, t2;  // (float)(xi m), (float)(xi m m)
  unsigned long long x;
};
__global__ void __launch_bounds__(MON_THREADS)
k_mon_mm(const __grid_constant__ DevCtx c, int which, int begin, uint32_t per) {
  constexpr int PER = MON_WIN / 32;
  constexpr uint32_t NONE = 0xFFFFFFFFu;
  __shared__ MonTerm tbuf[MON_THREADS / 32][MON_WIN];
  // a bit per droplet: rain, and where its zero term is not a number
  __shared__ uint32_t rbuf[MON_THREADS / 32][3][PER];
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mask = c.p.monitors;
  const double rlim = 40e-6 / R0;
  for (uint32_t g0 = warp * per; g0 < c.ngbxs; g0 += nwarps * per) {
    const uint32_t nb = c.ngbxs - g0 < per ? c.ngbxs - g0 : per;
    const bool own = (uint32_t)lane < nb;
    const uint32_t g = g0 + lane;
    uint32_t cur = own ? c.gstart[g] : 0u;
    const uint32_t e = own ? cur + c.gcount[g] : 0u;
    unsigned long long a0 = 0, r0 = 0;
    float a1 = 0.0f, a2 = 0.0f, r1 = 0.0f, r2 = 0.0f;
    const uint32_t hi = c.gstart[g0 + nb];
    uint32_t w0 = __reduce_min_sync(0xFFFFFFFFu, cur < e ? cur : NONE);
    while (w0 != NONE) {  // the window starts at the first element a lane still has to add
      const uint32_t w1 = hi - w0 < MON_WIN ? hi : w0 + MON_WIN;
      bool bad = false;
#pragma unroll 4
      for (int q = 0; q < PER; ++q) {
        const uint32_t k = w0 + 32 * q + lane;
        if (w0 + 32 * q >= w1) break;  // uniform across the warp
        const bool in = k < w1;
        const double r = in ? c.sd.r[k] : 0.0;
        const unsigned long long x = in ? c.sd.xi[k] : 0ull;
        const double mass = sd_mass(r, in ? c.sd.msol[k] : 0.0), xi = (double)x;
        const double p1 = xi * mass, p2 = xi * mass * mass;
        tbuf[wib][32 * q + lane] = MonTerm{(float)p1, (float)p2, x};
        const uint32_t mr = __ballot_sync(0xFFFFFFFFu, r >= rlim);
        const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, !(fabs(p1) <= DBLMAX));
        const uint32_t m2 = __ballot_sync(0xFFFFFFFFu, !(fabs(p2) <= DBLMAX));
        bad |= (m1 | m2) != 0u;
        if (lane == 0) {
          rbuf[wib][0][q] = mr;
          rbuf[wib][1][q] = m1;
          rbuf[wib][2][q] = m2;
        }
      }
      __syncwarp();
      const uint32_t b = e < w1 ? e : w1;
#pragma unroll 4
      for (uint32_t k = cur; k < b; ++k) {
        const uint32_t o = k - w0;
        const MonTerm t = tbuf[wib][o];
        const bool rain = (rbuf[wib][0][o >> 5] >> (o & 31)) & 1u;
        a0 += t.x;
        a1 += t.t1;
        a2 += t.t2;
        r0 += rain ? t.x : 0ull;
        r1 += rain ? t.t1 : 0.0f;
        r2 += rain ? t.t2 : 0.0f;
      }
      if (bad)  // (no number comes back from NaN, so its place in the sum does not matter)
        for (uint32_t k = cur; k < b; ++k) {
          const uint32_t o = k - w0, bit = 1u << (o & 31);
          const bool rain = rbuf[wib][0][o >> 5] & bit;
          if (!rain && (rbuf[wib][1][o >> 5] & bit)) r1 = __int_as_float(0x7FFFFFFF);
          if (!rain && (rbuf[wib][2][o >> 5] & bit)) r2 = __int_as_float(0x7FFFFFFF);
        }
      cur = cur < b ? b : cur;
      __syncwarp();
      w0 = __reduce_min_sync(0xFFFFFFFFu, cur < e ? cur : NONE);
    }
    if (!own) continue;
    for (int rain = 0; rain < 2; ++rain) {
      if (!begin && !(mask & (rain ? CLEO_MONITOR_RAINMASSMOMENTS : CLEO_MONITOR_MASSMOMENTS)))
        continue;
      const unsigned long long m0 = rain ? r0 : a0;
      const float m1 = rain ? r1 : a1, m2 = rain ? r2 : a2;
      if (!begin) {
        c.mm0[rain][which][g] += m0 - c.prev0[rain][g];
        c.mm1[rain][which][g] += m1 - c.prev1[rain][g];
        c.mm2[rain][which][g] += m2 - c.prev2[rain][g];
      }
      c.prev0[rain][g] = m0;
      c.prev1[rain][g] = m1;
      c.prev2[rain][g] = m2;
    }
  }
}
// the precipitation contributions of each gridbox's superdroplets, in their order (the reference
// adds them one by one as it moves the gridbox's superdroplets), onto its sum so far
__global__ void __launch_bounds__(SEQ_THREADS) k_mon_precip(const __grid_constant__ DevCtx c,
                                                            uint32_t per) {
  __shared__ double dbuf[SEQ_THREADS / 32][SEQ_WIN];
  __shared__ uint32_t ubuf[SEQ_THREADS / 32][SEQ_WIN];
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t g0 = warp * per; g0 < c.ngbxs; g0 += nwarps * per) {
    const uint32_t nb = c.ngbxs - g0 < per ? c.ngbxs - g0 : per;
    const bool own = (uint32_t)lane < nb;
    double acc;
    unsigned long long unused;
    warp_batch_sums(
        c, g0, nb, dbuf[wib], ubuf[wib],
        [&](uint32_t k) {
          const double v = c.precip_c[k];
          return v > 0.0 ? v : 0.0;  // (adding 0 to a sum of positive terms changes nothing)
        },
        [](uint32_t) { return 0u; }, acc, unused, false, own ? c.precip[g0 + lane] : 0.0);
    if (own) c.precip[g0 + lane] = acc;
  }
}

}  // namespace
