// pair_bound.h — the single-precision upper bound of a pair's collision probability with which the
// collision kernels leave a pair alone (batched.cuh, collide_pair), for device and host (the tests).
#pragma once

#include <cmath>
#include <cstdint>

#include "../../include/cleo_b200.h"
#include "constants.h"
#include "ddmath.h"

namespace cleo {

// a / b within 2 ulp, either way on the device; the host takes the end that makes the bound smaller
CLEO_MATH_HD float pair_div(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fdividef(a, b);
#else
  const float q = a / b;
  return std::nextafter(std::nextafter(q, INFINITY), INFINITY);
#endif
}
// the larger multiplicity of two, rounded up
CLEO_MATH_HD float pair_xi(uint64_t xa, uint64_t xb) {
  const uint64_t x = xa < xb ? xb : xa;
#if defined(__CUDA_ARCH__)
  return __ull2float_ru(x);
#else
  const float f = (float)x;
  return (unsigned __int128)f < x ? std::nextafter(f, INFINITY) : f;
#endif
}
// a random number's leading 24 bits, a lower bound of cleo_rng_to_unit's
CLEO_MATH_HD float pair_phi(uint64_t u) { return (float)(uint32_t)(u >> 40) * 0x1p-24f; }

// What the probabilities of all pairs share, in single precision: the kernel's constant and DELT.
// Not a number where there is no bound: a negative kernel (whose breakup compares phi with
// prob - floor(prob)), or one too small to be sure that no bits are lost below the normal range.
CLEO_MATH_HD float pair_bound_kernel(const cleo_b200_params& p) {
  double factor = 1.0;
  float k;
  if (p.coll_prob == CLEO_PROB_GOLOVIN) {
    k = (float)(1.5e3 * R0 * R0 * R0 * 4.0 / 3.0 * PI);
  } else if (p.coll_prob == CLEO_PROB_LONG) {
    factor = p.coaleff;
    k = (float)(PI * R0 * R0 * W0) * (float)factor;
  } else {
    factor = p.const_kernel;
    k = (float)factor;
  }
  k *= (float)p.coll_delt;
  return factor == 0.0 ? 0.0f : (k >= 1e-30f ? k : NAN);
}
// and what those of a gridbox share: scale_p / VOLUME with it, 0.5% up to cover every rounding of the
// bound. Not a number, as above: every pair is then evaluated.
CLEO_MATH_HD float pair_bound_coef(float kernel, uint32_t n, double VOLUME) {
  const float pairs = (float)(n / 2), volume = (float)VOLUME;
  const float coef =
      1.005f * ((float)n * ((float)n - 1.0f)) / (2.0f * pairs) * (kernel / volume);
  return kernel == 0.0f || (coef >= 1e-30f && volume >= 1e-30f) ? coef : NAN;
}
// Whether a pair surely does not collide: phi (at most the random number) above an upper bound of
// prob. Golovin: r1^3 + r2^3. Long: the collection efficiency (its 1 - k2 / rsmall with 1e-5 to
// spare), the squared sum of the radii, and for the difference of the terminal velocities the
// larger droplet's, at most 1.189e-4 r^2 m/s (Simmel's first branch, which the others, 0.06% above
// it where they meet, stay below beyond) and 9.18. NaN and overflow fail the comparison, and so does
// a random number of 0 whatever a bound that underflows.
CLEO_MATH_HD bool pair_apart(const cleo_b200_params& p, float coef, float r1, float r2, float xi,
                             float phi) {
  float k = 1.0f;
  if (p.coll_prob == CLEO_PROB_LONG) {
    const float rs = fminf(r1, r2), rb = fmaxf(r1, r2), rb2 = rb * rb, sum = r1 + r2;
    const float k1 = (float)(4.5e4 * R0 * R0 * 100 * 100), k2 = (float)(3e-4 / R0 / 100);
    float eff = fmaxf(k1 * rb2 * (1.00001f - pair_div(k2, rs)), 0.001f);
    if (!(rb < 49.9f)) eff = fmaxf(eff, 1.0f);
    k = eff * (sum * sum) * fminf(1.189e-4f / (float)W0 * rb2, 9.18f / (float)W0);
  } else if (p.coll_prob == CLEO_PROB_GOLOVIN) {
    k = r1 * r1 * r1 + r2 * r2 * r2;
  }
  return phi > coef * xi * k;
}

}  // namespace cleo
