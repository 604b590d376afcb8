// mlp.cu — training and inference entry points of the condensation surrogate (see mlp.cuh).
//
// Training runs on the GPU with this file's own kernels: a forward/backward kernel computes the
// gradient of the mean squared error of the standardised target over a minibatch (FP32,
// deterministic: each CTA adds its samples up in a fixed order into its own partial row, and
// the Adam kernel sums the rows in a fixed order), and an Adam kernel updates the FP32 master
// weights. After every change of the weights a packing kernel writes the BF16 inference copies.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/cleo_b200.h"
#include "mlp.cuh"

using namespace cleo;
using namespace cleo::mlp;

struct cleo_b200_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  float* params = nullptr;  // NPARAM FP32 master weights
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  float* norm = nullptr;  // NNORM
  float* fw = nullptr;    // NFW inference constants
  uint4* w2_umma = nullptr;
  uint32_t* w2_rm = nullptr;
  uint32_t* err = nullptr;
  DevError* phys_err = nullptr;
  float* partial = nullptr;  // [cap_blocks][NPARAM]
  float* loss_partial = nullptr;
  double* stats = nullptr;  // [cap_stat_blocks][32]
  uint32_t cap_blocks = 0, cap_stat_blocks = 0;
  uint64_t adam_t = 0;
};

namespace {

#define MLP_TRY(x)                                                                     \
  do {                                                                                 \
    cudaError_t e_ = (x);                                                              \
    if (e_ != cudaSuccess) {                                                           \
      fprintf(stderr, "cleo_b200 mlp: %s failed: %s\n", #x, cudaGetErrorString(e_)); \
      return CLEO_ERR_CUDA;                                                            \
    }                                                                                  \
  } while (0)

// The training kernel's tile: TR_S samples by TR_T threads. Rows of 64 units are padded to TR_LD
// floats: 16-byte aligned, and 8 adjacent rows start in different banks.
constexpr int TR_S = 64;
constexpr int TR_T = 256;
constexpr int TR_LD = 68;
constexpr uint32_t TR_BLOCKS_MAX = 148 * 2;  // two CTAs of TR_SMEM per SM
// floats: W2 and four activation arrays, W1 with its biases and the features (rows of 8), then b2,
// W3, targets, dL/dy, and two partial outputs per sample
constexpr size_t TR_SMEM =
    (size_t)(5 * TR_S * TR_LD + 2 * TR_S * 8 + 6 * TR_S) * sizeof(float);  // 92,672 B

// ---- features, standardisation targets and the Newton branch of each droplet ----
__global__ void k_mlp_features(uint32_t n, const double* __restrict__ radius,
                               const double* __restrict__ msol, const double* __restrict__ temp,
                               const double* __restrict__ press,
                               const double* __restrict__ s_ratio,
                               const double* __restrict__ delt,
                               const double* __restrict__ radius_new, float* __restrict__ feats,
                               float* __restrict__ target, uint8_t* __restrict__ direct,
                               DevError* err) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float x[NIN];
    raw_features(radius[i], msol[i], temp[i], press[i], s_ratio[i], delt[i], x);
#pragma unroll
    for (int q = 0; q < NIN; ++q) feats[(size_t)i * NIN + q] = x[q];
    if (target) target[i] = (float)(2.0 * log(radius_new[i] / radius[i]));
    if (direct) {
      // the branch of solve_condensation (impliciteuler.cpp:35-54) that a seed applies to
      const Where w{err, OOB, i};
      const double T = temp[i];
      const double psat = saturation_pressure(T, w);
      const double ffactor = diffusion_factor(press[i], T, psat);
      double akoh, bkoh;
      kohler_factors(msol[i], T, akoh, bkoh);
      const OdeConsts o = ode_consts(s_ratio[i], akoh, bkoh, ffactor / ventilation_factor(radius[i]));
      const double z0 = initialguess(o, radius[i]);
      direct[i] = (first_unique_criteria(o, radius[i], z0) || delt[i] <= critical_timestep(o))
                      ? 1
                      : 0;
    }
  }
}

// per-block sums and sums of squares of the 7 features and the target (FP64)
__global__ void k_mlp_stats(uint32_t n, const float* __restrict__ feats,
                            const float* __restrict__ target, double* __restrict__ out) {
  __shared__ double red[256];
  double s[8], q[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) s[c] = q[c] = 0.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double v = c < NIN ? (double)feats[(size_t)i * NIN + c] : (double)target[i];
      s[c] += v;
      q[c] += v * v;
    }
  }
  for (int c = 0; c < 16; ++c) {
    red[threadIdx.x] = c < 8 ? s[c] : q[c - 8];
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
      if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x * 32 + c] = red[0];
    __syncthreads();
  }
}

// ---- forward + backward ----
// Loss L = inv_count * sum_s (y_s - t_s)^2 over the standardised target t. random != 0 draws
// the samples uniformly (with replacement) from [0, n) by the counter generator keyed by
// (seed, step); otherwise sample = slot.
//
// The three 64 x 64 products of a sample (layer 2, its transpose in the backward pass, and the
// weights' gradient) are a third of a megaflop each for a tile of 64 samples: every thread keeps
// 4 x 4 outputs in registers and reads its operands four at a time, 16 bytes a load, from rows laid
// out so that a warp's loads meet no bank twice: 64 fused multiply-adds to 8 loads. A thread per
// sample with a row of weights per multiply-add kept 4 warps on each of 64 SMs busy with loads:
// 8192 samples took 77 us (cold, under the profiler), now 22, and a training step, its Adam update
// and launches with it, 76 us live, now 28.5. What bounds it is the chain of a tile's phases at two
// warps per scheduler, a quarter of the time shared-memory loads; 512 threads of 2 x 4 outputs
// read more (half the time) and took 33 us a step. A CTA takes several tiles when there are more
// than TR_BLOCKS_MAX, adding to the same registers, so the partial rows stay few.
//
// The kernels of consecutive steps are on the GPU together (launch_step): an update writes params
// while the next gradient kernel waits, a gradient kernel writes partial and loss_partial while its
// update waits. So no pointer to those carries __restrict__, which would say that nothing else
// writes them while the kernel runs and allow loads through the read-only path or ahead of the
// wait, and they are read from L2 (__ldcg), where the writer's stores are.
__device__ __forceinline__ void fma4x4(float acc[4][4], const float4 a[4], const float4 b[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[r][c] = __fmaf_rn(a[r].x, b[c].x, acc[r][c]);
      acc[r][c] = __fmaf_rn(a[r].y, b[c].y, acc[r][c]);
      acc[r][c] = __fmaf_rn(a[r].z, b[c].z, acc[r][c]);
      acc[r][c] = __fmaf_rn(a[r].w, b[c].w, acc[r][c]);
    }
}
// acc[r][c] += x * b[c] for the four components of b
__device__ __forceinline__ void fma1x4(float acc[4], float x, const float4& b) {
  acc[0] = __fmaf_rn(x, b.x, acc[0]);
  acc[1] = __fmaf_rn(x, b.y, acc[1]);
  acc[2] = __fmaf_rn(x, b.z, acc[2]);
  acc[3] = __fmaf_rn(x, b.w, acc[3]);
}
// GELU and its derivative from one erf
__device__ __forceinline__ void gelu_both(float a, float& h, float& d) {
  const float cdf = 0.5f * (1.0f + erff(a * 0.70710678118654752f));
  h = a * cdf;
  d = __fmaf_rn(a, 0.39894228040143268f * expf(-0.5f * a * a), cdf);
}
__global__ void __launch_bounds__(TR_T, 2)
k_mlp_fwdbwd(const float* params, const float* __restrict__ norm,
             const float* __restrict__ feats, const float* __restrict__ target, uint32_t n,
             uint32_t count, uint64_t seed, uint32_t step, int random,
             float* partial, float* loss_partial, float inv_count) {
  extern __shared__ __align__(16) float sm[];
  float* W2 = sm;                    // [j][k]
  float* H1 = W2 + TR_S * TR_LD;     // hidden 1 after GELU, [sample][k]
  float* D1 = H1 + TR_S * TR_LD;     // GELU'(a1), then dL/da1
  float* H2 = D1 + TR_S * TR_LD;     // hidden 2 after GELU
  float* D2 = H2 + TR_S * TR_LD;     // dL/da2
  float* W1 = D2 + TR_S * TR_LD;     // [k][8]: 7 weights and the bias
  float* X = W1 + TR_S * 8;          // [sample][8]: standardised features and 1
  float* B2 = X + TR_S * 8;
  float* W3 = B2 + TR_S;
  float* T = W3 + TR_S;              // standardised target
  float* DY = T + TR_S;              // dL/dy
  float* YP = DY + TR_S;             // [2][sample] partial outputs
  const uint32_t t = threadIdx.x;
  const uint32_t ntiles = (count + TR_S - 1) / TR_S;
  // a thread's 4 x 4 outputs: lanes 8 x 4 over (column group, row group)
  const uint32_t cg = (t & 7) + 8 * ((t >> 5) & 1), rg = ((t >> 3) & 3) + 4 * (t >> 6);
  cudaTriggerProgrammaticLaunchCompletion();
  // this tile's samples: four threads a sample, two of its 8 values (7 features, target) each
  float v0 = 0.0f, v1 = 0.0f;
  const uint32_t gs = t >> 2, gp = t & 3;
  const auto gather = [&](uint32_t tile) {
    const uint32_t slot = tile * TR_S + gs;
    v0 = v1 = 0.0f;
    if (slot < count) {
      uint32_t j = slot;
      if (random)
        j = (uint32_t)cleo_rng_mulhi(cleo_rng_u64(cleo_rng_key(seed, step, 0x4D4C50u), slot), n);
      v0 = feats[(size_t)j * NIN + 2 * gp];
      v1 = gp < 3 ? feats[(size_t)j * NIN + 2 * gp + 1] : target[j];
    }
  };
  // the samples are inputs that no earlier kernel of a training run writes: in flight while the
  // update before this step finishes (programmatic launch)
  gather(blockIdx.x);
  cudaGridDependencySynchronize();
  for (uint32_t i = t; i < (uint32_t)(NH * NH); i += TR_T)
    W2[(i / NH) * TR_LD + i % NH] = __ldcg(&params[OFF_W2 + i]);
  for (uint32_t i = t; i < (uint32_t)(NH * 8); i += TR_T)
    W1[i] = __ldcg(&params[(i & 7) < NIN ? OFF_W1 + (i >> 3) * NIN + (i & 7) : OFF_B1 + (i >> 3)]);
  if (t < NH) {
    B2[t] = __ldcg(&params[OFF_B2 + t]);
    W3[t] = __ldcg(&params[OFF_W3 + t]);
  }
  const float b3 = __ldcg(&params[OFF_B3]);
  float gw2[4][4], gw1[2] = {0.0f, 0.0f}, gv = 0.0f, gb3 = 0.0f, loss = 0.0f;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) gw2[r][c] = 0.0f;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const bool gvalid = tile * TR_S + gs < count;
    {  // standardise; an unused slot's features are zero
      const uint32_t q0 = 2 * gp, q1 = q0 + 1;
      X[gs * 8 + q0] = gvalid ? (v0 - norm[q0]) * norm[NIN + q0] : 0.0f;
      if (gp < 3) {
        X[gs * 8 + q1] = gvalid ? (v1 - norm[q1]) * norm[NIN + q1] : 0.0f;
      } else {
        X[gs * 8 + 7] = 1.0f;
        T[gs] = gvalid ? (v1 - norm[14]) / norm[15] : 0.0f;
      }
    }
    __syncthreads();
    if (tile + gridDim.x < ntiles) gather(tile + gridDim.x);
    {  // layer 1: sample t / 4, units t % 4 + 4 r
      const float4 xa = *reinterpret_cast<const float4*>(&X[gs * 8]);
      const float4 xb = *reinterpret_cast<const float4*>(&X[gs * 8 + 4]);
#pragma unroll 4
      for (int r = 0; r < 16; ++r) {
        const uint32_t k = gp + 4 * r;
        const float4 wa = *reinterpret_cast<const float4*>(&W1[k * 8]);
        const float4 wb = *reinterpret_cast<const float4*>(&W1[k * 8 + 4]);
        float a = wb.w;
        a = __fmaf_rn(wa.x, xa.x, a);
        a = __fmaf_rn(wa.y, xa.y, a);
        a = __fmaf_rn(wa.z, xa.z, a);
        a = __fmaf_rn(wa.w, xa.w, a);
        a = __fmaf_rn(wb.x, xb.x, a);
        a = __fmaf_rn(wb.y, xb.y, a);
        a = __fmaf_rn(wb.z, xb.z, a);
        gelu_both(a, H1[gs * TR_LD + k], D1[gs * TR_LD + k]);
      }
    }
    __syncthreads();
    float d2[4][4];  // W3 GELU'(a2), samples rg + 16 r, units cg + 16 c
    {
      float acc[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = B2[cg + 16 * c];
#pragma unroll 4
      for (int k = 0; k < NH; k += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          a[r] = *reinterpret_cast<const float4*>(&H1[(rg + 16 * r) * TR_LD + k]);
          b[r] = *reinterpret_cast<const float4*>(&W2[(cg + 16 * r) * TR_LD + k]);
        }
        fma4x4(acc, a, b);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float y = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float w3 = W3[cg + 16 * c];
          float h, d;
          gelu_both(acc[r][c], h, d);
          H2[(rg + 16 * r) * TR_LD + cg + 16 * c] = h;
          d2[r][c] = w3 * d;
          y = __fmaf_rn(w3, h, y);
        }
        // the sample's 16 column groups: 8 lanes here, two warps through YP
        y += __shfl_xor_sync(0xFFFFFFFFu, y, 1);
        y += __shfl_xor_sync(0xFFFFFFFFu, y, 2);
        y += __shfl_xor_sync(0xFFFFFFFFu, y, 4);
        if ((t & 7) == 0) YP[((t >> 5) & 1) * TR_S + rg + 16 * r] = y;
      }
    }
    __syncthreads();
    if (t < TR_S) {
      const float d = tile * TR_S + t < count ? (b3 + (YP[t] + YP[TR_S + t])) - T[t] : 0.0f;
      const float dy = 2.0f * d * inv_count;
      DY[t] = dy;
      loss = __fmaf_rn(d * inv_count, d, loss);
      gb3 += dy;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float dy = DY[rg + 16 * r];
#pragma unroll
      for (int c = 0; c < 4; ++c) D2[(rg + 16 * r) * TR_LD + cg + 16 * c] = dy * d2[r][c];
    }
    __syncthreads();
    {  // dL/dh1 = D2 W2: samples rg + 16 r, units 4 cg ..
      float acc[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.0f;
#pragma unroll 4
      for (int j = 0; j < NH; j += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          a[r] = *reinterpret_cast<const float4*>(&D2[(rg + 16 * r) * TR_LD + j]);
          b[r] = *reinterpret_cast<const float4*>(&W2[(j + r) * TR_LD + 4 * cg]);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          fma1x4(acc[r], a[r].x, b[0]);
          fma1x4(acc[r], a[r].y, b[1]);
          fma1x4(acc[r], a[r].z, b[2]);
          fma1x4(acc[r], a[r].w, b[3]);
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float4* d = reinterpret_cast<float4*>(&D1[(rg + 16 * r) * TR_LD + 4 * cg]);
        float4 v = *d;
        v.x *= acc[r][0];
        v.y *= acc[r][1];
        v.z *= acc[r][2];
        v.w *= acc[r][3];
        *d = v;
      }
    }
    __syncthreads();
    // parameter gradients, the samples in order
#pragma unroll 4
    for (int q = 0; q < TR_S; ++q) {  // W2: units 4 rg .. by 4 cg ..
      const float4 a = *reinterpret_cast<const float4*>(&D2[q * TR_LD + 4 * rg]);
      const float4 b = *reinterpret_cast<const float4*>(&H1[q * TR_LD + 4 * cg]);
      fma1x4(gw2[0], a.x, b);
      fma1x4(gw2[1], a.y, b);
      fma1x4(gw2[2], a.z, b);
      fma1x4(gw2[3], a.w, b);
    }
#pragma unroll 8
    for (int q = 0; q < TR_S; ++q) {  // W1 and b1: unit t / 4, columns 2 (t % 4) ..
      const float d = D1[q * TR_LD + gs];
      const float2 x = *reinterpret_cast<const float2*>(&X[q * 8 + 2 * gp]);
      gw1[0] = __fmaf_rn(d, x.x, gw1[0]);
      gw1[1] = __fmaf_rn(d, x.y, gw1[1]);
    }
    if (t < NH) {
#pragma unroll 8
      for (int q = 0; q < TR_S; ++q) gv += D2[q * TR_LD + t];
    } else if (t < 2 * NH) {
#pragma unroll 8
      for (int q = 0; q < TR_S; ++q) gv = __fmaf_rn(DY[q], H2[q * TR_LD + t - NH], gv);
    }
    __syncthreads();
  }
  float* out = partial + (size_t)blockIdx.x * NPARAM;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) out[OFF_W2 + (4 * rg + r) * NH + 4 * cg + c] = gw2[r][c];
  out[OFF_W1 + gs * NIN + 2 * gp] = gw1[0];
  if (gp < 3)
    out[OFF_W1 + gs * NIN + 2 * gp + 1] = gw1[1];
  else
    out[OFF_B1 + gs] = gw1[1];
  if (t < 2 * NH) out[(t < NH ? OFF_B2 : OFF_W3 - NH) + t] = gv;
  if (t < TR_S) {  // two warps: their lanes' sums over the samples
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      gb3 += __shfl_down_sync(0xFFFFFFFFu, gb3, o);
      loss += __shfl_down_sync(0xFFFFFFFFu, loss, o);
    }
    if ((t & 31) == 0) {
      YP[t >> 5] = gb3;
      YP[2 + (t >> 5)] = loss;
    }
  }
  __syncthreads();
  if (t == 0) {
    out[OFF_B3] = YP[0] + YP[1];
    loss_partial[blockIdx.x] = YP[2] + YP[3];
  }
}

// sum of the partial rows, then an optional Adam update. A block of AD_P parameters by AD_G groups
// of rows: group g adds rows g, g + AD_G, ... (coalesced, many in flight), the groups' sums are
// added in order (one thread a parameter took its rows one after another, on 19 blocks: 6.6 us for
// 64 rows; now 4.9 us for 128 rows).
constexpr int AD_P = 32, AD_G = 16;
__global__ void __launch_bounds__(AD_P * AD_G)
k_mlp_adam(float* params, float* m, float* v, const float* partial, uint32_t nblk, float lr_eff,
           float eps_eff, float beta1, float beta2, int apply, float* grad_out,
           const float* loss_partial, float* loss_out) {
  __shared__ float sums[AD_G][AD_P];
  const uint32_t p = threadIdx.x % AD_P, grp = threadIdx.x / AD_P;
  const uint32_t i = blockIdx.x * AD_P + p;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  float g = 0.0f;
  if (i < (uint32_t)NPARAM) {
#pragma unroll 8
    for (uint32_t b = grp; b < nblk; b += AD_G) g += __ldcg(&partial[(size_t)b * NPARAM + i]);
  }
  sums[grp][p] = g;
  __syncthreads();
  if (grp == 1 && blockIdx.x == 0 && loss_out) {  // a warp: the blocks' losses
    float l = 0.0f;
    for (uint32_t b = p; b < nblk; b += AD_P) l += __ldcg(&loss_partial[b]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xFFFFFFFFu, l, o);
    if (p == 0) *loss_out = l;
  }
  if (grp != 0 || i >= (uint32_t)NPARAM) return;
#pragma unroll
  for (int q = 1; q < AD_G; ++q) g += sums[q][p];
  if (grad_out) grad_out[i] = g;
  if (!apply) return;
  const float mi = beta1 * __ldcg(&m[i]) + (1.0f - beta1) * g;
  const float vi = beta2 * __ldcg(&v[i]) + (1.0f - beta2) * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] = __ldcg(&params[i]) - lr_eff * mi / (sqrtf(vi) + eps_eff);
}

// BF16 inference copies of the master weights
__global__ void k_mlp_pack(const float* __restrict__ params, const float* __restrict__ norm,
                           float* __restrict__ fw, uint16_t* __restrict__ w2_umma,
                           uint32_t* __restrict__ w2_rm) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (uint32_t)(NH * NH)) {
    const uint32_t nn = i / NH, k = i % NH;
    const uint16_t b = __bfloat16_as_ushort(__float2bfloat16_rn(params[OFF_W2 + i]));
    w2_umma[((k / 8) * 8 + nn / 8) * 64 + (nn % 8) * 8 + (k % 8)] = b;
    if ((k & 1) == 0)
      w2_rm[nn * 32 + k / 2] = pack_bf16x2(params[OFF_W2 + i], params[OFF_W2 + i + 1]);
  }
  if (i < (uint32_t)(NH * NIN)) fw[FW_W1 + i] = bf16_round(params[OFF_W1 + i]);
  if (i < (uint32_t)NH) {
    fw[FW_B1 + i] = params[OFF_B1 + i];
    fw[FW_B2 + i] = params[OFF_B2 + i];
    fw[FW_W3 + i] = bf16_round(params[OFF_W3 + i]);
  }
  if (i == 0) fw[FW_B3] = params[OFF_B3];
  if (i < (uint32_t)NNORM) fw[FW_NORM + i] = norm[i];
}

int pack(cleo_b200_mlp* m) {
  k_mlp_pack<<<(NH * NH + 255) / 256, 256, 0, m->stream>>>(
      m->params, m->norm, m->fw, reinterpret_cast<uint16_t*>(m->w2_umma), m->w2_rm);
  MLP_TRY(cudaGetLastError());
  return CLEO_OK;
}

int ensure_blocks(cleo_b200_mlp* m, uint32_t nblk) {
  if (nblk <= m->cap_blocks) return CLEO_OK;
  MLP_TRY(cudaStreamSynchronize(m->stream));
  cudaFree(m->partial);
  cudaFree(m->loss_partial);
  m->partial = nullptr;
  m->loss_partial = nullptr;
  m->cap_blocks = 0;
  MLP_TRY(cudaMalloc(&m->partial, (size_t)nblk * NPARAM * sizeof(float)));
  MLP_TRY(cudaMalloc(&m->loss_partial, (size_t)nblk * sizeof(float)));
  m->cap_blocks = nblk;
  return CLEO_OK;
}

int set_fwdbwd_smem() {  // the attribute is per function and device: set before each use
  MLP_TRY(cudaFuncSetAttribute(k_mlp_fwdbwd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)TR_SMEM));
  return CLEO_OK;
}

uint32_t train_blocks(uint32_t count) {
  const uint32_t tiles = (count + TR_S - 1) / TR_S;
  return tiles < TR_BLOCKS_MAX ? tiles : TR_BLOCKS_MAX;
}

// one gradient and its sum (or Adam update). The update may start while the gradient kernel ends,
// and with `follows` the gradient kernel while the update before it does (programmatic launch:
// each waits for the other's results on the device). The first gradient of a call is launched
// plainly: it reads features that the stream's earlier work may have produced.
int launch_step(cleo_b200_mlp* m, uint32_t nb, bool follows, const float* feats,
                const float* target, uint32_t n, uint32_t count, uint64_t seed, uint32_t step,
                int random, float inv_count, float lr_eff, float eps_eff, float beta1,
                float beta2, int apply, float* grad_out, float* loss_out) {
  cudaLaunchAttribute pdl{};
  pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nb);
  cfg.blockDim = dim3(TR_T);
  cfg.dynamicSmemBytes = TR_SMEM;
  cfg.stream = m->stream;
  cfg.attrs = &pdl;
  cfg.numAttrs = follows ? 1 : 0;
  const float *params = m->params, *norm = m->norm, *partial = m->partial,
              *losses = m->loss_partial;
  MLP_TRY(cudaLaunchKernelEx(&cfg, k_mlp_fwdbwd, params, norm, feats, target, n, count, seed, step,
                             random, m->partial, m->loss_partial, inv_count));
  cfg.gridDim = dim3((NPARAM + AD_P - 1) / AD_P);
  cfg.blockDim = dim3(AD_P * AD_G);
  cfg.dynamicSmemBytes = 0;
  cfg.numAttrs = 1;
  MLP_TRY(cudaLaunchKernelEx(&cfg, k_mlp_adam, m->params, m->adam_m, m->adam_v, partial, nb, lr_eff,
                             eps_eff, beta1, beta2, apply, grad_out, losses, loss_out));
  return CLEO_OK;
}

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

bool bad_mlp(const cleo_b200_mlp* m) { return m == nullptr || m->params == nullptr; }

}  // namespace

int cleo_mlp_infer_view(const cleo_b200_mlp* m, Infer* out) {
  if (bad_mlp(m) || !out) return CLEO_ERR_ARGUMENT;
  out->fw = m->fw;
  out->w2_umma = m->w2_umma;
  out->w2_rm = m->w2_rm;
  out->err = m->err;
  return CLEO_OK;
}

extern "C" {

int cleo_b200_mlp_create(void* stream, uint64_t seed, cleo_b200_mlp** out) {
  if (!out) return CLEO_ERR_ARGUMENT;
  *out = nullptr;
  cleo_b200_mlp* m = new cleo_b200_mlp();
  MLP_TRY(cudaGetDevice(&m->device));
  m->stream = static_cast<cudaStream_t>(stream);
  int rc = CLEO_OK;
  auto al = [&](void** p, size_t bytes) {
    if (rc == CLEO_OK && cudaMalloc(p, bytes) != cudaSuccess) rc = CLEO_ERR_CUDA;
  };
  al((void**)&m->params, NPARAM * sizeof(float));
  al((void**)&m->adam_m, NPARAM * sizeof(float));
  al((void**)&m->adam_v, NPARAM * sizeof(float));
  al((void**)&m->norm, NNORM * sizeof(float));
  al((void**)&m->fw, NFW * sizeof(float));
  al((void**)&m->w2_umma, W2_UMMA_BYTES);
  al((void**)&m->w2_rm, NH * NH / 2 * sizeof(uint32_t));
  al((void**)&m->err, sizeof(uint32_t));
  al((void**)&m->phys_err, sizeof(DevError));
  if (rc != CLEO_OK) {
    cleo_b200_mlp_destroy(m);
    return rc;
  }
  // Glorot-uniform weights, zero biases, identity standardisation
  std::vector<float> p(NPARAM, 0.0f);
  uint64_t st = seed ^ 0x6D6C702D696E6974ull;
  auto uni = [&](float a) {
    const double u = (double)(splitmix(st) >> 11) * (1.0 / 9007199254740992.0);
    return (float)((2.0 * u - 1.0) * a);
  };
  const float a1 = std::sqrt(6.0f / (NIN + NH)), a2 = std::sqrt(6.0f / (NH + NH)),
              a3 = std::sqrt(6.0f / (NH + 1));
  for (int i = 0; i < NH * NIN; ++i) p[OFF_W1 + i] = uni(a1);
  for (int i = 0; i < NH * NH; ++i) p[OFF_W2 + i] = uni(a2);
  for (int i = 0; i < NH; ++i) p[OFF_W3 + i] = uni(a3);
  float nrm[NNORM];
  for (int i = 0; i < NIN; ++i) {
    nrm[i] = 0.0f;
    nrm[NIN + i] = 1.0f;
  }
  nrm[14] = 0.0f;
  nrm[15] = 1.0f;
  rc = cleo_b200_mlp_set_params(m, p.data(), nrm);
  if (rc != CLEO_OK) {
    cleo_b200_mlp_destroy(m);
    return rc;
  }
  *out = m;
  return CLEO_OK;
}

int cleo_b200_mlp_destroy(cleo_b200_mlp* m) {
  if (!m) return CLEO_OK;
  if (m->stream) cudaStreamSynchronize(m->stream);
  cudaFree(m->params);
  cudaFree(m->adam_m);
  cudaFree(m->adam_v);
  cudaFree(m->norm);
  cudaFree(m->fw);
  cudaFree(m->w2_umma);
  cudaFree(m->w2_rm);
  cudaFree(m->err);
  cudaFree(m->phys_err);
  cudaFree(m->partial);
  cudaFree(m->loss_partial);
  cudaFree(m->stats);
  delete m;
  return CLEO_OK;
}

int cleo_b200_mlp_set_params(cleo_b200_mlp* m, const float* params, const float* norm) {
  if (bad_mlp(m) || !params || !norm) return CLEO_ERR_ARGUMENT;
  MLP_TRY(cudaMemcpyAsync(m->params, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice,
                          m->stream));
  MLP_TRY(cudaMemcpyAsync(m->norm, norm, NNORM * sizeof(float), cudaMemcpyHostToDevice,
                          m->stream));
  MLP_TRY(cudaMemsetAsync(m->adam_m, 0, NPARAM * sizeof(float), m->stream));
  MLP_TRY(cudaMemsetAsync(m->adam_v, 0, NPARAM * sizeof(float), m->stream));
  MLP_TRY(cudaMemsetAsync(m->err, 0, sizeof(uint32_t), m->stream));
  MLP_TRY(cudaMemsetAsync(m->phys_err, 0, sizeof(DevError), m->stream));
  m->adam_t = 0;
  const int rc = pack(m);
  if (rc != CLEO_OK) return rc;
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return CLEO_OK;
}

int cleo_b200_mlp_get_params(cleo_b200_mlp* m, float* params, float* norm) {
  if (bad_mlp(m)) return CLEO_ERR_ARGUMENT;
  if (params)
    MLP_TRY(cudaMemcpyAsync(params, m->params, NPARAM * sizeof(float), cudaMemcpyDeviceToHost,
                            m->stream));
  if (norm)
    MLP_TRY(cudaMemcpyAsync(norm, m->norm, NNORM * sizeof(float), cudaMemcpyDeviceToHost,
                            m->stream));
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return CLEO_OK;
}

int cleo_b200_mlp_features(cleo_b200_mlp* m, size_t n, const double* d_radius,
                           const double* d_msol, const double* d_temp, const double* d_press,
                           const double* d_s_ratio, const double* d_delt,
                           const double* d_radius_new, float* d_features, float* d_target,
                           uint8_t* d_direct) {
  if (bad_mlp(m) || n > 0xFFFFFFFFull) return CLEO_ERR_ARGUMENT;
  if (n == 0) return CLEO_OK;
  if (!d_radius || !d_msol || !d_temp || !d_press || !d_s_ratio || !d_delt || !d_features ||
      (d_target && !d_radius_new))
    return CLEO_ERR_ARGUMENT;
  const uint32_t nb = (uint32_t)std::min<size_t>((n + 255) / 256, 148 * 16);
  k_mlp_features<<<nb, 256, 0, m->stream>>>((uint32_t)n, d_radius, d_msol, d_temp, d_press,
                                            d_s_ratio, d_delt, d_radius_new, d_features,
                                            d_target, d_direct, m->phys_err);
  MLP_TRY(cudaGetLastError());
  DevError e{};
  MLP_TRY(cudaMemcpyAsync(&e, m->phys_err, sizeof(e), cudaMemcpyDeviceToHost, m->stream));
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return e.code != 0 ? e.code : CLEO_OK;
}

int cleo_b200_mlp_fit_normalisation(cleo_b200_mlp* m, size_t n, const float* d_features,
                                    const float* d_target) {
  if (bad_mlp(m) || n == 0 || n > 0xFFFFFFFFull || !d_features || !d_target)
    return CLEO_ERR_ARGUMENT;
  const uint32_t nb = (uint32_t)std::min<size_t>((n + 255) / 256, 148 * 4);
  if (nb > m->cap_stat_blocks) {
    MLP_TRY(cudaStreamSynchronize(m->stream));
    cudaFree(m->stats);
    m->stats = nullptr;
    m->cap_stat_blocks = 0;
    MLP_TRY(cudaMalloc(&m->stats, (size_t)nb * 32 * sizeof(double)));
    m->cap_stat_blocks = nb;
  }
  k_mlp_stats<<<nb, 256, 0, m->stream>>>((uint32_t)n, d_features, d_target, m->stats);
  MLP_TRY(cudaGetLastError());
  std::vector<double> h((size_t)nb * 32);
  MLP_TRY(cudaMemcpyAsync(h.data(), m->stats, h.size() * sizeof(double), cudaMemcpyDeviceToHost,
                          m->stream));
  MLP_TRY(cudaStreamSynchronize(m->stream));
  double s[8] = {0}, q[8] = {0};
  for (uint32_t b = 0; b < nb; ++b)
    for (int c = 0; c < 8; ++c) {
      s[c] += h[b * 32 + c];
      q[c] += h[b * 32 + 8 + c];
    }
  float nrm[NNORM];
  for (int c = 0; c < 8; ++c) {
    const double mean = s[c] / (double)n;
    double var = q[c] / (double)n - mean * mean;
    if (!(var > 1e-24)) var = 1.0;  // a constant input carries no information: leave unscaled
    const double sd = std::sqrt(var);
    if (c < NIN) {
      nrm[c] = (float)mean;
      nrm[NIN + c] = (float)(1.0 / sd);
    } else {
      nrm[14] = (float)mean;
      nrm[15] = (float)sd;
    }
  }
  MLP_TRY(cudaMemcpyAsync(m->norm, nrm, sizeof(nrm), cudaMemcpyHostToDevice, m->stream));
  const int rc = pack(m);
  if (rc != CLEO_OK) return rc;
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return CLEO_OK;
}

int cleo_b200_mlp_loss_grad(cleo_b200_mlp* m, size_t n, const float* d_features,
                            const float* d_target, float* d_grad, float* d_loss) {
  if (bad_mlp(m) || n == 0 || n > (1u << 24) || !d_features || !d_target || !d_grad)
    return CLEO_ERR_ARGUMENT;
  const uint32_t nb = train_blocks((uint32_t)n);
  int rc = ensure_blocks(m, nb);
  if (rc != CLEO_OK) return rc;
  rc = set_fwdbwd_smem();
  if (rc != CLEO_OK) return rc;
  rc = launch_step(m, nb, false, d_features, d_target, (uint32_t)n, (uint32_t)n, 0, 0, 0,
                   1.0f / (float)n, 0.f, 0.f, 0.f, 0.f, 0, d_grad, d_loss);
  if (rc != CLEO_OK) return rc;
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return CLEO_OK;
}

int cleo_b200_mlp_train(cleo_b200_mlp* m, size_t n, const float* d_features,
                        const float* d_target, uint32_t steps, uint32_t batch, float lr,
                        uint64_t seed, float* d_loss_per_step) {
  if (bad_mlp(m) || n == 0 || n > 0xFFFFFFFFull || !d_features || !d_target || batch == 0 ||
      batch % 128 != 0 || batch > (1u << 20) || !(lr > 0.0f))
    return CLEO_ERR_ARGUMENT;
  const uint32_t nb = train_blocks(batch);
  int rc = ensure_blocks(m, nb);
  if (rc != CLEO_OK) return rc;
  rc = set_fwdbwd_smem();
  if (rc != CLEO_OK) return rc;
  const double beta1 = 0.9, beta2 = 0.999, eps = 1e-8;
  const uint32_t warm = steps / 50 + 1;
  for (uint32_t s = 0; s < steps; ++s) {
    // linear warm-up, then cosine decay to 2% of lr
    double f = 0.02 + 0.98 * 0.5 * (1.0 + std::cos(3.141592653589793 * (double)s / (double)steps));
    if (s < warm) f *= (double)(s + 1) / (double)warm;
    const uint64_t t = ++m->adam_t;
    const double bc1 = 1.0 - std::pow(beta1, (double)t), bc2 = 1.0 - std::pow(beta2, (double)t);
    const float lr_eff = (float)(lr * f * std::sqrt(bc2) / bc1);
    const float eps_eff = (float)(eps * std::sqrt(bc2));
    rc = launch_step(m, nb, s > 0, d_features, d_target, (uint32_t)n, batch, seed, s, 1,
                     1.0f / (float)batch, lr_eff, eps_eff, (float)beta1, (float)beta2, 1, nullptr,
                     d_loss_per_step ? d_loss_per_step + s : nullptr);
    if (rc != CLEO_OK) return rc;
  }
  MLP_TRY(cudaGetLastError());
  rc = pack(m);
  if (rc != CLEO_OK) return rc;
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return CLEO_OK;
}

int cleo_b200_mlp_infer(cleo_b200_mlp* m, size_t n, const float* d_features, float* d_out,
                        int path) {
  if (bad_mlp(m) || n > 0xFFFFFFFFull || !d_features || !d_out) return CLEO_ERR_ARGUMENT;
  if (n == 0) return CLEO_OK;
  Infer w;
  cleo_mlp_infer_view(m, &w);
  const ArrayIO io{d_features, d_out};
  const uint32_t nn = (uint32_t)n;
  if (path == CLEO_MLP_TCGEN05) {
    const uint32_t tiles = (nn + TILE_M - 1) / TILE_M;
    const uint32_t grid = tiles < TC_GRID_MAX ? tiles : TC_GRID_MAX;
    k_mlp_tc<ArrayIO><<<grid, 128, TC_SMEM, m->stream>>>(w, io, nn);
  } else if (path == CLEO_MLP_MMA_SYNC) {
    const uint32_t tiles = (nn + 15) / 16;
    uint32_t grid = (tiles + MMA_WARPS - 1) / MMA_WARPS;
    if (grid > 148u * 8u) grid = 148u * 8u;
    k_mlp_mma<ArrayIO><<<grid, 128, 0, m->stream>>>(w, io, nn);
  } else if (path == CLEO_MLP_FP32) {
    uint32_t grid = (nn + 127) / 128;
    if (grid > 148u * 8u) grid = 148u * 8u;
    k_mlp_fp32<ArrayIO><<<grid, 128, 0, m->stream>>>(w, io, nn);
  } else {
    return CLEO_ERR_ARGUMENT;
  }
  MLP_TRY(cudaGetLastError());
  uint32_t e = 0;
  MLP_TRY(cudaMemcpyAsync(&e, m->err, sizeof(e), cudaMemcpyDeviceToHost, m->stream));
  MLP_TRY(cudaStreamSynchronize(m->stream));
  return e != 0 ? (int)e : CLEO_OK;
}

}  // extern "C"
