// One 32-token x D block of a producer (rule: dm_quant.cu), for the quantiser kernels and for pass 0 of small problems, which quantises
// its own dO tile (dm_delta.cu).
#pragma once
#include <cuda_bf16.h>
#include "dm_common.cuh"
#include "dm_kernels.h"

namespace dm {

__device__ __forceinline__ void bf16x8_to_float(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// kMean / kStale: the K tensor alone subtracts a mean and the dO tensor of the stale mode alone reads O; compiled out
// elsewhere, the kernel needs fewer registers and more of its small CTAs fit an SM (more loads in flight).
// Executed by 128 threads (tid 0-127), which meet at the named barrier `bar`.
template <int D, bool kMean, bool kStale>
__device__ __forceinline__ void quant_block(const QuantParams& p, int blk, int bh, float* wmax, int tid = threadIdx.x, int bar = 1,
                                            const float* mean_row = nullptr) {
  constexpr int kTpr = D / 16;           // threads per token row (16 elements each)
  constexpr int kRpp = 128 / kTpr;       // rows per pass
  constexpr int kPass = 32 / kRpp;
  const int b = bh / p.H, h = bh % p.H;
  const int c16 = tid % kTpr, r0 = tid / kTpr;
  const __nv_bfloat16* xb = p.x + b * p.sb + h * p.sh + static_cast<int64_t>(blk) * 32 * p.sn + c16 * 16;

  float mean[kMean ? 16 : 1];
  if (kMean) {
    const float4* mp = reinterpret_cast<const float4*>((mean_row != nullptr ? mean_row : p.mean + static_cast<size_t>(bh) * D) + c16 * 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = mp[i];
      mean[4 * i] = v.x; mean[4 * i + 1] = v.y; mean[4 * i + 2] = v.z; mean[4 * i + 3] = v.w;
    }
  }

  float y[kPass][16];
  float amax = 0.f;
#pragma unroll
  for (int ps = 0; ps < kPass; ++ps) {
    const int r = r0 + ps * kRpp;
    const uint4* src = reinterpret_cast<const uint4*>(xb + r * p.sn);
    const uint4 v0 = __ldg(src), v1 = __ldg(src + 1);
    bf16x8_to_float(v0, &y[ps][0]);
    bf16x8_to_float(v1, &y[ps][8]);
    if (kStale) {
      // stale delta = sum_d dO * O on the raw bf16 values (delta_matching/reference.py:500-501)
      const __nv_bfloat16* ob = p.o + b * p.o_sb + h * p.o_sh + (static_cast<int64_t>(blk) * 32 + r) * p.o_sn + c16 * 16;
      const uint4 o0 = __ldg(reinterpret_cast<const uint4*>(ob)), o1 = __ldg(reinterpret_cast<const uint4*>(ob) + 1);
      float of[16];
      bf16x8_to_float(o0, &of[0]);
      bf16x8_to_float(o1, &of[8]);
      float d = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) d = fmaf(y[ps][i], of[i], d);
#pragma unroll
      for (int off = kTpr / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
      if (c16 == 0) p.delta[static_cast<size_t>(bh) * p.N + blk * 32 + r] = d;
    }
    // (x - 0) * prescale and x * prescale are the same fp32 value, so leaving the subtraction out changes no bit
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      y[ps][i] = kMean ? (y[ps][i] - mean[i]) * p.prescale : y[ps][i] * p.prescale;
      amax = fmaxf(amax, fabsf(y[ps][i]));
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if ((tid & 31) == 0) wmax[tid >> 5] = amax;
  bar_sync(bar, 128);
  amax = fmaxf(fmaxf(wmax[0], wmax[1]), fmaxf(wmax[2], wmax[3]));
  const uint32_t sb = pow2_sb(amax, 127u);
  const float inv = sb_to_inv(sb);
  if (tid == 0) p.scales[static_cast<size_t>(bh) * (p.N / 32) + blk] = sb_to_scale(sb);

  uint8_t* cb = p.codes + (static_cast<size_t>(bh) * p.N + static_cast<size_t>(blk) * 32) * D + c16 * 16;
#pragma unroll
  for (int ps = 0; ps < kPass; ++ps) {
    const int r = r0 + ps * kRpp;
    uint4 w;
    w.x = cvt_e4m3x4(y[ps][0] * inv, y[ps][1] * inv, y[ps][2] * inv, y[ps][3] * inv);
    w.y = cvt_e4m3x4(y[ps][4] * inv, y[ps][5] * inv, y[ps][6] * inv, y[ps][7] * inv);
    w.z = cvt_e4m3x4(y[ps][8] * inv, y[ps][9] * inv, y[ps][10] * inv, y[ps][11] * inv);
    w.w = cvt_e4m3x4(y[ps][12] * inv, y[ps][13] * inv, y[ps][14] * inv, y[ps][15] * inv);
    *reinterpret_cast<uint4*>(cb + static_cast<size_t>(r) * D) = w;
  }
}

}  // namespace dm
