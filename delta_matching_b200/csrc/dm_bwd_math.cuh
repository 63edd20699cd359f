// The backward's arithmetic per (key row, 32 queries), shared by the key-stationary kernels (dm_bwd_kv.cu, dm_bwd_pipe.cu) and the
// tile-parallel one (dm_bwd_tiles.cu): a call may take any, so all have to produce the same bits.  And the write-out of accumulators.
#pragma once
#include <cuda_bf16.h>
#include "dm_common.cuh"

namespace dm {

// P = ex2(S_acc cc - lse log2e); cc: (ks qs) log2e twice; lse: shared address of the 32 values of -lse log2e.  Returns the maximum.
__device__ __forceinline__ float p_block(const uint32_t (&s)[32], float2 cc, uint32_t lse, float2 (&p)[16]) {
  float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    const float4 l = lds_f4(lse + 8 * e);
    p[e] = ex2_2(fma2(make_float2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), cc, make_float2(l.x, l.y)));
    p[e + 1] = ex2_2(fma2(make_float2(__uint_as_float(s[2 * e + 2]), __uint_as_float(s[2 * e + 3])), cc, make_float2(l.z, l.w)));
    m0 = max3(m0, p[e].x, p[e].y);
    m1 = max3(m1, p[e + 1].x, p[e + 1].y);
  }
  return fmaxf(m0, m1);
}

// -dS = P (delta - dP_acc a) in the place of P; na: -a = -(vs dos) twice, a power of two, so that the product is exact; the sign is
// undone by the codes' scale.  delta: shared address of the 32 values.  Returns the maximum of |dS|.
__device__ __forceinline__ float neg_ds_block(const uint32_t (&dp)[32], float2 na, uint32_t delta, float2 (&p)[16]) {
  float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    const float4 d = lds_f4(delta + 8 * e);
    const float2 t0 = fma2(make_float2(__uint_as_float(dp[2 * e]), __uint_as_float(dp[2 * e + 1])), na, make_float2(d.x, d.y));
    const float2 t1 = fma2(make_float2(__uint_as_float(dp[2 * e + 2]), __uint_as_float(dp[2 * e + 3])), na, make_float2(d.z, d.w));
    p[e] = mul2(p[e], t0);
    p[e + 1] = mul2(p[e + 1], t1);
    m0 = max3(m0, fabsf(p[e].x), fabsf(p[e].y));
    m1 = max3(m1, fabsf(p[e + 1].x), fabsf(p[e + 1].y));
  }
  return fmaxf(m0, m1);
}

// The codes of query block `blk` into row r of a [key][query] code tile in 128-byte-swizzled shared memory (16-byte chunk j of row
// r at chunk j ^ (r % 8)); row: shared address of the row.
__device__ __forceinline__ void stage_codes(uint32_t row, int r, int blk, const uint32_t (&w)[8]) {
  const int j = 2 * blk;
  sts_u4(row + ((j ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
  sts_u4(row + (((j + 1) ^ (r & 7)) << 4), w[4], w[5], w[6], w[7]);
}

// 32 columns of the warp's 32 TMEM lanes, times mul, to bf16 rows; dst: the warp's first row, sn: elements between rows.  A thread that
// held a row would write 16 bytes into each of 32 lines per instruction.  Four threads share a row instead: loaded as MMA
// fragments, a 4 x 4 exchange gives each of them 16 contiguous bytes of the row's 64.  Streaming kernel, us: 48.6 -> 45.8 (B=3 N=1792
// H=15 Hk=5), 271 -> 267 (B=4 N=4096 H=32 Hk=8), 697 -> 667 (head_dim 256, B=2 N=8192 H=16); an item of dm_bwd_pipe.cu 3.3 us -> 1.
__device__ __forceinline__ void store_rows32(uint32_t taddr, float mul, __nv_bfloat16* dst, int64_t sn) {
  const int lane = threadIdx.x & 31, i = lane & 3;
  dst += (lane >> 2) * sn + 8 * i;
#pragma unroll
  for (int x = 0; x < 2; ++x) {                          // lanes 0 - 15, then 16 - 31
    uint32_t rr[16];
    tmem_ld_frag32(taddr + (static_cast<uint32_t>(16 * x) << 16), rr);
    tmem_wait_ld();
#pragma unroll
    for (int h = 0; h < 2; ++h) {                        // rows lane / 4 and lane / 4 + 8
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(rr[4 * j + 2 * h]) * mul, __uint_as_float(rr[4 * j + 2 * h + 1]) * mul);
        w[j] = *reinterpret_cast<uint32_t*>(&v);         // columns 8 j + 2 i and the next
      }
      // 4 x 4 transposition in the group of four lanes: word j of lane i <-> word i of lane j
#pragma unroll
      for (int bit = 1; bit < 4; bit *= 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j & bit) continue;
          const bool up = (i & bit) != 0;
          const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? w[j] : w[j | bit], bit);
          if (up) w[j] = got; else w[j | bit] = got;
        }
      }
      *reinterpret_cast<uint4*>(dst + (16 * x + 8 * h) * sn) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

}  // namespace dm
