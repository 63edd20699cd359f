// The backward's arithmetic per (key row, 32 queries), shared by the key-stationary kernel (dm_bwd_kv.cu) and the tile-parallel
// one (dm_bwd_tiles.cu): a call may take either, so both have to produce the same bits.
#pragma once
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

}  // namespace dm
