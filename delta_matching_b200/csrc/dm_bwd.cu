// dQ of the backward without a workspace, on sm_100a: all matmuls on tcgen05 with TMEM accumulators, bit-deterministic (one
// writer per output element, fixed loop orders, no atomics).  dK and dV: dm_bwd_pipe.cu and
// dm_bwd_kv.cu; dQ from stored dS tiles: dm_bwd_p2.cu.
//
//   Query-stationary: CTA = (128-query tile, query head, batch); loops over key tiles: S, dP recomputed, dS codes staged in
//   shared memory, dQ += dS K block-scaled; dQ * softmax_scale rounded to bf16 once.  Also the form of the identity probe.
//
// Numerics (delta_matching/reference.py:476-518 with preset "sm100-mx", :612-613; kernel-side rules
// delta_matching/sm100/dm_bwd_sm100.py:5413-5433, 6175-6224 and attention_math_sm100.py:26-45):
//   P = ex2(fma(S_acc, (ks*qs)*log2e, -lse*log2e));  dP = dP_acc * (vs*dos);  dS = P * (dP - delta)   (fp32)
//   P^T codes: power-of-two scale per (key, 32 queries), amax 0 -> byte 0;   SFA_dV = p_sb (+) dos_sb
//   dS codes:  power-of-two scale per (128 queries x 32 keys), amax 0 -> scale 1;  SFA_dK = ds_sb (+) qs_sb,
//              dQ's scale along keys = ds_sb (+) ks_sb;  dQ = (dS K) * D^-0.5.
// P and dS are evaluated with the operations of the dK / dV kernel on the same accumulators, so the dS codes are that kernel's
// whenever the two MMA orientations return the same fp32 sums.
#include <cuda_bf16.h>
#include "dm_common.cuh"
#include "dm_kernels.h"

namespace dm {

// Row of an fp32 TMEM accumulator (32-column chunk c) -> bf16, 64 bytes to global.
__device__ __forceinline__ void store_bf16_chunk(const uint32_t (&r)[32], float mul, __nv_bfloat16* dst) {
  uint32_t w[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[2 * e]) * mul, __uint_as_float(r[2 * e + 1]) * mul);
    w[e] = *reinterpret_cast<uint32_t*>(&v);
  }
  uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
  for (int e = 0; e < 4; ++e) d4[e] = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
}

// ================================================================================================ dQ
template <int D>
struct DqSerialCfg {
  static constexpr int kSub = D / 128;
  static constexpr int kTileBytes = 128 * D;
  static constexpr int kStages = 2;
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0;
  static constexpr int kColSfa = 32;         // written after S is consumed: bytes = ds_sb (+) ks_sb per 32-key step
  static constexpr int kColOne = 36;
  static constexpr int kColDp = 128;
  static constexpr int kColDq = 256;
  static constexpr int kSmemQ = 0;
  static constexpr int kSmemDo = kTileBytes;
  static constexpr int kSmemK = 2 * kTileBytes;                      // [kStages]
  static constexpr int kSmemV = kSmemK + kStages * kTileBytes;       // [kStages]
  static constexpr int kSmemDs = kSmemV + kStages * kTileBytes;      // 128 x 128 dS codes, rows = queries
  static constexpr int kSmemRed = kSmemDs + 16384;                   // 2 x [4 warps][4 blocks] floats
  static constexpr int kSmemBar = kSmemRed + 2 * 16 * 4;
  static constexpr int kSmemBytes = kSmemBar + 256 + 1024;
};

template <int D>
__global__ void __launch_bounds__(192, 1)
bwd_dq_serial_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
              const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, const BwdParams p) {
  using C = DqSerialCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + C::kSmemQ;
  uint8_t* sDo = smem + C::kSmemDo;
  uint8_t* sK = smem + C::kSmemK;
  uint8_t* sV = smem + C::kSmemV;
  uint8_t* sDs = smem + C::kSmemDs;
  float* sRed = reinterpret_cast<float*>(smem + C::kSmemRed);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  uint64_t* bar_q = bars + 0;
  uint64_t* bar_s = bars + 1;
  uint64_t* bar_p = bars + 2;
  uint64_t* bar_done = bars + 3;
  uint64_t* full = bars + 4;
  uint64_t* empty = bars + 6;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 11);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int n_t = p.N / 128;
  const int qt = n_t - 1 - static_cast<int>(blockIdx.x);
  const int bh = blockIdx.y;
  const int b = bh / p.H, h = bh % p.H;
  const int bhk = b * p.Hk + h / (p.H / p.Hk);
  const int n_it = p.causal ? (qt + 1) : n_t;

  if (tid == 0) {
    mbar_init(bar_q, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_p, 128);
    mbar_init(bar_done, 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dep_wait();

  if (warp == 4) {
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_do);
      mbar_expect_tx(bar_q, 2 * C::kTileBytes);
      for (int s = 0; s < C::kSub; ++s) {
        tma_load_2d(sQ + s * 16384, &tm_q, bar_q, s * 128, bh * p.N + qt * 128);
        tma_load_2d(sDo + s * 16384, &tm_do, bar_q, s * 128, bh * p.N + qt * 128);
      }
      for (int it = 0; it < n_it; ++it) {
        const int st = it % C::kStages;
        if (it >= C::kStages) {
          if (!wait_or_abort(empty + st, ((it / C::kStages) - 1) & 1, abort_flag)) {
            raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInDq);
            break;
          }
        }
        const int row = bhk * p.N + it * 128;
        mbar_expect_tx(full + st, 2 * C::kTileBytes);
        for (int s = 0; s < C::kSub; ++s) {
          tma_load_2d(sK + st * C::kTileBytes + s * 16384, &tm_k, full + st, s * 128, row);
          tma_load_2d(sV + st * C::kTileBytes + s * 16384, &tm_v, full + st, s * 128, row);
        }
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      constexpr uint32_t kIdesc = idesc_f8(128, 128, false, false);
      const uint32_t q_lo = desc_lo(smem_u32(sQ)), do_lo = desc_lo(smem_u32(sDo)), ds_lo = desc_lo(smem_u32(sDs));
      const uint32_t k_lo0 = desc_lo(smem_u32(sK)), v_lo0 = desc_lo(smem_u32(sV));
      bool ok = wait_or_abort(bar_q, 0, abort_flag);
      for (int it = 0; ok && it < n_it; ++it) {
        const int st = it % C::kStages;
        if (!(ok = wait_or_abort(full + st, (it / C::kStages) & 1, abort_flag))) break;
        if (it > 0 && !(ok = wait_or_abort(bar_done, (it - 1) & 1, abort_flag))) break;
        tc_fence_after();
        const uint32_t k_lo = k_lo0 + st * (C::kTileBytes >> 4), v_lo = v_lo0 + st * (C::kTileBytes >> 4);
#pragma unroll
        for (int ks = 0; ks < D / 32; ++ks) {
          const uint32_t off = (ks / 4) * 1024 + (ks % 4) * 2;      // descriptor units of 16 bytes
          mma_f8_ss(tmem + C::kColS, q_lo + off, k_lo + off, kIdesc, ks > 0);
        }
#pragma unroll
        for (int ks = 0; ks < D / 32; ++ks) {
          const uint32_t off = (ks / 4) * 1024 + (ks % 4) * 2;
          mma_f8_ss(tmem + C::kColDp, do_lo + off, v_lo + off, kIdesc, ks > 0);
        }
        tc_commit(bar_s);
        if (!(ok = wait_or_abort(bar_p, it & 1, abort_flag))) break;
        tc_fence_after();
        // dQ += dS K: A = dS codes in shared memory (rows = queries, K-major), B = K tile MN-major (32 key rows per step)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
          for (int s = 0; s < C::kSub; ++s) {
            mma_mxf8_ss(tmem + C::kColDq + s * 128, ds_lo + ks * 2, k_lo + s * 1024 + ks * 256,
                        idesc_mxf8(128, 128, false, true, ks, ks), tmem + C::kColSfa, tmem + C::kColOne,
                        (it > 0) || (ks > 0));
          }
        }
        tc_commit(empty + st);
        tc_commit(bar_done);
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInDq);
    }
  } else {
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const int row = qt * 128 + tid;
    const int nblk = p.N / 32;
    const float qs = p.qs[static_cast<size_t>(bh) * nblk + row / 32];
    const float dos = p.dos[static_cast<size_t>(bh) * nblk + row / 32];
    const float neg_l2 = -(p.lse[static_cast<size_t>(bh) * p.N + row] * kLog2e);
    const float dlt = p.delta[static_cast<size_t>(bh) * p.N + row];
    const bool probe = p.rowsum_ds != nullptr;
    double rs_acc = 0.0, ap_acc = 0.0;
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const float4 ks4 = *reinterpret_cast<const float4*>(p.ks + static_cast<size_t>(bhk) * nblk + it * 4);
      const float4 vs4 = *reinterpret_cast<const float4*>(p.vs + static_cast<size_t>(bhk) * nblk + it * 4);
      const float ksv[4] = {ks4.x, ks4.y, ks4.z, ks4.w};
      const float vsv[4] = {vs4.x, vs4.y, vs4.z, vs4.w};
      const bool diag = p.causal && (it == qt);
      if (ok) ok = wait_warp(bar_s, it & 1, abort_flag);
      tc_fence_after();
      float ds[128];
      float bmax[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; ok && c < 4; ++c) {
        const float cc = (ksv[c] * qs) * kLog2e;
        const float aa = vsv[c] * dos;
        uint32_t rs[32], rd[32];
        tmem_ld32(tmem + lane_base + C::kColS + 32 * c, rs);
        tmem_ld32(tmem + lane_base + C::kColDp + 32 * c, rd);
        tmem_wait_ld();
        float am = 0.f, rsum = 0.f, asum = 0.f;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float s = __uint_as_float(rs[e]);
          if (diag && (32 * c + e > tid)) s = -INFINITY;
          const float pe = ex2_approx(fmaf(s, cc, neg_l2));
          const float dp = __uint_as_float(rd[e]) * aa;
          const float v = pe * (dp - dlt);
          ds[32 * c + e] = v;
          am = fmaxf(am, fabsf(v));
          if (probe) {
            rsum += v;
            asum += fabsf(pe * dp);
          }
        }
        bmax[c] = am;
        if (probe) {
          rs_acc += static_cast<double>(rsum);
          ap_acc += static_cast<double>(asum);
        }
      }
      // one scale per (this tile's 128 queries x 32 keys): reduce the block maxima over the four warps
      // (with 32 x 32 dS blocks the warp's own maximum is the block's)
      float* red = sRed + (it & 1) * 16;
      float wmx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        wmx[c] = warp_max(bmax[c]);
        if ((tid & 31) == 0) red[warp * 4 + c] = wmx[c];
      }
      bar_sync(1, 128);          // reached by every compute warp in every iteration, also after a failed wait
      if (!ok) continue;
      uint32_t sfw[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float am = p.ds32 ? wmx[c] : fmaxf(fmaxf(red[c], red[4 + c]), fmaxf(red[8 + c], red[12 + c]));
        const uint32_t dsb = pow2_sb(am, 127u);
        const float inv = sb_to_inv(dsb);
        sfw[c] = sb_mul(dsb, scale_to_sb(ksv[c]));
        // row tid of the dS tile: 16-byte chunk j of the row lands at chunk (j ^ (tid % 8)) (128-byte swizzle)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int e0 = 32 * c + 16 * j;
          uint4 w;
          w.x = cvt_e4m3x4(ds[e0 + 0] * inv, ds[e0 + 1] * inv, ds[e0 + 2] * inv, ds[e0 + 3] * inv);
          w.y = cvt_e4m3x4(ds[e0 + 4] * inv, ds[e0 + 5] * inv, ds[e0 + 6] * inv, ds[e0 + 7] * inv);
          w.z = cvt_e4m3x4(ds[e0 + 8] * inv, ds[e0 + 9] * inv, ds[e0 + 10] * inv, ds[e0 + 11] * inv);
          w.w = cvt_e4m3x4(ds[e0 + 12] * inv, ds[e0 + 13] * inv, ds[e0 + 14] * inv, ds[e0 + 15] * inv);
          const int chunk = (2 * c + j) ^ (tid & 7);
          *reinterpret_cast<uint4*>(sDs + tid * 128 + chunk * 16) = w;
        }
      }
      const uint32_t w = pack4(sfw[0], sfw[1], sfw[2], sfw[3]);
      tmem_st4(tmem + lane_base + C::kColSfa, w, w, w, w);
      tmem_st4(tmem + lane_base + C::kColOne, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
      tmem_wait_st();
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(bar_p);
    }
    if (ok) ok = wait_warp(bar_done, (n_it - 1) & 1, abort_flag);
    if (!ok) {
      raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDq);
    } else {
      tc_fence_after();
      __nv_bfloat16* dst = p.dq + static_cast<int64_t>(b) * p.dq_sb + static_cast<int64_t>(row) * p.dq_sn +
                           static_cast<int64_t>(h) * p.dq_sh;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_base + C::kColDq + 32 * c, r);
        tmem_wait_ld();
        store_bf16_chunk(r, p.sm_scale, dst + 32 * c);
      }
      if (probe) {
        p.rowsum_ds[static_cast<size_t>(bh) * p.N + row] = static_cast<float>(rs_acc);
        p.sum_abs_pdp[static_cast<size_t>(bh) * p.N + row] = static_cast<float>(ap_acc);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem, C::kTmemCols);
}


// ================================================================================================ dQ, pipelined (D = 128)
// One CTA per SM, 576 threads.  Warps 0-15: four compute groups of four warps; group g owns key block g of every tile
// (32 key columns = one whole dS scale block of 128 queries x 32 keys; thread t % 128 = query row = TMEM lane), which
// puts four compute warps on every scheduler.  Warp 16: TMA.  Warp 17: MMA.  The groups pull S and dP of tile i into
// registers and hand the accumulators back at once, so the tensor pipe computes S, dP of tile i+1 while the groups take
// the exponentials of tile i; dS codes go to shared memory (double-buffered), the scale words to TMEM columns of their
// own, and dQ += dS K runs behind the next tile's compute.
struct DqCfg {
  static constexpr int kTileBytes = 128 * 128;
  static constexpr int kStages = 4;
  static constexpr int kGroups = 4;
  static constexpr int kThreads = kGroups * 128 + 64;
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0, kColDp = 128, kColDq = 256;
  static constexpr int kColX = 384;          // 4 x 4 columns: scale word of key block g at kColX + 4 g (byte 0)
  static constexpr int kColOne = 400;        // 4 columns of 0x7F7F7F7F: scale 1.0 for the B operand
  static constexpr int kSmemQ = 0;
  static constexpr int kSmemDo = kTileBytes;
  static constexpr int kSmemK = 2 * kTileBytes;
  static constexpr int kSmemV = kSmemK + kStages * kTileBytes;
  static constexpr int kSmemDs = kSmemV + kStages * kTileBytes;      // 2 x (128 x 128 dS codes, rows = queries)
  static constexpr int kSmemRed = kSmemDs + 2 * kTileBytes;          // 2 x [16 warps] block maxima, then probe sums
  static constexpr int kSmemProbe = kSmemRed + 2 * 16 * 4;           // 3 slots x 3 groups x 128 rows x 2 doubles
  static constexpr int kSmemBar = kSmemProbe + 3 * 3 * 128 * 16;
  static constexpr int kSmemBytes = kSmemBar + 256 + 1024;
};

// Work item = one 128-query tile of one (batch, query head); persistent CTAs (one per SM) walk the item list with stride
// gridDim.x, heaviest items first, and the TMA / MMA pipeline runs across item boundaries.
struct DqWalk {                      // position of a role in the CTA's sequence of (item, key tile) pairs
  int item, it, n_it, qt, bh;
  uint32_t n_done;                   // items finished before the current one
};
__device__ __forceinline__ void dq_walk_set(DqWalk& w, const BwdParams& p, int n_t, int bh_count) {
  w.qt = n_t - 1 - w.item / bh_count;
  w.bh = w.item % bh_count;
  w.n_it = p.causal ? (w.qt + 1) : n_t;
  w.it = 0;
}

__global__ void __launch_bounds__(DqCfg::kThreads, 1)
bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
              const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, const BwdParams p) {
  using C = DqCfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + C::kSmemQ;
  uint8_t* sDo = smem + C::kSmemDo;
  uint8_t* sK = smem + C::kSmemK;
  uint8_t* sV = smem + C::kSmemV;
  uint8_t* sDs = smem + C::kSmemDs;
  float* sRed = reinterpret_cast<float*>(smem + C::kSmemRed);
  double* sProbe = reinterpret_cast<double*>(smem + C::kSmemProbe);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  uint64_t* bar_q = bars + 0;        // Q and dO of the item landed
  uint64_t* bar_qfree = bars + 1;    // every MMA that reads Q / dO of the item is done
  uint64_t* bar_s = bars + 2;        // S and dP of the tile ready (MMA commit)
  uint64_t* bar_free = bars + 3;     // every compute warp holds its part of the tile in registers (16 arrivals)
  uint64_t* bar_p = bars + 4;        // dS codes and scale words written (16 arrivals)
  uint64_t* bar_done = bars + 5;     // dQ chain of the tile done (MMA commit)
  uint64_t* bar_dqfree = bars + 6;   // the item's dQ accumulator has been read out (16 arrivals)
  uint64_t* full = bars + 7;         // [kStages]
  uint64_t* empty = bars + 7 + C::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7 + 2 * C::kStages);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 8 + 2 * C::kStages);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int n_t = p.N / 128;
  const int bh_count = p.B * p.H;
  const int n_items = n_t * bh_count;

  if (tid == 0) {
    mbar_init(bar_q, 1);
    mbar_init(bar_qfree, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_free, C::kGroups * 4);
    mbar_init(bar_p, C::kGroups * 4);
    mbar_init(bar_done, 1);
    mbar_init(bar_dqfree, C::kGroups * 4);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 17) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dep_wait();

  if (warp == 16) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_do);
      uint32_t g = 0, n_done = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < n_items; item += gridDim.x, ++n_done) {
        const int qt = n_t - 1 - item / bh_count, bh = item % bh_count;
        const int bhk = (bh / p.H) * p.Hk + (bh % p.H) / (p.H / p.Hk);
        const int n_it = p.causal ? (qt + 1) : n_t;
        if (n_done > 0 && !(ok = wait_or_abort(bar_qfree, (n_done - 1) & 1, abort_flag))) break;
        mbar_expect_tx(bar_q, 2 * C::kTileBytes);
        tma_load_2d(sQ, &tm_q, bar_q, 0, bh * p.N + qt * 128);
        tma_load_2d(sDo, &tm_do, bar_q, 0, bh * p.N + qt * 128);
        for (int it = 0; it < n_it; ++it, ++g) {
          const uint32_t st = g % C::kStages;
          if (g >= C::kStages && !(ok = wait_or_abort(empty + st, ((g / C::kStages) - 1) & 1, abort_flag))) break;
          const int row = bhk * p.N + it * 128;
          mbar_expect_tx(full + st, 2 * C::kTileBytes);
          tma_load_2d(sK + st * C::kTileBytes, &tm_k, full + st, 0, row);
          tma_load_2d(sV + st * C::kTileBytes, &tm_v, full + st, 0, row);
        }
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInDq);
    }
  } else if (warp == 17) {
    // ------------------------------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t kIdesc = idesc_f8(128, 128, false, false);
      const uint32_t q_lo = desc_lo(smem_u32(sQ)), do_lo = desc_lo(smem_u32(sDo)), ds_lo0 = desc_lo(smem_u32(sDs));
      const uint32_t k_lo0 = desc_lo(smem_u32(sK)), v_lo0 = desc_lo(smem_u32(sV));
      bool ok = true;
      // `nx` runs one tile ahead of `cur`: S / dP of the next tile (possibly the first tile of the next item) are
      // issued as soon as the compute warps hold the current tile in registers.
      DqWalk cur{static_cast<int>(blockIdx.x), 0, 0, 0, 0, 0}, nx = cur;
      uint32_t g_nx = 0;                                // tiles whose S / dP have been issued
      auto issue_s_dp = [&]() -> bool {                 // for the tile `nx` points at; advances nx
        if (nx.it == 0 && !wait_or_abort(bar_q, nx.n_done & 1, abort_flag)) return false;
        const uint32_t st = g_nx % C::kStages;
        if (!wait_or_abort(full + st, (g_nx / C::kStages) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t k_lo = k_lo0 + st * (C::kTileBytes >> 4), v_lo = v_lo0 + st * (C::kTileBytes >> 4);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_f8_ss(tmem + C::kColS, q_lo + ks * 2, k_lo + ks * 2, kIdesc, ks > 0);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_f8_ss(tmem + C::kColDp, do_lo + ks * 2, v_lo + ks * 2, kIdesc, ks > 0);
        tc_commit(bar_s);
        ++g_nx;
        if (++nx.it == nx.n_it) {                       // last tile of the item: its Q / dO may be replaced
          tc_commit(bar_qfree);
          nx.item += gridDim.x;
          ++nx.n_done;
          if (nx.item < n_items) dq_walk_set(nx, p, n_t, bh_count);
        }
        return true;
      };
      if (cur.item < n_items) {
        dq_walk_set(cur, p, n_t, bh_count);
        nx = cur;
        ok = issue_s_dp();
      }
      uint32_t g = 0;                                   // tiles whose dQ chain has been issued
      while (ok && cur.item < n_items) {
        const uint32_t st = g % C::kStages;
        if (!(ok = wait_or_abort(bar_free, g & 1, abort_flag))) break;
        if (nx.item < n_items && !(ok = issue_s_dp())) break;
        if (!(ok = wait_or_abort(bar_p, g & 1, abort_flag))) break;
        // the first chain of an item overwrites the accumulator: the previous item's dQ must have been read out
        if (cur.it == 0 && cur.n_done > 0 && !(ok = wait_or_abort(bar_dqfree, (cur.n_done - 1) & 1, abort_flag))) break;
        tc_fence_after();
        // dQ += dS K: A = dS codes in shared memory (rows = queries, K-major), B = K tile MN-major (32 key rows per step)
        const uint32_t ds_lo = ds_lo0 + (g & 1) * (C::kTileBytes >> 4), k_lo = k_lo0 + st * (C::kTileBytes >> 4);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_mxf8_ss(tmem + C::kColDq, ds_lo + ks * 2, k_lo + ks * 256, idesc_mxf8(128, 128, false, true, 0, 0),
                      tmem + C::kColX + 4 * ks, tmem + C::kColOne, (cur.it > 0) || (ks > 0));
        tc_commit(empty + st);
        tc_commit(bar_done);
        ++g;
        if (++cur.it == cur.n_it) {
          cur.item += gridDim.x;
          ++cur.n_done;
          if (cur.item < n_items) dq_walk_set(cur, p, n_t, bh_count);
        }
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInDq);
    }
  } else {
    // ------------------------------------------------------------------------------------------ compute groups
    const int wg = warp >> 2;
    const int r = tid & 127;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int nblk = p.N / 32;
    const bool probe = p.rowsum_ds != nullptr;
    uint32_t g = 0, n_done = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++n_done) {
      const int qt = n_t - 1 - item / bh_count, bh = item % bh_count;
      const int b = bh / p.H, h = bh % p.H;
      const int bhk = b * p.Hk + h / (p.H / p.Hk);
      const int n_it = p.causal ? (qt + 1) : n_t;
      const int row = qt * 128 + r;
      const float qs = p.qs[static_cast<size_t>(bh) * nblk + row / 32];
      const float dos = p.dos[static_cast<size_t>(bh) * nblk + row / 32];
      const float2 nl2 = splat2(-(p.lse[static_cast<size_t>(bh) * p.N + row] * kLog2e));
      const float2 ndl = splat2(-p.delta[static_cast<size_t>(bh) * p.N + row]);
      const float* ks_base = p.ks + static_cast<size_t>(bhk) * nblk + wg;
      const float* vs_base = p.vs + static_cast<size_t>(bhk) * nblk + wg;
      float ks1 = *ks_base, vs1 = *vs_base;
      double rs_acc = 0.0, ap_acc = 0.0;
      for (int it = 0; it < n_it; ++it, ++g) {
        const float ksv = ks1, vsv = vs1;
        if (it + 1 < n_it) {
          ks1 = ks_base[(it + 1) * 4];
          vs1 = vs_base[(it + 1) * 4];
        }
        const bool diag = p.causal && (it == qt);
        float2 v[16];
        float wm = 0.f;
        if (ok) ok = wait_warp(bar_s, g & 1, abort_flag);
        if (ok) {
          tc_fence_after();
          uint32_t rs[32], rd[32];
          tmem_ld32(tmem + lane_base + C::kColS + 32 * wg, rs);
          tmem_ld32(tmem + lane_base + C::kColDp + 32 * wg, rd);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if ((tid & 31) == 0) mbar_arrive(bar_free);    // this warp's part of the accumulators may be overwritten now
          if (diag) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (32 * wg + e > r) rs[e] = 0xff800000u;  // -inf: key index above the query index
          }
          const float2 cc = splat2((ksv * qs) * kLog2e), aa = splat2(vsv * dos);
          float am0 = 0.f, am1 = 0.f;
          float2 rsum = make_float2(0.f, 0.f), asum = rsum;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 pe = ex2_2(fma2(make_float2(__uint_as_float(rs[2 * e]), __uint_as_float(rs[2 * e + 1])), cc, nl2));
            const float2 dp = make_float2(__uint_as_float(rd[2 * e]), __uint_as_float(rd[2 * e + 1]));
            const float2 t = fma2(dp, aa, ndl);          // dP_acc * a - delta: a is a power of two, the product is exact
            const float2 d = mul2(pe, t);
            v[e] = d;
            if (e & 1) am1 = max3(am1, fabsf(d.x), fabsf(d.y));
            else am0 = max3(am0, fabsf(d.x), fabsf(d.y));
            if (probe) {
              rsum = add2(rsum, d);
              const float2 pd = mul2(pe, mul2(dp, aa));
              asum = add2(asum, make_float2(fabsf(pd.x), fabsf(pd.y)));
            }
          }
          if (probe) {
            rs_acc += static_cast<double>(rsum.x) + static_cast<double>(rsum.y);
            ap_acc += static_cast<double>(asum.x) + static_cast<double>(asum.y);
          }
          // one scale per (128 queries x 32 keys): the maxima of this group's four warps meet in shared memory
          // (with 32 x 32 dS blocks the warp's own maximum is the block's)
          wm = warp_max(fmaxf(am0, am1));
          if ((tid & 31) == 0) sRed[(g & 1) * 16 + warp] = wm;
        }
        bar_sync(1 + wg, 128);        // reached by every warp of the group in every iteration, also after a failed wait
        if (ok && g > 0) ok = wait_warp(bar_done, (g - 1) & 1, abort_flag);   // the previous chain has read its scale words
        if (!ok) continue;
        const float* red = sRed + (g & 1) * 16 + wg * 4;
        const uint32_t dsb = pow2_sb(p.ds32 ? wm : fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])), 127u);
        uint32_t w[8];
        codes32(v, sb_to_inv(dsb), w);
        // row r of the dS tile: 16-byte chunk j of the row lands at chunk (j ^ (r % 8)) (128-byte swizzle)
        uint8_t* ds_row = sDs + (g & 1) * C::kTileBytes + r * 128;
        sts_u4(ds_row + (((2 * wg) ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
        sts_u4(ds_row + (((2 * wg + 1) ^ (r & 7)) << 4), w[4], w[5], w[6], w[7]);
        const uint32_t word = sb_mul(dsb, scale_to_sb(ksv));
        tmem_st4(tmem + lane_base + C::kColX + 4 * wg, word, word, word, word);
        if (wg == 0) tmem_st4(tmem + lane_base + C::kColOne, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
        tmem_wait_st();
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bar_p);
      }
      // item epilogue: dQ of the item out of TMEM, then hand the accumulator to the next item
      if (ok) ok = wait_warp(bar_done, (g - 1) & 1, abort_flag);
      if (ok) {
        tc_fence_after();
        __nv_bfloat16* dst = p.dq + static_cast<int64_t>(b) * p.dq_sb + static_cast<int64_t>(row) * p.dq_sn +
                             static_cast<int64_t>(h) * p.dq_sh + 32 * wg;
        uint32_t rr[32];
        tmem_ld32(tmem + lane_base + C::kColDq + 32 * wg, rr);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bar_dqfree);
        store_bf16_chunk(rr, p.sm_scale, dst);
      }
      if (probe) {                     // identity probe: the groups' partial row sums meet in shared memory
        const int slot = n_done % 3;   // slots and barriers rotate: a warp is at most two items ahead of another
        double* pr = sProbe + slot * (3 * 128 * 2);
        if (wg > 0) {
          pr[((wg - 1) * 128 + r) * 2] = rs_acc;
          pr[((wg - 1) * 128 + r) * 2 + 1] = ap_acc;
          bar_arrive(5 + slot, C::kGroups * 128);
        } else {
          bar_sync(5 + slot, C::kGroups * 128);
          for (int gi = 0; gi < C::kGroups - 1; ++gi) {
            rs_acc += pr[(gi * 128 + r) * 2];
            ap_acc += pr[(gi * 128 + r) * 2 + 1];
          }
          if (ok) {
            p.rowsum_ds[static_cast<size_t>(bh) * p.N + row] = static_cast<float>(rs_acc);
            p.sum_abs_pdp[static_cast<size_t>(bh) * p.N + row] = static_cast<float>(ap_acc);
          }
        }
      }
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDq);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 17) tmem_dealloc(tmem, C::kTmemCols);
}

// ================================================================================================ launchers
template <typename K>
static cudaError_t set_smem(K kernel, int bytes, bool* done) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    done[dev] = true;
  }
  return cudaSuccess;
}

template <int D>
static cudaError_t launch_dq_serial_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                      const CUtensorMap& tdo, const BwdParams& p, cudaStream_t stream) {
  using C = DqSerialCfg<D>;
  static bool done[64] = {};
  cudaError_t e = set_smem(bwd_dq_serial_kernel<D>, C::kSmemBytes, done);
  if (e != cudaSuccess) return e;
  dim3 grid(p.N / 128, p.B * p.H);
  count_launch();
  return launch_chained(bwd_dq_serial_kernel<D>, grid, 192, C::kSmemBytes, stream, tq, tk, tv, tdo, p);
}

cudaError_t launch_bwd_dq(int D, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                          const CUtensorMap& tdo, const BwdParams& p, cudaStream_t stream) {
  // head_dim 256: dQ alone fills 256 TMEM columns, which leaves no room for the pipelined kernel's separate scale-word
  // columns; it keeps the kernel that serialises MMA and compute inside a CTA.
  if (D != 128) return launch_dq_serial_t<256>(tq, tk, tv, tdo, p, stream);
  static bool done[64] = {};
  cudaError_t e = set_smem(bwd_dq_kernel, DqCfg::kSmemBytes, done);
  if (e != cudaSuccess) return e;
  const int sms = sm_count();
  const int n_items = (p.N / 128) * p.B * p.H;
  count_launch();
  return launch_chained(bwd_dq_kernel, n_items < sms ? n_items : sms, DqCfg::kThreads, DqCfg::kSmemBytes, stream, tq, tk, tv, tdo, p);
}

}  // namespace dm
