// Backward of small problems, tile-parallel: every live 128 x 128 (key x query) tile on its own, its P^T and dS^T codes and
// scale words left in a workspace, from which one streaming launch (dm_bwd_p2.cu) makes dV, dK and dQ.
//
// The key-stationary kernels (dm_bwd_pipe.cu, dm_bwd_kv.cu) walk all tiles of a key tile, the whole GQA group's, in one CTA: a chain of
// (H / Hk) (N / 128) tiles at about 1.6 us each, however many SMs are idle.  At B=1 N=1024 H=8 Hk=2 that is 16 chains of up to
// 32 tiles on 148 SMs.  Here the tiles are dealt out evenly, and what stays a chain is the accumulation alone, at about a
// fifth of the time per tile.  The arithmetic, the order of every sum and so the bits are those of the key-stationary kernel.
#include <cuda_bf16.h>
#include "dm_bwd_math.cuh"
#include "dm_common.cuh"
#include "dm_kernels.h"

namespace dm {

// Four compute warpgroups share a tile (thread = key row = TMEM lane, and one block of 32 queries; eight warps with two blocks
// each take as long), then the MMA, TMA, vector and store warps.  S^T and dP^T are double-buffered in TMEM (2 x (128 + 128) columns) and nothing else is
// there, so the MMAs of the next tile run under the arithmetic of this one and a Q / dO stage is free as soon as they are done.
template <int D>
struct TilesCfg {
  static constexpr int kSub = D / 128;                 // 128-byte-wide sub-tiles of an operand row
  static constexpr int kTileBytes = 128 * D;           // K, V, Q, dO tile
  static constexpr int kCodeBytes = 128 * 128;
  static constexpr int kKvBufs = (D == 128) ? 2 : 1;
  static constexpr int kStages = (D == 128) ? 2 : 1;
  static constexpr int kVecs = 4;
  static constexpr int kComputeWarps = 16;
  static constexpr int kThreads = (kComputeWarps + 4) * 32;
  static constexpr int kSmemK = 0;                                        // [kKvBufs] K, V
  static constexpr int kSmemQ = kKvBufs * 2 * kTileBytes;                 // [kStages]
  static constexpr int kSmemDo = kSmemQ + kStages * kTileBytes;           // [kStages]
  static constexpr int kSmemOut = kSmemDo + kStages * kTileBytes;         // [2] P^T codes, dS^T codes
  static constexpr int kSmemVec = kSmemOut + 4 * kCodeBytes;              // [kVecs] vectors of the query tile (bytes):
  static constexpr int kVecLse = 0, kVecDelta = 512, kVecQs = 1024, kVecDos = 1040, kVecBytes = 1056;
  static constexpr int kSmemXch = kSmemVec + kVecs * kVecBytes;           // [2 parities][16 warps] floats
  static constexpr int kSmemBar = kSmemXch + 2 * 16 * 4;
  static constexpr int kSmemBytes = kSmemBar + 512;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
};

// Position in the list of live tiles: kv head, key tile, head of the group, query tile, the last one fastest.
struct TileWalk {
  int bhk, kt, g, qt;
  int row, tile;               // code row of the tile's Q / dO; index of the tile in the workspace
  __device__ __forceinline__ void place(const BwdParams& p, int n_t, int rep) {
    const int bh = bhk * rep + g;
    row = bh * p.N + qt * 128;
    tile = (bh * n_t + qt) * n_t + kt;
  }
  __device__ __forceinline__ void seek(const BwdParams& p, int n_t, int rep, int index) {
    const int per_kv = rep * (p.causal ? n_t * (n_t + 1) / 2 : n_t * n_t);
    bhk = index / per_kv;
    index %= per_kv;
    kt = 0;
    for (int per = rep * n_t; index >= per; index -= per, per -= p.causal ? rep : 0) ++kt;
    const int q0 = p.causal ? kt : 0;
    g = index / (n_t - q0);
    qt = q0 + index % (n_t - q0);
    place(p, n_t, rep);
  }
  __device__ __forceinline__ bool next(const BwdParams& p, int n_t, int rep) {       // true: another key tile
    row += 128;
    tile += n_t;
    if (++qt < n_t) return false;
    bool fresh = false;
    if (++g == rep) {
      fresh = true;
      g = 0;
      if (++kt == n_t) {
        kt = 0;
        ++bhk;
      }
    }
    qt = p.causal ? kt : 0;
    place(p, n_t, rep);
    return fresh;
  }
};

template <int D, bool DS32>
__global__ void __launch_bounds__(TilesCfg<D>::kThreads, 1)
bwd_tiles_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                 const __grid_constant__ CUtensorMap tm_ds, const __grid_constant__ CUtensorMap tm_p, const BwdParams p) {
  using C = TilesCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  uint64_t* kv_full = bars + 0;      // [2] K and V landed
  uint64_t* kv_empty = bars + 2;     // [2] the last MMA that reads them is done (MMA commit)
  uint64_t* full_q = bars + 4;       // [2] Q landed
  uint64_t* full_d = bars + 6;       // [2] dO landed
  uint64_t* empty_q = bars + 8;      // [2] S^T of the stage is done (MMA commit)
  uint64_t* empty_d = bars + 10;     // [2] dP^T of the stage is done
  uint64_t* bar_s = bars + 12;       // [2] S^T of the buffer landed
  uint64_t* bar_dp = bars + 14;      // [2] dP^T of the buffer landed
  uint64_t* s_free = bars + 16;      // [2] the compute warps hold the buffer's S^T (one arrival per warp)
  uint64_t* dp_free = bars + 18;     // [2] likewise, dP^T
  uint64_t* staged = bars + 20;      // [2] codes of the tile written to the staging tiles (one arrival per warp)
  uint64_t* stage_free = bars + 22;  // [2] they have been read by the TMA stores
  uint64_t* vec_full = bars + 24;    // [kVecs] vectors landed
  uint64_t* vec_ok = bars + 28;      // [kVecs] -lse * log2e is written
  uint64_t* vec_empty = bars + 32;   // [kVecs] the compute warps have read them (one arrival per warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 36);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 37);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // a warp-uniform value, also to the compiler
  const int n_t = p.N / 128, rep = p.H / p.Hk;
  const int total = p.B * p.H * (p.causal ? n_t * (n_t + 1) / 2 : n_t * n_t);
  const int begin = static_cast<int>(static_cast<long long>(total) * blockIdx.x / gridDim.x);
  const int n_it = static_cast<int>(static_cast<long long>(total) * (blockIdx.x + 1) / gridDim.x) - begin;

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_empty + s, 1);
      mbar_init(full_q + s, 1);
      mbar_init(full_d + s, 1);
      mbar_init(empty_q + s, 1);
      mbar_init(empty_d + s, 1);
      mbar_init(bar_s + s, 1);
      mbar_init(bar_dp + s, 1);
      mbar_init(s_free + s, C::kComputeWarps);
      mbar_init(dp_free + s, C::kComputeWarps);
      mbar_init(staged + s, C::kComputeWarps);
      mbar_init(stage_free + s, 1);
    }
    for (int s = 0; s < C::kVecs; ++s) {
      mbar_init(vec_full + s, 1);
      mbar_init(vec_ok + s, 1);
      mbar_init(vec_empty + s, C::kComputeWarps);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == C::kComputeWarps) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem = 0;                         // 512 columns are all there are: the allocation starts at column 0
  grid_dep_wait();

  TileWalk w;
  w.seek(p, n_t, rep, begin);
  bool ok = true;
  if (warp == C::kComputeWarps + 1) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_do);
      bool fresh = true;                                 // the tile has another K / V than the one before
      for (int i = 0, kv = 0; ok && i < n_it; ++i) {
        const int row = w.row;
        const int vs = i % C::kVecs, st = i % C::kStages;
        if (fresh) {
          const int buf = kv % C::kKvBufs;
          if (kv >= C::kKvBufs && !(ok = wait_or_abort(kv_empty + buf, ((kv / C::kKvBufs) - 1) & 1, abort_flag))) break;
          mbar_expect_tx(kv_full + buf, 2 * C::kTileBytes);
          uint8_t* dst = smem + C::kSmemK + buf * 2 * C::kTileBytes;
          for (int s = 0; s < C::kSub; ++s) {
            tma_load_2d(dst + s * 16384, &tm_k, kv_full + buf, s * 128, w.bhk * p.N + w.kt * 128);
            tma_load_2d(dst + C::kTileBytes + s * 16384, &tm_v, kv_full + buf, s * 128, w.bhk * p.N + w.kt * 128);
          }
          ++kv;
        }
        const uint32_t eph = ((i / C::kStages) - 1) & 1;
        if (i >= C::kStages && !(ok = wait_or_abort(empty_q + st, eph, abort_flag))) break;
        mbar_expect_tx(full_q + st, C::kTileBytes);
        for (int s = 0; s < C::kSub; ++s)
          tma_load_2d(smem + C::kSmemQ + st * C::kTileBytes + s * 16384, &tm_q, full_q + st, s * 128, row);
        if (i >= C::kVecs && !(ok = wait_or_abort(vec_empty + vs, ((i / C::kVecs) - 1) & 1, abort_flag))) break;
        uint8_t* v = smem + C::kSmemVec + vs * C::kVecBytes;
        mbar_expect_tx(vec_full + vs, 1056);
        bulk_load_1d(v + C::kVecLse, p.lse + row, 512, vec_full + vs);
        bulk_load_1d(v + C::kVecDelta, p.delta + row, 512, vec_full + vs);
        bulk_load_1d(v + C::kVecQs, p.qs + row / 32, 16, vec_full + vs);
        bulk_load_1d(v + C::kVecDos, p.dos + row / 32, 16, vec_full + vs);
        if (i >= C::kStages && !(ok = wait_or_abort(empty_d + st, eph, abort_flag))) break;
        mbar_expect_tx(full_d + st, C::kTileBytes);
        for (int s = 0; s < C::kSub; ++s)
          tma_load_2d(smem + C::kSmemDo + st * C::kTileBytes + s * 16384, &tm_do, full_d + st, s * 128, row);
        fresh = w.next(p, n_t, rep);
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInTiles);
    }
  } else if (warp == C::kComputeWarps + 2) {
    // ------------------------------------------------------------------------------------------ vector warp
    // -lse * log2e once per query, in place, fenced for the bulk copy that will replace it (as in dm_bwd_kv.cu)
    const int lane = tid & 31;
    for (int i = 0; i < n_it; ++i) {
      const int vs = i % C::kVecs;
      if (!(ok = wait_warp(vec_full + vs, (i / C::kVecs) & 1, abort_flag))) break;
      const uint32_t v = smem_u32(smem + C::kSmemVec) + vs * C::kVecBytes + C::kVecLse + 16 * lane;
      const float4 l = lds_f4(v);
      const float2 x = mul2(make_float2(l.x, l.y), splat2(-kLog2e)), y = mul2(make_float2(l.z, l.w), splat2(-kLog2e));
      sts_u4(v, __float_as_uint(x.x), __float_as_uint(x.y), __float_as_uint(y.x), __float_as_uint(y.y));
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(vec_ok + vs);
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInTiles);
  } else if (warp == C::kComputeWarps + 3) {
    // ------------------------------------------------------------------------------------------ store warp
    if (elect_one()) {
      for (int i = 0; i < n_it; ++i) {
        const int buf = i & 1, row = w.tile * 128;
        if (!(ok = wait_or_abort(staged + buf, (i >> 1) & 1, abort_flag))) break;
        tma_store_2d(&tm_p, smem + C::kSmemOut + buf * 2 * C::kCodeBytes, 0, row);
        tma_store_2d(&tm_ds, smem + C::kSmemOut + buf * 2 * C::kCodeBytes + C::kCodeBytes, 0, row);
        bulk_commit_group();
        bulk_wait_group_read<0>();
        mbar_arrive(stage_free + buf);
        w.next(p, n_t, rep);
      }
      bulk_wait_group<0>();
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInTiles);
    }
  } else if (warp == C::kComputeWarps) {
    // ------------------------------------------------------------------------------------------ MMA issuer
    constexpr uint32_t kIdesc = idesc_f8(128, 128, false, false);
    const uint32_t lo0 = desc_lo(smem_u32(smem));
    auto chain_kmajor = [&](uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo) {
#pragma unroll
      for (int ks = 0; ks < D / 32; ++ks) {
        const uint32_t off = (ks / 4) * 1024 + (ks % 4) * 2;        // descriptor units of 16 bytes
        mma_f8_ss(d_tmem, a_lo + off, b_lo + off, kIdesc, ks > 0);
      }
    };
    int kv = -1;
    bool fresh = true;
    for (int i = 0; i < n_it; ++i) {
      const int buf = i & 1, st = i % C::kStages;
      const uint32_t sph = (i / C::kStages) & 1, fph = ((i >> 1) - 1) & 1;
      if (fresh) {
        ++kv;
        if (!(ok = wait_warp(kv_full + kv % C::kKvBufs, (kv / C::kKvBufs) & 1, abort_flag))) break;
      }
      fresh = w.next(p, n_t, rep);
      const uint32_t k_lo = lo0 + (C::kSmemK >> 4) + static_cast<uint32_t>(kv % C::kKvBufs) * (2 * C::kTileBytes >> 4);
      const uint32_t q_lo = lo0 + (C::kSmemQ >> 4) + static_cast<uint32_t>(st) * (C::kTileBytes >> 4);
      const uint32_t d_lo = lo0 + (C::kSmemDo >> 4) + static_cast<uint32_t>(st) * (C::kTileBytes >> 4);
      if (!(ok = wait_warp(full_q + st, sph, abort_flag))) break;
      if (i >= 2 && !(ok = wait_warp(s_free + buf, fph, abort_flag))) break;
      tc_fence_after();
      if (elect_one()) {
        chain_kmajor(tmem + 256 * buf, k_lo, q_lo);                            // S^T = K Q^T
        tc_commit(bar_s + buf);
        tc_commit(empty_q + st);
      }
      if (!(ok = wait_warp(full_d + st, sph, abort_flag))) break;
      if (i >= 2 && !(ok = wait_warp(dp_free + buf, fph, abort_flag))) break;
      tc_fence_after();
      if (elect_one()) {
        chain_kmajor(tmem + 256 * buf + 128, k_lo + (C::kTileBytes >> 4), d_lo);   // dP^T = V dO^T
        tc_commit(bar_dp + buf);
        tc_commit(empty_d + st);
        if (fresh) tc_commit(kv_empty + kv % C::kKvBufs);
      }
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInTiles);
  } else {
    // ------------------------------------------------------------------------------------------ compute warps
    // As in dkdv_tile (dm_bwd_kv.cu), but the codes go to shared memory instead of TMEM.
    const int part = warp >> 2;                        // query block of every tile: columns [32 part, 32 part + 32)
    const int quad = warp & 3;                         // lane quadrant = 32-key block of the dS scale
    const int r = tid & 127;                           // key row inside the tile = TMEM lane
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(quad * 32) << 16) + 32 * part;
    const int nblk = p.N / 32;
    const uint32_t vec_a = smem_u32(smem + C::kSmemVec), xch_a = smem_u32(smem + C::kSmemXch);
    const uint32_t out_a = smem_u32(smem + C::kSmemOut) + r * 128;
    // the key scales of the next tile are in flight during this one
    float ks_n, vs_n;
    auto fetch = [&]() {
      const int at = w.bhk * nblk + w.kt * 4 + quad;
      ks_n = p.ks[at];
      vs_n = p.vs[at];
    };
    fetch();
    for (int i = 0; i < n_it; ++i) {
      const uint32_t buf = i & 1, ph = (i >> 1) & 1;
      const int vs = i % C::kVecs;
      const bool diag = p.causal && (w.qt == w.kt);
      const float ks_row = ks_n, vs_row = vs_n;
      const size_t tile = w.tile;
      w.next(p, n_t, rep);
      if (i + 1 < n_it) fetch();
      const uint32_t va = vec_a + vs * C::kVecBytes + 128 * part, sc = vec_a + vs * C::kVecBytes + 4 * part;
      const uint32_t t_s = t_lane + 256 * buf, o_row = out_a + buf * 2 * C::kCodeBytes;
      float2 pr[16];                                   // P, then -dS
      float dos_c, am;
      uint32_t xv = 0;
      if (ok) ok = wait_warp(vec_ok + vs, (i / C::kVecs) & 1, abort_flag);
      if (ok) ok = wait_warp(bar_s + buf, ph, abort_flag);
      if (ok) {
        tc_fence_after();
        const float qs_c = lds_f(sc + C::kVecQs);
        dos_c = lds_f(sc + C::kVecDos);
        uint32_t rs[32];
        tmem_ld32(t_s, rs);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(s_free + buf);
        if (i >= 2) ok = wait_warp(stage_free + buf, ph ^ 1, abort_flag);     // the tile's staging is free
        if (diag) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (r > 32 * part + e) rs[e] = 0xff800000u;                        // -inf: key index above the query index
        }
        const float pm = p_block(rs, splat2((ks_row * qs_c) * kLog2e), va + C::kVecLse, pr);
        // P^T codes: one power-of-two scale per (key row, 32 queries) = per thread
        const uint32_t psb = pow2_sb(pm, 0u);
        uint32_t wd[8];
        codes32(pr, sb_to_inv(psb), wd);
        stage_codes(o_row, r, part, wd);
        xv = sb_mul(psb, scale_to_sb(dos_c));
        if (ok) ok = wait_warp(bar_dp + buf, ph, abort_flag);
      }
      if (ok) {
        tc_fence_after();
        uint32_t rd[32];
        tmem_ld32(t_s + 128, rd);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(dp_free + buf);
        am = warp_max(neg_ds_block(rd, splat2(-(vs_row * dos_c)), va + C::kVecDelta, pr));
        if (!DS32 && (tid & 31) == 0) sts_f(xch_a + 4 * (buf * 16 + warp), am);
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(vec_empty + vs);
      }
      // one dS scale per (128 queries x this quadrant's 32 keys): the warps of the quadrant meet here (reached for every tile,
      // also after a failed wait).  With 32 x 32 blocks the warp's own maximum is the block's.
      if (!DS32) bar_sync(1 + quad, 128);
      if (ok) {
        if (!DS32) {
          am = lds_f(xch_a + 4 * (buf * 16 + quad));
#pragma unroll
          for (int g = 1; g < 4; ++g) am = fmaxf(am, lds_f(xch_a + 4 * (buf * 16 + 4 * g + quad)));
        }
        const uint32_t dsb = pow2_sb(am, 127u);
        uint32_t wd[8];
        codes32(pr, -sb_to_inv(dsb), wd);
        stage_codes(o_row + C::kCodeBytes, r, part, wd);
        fence_async_smem();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(staged + buf);
        // the scale bytes last: global stores that are under way would hold up the proxy fence
        p.p_words[tile * 512 + r * 4 + part] = static_cast<uint8_t>(xv);                              // [key][query block]
        if ((tid & 31) == 0) p.ds_words[tile * 16 + part * 4 + quad] = static_cast<uint8_t>(dsb);     // [query block][key block]
      }
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInTiles);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == C::kComputeWarps) tmem_dealloc(tmem, 512);
}

template <int D, bool DS32>
static cudaError_t launch_tiles_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                  const CUtensorMap& tds, const CUtensorMap& tp, const BwdParams& p, cudaStream_t stream) {
  using C = TilesCfg<D>;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(bwd_tiles_kernel<D, DS32>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return e;
    done[dev] = true;
  }
  const int n_t = p.N / 128;
  const int total = p.B * p.H * (p.causal ? n_t * (n_t + 1) / 2 : n_t * n_t);
  const int sms = sm_count();
  count_launch();
  return launch_chained(bwd_tiles_kernel<D, DS32>, total < sms ? total : sms, C::kThreads, C::kSmemBytes, stream, tq, tk, tv, tdo,
                        tds, tp, p);
}

cudaError_t launch_bwd_tiles(int D, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                             const CUtensorMap& tds, const CUtensorMap& tp, const BwdParams& p, cudaStream_t stream) {
  if (D == 128) return (p.ds32 ? launch_tiles_t<128, true> : launch_tiles_t<128, false>)(tq, tk, tv, tdo, tds, tp, p, stream);
  return (p.ds32 ? launch_tiles_t<256, true> : launch_tiles_t<256, false>)(tq, tk, tv, tdo, tds, tp, p, stream);
}

}  // namespace dm
