// Backward pass 1 of delta-matching fp8 attention on sm_100a with dK and dV made by different CTAs, or dV elsewhere: head_dim 256, and
// small grids at head_dim 128 (the others: dm_bwd_pipe.cu).  Key-stationary, bit-deterministic (one writer per output element, fixed loop
// order, no atomics).
//
//   CTA = (128-key tile, kv head, batch); it walks the query heads of the GQA group and their 128-query tiles:
//   dP^T = V8 dO8^T and S^T = K8 Q8^T (kind::f8f6f4), P^T codes and dS^T codes written to TMEM, dV += P^T dO and
//   dK += dS^T Q as block-scaled chains (kind::mxf8f6f4).  The group is reduced in TMEM, dK / dV are rounded to bf16 once per
//   kv head.  With a workspace the dS^T code tiles also go there for the streaming dQ kernel (dm_bwd_p2.cu).
//
// Numerics (delta_matching/reference.py:476-518 with preset "sm100-mx", :612-613; kernel-side rules
// delta_matching/sm100/dm_bwd_sm100.py:5413-5433, 6175-6224 and attention_math_sm100.py:26-45):
//   P = ex2(fma(S_acc, (ks*qs)*log2e, -lse*log2e));  dP = dP_acc * (vs*dos);  dS = P * (dP - delta)   (fp32)
//   P^T codes: power-of-two scale per (key, 32 queries), amax 0 -> byte 0;   SFA_dV = p_sb (+) dos_sb
//   dS codes:  power-of-two scale per (128 queries x 32 keys), amax 0 -> scale 1;  SFA_dK = ds_sb (+) qs_sb.
#include <cuda_bf16.h>
#include "dm_bwd_math.cuh"
#include "dm_common.cuh"
#include "dm_kernels.h"

namespace dm {

// Eight compute warps (two per SM quarter, up to 168 registers a thread) and four that issue.  A tile of 128 keys x 128 queries
// is a chain: S^T MMA -> exponentials and P^T codes -> dP^T -> dS, block maximum, dS^T codes -> dV or dK MMAs.  S^T and dP^T
// have TMEM columns of their own; a thread holds 64 values each of P and dP (one key row, 64 queries), so that both TMEM regions are in
// registers early.
//
// Head_dim 256: one accumulator fills 256 columns.  Either a key tile is two CTAs (and so it is in small grids at head_dim 128): a
// DV role (S^T, P^T codes, dV; the columns of dP^T are a second S^T buffer, and the words lie beside the codes) and a DK role
// (S^T, dP^T, dS codes, dK and the dS tiles for the workspace; the scale words and the dS^T codes over dP^T), each with the other half of
// the work compiled out.  Or, PO, the DK role also leaves the P^T tiles in the workspace, and dV is streamed from them beside dQ
// (dm_bwd_p2.cu), which saves the DV role's S^T and exponentials.
// DK: the DK role, else the DV role.
template <int D, bool DK, bool PO = false>
struct KvCfg {
  static_assert((D == 128 || D == 256) && (DK || !PO), "P^T tiles go out of the DK role");
  static constexpr int kSub = D / 128;                 // 128-byte-wide sub-tiles of an operand row
  static constexpr int kTileBytes = 128 * D;           // K, V, Q, dO tile
  static constexpr int kCodeBytes = 128 * 128;         // dS^T code tile (does not depend on head_dim)
  static constexpr int kStages = (D == 128) ? 4 : 2;
  static constexpr int kComputeWarps = 8;
  static constexpr int kThreads = (kComputeWarps + 4) * 32;
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0, kColDp = 128;        // fp32 accumulators, 128 columns each
  // What a warp writes over the 64 columns [64 h, 64 h + 64) that it has read, relative to the region (DV role: S^T, DK role: dP^T):
  static constexpr int kColCodes = 0;        // 64 h + 8 c: codes of query block 2 h + c
  static constexpr int kColWord = 16;        // 64 h + 16: 4 columns of the scale word of half h (byte c = block 2 h + c)
  static constexpr int kColOne = 24;         // 4 columns of 0x7F7F7F7F (written by h = 0)
  static constexpr int kColAcc = 256;        // dV or dK
  static constexpr int kSmemK = 0;
  static constexpr int kSmemV = kTileBytes;                          // the DV role has no V tile
  static constexpr int kSmemQ = DK ? 2 * kTileBytes : kTileBytes;    // [kStages]
  static constexpr int kSmemDo = kSmemQ + kStages * kTileBytes;      // [kStages]
  static constexpr int kSmemWs = kSmemDo + kStages * kTileBytes;     // two staging tiles of dS^T codes (PO: one, and one of P^T codes)
  static constexpr int kSmemVec = kSmemWs + (DK ? 2 * kCodeBytes : 0);   // [kStages] vectors of the query tile (bytes):
  static constexpr int kVecLse = 0, kVecDelta = 512, kVecQs = 1024, kVecDos = 1040, kVecBytes = 1056;
  static constexpr int kSmemXch = kSmemVec + kStages * kVecBytes;    // [2 parities][8 warps] floats
  static constexpr int kSmemBar = kSmemXch + 2 * 8 * 4;
  static constexpr int kSmemBytes = kSmemBar + 256;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
};

// Row of an fp32 TMEM accumulator (32-column chunk) -> bf16, 64 bytes to global.
__device__ __forceinline__ void store_bf16_row32(const uint32_t (&r)[32], __nv_bfloat16* dst) {
  uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[8 * e + 2 * j]), __uint_as_float(r[8 * e + 2 * j + 1]));
      w[j] = *reinterpret_cast<uint32_t*>(&v);
    }
    d4[e] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// DS32: the dS scale is taken per (32 queries x 32 keys), which is one 32-column block of one warp, instead of the contract's
// (128 queries x 32 keys), for which the two warps of a key quadrant exchange their maxima.
template <int D, bool DK, bool DS32, bool PO = false>
__device__ __forceinline__ void dkdv_tile(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v,
                                          const CUtensorMap& tm_do, const CUtensorMap& tm_ds, const CUtensorMap& tm_p, const BwdParams& p) {
  using C = KvCfg<D, DK, PO>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  uint64_t* bar_kv = bars + 0;       // K and V landed
  uint64_t* bar_s = bars + 1;        // [2] S^T landed (MMA commit); the second one: the second buffer of the DV role
  uint64_t* bar_dp = bars + 3;       // dP^T landed
  uint64_t* bar_p = bars + 4;        // P^T codes and words written (DK role: S^T in registers); one arrival per compute warp
  uint64_t* bar_p1 = bars + 26;      // DV role: the same for odd tiles.  S^T of tile i + 1 is issued before the MMA warp has seen the
                                     // codes of tile i, so the compute warps can be two hand-offs ahead of it: with one barrier its
                                     // parity test could miss a phase and wait for good
  uint64_t* bar_k = bars + 5;        // dS^T codes and words written
  uint64_t* bar_done = bars + 6;     // the tile's chains done (MMA commit): columns and staging tile are free
  uint64_t* bar_acc = bars + 7;      // every chain of the CTA done (MMA commit behind the last one)
  uint64_t* full_q = bars + 8;       // [kStages] Q and the vectors landed
  uint64_t* full_d = bars + 12;      // [kStages] dO landed
  uint64_t* vec_ok = bars + 16;      // [kStages] the vectors landed and -lse * log2e is written
  uint64_t* empty = bars + 20;       // [kStages] the chains of the stage's tile are done (MMA commit)
  uint64_t* bar_po = bars + 27;      // PO: P^T codes of the tile in their staging tile (one arrival per compute warp)
  uint64_t* po_free = bars + 28;     // PO: they have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 25);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // a warp-uniform value, also to the compiler
  const int n_t = p.N / 128;
  // Heaviest first: under a causal mask key tile 0 has the most query tiles, so the tiles of one rank of all heads are
  // neighbours in the grid, and the last CTAs to start are the lightest.
  const int kt = blockIdx.y;
  const int bhk = blockIdx.x;
  const int b = bhk / p.Hk, hk = bhk % p.Hk;
  const int rep = p.H / p.Hk;
  const int qt0 = p.causal ? kt : 0;
  const int n_qi = n_t - qt0;
  const int n_it = rep * n_qi;                        // tile i = (query head of the group, query tile)

  if (tid == 0) {
    mbar_init(bar_kv, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_s + 1, 1);
    mbar_init(bar_dp, 1);
    mbar_init(bar_p, C::kComputeWarps);
    mbar_init(bar_p1, C::kComputeWarps);
    mbar_init(bar_k, C::kComputeWarps);
    mbar_init(bar_done, 1);
    mbar_init(bar_acc, 1);
    mbar_init(bar_po, C::kComputeWarps);
    mbar_init(po_free, 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full_q + s, 1);
      mbar_init(full_d + s, 1);
      mbar_init(vec_ok + s, 1);
      mbar_init(empty + s, 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == C::kComputeWarps) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem = 0;                         // 512 columns are all there are: the allocation starts at column 0
  grid_dep_wait();

  if (warp == C::kComputeWarps + 1) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_do);
      mbar_expect_tx(bar_kv, (DK ? 2 : 1) * C::kTileBytes);
      for (int s = 0; s < C::kSub; ++s) {
        tma_load_2d(smem + C::kSmemK + s * 16384, &tm_k, bar_kv, s * 128, bhk * p.N + kt * 128);
        if (DK) tma_load_2d(smem + C::kSmemV + s * 16384, &tm_v, bar_kv, s * 128, bhk * p.N + kt * 128);
      }
      int row = (b * p.H + hk * rep) * p.N + qt0 * 128, left = n_qi;
      for (int i = 0; i < n_it; ++i) {
        const int st = i % C::kStages;
        if (i >= C::kStages && !wait_or_abort(empty + st, ((i / C::kStages) - 1) & 1, abort_flag)) {
          raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInDkDv);
          break;
        }
        uint8_t* v = smem + C::kSmemVec + st * C::kVecBytes;
        mbar_expect_tx(full_q + st, C::kTileBytes + (DK ? 1056 : 544));
        for (int s = 0; s < C::kSub; ++s)
          tma_load_2d(smem + C::kSmemQ + st * C::kTileBytes + s * 16384, &tm_q, full_q + st, s * 128, row);
        bulk_load_1d(v + C::kVecLse, p.lse + row, 512, full_q + st);
        if (DK) bulk_load_1d(v + C::kVecDelta, p.delta + row, 512, full_q + st);
        bulk_load_1d(v + C::kVecQs, p.qs + row / 32, 16, full_q + st);
        bulk_load_1d(v + C::kVecDos, p.dos + row / 32, 16, full_q + st);
        mbar_expect_tx(full_d + st, C::kTileBytes);
        for (int s = 0; s < C::kSub; ++s)
          tma_load_2d(smem + C::kSmemDo + st * C::kTileBytes + s * 16384, &tm_do, full_d + st, s * 128, row);
        row += 128;
        if (--left == 0) {                               // the next head of the group
          left = n_qi;
          row += qt0 * 128;
        }
      }
    }
  } else if (warp == C::kComputeWarps + 2) {
    // ------------------------------------------------------------------------------------------ vector warp
    // -lse * log2e once per query instead of once per (key, query): the same fp32 product.  Written in place, and fenced for
    // the bulk copy that will replace it.
    bool ok = true;
    const int lane = tid & 31;
    for (int i = 0; i < n_it; ++i) {
      const int st = i % C::kStages;
      if (!(ok = wait_warp(full_q + st, (i / C::kStages) & 1, abort_flag))) break;
      const uint32_t v = smem_u32(smem + C::kSmemVec) + st * C::kVecBytes + C::kVecLse + 16 * lane;
      const float4 l = lds_f4(v);
      const float2 x = mul2(make_float2(l.x, l.y), splat2(-kLog2e)), y = mul2(make_float2(l.z, l.w), splat2(-kLog2e));
      sts_u4(v, __float_as_uint(x.x), __float_as_uint(x.y), __float_as_uint(y.x), __float_as_uint(y.y));
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(vec_ok + st);
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDkDv);
  } else if (PO && warp == C::kComputeWarps + 3) {
    // ------------------------------------------------------------------------------------------ P^T store warp
    if (elect_one()) {
      bool ok = true;
      int row = (((b * p.H + hk * rep) * n_t + qt0) * n_t + kt) * 128, left = n_qi;
      for (int i = 0; i < n_it; ++i) {
        if (!(ok = wait_or_abort(bar_po, i & 1, abort_flag))) break;
        tma_store_2d(&tm_p, smem + C::kSmemWs + C::kCodeBytes, 0, row);
        bulk_commit_group();
        bulk_wait_group_read<0>();
        mbar_arrive(po_free);
        row += 128 * n_t;
        if (--left == 0) {
          left = n_qi;
          row += 128 * n_t * qt0;
        }
      }
      bulk_wait_group<0>();
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInDkDv);
    }
  } else if (warp == C::kComputeWarps) {
    // ------------------------------------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop (uniform values stay in uniform registers), one elected thread issues.
    constexpr uint32_t kIdesc = idesc_f8(128, 128, false, false);
    const uint32_t lo0 = desc_lo(smem_u32(smem));      // descriptor low word of the start of shared memory
    auto q_lo = [&](int i) { return lo0 + (C::kSmemQ >> 4) + static_cast<uint32_t>(i % C::kStages) * (C::kTileBytes >> 4); };
    auto do_lo = [&](int i) { return lo0 + (C::kSmemDo >> 4) + static_cast<uint32_t>(i % C::kStages) * (C::kTileBytes >> 4); };
    auto landed = [&](uint64_t* full, int i) { return wait_warp(full + i % C::kStages, (i / C::kStages) & 1, abort_flag); };
    // S^T or dP^T: both operands K-major, D / 32 steps of 32 bytes inside the 128-byte swizzle rows
    auto chain_kmajor = [&](uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo) {
#pragma unroll
      for (int ks = 0; ks < D / 32; ++ks) {
        const uint32_t off = (ks / 4) * 1024 + (ks % 4) * 2;        // descriptor units of 16 bytes
        mma_f8_ss(d_tmem, a_lo + off, b_lo + off, kIdesc, ks > 0);
      }
    };
    // dV or dK: A = codes in TMEM (8 columns per 32-query step), B = dO / Q tile MN-major (32 query rows per step), one
    // 128-column accumulator slice per sub-tile of head_dim; step ks = block ks & 1 of half ks / 2
    auto chain_acc = [&](uint32_t d_tmem, uint32_t codes, uint32_t words, uint32_t ones, uint32_t b_lo, bool first) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint32_t h = 64 * (ks / 2);
#pragma unroll
        for (int s = 0; s < C::kSub; ++s)
          mma_mxf8_ts(d_tmem + s * 128, codes + h + 8 * (ks % 2), b_lo + s * 1024 + ks * 256, idesc_mxf8(128, 128, false, true, ks % 2, 0),
                      words + h, ones, !first || (ks > 0));
      }
    };
    // S^T of tile i: into the one S^T region, or alternating (DV role)
    auto issue_s = [&](int i) -> bool {
      if (!landed(full_q, i)) return false;
      tc_fence_after();
      const uint32_t b_lo = q_lo(i), d = tmem + (DK ? C::kColS : 128 * (i & 1));
      uint64_t* bar = bar_s + (DK ? 0 : (i & 1));
      if (elect_one()) {
        chain_kmajor(d, lo0 + (C::kSmemK >> 4), b_lo);
        tc_commit(bar);
      }
      return true;
    };
    auto issue_dp = [&](int i) -> bool {
      if (!landed(full_d, i)) return false;
      tc_fence_after();
      const uint32_t b_lo = do_lo(i);
      if (elect_one()) {
        chain_kmajor(tmem + C::kColDp, lo0 + (C::kSmemV >> 4), b_lo);
        tc_commit(bar_dp);
      }
      return true;
    };
    bool ok = wait_warp(bar_kv, 0, abort_flag) && issue_s(0) && (!DK || issue_dp(0));
    int ws_row = (((b * p.H + hk * rep) * n_t + qt0) * n_t + kt) * 128, left = n_qi;      // workspace row of tile i's dS
    for (int i = 0; ok && i < n_it; ++i) {
      const uint32_t ph = i & 1;
      if (!DK && i + 1 < n_it) {                         // the other buffer: its codes were read by the chains of tile i - 1
        if (i > 0 && !(ok = wait_warp(bar_done, ph ^ 1, abort_flag))) break;
        if (!(ok = issue_s(i + 1))) break;
      }
      if (!(ok = DK ? wait_warp(bar_p, ph, abort_flag) : wait_warp((i & 1) ? bar_p1 : bar_p, (i >> 1) & 1, abort_flag))) break;
      if (!DK) {
        if (!(ok = landed(full_d, i))) break;
        tc_fence_after();
        const uint32_t b_lo = do_lo(i), region = tmem + 128 * (i & 1);
        if (elect_one()) {                               // dV += P^T dO
          chain_acc(tmem + C::kColAcc, region + C::kColCodes, region + C::kColWord, region + C::kColOne, b_lo, i == 0);
          tc_commit(bar_done);
          tc_commit(empty + i % C::kStages);
          if (i == n_it - 1) tc_commit(bar_acc);
        }
      }
      if (DK) {
        if (i + 1 < n_it && !(ok = issue_s(i + 1))) break;
        if (!(ok = wait_warp(bar_k, ph, abort_flag))) break;
        tc_fence_after();
        const uint32_t b_lo = q_lo(i);
        if (elect_one()) {                               // dK += dS^T Q
          chain_acc(tmem + C::kColAcc, tmem + C::kColDp + C::kColCodes, tmem + C::kColDp + C::kColWord, tmem + C::kColDp + C::kColOne, b_lo, i == 0);
          tc_commit(bar_done);
          tc_commit(empty + i % C::kStages);
          if (i == n_it - 1) tc_commit(bar_acc);
          if (p.ds_codes != nullptr) {                   // the dS^T codes of the tile, from its staging tile, to the workspace
            tma_store_2d(&tm_ds, smem + C::kSmemWs + (PO ? 0 : (i & 1) * C::kCodeBytes), 0, ws_row);
            bulk_commit_group();
          }
        }
        ws_row += 128 * n_t;
        if (--left == 0) {                               // the next head of the group
          left = n_qi;
          ws_row += 128 * n_t * qt0;
        }
        if (i + 1 < n_it) {
          // the scale words of these chains lie where dP^T of the next tile lands
          if (!(ok = wait_warp(bar_done, ph, abort_flag))) break;
          bulk_wait_group_read<PO ? 0 : 1>();            // tile i + 1 writes its codes where those of tile i - 1 (PO: i) were
          if (!(ok = issue_dp(i + 1))) break;
        }
      }
    }
    if (DK && p.ds_codes != nullptr) bulk_wait_group<0>();
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInDkDv);
  } else if (warp < C::kComputeWarps) {
    // ------------------------------------------------------------------------------------------ compute warps
    const int half = warp >> 2;                        // query columns [64 half, 64 half + 64) of every tile
    const int quad = warp & 3;                         // lane quadrant = 32-key block of the dS scale
    const int r = tid & 127;                           // key row inside the tile = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s0 = tmem + lane_base + 64 * half, t_dp = t_s0 + C::kColDp;
    const int key = kt * 128 + r;
    const int nblk = p.N / 32;
    const float ks_row = p.ks[static_cast<size_t>(bhk) * nblk + key / 32];
    const float vs_row = DK ? p.vs[static_cast<size_t>(bhk) * nblk + key / 32] : 0.f;
    const uint32_t vec_a = smem_u32(smem + C::kSmemVec) + 256 * half;       // this half's entries of the 128-query vectors
    const uint32_t xch_a = smem_u32(smem + C::kSmemXch);
    const uint32_t ws_a = smem_u32(smem + C::kSmemWs) + r * 128;
    bool ok = true;
    int left = n_qi;                                     // query tiles of the head that are still to come, this one included
    int ws_tile = ((b * p.H + hk * rep) * n_t + qt0) * n_t + kt;            // workspace tile
    for (int i = 0; i < n_it; ++i) {
      const uint32_t ph = i & 1;
      const int st = i % C::kStages;
      const bool diag = p.causal && (left == n_qi);      // the first query tile of a causal sweep is the diagonal one
      const uint32_t va = vec_a + st * C::kVecBytes, sc = va - 248 * half;  // sc: the scales of this half's two blocks
      const uint32_t t_s = t_s0 + (DK ? 0 : 128 * ph);
      float2 pr[2][16];                                   // P, then (DK) -dS
      float2 qs2, dos2;
      uint32_t xv = 0;
      if (ok) ok = wait_warp(vec_ok + st, (i / C::kStages) & 1, abort_flag);
      if (ok) ok = wait_warp(bar_s + (DK ? 0 : ph), DK ? ph : ((i >> 1) & 1), abort_flag);
      if (ok) {
        tc_fence_after();
        qs2 = lds_f2(sc + C::kVecQs);
        dos2 = lds_f2(sc + C::kVecDos);
        uint32_t rs[2][32];
        tmem_ld32(t_s, rs[0]);
        tmem_ld32(t_s + 32, rs[1]);
        tmem_wait_ld();
        if (DK) {                                        // S^T of the next tile may land
          tc_fence_before();
          __syncwarp();
          if ((tid & 31) == 0) mbar_arrive(bar_p);
        }
        if (diag) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (r > 64 * half + 32 * c + e) rs[c][e] = 0xff800000u;   // -inf: key index above the query index
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float2 cc = splat2((ks_row * (c ? qs2.y : qs2.x)) * kLog2e);
          if (PO && c == 0 && i > 0) ok = wait_warp(po_free, ph ^ 1, abort_flag);
          const float pm = p_block(rs[c], cc, va + C::kVecLse + 128 * c, pr[c]);
          if (!DK || PO) {
            // P^T codes: one power-of-two scale per (key row, 32 queries) = per thread and block
            const uint32_t psb = pow2_sb(pm, 0u);
            uint32_t w[8];
            codes32(pr[c], sb_to_inv(psb), w);
            if (!DK) tmem_st8(t_s + C::kColCodes + 8 * c, w);
            if (PO) stage_codes(ws_a + C::kCodeBytes, r, 2 * half + c, w);     // like the dS^T codes below
            xv |= sb_mul(psb, scale_to_sb(c ? dos2.y : dos2.x)) << (8 * c);
          }
        }
        if (!DK) {                                       // DV role: the words go beside the codes, and that is the tile
          tmem_st4(t_s + C::kColWord, xv, xv, xv, xv);
          if (half == 0) tmem_st4(t_s + C::kColOne, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if ((tid & 31) == 0) mbar_arrive(ph ? bar_p1 : bar_p);
        }
      }
      if (PO && ok) {
        fence_async_smem();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bar_po);
      }
      float am[2] = {0.f, 0.f};
      if (DK && ok) ok = wait_warp(bar_dp, ph, abort_flag);
      if (DK && ok) {
        tc_fence_after();
        uint32_t rd[2][32];
        tmem_ld32(t_dp, rd[0]);
        tmem_ld32(t_dp + 32, rd[1]);
        tmem_wait_ld();
        if (half == 0) tmem_st4(t_dp + C::kColOne, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float2 na = splat2(-(vs_row * (c ? dos2.y : dos2.x)));
          am[c] = neg_ds_block(rd[c], na, va + C::kVecDelta + 128 * c, pr[c]);
        }
        if (!DS32) {
          am[0] = warp_max(fmaxf(am[0], am[1]));
          if ((tid & 31) == 0) sts_f(xch_a + 4 * (ph * 8 + warp), am[0]);
        }
      }
      if (DK) {
        // one dS scale per (128 queries x this quadrant's 32 keys): the two warps of the quadrant meet here (reached for every
        // tile, also after a failed wait).  With 32 x 32 blocks the warp's own maxima are the blocks'.
        if (!DS32) bar_sync(1 + quad, 64);
        if (ok) {
          uint32_t dsb[2];
          if (DS32) {
#pragma unroll
            for (int c = 0; c < 2; ++c) dsb[c] = pow2_sb(warp_max(am[c]), 127u);
          } else {
            const float mx = fmaxf(lds_f(xch_a + 4 * (ph * 8 + quad)), lds_f(xch_a + 4 * (ph * 8 + 4 + quad)));
            dsb[0] = dsb[1] = pow2_sb(mx, 127u);
          }
          const uint32_t ws_row = ws_a + (PO ? 0 : ph * C::kCodeBytes);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t w[8];
            codes32(pr[c], -sb_to_inv(dsb[c]), w);
            tmem_st8(t_dp + C::kColCodes + 8 * c, w);
            // the same codes as a [key][query] tile, which the MMA warp stores to the workspace for pass 2
            if (p.ds_codes != nullptr) stage_codes(ws_row, r, 2 * half + c, w);
          }
          const uint32_t xk = sb_mul(dsb[0], scale_to_sb(qs2.x)) | (sb_mul(dsb[1], scale_to_sb(qs2.y)) << 8);
          tmem_st4(t_dp + C::kColWord, xk, xk, xk, xk);
          if (p.ds_codes != nullptr) {
            fence_async_smem();
            // scale bytes of the tile for pass 2, [query block][key block]
            if ((tid & 31) == 0) {
#pragma unroll
              for (int c = 0; c < 2; ++c) p.ds_words[static_cast<size_t>(ws_tile) * 16 + (2 * half + c) * 4 + quad] = static_cast<uint8_t>(dsb[c]);
            }
          }
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if ((tid & 31) == 0) mbar_arrive(bar_k);
          if (PO)                                          // dV scale bytes of the tile, [key][query block]
            *reinterpret_cast<uint16_t*>(p.p_words + static_cast<size_t>(ws_tile) * 512 + r * 4 + 2 * half) = static_cast<uint16_t>(xv);
        }
      }
      ws_tile += n_t;
      if (--left == 0) {                                 // the next head of the group
        left = n_qi;
        ws_tile += qt0 * n_t;
      }
    }
    // A barrier of its own: waiting for a phase of bar_done by its parity would, for a warp that comes late, mistake the end of
    // the phase after it for one that is still to come.
    if (ok) ok = wait_warp(bar_acc, 0, abort_flag);
    if (!ok) {
      raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDkDv);
    } else {
      tc_fence_after();
      // two warps per lane quadrant: each writes 64 columns of every 128-column slice of the accumulator
#pragma unroll 1
      for (int s = 0; s < 2 * C::kSub; ++s) {
        const int col = 128 * (s / 2) + 64 * half + 32 * (s % 2);
        uint32_t rr[32];
        tmem_ld32(tmem + lane_base + C::kColAcc + col, rr);
        tmem_wait_ld();
        __nv_bfloat16* out = DK ? p.dk + static_cast<int64_t>(b) * p.dk_sb + static_cast<int64_t>(key) * p.dk_sn + static_cast<int64_t>(hk) * p.dk_sh
                                : p.dv + static_cast<int64_t>(b) * p.dv_sb + static_cast<int64_t>(key) * p.dv_sn + static_cast<int64_t>(hk) * p.dv_sh;
        store_bf16_row32(rr, out + col);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == C::kComputeWarps) tmem_dealloc(tmem, C::kTmemCols);
}

// How dK and dV of a key tile are made: by two CTAs, both kinds in one grid, the longer one (dK) first; or dK here and dV from the P^T
// tiles that the launch leaves in the workspace.
enum KvForm { kKvRoles, kKvDkAndP };

template <int D, int Form>
struct KvLaunch {
  using Dk = KvCfg<D, true, Form == kKvDkAndP>;
  using Dv = KvCfg<D, false>;
  static constexpr int kThreads = Dk::kThreads;
  static constexpr int kSmemBytes = Dk::kSmemBytes > Dv::kSmemBytes ? Dk::kSmemBytes : Dv::kSmemBytes;
};

template <int D, int Form, bool DS32>
__global__ void __launch_bounds__(KvLaunch<D, Form>::kThreads, 1)
bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_ds, const __grid_constant__ CUtensorMap tm_p, const BwdParams p) {
  if constexpr (Form == kKvDkAndP) dkdv_tile<D, true, DS32, true>(tm_q, tm_k, tm_v, tm_do, tm_ds, tm_p, p);
  else if (blockIdx.z == 0) dkdv_tile<D, true, DS32>(tm_q, tm_k, tm_v, tm_do, tm_ds, tm_p, p);
  else dkdv_tile<D, false, DS32>(tm_q, tm_k, tm_v, tm_do, tm_ds, tm_p, p);
}

template <int D, int Form, bool DS32>
static cudaError_t launch_kv_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                               const CUtensorMap& tds, const CUtensorMap& tp, const BwdParams& p, cudaStream_t stream) {
  using L = KvLaunch<D, Form>;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(bwd_dkdv_kernel<D, Form, DS32>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmemBytes);
    if (e != cudaSuccess) return e;
    done[dev] = true;
  }
  const dim3 grid(p.B * p.Hk, p.N / 128, Form == kKvRoles ? 2 : 1);
  count_launch();
  return launch_chained(bwd_dkdv_kernel<D, Form, DS32>, grid, L::kThreads, L::kSmemBytes, stream, tq, tk, tv, tdo, tds, tp, p);
}

cudaError_t launch_bwd_dkdv(int D, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                            const CUtensorMap& tdo, const CUtensorMap* tds_or_null, const BwdParams& p,
                            cudaStream_t stream) {
  const CUtensorMap& tds = (tds_or_null != nullptr) ? *tds_or_null : tq;     // unused by the kernel without a workspace
  // At head_dim 128 the roles cost a second S^T and a second exponential per element, so they are for grids that leave half of
  // the SMs without a CTA (the same bits: the accumulators do not depend on each other).  There the dK role is a little shorter than the
  // pipeline, per tile (1.51 against 1.53 us; 32 x 32 dS blocks 1.31 against 1.40) and by some 2 us a launch, as dV is written out elsewhere.
  // Pipeline -> roles, us of this pass alone: 20.6 -> 18.5 (N=1024 H=2), 32.9 -> 30.8 (N=512 H=8 Hk=2), 12.4 -> 10.3 (B=36 N=256 H=1), 70.0 ->
  // 67.8 (N=1280 H=16 Hk=4), 400 -> 394 (N=4096 H=8 Hk=1), 463 -> 456 (N=9472 H=4 Hk=1); 32 x 32 blocks: 367 -> 342 and 425 -> 396 for the
  // last two.  (Causal calls; bidirectional ones gain the same, with 32 x 32 blocks less: 371 -> 362, 429 -> 423.)  With more key tiles some SM
  // has two roles in a row; whole step, bidirectional: 822 -> 928 (N=9728 H=4 Hk=1, 76 key tiles), 93 -> 108 (B=18 N=512 H=8 Hk=2, 144).
  if (D != 128) return (p.ds32 ? launch_kv_t<256, kKvRoles, true> : launch_kv_t<256, kKvRoles, false>)(tq, tk, tv, tdo, tds, tq, p, stream);
  if (2ll * p.B * p.Hk * (p.N / 128) <= sm_count())
    return (p.ds32 ? launch_kv_t<128, kKvRoles, true> : launch_kv_t<128, kKvRoles, false>)(tq, tk, tv, tdo, tds, tq, p, stream);
  return launch_bwd_pipe(tq, tk, tv, tdo, tds, p, stream);
}

cudaError_t launch_bwd_dk_and_p(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                const CUtensorMap& tds, const CUtensorMap& tp, const BwdParams& p, cudaStream_t stream) {
  return (p.ds32 ? launch_kv_t<256, kKvDkAndP, true> : launch_kv_t<256, kKvDkAndP, false>)(tq, tk, tv, tdo, tds, tp, p, stream);
}

}  // namespace dm
