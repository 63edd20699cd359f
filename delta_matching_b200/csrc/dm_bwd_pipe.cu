// Backward pass 1 of delta-matching fp8 attention on sm_100a at head_dim 128: dK and dV, key-stationary, bit-deterministic (one
// writer per output element, fixed order, no atomics), and the dS^T code tiles for the streaming dQ kernel (dm_bwd_p2.cu).  Numerics:
// see dm_bwd_kv.cu, whose arithmetic per (key row, 32 queries) this shares (dm_bwd_math.cuh).
//
// Work item = one 128-key tile of one (batch, kv head); it goes through the query heads of the GQA group and their 128-query tiles:
// S^T = K8 Q8^T, dP^T = V8 dO8^T, exponentials, P^T codes, dS, dS^T codes, dV += P^T dO, dK += dS^T Q.  dV (128 columns), dK (128), S^T
// (128) and dP^T (128) fill the TMEM, so neither accumulator of a tile can be doubled.  What bounds a tile is that its sixteen compute warps
// are in one phase of the loop  accumulator lands -> registers -> codes written -> chain that reads them -> accumulator of the next tile:
// in 39 % of the 2904 cycles a scheduler has no warp that can issue (all wait for the same hand-off, or each for its own latencies),
// in the others 2.3 of its five warps are ready at once (7109 warp instructions, issue slots 61 % used, 1.40 eligible warps a cycle).  No pipe is near
// its limit: tensor 35 %, MUFU 35 %, ALU 30 %, FMA 27 %.  Hence:
//   - codes lie over the accumulator that is free at the time: dS^T codes of tile g - 1 over S^T of tile g, once that is in registers,
//     P^T codes of tile g over its dP^T.  S^T of tile g + 1 waits for the dK chain of tile g - 1 only, dP^T of tile g + 1 for the dV chain
//     of tile g only, and neither is needed before half a tile of other work has gone by.  (In registers dS waits for its scale, the
//     maximum over four warps, through the same time.)
//   - the two loops have an issuing warp each.  One warp for both spent 1250 cycles a tile between hand-off and next accumulator:
//     791 -> 777 us (B=4 N=4096 H=32 Hk=8 causal).
//   - sixteen compute warps of 32 queries with 104 registers each (setmaxnreg: with 96 the loop spills, and behind a spill the fence of
//     the staging tile waits for local memory).  Eight warps of 64 queries were 840 us in the same form.
//   - persistent CTAs whose items follow each other without a break: Q / dO of the next item are loaded, its first S^T and dP^T computed
//     while the last tile of the one before is worked on, and that one is written out behind the first exponentials of the next.
//     With a CTA per item its start and end cost 8 us: 777 -> 742 us, and 474 -> 394 (B=8 N=2048 H=16 bidirectional, 16 tiles an item).
//   - one copy of each role's loop (48 KB of code in all): at 88 KB the warps waited for instructions a fifth of the time (920 us).
// Before (eight compute warps on one phase, one issuing warp, a CTA per item): 836, 490 and 230 us (B=1) -> 742, 394, 209; barriers by their
// shared addresses and a shorter scale byte: 762 -> 756 on another GPU of the same model.
#include <cuda_bf16.h>
#include "dm_bwd_math.cuh"
#include "dm_common.cuh"
#include "dm_kernels.h"

namespace dm {

struct PipeCfg {
  static constexpr int kTileBytes = 128 * 128;         // K, V, Q, dO and code tile
  static constexpr uint32_t kStages = 4;
  static constexpr int kComputeWarps = 16;             // warp = (32-query block, 32-key quadrant)
  static constexpr int kThreads = (kComputeWarps + 4) * 32;
  // Registers a thread: 640 x 96 at launch = 512 x 104 + 128 x 64.
  static constexpr int kRegsCompute = 104, kRegsIssue = 64;
  static_assert(512 * kRegsCompute + 128 * kRegsIssue <= kThreads * 96, "a split above the launch's own registers would wait for ever");
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0, kColDp = 128;        // fp32 accumulators, 128 columns each
  // What a warp writes over the 32 columns of its query block that it has read, relative to them: dS^T codes and the scale word of dK
  // over S^T, P^T codes and the scale word of dV over dP^T.
  static constexpr int kColCodes = 0;                  // 8 columns
  static constexpr int kColWord = 8;                   // 4 columns: byte 0 the scale, byte 1 one
  static constexpr int kColDv = 256, kColDk = 384;
  static constexpr int kSmemK = 0;
  static constexpr int kSmemV = kTileBytes;
  static constexpr int kSmemQ = 2 * kTileBytes;                      // [kStages]
  static constexpr int kSmemDo = kSmemQ + kStages * kTileBytes;      // [kStages]
  static constexpr int kSmemWs = kSmemDo + kStages * kTileBytes;     // two staging tiles of dS^T codes
  static constexpr int kSmemVec = kSmemWs + 2 * kTileBytes;          // [kStages] vectors of the query tile (bytes):
  static constexpr int kVecLse = 0, kVecDelta = 512, kVecQs = 1024, kVecDos = 1040, kVecRec = 1056, kVecBytes = 1120;
  static constexpr int kSmemXch = kSmemVec + kStages * kVecBytes;    // [2 parities][4 quadrants][4 query blocks] floats
  static constexpr int kSmemBar = kSmemXch + 2 * 16 * 4;
  static constexpr int kSmemBytes = kSmemBar + 512;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
};

template <bool DS32>
__global__ void __launch_bounds__(PipeCfg::kThreads, 1)
bwd_dkdv_pipe_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_ds, const BwdParams p) {
  using C = PipeCfg;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  // Pairs: [0] for S^T and dK, [1] for dP^T and dV.
  uint64_t* bar_s = bars + 0;        // S^T landed (MMA commit)
  uint64_t* bar_dp = bars + 1;       // dP^T landed
  uint64_t* bar_k = bars + 2;        // S^T of tile g in registers, dS^T codes and word of tile g - 1 written, its maxima read by the warp
                                     // that stores the tile; one arrival per warp
  uint64_t* bar_p = bars + 3;        // dP^T of tile g in registers, its P^T codes and word written
  uint64_t* bar_done = bars + 4;     // [2] the chain that reads them is done (MMA commit): the columns are free
  uint64_t* kv_full = bars + 6;      // [2] K, V of an item landed
  uint64_t* kv_free = bars + 8;      // [2] the item's last S^T, dP^T chain has read them (MMA commit)
  uint64_t* bar_acc = bars + 10;     // the last chains of dK and dV of an item are done (a commit of either issuer)
  uint64_t* full_q = bars + 11;      // [kStages] Q and the vectors landed
  uint64_t* full_d = bars + 15;      // [kStages] dO landed (kStages behind full_q)
  uint64_t* vec_ok = bars + 19;      // [kStages] the vectors landed and -lse * log2e is written
  uint64_t* empty = bars + 23;       // [kStages] the dK and the dV chain of the stage's tile are done (a commit of either issuer)
  uint64_t* bar_x = bars + 27;       // [parity][quadrant] the dS maxima of the quadrant's four query blocks are in their slots
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 35);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 36);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // a warp-uniform value, also to the compiler
  // Item k of this CTA: key tile kt of the (batch, kv head) bhk, n_q query tiles of each head of the group, n tiles in all (0: there is no
  // such item).  Items are numbered heaviest first: under a causal mask key tile 0 has the most query tiles.
  struct Item {
    int kt, bhk, n_q, n;
  };
  auto item_of = [&p](int k) -> Item {
    const int item = sched_item(k, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
    const int n_t = p.N >> 7, bhk_count = p.B * p.Hk, kt = item / bhk_count, n_q = p.causal ? n_t - kt : n_t;
    return {kt, item - kt * bhk_count, n_q, kt < n_t ? p.H / p.Hk * n_q : 0};
  };

  if (tid == 0) {
    for (int s = 0; s < 27; ++s)
      mbar_init(bars + s, bars + s == bar_k ? C::kComputeWarps + 1 : bars + s == bar_p ? C::kComputeWarps : (bars + s == bar_acc || bars + s >= empty) ? 2 : 1);
    for (int s = 0; s < 8; ++s) mbar_init(bar_x + s, 4);
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

  if (warp < C::kComputeWarps) {
    // ------------------------------------------------------------------------------------------ compute warps
    reg_inc<C::kRegsCompute>();
    const int qb = warp >> 2;                          // 32-query block of every tile
    const int quad = warp & 3;                         // lane quadrant = 32-key block of the dS scale
    const int r = tid & 127;                           // key row inside the tile = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem + lane_base + C::kColS + 32 * qb, t_dp = t_s + C::kColDp;
    const uint32_t vec_a = smem_u32(smem + C::kSmemVec);
    const uint32_t xch_a = smem_u32(smem + C::kSmemXch) + 16 * quad;
    const uint32_t ws_a = smem_u32(smem + C::kSmemWs) + r * 128;
    const uint32_t ws_c0 = ws_a + (((2 * qb) ^ (r & 7)) << 4);      // its neighbour is 16 bytes up or down
    // barriers by their shared addresses
    const uint32_t s_bar = smem_u32(bar_s), dp_bar = smem_u32(bar_dp), k_bar = smem_u32(bar_k), p_bar = smem_u32(bar_p);
    const uint32_t vec_bar = smem_u32(vec_ok), x_bar = smem_u32(bar_x) + 8 * quad;
    const bool leader = (tid & 31) == 0;
    bool ok = true;
    float ks_row = 0.f, vs_row = 0.f;                    // scales of the item's key row
    float2 pr[16];                                       // -dS of tile g - 1
#pragma unroll
    for (int e = 0; e < 16; ++e) pr[e] = make_float2(0.f, 0.f);
    float am = 0.f;                                      // maximum of the block's |dS| (DS32)
    uint32_t sbq = 0;                                    // byte of its Q scale
    // dV and dK of the CTA's item k: each warp writes 32 columns of its rows
    auto write_out = [&](int k, int kt, int bhk) -> bool {
      if (!wait_warp(bar_acc, k & 1, abort_flag)) return false;
      tc_fence_after();
      const int64_t b = bhk / p.Hk, hk = bhk - b * p.Hk, key = kt * 128 + 32 * quad;
#pragma unroll 1
      for (int x = 0; x < 2; ++x) {
        const int64_t sn = x ? p.dk_sn : p.dv_sn;
        store_rows32(tmem + lane_base + (x ? C::kColDk : C::kColDv) + 32 * qb, 1.0f,
                     (x ? p.dk + b * p.dk_sb + hk * p.dk_sh : p.dv + b * p.dv_sb + hk * p.dv_sh) + key * sn + 32 * qb, sn);
      }
      return true;
    };
    // Step g: the dS^T codes of tile g - 1 (zeros at g = 0, which nothing reads), then exponentials and dS of tile g.  Items follow each
    // other without a break: the first tile of an item takes its exponentials while the last dK chain of the item before runs, then
    // writes that one out.  One copy of this code for all cases: the loops of all roles share the SM's instruction cache.
    int k = 0, n = 0, left = 0;                          // items begun; tiles and query tiles of the head that are still to come
    int kt_done = 0, bhk_done = 0;                       // the item before, in an item's first tile
    Item it{0, 0, 0, 0};
    uint32_t g = 0;
#pragma unroll 1
    for (;; ++g) {
      const bool first = n == 0;
      if (first) {
        kt_done = it.kt;
        bhk_done = it.bhk;
        it = item_of(k++);
        n = it.n;
        left = 0;
        if (n > 0) {
          const size_t row = static_cast<size_t>(it.bhk) * (p.N >> 5) + it.kt * 4 + quad;
          ks_row = p.ks[row];
          vs_row = p.vs[row];
        }
      }
      const bool more = n > 0, diag = p.causal && left == 0;      // the first query tile of a causal sweep is the diagonal one
      if (left == 0) left = it.n_q;
      --left;
      --n;
      const uint32_t va = vec_a + (g % C::kStages) * C::kVecBytes;
      const uint32_t bx = x_bar + 32 * ((g - 1) & 1);
      // S^T, the vectors, and the maxima of the tile before, in one look
      {
        const bool need_x = !DS32 && g > 0;
        bool seen = mbar_test_wait(s_bar, g & 1);
        if (more) seen = mbar_test_wait(vec_bar + 8 * (g % C::kStages), (g / C::kStages) & 1) && seen;
        if (need_x) seen = mbar_test_wait(bx, ((g - 1) >> 1) & 1) && seen;
        if (!__all_sync(0xffffffffu, seen)) {
          seen = poll_or_abort(s_bar, g & 1, abort_flag);
          if (more) seen = seen && poll_or_abort(vec_bar + 8 * (g % C::kStages), (g / C::kStages) & 1, abort_flag);
          if (need_x) seen = seen && poll_or_abort(bx, ((g - 1) >> 1) & 1, abort_flag);
          if (!(ok = __all_sync(0xffffffffu, seen))) break;
        }
      }
      tc_fence_after();
      uint32_t rs[32];
      tmem_ld32(t_s, rs);                                // (behind the last tile: of no use)
      {
        // one dS scale per (128 queries x this quadrant's 32 keys), or per block
        float mx = am;
        if (!DS32) {
          const float4 m = lds_f4(xch_a + 64 * ((g - 1) & 1));
          mx = fmaxf(max3(m.x, m.y, m.z), m.w);
        }
        const uint32_t dsb = pow2_sb(mx, 127u);
        uint32_t w[8];
        codes32(pr, -sb_to_inv(dsb), w);
        const uint32_t off = ((g - 1) & 1) * C::kTileBytes, word = sb_mul(dsb, sbq) | 0x7F00u;
        sts_u4(ws_c0 + off, w[0], w[1], w[2], w[3]);
        sts_u4((ws_c0 ^ 16) + off, w[4], w[5], w[6], w[7]);
        tmem_wait_ld();
        tmem_st8(t_s + C::kColCodes, w);
        tmem_st4(t_s + C::kColWord, word, word, word, word);
        fence_async_smem();
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (leader) mbar_arrive(k_bar);
      }
      if (!more) break;
      const float4 rec = lds_f4(va + C::kVecRec + 16 * qb);
      sbq = __float_as_uint(rec.z);
      if (diag) {
#pragma unroll
        for (int e = 0; e < 32; ++e)
          if (r > 32 * qb + e) rs[e] = 0xff800000u;      // -inf: key index above the query index
      }
      const float pm = p_block(rs, splat2(ks_row * rec.x), va + C::kVecLse + 128 * qb, pr);
      if (first && g > 0 && !(ok = write_out(k - 2, kt_done, bhk_done))) break;
      // P^T codes: one scale per (key row, 32 queries)
      if (!(ok = wait_warp(dp_bar, g & 1, abort_flag))) break;
      tc_fence_after();
      uint32_t rd[32];
      tmem_ld32(t_dp, rd);
      const uint32_t psb = pow2_sb(pm, 0u);
      uint32_t w[8];
      codes32(pr, sb_to_inv(psb), w);
      const uint32_t word = sb_mul(psb, __float_as_uint(rec.w)) | 0x7F00u;
      tmem_wait_ld();
      tmem_st8(t_dp + C::kColCodes, w);
      tmem_st4(t_dp + C::kColWord, word, word, word, word);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (leader) mbar_arrive(p_bar);
      am = warp_max(neg_ds_block(rd, splat2(vs_row * rec.y), va + C::kVecDelta + 128 * qb, pr));
      if (leader) {
        sts_f(xch_a + 64 * (g & 1) + 4 * qb, am);
        mbar_arrive(x_bar + 32 * (g & 1));
      }
    }
    if (ok) ok = write_out(k - 2, kt_done, bhk_done);
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDkDv);
  } else {
    reg_dec<C::kRegsIssue>();
    if (warp == C::kComputeWarps + 2) {
      // ------------------------------------------------------------------------------------------ TMA producer
      if (elect_one()) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_do);
        bool ok = true;
        uint32_t g = 0;
#pragma unroll 1
        for (int k = 0; ok; ++k) {
          const Item it = item_of(k);
          if (it.n == 0) break;
          const int skip = p.causal ? it.kt * 128 : 0;
          int row = it.bhk * (p.H / p.Hk) * p.N + skip, left = it.n_q;
#pragma unroll 1
          for (int i = 0; i < it.n; ++i, ++g) {
            const uint32_t st = g % C::kStages;
            if (g >= C::kStages && !(ok = wait_or_abort(empty + st, ((g / C::kStages) - 1) & 1, abort_flag))) break;
            uint8_t* v = smem + C::kSmemVec + st * C::kVecBytes;
            mbar_expect_tx(full_q + st, C::kTileBytes + 1056);
            tma_load_2d(smem + C::kSmemQ + st * C::kTileBytes, &tm_q, full_q + st, 0, row);
            bulk_load_1d(v + C::kVecLse, p.lse + row, 512, full_q + st);
            bulk_load_1d(v + C::kVecDelta, p.delta + row, 512, full_q + st);
            bulk_load_1d(v + C::kVecQs, p.qs + row / 32, 16, full_q + st);
            bulk_load_1d(v + C::kVecDos, p.dos + row / 32, 16, full_q + st);
            mbar_expect_tx(full_d + st, C::kTileBytes);
            tma_load_2d(smem + C::kSmemDo + st * C::kTileBytes, &tm_do, full_d + st, 0, row);
            if (i == 0) {                                // K and V of the item, over those of the one before
#pragma unroll 1
              for (int h = 0; ok && h < 2; ++h) {
                if (k > 0 && !(ok = wait_or_abort(kv_free + h, (k - 1) & 1, abort_flag))) break;
                mbar_expect_tx(kv_full + h, C::kTileBytes);
                tma_load_2d(smem + C::kSmemK + h * C::kTileBytes, h ? &tm_v : &tm_k, kv_full + h, 0, it.bhk * p.N + it.kt * 128);
              }
              if (!ok) break;
            }
            row += 128;
            if (--left == 0) {                           // the next head of the group
              left = it.n_q;
              row += skip;
            }
          }
        }
        if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInDkDv);
      }
    } else if (warp == C::kComputeWarps + 3) {
      // ------------------------------------------------------------------------------------------ vectors and dS tiles
      // Of tile g: -lse * log2e once per query instead of once per (key, query), the same fp32 product, written in place; the scalars
      // of the query blocks.  Fenced for the bulk copies that will replace them.  Of tile g - 2: the dS^T codes and their scale bytes
      // ([query block][key block], a lane each) to the workspace.
      bool ok = true;
      const int lane = tid & 31, kb = lane & 3, qb = (lane >> 2) & 3;
      if (lane == 0) mbar_arrive(bar_k);
      int k = 0, n = 0, left = 0;
      uint32_t tile = 0, tile1 = 0, tile2 = 0;           // workspace index of tiles g, g - 1, g - 2
      Item it{0, 0, 0, 0};
      uint32_t total = 0xffffffffu;                      // tiles of the CTA, once known
#pragma unroll 1
      for (uint32_t g = 0; g < 2 || g - 2 < total; ++g) {
        tile2 = tile1;
        tile1 = tile;
        if (n == 0 && g < total) {
          it = item_of(k++);
          n = it.n;
          left = it.n_q;
          tile = (it.bhk * (p.H / p.Hk) * (p.N >> 7) + (p.causal ? it.kt : 0)) * (p.N >> 7) + it.kt;
          if (n == 0) total = g;
        } else {
          tile += p.N >> 7;
          if (--left == 0) {                             // the next head of the group
            left = it.n_q;
            if (p.causal) tile += it.kt * (p.N >> 7);
          }
        }
        if (g < total) {
          --n;
          const uint32_t st = g % C::kStages;
          if (!(ok = wait_warp(full_q + st, (g / C::kStages) & 1, abort_flag))) break;
          const uint32_t va = smem_u32(smem + C::kSmemVec) + st * C::kVecBytes, v = va + C::kVecLse + 16 * lane;
          const float4 l = lds_f4(v);
          const float2 x = mul2(make_float2(l.x, l.y), splat2(-kLog2e)), y = mul2(make_float2(l.z, l.w), splat2(-kLog2e));
          sts_u4(v, __float_as_uint(x.x), __float_as_uint(x.y), __float_as_uint(y.x), __float_as_uint(y.y));
          if (lane < 4) {                                // powers of two: the products are exact
            const float qs = lds_f(va + C::kVecQs + 4 * lane), dos = lds_f(va + C::kVecDos + 4 * lane);
            sts_u4(va + C::kVecRec + 16 * lane, __float_as_uint(qs * kLog2e), __float_as_uint(-dos), scale_to_sb(qs), scale_to_sb(dos));
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(vec_ok + st);
        }
        if (g >= 2) {
          const uint32_t t = g - 2;
          if (!(ok = wait_warp(bar_x + 4 * (t & 1) + kb, (t >> 1) & 1, abort_flag))) break;
          const float4 m = lds_f4(smem_u32(smem + C::kSmemXch) + 64 * (t & 1) + 16 * kb);
          const float mx = DS32 ? (qb == 0 ? m.x : qb == 1 ? m.y : qb == 2 ? m.z : m.w) : fmaxf(fmaxf(m.x, m.y), fmaxf(m.z, m.w));
          bulk_wait_group_read<0>();                     // behind this hand-off, tile t + 1 writes its dS^T codes where those of tile t - 1 were
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_k);
          if (p.ds_codes != nullptr && lane < 16) p.ds_words[static_cast<size_t>(tile2) * 16 + lane] = static_cast<uint8_t>(pow2_sb(mx, 127u));
          if (p.ds_codes != nullptr) {                   // the tile's dS^T codes, complete with the hand-off of tile t + 1, to the workspace
            if (!(ok = wait_warp(bar_k, (t + 1) & 1, abort_flag))) break;
            if (elect_one()) {
              tma_store_2d(&tm_ds, smem + C::kSmemWs + (t & 1) * C::kTileBytes, 0, static_cast<int>(tile2) * 128);
              bulk_commit_group();
            }
          }
        }
      }
      if (p.ds_codes != nullptr) bulk_wait_group<0>();
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDkDv);
    } else {
      // ------------------------------------------------------------------------------------------ MMA issuers
      // Two warps, one for S^T and dK, one for dP^T and dV: either loop is hand-off -> chain -> completion -> next accumulator, and
      // most of its time is latency of the issuing warp, so the two do not wait for each other.  They run the same code.  The whole warp
      // walks the loop (uniform values stay in uniform registers), one elected thread issues.
      constexpr uint32_t kIdesc = idesc_f8(128, 128, false, false), kIdescMx = idesc_mxf8(128, 128, false, true, 0, 1);
      const int role = warp - C::kComputeWarps;          // 0: S^T, dK; 1: dP^T, dV
      const uint32_t lag = 1 - role;                     // hand-off g is followed by the chain of tile g - lag
      const uint32_t lo0 = desc_lo(smem_u32(smem));      // descriptor low word of the start of shared memory
      const uint32_t a_lo = lo0 + ((C::kSmemK + role * C::kTileBytes) >> 4), b_lo = lo0 + ((role ? C::kSmemDo : C::kSmemQ) >> 4);
      const uint32_t region = tmem + C::kColS + 128 * role, acc = tmem + (role ? C::kColDv : C::kColDk);
      uint64_t* full = full_q + role * C::kStages;
      bool ok = true;
      int k = 0, n = item_of(0).n, i = 0;                // tile g + 1 is tile i of n of item k (n = 0: there is none)
      int ka = 0, na = n, ia = 0;                        // the next tile of the chains likewise
#pragma unroll 1
      for (uint32_t g = 0xffffffffu;; ++g) {             // from -1 on
        const bool more = n > 0;
        if (more && !(ok = wait_warp(full + (g + 1) % C::kStages, ((g + 1) / C::kStages) & 1, abort_flag))) break;
        if (more && i == 0 && !(ok = wait_warp(kv_full + role, k & 1, abort_flag))) break;
        bool over = false;                               // the CTA's last chain
        if (g != 0xffffffffu) {
          if (!(ok = wait_warp(bar_k + role, g & 1, abort_flag))) break;
          tc_fence_after();
          if (g >= lag) {
            const uint32_t c_lo = b_lo + ((g - lag) % C::kStages) * (C::kTileBytes >> 4);
            if (elect_one()) {
              // dK += dS^T Q or dV += P^T dO: A = codes in TMEM (8 columns per 32-query step), B = Q / dO tile MN-major (32 query rows)
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                const uint32_t c = region + 32 * ks;
                mma_mxf8_ts(acc, c + C::kColCodes, c_lo + ks * 256, kIdescMx, c + C::kColWord, c + C::kColWord, ia > 0 || ks > 0);
              }
              tc_commit(bar_done + role);
            }
            // the words lie where the next accumulator lands, and for scale-factor reads the PTX ISA promises no order
            if (!(ok = wait_warp(bar_done + role, (g - lag) & 1, abort_flag))) break;
            tc_fence_after();
          }
        }
        const bool chained = g != 0xffffffffu && g >= lag, last = ia + 1 == na;
        if (elect_one()) {
          if (more) {
            // S^T or dP^T of tile g + 1: both operands K-major, four steps of 32 bytes inside the 128-byte swizzle rows
            const uint32_t c_lo = b_lo + ((g + 1) % C::kStages) * (C::kTileBytes >> 4);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_f8_ss(region, a_lo + 2 * ks, c_lo + 2 * ks, kIdesc, ks > 0);
            tc_commit(bar_s + role);
            if (i + 1 == n) tc_commit(kv_free + role);
          }
          // what nobody waits for comes behind the chain that somebody does
          if (chained) {
            if (last) tc_commit(bar_acc);
            tc_commit(empty + (g - lag) % C::kStages);
          }
        }
        if (chained && ++ia == na) {
          na = item_of(++ka).n;
          ia = 0;
          over = na == 0;
        }
        if (over) break;
        if (more) {
          if (++i == n) {
            n = item_of(++k).n;
            i = 0;
          }
        } else if (elect_one()) {
          mbar_arrive(bar_s + role);                     // no further tile: the columns are free for the last codes
        }
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInDkDv);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == C::kComputeWarps) tmem_dealloc(tmem, C::kTmemCols);
}

template <bool DS32>
static cudaError_t launch_pipe_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                 const CUtensorMap& tds, const BwdParams& p, cudaStream_t stream) {
  using C = PipeCfg;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    // the register split draws on what the launch has: with fewer the compute warps would wait for ever
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, bwd_dkdv_pipe_kernel<DS32>);
    if (e != cudaSuccess) return e;
    if (attr.numRegs * C::kThreads < C::kComputeWarps * 32 * C::kRegsCompute + 128 * C::kRegsIssue) return cudaErrorLaunchOutOfResources;
    e = cudaFuncSetAttribute(bwd_dkdv_pipe_kernel<DS32>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return e;
    done[dev] = true;
  }
  const int items = p.B * p.Hk * (p.N / 128), sms = sm_count();
  count_launch();
  return launch_chained(bwd_dkdv_pipe_kernel<DS32>, items < sms ? items : sms, C::kThreads, C::kSmemBytes, stream, tq, tk, tv, tdo, tds, p);
}

cudaError_t launch_bwd_pipe(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                            const CUtensorMap& tds, const BwdParams& p, cudaStream_t stream) {
  return (p.ds32 ? launch_pipe_t<true> : launch_pipe_t<false>)(tq, tk, tv, tdo, tds, p, stream);
}

}  // namespace dm
