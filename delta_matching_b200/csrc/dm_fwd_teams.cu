// Forward of delta-matching fp8 attention on sm_100a at head_dim 128 (numerics: see dm_fwd.cu, whose arithmetic and order this keeps, so
// that either kernel gives the same bits).
//
// Work item = one 128-query tile of one (batch, query head); a persistent CTA per SM walks a list of items.  The key tiles of an item go
// round three teams of four softmax warps (thread = query row), a team to an S accumulator of 128 TMEM columns; O has the other 128.  The
// exponentials of a tile need nothing from the tile before (P codes have a basis of their own per 32 keys): only the running maximum and
// sum go from team to team, at a tile's end.  So a team's round trip P codes -> PV chain -> completion -> S chain runs behind the
// exponentials of the other two, also where an SM has a single item.  (Cycles of a tile there: S issued -> seen by the team 700, exponentials and
// codes 1650 - 2100, hand-over and words 700, P codes -> PV chain 240, PV chain -> next S 500 - 650; a third of it per tile with three teams.)
//
// With many items the exponentials of a call bound neither this nor the two CTAs per SM of dm_fwd.cu: 450 us at B=4 N=4096 H=32 Hk=8 causal become
// 378 without any exponential and 279 without three quarters of the softmax; MUFU 55 %, issue slots 55 %.  What the teams gain there
// is the end of a call.  us, two CTAs per SM -> teams, the forward alone in single calls: N=1024 H=8 Hk=2 causal 16.4 -> 12.8, N=4096 H=9 56.5 -> 34.9, N=8192 H=6 105.8 -> 84.1;
// bidirectional N=2048 H=42 88.8 -> 74.4, B=8 N=2048 H=16 214 -> 200 (dm_fwd.cu says which calls come here, and what the others would take).
// Slower: K and V by a producer warp each (441 -> 448 at B=4 N=4096 H=32), a staging row for each team in the place of a second Q tile and the fourth
// stages (200 -> 216 at B=8 N=2048 H=16).
#include <type_traits>
#include <cuda_bf16.h>
#include "dm_common.cuh"
#include "dm_kernels.h"

namespace dm {

struct FwdTeamsCfg {
  static constexpr int kTileBytes = 128 * 128;
  static constexpr int kTeams = 3, kStages = 4;
  static constexpr int kSoftmaxWarps = 4 * kTeams;
  static constexpr int kThreads = (kSoftmaxWarps + 4) * 32;
  // Registers a thread: 512 x 128 at launch = 384 x 152 + 128 x 56.
  static constexpr int kRegsSoftmax = 152, kRegsIssue = 56;
  static_assert(384 * kRegsSoftmax + 128 * kRegsIssue <= kThreads * 128, "a split above the launch's own registers would wait for ever");
  static constexpr int kTmemCols = 512;
  static constexpr int kColO = 128 * kTeams;           // behind the S accumulators: O, 128 fp32 columns
  // Relative to a team's S accumulator, over columns that the writing warp itself has loaded: P codes of 32 keys in 8 columns each, then
  static constexpr int kColSfa = 32;                   // 4 columns, each this row's SFA word
  static constexpr int kColSfb = 36;                   // 4 columns, each the tile's V scale word
  // shared memory: Q (two items) | K stages | V stages | ...
  static constexpr int kSmemQ = 0;
  static constexpr int kSmemK = 2 * kTileBytes;
  static constexpr int kSmemV = kSmemK + kStages * kTileBytes;
  static constexpr int kSmemOut = kSmemV + kStages * kTileBytes;   // 128 rows of O on their way out
  static constexpr int kOutRow = 272;                              // 256 bytes + 16 of padding (bank spread)
  static constexpr int kSmemMl = kSmemOut + 128 * kOutRow;   // running maximum and sum of a row behind a team's tile
  // [kStages] scales of a key tile (K, V; four each) and of the query tile (four), which travel with V
  static constexpr int kSmemVec = kSmemMl + kTeams * 128 * 8;
  static constexpr int kSmemBar = kSmemVec + kStages * 48;
  static constexpr int kSmemBytes = kSmemBar + 512 + 1024;   // + slack for the 1024-byte alignment of the tile base
  static_assert(kSmemBytes <= 232448, "shared memory budget");
};

// Persistent: the grid is the SM count; CTA j processes the work items sched_item(0, j), sched_item(1, j), ... of a list ordered by
// decreasing number of key tiles (item -> query tile n_qt - 1 - item / (B H), head item % (B H)).  The CTA's tiles are counted through
// all its items; tile g belongs to team g % 3 and its S accumulator, as number g / 3 of every barrier of that team.
// S of tile g + 3 waits for the completion of the PV chain of tile g.  It overwrites the TMEM columns from which that chain reads its codes and
// scale-factor words, and two threads issue the two: nothing but completion orders them (dm_fwd.cu's kOrdered asks what issue order gives within
// one thread).  The softmax warps' parity waits for a PV chain rest on the same wait: with S of a tile landed, the PV chain before it in that
// accumulator is complete, so a barrier of PV chains is never more than one phase away from the one that is tested.
__global__ void __launch_bounds__(FwdTeamsCfg::kThreads, 1)
fwd_teams_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  using C = FwdTeamsCfg;
  constexpr int T = C::kTeams;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + C::kSmemQ;
  uint8_t* sK = smem + C::kSmemK;
  uint8_t* sV = smem + C::kSmemV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  uint64_t* bar_s = bars + 0;                // [T] S accumulator ready (MMA commit)
  uint64_t* bar_p = bar_s + T;               // [T] P codes + scale words written (one arrival per softmax warp)
  uint64_t* bar_o = bar_p + T;               // [T] PV chain done (MMA commit)
  uint64_t* bar_ml = bar_o + T;              // [T][4] running maximum and sum of a row quarter behind the tile are written
  uint64_t* full_k = bar_ml + 4 * T;         // [kStages]
  uint64_t* full_v = full_k + C::kStages;    // [kStages] V and the scales
  uint64_t* empty_k = full_v + C::kStages;   // [kStages] K stage free again (MMA commit behind the S chain)
  uint64_t* empty_v = empty_k + C::kStages;  // [kStages] V stage free again (MMA commit behind the PV chain)
  uint64_t* bar_q = empty_v + C::kStages;    // [2] Q of an item landed
  uint64_t* bar_qfree = bar_q + 2;           // [2] the item's last S chain has read Q (MMA commit)
  uint64_t* bar_ofree = bar_qfree + 2;       // O of an item is in registers (one arrival per warp that writes it out)
  uint64_t* bar_out = bar_ofree + 1;         // ... and has left its rows in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_out + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_out + 2);
  static_assert((7 * T + 4 * C::kStages + 8) * 8 <= 512, "barrier block");

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);     // a warp-uniform value, also to the compiler
  const int n_qt = p.N / 128;
  const int BH = p.B * p.H;
  const int n_items = n_qt * BH;
  const int rep = p.H / p.Hk;
  const int first_item = static_cast<int>(blockIdx.x), item_step = static_cast<int>(gridDim.x);

  if (tid == 0) {
    for (int s = 0; s < 7 * T + 4 * C::kStages + 6; ++s) mbar_init(bars + s, (bars + s >= bar_p && bars + s < bar_o) || bars + s >= bar_ofree ? 4 : 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == C::kSoftmaxWarps) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem = 0;                         // 512 columns are all there are: the allocation starts at column 0
  // The next kernel does not start its set-up under this one.  Its CTAs would come onto each SM straight behind the one here and keep the
  // division of that SM's 256 KB that 199 KB of shared memory call for, so that the producers of the next call run with the smallest L1 (with a
  // carve-out of their own they did not).  us, producers and forward in a run, two CTAs per SM -> teams with that start -> without, bidirectional:
  // 14.5 -> 13.7 -> 11.5 (N=256, 71 heads), 64.8 -> 68.4 -> 62.0 (N=768, 122), 236 -> 250 -> 227 (N=512, 775), 507 -> 554 -> 509 (N=768, 1010).
  grid_dep_wait_alone();

  if (warp >= C::kSoftmaxWarps) {
    reg_dec<C::kRegsIssue>();
    if (warp == C::kSoftmaxWarps + 2) {
      // ------------------------------------------------------------------------------------------ TMA producer
      if (elect_one()) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        bool ok = true;
        uint32_t g = 0;                                // tiles issued so far by this CTA
        for (int k = 0, item; ok && (item = sched_item(k, first_item, item_step)) < n_items; ++k) {
          const int qt = n_qt - 1 - item / BH, bh = item % BH;
          const int bhk = (bh / p.H) * p.Hk + (bh % p.H) / rep;
          const int n_it = p.causal ? (qt + 1) : n_qt;
          const int q_row = bh * p.N + qt * 128, slot = k & 1;
          int row = bhk * p.N + (n_it - 1) * 128;
          if (k >= 2 && !(ok = wait_or_abort(bar_qfree + slot, ((k >> 1) - 1) & 1, abort_flag))) break;
          mbar_expect_tx(bar_q + slot, C::kTileBytes);
          tma_load_2d(sQ + slot * C::kTileBytes, &tm_q, bar_q + slot, 0, q_row);
          for (int it = 0; it < n_it; ++it, ++g, row -= 128) {
            const uint32_t st = g % C::kStages, eph = ((g / C::kStages) - 1) & 1;
            if (g >= C::kStages && !(ok = wait_or_abort(empty_k + st, eph, abort_flag))) break;
            mbar_expect_tx(full_k + st, C::kTileBytes);
            tma_load_2d(sK + st * C::kTileBytes, &tm_k, full_k + st, 0, row);
            if (g >= C::kStages && !(ok = wait_or_abort(empty_v + st, eph, abort_flag))) break;
            uint8_t* vec = smem + C::kSmemVec + st * 48;
            mbar_expect_tx(full_v + st, C::kTileBytes + 48);
            tma_load_2d(sV + st * C::kTileBytes, &tm_v, full_v + st, 0, row);
            bulk_load_1d(vec, p.ks + row / 32, 16, full_v + st);
            bulk_load_1d(vec + 16, p.vs + row / 32, 16, full_v + st);
            bulk_load_1d(vec + 32, p.qs + q_row / 32, 16, full_v + st);
          }
        }
        if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInForward);
      }
    } else if (warp < C::kSoftmaxWarps + 2) {
      // ------------------------------------------------------------------------------------------ MMA issuers
      // A warp for the S chains and one for the PV chains: neither waits behind what the other waits for.
      const bool pv = warp == C::kSoftmaxWarps + 1;
      if (elect_one()) {
        constexpr uint32_t kIdescS = idesc_f8(128, 128, false, false);
        const uint32_t q_lo0 = desc_lo(smem_u32(sQ)), k_lo0 = desc_lo(smem_u32(sK)), v_lo0 = desc_lo(smem_u32(sV));
        bool ok = true;
        int st = 0, team = 0;                          // the tile's ring stage and team, and the phases of their barriers
        uint32_t st_ph = 0, ph = 0;
        bool again = false;                            // the accumulator has been in use before
        for (int k = 0, item; ok && (item = sched_item(k, first_item, item_step)) < n_items; ++k) {
          const int n_it = p.causal ? (n_qt - item / BH) : n_qt;
          const uint32_t q_lo = q_lo0 + (k & 1) * (C::kTileBytes >> 4);
          if (!pv && !(ok = wait_or_abort(bar_q + (k & 1), (k >> 1) & 1, abort_flag))) break;
          for (int it = 0; it < n_it; ++it) {
            const uint32_t s_col = tmem + 128 * team;
            if (!pv) {
              // S = Q K^T: both operands K-major, k-step of 32 bytes inside the 128-byte swizzle row
              if (!(ok = wait_or_abort(full_k + st, st_ph, abort_flag))) break;
              if (again && !(ok = wait_or_abort(bar_o + team, ph ^ 1, abort_flag))) break;
              tc_fence_after();
              const uint32_t k_lo = k_lo0 + st * (C::kTileBytes >> 4);
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) mma_f8_ss(s_col, q_lo + 2 * ks, k_lo + 2 * ks, kIdescS, ks > 0);
              tc_commit(bar_s + team);
              tc_commit(empty_k + st);                 // the K stage is free as soon as this chain has read it
              if (it == n_it - 1) tc_commit(bar_qfree + (k & 1));
            } else {
              // O += P V: A = P codes in TMEM (8 columns per 32-key step), B = V tile MN-major (32 key rows per step).  The first
              // chain of an item overwrites O.
              if (!(ok = wait_or_abort(full_v + st, st_ph, abort_flag))) break;
              if (it == 0 && k > 0 && !(ok = wait_or_abort(bar_ofree, (k - 1) & 1, abort_flag))) break;
              if (!(ok = wait_or_abort(bar_p + team, ph, abort_flag))) break;
              tc_fence_after();
              const uint32_t v_lo = v_lo0 + st * (C::kTileBytes >> 4);
#pragma unroll
              for (int ks = 0; ks < 4; ++ks)
                mma_mxf8_ts(tmem + C::kColO, s_col + 8 * ks, v_lo + ks * 256, idesc_mxf8(128, 128, false, true, ks, ks), s_col + C::kColSfa,
                            s_col + C::kColSfb, (it > 0) || (ks > 0));
              tc_commit(bar_o + team);
              tc_commit(empty_v + st);
            }
            if (++st == C::kStages) {
              st = 0;
              st_ph ^= 1;
            }
            if (++team == T) {
              team = 0;
              ph ^= 1;
              again = true;
            }
          }
        }
        if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInForward);
      }
    }
  } else {
    // ------------------------------------------------------------------------------------------ softmax / epilogue
    reg_inc<C::kRegsSoftmax>();
    const int team = warp >> 2;
    const int quad = warp & 3;
    const int trow = tid & 127;                                            // row of the tile = TMEM lane
    const int before = (team == 0 ? T : team) - 1;                         // the team of the tile before
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem + lane_base + 128 * team;
    const uint32_t ml_a = smem_u32(smem + C::kSmemMl) + 8 * trow;
    const uint32_t s_bar = smem_u32(bar_s + team), p_bar = smem_u32(bar_p + team);
    const uint32_t ml_bar = smem_u32(bar_ml + 4 * team + quad), ml_bar_b = smem_u32(bar_ml + 4 * before + quad);
    const uint32_t vec_a = smem_u32(smem + C::kSmemVec), v_bar = smem_u32(full_v);
    bool ok = true;
    // The team's tile number n, the CTA's tile g, is tile `it` of the n_it of its item k.
    int k = 0, item = first_item, it = team, n_it = 0;
    uint32_t g = team;
    for (uint32_t n = 0;; ++n, g += T, it += T) {
      for (; item < n_items; item = sched_item(++k, first_item, item_step)) {
        n_it = p.causal ? (n_qt - item / BH) : n_qt;
        if (it < n_it) break;
        it -= n_it;
      }
      if (item >= n_items) break;
      const uint32_t ph = n & 1, ph_b = (team == 0 ? ph ^ 1 : ph);         // of this team's barriers; of the team's before
      float m, l;
      // One key tile.  kDiag: the tile on the diagonal of a causal problem (always the first one visited), where keys
      // above the query index are masked; a compile-time variant so that the other tiles carry no select per element.
      auto tile = [&](auto diag_tag) -> bool {
        constexpr bool kDiag = decltype(diag_tag)::value;
        const uint32_t st = g % C::kStages, va = vec_a + 48 * st, st_ph = (g / C::kStages) & 1;
        // S and the scales, in one look.  (The scales second: with S of this tile landed, those of the stage's former tile have.)
        bool seen = mbar_test_wait(s_bar, ph);
        seen = mbar_test_wait(v_bar + 8 * st, st_ph) && seen;
        if (!__all_sync(0xffffffffu, seen)) {
          seen = poll_or_abort(s_bar, ph, abort_flag);
          seen = seen && poll_or_abort(v_bar + 8 * st, st_ph, abort_flag);
          if (!__all_sync(0xffffffffu, seen)) return false;
        }
        tc_fence_after();
        float bsum[4], kb[4], bmax[4];
        uint32_t r[2][32];
        tmem_ld32(t_s, r[0]);
        const float qsl = lds_f(va + 32 + 4 * quad) * kLog2e;
        const float4 ks4 = lds_f4(va);
        const float cb[4] = {qsl * ks4.x, qsl * ks4.y, qsl * ks4.z, qsl * ks4.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t (&rc)[32] = r[c & 1];
          tmem_wait_ld();
          if (c < 3) tmem_ld32(t_s + 32 * (c + 1), r[(c + 1) & 1]);        // next chunk in flight
          if (c == 1) {                                                    // the columns of the words are in registers
            const float4 vs4 = lds_f4(va + 16);
            const uint32_t sfb = pack4(scale_to_sb(vs4.x), scale_to_sb(vs4.y), scale_to_sb(vs4.z), scale_to_sb(vs4.w));
            tmem_st4(t_s + C::kColSfb, sfb, sfb, sfb, sfb);
          }
          if (kDiag) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (32 * c + e > trow) rc[e] = 0xff800000u;                  // -inf: key index above the query index
          }
          float2 s2[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) s2[e] = make_float2(__uint_as_float(rc[2 * e]), __uint_as_float(rc[2 * e + 1]));
          bmax[c] = max32(s2) * cb[c];
          kb[c] = fmaxf(floorf(bmax[c]), -1e30f);
          const float2 c2 = splat2(cb[c]), bias2 = splat2(7.0f - kb[c]);
          float2 sum0 = make_float2(0.f, 0.f), sum1 = make_float2(0.f, 0.f);
          uint32_t codes[8];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float2 p0 = ex2_2(fma2(s2[e], c2, bias2));
            // three of the sixteen pairs take the polynomial: the MUFU pipe is the floor of this loop, the FMA pipe has room
            const float2 p1 = (e == 2 || e == 8 || e == 14) ? ex2_poly2(fma2(s2[e + 1], c2, bias2)) : ex2_2(fma2(s2[e + 1], c2, bias2));
            sum0 = add2(sum0, p0);
            sum1 = add2(sum1, p1);
            codes[e / 2] = cvt_e4m3x4(p0.x, p0.y, p1.x, p1.y);
          }
          sum0 = add2(sum0, sum1);
          bsum[c] = sum0.x + sum0.y;
          tmem_st8(t_s + 8 * c, codes);
        }
        const float mcand = ceilf(fmaxf(fmaxf(bmax[0], bmax[1]), fmaxf(bmax[2], bmax[3])));
        // Running maximum and sum of the row, from the team of the tile before and on to the team of the next.  (The wait also between
        // items, where nothing is handed on: a slot is then written again behind its reader's own hand-over.)
        if ((n > 0 || team > 0) && !wait_warp(ml_bar_b, ph_b, abort_flag)) return false;
        float acc_scale = 1.0f;
        if (it == 0) {
          m = mcand;
          l = 0.f;
        } else {
          const float2 ml = lds_f2(ml_a + 1024 * before);
          m = ml.x;
          l = ml.y;
          if (mcand > m + 32.0f) {
            acc_scale = sb_to_scale(static_cast<uint32_t>(max(0, min(__float2int_rn(m - mcand) + 127, 254))));
            m = mcand;
          }
        }
        l *= acc_scale;
        uint32_t sb[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int e = __float2int_rn(kb[c] - 7.0f - m);      // saturates for fully masked blocks
          sb[c] = static_cast<uint32_t>(max(0, min(max(e, -1000) + 127, 254)));
          l = fmaf(bsum[c], __uint_as_float(sb[c] << 23), l);
        }
        sts_f2(ml_a + 1024 * team, m, l);
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(ml_bar);
        if (__any_sync(0xffffffffu, acc_scale != 1.0f)) {
          // rare: the running max moved by more than 32 binades; rescale this warp's O rows in place, between the PV chains of the
          // tile before and of this one
          if (!wait_warp(smem_u32(bar_o + before), ph_b, abort_flag)) return false;
          tc_fence_after();
          for (int c = 0; c < 4; ++c) {
            uint32_t ro[32];
            tmem_ld32(tmem + lane_base + C::kColO + 32 * c, ro);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; ++e) ro[e] = __float_as_uint(__uint_as_float(ro[e]) * acc_scale);
            tmem_st32(tmem + lane_base + C::kColO + 32 * c, ro);
          }
        }
        const uint32_t sfa = pack4(sb[0], sb[1], sb[2], sb[3]);
        tmem_st4(t_s + C::kColSfa, sfa, sfa, sfa, sfa);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(p_bar);
        return true;
      };
      if (!(ok = (p.causal && it == 0) ? tile(std::true_type{}) : tile(std::false_type{}))) break;
      if (it != n_it - 1) continue;
      // the item's last tile: this team writes O out
      if (!(ok = wait_warp(smem_u32(bar_o + team), ph, abort_flag))) break;
      tc_fence_after();
      const float inv_l = 1.0f / l;
      // A thread holds one row of O: it leaves as one bulk copy per row, out of shared memory (behind the copies of the item before), so
      // that the next item's first PV chain waits for little more than the loads.
      const int lane = tid & 31;
      const uint32_t stage = smem_u32(smem + C::kSmemOut) + trow * C::kOutRow;
      if (k > 0 && !(ok = wait_warp(bar_out, (k - 1) & 1, abort_flag))) break;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_base + C::kColO + 32 * c, r);
        tmem_wait_ld();
        if (c == 3) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_ofree);
        }
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[2 * e]) * inv_l, __uint_as_float(r[2 * e + 1]) * inv_l);
          w[e] = *reinterpret_cast<uint32_t*>(&v);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sts_u4(stage + 64 * c + 16 * e, w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
      }
      fence_async_smem();
      const int qt = n_qt - 1 - item / BH, bh = item % BH, b = bh / p.H, h = bh % p.H;
      bulk_store_1d(p.o + static_cast<int64_t>(b) * p.o_sb + static_cast<int64_t>(h) * p.o_sh + static_cast<int64_t>(qt * 128 + trow) * p.o_sn, stage, 256);
      bulk_commit_group();
      p.lse[static_cast<size_t>(bh) * p.N + qt * 128 + trow] = (m + log2f(l)) * kLn2;
      bulk_wait_group_read<0>();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_out);
    }
    bulk_wait_group<0>();
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInForward);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == C::kSoftmaxWarps) tmem_dealloc(tmem, C::kTmemCols);
}

cudaError_t launch_fwd_teams(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream) {
  using C = FwdTeamsCfg;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    // the register split draws on what the launch has: with fewer the softmax warps would wait for ever
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, fwd_teams_kernel);
    if (e != cudaSuccess) return e;
    if (attr.numRegs * C::kThreads < C::kSoftmaxWarps * 32 * C::kRegsSoftmax + 128 * C::kRegsIssue) return cudaErrorLaunchOutOfResources;
    e = cudaFuncSetAttribute(fwd_teams_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return e;
    done[dev] = true;
  }
  const int items = p.B * p.H * (p.N / 128), sms = sm_count();
  count_launch();
  return launch_chained(fwd_teams_kernel, items < sms ? items : sms, C::kThreads, C::kSmemBytes, stream, tq, tk, tv, p);
}

}  // namespace dm
