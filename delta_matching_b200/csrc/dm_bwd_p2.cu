// Streaming pass of the backward: dQ = dS K from the quantised dS tiles that an earlier kernel left in a workspace, and, where it
// left P^T tiles too, dV, or dV and dK.
//
// Reference structure: pass 1 writes dS codes, pass 2 multiplies them with K
// (csrc/fq8_dq_pass2_hd128.h:407-442, launched from csrc/flash_bwd_fp8v10_launch.h:158-163).  The alternative without a
// workspace (dm_bwd.cu: bwd_dq_kernel) recomputes S, dP and the exponentials per tile; this kernel only streams
// 16 KiB code tiles and operand tiles through one block-scaled MMA chain per tile, so it is bound by the L2 / HBM stream.
//
// Workspace: tile (head bh, query tile qt, key tile kt) at index (bh * n_t + qt) * n_t + kt holds 128 x 128 e4m3 codes
// as [key][query] (the layout the dK chain consumes), followed after all tiles by four 32-bit words per tile: word b
// belongs to query block b (32 queries) and its byte j is the UE8M0 scale of key block j (32 keys).  With the contract's
// dS blocks of 128 queries x 32 keys the four words of a tile are equal; with 32 x 32 blocks they differ.  The tile is the A operand of dQ in MN-major form
// (M = queries contiguous); K is the B operand in MN-major form as in the other kernels.
//
// Behind the tile-parallel pass (dm_bwd_tiles.cu) the same kernel also makes dV = sum P^T dO and dK = sum dS^T Q of
// every (key tile, kv head), over the group's heads and their query tiles in the order of the key-stationary kernel: there
// the code tile is the A operand as it lies, K-major (M = keys), and dO / Q the MN-major B operand.  P^T tiles have a word per key row
// (byte = query block), ready to use.  Behind the head_dim-256 DK role (dm_bwd_kv.cu) it makes dV and dQ.
//
// One persistent CTA per SM, 320 threads: warps 0-3 write the per-tile scale words into TMEM (code scale x operand scale of the four
// blocks that a row is summed over; warp b writes rows [32 b, 32 b + 32), whose words are one and the same for dQ and dK), warps
// 4-7 write the finished accumulator out (at head_dim 128 two accumulators alternate between items; at head_dim 256 one
// accumulator fills the columns, and an item's first chain waits for the read-out of the previous item), warp 8 TMA, warp 9 MMA.
// Items = (query tile, head) for dQ and (key tile, kv head) for dK and dV, in the order of stream_item.
#include <cuda_bf16.h>
#include "dm_bwd_math.cuh"
#include "dm_common.cuh"
#include "dm_kernels.h"
#include "dm_ptx.cuh"

namespace dm {

template <int D>
struct DqP2Cfg {
  static constexpr int kSub = D / 128;           // 128-byte-wide sub-tiles of a K row
  static constexpr int kDsBytes = 128 * 128;     // dS^T tile
  static constexpr int kKBytes = 128 * D;        // K tile
  static constexpr int kStages = (D == 128) ? 7 : 4;   // dS^T tile + K tile + scale word per stage (224 / 192 KiB)
  static constexpr int kAccs = (D == 128) ? 2 : 1;     // dQ accumulators of D fp32 columns
  static constexpr int kThreads = 320;
  static constexpr int kTmemCols = 512;
  static constexpr int kColDq = 0;
  static constexpr int kColSf = 256;           // kStages x 4 columns: the tile's scale word
  static constexpr int kColOne = 256 + 4 * kStages;   // 4 columns of 0x7F7F7F7F: scale 1.0 for the B operand
  static constexpr int kSmemDs = 0;
  static constexpr int kSmemK = kStages * kDsBytes;
  static constexpr int kSmemBar = kStages * (kDsBytes + kKBytes);
  static constexpr int kSmemBytes = kSmemBar + 256 + 1024;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
};

// A work item: one accumulator.  kDq: (head, query tile), over key tiles.  kDk, kDv: (kv head, key tile), over (head of the
// group, query tile).  dK and dV of all key tiles come first, the most tiles first, then dQ likewise.
enum : int { kDq = 0, kDk = 1, kDv = 2 };
enum : int { kOnlyDq = 0, kDqDkDv = 1, kDqDv = 2 };      // Kinds of items in a launch
struct StreamItem {
  int kind, head, tile;        // head: query head (kDq) or kv head; tile: query tile or key tile
  int n_it, first, per_head;   // tiles; kDk, kDv: first query tile, query tiles per head
};
template <int Kinds>
__device__ __forceinline__ int stream_item_count(const BwdParams& p, int n_t) {
  return n_t * p.B * (p.H + (Kinds == kDqDkDv ? 2 * p.Hk : Kinds == kDqDv ? p.Hk : 0));
}
template <int Kinds>
__device__ __forceinline__ StreamItem stream_item(const BwdParams& p, int n_t, int item) {
  StreamItem r;
  const int BH = p.B * p.H, BHk = p.B * p.Hk, kv_items = Kinds == kDqDkDv ? 2 * n_t * BHk : Kinds == kDqDv ? n_t * BHk : 0;
  if (item < kv_items) {
    r.kind = kDv;
    if (Kinds == kDqDkDv) {
      r.kind = kDk + (item & 1);
      item >>= 1;
    }
    r.tile = item / BHk;
    r.head = item % BHk;
    r.first = p.causal ? r.tile : 0;
    r.per_head = n_t - r.first;
    r.n_it = r.per_head * (p.H / p.Hk);
  } else {
    item -= kv_items;
    r.kind = kDq;
    r.tile = n_t - 1 - item / BH;
    r.head = item % BH;
    r.n_it = p.causal ? (r.tile + 1) : n_t;
    r.first = 0;
    r.per_head = r.n_it;
  }
  return r;
}
// Position inside an item: the tile's index in the workspace and its B operand's row (K, Q or dO codes).
template <int Kinds>
struct StreamWalk {
  int ws, ws_step, row, left, per_head, ws_wrap, row_wrap;
  __device__ __forceinline__ void set(const BwdParams& p, int n_t, const StreamItem& it) {
    const int rep = p.H / p.Hk;
    if (Kinds == kOnlyDq || it.kind == kDq) {
      ws = (it.head * n_t + it.tile) * n_t;
      ws_step = 1;
      row = ((it.head / p.H) * p.Hk + (it.head % p.H) / rep) * p.N;
      ws_wrap = row_wrap = 0;
    } else {
      const int bh = (it.head / p.Hk) * p.H + (it.head % p.Hk) * rep;
      ws = (bh * n_t + it.first) * n_t + it.tile;
      ws_step = n_t;
      row = bh * p.N + it.first * 128;
      ws_wrap = it.first * n_t;                // from the end of one head to the first live query tile of the next
      row_wrap = it.first * 128;
    }
    left = per_head = it.per_head;
  }
  __device__ __forceinline__ void next() {
    ws += ws_step;
    row += 128;
    if (Kinds != kOnlyDq && --left == 0) {
      left = per_head;
      ws += ws_wrap;
      row += row_wrap;
    }
  }
};

template <int D, int Kinds>
__global__ void __launch_bounds__(DqP2Cfg<D>::kThreads, 1)
bwd_stream_kernel(const __grid_constant__ CUtensorMap tm_ds, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_q,
                  const __grid_constant__ CUtensorMap tm_do, const BwdParams p) {
  using C = DqP2Cfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sDs = smem + C::kSmemDs;
  uint8_t* sK = smem + C::kSmemK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kSmemBar);
  // One barrier pair per stage keeps the MMA thread's loop short (one wait, four MMAs, one commit per tile): `full`
  // collects the TMA transaction and one arrival per scale warp, `empty` (MMA commit) releases the stage's shared memory
  // to the TMA warp and its scale-word columns to the scale warps.
  uint64_t* full = bars + 0;          // [kStages] tiles landed and scale word written
  uint64_t* empty = bars + C::kStages;          // [kStages] the stage's chain has read them (MMA commit)
  uint64_t* dq_full = bars + 2 * C::kStages;     // [2] last chain of the item done (MMA commit)
  uint64_t* dq_free = bars + 2 * C::kStages + 2; // [2] accumulator read out (one arrival per epilogue warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::kStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * C::kStages + 5);
  static_assert(2 * C::kStages + 6 <= 32, "barrier block is 256 bytes");

  const int tid = threadIdx.x, warp = tid >> 5;
  const int n_t = p.N / 128;
  const int n_items = stream_item_count<Kinds>(p, n_t);
  const int first_item = static_cast<int>(blockIdx.x), item_step = static_cast<int>(gridDim.x);

  if (tid == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full + s, 1 + 4);
      mbar_init(empty + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(dq_full + s, 1);
      mbar_init(dq_free + s, 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dep_wait();

  if (warp == 8) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_ds);
      tma_prefetch_desc(&tm_k);
      bool ok = true;
      uint32_t g = 0;
      for (int k = 0, item; ok && (item = sched_item(k, first_item, item_step)) < n_items; ++k) {
        const StreamItem itm = stream_item<Kinds>(p, n_t, item);
        StreamWalk<Kinds> wk;
        wk.set(p, n_t, itm);
        const CUtensorMap* ta = (Kinds != kOnlyDq && itm.kind == kDv) ? &tm_p : &tm_ds;
        const CUtensorMap* tb = Kinds == kOnlyDq || itm.kind == kDq ? &tm_k : itm.kind == kDk ? &tm_q : &tm_do;
        for (int it = 0; it < itm.n_it; ++it, ++g, wk.next()) {
          const uint32_t st = g % C::kStages;
          if (g >= C::kStages && !(ok = wait_or_abort(empty + st, ((g / C::kStages) - 1) & 1, abort_flag))) break;
          mbar_expect_tx(full + st, C::kDsBytes + C::kKBytes);
          tma_load_2d(sDs + st * C::kDsBytes, ta, full + st, 0, wk.ws * 128);
          for (int sub = 0; sub < C::kSub; ++sub)
            tma_load_2d(sK + st * C::kKBytes + sub * 16384, tb, full + st, sub * 128, wk.row);
        }
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutProducer + kInDqPass2);
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t ds_lo0 = desc_lo(smem_u32(sDs)), k_lo0 = desc_lo(smem_u32(sK));
      bool ok = true;
      uint32_t g = 0, n_done = 0;
      for (int k = 0, item; ok && (item = sched_item(k, first_item, item_step)) < n_items; ++k, ++n_done) {
        const StreamItem itm = stream_item<Kinds>(p, n_t, item);
        const int n_it = itm.n_it;
        const bool kv_item = Kinds != kOnlyDq && itm.kind != kDq;
        const uint32_t a_step = kv_item ? 2 : 256, idesc = kv_item ? idesc_mxf8(128, 128, false, true, 0, 0) : idesc_mxf8(128, 128, true, true, 0, 0);
        const uint32_t acc = n_done % C::kAccs;
        // the accumulator was last used kAccs items ago: its read-out must be complete
        if (n_done >= C::kAccs && !(ok = wait_or_abort(dq_free + acc, ((n_done / C::kAccs) - 1) & 1, abort_flag))) break;
        for (int it = 0; it < n_it; ++it, ++g) {
          const uint32_t st = g % C::kStages;
          if (!(ok = wait_or_abort(full + st, (g / C::kStages) & 1, abort_flag))) break;
          tc_fence_after();
          // dQ += dS K over the tile's 128 keys: A = dS^T tile read MN-major, B = K tile read MN-major; both advance
          // by 32 key rows (4096 bytes) per step; byte ks of the scale word belongs to key block ks.  dK, dV: A K-major, 32
          // bytes (queries) per step.
          const uint32_t ds_lo = ds_lo0 + st * (C::kDsBytes >> 4), k_lo = k_lo0 + st * (C::kKBytes >> 4);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
            for (int sub = 0; sub < C::kSub; ++sub)
              mma_mxf8_ss(tmem + C::kColDq + D * acc + 128 * sub, ds_lo + ks * a_step, k_lo + sub * 1024 + ks * 256,
                          idesc | (static_cast<uint32_t>(ks) << 29), tmem + C::kColSf + 4 * st, tmem + C::kColOne,
                          (it > 0) || (ks > 0));
          }
          tc_commit(empty + st);
          if (it == n_it - 1) tc_commit(dq_full + acc);
        }
      }
      if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutMma + kInDqPass2);
    }
  } else if (warp < 4) {
    // ------------------------------------------------------------------------------------------ scale words
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    tmem_st4(tmem + lane_base + C::kColOne, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
    bool ok = true;
    // The tile's scale word and the four scales it is multiplied with come from global memory: they are requested kAhead
    // tiles before they are used, through a walk over the CTA's (item, tile) sequence that runs ahead of the consuming one.
    //   dQ: the word of this warp's query block (byte = key block) and the tile's four K scales
    //   dK: byte `warp` (this warp's key block) of the words of the four query blocks and their Q scales
    //   dV: this row's own word, finished
    // The slots stay where they are and the loop is unrolled over them: a queue that moves up by a slot per tile waits, in the
    // move, for the load of the tile before.  Forward + backward on the GPU: N=1024 H=8 Hk=2 59.5 -> 57.4 us, N=1920 H=6 Hk=2 D=256 89.9 ->
    // 86.0, B=2 N=1536 H=8 Hk=1 115.9 -> 110.1, B=3 N=1792 H=15 Hk=5 198.5 -> 196.5; N=4096 H=8 Hk=1 D=256 309 -> 318.
    // (dV and dQ of head_dim 256, bound by their stream: 0.7 % slower per step with four than with one.)
    constexpr int kAhead = Kinds == kDqDv ? 1 : 4;
    int pre_k = 0, pre_item = first_item, pre_left = 0, pre_kind = kDq;
    StreamWalk<Kinds> pre;
    auto pre_set = [&]() {
      if (pre_item >= n_items) return;
      const StreamItem itm = stream_item<Kinds>(p, n_t, pre_item);
      pre.set(p, n_t, itm);
      pre_left = itm.n_it;
      pre_kind = itm.kind;
    };
    pre_set();
    struct Slot {
      uint4 w;
      float4 f;
      int kind;            // -1: the sequence has ended
    } slot[kAhead];
    auto request = [&](Slot& q) {
      q.kind = -1;
      if (pre_item >= n_items) return;
      q.kind = pre_kind;
      if (Kinds == kOnlyDq || pre_kind == kDq) {
        q.w.x = reinterpret_cast<const uint32_t*>(p.ds_words)[static_cast<size_t>(pre.ws) * 4 + warp];
        q.f = *reinterpret_cast<const float4*>(p.ks + pre.row / 32);
      } else if (pre_kind == kDk) {
        q.w = *reinterpret_cast<const uint4*>(p.ds_words + static_cast<size_t>(pre.ws) * 16);
        q.f = *reinterpret_cast<const float4*>(p.qs + pre.row / 32);
      } else {
        q.w.x = reinterpret_cast<const uint32_t*>(p.p_words)[static_cast<size_t>(pre.ws) * 128 + tid];
        q.f = make_float4(1.f, 1.f, 1.f, 1.f);
      }
      if (--pre_left == 0) {
        pre_item = sched_item(++pre_k, first_item, item_step);
        pre_set();
      } else {
        pre.next();
      }
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      slot[i].w = make_uint4(0, 0, 0, 0);
      request(slot[i]);
    }
    uint32_t g = 0;
    for (bool more = true; more;) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        if (!more || slot[i].kind < 0) {
          more = false;
          continue;
        }
        uint32_t w = slot[i].w.x;
        if (Kinds != kOnlyDq && slot[i].kind == kDk) {
          const uint4 v = slot[i].w;
          const int sh = 8 * warp;
          w = pack4((v.x >> sh) & 0xFF, (v.y >> sh) & 0xFF, (v.z >> sh) & 0xFF, (v.w >> sh) & 0xFF);
        }
        const float4 f = slot[i].f;
        const uint32_t word = pack4(sb_mul(w & 0xFF, scale_to_sb(f.x)), sb_mul((w >> 8) & 0xFF, scale_to_sb(f.y)),
                                    sb_mul((w >> 16) & 0xFF, scale_to_sb(f.z)), sb_mul(w >> 24, scale_to_sb(f.w)));
        request(slot[i]);
        const uint32_t st = g % C::kStages;
        if (g >= C::kStages && !(ok = wait_warp(empty + st, ((g / C::kStages) - 1) & 1, abort_flag))) {
          more = false;
          continue;
        }
        tc_fence_after();
        tmem_st4(tmem + lane_base + C::kColSf + 4 * st, word, word, word, word);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(full + st);
        ++g;
      }
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDqPass2);
  } else {
    // ------------------------------------------------------------------------------------------ dQ read-out
    const int quad = warp & 3;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    bool ok = true;
    uint32_t n_done = 0;
    for (int k = 0, item; ok && (item = sched_item(k, first_item, item_step)) < n_items; ++k, ++n_done) {
      const StreamItem itm = stream_item<Kinds>(p, n_t, item);
      const bool kv_item = Kinds != kOnlyDq && itm.kind != kDq;
      const int heads = kv_item ? p.Hk : p.H, b = itm.head / heads, h = itm.head % heads;
      const float mul = kv_item ? 1.0f : p.sm_scale;
      const uint32_t acc = n_done % C::kAccs;
      if (!(ok = wait_warp(dq_full + acc, (n_done / C::kAccs) & 1, abort_flag))) break;
      tc_fence_after();
      __nv_bfloat16* dst = p.dq + b * p.dq_sb + h * p.dq_sh;
      int64_t sn = p.dq_sn;
      if (Kinds != kOnlyDq && itm.kind == kDk) {
        dst = p.dk + b * p.dk_sb + h * p.dk_sh;
        sn = p.dk_sn;
      }
      if (Kinds != kOnlyDq && itm.kind == kDv) {
        dst = p.dv + b * p.dv_sb + h * p.dv_sh;
        sn = p.dv_sn;
      }
      dst += (static_cast<int64_t>(itm.tile) * 128 + quad * 32) * sn;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) store_rows32(tmem + lane_base + C::kColDq + D * acc + 32 * c, mul, dst + 32 * c, sn);
      tc_fence_before();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(dq_free + acc);
    }
    if (!ok) raise_abort(abort_flag, p.status, kStatusTimeoutCompute + kInDqPass2);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, C::kTmemCols);
}

template <int D, int Kinds>
static cudaError_t launch_stream_t(const CUtensorMap& tds, const CUtensorMap& tk, const CUtensorMap& tp, const CUtensorMap& tq,
                                   const CUtensorMap& tdo, const BwdParams& p, cudaStream_t stream) {
  using C = DqP2Cfg<D>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(bwd_stream_kernel<D, Kinds>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  const int sms = sm_count();
  const int items = (p.N / 128) * p.B * (p.H + (Kinds == kDqDkDv ? 2 * p.Hk : Kinds == kDqDv ? p.Hk : 0));
  count_launch();
  return launch_chained(bwd_stream_kernel<D, Kinds>, items < sms ? items : sms, C::kThreads, C::kSmemBytes, stream, tds, tk, tp, tq, tdo, p);
}

cudaError_t launch_bwd_dq_p2(int D, const CUtensorMap& tds, const CUtensorMap& tk, const BwdParams& p, cudaStream_t stream) {
  return (D == 128 ? launch_stream_t<128, kOnlyDq> : launch_stream_t<256, kOnlyDq>)(tds, tk, tds, tk, tk, p, stream);   // the last three unused
}

cudaError_t launch_bwd_stream(int D, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tdo, const CUtensorMap& tds,
                              const CUtensorMap& tp, const BwdParams& p, cudaStream_t stream) {
  return (D == 128 ? launch_stream_t<128, kDqDkDv> : launch_stream_t<256, kDqDkDv>)(tds, tk, tp, tq, tdo, p, stream);
}

cudaError_t launch_bwd_stream_dq_dv(const CUtensorMap& tk, const CUtensorMap& tdo, const CUtensorMap& tds, const CUtensorMap& tp,
                                    const BwdParams& p, cudaStream_t stream) {
  return launch_stream_t<256, kDqDv>(tds, tk, tp, tk, tdo, p, stream);
}

}  // namespace dm
