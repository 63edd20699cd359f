// Quantisation producers: bf16 Q / K / V / dO -> e4m3 codes with one power-of-two scale per 32 tokens over all of
// head_dim, K centred by its per-(batch, kv head) mean over tokens, optional stale delta rowsum(dO * O).
//
// Rule (delta_matching/sm100/quant.py:1-12, 160-176; emulation delta_matching/reference.py:96-107):
//   y = (x - mean) * prescale (fp32);  amax over the 32 x D block = m * 2^E;
//   scale = 2^(E-8) if m <= 1.75 else 2^(E-7)  (the smallest power of two with amax <= 448 * scale; 1 if amax == 0);
//   code = e4m3_rne(y * 2^-e)  (exact scaling, never saturates).
// K mean (delta_matching/reference.py:328-338): fp32 sums of 64-token chunks folded serially in chunk order, / N.
// HBM-bound kernels: 16-byte loads, 16-byte code stores, one 32-token block per 128-thread CTA.
#include <cuda_bf16.h>
#include "dm_common.cuh"
#include "dm_kernels.h"
#include "dm_quant_block.cuh"

namespace dm {

// ------------------------------------------------------------------------------------------------ K mean
// Stage 1: one CTA per (64-token chunk, batch * kv head): column sums of the chunk, rows folded in a fixed order.
template <int D>
struct KMeanTile {
  static constexpr int kTpr = D / 8;            // threads per token row (16 bytes each)
  static constexpr int kRpp = 128 / kTpr;       // rows per pass
};

template <int D>
__device__ __forceinline__ void kmean_block(const KMeanParams& p, int chunk, int bh, float (*red)[D]) {
  constexpr int kTpr = KMeanTile<D>::kTpr, kRpp = KMeanTile<D>::kRpp;
  const int b = bh / p.Hk, h = bh % p.Hk;
  const int tid = threadIdx.x;
  const int c8 = tid % kTpr, r0 = tid / kTpr;
  const __nv_bfloat16* base = p.k + b * p.sb + h * p.sh + static_cast<int64_t>(chunk) * 64 * p.sn + c8 * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int r = r0; r < 64; r += kRpp) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(base + r * p.sn));
    float f[8];
    bf16x8_to_float(v, f);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += f[i];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[r0][c8 * 8 + i] = acc[i];
  __syncthreads();
  for (int c = tid; c < D; c += 128) {
    float s = red[0][c];
#pragma unroll
    for (int r = 1; r < kRpp; ++r) s += red[r][c];
    p.partial[(static_cast<size_t>(bh) * (p.N / 64) + chunk) * D + c] = s;
  }
}

template <int D>
__global__ void __launch_bounds__(128) kmean_partial_kernel(const KMeanParams p) {
  __shared__ float red[KMeanTile<D>::kRpp][D];
  grid_dep_wait();
  kmean_block<D>(p, blockIdx.x, blockIdx.y, red);
}

// Mean of one column: serial fold of the chunk sums in chunk order, divided by N.  Bound by the latency of its loads, 0.6 us a
// batch: 32 in flight, added in chunk order (with eight the fold of 512 chunks took longer than the chunk sums themselves: q, k, v
// producers at N=32768 H=64 Hk=8 206 -> 181 us).
__device__ __forceinline__ float kmean_column(const KMeanParams& p, int bh, int c) {
  const int nchunk = p.N / 64;
  const float* src = p.partial + static_cast<size_t>(bh) * nchunk * p.D + c;
  float s = 0.f;
  int j = 0;
  for (; j + 32 <= nchunk; j += 32) {
    float v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) v[u] = src[static_cast<size_t>(j + u) * p.D];
#pragma unroll
    for (int u = 0; u < 32; ++u) s += v[u];
  }
  if (j < nchunk) {
    float v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) v[u] = (j + u < nchunk) ? src[static_cast<size_t>(j + u) * p.D] : 0.f;
#pragma unroll
    for (int u = 0; u < 32; ++u)
      if (j + u < nchunk) s += v[u];
  }
  return s / static_cast<float>(p.N);
}

// Stage 2: one CTA per (batch, kv head).
__global__ void kmean_fold_kernel(const KMeanParams p) {
  grid_dep_wait();
  const int bh = blockIdx.x;
  for (int c = threadIdx.x; c < p.D; c += blockDim.x) p.mean[static_cast<size_t>(bh) * p.D + c] = kmean_column(p, bh, c);
}

cudaError_t launch_kmean(const KMeanParams& p, cudaStream_t stream) {
  dim3 grid(p.N / 64, p.B * p.Hk);
  cudaError_t e = launch_chained(p.D == 128 ? kmean_partial_kernel<128> : kmean_partial_kernel<256>, grid, 128, 0, stream, p);
  if (e == cudaSuccess) e = launch_chained(kmean_fold_kernel, p.B * p.Hk, 128, 0, stream, p);
  count_launch(2);
  return e;
}

// ------------------------------------------------------------------------------------------------ quantiser
cudaError_t launch_quant(const QuantParams& p, cudaStream_t stream);
template <int D, bool kMean, bool kStale>
__global__ void __launch_bounds__(128, D == 128 ? 10 : 6) quant_kernel(const QuantParams p) {
  __shared__ float wmax[4];
  grid_dep_wait();
  quant_block<D, kMean, kStale>(p, blockIdx.x, blockIdx.y, wmax);
}

// Longer sequences.  Q, V and the chunk sums of the K mean in one launch: the three need nothing from each other, and as separate launches
// of a few microseconds each they spend a good part of their time filling and draining the GPU.  The grid is the
// concatenation [K-mean chunks | Q blocks | V blocks] (the chunk sums first: the fold and the K quantiser wait for them).
template <int D>
__global__ void __launch_bounds__(128, D == 128 ? 10 : 6) quant_qv_kmean_kernel(const QuantParams pq, const QuantParams pv, const KMeanParams pk) {
  __shared__ float wmax[4];
  __shared__ float red[KMeanTile<D>::kRpp][D];
  grid_dep_wait();
  const int n_km = (pk.N / 64) * pk.B * pk.Hk;
  const int n_q = (pq.N / 32) * pq.B * pq.H;
  int i = static_cast<int>(blockIdx.x);
  if (i < n_km) {
    kmean_block<D>(pk, i % (pk.N / 64), i / (pk.N / 64), red);
  } else if ((i -= n_km) < n_q) {
    quant_block<D, false, false>(pq, i % (pq.N / 32), i / (pq.N / 32), wmax);
  } else {
    i -= n_q;
    quant_block<D, false, false>(pv, i % (pv.N / 32), i / (pv.N / 32), wmax);
  }
}

// K with the fold of its chunk sums: a CTA of four groups of 128 threads folds all columns of its head into shared memory, then
// each group quantises 32 tokens.
template <int D>
__global__ void __launch_bounds__(512, D == 128 ? 2 : 1) quant_k_fold_kernel(const QuantParams p, const KMeanParams pm) {
  __shared__ float mean[D];
  __shared__ float wmax[16];
  grid_dep_wait();
  const int bh = blockIdx.y, group = threadIdx.x / 128;
  if (threadIdx.x < D) {
    mean[threadIdx.x] = kmean_column(pm, bh, threadIdx.x);
    if (blockIdx.x == 0) pm.mean[static_cast<size_t>(bh) * D + threadIdx.x] = mean[threadIdx.x];
  }
  __syncthreads();
  quant_block<D, true, false>(p, 4 * blockIdx.x + group, bh, wmax + 4 * group, threadIdx.x % 128, 1 + group, mean);
}

// Q, K and V of a short sequence in one launch.  A CTA has one group of 128 threads per 64 tokens; the K CTA of a (batch, kv
// head) holds the whole head in registers between the chunk sums, their fold and the quantisation (K is read once), the other
// CTAs take one 32-token block of Q or V per group.  For N / 64 groups of 32 x D / 128 bf16 values a thread: up to
// kShortTokens tokens.  Three launches of one or two microseconds each before (N=256: 6.6 us and three times the host's launch time).
template <int D>
constexpr int kShortTokens = (D == 128) ? 512 : 256;

// The packed values are what stays in registers between the passes over them, not their fp32 forms.
template <int N>
__device__ __forceinline__ void keep_packed(uint4 (&x)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(x[i].x), "+r"(x[i].y), "+r"(x[i].z), "+r"(x[i].w));
}

template <int D>
__device__ __forceinline__ void quant_k_head(const QuantParams& p, float* mean_out, int bh, float* red, float* mean, float* wmax) {
  constexpr int kTpr = D / 8, kRpp = 128 / kTpr, kPass = 64 / kRpp;      // thread layout of the chunk sums (kmean_block)
  const int b = bh / p.H, h = bh % p.H;
  const int group = threadIdx.x / 128, tid = threadIdx.x % 128, n_chunk = p.N / 64;
  const int c8 = tid % kTpr, r0 = tid / kTpr;
  const __nv_bfloat16* base = p.x + b * p.sb + h * p.sh + static_cast<int64_t>(group) * 64 * p.sn + c8 * 8;
  uint4 x[kPass];
#pragma unroll
  for (int i = 0; i < kPass; ++i) x[i] = __ldg(reinterpret_cast<const uint4*>(base + (r0 + i * kRpp) * p.sn));
  {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < kPass; ++i) {
      float f[8];
      bf16x8_to_float(x[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += f[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) red[(group * kRpp + r0) * D + c8 * 8 + j] = acc[j];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += blockDim.x) {      // the sums of the chunks, then their fold, in the order of kmean_block
    float s = 0.f;
    for (int g = 0; g < n_chunk; ++g) {
      float t = red[g * kRpp * D + c];
#pragma unroll
      for (int r = 1; r < kRpp; ++r) t += red[(g * kRpp + r) * D + c];
      s += t;
    }
    s /= static_cast<float>(p.N);
    mean[c] = s;
    mean_out[static_cast<size_t>(bh) * D + c] = s;
  }
  __syncthreads();
  keep_packed(x);
  float m[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) m[j] = mean[c8 * 8 + j];
#pragma unroll
  for (int half = 0; half < 2; ++half) {                   // the two 32-token blocks of the group's chunk
    float amax = 0.f;
#pragma unroll
    for (int i = half * kPass / 2; i < (half + 1) * kPass / 2; ++i) {
      float f[8];
      bf16x8_to_float(x[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf((f[j] - m[j]) * p.prescale));
    }
    amax = warp_max(amax);
    if ((tid & 31) == 0) wmax[group * 8 + half * 4 + (tid >> 5)] = amax;
  }
  bar_sync(1 + group, 128);
  keep_packed(x);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const float* w4 = wmax + group * 8 + half * 4;
    const uint32_t sb = pow2_sb(fmaxf(fmaxf(w4[0], w4[1]), fmaxf(w4[2], w4[3])), 127u);
    const float inv = sb_to_inv(sb);
    if (tid == 0) p.scales[static_cast<size_t>(bh) * (p.N / 32) + group * 2 + half] = sb_to_scale(sb);
#pragma unroll
    for (int i = half * kPass / 2; i < (half + 1) * kPass / 2; ++i) {
      float f[8];
      bf16x8_to_float(x[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = ((f[j] - m[j]) * p.prescale) * inv;
      uint2 w;
      w.x = cvt_e4m3x4(f[0], f[1], f[2], f[3]);
      w.y = cvt_e4m3x4(f[4], f[5], f[6], f[7]);
      *reinterpret_cast<uint2*>(p.codes + (static_cast<size_t>(bh) * p.N + group * 64 + r0 + i * kRpp) * D + c8 * 8) = w;
    }
  }
}

template <int D>
__global__ void __launch_bounds__(kShortTokens<D> * 2) quant_qkv_short_kernel(const QuantParams pq, const QuantParams pk, const QuantParams pv, float* mean_out) {
  constexpr int kGroups = kShortTokens<D> / 64, kRpp = KMeanTile<D>::kRpp;
  __shared__ float red[kGroups * kRpp * D];
  __shared__ float mean[D];
  __shared__ float wmax[kGroups * 8];
  grid_dep_wait();
  const int n_k = pk.B * pk.H, groups = blockDim.x / 128;
  if (static_cast<int>(blockIdx.x) < n_k) {
    quant_k_head<D>(pk, mean_out, blockIdx.x, red, mean, wmax);
    return;
  }
  const int group = threadIdx.x / 128, blocks = pq.N / 32;
  int i = (static_cast<int>(blockIdx.x) - n_k) * groups + group;
  const int n_q = blocks * pq.B * pq.H, n_v = blocks * pv.B * pv.H;
  if (i < n_q) quant_block<D, false, false>(pq, i % blocks, i / blocks, wmax + 4 * group, threadIdx.x % 128, 1 + group);
  else if ((i -= n_q) < n_v) quant_block<D, false, false>(pv, i % blocks, i / blocks, wmax + 4 * group, threadIdx.x % 128, 1 + group);
}

cudaError_t launch_quant_qkv(const QuantParams& pq, const QuantParams& pk, const QuantParams& pv, const KMeanParams& pm,
                             cudaStream_t stream) {
  const int short_tokens = pq.D == 128 ? kShortTokens<128> : kShortTokens<256>;
  if (pm.N <= short_tokens) {
    const int groups = pm.N / 64;                        // 2 .. 8 (N is a multiple of 128)
    const long long qv = static_cast<long long>(pq.N / 32) * (pq.B * pq.H + pv.B * pv.H);
    count_launch();
    return launch_chained(pq.D == 128 ? quant_qkv_short_kernel<128> : quant_qkv_short_kernel<256>,
                          static_cast<unsigned>(pk.B * pk.H + (qv + groups - 1) / groups), groups * 128, 0, stream, pq, pk, pv, pm.mean);
  }
  const long long blocks = static_cast<long long>(pm.N / 64) * pm.B * pm.Hk + static_cast<long long>(pq.N / 32) * pq.B * pq.H +
                           static_cast<long long>(pv.N / 32) * pv.B * pv.H;
  if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
  cudaError_t e = launch_chained(pq.D == 128 ? quant_qv_kmean_kernel<128> : quant_qv_kmean_kernel<256>, static_cast<unsigned>(blocks), 128,
                                 0, stream, pq, pv, pm);
  count_launch();
  if (e != cudaSuccess) return e;
  // Then K, centred.  Every CTA of K folds the chunk sums for itself, which saves the fold's launch, as long as what they read
  // for it together is small (a head's sums, N / 64 rows, once per 128 tokens).  Forward + backward: N=1024 H=8 Hk=2 80.0 -> 77.1 us,
  // N=1920 H=6 Hk=2 D=256 (0.9 MiB) 94.2 -> 91.3; B=3 N=1792 H=15 Hk=5 (2.9 MiB) 203.1 -> 204.2, N=4096 H=32 Hk=8 (8 MiB) 470 -> 473.
  if (static_cast<long long>(pm.B) * pm.Hk * (pm.N / 128) * (pm.N / 64) * pm.D * 4 <= (1ll << 20)) {
    count_launch();
    return launch_chained(pq.D == 128 ? quant_k_fold_kernel<128> : quant_k_fold_kernel<256>, dim3(pm.N / 128, pm.B * pm.Hk), 512, 0, stream, pk, pm);
  }
  e = launch_chained(kmean_fold_kernel, pm.B * pm.Hk, 128, 0, stream, pm);
  count_launch();
  if (e != cudaSuccess) return e;
  return launch_quant(pk, stream);
}

cudaError_t launch_quant(const QuantParams& p, cudaStream_t stream) {
  dim3 grid(p.N / 32, p.B * p.H);
  const bool mean = p.mean != nullptr, stale = p.o != nullptr;
  auto* kernel = p.D == 128 ? (stale ? quant_kernel<128, false, true> : mean ? quant_kernel<128, true, false> : quant_kernel<128, false, false>)
                            : (stale ? quant_kernel<256, false, true> : mean ? quant_kernel<256, true, false> : quant_kernel<256, false, false>);
  count_launch();
  return launch_chained(kernel, grid, 128, 0, stream, p);
}

}  // namespace dm
