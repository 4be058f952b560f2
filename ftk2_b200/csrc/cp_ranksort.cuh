// Sorting a few thousand keys in one launch: every block copies all keys into
// shared memory and each warp counts, for four keys at a time, the keys below
// them; a key's rank is its place.
//
// n^2 / 128 warp steps in all, each a shared-memory read and four compares a
// lane, so a few thousand keys are bound by the launch.  An LSD radix sort of the same
// keys is three launches per 8 bits, and a 55-bit tuple takes two such sorts.  A
// stream's push, whose window of some 500 features was sorted that way, went
// from 165 to 110 us (96 x 101 x 88 float) and from 880 to 720 us (100 x 100 x 40
// tets); its result from 270 to 102 us (2,200 features).  Larger sets take the
// radix passes.
#pragma once

#include <cuda_runtime.h>

#include "cp_pdl.cuh"

namespace ftk2b {

constexpr int kRankThreads = 512;
// Keys of one word: where a push of that many takes as long by the radix passes
// (2D and 3D noise, by rank / by passes: 12,600 keys 160 / 169 us, 14,800 185 /
// 187, 16,600 191 / 171, 18,600 258 / 181; 231 before there was a rank sort).
constexpr unsigned kRankCap1 = 15360;
// Keys of two words, whose passes are twice as many: what 192 KB hold (a push of
// 12,000 tuples 332 / 454 us).
constexpr unsigned kRankCap2 = 12288;

// How many keys there are: `add`, plus *n where n is not null; none when that is
// more than the launch holds, *gate (not null) is above gate_max, or *err (not
// null) is set, so that a launch may precede the host's look at the counters: a
// step that failed must leave no trace in what the launches behind it update.
struct RankCount {
  unsigned add;
  const unsigned* n = nullptr;
  const unsigned* gate = nullptr;
  unsigned gate_max = 0;
  const unsigned* err = nullptr;
};

// Keys of W 64-bit words, compared word by word, equal keys by index.
//   load(i, k)          writes the W words of key i
//   store(pos, i, k)    called once per key: key i is the pos-th smallest
// for i below the count, which is also written to *n_out when that is not null.
// Shared memory: W * cap words.
template <int W, typename Load, typename Store>
__global__ void __launch_bounds__(kRankThreads, 1)
    rank_sort_kernel(Load load, Store store, RankCount count, unsigned cap, unsigned* n_out) {
  extern __shared__ unsigned long long rank_keys[];
  pdl_enter();
  const unsigned long long all = (unsigned long long)count.add + (count.n ? *count.n : 0u);
  const bool none = all > cap || (count.gate && *count.gate > count.gate_max) || (count.err && *count.err);
  const unsigned n = none ? 0u : (unsigned)all;
  if (n_out && blockIdx.x == 0 && threadIdx.x == 0) *n_out = n;
  if (blockIdx.x * (kRankThreads / 8) >= n) return;  // no key of this block's
  for (unsigned i = threadIdx.x; i < n; i += kRankThreads) {
    unsigned long long k[W];
    load(i, k);
#pragma unroll
    for (int w = 0; w < W; ++w) rank_keys[w * (size_t)cap + i] = k[w];
  }
  __syncthreads();
  constexpr int U = 4;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (unsigned e0 = (blockIdx.x * (kRankThreads / 32) + warp) * U; e0 < n;
       e0 += gridDim.x * (kRankThreads / 32) * U) {
    unsigned long long k[U][W];
    unsigned below[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      below[u] = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) k[u][w] = rank_keys[w * (size_t)cap + min(e0 + u, n - 1)];
    }
    for (unsigned j = lane; j < n; j += 32) {
      unsigned long long x[W];
#pragma unroll
      for (int w = 0; w < W; ++w) x[w] = rank_keys[w * (size_t)cap + j];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        bool less = j < e0 + u;
#pragma unroll
        for (int w = W - 1; w >= 0; --w) less = x[w] < k[u][w] || (x[w] == k[u][w] && less);
        below[u] += less ? 1u : 0u;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned pos = __reduce_add_sync(0xFFFFFFFFu, below[u]);
      if (lane == (unsigned)u && e0 + u < n) store(pos, e0 + u, k[u]);
    }
  }
}

template <int W, typename Load, typename Store>
inline cudaError_t launch_rank_sort(const Load& load, const Store& store, const RankCount& count, unsigned cap,
                                    unsigned* n_out, int num_sms, cudaStream_t st) {
  auto k = rank_sort_kernel<W, Load, Store>;
  const size_t smem = 8 * (size_t)W * (cap ? cap : 1);
  // always the most any call needs: another thread may be launching the same kernel
  constexpr int kMost = 8 * (W == 1 ? kRankCap1 : W * kRankCap2);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
  if (e) return e;
  unsigned grid = (cap + kRankThreads / 8 - 1) / (kRankThreads / 8);
  if (grid > (unsigned)num_sms) grid = (unsigned)num_sms;
  e = launch_pdl(k, grid ? grid : 1, kRankThreads, smem, st, load, store, count, cap, n_out);
  return e ? e : cudaGetLastError();
}

}  // namespace ftk2b
