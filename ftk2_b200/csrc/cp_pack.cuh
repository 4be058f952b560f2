// Device side of result delivery: the writers of the packed block's arrays
// (pack_layout) that the pack kernel and the short chain's last step share.
#pragma once

#include <cuda_runtime.h>

#include "cp_pack.h"

namespace ftk2b {

// Words [0, n) of an array by threads t of nt: consecutive lanes store
// consecutive words, so a warp's stores leave as whole 128-byte lines.
template <typename W, typename F>
__device__ __forceinline__ void pack_words(unsigned char* dst, unsigned long long n, unsigned long long t,
                                           unsigned long long nt, F word) {
  W* out = reinterpret_cast<W*>(dst);
  for (unsigned long long i = t; i < n; i += nt) out[i] = word(i);
}

// The arrays that neither trajectories nor classes go into.
__device__ __forceinline__ void pack_records(const PackArgs& a, const PackLayout& L, unsigned n, unsigned long long t,
                                             unsigned long long nt) {
  const unsigned k = (unsigned)a.k;
  pack_words<double>(a.dst + L.lam, (unsigned long long)n * k, t, nt,
                     [&](unsigned long long i) { return k == 4 ? a.lam4[i] : a.lam4[i / k * 4 + i % k]; });
  pack_words<unsigned long long>(a.dst + L.simplices, (unsigned long long)n * k, t, nt,
                                 [&](unsigned long long i) { return a.simplices[i]; });
  pack_words<float>(a.dst + L.bary, (unsigned long long)n * k, t, nt, [&](unsigned long long i) { return a.bary[i]; });
  pack_words<float>(a.dst + L.scalar, n, t, nt, [&](unsigned long long i) { return a.scalar[i]; });
}

// Track ids (track(i): feature i's, where the run has edges) and classes.
template <typename F>
__device__ __forceinline__ void pack_labels(const PackArgs& a, const PackLayout& L, unsigned n, unsigned long long t,
                                            unsigned long long nt, F track) {
  pack_words<unsigned long long>(a.dst + L.track, n, t, nt,
                                 [&](unsigned long long i) -> unsigned long long { return a.want_edges ? track(i) : i; });
  if (a.classify) pack_words<unsigned>(a.dst + L.cls, n, t, nt, [&](unsigned long long i) { return a.cls[i]; });
}

}  // namespace ftk2b
