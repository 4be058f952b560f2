// Delivery of critical-point results to the host: the layout of a result's
// arrays in one block, and the kernel that writes them there.
#pragma once

#include <cstddef>
#include <cstdint>

#include "cp_internal.h"

#include "../../include/ftk2b.h"

namespace ftk2b {

// Byte offsets of a result's arrays in one block of host memory, each on a
// 16-byte boundary.  The pack kernel writes [0, packed); what follows (the
// types, and the classes of an unclassified run) is zero.
struct PackLayout {
  unsigned long long lam, simplices, track, bary, scalar, edges, cls, type;
  unsigned long long packed, total;
};

__host__ __device__ inline PackLayout pack_layout(unsigned long long n, unsigned long long ne, int k, int classify) {
  PackLayout L;
  unsigned long long o = 0;
  auto take = [&o](unsigned long long bytes) {
    const unsigned long long at = o;
    o += (bytes + 15) & ~15ull;
    return at;
  };
  L.lam = take(8 * n * (unsigned)k);
  L.simplices = take(8 * n * (unsigned)k);
  L.track = take(8 * n);
  L.bary = take(4 * n * (unsigned)k);
  L.scalar = take(4 * n);
  L.edges = take(8 * ne);
  if (!classify) L.packed = o;
  L.cls = take(4 * n);
  if (classify) L.packed = o;
  L.type = take(4 * n);
  L.total = o;
  return L;
}

// One run's device results.  The numbers of features and edges are *count and
// *n_edges (0 when null), or n and ne when count is null; when either exceeds
// its capacity, or the block's packed part exceeds dst_bytes, nothing but the
// counters is written (the host sees the same numbers and takes another way).
struct PackArgs {
  const unsigned* counters;            // the run's counters, copied to h_counters
  unsigned* h_counters;                // null: not copied
  int n_counters;
  const unsigned* count;
  const unsigned* n_edges;
  unsigned n, ne;
  unsigned cap, edge_cap;
  int k;                               // vertices per simplex
  int classify, want_edges;
  const double* lam4;                  // rows of 4
  const unsigned long long* simplices; // rows of k
  const float* bary;                   // rows of k
  const float* scalar;
  const unsigned long long* track;
  const unsigned* cls;
  const unsigned* edges;
  unsigned char* dst;                  // mapped pinned host memory, 16-byte aligned
  unsigned long long dst_bytes;
};

cudaError_t launch_pack(const PackArgs& a, int num_sms, cudaStream_t st);

// A result whose arrays follow it in the same allocation (freed as one), laid
// out by pack_layout from kResultHeader on; null when the host is out of memory.
constexpr size_t kResultHeader = (sizeof(ftk2b_cp_result) + 63) & ~size_t(63);
ftk2b_cp_result* new_result(uint64_t n, uint64_t ne, int m, int classify, PackLayout* L);

}  // namespace ftk2b
