// Result delivery: one kernel gathers every array of a result into the final
// layout of the host block and stores it straight into mapped pinned memory.
//
// Bound by the PCIe writes of the packed bytes (about 100 per feature) and, for
// small results, by its launch; an extraction captures it as its graph's last
// node, so a result costs no wait of its own.  The seven copies into pageable
// memory it replaces were staged copies the host waited for: an extraction of
// 533 features (64 x 64 x 10) went from 189 to 109 us per call, one of 5,700
// (128^3 x 16) from 600 to 470 us.
#include <cstdlib>
#include <cstring>

#include "cp_host.h"
#include "cp_pack.cuh"
#include "cp_pdl.cuh"

namespace ftk2b {

namespace {

constexpr int kPackThreads = 256;

__global__ void __launch_bounds__(kPackThreads) pack_kernel(PackArgs a) {
  pdl_enter();
  const unsigned long long t = blockIdx.x * (unsigned long long)kPackThreads + threadIdx.x;
  const unsigned long long nt = (unsigned long long)gridDim.x * kPackThreads;
  if (a.h_counters && t < (unsigned)a.n_counters) a.h_counters[t] = a.counters[t];
  const unsigned n = a.count ? *a.count : a.n;
  const unsigned ne = !a.count ? a.ne : a.n_edges ? *a.n_edges : 0u;
  if (n > a.cap || ne > a.edge_cap) return;
  const PackLayout L = pack_layout(n, ne, a.k, a.classify);
  if (L.packed > a.dst_bytes) return;
  pack_records(a, L, n, t, nt);
  pack_labels(a, L, n, t, nt, [&](unsigned long long i) { return a.track[i]; });
  pack_words<unsigned>(a.dst + L.edges, 2ull * ne, t, nt, [&](unsigned long long i) { return a.edges[i]; });
}

}  // namespace

cudaError_t launch_pack(const PackArgs& a, int num_sms, cudaStream_t st) {
  const cudaError_t e = launch_pdl(pack_kernel, num_sms, kPackThreads, 0, st, a);
  return e ? e : cudaGetLastError();
}

ftk2b_cp_result* new_result(uint64_t n, uint64_t ne, int m, int classify, PackLayout* out) {
  const PackLayout L = pack_layout(n, ne, m + 1, classify);
  unsigned char* b = static_cast<unsigned char*>(host_alloc(kResultHeader + L.total));
  if (!b) return nullptr;
  ftk2b_cp_result* r = reinterpret_cast<ftk2b_cp_result*>(b);
  std::memset(r, 0, sizeof(*r));
  unsigned char* d = b + kResultHeader;
  std::memset(d + L.packed, 0, L.total - L.packed);
  r->m = m;
  r->n_features = n;
  r->n_edges = ne;
  r->lambda = reinterpret_cast<double*>(d + L.lam);
  r->simplices = reinterpret_cast<uint64_t*>(d + L.simplices);
  r->track_id = reinterpret_cast<uint64_t*>(d + L.track);
  r->barycentric = reinterpret_cast<float*>(d + L.bary);
  r->scalar = reinterpret_cast<float*>(d + L.scalar);
  r->edges = reinterpret_cast<uint32_t*>(d + L.edges);
  r->cp_class = reinterpret_cast<uint32_t*>(d + L.cls);
  r->type = reinterpret_cast<uint32_t*>(d + L.type);
  if (out) *out = L;
  return r;
}

}  // namespace ftk2b

// every result is one allocation (new_result)
extern "C" void ftk2b_cp_result_free(ftk2b_cp_result* r) { std::free(r); }
