// Critical-point extraction over an extruded unstructured spacetime mesh:
// ExtrudedSimplicialMesh(UnstructuredSimplicialMesh(cells), n_layers)
// (mesh.hpp:542-730, unstructured_mesh.hpp:12-116) with per-vertex fields
// indexed by vertex id = spatial id + t * n_spatial (engine.hpp:999-1009).
//
// The spacetime mesh has three kinds of m-simplices (m = base cell dim):
//   spatial   every base cell at every time layer t = 0..L
//   lateral   the m Kuhn pieces of the prism over every (m-1)-face of the
//             base between layers t and t+1: f[0..j]@t + f[j..m-1]@t+1
//   interior  the m simplices between consecutive top cells of the prism
//             over a base cell: u[0..s-1]@t + u[s..m]@t+1, s = 1..m
// whose top cells are the m+1 pieces u[0..p]@t + u[p..m]@t+1 of each prism.
// Spatial and lateral simplices are what the reference's phase 1 iterates
// (mesh.hpp:568-599); interior ones it finds while patching (engine.hpp:
// 1352-1367), so they number after all phase-1 nodes.
//
// Pipeline (all on the context's stream):
//   0. base-mesh preparation, cached by content: cells sorted and narrowed to
//      32 bits, every (m-1)-face keyed, radix-sorted, de-duplicated, and the
//      coface cells of each unique face gathered (unstructured_mesh.hpp:44-53)
//   1. cull words of every spacetime vertex: one coalesced pass over the field
//   2. one thread per (base cell, layer): the AND of the prism's vertex words
//      culls all its simplices at once; those of the prisms left are culled by
//      their own words or run the exact integer SoS and the bit-exact solve;
//      accepted simplices are compacted by ballot
//   3. canonical order: one rank sort of the packed vertex tuples, or two stable
//      radix sorts where they are too many for it
//   4. star edges per top cell, centre = smallest node id (phase, then
//      canonical position: engine.hpp:1375-1387 for non-regular meshes)
//   5. union-find over the edges, plus for 4-D meshes the extra coface unions
//      of get_complex (engine.hpp:896-963) as ExtrudedSimplicialMesh::cofaces
//      reports them (mesh.hpp:601-712), then labels = component minimum.
#include <algorithm>
#include <cstring>
#include <vector>

#include "cp_api_internal.h"
#include "cp_host.h"
#include "cp_stream.h"
#include "cp_stream_kernels.cuh"
#include "cp_cull.cuh"
#include "cp_device.cuh"
#include "cp_uf.cuh"

namespace ftk2b {

namespace {

enum { kCountPrepEntries = 5, kCountFaces = 6 };
enum { kErrBadVertex = 4u, kErrCofaces = 8u };

constexpr int kThreadsX = 256;
constexpr int kMaxOthers = 32;  // star partners of one centre: 8 coface cells x 4

struct ExtMeshDev {
  int cd;                            // base cell dim = m = number of components
  unsigned ns;                       // spatial vertices: vertex id = s + t * ns
  unsigned L;                        // time slabs; vertex layers t0..t0+L
  unsigned t0;                       // global layer of the first local layer
  unsigned tflip;                    // storage slot of local layer l = l xor tflip
  int skip_first_spatial;            // 1: no spatial simplices at local layer 0
  unsigned ncell, nface;
  int fbits;                         // bits per base vertex id in a face key
  const unsigned* cells;             // [ncell][cd+1], ascending
  const unsigned long long* fkeys;   // [nface], ascending packed faces
  const unsigned* cof_start;         // [nface+1]
  const unsigned* cof;               // coface cells, grouped by face
  const unsigned* own;               // [ncell], byte r: 1 when the face without vertex r is this cell's to extract
};

struct ExtSink {
  unsigned long long* hi;   // packed v0, v1
  unsigned long long* lo;   // packed v2, v3 (m = 3) or v2 (m = 2)
  unsigned* phase;          // 0 = spatial / lateral, 1 = interior
  double* lam;
  float* bary4;
  float* scalar;
  unsigned* count;
  unsigned cap;
};

__device__ __forceinline__ unsigned long long face_key(const unsigned* w, int n, int fbits) {
  unsigned long long k = 0;
  for (int i = 0; i < n; ++i) k = (k << fbits) | w[i];
  return k;
}

template <int M>
__device__ __forceinline__ void pack_tuple(const unsigned long long* v, int vb, unsigned long long& hi,
                                           unsigned long long& lo) {
  hi = (v[0] << vb) | v[1];
  lo = (M == 3) ? ((v[2] << vb) | v[3]) : v[2];
}

template <int M>
__device__ __forceinline__ void unpack_tuple(unsigned long long hi, unsigned long long lo, int vb,
                                             unsigned long long* v) {
  const unsigned long long mask = (vb >= 64) ? ~0ull : ((1ull << vb) - 1ull);
  v[0] = hi >> vb;
  v[1] = hi & mask;
  if (M == 3) {
    v[2] = lo >> vb;
    v[3] = lo & mask;
  } else {
    v[2] = lo;
  }
}

__device__ __forceinline__ long long find_tuple(const unsigned long long* __restrict__ H,
                                                const unsigned long long* __restrict__ Lo, unsigned n,
                                                unsigned long long h, unsigned long long l) {
  unsigned a = 0, b = n;
  while (a < b) {
    const unsigned mid = (a + b) >> 1;
    const unsigned long long hm = H[mid], lm = Lo[mid];
    if (hm == h && lm == l) return mid;
    if (hm < h || (hm == h && lm < l)) a = mid + 1;
    else b = mid;
  }
  return -1;
}

// ---------------------------------------------------------------------------
// 0. base-mesh preparation

__global__ void ext_prep_cells_kernel(const unsigned long long* __restrict__ cells64, unsigned ncell,
                                      int cd, unsigned ns, int fbits, unsigned* __restrict__ cells,
                                      unsigned long long* __restrict__ fkey, unsigned* __restrict__ fval,
                                      unsigned* counters, unsigned* err) {
  const unsigned nv = (unsigned)cd + 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) counters[kCountPrepEntries] = ncell * nv;
  for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
    unsigned v[4] = {0, 0, 0, 0};
    for (unsigned i = 0; i < nv; ++i) {
      const unsigned long long x = cells64[(size_t)c * nv + i];
      if (x >= ns) atomicOr(err, kErrBadVertex);
      v[i] = x < ns ? (unsigned)x : 0u;
    }
    for (unsigned i = 1; i < nv; ++i)
      for (unsigned j = i; j > 0 && v[j - 1] > v[j]; --j) {
        const unsigned t = v[j];
        v[j] = v[j - 1];
        v[j - 1] = t;
      }
    for (unsigned i = 0; i < nv; ++i) cells[(size_t)c * nv + i] = v[i];
    for (unsigned r = 0; r < nv; ++r) {
      unsigned w[3];
      int k = 0;
      for (unsigned i = 0; i < nv; ++i)
        if (i != r) w[k++] = v[i];
      fkey[(size_t)c * nv + r] = face_key(w, cd, fbits);
      fval[(size_t)c * nv + r] = c * nv + r;
    }
  }
}

__global__ void ext_face_flags_kernel(const unsigned long long* __restrict__ k, unsigned n,
                                      unsigned* __restrict__ flag) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    flag[i] = (i == 0 || k[i] != k[i - 1]) ? 1u : 0u;
}

// pos = exclusive scan of the head flags: entry i belongs to face pos[i]
// (a head) or pos[i] - 1
__global__ void ext_face_build_kernel(const unsigned long long* __restrict__ k,
                                      const unsigned* __restrict__ v, const unsigned* __restrict__ pos,
                                      unsigned n, int cd, unsigned long long* __restrict__ fkeys,
                                      unsigned* __restrict__ cof_start, unsigned* __restrict__ cof,
                                      unsigned char* __restrict__ own) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const bool head = i == 0 || k[i] != k[i - 1];
    const unsigned f = head ? pos[i] : pos[i] - 1;
    if (head) {
      fkeys[f] = k[i];
      cof_start[f] = i;
    }
    if (i == n - 1) cof_start[f + 1] = n;
    const unsigned c = v[i] / (unsigned)(cd + 1);
    cof[i] = c;
    own[4 * (size_t)c + (v[i] - c * (unsigned)(cd + 1))] = head;  // a face is its first coface cell's
  }
}

// ---------------------------------------------------------------------------
// 1. cull words of every spacetime vertex

template <typename T, int M>
__global__ void __launch_bounds__(256) ext_words_kernel(FieldAccess fa, unsigned long long nv,
                                                        unsigned* __restrict__ words) {
  __shared__ unsigned band_tbl[kBandTable];
  fill_band_table<T>(band_tbl, threadIdx.x, blockDim.x);
  __syncthreads();
  const T* c0 = static_cast<const T*>(fa.comp[0]);
  const T* c1 = static_cast<const T*>(fa.comp[1]);
  const T* c2 = static_cast<const T*>(fa.comp[M == 3 ? 2 : 1]);
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < nv;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned h[M];
    h[0] = hi_word<T>(__ldcs(c0 + i));
    h[1] = hi_word<T>(__ldcs(c1 + i));
    if (M == 3) h[M - 1] = hi_word<T>(__ldcs(c2 + i));
    words[i] = vertex_word_hi<T, M>(h, band_tbl);
  }
}

// ---------------------------------------------------------------------------
// 2. per-simplex exact test

template <typename T, int M>
__device__ __forceinline__ bool ext_test(const FieldAccess& fa, const ExtractConfig& cfg,
                                         const unsigned long long* sidx, double lam_out[4],
                                         float bary_out[4], float& sc_out) {
  T vals[M + 1][M];
#pragma unroll
  for (int i = 0; i <= M; ++i)
#pragma unroll
    for (int j = 0; j < M; ++j) {
      vals[i][j] = static_cast<const T*>(fa.comp[j])[sidx[i]];
      if (cfg.fiber) vals[i][j] = fp<T>::sub(vals[i][j], (T)cfg.fthr[j]);  // values[i][j] - thresholds[j]
    }
  bool inside;
  if constexpr (M == 2) inside = sos_inside2<T>(vals, cfg.Q);
  else inside = sos_inside3<T>(vals, cfg.Q);
  if (!inside) return false;
  T lam[M + 1];
  if (!solve_exact<M, T>(vals, lam)) {
    if (!cfg.fiber) return false;
    // FiberPredicate keeps the simplex at the centroid: (T)1.0 / 3.0
#pragma unroll
    for (int i = 0; i <= M; ++i) lam[i] = (T)((double)(T)1.0 / 3.0);
  }
#pragma unroll
  for (int i = 0; i <= M; ++i) {
    lam_out[i] = (double)lam[i];
    bary_out[i] = (float)lam[i];
  }
  if (fa.has_scalar) {
    using F = fp<T>;
    const T* s = static_cast<const T*>(fa.scalar);
    T sc = T(0);
#pragma unroll
    for (int i = 0; i <= M; ++i) sc = F::add(sc, F::mul(lam[i], s[sidx[i]]));
    sc_out = (float)sc;
  }
  if (cfg.refined) {
    double rr[M + 1];
    if (solve_refined<M, T>(vals, rr))
#pragma unroll
      for (int i = 0; i <= M; ++i) lam_out[i] = rr[i];
  }
  return true;
}

// The simplices a prism gives: its lower spatial cell, the M interior ones, M
// pieces over each of its M + 1 faces, and its upper spatial cell.
template <int M>
constexpr int kPrismSlots = 2 + M + M * (M + 1);

// Slot s of a prism: output vertex k is base vertex src(k) of the cell, at the
// upper layer when k > split.  face: the base vertex a lateral piece leaves
// out (M + 1: not lateral).  live: the bit of a cell that asks for the slot.
template <int M>
struct PrismSlot {
  int split, face, live;
  __device__ __forceinline__ explicit PrismSlot(int s) {
    face = M + 1;
    if (s == 0 || s == kPrismSlots<M> - 1) {
      split = s ? -1 : M;
      live = s ? M + 3 : 0;
    } else if (s <= M) {
      split = s - 1;  // u[0..split]@t, u[split+1..M]@t+1
      live = 1;
    } else {
      face = (s - M - 1) / M;
      split = (s - M - 1) % M;  // f[0..split]@t, f[split..M-1]@t+1
      live = 2 + face;
    }
  }
  __device__ __forceinline__ bool interior() const { return live == 1; }
  __device__ __forceinline__ int upper(int k) const { return k > split ? 1 : 0; }
  __device__ __forceinline__ int src(int k) const {
    if (face > M) return k;
    const int f = k - upper(k);
    return f + (f >= face ? 1 : 0);
  }
};

// grid: x over the base cells, y = slab between local layers t and t + 1 (the
// last one also has the upper layer's spatial cells; one layer alone is slab 0
// without a prism).  Values and words of local layer l sit at storage layer
// l xor tflip; vertex ids use the global layer t0 + l.
//
// A thread ANDs the words of its cells' prisms.  What is culled on a superset
// is culled on every simplex of it, so a prism whose AND is culled has no
// simplex to test: a cell costs one 16-byte load and eight gathers instead of
// one pass for the cell, one for its interior and one for each of its faces.
// The few prisms left are listed in shared memory, a thread per simplex of them
// ANDs that simplex's words, and the simplices left after that run the exact
// test in full warps.  A face belongs to its first coface cell (X.own).  Bound
// by the latency of the gathers, so a thread has kCellsPer cells in flight and
// the exact test, rare here, gives up registers (164 unbounded) for three
// blocks an SM.  2.3M tets, one slab, float: 525 us with a thread per cell,
// face and interior, 110 with one 256-cell block an SM, 48 with three, 35 with
// two cells a thread; 364,000 tets, four slabs, double: 253 -> 21 us.
constexpr int kCellsPer = 2;

template <typename T, int M>
__global__ void __launch_bounds__(kThreadsX, 3) ext_extract_kernel(ExtMeshDev X, FieldAccess fa,
                                                                   const unsigned* __restrict__ words,
                                                                   ExtractConfig cfg, ExtSink sink, int vb) {
  constexpr int NS = kPrismSlots<M>, NC = kCellsPer * kThreadsX;
  __shared__ unsigned s_u[M + 1][NC], s_w[2][M + 1][NC];  // listed cells: vertices, words per layer
  __shared__ unsigned short s_live[NC];                   // PrismSlot::live bits
  __shared__ unsigned short s_list[NC * NS];
  __shared__ unsigned s_n[2];  // cells, simplices listed
  const unsigned t = blockIdx.y;
  const bool slab = t < X.L, spatial = !(X.skip_first_spatial && t == 0), top = t + 1 == X.L;
  const unsigned long long bt = (unsigned long long)(X.t0 + t) * X.ns, bt1 = bt + X.ns;
  const unsigned long long st = (unsigned long long)(t ^ X.tflip) * X.ns;
  const unsigned long long st1 = (unsigned long long)((t + 1) ^ X.tflip) * X.ns;
  const unsigned tid = threadIdx.x, lane = tid & 31, below = (1u << lane) - 1;
  for (unsigned long long base = blockIdx.x * (unsigned long long)NC; base < X.ncell;
       base += gridDim.x * (unsigned long long)NC) {
    if (tid < 2) s_n[tid] = 0;
    __syncthreads();
    unsigned u[kCellsPer][M + 1], w[2][kCellsPer][M + 1], live[kCellsPer];
#pragma unroll
    for (int q = 0; q < kCellsPer; ++q) {
      const unsigned long long c = min(base + q * kThreadsX + tid, (unsigned long long)X.ncell - 1);
      if constexpr (M == 3) {
        const uint4 v = *reinterpret_cast<const uint4*>(X.cells + 4 * c);
        u[q][0] = v.x;
        u[q][1] = v.y;
        u[q][2] = v.z;
        u[q][M] = v.w;
      } else {
#pragma unroll
        for (int k = 0; k <= M; ++k) u[q][k] = X.cells[c * (M + 1) + k];
      }
    }
#pragma unroll
    for (int q = 0; q < kCellsPer; ++q)
#pragma unroll
      for (int k = 0; k <= M; ++k) {
        w[0][q][k] = words[st + u[q][k]];
        w[1][q][k] = slab ? words[st1 + u[q][k]] : kAbsent;
      }
#pragma unroll
    for (int q = 0; q < kCellsPer; ++q) {
      const unsigned long long c = base + q * kThreadsX + tid;
      unsigned lo = kAbsent, hi = kAbsent;
#pragma unroll
      for (int k = 0; k <= M; ++k) {
        lo &= w[0][q][k];
        hi &= w[1][q][k];
      }
      live[q] = 0;
      if (c < X.ncell) {
        // the cull words assume an accepted simplex has a successful solve,
        // which fibers do not require
        if (spatial && (cfg.fiber || !word_culled(lo))) live[q] = 1;
        if (slab && (cfg.fiber || !word_culled(lo & hi))) {
          const unsigned own = X.own[c];
          live[q] |= 2;
#pragma unroll
          for (int r = 0; r <= M; ++r) live[q] |= ((own >> (8 * r)) & 1u) << (2 + r);
        }
        if (top && (cfg.fiber || !word_culled(hi))) live[q] |= 1u << (M + 3);
      }
    }
#pragma unroll
    for (int q = 0; q < kCellsPer; ++q) {
      const unsigned ball = __ballot_sync(0xFFFFFFFFu, live[q] != 0);
      if (!ball) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&s_n[0], (unsigned)__popc(ball));
      at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(ball & below);
      if (live[q]) {
        s_live[at] = (unsigned short)live[q];
#pragma unroll
        for (int k = 0; k <= M; ++k) {
          s_u[k][at] = u[q][k];
          s_w[0][k][at] = w[0][q][k];
          s_w[1][k][at] = w[1][q][k];
        }
      }
    }
    __syncthreads();
    const unsigned n_slots = s_n[0] * NS;
    for (unsigned i0 = 0; i0 < n_slots; i0 += kThreadsX) {
      const unsigned i = i0 + tid;
      bool keep = false;
      if (i < n_slots) {
        const unsigned cell = i / NS;
        const PrismSlot<M> p((int)(i % NS));
        if ((s_live[cell] >> p.live) & 1u) {
          unsigned acc = kAbsent;
#pragma unroll
          for (int k = 0; k <= M; ++k) acc &= s_w[p.upper(k)][p.src(k)][cell];
          keep = cfg.fiber || !word_culled(acc);
        }
      }
      const unsigned kb = __ballot_sync(0xFFFFFFFFu, keep);
      if (!kb) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&s_n[1], (unsigned)__popc(kb));
      at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(kb & below);
      if (keep) s_list[at] = (unsigned short)i;
    }
    __syncthreads();
    const unsigned n_list = s_n[1];
    for (unsigned i0 = 0; i0 < n_list; i0 += kThreadsX) {
      const unsigned i = i0 + tid;
      bool acc = false, interior = false;
      unsigned long long vid[M + 1], sidx[M + 1];
      double lam_out[4] = {0, 0, 0, 0};
      float bary_out[4] = {0.f, 0.f, 0.f, 0.f};
      float sc_out = 0.f;
      if (i < n_list) {
        const unsigned e = s_list[i], cell = e / NS;
        const PrismSlot<M> p((int)(e % NS));
        interior = p.interior();
#pragma unroll
        for (int k = 0; k <= M; ++k) {
          const unsigned x = s_u[p.src(k)][cell];
          vid[k] = (p.upper(k) ? bt1 : bt) + x;
          sidx[k] = (p.upper(k) ? st1 : st) + x;
        }
        acc = ext_test<T, M>(fa, cfg, sidx, lam_out, bary_out, sc_out);
      }
      const unsigned ab = __ballot_sync(0xFFFFFFFFu, acc);
      if (!ab) continue;
      unsigned basei = 0;
      if (lane == 0) basei = atomicAdd(sink.count, (unsigned)__popc(ab));
      basei = __shfl_sync(0xFFFFFFFFu, basei, 0);
      const unsigned idx = basei + __popc(ab & below);
      if (acc && idx < sink.cap) {
        unsigned long long hi, lo;
        pack_tuple<M>(vid, vb, hi, lo);
        sink.hi[idx] = hi;
        sink.lo[idx] = lo;
        sink.phase[idx] = interior ? 1u : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sink.lam[4 * (size_t)idx + k] = lam_out[k];
          sink.bary4[4 * (size_t)idx + k] = bary_out[k];
        }
        sink.scalar[idx] = sc_out;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// 3. canonical order

__global__ void ext_gather_by_perm_kernel(const unsigned long long* __restrict__ src,
                                          const unsigned* __restrict__ perm, const unsigned* n_ptr,
                                          unsigned cap, unsigned long long* __restrict__ dst) {
  const unsigned n = min(*n_ptr, cap);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dst[i] = src[perm[i]];
}

// Features in canonical order.
struct ExtSorted {
  unsigned long long *hi, *lo;
  unsigned* phase;
  double* lam;
  float* scalar;
  unsigned long long* simplices;
  float* bary;
  unsigned* parent;
};

// feature p of the extraction is the i-th of the canonical order
template <int M>
__device__ __forceinline__ void ext_finalize(const ExtSink& in, unsigned p, int vb, const ExtSorted& out, unsigned i) {
  const unsigned long long h = in.hi[p], l = in.lo[p];
  out.hi[i] = h;
  out.lo[i] = l;
  out.phase[i] = in.phase[p];
  out.parent[i] = i;
#pragma unroll
  for (int k = 0; k < 4; ++k) out.lam[4 * (size_t)i + k] = in.lam[4 * (size_t)p + k];
  out.scalar[i] = in.scalar[p];
  unsigned long long v[4];
  unpack_tuple<M>(h, l, vb, v);
#pragma unroll
  for (int k = 0; k <= M; ++k) {
    out.simplices[(size_t)i * (M + 1) + k] = v[k];
    out.bary[(size_t)i * (M + 1) + k] = in.bary4[4 * (size_t)p + k];
  }
}

template <int M>
__global__ void ext_finalize_kernel(const unsigned* __restrict__ perm, const unsigned* n_ptr, unsigned cap, int vb,
                                    ExtSink in, ExtSorted out) {
  const unsigned n = min(*n_ptr, cap);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    ext_finalize<M>(in, perm[i], vb, out, i);
}

// ---------------------------------------------------------------------------
// 4. star edges and 5. coface unions

struct ExtFeatures {
  const unsigned long long* hi;
  const unsigned long long* lo;
  const unsigned* phase;
  const unsigned* n_ptr;
  unsigned cap;
  int vb;
};

__global__ void ext_unpack_edges_kernel(const unsigned long long* __restrict__ ekeys, const unsigned* ne_ptr,
                                        unsigned edge_cap, unsigned* __restrict__ edges) {
  const unsigned ne = min(*ne_ptr, edge_cap);
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += gridDim.x * blockDim.x) {
    const unsigned long long k = ekeys[e];
    edges[2 * (size_t)e] = (unsigned)(k >> 32);
    edges[2 * (size_t)e + 1] = (unsigned)k;
  }
}

// Where a set of features' star edges and unions go.
struct ExtStars {
  const unsigned* ids;        // union-find index of each feature (null: the feature's own)
  unsigned* parent;           // initialised
  unsigned long long* ekeys;  // packed (min << 32 | max) feature indices, or
  unsigned* pairs;            // (null: ekeys) pairs of ids, from row `base` on
  unsigned base, cap;         // rows of ekeys or pairs
  unsigned* n_edges;
  unsigned* err;
};

constexpr int kStarLanes = 16;

// The face with key k, searched by a group's 16 lanes (gm): each round keeps a
// sixteenth of the range, so 4.6 million faces take six dependent loads.
__device__ __forceinline__ long long find_face_group(const ExtMeshDev& X, unsigned long long k, unsigned gm,
                                                     unsigned hl, unsigned shift) {
  unsigned lo = 0, len = X.nface;
  while (len > kStarLanes) {
    const unsigned step = (len + kStarLanes - 1) / kStarLanes;
    const bool le = hl * step < len && X.fkeys[lo + hl * step] <= k;
    const unsigned c = __popc(__ballot_sync(gm, le) >> shift & 0xFFFFu);
    if (c == 0) return -1;
    lo += (c - 1) * step;
    len = min(step, len - (c - 1) * step);
  }
  const bool hit = hl < len && X.fkeys[lo + hl] == k;
  const unsigned ball = __ballot_sync(gm, hit) >> shift & 0xFFFFu;
  return ball ? (long long)(lo + __ffs(ball) - 1) : -1;
}

// Star edges and unions of the features: 16 lanes a feature, a lane per face
// of its top cells (three cells of five faces, four of four, at a time).
//
// A feature's top cells: of a spatial simplex (a base cell at layer t) piece m
// of slab t and piece 0 of slab t - 1; of an interior simplex s of the prism
// over a base cell, pieces s - 1 and s; of a lateral piece j over base face f,
// piece j + (e <= j) of the prism over every cell that contains f, e the
// position of the cell's vertex outside f.  The features among a cell's faces
// form a star around the one with the smallest node id (phase, then canonical
// position), which emits the edges.
//
// 4-D meshes: every non-spatial feature is also united with the features among
// the faces of the top cells that ExtrudedSimplicialMesh::cofaces lists for it.
// That routine lifts the base face obtained by dropping the vertex after the
// last layer-t vertex: for a lateral piece that is its own base face (the true
// cofaces); for an interior simplex it is a face of its cell, and the pieces
// of the neighbouring cell across that face join the component as well.
//
// Bound by chains of dependent loads (the face, its cells, the features'
// binary searches).  A thread a feature walked them one after the other, twice
// for the edges and once more for the cofaces: 57 + 54 + 37 us for the 570
// features of a 100 x 100 x 40 tet slab, now 19 for all three.
template <int M>
__global__ void __launch_bounds__(256) ext_stars_kernel(ExtMeshDev X, ExtFeatures Fs, ExtStars out) {
  constexpr int kFaces = M + 2, kCells = kStarLanes / kFaces;
  const unsigned n = min(*Fs.n_ptr, Fs.cap);
  const unsigned lane = threadIdx.x & 31, hl = lane & (kStarLanes - 1), shift = lane & kStarLanes;
  const unsigned gm = 0xFFFFu << shift;
  const unsigned q_lane = hl / kFaces, r = hl % kFaces;  // this lane's cell of the round and the vertex its face leaves out
  const bool used = q_lane < kCells;
  const unsigned first = shift + (used ? q_lane * kFaces : 0u);  // lane of the cell's first face
  const unsigned long long ns = X.ns;
  for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) / kStarLanes; i < n;
       i += gridDim.x * blockDim.x / kStarLanes) {
    unsigned long long v[4];
    unpack_tuple<M>(Fs.hi[i], Fs.lo[i], Fs.vb, v);
    const unsigned long long t = v[0] / ns;
    unsigned sp[M + 1];
    int n_at_t = 0;
#pragma unroll
    for (int k = 0; k <= M; ++k) {
      const unsigned long long tk = v[k] / ns;
      sp[k] = (unsigned)(v[k] - tk * ns);
      n_at_t += tk == t;
    }
    const unsigned id = out.ids ? out.ids[i] : i;
    const bool spatial = n_at_t == M + 1;
    const int j = n_at_t - 1;
    bool lateral = false;
#pragma unroll
    for (int k = 0; k < M; ++k) lateral |= !spatial && k == j && sp[k] == sp[k + 1];
    // base face without the vertex after the last layer-t one
    unsigned f[M];
    long long fi = -1;
    if (!spatial && (lateral || M == 3)) {
#pragma unroll
      for (int k = 0; k < M; ++k) f[k] = k <= j ? sp[k] : sp[k + 1];
      fi = find_face_group(X, face_key(f, M, X.fbits), gm, hl, shift);
    }
    unsigned others = 0;
    // star: the feature's own top cells; the second pass (interior simplices
    // of 4-D meshes): the lifted face's
    for (int pass = 0; pass < 2; ++pass) {
      const bool over_face = pass ? M == 3 && !spatial && !lateral : lateral;
      if (pass && !over_face) break;
      const bool star = pass == 0;
      const bool unite_all = M == 3 && (pass || lateral);
      const unsigned q0 = over_face ? (fi < 0 ? 0u : X.cof_start[fi]) : 0u;
      const unsigned nq = over_face ? (fi < 0 ? 0u : X.cof_start[fi + 1] - q0) : 2u;
      for (unsigned qb = 0; qb < nq; qb += kCells) {
        const unsigned q = qb + q_lane;
        bool valid = used && q < nq;
        unsigned u[M + 1];
        unsigned long long tt = t;
        int p = 0;
#pragma unroll
        for (int k = 0; k <= M; ++k) u[k] = sp[k];
        if (valid && over_face) {
          const unsigned* cell = X.cells + (size_t)X.cof[q0 + q] * (M + 1);
          int e = -1, wi = 0;
#pragma unroll
          for (int k = 0; k <= M; ++k) {
            u[k] = cell[k];
            const unsigned fw = wi == 0 ? f[0] : wi == 1 ? f[1] : f[M - 1];
            if (wi < M && u[k] == fw) ++wi;
            else e = k;
          }
          valid = e >= 0;
          p = j + (e <= j ? 1 : 0);
        } else if (spatial) {
          p = q ? 0 : M;
          tt = q ? t - 1 : t;
          valid = valid && (q ? t > X.t0 : t < (unsigned long long)X.t0 + X.L);
        } else {
          p = j + (int)q;
        }
        // the cell u[0..p]@tt, u[p..M]@tt+1 without its vertex r
        long long idx = -1;
        if (valid) {
          unsigned long long face[M + 1];
#pragma unroll
          for (int k = 0; k <= M; ++k) {
            const unsigned long long a = k <= p ? tt * ns + u[k] : (tt + 1) * ns + u[k ? k - 1 : 0];
            const unsigned long long b = k + 1 <= p ? tt * ns + u[k < M ? k + 1 : M] : (tt + 1) * ns + u[k];
            face[k] = k < (int)r ? a : b;
          }
          unsigned long long h, l;
          pack_tuple<M>(face, Fs.vb, h, l);
          idx = find_tuple(Fs.hi, Fs.lo, n, h, l);
        }
        bool emit = false;
        if (star) {
          const unsigned long long node =
              idx >= 0 ? ((unsigned long long)Fs.phase[idx] << 32) | (unsigned long long)idx : ~0ull;
          unsigned long long centre = ~0ull;
#pragma unroll
          for (int k = 0; k < kFaces; ++k) {
            const unsigned long long o = __shfl_sync(gm, node, first + k);
            if (o < centre) centre = o;
          }
          emit = idx >= 0 && (unsigned)centre == i && idx != (long long)i;
        }
        const unsigned ball = __ballot_sync(gm, emit) >> shift & 0xFFFFu;
        if (ball) {
          others += __popc(ball);
          unsigned at = 0;
          if (hl == 0) at = atomicAdd(out.n_edges, (unsigned)__popc(ball));
          at = __shfl_sync(gm, at, shift) + __popc(ball & ((1u << hl) - 1));
          if (emit) {
            const unsigned x = (unsigned)idx, lo = min(x, i), hi = max(x, i);
            if (!out.pairs) {
              if (at < out.cap) out.ekeys[at] = ((unsigned long long)lo << 32) | hi;
            } else if (at < out.cap - out.base) {
              out.pairs[2 * (size_t)(out.base + at)] = out.ids ? out.ids[lo] : lo;
              out.pairs[2 * (size_t)(out.base + at) + 1] = out.ids ? out.ids[hi] : hi;
            }
          }
        }
        if (idx >= 0 && (emit || unite_all))
          uf_unite(out.parent, id, out.ids ? out.ids[idx] : (unsigned)idx, out.err);
        __syncwarp(gm);
      }
    }
    if (others > kMaxOthers && hl == 0) atomicOr(out.err, kErrCofaces);
  }
}

// ---------------------------------------------------------------------------
// host side

int bits_of(unsigned long long v) {
  int b = 0;
  while (b < 64 && (v >> b) != 0) ++b;
  return b < 1 ? 1 : b;
}

int grid_of(unsigned long long n, int threads, int max_blocks) {
  unsigned long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > (unsigned long long)max_blocks) b = max_blocks;
  return (int)b;
}

ftk2b_status ext_fail(ftk2b_ctx* ctx, ftk2b_status st, const std::string& msg) {
  ctx->err = msg;
  return st;
}

#define EXT_TRY(call)                                                                              \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess)                                                                         \
      return ext_fail(ctx, e_ == cudaErrorMemoryAllocation ? FTK2B_OOM : FTK2B_CUDA_ERROR,          \
                      std::string(#call) + " failed: " + cudaGetErrorString(e_));                  \
  } while (0)

ftk2b_status validate_mesh(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, int* fbits) {
  const int cd = mesh->base_cell_dim;
  if (cd != 2 && cd != 3)
    return ext_fail(ctx, FTK2B_UNSUPPORTED, "extruded meshes need triangle (2) or tet (3) base cells");
  if (mesh->n_base_verts < 1) return ext_fail(ctx, FTK2B_INVALID_ARG, "extruded mesh without base vertices");
  if (mesh->n_base_cells > 0 && !mesh->base_cells)
    return ext_fail(ctx, FTK2B_INVALID_ARG, "base_cells is null");
  if (mesh->n_base_cells * (uint64_t)(cd + 1) >= (1ull << 31))
    return ext_fail(ctx, FTK2B_UNSUPPORTED, "more than 2^31 base cell vertices");
  if (mesh->n_layers >= 65535) return ext_fail(ctx, FTK2B_UNSUPPORTED, "n_layers must be below 65535");
  if (mesh->n_base_verts * (mesh->n_layers + 1) > 0xFFFFFFFFull)
    return ext_fail(ctx, FTK2B_UNSUPPORTED, "spacetime vertex ids exceed 32 bits");
  *fbits = bits_of(mesh->n_base_verts - 1);
  if (*fbits * cd > 64)
    return ext_fail(ctx, FTK2B_UNSUPPORTED, "base vertex ids too wide to pack a face into 64 bits");
  return FTK2B_OK;
}

// Builds (or reuses) the device copy of the base mesh.
ftk2b_status prepare_base(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, int fbits, unsigned long long* nl,
                          const uint64_t* known_hash = nullptr) {
  ExtCache& C = ctx->ext;
  const int cd = mesh->base_cell_dim;
  const uint64_t nent64 = mesh->n_base_cells * (uint64_t)(cd + 1);
  const uint64_t h = known_hash ? *known_hash : hash_words(mesh->base_cells, nent64);
  if (C.valid && C.hash == h && C.ncell == mesh->n_base_cells && C.ns == mesh->n_base_verts && C.cd == cd)
    return FTK2B_OK;
  C.valid = false;
  const unsigned nent = (unsigned)nent64;
  const unsigned ncell = (unsigned)mesh->n_base_cells;
  const size_t ne = nent ? nent : 1;
  EXT_TRY(C.cells.ensure(sizeof(unsigned) * ne));
  EXT_TRY(C.fkeys.ensure(sizeof(unsigned long long) * ne));
  EXT_TRY(C.cof_start.ensure(sizeof(unsigned) * (ne + 1)));
  EXT_TRY(C.cof.ensure(sizeof(unsigned) * ne));
  EXT_TRY(C.own.ensure(sizeof(unsigned) * (ncell ? ncell : 1)));
  EXT_TRY(C.ekeys.ensure(sizeof(unsigned long long) * ne));
  EXT_TRY(C.sort_k.ensure(sizeof(unsigned long long) * ne));
  EXT_TRY(C.sort_k2.ensure(sizeof(unsigned long long) * ne));
  EXT_TRY(C.sort_v.ensure(sizeof(unsigned) * ne));
  EXT_TRY(C.sort_v2.ensure(sizeof(unsigned) * ne));
  EXT_TRY(ctx->counters.ensure(sizeof(unsigned) * kNumCounters));
  const int sgrid = ctx->sort_grid(nent);
  EXT_TRY(ctx->hist.ensure(sizeof(unsigned) * 256 * (size_t)(sgrid > 1 ? sgrid : 1) + 1024));
  cudaStream_t st = ctx->stream;
  unsigned* counters = (unsigned*)ctx->counters.p;
  EXT_TRY(cudaMemsetAsync(counters, 0, sizeof(unsigned) * kNumCounters, st));
  unsigned nface = 0;
  if (nent) {
    EXT_TRY(cudaMemcpyAsync(C.ekeys.p, mesh->base_cells, sizeof(uint64_t) * nent, cudaMemcpyHostToDevice, st));
    ext_prep_cells_kernel<<<grid_of(ncell, 256, 8 * ctx->num_sms), 256, 0, st>>>(
        (const unsigned long long*)C.ekeys.p, ncell, cd, (unsigned)mesh->n_base_verts, fbits,
        (unsigned*)C.cells.p, (unsigned long long*)C.sort_k.p, (unsigned*)C.sort_v.p, counters,
        counters + kCountErr);
    *nl += 1;
    const bool alt = radix_sort((unsigned long long*)C.sort_k.p, (unsigned*)C.sort_v.p,
                                (unsigned long long*)C.sort_k2.p, (unsigned*)C.sort_v2.p,
                                counters + kCountPrepEntries, nent, fbits * cd, (unsigned*)ctx->hist.p,
                                sgrid, st, nl);
    const unsigned long long* k = (const unsigned long long*)(alt ? C.sort_k2.p : C.sort_k.p);
    const unsigned* v = (const unsigned*)(alt ? C.sort_v2.p : C.sort_v.p);
    unsigned* flags = (unsigned*)(alt ? C.sort_v.p : C.sort_v2.p);
    const int g = grid_of(nent, 256, 16 * ctx->num_sms);
    ext_face_flags_kernel<<<g, 256, 0, st>>>(k, nent, flags);
    EXT_TRY(launch_scan(flags, nent, counters + kCountFaces, nullptr, st));
    ext_face_build_kernel<<<g, 256, 0, st>>>(k, v, flags, nent, cd, (unsigned long long*)C.fkeys.p,
                                             (unsigned*)C.cof_start.p, (unsigned*)C.cof.p,
                                             (unsigned char*)C.own.p);
    *nl += 3;
    EXT_TRY(cudaGetLastError());
    EXT_TRY(cudaMemcpyAsync(ctx->h_counters, counters, sizeof(unsigned) * kNumCounters,
                            cudaMemcpyDeviceToHost, st));
    EXT_TRY(ctx->sync());
    if (ctx->h_counters[kCountErr] & kErrBadVertex)
      return ext_fail(ctx, FTK2B_INVALID_ARG, "a base cell lists a vertex id >= n_base_verts");
    nface = ctx->h_counters[kCountFaces];
  }
  C.hash = h;
  C.ncell = mesh->n_base_cells;
  C.ns = mesh->n_base_verts;
  C.cd = cd;
  C.nface = nface;
  C.fbits = fbits;
  C.valid = true;
  return FTK2B_OK;
}

template <typename T, int M>
cudaError_t enqueue_extract(ftk2b_ctx* ctx, const ExtMeshDev& X, const FieldAccess& fa,
                            const ExtractConfig& cfg, const ExtSink& sink, int vb, unsigned long long nv,
                            unsigned long long* nl) {
  cudaStream_t st = ctx->stream;
  ext_words_kernel<T, M><<<grid_of(nv, 256, 32 * ctx->num_sms), 256, 0, st>>>(fa, nv,
                                                                              (unsigned*)ctx->ext.words.p);
  const dim3 grid((unsigned)grid_of(X.ncell, kCellsPer * kThreadsX, 1 << 20), std::max(X.L, 1u));
  ext_extract_kernel<T, M><<<grid, kThreadsX, 0, st>>>(X, fa, (const unsigned*)ctx->ext.words.p, cfg, sink, vb);
  *nl += 2;
  return cudaGetLastError();
}

// The packed edges of C.ekeys in order to the context's edges, any number of them.
cudaError_t sort_edges(ftk2b_ctx* ctx, unsigned edge_cap, unsigned long long* nl) {
  ExtCache& C = ctx->ext;
  const unsigned* n_edges = (const unsigned*)ctx->counters.p + kCountEdges;
  const bool alt = radix_sort((unsigned long long*)C.ekeys.p, (unsigned*)C.sort_v.p, (unsigned long long*)C.sort_k2.p,
                              (unsigned*)C.sort_v2.p, n_edges, edge_cap, 64, (unsigned*)ctx->hist.p,
                              ctx->sort_grid(edge_cap), ctx->stream, nl);
  ext_unpack_edges_kernel<<<grid_of(edge_cap, 256, 4096), 256, 0, ctx->stream>>>(
      (const unsigned long long*)(alt ? C.sort_k2.p : C.ekeys.p), n_edges, edge_cap, (unsigned*)ctx->edges.p);
  *nl += 1;
  return cudaGetLastError();
}

// The features of one extraction in canonical order by one rank sort of their
// tuples (cp_ranksort.cuh); each also becomes a component of its own.
struct LoadFound {
  const unsigned long long *hi, *lo;
  __device__ __forceinline__ void operator()(unsigned i, unsigned long long (&k)[2]) const {
    k[0] = hi[i];
    k[1] = lo[i];
  }
};
template <int M>
struct StoreFound {
  ExtSink in;
  ExtSorted out;
  int vb;
  __device__ __forceinline__ void operator()(unsigned pos, unsigned i, const unsigned long long (&)[2]) const {
    ext_finalize<M>(in, i, vb, out, pos);
  }
};
// their star edges in order
struct LoadEdgeKey {
  const unsigned long long* key;
  __device__ __forceinline__ void operator()(unsigned e, unsigned long long (&k)[1]) const { k[0] = key[e]; }
};

// Canonical order, star edges, trajectories.  n: the features found (at most
// cap).  Sets kCountEdges and kCountRoots; *edges_ranked says whether the edges
// were sorted by one launch that holds for up to kRankCap1 of them.
template <int M>
cudaError_t enqueue_post(ftk2b_ctx* ctx, const ExtMeshDev& X, const ExtSink& sink, unsigned n, unsigned cap,
                         unsigned edge_cap, int vb, int want_edges, bool* edges_ranked, unsigned long long* nl) {
  cudaStream_t st = ctx->stream;
  ExtCache& C = ctx->ext;
  unsigned* counters = (unsigned*)ctx->counters.p;
  unsigned* count = counters + kCountFeatures;
  cudaError_t e;
  const ExtSorted out{(unsigned long long*)C.hi_s.p, (unsigned long long*)C.lo_s.p, (unsigned*)C.phase_s.p,
                      (double*)ctx->lam_s.p, (float*)ctx->scalar_s.p, (unsigned long long*)ctx->simplices.p,
                      (float*)ctx->bary.p, (unsigned*)ctx->parent.p};
  const bool ranked = n <= kRankCap2;
  *edges_ranked = ranked;
  if (ranked) {
    const LoadFound ld{sink.hi, sink.lo};
    const StoreFound<M> sw{sink, out, vb};
    if ((e = launch_rank_sort<2>(ld, sw, RankCount{n}, n ? n : 1, nullptr, ctx->num_sms, st))) return e;
    *nl += 1;
  } else {
    const int sgrid = ctx->sort_grid(cap);
    unsigned* hist = (unsigned*)ctx->hist.p;
    const int g = grid_of(n, 256, 4096);
    // stable sort by the low word, then by the high word
    if ((e = cudaMemcpyAsync(C.sort_k.p, sink.lo, sizeof(unsigned long long) * n, cudaMemcpyDeviceToDevice, st)))
      return e;
    if ((e = launch_iota((unsigned*)ctx->perm0.p, count, n, st))) return e;
    const int lo_bits = (M == 3) ? 2 * vb : vb;
    bool alt = radix_sort((unsigned long long*)C.sort_k.p, (unsigned*)ctx->perm0.p,
                          (unsigned long long*)C.sort_k2.p, (unsigned*)ctx->perm1.p, count, cap, lo_bits,
                          hist, sgrid, st, nl);
    unsigned* p1 = (unsigned*)(alt ? ctx->perm1.p : ctx->perm0.p);
    unsigned* p1_other = (unsigned*)(alt ? ctx->perm0.p : ctx->perm1.p);
    ext_gather_by_perm_kernel<<<g, 256, 0, st>>>(sink.hi, p1, count, cap, (unsigned long long*)C.sort_k.p);
    alt = radix_sort((unsigned long long*)C.sort_k.p, p1, (unsigned long long*)C.sort_k2.p, p1_other, count, cap,
                     2 * vb, hist, sgrid, st, nl);
    const unsigned* perm = alt ? p1_other : p1;
    ext_finalize_kernel<M><<<g, 256, 0, st>>>(perm, count, cap, vb, sink, out);
    *nl += 3;  // iota, gather, finalize
  }
  if (!want_edges) return cudaGetLastError();
  const ExtFeatures Fs{out.hi, out.lo, out.phase, count, cap, vb};
  const ExtStars stars{nullptr, out.parent, (unsigned long long*)C.ekeys.p, nullptr, 0u, edge_cap,
                       counters + kCountEdges, counters + kCountErr};
  ext_stars_kernel<M><<<grid_of(kStarLanes * (unsigned long long)n, 256, 4096), 256, 0, st>>>(X, Fs, stars);
  // (min, max) pairs sorted lexicographically; a pair spans exactly one top
  // cell, so there are no duplicates
  if (ranked) {
    const LoadEdgeKey ld{(const unsigned long long*)C.ekeys.p};
    const StoreEdge so{(unsigned*)ctx->edges.p};
    if ((e = launch_rank_sort<1>(ld, so, RankCount{0, counters + kCountEdges}, std::min(edge_cap, kRankCap1), nullptr,
                                 ctx->num_sms, st)))
      return e;
    *nl += 1;
  } else if ((e = sort_edges(ctx, edge_cap, nl))) {
    return e;
  }
  if ((e = launch_uf_label(out.parent, count, n ? n : 1, (unsigned long long*)ctx->track.p, counters + kCountRoots,
                           st)))
    return e;
  *nl += 2;
  return cudaGetLastError();
}

}  // namespace

}  // namespace ftk2b

using namespace ftk2b;

// ---------------------------------------------------------------------------
// extruded time streams (the driver and its contract: cp_stream.cu)

namespace ftk2b {
namespace {

enum { kSWin = 5, kSWinEdges = 6, kSPrev = 7 };
constexpr int kStreamVb = 32;  // fixed id width of a stream's packed tuples

__global__ void ext_window_build_kernel(const unsigned long long* __restrict__ lo, const unsigned* __restrict__ prev,
                                        unsigned n_prev, unsigned first_new, unsigned n_new,
                                        unsigned long long* __restrict__ k_out, unsigned* __restrict__ id_out) {
  const unsigned nS = n_prev + n_new;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < nS; i += gridDim.x * blockDim.x) {
    const unsigned id = i < n_prev ? prev[i] : first_new + (i - n_prev);
    k_out[i] = lo[id];
    id_out[i] = id;
  }
}

__global__ void ext_gather_key_kernel(const unsigned long long* __restrict__ src, const unsigned* __restrict__ ids,
                                      const unsigned* n_ptr, unsigned cap, unsigned long long* __restrict__ dst) {
  const unsigned n = min(*n_ptr, cap);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[ids[i]];
}

__global__ void ext_window_fill_kernel(const unsigned* __restrict__ ids, const unsigned* n_ptr, unsigned cap,
                                       const unsigned long long* __restrict__ hi,
                                       const unsigned long long* __restrict__ lo, const unsigned* __restrict__ phase,
                                       unsigned long long* __restrict__ hi_s, unsigned long long* __restrict__ lo_s,
                                       unsigned* __restrict__ phase_s) {
  const unsigned n = min(*n_ptr, cap);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned id = ids[i];
    hi_s[i] = hi[id];
    lo_s[i] = lo[id];
    phase_s[i] = phase[id];
  }
}

// The window in Simplex order by one rank sort of its tuples (cp_ranksort.cuh):
// the spatial features of the previous layer, then the new ones, which also
// become components of their own and, when they lie in the newest layer, go
// to its list.
struct LoadTuple {
  const unsigned long long *hi, *lo;
  const unsigned* prev;  // null: ids 0, 1, ..
  unsigned n_prev, first_new;
  __device__ __forceinline__ unsigned id(unsigned i) const {
    return i < n_prev ? prev[i] : first_new + (i - n_prev);
  }
  __device__ __forceinline__ void operator()(unsigned i, unsigned long long (&k)[2]) const {
    const unsigned j = id(i);
    k[0] = hi[j];
    k[1] = lo[j];
  }
};
template <int M>
struct StoreTuple {
  LoadTuple in;
  unsigned long long *hi_s, *lo_s;
  const unsigned* phase;
  unsigned *phase_s, *ids;
  unsigned* parent;
  unsigned *newest, *n_newest;
  unsigned long long ns, t;
  __device__ __forceinline__ void operator()(unsigned pos, unsigned i, const unsigned long long (&k)[2]) const {
    const unsigned id = in.id(i);
    hi_s[pos] = k[0];
    lo_s[pos] = k[1];
    phase_s[pos] = phase[id];
    ids[pos] = id;
    if (i < in.n_prev) return;
    parent[id] = id;
    unsigned long long v[4];
    unpack_tuple<M>(k[0], k[1], kStreamVb, v);
    if (v[0] / ns == t && v[M] / ns == t) newest[atomicAdd(n_newest, 1u)] = id;
  }
};
struct StoreTupleOrder {
  StoreOrder order;
  __device__ __forceinline__ void operator()(unsigned pos, unsigned i, const unsigned long long (&)[2]) const {
    order.put(pos, i);
  }
};

template <int M>
__global__ void ext_collect_spatial_kernel(const unsigned long long* __restrict__ hi,
                                           const unsigned long long* __restrict__ lo, unsigned first_new,
                                           unsigned n_new, unsigned long long ns, unsigned long long t,
                                           unsigned* __restrict__ prev, unsigned* prev_n) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n_new; i += gridDim.x * blockDim.x) {
    const unsigned id = first_new + i;
    unsigned long long v[4];
    unpack_tuple<M>(hi[id], lo[id], kStreamVb, v);
    if (v[0] / ns == t && v[M] / ns == t) prev[atomicAdd(prev_n, 1u)] = id;
  }
}

template <int M>
__global__ void ext_stream_expand_kernel(const unsigned* __restrict__ perm, unsigned n,
                                         const unsigned long long* __restrict__ hi,
                                         const unsigned long long* __restrict__ lo, const float* __restrict__ bary4_s,
                                         unsigned long long* __restrict__ simplices, float* __restrict__ bary) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned p = perm[i];
    unsigned long long v[4];
    unpack_tuple<M>(hi[p], lo[p], kStreamVb, v);
    for (int k = 0; k <= M; ++k) {
      simplices[(size_t)i * (M + 1) + k] = v[k];
      bary[(size_t)i * (M + 1) + k] = bary4_s[4 * (size_t)i + k];
    }
  }
}

ExtMeshDev stream_mesh(ftk2b_ctx* ctx, const ftk2b_stream* s, unsigned t0, unsigned L) {
  ExtCache& C = ctx->ext;
  ExtMeshDev X;
  X.cd = s->m;
  X.ns = (unsigned)s->emesh.n_base_verts;
  X.L = L;
  X.t0 = t0;
  X.tflip = t0 & 1u;
  X.skip_first_spatial = 0;
  X.ncell = (unsigned)C.ncell;
  X.nface = C.nface;
  X.fbits = C.fbits;
  X.cells = (const unsigned*)C.cells.p;
  X.fkeys = (const unsigned long long*)C.fkeys.p;
  X.cof_start = (const unsigned*)C.cof_start.p;
  X.cof = (const unsigned*)C.cof.p;
  X.own = (const unsigned*)C.own.p;
  return X;
}

// sorts ids [0, n) (in k0/v0 order of the window or store) by (hi, lo);
// returns the buffer holding the sorted ids
unsigned* sort_by_tuple(ftk2b_ctx* ctx, ftk2b_stream* s, const unsigned* n_ptr, unsigned cap, int bits,
                        unsigned long long* nl) {
  cudaStream_t st = ctx->stream;
  const int sgrid = ctx->sort_grid(cap);
  unsigned* hist = (unsigned*)ctx->hist.p;
  bool alt = radix_sort((unsigned long long*)s->s_key.p, (unsigned*)s->s_id.p, (unsigned long long*)s->s_key2.p,
                        (unsigned*)s->s_id2.p, n_ptr, cap, bits, hist, sgrid, st, nl);
  unsigned* ids = (unsigned*)(alt ? s->s_id2.p : s->s_id.p);
  unsigned* ids_other = (unsigned*)(alt ? s->s_id.p : s->s_id2.p);
  unsigned long long* kfree = (unsigned long long*)(alt ? s->s_key.p : s->s_key2.p);
  unsigned long long* kother = (unsigned long long*)(alt ? s->s_key2.p : s->s_key.p);
  ext_gather_key_kernel<<<grid_of(cap, 256, 4096), 256, 0, st>>>((const unsigned long long*)s->hi.p, ids, n_ptr, cap,
                                                                 kfree);
  alt = radix_sort(kfree, ids, kother, ids_other, n_ptr, cap, bits, hist, sgrid, st, nl);
  *nl += 1;
  return alt ? ids_other : ids;
}

template <typename T, int M>
ftk2b_status push_extruded_t(ftk2b_stream* s) {
  ftk2b_ctx* ctx = s->ctx;
  cudaStream_t st = ctx->stream;
  unsigned long long nl = 0;
  int fbits = 0;
  ftk2b_status rc = validate_mesh(ctx, &s->emesh, &fbits);
  if (rc) return rc;
  const uint64_t tnow = s->T;
  const unsigned long long ns = s->emesh.n_base_verts;
  if (ns * (tnow + 1) > 0xFFFFFFFFull) return ext_fail(ctx, FTK2B_UNSUPPORTED, "spacetime vertex ids exceed 32 bits");
  rc = prepare_base(ctx, &s->emesh, fbits, &nl, &s->ebase_hash);
  if (rc) return rc;
  if (nl) s->counters_clear = false;  // the preparation counts too
  const unsigned t0 = tnow ? (unsigned)(tnow - 1) : 0u, L = tnow ? 1u : 0u;
  ExtMeshDev X = stream_mesh(ctx, s, t0, L);
  X.skip_first_spatial = tnow > 0;
  FieldAccess fa;
  memset(&fa, 0, sizeof(fa));
  fa.per_vertex = 1;
  for (int j = 0; j < M; ++j) fa.comp[j] = s->ring[j].p;
  ExtractConfig cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.Q = s->prm.sos_q;
  cfg.refined = s->prm.precision == FTK2B_PRECISION_REFINED;
  const unsigned long long nv = ns * (L + 1);
  ExtCache& C = ctx->ext;
  EXT_TRY(C.words.ensure(sizeof(unsigned) * nv));
  EXT_TRY(ctx->counters.ensure(sizeof(unsigned) * kNumCounters));
  unsigned* counters = (unsigned*)ctx->counters.p;
  unsigned n_new = 0;
  // window: spatial features of layer t-1 plus the new ones, in Simplex order;
  // it goes ahead of the host's look at the counters as in regular streams
  const unsigned first_new = s->n;
  const unsigned* ids = nullptr;
  auto room = [&](unsigned wcap) -> ftk2b_status {
    EXT_TRY(s->s_id.ensure(4 * (size_t)wcap));
    EXT_TRY(s->s_hi.ensure(8 * (size_t)wcap));
    EXT_TRY(s->s_lo.ensure(8 * (size_t)wcap));
    EXT_TRY(s->s_phase.ensure(4 * (size_t)wcap));
    return ensure_stream_edges(s, (unsigned long long)kMaxOthers * wcap);
  };
  auto window = [&](const RankCount& count, unsigned wcap) -> cudaError_t {
    const LoadTuple ld{(const unsigned long long*)s->hi.p, (const unsigned long long*)s->lo.p,
                       (const unsigned*)s->prev_ids.p, s->n_prev, first_new};
    const StoreTuple<M> sw{ld, (unsigned long long*)s->s_hi.p, (unsigned long long*)s->s_lo.p,
                           (const unsigned*)s->phase.p, (unsigned*)s->s_phase.p, (unsigned*)s->s_id.p,
                           (unsigned*)s->parent.p, (unsigned*)s->prev_ids2.p, counters + kSPrev, ns, tnow};
    ids = sw.ids;
    nl += 1;
    return launch_rank_sort<2>(ld, sw, count, wcap, counters + kSWin, ctx->num_sms, st);
  };
  auto stars = [&](unsigned wcap) -> cudaError_t {
    const ExtFeatures Fs{(const unsigned long long*)s->s_hi.p, (const unsigned long long*)s->s_lo.p,
                         (const unsigned*)s->s_phase.p, counters + kSWin, wcap, kStreamVb};
    const ExtStars to{ids, (unsigned*)s->parent.p, nullptr, (unsigned*)s->edges.p, s->n_edges, s->edge_cap,
                      counters + kSWinEdges, counters + kCountErr};
    ext_stars_kernel<M><<<grid_of(kStarLanes * (unsigned long long)wcap, 256, 4096), 256, 0, st>>>(X, Fs, to);
    nl += 1;
    return cudaGetLastError();
  };
  const unsigned guess = window_guess(s, kRankCap2);
  if (guess) {
    rc = room(guess);
    if (rc) return rc;
  }
  for (int attempt = 0;; ++attempt) {
    if (attempt == 6) return ext_fail(ctx, FTK2B_OVERFLOW_RETRY, "stream buffers kept overflowing");
    if (s->cap < s->n + 1024) {
      rc = ensure_stream_store(s, s->n + 1024);
      if (rc) return rc;
    }
    if (!s->counters_clear) EXT_TRY(cudaMemsetAsync(counters, 0, sizeof(unsigned) * kNumCounters, st));
    s->counters_clear = false;
    ExtSink sink;
    sink.hi = (unsigned long long*)s->hi.p + s->n;
    sink.lo = (unsigned long long*)s->lo.p + s->n;
    sink.phase = (unsigned*)s->phase.p + s->n;
    sink.lam = (double*)s->lam.p + 4 * (size_t)s->n;
    sink.bary4 = (float*)s->bary4.p + 4 * (size_t)s->n;
    sink.scalar = (float*)s->scalar.p + s->n;
    sink.count = counters + kCountFeatures;
    sink.cap = s->cap - s->n;
    EXT_TRY((enqueue_extract<T, M>(ctx, X, fa, cfg, sink, kStreamVb, nv, &nl)));
    if (guess) {
      EXT_TRY(window({s->n_prev, counters + kCountFeatures, counters + kCountFeatures, sink.cap}, guess));
      EXT_TRY(stars(guess));
    }
    EXT_TRY(cudaMemcpyAsync(ctx->h_counters, counters, sizeof(unsigned) * kNumCounters, cudaMemcpyDeviceToHost, st));
    EXT_TRY(cudaEventRecord(ctx->ev1, st));
    EXT_TRY(ctx->sync());
    const unsigned got = ctx->h_counters[kCountFeatures];
    if (got > s->cap - s->n) {
      rc = ensure_stream_store(s, s->n + got + got / 4 + 1024);
      if (rc) return rc;
      continue;
    }
    n_new = got;
    break;
  }

  const unsigned nS = s->n_prev + n_new;
  const unsigned wcap = nS ? nS : 1;
  const bool ranked = wcap <= kRankCap2;
  const bool done = guess && nS <= guess;  // the window that went ahead held it
  if (!done) {
    rc = room(wcap);
    if (rc) return rc;
  }
  if (!done && ranked) {
    EXT_TRY(window({nS}, wcap));
    EXT_TRY(stars(wcap));
  } else if (!done) {
    EXT_TRY(s->s_key.ensure(8 * (size_t)wcap));
    EXT_TRY(s->s_key2.ensure(8 * (size_t)wcap));
    EXT_TRY(s->s_id2.ensure(4 * (size_t)wcap));
    EXT_TRY(ctx->hist.ensure(sizeof(unsigned) * 256 * (size_t)ctx->sort_grid(wcap)));
    const int g = grid_of(wcap, 256, 4096);
    set_u32_kernel<<<1, 1, 0, st>>>(counters + kSWin, nS);
    ext_window_build_kernel<<<g, 256, 0, st>>>((const unsigned long long*)s->lo.p, (const unsigned*)s->prev_ids.p,
                                               s->n_prev, first_new, n_new, (unsigned long long*)s->s_key.p,
                                               (unsigned*)s->s_id.p);
    const int bits = kStreamVb + bits_of(ns * (tnow + 1));
    ids = sort_by_tuple(ctx, s, counters + kSWin, wcap, bits, &nl);
    ext_window_fill_kernel<<<g, 256, 0, st>>>(ids, counters + kSWin, wcap, (const unsigned long long*)s->hi.p,
                                              (const unsigned long long*)s->lo.p, (const unsigned*)s->phase.p,
                                              (unsigned long long*)s->s_hi.p, (unsigned long long*)s->s_lo.p,
                                              (unsigned*)s->s_phase.p);
    if (n_new)
      uf_init_range_kernel<<<grid_of(n_new, 256, 4096), 256, 0, st>>>((unsigned*)s->parent.p, first_new, n_new);
    EXT_TRY(stars(wcap));
    if (n_new)
      ext_collect_spatial_kernel<M><<<grid_of(n_new, 256, 4096), 256, 0, st>>>(
        (const unsigned long long*)s->hi.p, (const unsigned long long*)s->lo.p, first_new, n_new, ns, tnow,
        (unsigned*)s->prev_ids2.p, counters + kSPrev);
    nl += 5;
  }
  EXT_TRY(cudaGetLastError());
  if (!done) {
    EXT_TRY(cudaMemcpyAsync(ctx->h_counters, counters, sizeof(unsigned) * kNumCounters, cudaMemcpyDeviceToHost, st));
    EXT_TRY(cudaEventRecord(ctx->ev1, st));
    EXT_TRY(ctx->sync());
  }
  ctx->launches += nl;
  const unsigned* h = ctx->h_counters;
  if (h[kCountErr] & kErrCofaces) return ext_fail(ctx, FTK2B_UNSUPPORTED, "a base face has more than 8 coface cells");
  if (h[kCountErr] & 1u) return ext_fail(ctx, FTK2B_TIMEOUT, "union-find retry bound reached");
  s->n_edges += h[kSWinEdges];
  s->last_window = nS;
  s->n_prev = h[kSPrev];
  std::swap(s->prev_ids, s->prev_ids2);
  s->n += n_new;
  if (tnow == 0) s->n_first = n_new;
  s->last_new = n_new;
  return FTK2B_OK;
}

template <int M>
ftk2b_status result_extruded_t(ftk2b_stream* s, ftk2b_cp_result** out) {
  ftk2b_ctx* ctx = s->ctx;
  cudaStream_t st = ctx->stream;
  unsigned long long nl = 0;
  const unsigned n = s->n, ne = s->n_edges;
  const unsigned nc = n ? n : 1, ec = ne ? ne : 1, mc = nc > ec ? nc : ec;
  EXT_TRY(ctx->counters.ensure(sizeof(unsigned) * kNumCounters));
  unsigned* counters = (unsigned*)ctx->counters.p;
  EXT_TRY(s->s_key.ensure(8 * (size_t)mc));
  EXT_TRY(s->s_key2.ensure(8 * (size_t)mc));
  EXT_TRY(s->s_id.ensure(4 * (size_t)mc));
  EXT_TRY(s->s_id2.ensure(4 * (size_t)mc));
  EXT_TRY(ctx->perm0.ensure(4 * (size_t)nc));
  EXT_TRY(ctx->perm1.ensure(4 * (size_t)nc));
  EXT_TRY(ctx->parent.ensure(4 * (size_t)nc));
  EXT_TRY(ctx->lam_s.ensure(32 * (size_t)nc));
  EXT_TRY(ctx->bary4_s.ensure(16 * (size_t)nc));
  EXT_TRY(ctx->scalar_s.ensure(4 * (size_t)nc));
  EXT_TRY(ctx->cls.ensure(4 * (size_t)nc));
  EXT_TRY(ctx->track.ensure(8 * (size_t)nc));
  EXT_TRY(ctx->simplices.ensure(8 * (size_t)(M + 1) * nc));
  EXT_TRY(ctx->bary.ensure(4 * (size_t)(M + 1) * nc));
  EXT_TRY(ctx->edges.ensure(8 * (size_t)ec));
  EXT_TRY(ctx->hist.ensure(sizeof(unsigned) * 256 * (size_t)ctx->sort_grid(mc)));
  const int g = grid_of(mc, 256, 4096);
  EXT_TRY(cudaMemsetAsync(counters, 0, sizeof(unsigned) * kNumCounters, st));
  unsigned* inv = (unsigned*)ctx->perm0.p;
  unsigned* root = (unsigned*)ctx->perm1.p;
  unsigned* cmin = (unsigned*)ctx->parent.p;
  const unsigned* perm;
  if (nc <= kRankCap2) {
    const LoadTuple ld{(const unsigned long long*)s->hi.p, (const unsigned long long*)s->lo.p, nullptr, 0u, 0u};
    const StoreTupleOrder so{{(unsigned*)s->s_id.p, inv, cmin}};
    EXT_TRY(launch_rank_sort<2>(ld, so, RankCount{n}, nc, counters + kSWin, ctx->num_sms, st));
    perm = so.order.perm;
  } else {
    set_u32_kernel<<<1, 1, 0, st>>>(counters + kSWin, n);
    EXT_TRY(cudaMemcpyAsync(s->s_key.p, s->lo.p, 8 * (size_t)n, cudaMemcpyDeviceToDevice, st));
    iota_u32_kernel<<<g, 256, 0, st>>>((unsigned*)s->s_id.p, n);
    const unsigned long long ns = s->emesh.n_base_verts;
    perm = sort_by_tuple(ctx, s, counters + kSWin, nc, kStreamVb + bits_of(ns * (s->T + 1)), &nl);
    invert_kernel<<<g, 256, 0, st>>>(perm, n, inv);
    fill_u32_kernel<<<g, 256, 0, st>>>(cmin, n, 0xFFFFFFFFu);
  }
  comp_min_kernel<<<g, 256, 0, st>>>((unsigned*)s->parent.p, inv, n, root, cmin, counters + kCountRoots);
  gather_result_kernel<<<g, 256, 0, st>>>(perm, n, root, cmin, (const double*)s->lam.p, (const float*)s->bary4.p,
                                          (const float*)s->scalar.p, (const unsigned*)s->cls.p, (double*)ctx->lam_s.p,
                                          (float*)ctx->bary4_s.p, (float*)ctx->scalar_s.p, (unsigned*)ctx->cls.p,
                                          (unsigned long long*)ctx->track.p);
  ext_stream_expand_kernel<M><<<g, 256, 0, st>>>(perm, n, (const unsigned long long*)s->hi.p,
                                                 (const unsigned long long*)s->lo.p, (const float*)ctx->bary4_s.p,
                                                 (unsigned long long*)ctx->simplices.p, (float*)ctx->bary.p);
  nl += 4;
  EXT_TRY(cudaGetLastError());
  ctx->launches += nl;
  // edges in canonical ids, sorted; the id and key buffers are free after the gathers
  const ftk2b_status rc = canonical_edges(s, inv, (unsigned long long*)s->s_key.p, (unsigned long long*)s->s_key2.p);
  if (rc) return rc;
  ctx->last.kind = FTK2B_MESH_EXTRUDED;
  ctx->last.m = M;
  ctx->last.f64 = s->dtype == FTK2B_F64;
  ctx->pack_ready = false;
  ctx->last.n = n;
  ctx->last.ne = s->prm.want_edges ? ne : 0;
  // m-simplices of the T-timestep mesh, from the prepared base mesh's counts
  const uint64_t L = s->T ? s->T - 1 : 0;
  ctx->last.n_simplices =
      s->T ? ctx->ext.ncell * (L + 1) + (uint64_t)ctx->ext.nface * L * M + ctx->ext.ncell * L * M : 0;
  ctx->last.device_ms = 0;
  ctx->last.classify = 0;
  ctx->last.want_edges = s->prm.want_edges;
  return stream_fetch(s, out);
}

}  // namespace

}  // namespace ftk2b

ftk2b_status stream_push_extruded(ftk2b_stream* s) {
  if (s->prm.classify) {
    s->ctx->err = "classification of extruded meshes is not available";
    return FTK2B_UNSUPPORTED;
  }
  const bool f64 = s->dtype == FTK2B_F64;
  if (s->m == 3) return f64 ? push_extruded_t<double, 3>(s) : push_extruded_t<float, 3>(s);
  return f64 ? push_extruded_t<double, 2>(s) : push_extruded_t<float, 2>(s);
}

ftk2b_status stream_result_extruded(ftk2b_stream* s, ftk2b_cp_result** out) {
  return s->m == 3 ? result_extruded_t<3>(s, out) : result_extruded_t<2>(s, out);
}

uint64_t extruded_simplex_count(const ftk2b_mesh_desc* mesh, int m) {
  const int cd = mesh->base_cell_dim;
  if ((cd != 2 && cd != 3) || m != cd || (mesh->n_base_cells && !mesh->base_cells)) return 0;
  // unique (cd-1)-faces of the base, counted on the host from packed keys
  // (base vertex ids below 2^21 for tets, 2^32 for triangles; wider ids are
  // not supported by the extruded path either)
  const int fbits = bits_of(mesh->n_base_verts ? mesh->n_base_verts - 1 : 0);
  if (fbits * cd > 64) return 0;
  std::vector<uint64_t> keys;
  keys.reserve(mesh->n_base_cells * (cd + 1));
  for (uint64_t c = 0; c < mesh->n_base_cells; ++c) {
    uint64_t v[4];
    for (int i = 0; i <= cd; ++i) v[i] = mesh->base_cells[c * (cd + 1) + i];
    std::sort(v, v + cd + 1);
    for (int r = 0; r <= cd; ++r) {
      uint64_t k = 0;
      for (int i = 0; i <= cd; ++i)
        if (i != r) k = (k << fbits) | v[i];
      keys.push_back(k);
    }
  }
  std::sort(keys.begin(), keys.end());
  const uint64_t nface = (uint64_t)(std::unique(keys.begin(), keys.end()) - keys.begin());
  const uint64_t L = mesh->n_layers;
  return mesh->n_base_cells * (L + 1) + nface * L * cd + mesh->n_base_cells * L * cd;
}

ftk2b_status run_extruded(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, const ftk2b_field_desc* field,
                          const ftk2b_cp_params* prm, const double* fiber_thr, bool pack) {
  int fbits = 0;
  ftk2b_status st = validate_mesh(ctx, mesh, &fbits);
  if (st) return st;
  const int M = mesh->base_cell_dim;
  if (field->ncomp != M)
    return ext_fail(ctx, FTK2B_INVALID_ARG, "an extruded mesh over dimension-" + std::to_string(M) +
                                                " cells needs " + std::to_string(M) + " components");
  if (field->layout == FTK2B_LAYOUT_MULTICOMPONENT)
    return ext_fail(ctx, FTK2B_UNSUPPORTED,
                    "extruded meshes take per-vertex arrays (the reference indexes multicomponent arrays "
                    "by grid coordinates, which an unstructured mesh does not have)");
  if (field->layout == FTK2B_LAYOUT_SEPARATE && field->nd != 1)
    return ext_fail(ctx, FTK2B_INVALID_ARG, "extruded meshes take 1-D per-vertex arrays");
  const unsigned ns = (unsigned)mesh->n_base_verts;
  const unsigned L = (unsigned)mesh->n_layers;
  const unsigned long long nv = (unsigned long long)ns * (L + 1);
  FieldAccess fa;
  st = prepare_field(ctx, field, 1, nullptr, nullptr, nv, fa);
  if (st) return st;
  if (!fa.per_vertex) return ext_fail(ctx, FTK2B_INVALID_ARG, "extruded meshes take per-vertex arrays");
  if (fa.has_scalar && !fa.scalar_per_vertex)
    return ext_fail(ctx, FTK2B_INVALID_ARG, "the scalar of an extruded mesh must be a per-vertex array");

  unsigned long long nl = 0;
  st = prepare_base(ctx, mesh, fbits, &nl);
  if (st) return st;
  ExtCache& C = ctx->ext;
  ExtMeshDev X;
  X.cd = M;
  X.ns = ns;
  X.L = L;
  X.ncell = (unsigned)C.ncell;
  X.nface = C.nface;
  X.fbits = C.fbits;
  X.cells = (const unsigned*)C.cells.p;
  X.fkeys = (const unsigned long long*)C.fkeys.p;
  X.cof_start = (const unsigned*)C.cof_start.p;
  X.cof = (const unsigned*)C.cof.p;
  X.own = (const unsigned*)C.own.p;
  X.t0 = 0;
  X.tflip = 0;
  X.skip_first_spatial = 0;
  const int vb = bits_of(nv - 1);
  const uint64_t nsimp = C.ncell * (uint64_t)(L + 1) + (uint64_t)C.nface * L * M + C.ncell * (uint64_t)L * M;

  ExtractConfig cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.Q = prm->sos_q;
  cfg.refined = prm->precision == FTK2B_PRECISION_REFINED;
  if (fiber_thr) {  // FiberPredicate: every simplex tested, values minus thresholds
    cfg.fiber = 1;
    cfg.fthr[0] = fiber_thr[0];
    cfg.fthr[1] = fiber_thr[1];
    cfg.refined = 0;
  }
  const int f64 = field->dtype == FTK2B_F64;
  EXT_TRY(C.words.ensure(sizeof(unsigned) * nv));

  unsigned cap = ctx->cap_hint ? ctx->cap_hint : 65536u;
  for (int attempt = 0; attempt < 4; ++attempt) {
    const unsigned edge_cap = cap * 2;
    st = ensure_feature_buffers(ctx, cap, edge_cap, M);
    if (st) return st;
    const size_t wk = std::max<size_t>(std::max<size_t>(cap, edge_cap), C.ncell * (size_t)(M + 1));
    EXT_TRY(C.hi.ensure(sizeof(unsigned long long) * cap));
    EXT_TRY(C.lo.ensure(sizeof(unsigned long long) * cap));
    EXT_TRY(C.phase.ensure(sizeof(unsigned) * cap));
    EXT_TRY(C.hi_s.ensure(sizeof(unsigned long long) * cap));
    EXT_TRY(C.lo_s.ensure(sizeof(unsigned long long) * cap));
    EXT_TRY(C.phase_s.ensure(sizeof(unsigned) * cap));
    EXT_TRY(C.sort_k.ensure(sizeof(unsigned long long) * wk));
    EXT_TRY(C.sort_k2.ensure(sizeof(unsigned long long) * wk));
    EXT_TRY(C.sort_v.ensure(sizeof(unsigned) * wk));
    EXT_TRY(C.sort_v2.ensure(sizeof(unsigned) * wk));
    EXT_TRY(C.ekeys.ensure(sizeof(unsigned long long) * wk));
    EXT_TRY(ctx->hist.ensure(sizeof(unsigned) * 256 * (size_t)ctx->sort_grid((unsigned)wk)));
    ExtSink sink;
    sink.hi = (unsigned long long*)C.hi.p;
    sink.lo = (unsigned long long*)C.lo.p;
    sink.phase = (unsigned*)C.phase.p;
    sink.lam = (double*)ctx->lam.p;
    sink.bary4 = (float*)ctx->bary4.p;
    sink.scalar = (float*)ctx->scalar.p;
    sink.count = (unsigned*)ctx->counters.p + kCountFeatures;
    sink.cap = cap;
    cudaStream_t s = ctx->stream;
    EXT_TRY(cudaEventRecord(ctx->ev0, s));
    EXT_TRY(cudaMemsetAsync(ctx->counters.p, 0, sizeof(unsigned) * kNumCounters, s));
    cudaError_t e;
    if (M == 3)
      e = f64 ? enqueue_extract<double, 3>(ctx, X, fa, cfg, sink, vb, nv, &nl)
              : enqueue_extract<float, 3>(ctx, X, fa, cfg, sink, vb, nv, &nl);
    else
      e = f64 ? enqueue_extract<double, 2>(ctx, X, fa, cfg, sink, vb, nv, &nl)
              : enqueue_extract<float, 2>(ctx, X, fa, cfg, sink, vb, nv, &nl);
    EXT_TRY(e);
    EXT_TRY(cudaEventRecord(ctx->ev_x, s));
    // the number of features decides how they are sorted: reading it costs a
    // wait (about 12 us), the radix passes for a capacity unread some 150 us
    EXT_TRY(cudaMemcpyAsync(ctx->h_counters, ctx->counters.p, sizeof(unsigned) * kNumCounters,
                            cudaMemcpyDeviceToHost, s));
    EXT_TRY(ctx->sync());
    const unsigned n = ctx->h_counters[kCountFeatures];
    if (n > cap) {
      const uint64_t want = (uint64_t)n + n / 4 + 1024;
      if (want > 0x7FFFFFF0ull) return ext_fail(ctx, FTK2B_OVERFLOW_RETRY, "feature count exceeds 2^31");
      cap = (unsigned)want;
      ctx->cap_hint = cap;
      continue;
    }
    bool edges_ranked = false;
    e = (M == 3) ? enqueue_post<3>(ctx, X, sink, n, cap, edge_cap, vb, prm->want_edges, &edges_ranked, &nl)
                 : enqueue_post<2>(ctx, X, sink, n, cap, edge_cap, vb, prm->want_edges, &edges_ranked, &nl);
    EXT_TRY(e);
    LastRun r;
    r.m = M;
    r.want_edges = prm->want_edges;
    if (pack) {
      PackArgs a = ctx->pack_args(r);
      a.h_counters = (unsigned*)ctx->pin.d;
      a.cap = cap;
      a.edge_cap = edges_ranked ? std::min(edge_cap, kRankCap1) : edge_cap;
      EXT_TRY(launch_pack(a, ctx->num_sms, s));
      nl += 1;
    } else {
      EXT_TRY(cudaMemcpyAsync(ctx->h_counters, ctx->counters.p, sizeof(unsigned) * kNumCounters,
                              cudaMemcpyDeviceToHost, s));
    }
    EXT_TRY(cudaEventRecord(ctx->ev1, s));
    EXT_TRY(ctx->sync());
    ctx->launches += nl;
    nl = 0;
    unsigned h[kNumCounters];
    memcpy(h, ctx->h_counters, sizeof(h));
    float ms = 0.f, xms = 0.f;
    if (cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1) != cudaSuccess) ms = 0.f;
    if (cudaEventElapsedTime(&xms, ctx->ev0, ctx->ev_x) != cudaSuccess) xms = 0.f;
    cudaGetLastError();
    ctx->last_extract_ms = xms;
    if (h[kCountErr] & kErrCofaces)
      return ext_fail(ctx, FTK2B_UNSUPPORTED, "a base face has more than 8 coface cells");
    if (h[kCountErr] & 1u) return ext_fail(ctx, FTK2B_TIMEOUT, "union-find retry bound reached");
    if (h[kCountEdges] > edge_cap) {
      const uint64_t want = ((uint64_t)h[kCountEdges] + 1) / 2 + 1024;
      if (want > 0x7FFFFFF0ull) return ext_fail(ctx, FTK2B_OVERFLOW_RETRY, "feature count exceeds 2^31");
      cap = (unsigned)want;
      ctx->cap_hint = cap;
      continue;
    }
    const bool edges_left = edges_ranked && h[kCountEdges] > kRankCap1;  // few features, very many edges
    if (edges_left) {
      EXT_TRY(sort_edges(ctx, edge_cap, &nl));
      EXT_TRY(ctx->sync());
      ctx->launches += nl;
    }
    ctx->last.kind = FTK2B_MESH_EXTRUDED;
    ctx->last.m = M;
    ctx->last.f64 = field->dtype == FTK2B_F64;
    ctx->last.n = h[kCountFeatures];
    ctx->last.ne = prm->want_edges ? h[kCountEdges] : 0;
    ctx->last.n_roots = h[kCountRoots];
    ctx->last.n_simplices = nsimp;
    ctx->last.device_ms = ms;
    ctx->last.classify = 0;
    ctx->last.want_edges = prm->want_edges;
    ctx->pack_ready =
        pack && !edges_left && pack_layout(ctx->last.n, ctx->last.ne, M + 1, 0).packed <= ctx->pack_bytes();
    return FTK2B_OK;
  }
  return ext_fail(ctx, FTK2B_OVERFLOW_RETRY, "feature buffer overflow persisted after retries");
}
