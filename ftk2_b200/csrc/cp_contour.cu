// Level sets of a scalar field on a regular spacetime mesh: the
// SimplicialEngine<T, ContourPredicate<T>> path (execute + get_complex,
// engine.hpp:95-215 and 822-996; ContourPredicate predicate.hpp:135-183;
// marching_pentatope / marching_tetrahedron engine.hpp:1210-1339) as one
// device pipeline:
//
//   ct_sign    one pass over the field: the simulation-of-simplicity sign of
//              value - threshold at every vertex (sos.hpp:12-20), one bit
//   ct_mask    per vertex c, the directions e in {0,1}^d \ 0 whose edge to
//              c + e crosses (the signs differ, origin_inside<1>,
//              sos.hpp:211-220), per-block counts, and the hypercubes whose
//              corners differ in sign
//   scan       block offsets.  Every Freudenthal edge joins some c to c + e,
//              so the edges in simplex order are the (c, e) pairs in vertex
//              order with e read as a binary number, x lowest: a feature's
//              rank is its block offset plus a prefix count, no sort needed
//   ct_emit    vertex ids and barycentrics of every feature at its rank
//   ct_join    the two crossing edges of every crossed triangle united
//   ct_first   (2D+t) the position at which the reference's sequential
//              patching first meets each node whose edge starts on an upper
//              boundary face (those are numbered in meeting order, after the
//              first pass's nodes, and 2D+t quads are cut along the diagonal
//              from their smallest-numbered node)
//   ct_cells   marching tetrahedra / pentatopes over every Kuhn simplex of the
//              listed hypercubes: manifold cells
//   buckets    cells into lexicographic order: counted and scattered by
//              their leading node, each bucket's few rows sorted, duplicates
//              flagged
//   label      track id = the component's smallest feature index
#include <algorithm>
#include <array>
#include <vector>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "../../include/ftk2b.h"
#include "cp_api_internal.h"
#include "cp_device.cuh"
#include "cp_host.h"
#include "cp_post.h"
#include "cp_uf.cuh"

using namespace ftk2b;

namespace {

constexpr int kCtThreads = 256;

struct CtGeom {
  int d;                        // mesh dims: 3 (2D+t) or 4 (3D+t)
  int per_vertex;               // field indexed by global vertex id
  unsigned long long L[4];      // local dims
  unsigned long long as[4];     // array strides of the local coordinates
  unsigned long long gs[4];     // global id strides
  unsigned long long g0;        // global id of the local origin
  unsigned long long nv;        // local vertices
  unsigned long long ncube;     // local hypercubes
  unsigned long long loff[16];  // local linear step to corner e
  unsigned long long goff[16];  // global id step to corner e
  unsigned long long aoff[16];  // array step to corner e
  unsigned long long lstr[4];   // local linear strides
  unsigned char perm[24][4];    // axis order of the p-th Kuhn simplex (CPU mesh order)
  int linear;                   // array index = local linear index
  int small;                    // nv < 2^31: i / L[k] = (i * mul[k]) >> shf[k]
  unsigned mul[4];
  int shf[4];
};

// Local coordinates of local vertex i.  Meshes below 2^31 vertices divide by
// multiplying with rounded-up reciprocals (exact for such i): three or four
// 64-bit divisions a vertex bounded every kernel that walks the vertices.
__device__ __forceinline__ void ct_coords(const CtGeom& g, unsigned long long i, unsigned long long* c) {
  if (g.small) {
    unsigned r = (unsigned)i;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned q = k + 1 < g.d ? (unsigned)(((unsigned long long)r * g.mul[k]) >> g.shf[k]) : 0u;
      c[k] = k < g.d ? r - q * (unsigned)g.L[k] : 0u;
      r = q;
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k < g.d) {
      c[k] = i % g.L[k];
      i /= g.L[k];
    } else {
      c[k] = 0;
    }
  }
}

__device__ __forceinline__ unsigned long long ct_gid(const CtGeom& g, const unsigned long long* c) {
  unsigned long long v = g.g0;
#pragma unroll
  for (int k = 0; k < 4; ++k) v += c[k] * g.gs[k];  // strides of axes the mesh has not are 0
  return v;
}

__device__ __forceinline__ unsigned long long ct_aidx(const CtGeom& g, const unsigned long long* c) {
  unsigned long long v = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) v += c[k] * g.as[k];
  return v;
}

template <typename T>
__device__ __forceinline__ T ct_adj(const CtGeom& g, const T* __restrict__ a, unsigned long long aidx,
                                    unsigned long long gid, T thr) {
  const T v = g.per_vertex ? __ldg(a + gid) : __ldg(a + aidx);
  return fp<T>::sub(v, thr);
}

// sos::sign(v, id, Q) > 0: (int)(double(v) * Q + (v > 0 ? 0.5 : -0.5)) is
// positive exactly when the rounded sum is >= 1, negative when <= -1; zero
// goes by the parity of the vertex id.  Multiply and add rounded separately.
template <typename T>
__device__ __forceinline__ bool ct_positive(T adj, unsigned long long gid, double q) {
  const double x = __dadd_rn(__dmul_rn((double)adj, q), adj > T(0) ? 0.5 : -0.5);
  if (x >= 1.0) return true;
  if (x <= -1.0) return false;
  return (gid & 1ull) == 0;
}

// Bit planes: bit i & 31 of word i >> 5 belongs to local vertex i.  The 32
// neighbours of 32 consecutive vertices in one corner direction are then one
// shifted word, and a warp settles its vertices with a word per corner and lane
// instead of a load per corner and vertex.
__host__ __device__ inline unsigned long long ct_words(const CtGeom& g) {
  return (g.nv + g.loff[(1 << g.d) - 1]) / 32 + 2;  // the corners of out-of-mesh cubes included
}

// Each warp takes 128 consecutive vertices, four per lane in flight:
// load(i, j) by every lane (the last vertex again beyond the end; it must not
// use the value), then words(w, j) by the whole warp for the 32 of word w.
template <typename Load, typename Words>
__device__ __forceinline__ void ct_each_word(unsigned long long n, Load load, Words words) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x * 4;
  for (unsigned long long i0 = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x - lane) * 4; i0 < n;
       i0 += step) {
#pragma unroll
    for (int j = 0; j < 4; ++j) load(min(i0 + 32 * j + lane, n - 1), j);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + 32 * j < n) words(i0 / 32 + j, j);
  }
}

// step from a vertex to its corner e (lane-varying, so not from the table)
__device__ __forceinline__ unsigned long long ct_corner_step(const CtGeom& g, unsigned e) {
  unsigned long long v = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) v += (e >> k) & 1u ? g.lstr[k] : 0ull;
  return v;
}

// array index of local vertex i
__device__ __forceinline__ unsigned long long ct_index(const CtGeom& g, unsigned long long i) {
  if (g.linear) return i;
  unsigned long long c[4];
  ct_coords(g, i, c);
  return g.per_vertex ? ct_gid(g, c) : ct_aidx(g, c);
}

// Bound by the field's bytes (96^3 x 6 double: 56 us with 64-bit divisions for
// each vertex's coordinates, which only ties need, now 14).
template <typename T>
__global__ void ct_sign_kernel(CtGeom g, const T* __restrict__ a, T thr, double q, unsigned* __restrict__ pos) {
  const unsigned lane = threadIdx.x & 31;
  T v[4];
  ct_each_word(
      g.nv, [&](unsigned long long i, int j) { v[j] = __ldg(a + ct_index(g, i)); },
      [&](unsigned long long w, int j) {
        const unsigned long long i = 32 * w + lane;
        bool p = false;
        if (i < g.nv) {
          const T y = fp<T>::sub(v[j], thr);
          const double x = __dadd_rn(__dmul_rn((double)y, q), y > T(0) ? 0.5 : -0.5);
          p = x >= 1.0;
          if (!p && !(x <= -1.0)) {
            unsigned long long c[4];
            ct_coords(g, i, c);
            p = ct_positive(y, ct_gid(g, c), q);
          }
        }
        const unsigned word = __ballot_sync(0xffffffffu, p);
        if (lane == 0) pos[w] = word;
      });
}

// block-wide exclusive scan of one count per thread; returns the thread's
// prefix, *total the block's sum
__device__ __forceinline__ unsigned ct_block_scan(unsigned v, unsigned* total) {
  __shared__ unsigned wsum[kCtThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    unsigned w = lane < kCtThreads / 32 ? wsum[lane] : 0;
    unsigned wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < kCtThreads / 32) wsum[lane] = wi - w;
    if (lane == kCtThreads / 32 - 1) *total = wi;
  }
  __syncthreads();
  return wsum[warp] + incl - v;
}

// Kernels over the vertices of a regular mesh give a block kCtPer shares of
// kCtThreads consecutive vertices: vertex share * kCtThreads + thread.  One
// atomic per block then reserves list rows or adds to a total; one per warp on
// the same address took longer than everything else these kernels do.
constexpr int kCtPer = 4;
constexpr int kCtBlock = kCtPer * kCtThreads;

// Exclusive prefix in vertex order over the block of kCtPer counts per thread;
// returns the block's sum.
__device__ __forceinline__ unsigned ct_block_ranks(unsigned (&v)[kCtPer]) {
  constexpr int kWarps = kCtThreads / 32;
  static_assert(kCtPer * kWarps == 32, "one warp scans the words' sums");
  __shared__ unsigned sum[32], total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    unsigned incl = v[j];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) sum[j * kWarps + warp] = incl;
    v[j] = incl - v[j];
  }
  __syncthreads();
  if (warp == 0) {
    const unsigned w = sum[lane];
    unsigned wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    sum[lane] = wi - w;
    if (lane == 31) total = wi;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) v[j] += sum[j * kWarps + warp];
  return total;
}

__device__ __forceinline__ unsigned ct_inbounds(const CtGeom& g, const unsigned long long* c) {
  unsigned inb = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (c[k] + 1 < g.L[k]) inb |= 1u << k;
  return inb;
}

// Crossing mask of every vertex (bit e - 1: the edge to corner e), the counts
// of each block, and the list of mixed hypercubes (corner signs not all equal),
// each one word: base vertex (local linear index) << 20 | upper-face axes << 16
// | corner signs (bit e: corner e positive).  An upper-face axis k is one where
// the cube's corners with bit k set lie on the mesh's last layer (c_k = L_k - 2).
// A cube's signs are its lowest vertex's and mask, so the cubes need no pass of
// their own (96^3 x 6: 90 + 57 us for both, now 38).
constexpr int kCtBaseShift = 20;

__global__ void __launch_bounds__(kCtThreads) ct_mask_kernel(
    CtGeom g, const unsigned* __restrict__ pos, unsigned short* __restrict__ mask, unsigned* __restrict__ blk,
    unsigned long long* __restrict__ total64, unsigned long long* __restrict__ list,
    unsigned* __restrict__ list_cnt) {
  __shared__ unsigned s_at;
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock + threadIdx.x;
  const int ne = 1 << g.d;
  const unsigned lane = threadIdx.x & 31;
  // lane e: the signs of the warp's vertices, and those at their corners e
  unsigned here[kCtPer], cross[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long w0 = i0 - lane + j * kCtThreads;
    here[j] = cross[j] = 0;
    if (w0 < g.nv) {
      here[j] = pos[w0 / 32];
      if ((int)lane < ne) {
        const unsigned long long o = w0 + ct_corner_step(g, lane);
        cross[j] = here[j] ^ __funnelshift_r(pos[o / 32], pos[o / 32 + 1], (unsigned)o & 31u);
      }
    }
  }
  unsigned rank[kCtPer];  // crossing edges, mixed cubes << 16
  unsigned upper[kCtPer], m[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long i = i0 + j * kCtThreads;
    m[j] = upper[j] = rank[j] = 0;
    if (__any_sync(0xffffffffu, cross[j] != 0)) {
      unsigned long long c[4];
      ct_coords(g, i, c);
      const unsigned inb = i < g.nv ? ct_inbounds(g, c) : 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const unsigned in = __ballot_sync(0xffffffffu, (inb >> k) & 1u);
        if ((lane >> k) & 1u) cross[j] &= in;
        if (c[k] + 2 == g.L[k]) upper[j] |= 1u << k;
      }
#pragma unroll
      for (int e = 1; e < 16; ++e) m[j] |= ((__shfl_sync(0xffffffffu, cross[j], e) >> lane) & 1u) << (e - 1);
      rank[j] = __popc(m[j]);
      if (m[j] != 0 && inb == (1u << g.d) - 1u) rank[j] |= 1u << 16;
    }
    if (i < g.nv) mask[i] = (unsigned short)m[j];
  }
  bool mixed[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) mixed[j] = rank[j] >> 16;
  const unsigned n = ct_block_ranks(rank);
  if (threadIdx.x == 0) {
    blk[blockIdx.x] = n & 0xFFFFu;
    if (n & 0xFFFFu) atomicAdd(total64, (unsigned long long)(n & 0xFFFFu));  // exact: the offsets are 32-bit
    if (n >> 16) s_at = atomicAdd(list_cnt, n >> 16);
  }
  if (n >> 16 == 0) return;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    if (!mixed[j]) continue;
    const unsigned all = (1u << ne) - 1u, sgn = (here[j] >> lane) & 1u ? ~(m[j] << 1) & all : m[j] << 1;
    list[s_at + (rank[j] >> 16)] =
        ((i0 + j * kCtThreads) << kCtBaseShift) | ((unsigned long long)upper[j] << 16) | sgn;
  }
}

// ZeroCrossingSolver<1,T>::solve (zero_crossing.hpp:93-104) with the
// predicate's fallback to the midpoint (predicate.hpp:149), in T, each
// operation rounded on its own
template <typename T>
__device__ __forceinline__ void ct_solve(T a0, T a1, T* l0, T* l1) {
  using F = fp<T>;
  const T dd = F::sub(a0, a1);
  bool ok = !(F::abs(dd) < T(1e-12));
  T x0 = T(0.5), x1 = T(0.5);
  if (ok) {
    x0 = F::div(-a1, dd);
    x1 = F::sub(T(1.0), x0);
    const T eps = T(1e-9);
    ok = x0 >= -eps && x0 <= F::add(T(1.0), eps);
  }
  *l0 = ok ? x0 : T(0.5);
  *l1 = ok ? x1 : T(0.5);
}

// The crossing edges of a block's vertices in rank order: entry k is vertex of
// the block << 4 | corner.  Returns their number; n edges start at rank
// blk_off[block].  s_mask: the vertices' masks.
struct CtEdges {
  unsigned short edge[kCtBlock * 15];
  unsigned short mask[kCtBlock];
};
__device__ __forceinline__ unsigned ct_list_edges(const CtGeom& g, const unsigned short* __restrict__ mask,
                                                  unsigned base, unsigned* __restrict__ voff, CtEdges& s) {
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock;
  unsigned m[kCtPer], rank[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long i = i0 + j * kCtThreads + threadIdx.x;
    m[j] = i < g.nv ? mask[i] : 0u;
    rank[j] = __popc(m[j]);
  }
  const unsigned n = ct_block_ranks(rank);
  if (n == 0) return 0;
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned v = j * kCtThreads + threadIdx.x;
    unsigned w = rank[j];
    s.mask[v] = (unsigned short)m[j];
    if (m[j] && voff) voff[i0 + v] = base + w;
    for (unsigned x = m[j]; x; x &= x - 1) s.edge[w++] = (unsigned short)(v << 4 | __ffs(x));
  }
  __syncthreads();
  return n;
}

// number of crossing edges of mask m below corner e
__device__ __forceinline__ unsigned ct_below(unsigned m, unsigned e) { return __popc(m & ((1u << (e - 1)) - 1u)); }
// The crossing edges at one vertex that certainly belong together: all of them
// when the main diagonal is one (every corner is a subset of it), else those
// whose corner contains the first one's (a triangle holds both edges).  The
// others stand alone until a triangle joins them.
__device__ __forceinline__ bool ct_with_first(unsigned m, unsigned e, unsigned diag) {
  const unsigned f = __ffs(m);
  return ((m >> (diag - 1)) & 1u) || (e & f) == f;
}

// A thread per crossing edge; listed in shared memory first, so the rows leave
// in whole lines (96^3 x 6 double: 106 us with a thread per vertex, now 28).
// voff (first rank) is written where a vertex has edges; parent starts at the
// vertex's first edge where the two belong together (a mesh of single layers
// has triangles but no cells, which are what joins).
template <typename T>
__global__ void __launch_bounds__(kCtThreads) ct_emit_kernel(
    CtGeom g, const T* __restrict__ a, T thr, const unsigned short* __restrict__ mask,
    const unsigned* __restrict__ blk_off, unsigned* __restrict__ voff, unsigned long long* __restrict__ simp,
    double* __restrict__ lam, float* __restrict__ bary, unsigned* __restrict__ parent) {
  __shared__ CtEdges s;
  const unsigned base = blk_off[blockIdx.x];
  const unsigned n = ct_list_edges(g, mask, base, voff, s);
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock;
  for (unsigned k = threadIdx.x; k < n; k += kCtThreads) {
    const unsigned x = s.edge[k] >> 4, e = s.edge[k] & 15u;
    unsigned long long c[4];
    ct_coords(g, i0 + x, c);
    const unsigned long long gid = ct_gid(g, c), ai = ct_aidx(g, c);
    const T a0 = ct_adj(g, a, ai, gid, thr), a1 = ct_adj(g, a, ai + g.aoff[e], gid + g.goff[e], thr);
    T l0, l1;
    ct_solve(a0, a1, &l0, &l1);
    const unsigned r = base + k, m = s.mask[x];
    reinterpret_cast<ulonglong2*>(simp)[r] = make_ulonglong2(gid, gid + g.goff[e]);
    reinterpret_cast<double2*>(lam)[r] = make_double2((double)l0, (double)l1);
    reinterpret_cast<float2*>(bary)[r] = make_float2((float)l0, (float)l1);
    parent[r] = g.ncube && ct_with_first(m, e, (1u << g.d) - 1u) ? r - ct_below(m, e) : r;
  }
}

// The first crossing edge (v, v + e) of every vertex starts at an edge of a lower
// vertex w = v - a, a an axis outside e: in the triangle (w, w + a, w + a + e)
// exactly one of (w, a) and (w, a + e) crosses too.  Most edges then hang in
// one long tree before the joins, which otherwise meet everywhere at once.
__global__ void __launch_bounds__(kCtThreads) ct_hook_kernel(CtGeom g, const unsigned short* __restrict__ mask,
                                                             const unsigned* __restrict__ voff,
                                                             unsigned* __restrict__ parent) {
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock + threadIdx.x;
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long i = i0 + j * kCtThreads;
    const unsigned m = i < g.nv ? mask[i] : 0u;
    if (!m) continue;
    unsigned long long c[4];
    ct_coords(g, i, c);
    const unsigned e = __ffs(m);
    for (int k = g.d - 1; k >= 0; --k) {
      if (((e >> k) & 1u) || c[k] == 0) continue;
      const unsigned long long w = i - g.lstr[k];
      const unsigned mw = mask[w], a = 1u << k;
      parent[voff[i]] = voff[w] + ct_below(mw, (mw >> (a - 1)) & 1u ? a : a | e);
      break;
    }
  }
}

// Joins the crossing edges of every mesh triangle that has two.  The crossing
// edges of a simplex hang together through its triangles, so this gives the
// components of the cells; a triangle (v, v + a, v + b), a a subset of b, is met
// once, at a vertex with crossing edges (one of the two is at v):
//   (v, a) and (v, b)            unless the vertex's edges started joined
//   (v, a) and (v + a, b - a)    all edges at v + a disjoint from a
//   (v, b) and (v + a, b - a)    v has no edge to a
// A thread takes one vertex and corner a; of edges that started joined on both
// sides one pair is enough.  Bound by the dependent loads of ranks and roots, so
// what counts is how many threads are at it: while the mesh has fewer than
// kJoinBlocks shares of vertices an SM, several blocks (grid y) list the vertices
// of one share and take its items in turn, up to one item a thread.  White noise
// on 16 x 16 x 4 vertices (2,800 edges): 498 us with one block a share, 33 so; a
// whole level set of 16^3 x 3 noise 2251 -> 270 us on the device, of 96^3 x 6
// blobs (936,000 edges) 702 -> 660 (16 an SM: 703).  Joining every cell's nodes
// from the cells kernel took four times as many unions from divergent lanes.
//
// From kCtHooked edges on, threads that join the same two large trees queue on
// their roots: there the first edges are hooked ahead and the trees flattened,
// one vertex of kCtSample joins along its axes, the trees (few by then) are
// flattened again, and the rest mostly finds equal parents.  Whole level sets with
// and without: 128^3 x 16 (9.0 million edges) 4.68 / 5.07 ms, 128^3 x 8 (4.4)
// 2.37 / 2.57, 24^3 x 16 noise (1.5) 1.22 / 1.22, 96^3 x 6 (0.94) 0.66 / 0.66, 48^3
// x 4 (0.15) 0.26 / 0.23, 1000 x 700 x 12 (0.06) 0.28 / 0.24.
constexpr unsigned kJoinBlocks = 64;
constexpr unsigned kCtHooked = 1u << 20;
constexpr unsigned kCtSample = 4;

__global__ void __launch_bounds__(kCtThreads) ct_join_kernel(CtGeom g, const unsigned short* __restrict__ mask,
                                                             const unsigned* __restrict__ voff, unsigned* parent,
                                                             unsigned* err, bool sample) {
  __shared__ unsigned short s_vert[kCtBlock], s_mask[kCtBlock];
  __shared__ unsigned long long s_off[16];
  if (threadIdx.x < 16) s_off[threadIdx.x] = ct_corner_step(g, threadIdx.x);
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock;
  unsigned m[kCtPer], at[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long i = i0 + j * kCtThreads + threadIdx.x;
    m[j] = i < g.nv ? mask[i] : 0u;
    at[j] = m[j] ? 1u : 0u;
  }
  const unsigned n = ct_block_ranks(at);
  if (n == 0) return;
#pragma unroll
  for (int j = 0; j < kCtPer; ++j)
    if (m[j]) {
      s_vert[at[j]] = (unsigned short)(j * kCtThreads + threadIdx.x);
      s_mask[at[j]] = (unsigned short)m[j];
    }
  __syncthreads();
  const unsigned diag = (1u << g.d) - 1u;
  const unsigned per = sample ? (unsigned)g.d : diag, step = sample ? kCtSample : 1u;
  for (unsigned k = blockIdx.y * kCtThreads + threadIdx.x; k < (n + step - 1) / step * per;
       k += gridDim.y * kCtThreads) {
    const unsigned z = k / per * step, mv = s_mask[z], a = sample ? 1u << k % per : k % per + 1;
    const bool edge = (mv >> (a - 1)) & 1u;
    unsigned with = 0;  // no edge to a: the corners b above a that have one
    if (!edge) {
      for (unsigned y = mv; y; y &= y - 1) {
        const unsigned b = __ffs(y);
        if ((b & a) == a) with |= 1u << (b - 1);
      }
      if (!with) continue;
    }
    const unsigned long long v = i0 + s_vert[z], u = v + s_off[a];
    const unsigned mu = mask[u], ov = voff[v];
    const unsigned ou = mu ? voff[u] : 0u;
    bool met = false;
    if (edge) {
      const unsigned r = ov + ct_below(mv, a);
      for (unsigned y = mu; y; y &= y - 1) {
        const unsigned f = __ffs(y);
        if (f & a) continue;
        if (ct_with_first(mu, f, diag)) {
          if (met) continue;
          met = true;
        }
        uf_unite_flat(parent, r, ou + ct_below(mu, f), err);
      }
      if (!ct_with_first(mv, a, diag))
        for (unsigned y = mv; y; y &= y - 1) {
          const unsigned b = __ffs(y);
          if ((b & a) == a && b != a) uf_unite_flat(parent, r, ov + ct_below(mv, b), err);
        }
    } else {
      for (unsigned y = with; y; y &= y - 1) {
        const unsigned b = __ffs(y);
        if (ct_with_first(mv, b, diag) && ct_with_first(mu, b ^ a, diag)) {
          if (met) continue;
          met = true;
        }
        uf_unite_flat(parent, ov + ct_below(mv, b), ou + ct_below(mu, b ^ a), err);
      }
    }
  }
}

// A warp takes 32 / (D!) listed cubes, a lane per Kuhn simplex.  A lane's path
// (corner masks along the CPU mesh's permutation order) is the same for every
// cube, so its corners and their steps lie in shared memory, a column per lane:
// lane-varying indexes into the kernel's parameters are served one address at
// a time, and indexes into arrays of a thread's own go through local memory.
template <int D>
struct CtPaths {
  unsigned corner[D + 1][32];
  unsigned long long off[D + 1][32];
};
template <int D>
struct CtLane {
  static constexpr int kSimp = D == 3 ? 6 : 24, kCubes = 32 / kSimp;
  unsigned lane, sub, simp;
  bool active;
  const CtPaths<D>* P;

  // by all threads of the block
  __device__ __forceinline__ CtLane(const CtGeom& g, CtPaths<D>& paths) {
    lane = threadIdx.x & 31;
    sub = lane / kSimp;
    simp = lane % kSimp;
    active = sub < kCubes;
    P = &paths;
    if (threadIdx.x < 32) {
      unsigned c = 0;
      for (int i = 0; i <= D; ++i) {
        paths.corner[i][lane] = c;
        paths.off[i][lane] = ct_corner_step(g, c);
        if (i < D) c |= 1u << g.perm[simp][i];
      }
    }
    __syncthreads();
  }
  // bit i: path vertex i positive, given the cube's corner signs
  __device__ __forceinline__ unsigned signs(unsigned sgn) const {
    unsigned ps = 0;
#pragma unroll
    for (int i = 0; i <= D; ++i) ps |= ((sgn >> P->corner[i][lane]) & 1u) << i;
    return ps;
  }
  __device__ __forceinline__ unsigned corner(int i) const { return P->corner[i][lane]; }
  // feature index of the crossing edge between path vertices a and b of the
  // cube at local vertex base
  __device__ __forceinline__ unsigned node(unsigned long long base, const unsigned short* __restrict__ mask,
                                           const unsigned* __restrict__ voff, int a, int b) const {
    const int lo = min(a, b), hi = max(a, b);
    const unsigned long long v = base + P->off[lo][lane];
    const unsigned dir = P->corner[hi][lane] ^ P->corner[lo][lane];
    return __ldg(voff + v) + __popc((unsigned)__ldg(mask + v) & ((1u << (dir - 1)) - 1u));
  }
};

// The sides of a simplex's sign split in path order: `few` the vertices of the
// smaller side (of two positives and two negatives the positives), `rest` the
// others; n: how many few has (0: not crossed).
template <int D>
struct CtSplit {
  unsigned few, rest;
  int n;
  __device__ __forceinline__ explicit CtSplit(unsigned ps) {
    constexpr unsigned kAll = (1u << (D + 1)) - 1u;
    const int np = __popc(ps);
    const bool pos = 2 * np <= D + 1;
    n = pos ? np : D + 1 - np;
    few = pos ? ps : ps ^ kAll;
    rest = few ^ kAll;
  }
};

__device__ __forceinline__ int ct_pop(unsigned& bits) {
  const int i = __ffs(bits) - 1;
  bits &= bits - 1;
  return i;
}

// (2D+t) where the reference's sequential patching first meets each node whose
// edge starts on an upper boundary face: (cube base, permutation index,
// position in the marching enumeration), minimised over every meeting.  The
// marching functions meet the lone vertex with the others in order, or
// positives outer and others inner.
__global__ void ct_first_kernel(CtGeom g, const unsigned long long* __restrict__ list, const unsigned* list_cnt,
                                const unsigned short* __restrict__ mask, const unsigned* __restrict__ voff,
                                unsigned long long* __restrict__ first) {
  __shared__ CtPaths<3> paths;
  const CtLane<3> ln(g, paths);
  const unsigned nl = *list_cnt;
  const unsigned long long warp = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  for (unsigned long long it = warp * ln.kCubes + ln.sub; ln.active && it < nl; it += nwarps * ln.kCubes) {
    const unsigned long long w = list[it];
    const unsigned long long base = w >> kCtBaseShift;
    const unsigned upper = (unsigned)(w >> 16) & 0xFu;
    const CtSplit<3> x(ln.signs((unsigned)w & 0xFFFFu));
    int k = 0;
    for (unsigned f = x.few; f;) {
      const int a = ct_pop(f);
      for (unsigned r = x.rest; r; ++k) {
        const int b = ct_pop(r);
        if (!(ln.corner(min(a, b)) & upper)) continue;  // the edge starts at a hypercube base
        const unsigned nd = ln.node(base, mask, voff, a, b);
        const unsigned long long key = ((base * 6ull) + (unsigned long long)ln.simp) * 4ull + (unsigned long long)k;
        atomicMin(first + nd, key);
      }
    }
  }
}

__device__ __forceinline__ void ct_sort4(unsigned* v, int k) {
  for (int i = 1; i < k; ++i)
    for (int j = i; j > 0 && v[j - 1] > v[j]; --j) {
      const unsigned x = v[j - 1];
      v[j - 1] = v[j];
      v[j] = x;
    }
}

__device__ __forceinline__ void ct_order(unsigned& a, unsigned& b) {
  const unsigned lo = min(a, b);
  b = max(a, b);
  a = lo;
}

// row `slot` of the cells, its D entries ascending, counted at its leading node
template <int D>
__device__ __forceinline__ void ct_put_cell(unsigned* __restrict__ cells, unsigned long long slot, unsigned cap,
                                            unsigned* __restrict__ bcount, unsigned a, unsigned b, unsigned c,
                                            unsigned d) {
  if constexpr (D == 4) {
    ct_order(a, b), ct_order(c, d), ct_order(a, c), ct_order(b, d), ct_order(b, c);
    if (slot < cap) {
      reinterpret_cast<uint4*>(cells)[slot] = make_uint4(a, b, c, d);
      atomicAdd(bcount + a, 1u);
    }
  } else {
    ct_order(a, b), ct_order(b, c), ct_order(a, b);
    if (slot < cap) {
      cells[3 * slot] = a;
      cells[3 * slot + 1] = b;
      cells[3 * slot + 2] = c;
      atomicAdd(bcount + a, 1u);
    }
  }
}

// Marching tetrahedra (2D+t) / pentatopes (3D+t) on the listed cubes, one
// Kuhn simplex per lane: up to three cells each.  A warp reserves the slots of
// kCtBatch rounds at once: the signs alone give the number of cells, and the
// counter takes one atomic at a time.  Bound by the gathers of ranks and masks.
// 96^3 x 6 double, 7.5 million tets: 938 us with the joins, paths indexed in
// the kernel's parameters and an atomic per warp and round, now 89.
template <int D>
__global__ void __launch_bounds__(256) ct_cells_kernel(
    CtGeom g, const unsigned long long* __restrict__ list, const unsigned* list_cnt,
    const unsigned short* __restrict__ mask, const unsigned* __restrict__ voff,
    const unsigned long long* __restrict__ first, unsigned n, unsigned* __restrict__ cells, unsigned long long* cnt,
    unsigned cap, unsigned* __restrict__ bcount) {
  constexpr int kCtBatch = 8;
  __shared__ CtPaths<D> paths;
  const CtLane<D> ln(g, paths);
  const unsigned lane = ln.lane, nl = *list_cnt;
  const unsigned long long warp = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  for (unsigned long long r0 = warp * kCtBatch; r0 * ln.kCubes < nl; r0 += nwarps * kCtBatch) {
    unsigned mine = 0;
    for (int r = 0; r < kCtBatch; ++r) {
      const unsigned long long it = (r0 + r) * ln.kCubes + ln.sub;
      if (!ln.active || it >= nl) break;
      const CtSplit<D> x(ln.signs((unsigned)list[it] & 0xFFFFu));
      mine += x.n == 0 ? 0u : x.n == 1 ? 1u : (unsigned)D - 1u;
    }
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const unsigned wtot = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long wbase = 0;
    if (lane == 31 && wtot) wbase = atomicAdd(cnt, (unsigned long long)wtot);
    unsigned long long slot = __shfl_sync(0xffffffffu, wbase, 31) + incl - mine;
    for (int r = 0; r < kCtBatch; ++r) {
      const unsigned long long it = (r0 + r) * ln.kCubes + ln.sub;
      if (!ln.active || it >= nl) break;
      const unsigned long long w = list[it];
      const unsigned long long base = w >> kCtBaseShift;
      const CtSplit<D> x(ln.signs((unsigned)w & 0xFFFFu));
      if (x.n == 0) continue;
      unsigned few = x.few, rest = x.rest;
      if (x.n == 1) {  // 1-vs-rest: one cell
        const int a = ct_pop(few);
        unsigned nd[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < D; ++k) nd[k] = ln.node(base, mask, voff, a, ct_pop(rest));
        ct_put_cell<D>(cells, slot++, cap, bcount, nd[0], nd[1], nd[2], nd[3]);
      } else if constexpr (D == 3) {  // 2D+t 2-2 split: the quad cut along the diagonal from the
                                      // node the reference numbered first
        const int p0 = ct_pop(few), p1 = ct_pop(few), q0 = ct_pop(rest), q1 = ct_pop(rest);
        unsigned nd[4] = {ln.node(base, mask, voff, p0, q0), ln.node(base, mask, voff, p0, q1),
                          ln.node(base, mask, voff, p1, q0), ln.node(base, mask, voff, p1, q1)};
        unsigned long long key[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned long long f = first[nd[k]];
          key[k] = f == ~0ull ? (unsigned long long)nd[k] : (unsigned long long)n + f;
        }
#pragma unroll
        for (int i = 1; i < 4; ++i)
#pragma unroll
          for (int j = i; j > 0; --j)
            if (key[j - 1] > key[j]) {
              const unsigned long long kx = key[j - 1];
              key[j - 1] = key[j];
              key[j] = kx;
              const unsigned nx = nd[j - 1];
              nd[j - 1] = nd[j];
              nd[j] = nx;
            }
        ct_put_cell<D>(cells, slot++, cap, bcount, nd[0], nd[1], nd[2], 0);
        ct_put_cell<D>(cells, slot++, cap, bcount, nd[0], nd[2], nd[3], 0);
      } else {  // pentatope 2-3 split
        const int a = ct_pop(few), b = ct_pop(few);
        unsigned T0[3], T1[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int c = ct_pop(rest);
          T0[k] = ln.node(base, mask, voff, a, c);
          T1[k] = ln.node(base, mask, voff, b, c);
        }
        ct_put_cell<D>(cells, slot++, cap, bcount, T0[0], T0[1], T0[2], T1[2]);
        ct_put_cell<D>(cells, slot++, cap, bcount, T0[0], T0[1], T1[1], T1[2]);
        ct_put_cell<D>(cells, slot++, cap, bcount, T0[0], T1[0], T1[1], T1[2]);
      }
    }
  }
}

__global__ void ct_iota_kernel(unsigned* __restrict__ v, unsigned n) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

__global__ void ct_fill_u64_kernel(unsigned long long* __restrict__ v, unsigned long long x, unsigned n) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = x;
}

// Lexicographic order of the cells.  Each row is sorted, so the rows fall
// into buckets by their leading node: counts per leading node, a scan, a
// scatter into the buckets, then a small sort of each bucket's rows (a few
// rows: the cells at one crossing edge).
__global__ void ct_bucket_count_kernel(const unsigned* __restrict__ cells, unsigned m, int k,
                                       unsigned* __restrict__ bcount) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    atomicAdd(bcount + cells[(size_t)i * k], 1u);
}

__global__ void ct_bucket_scatter_kernel(const unsigned* __restrict__ cells, unsigned m, int k,
                                         const unsigned* __restrict__ boff, unsigned* __restrict__ bcur,
                                         unsigned* __restrict__ out) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const unsigned* c = cells + (size_t)i * k;
    const unsigned a = c[0];
    const unsigned dst = boff[a] + atomicAdd(bcur + a, 1u);
    for (int j = 0; j < k; ++j) out[(size_t)dst * k + j] = c[j];
  }
}

__device__ __forceinline__ bool ct_row_less(const unsigned* x, const unsigned* y, int k) {
  for (int j = 1; j < k; ++j)
    if (x[j] != y[j]) return x[j] < y[j];
  return false;
}

// Sorts each bucket's rows by their remaining entries: a block takes the buckets
// of kSortNodes leading nodes, copies their rows to shared memory, and a thread
// per row counts the rows of its bucket below it.  Without uniq, equal rows
// (duplicate cells) raise bit 1 of *err; with uniq, they are dropped (the unique
// rows stay at the start of the bucket, their count in uniq[a]).  Blocks whose
// rows do not fit sort each bucket by insertion where it lies.  96^3 x 6 double,
// 7.5 million tets: 480 us when every bucket was sorted that way by one thread,
// now 112.
constexpr int kSortNodes = 128;
constexpr unsigned kSortRows = 1536;

template <int K>
__global__ void __launch_bounds__(kCtThreads) ct_bucket_sort_kernel(unsigned* __restrict__ rows,
                                                                    const unsigned* __restrict__ boff, unsigned n,
                                                                    unsigned* err, unsigned* __restrict__ uniq) {
  __shared__ unsigned s_row[K][kSortRows];
  __shared__ unsigned s_off[kSortNodes + 1], s_uniq[kSortNodes];
  __shared__ unsigned char s_first[kSortRows];
  const unsigned a0 = blockIdx.x * kSortNodes, na = min((unsigned)kSortNodes, n - a0);
  for (unsigned i = threadIdx.x; i <= na; i += kCtThreads) s_off[i] = boff[a0 + i];
  if (threadIdx.x < kSortNodes) s_uniq[threadIdx.x] = 0;
  __syncthreads();
  const unsigned lo = s_off[0], cnt = s_off[na] - lo;
  if (cnt > kSortRows) {
    for (unsigned a = threadIdx.x; a < na; a += kCtThreads) {
      const unsigned first = s_off[a], last = s_off[a + 1];
      for (unsigned i = first + 1; i < last; ++i) {
        unsigned cur[K];
        for (int j = 0; j < K; ++j) cur[j] = rows[(size_t)i * K + j];
        unsigned p = i;
        while (p > first && ct_row_less(cur, rows + (size_t)(p - 1) * K, K)) {
          for (int j = 0; j < K; ++j) rows[(size_t)p * K + j] = rows[(size_t)(p - 1) * K + j];
          --p;
        }
        for (int j = 0; j < K; ++j) rows[(size_t)p * K + j] = cur[j];
      }
      unsigned w = first;
      for (unsigned i = first; i < last; ++i) {
        if (i > first && !ct_row_less(rows + (size_t)(w - 1) * K, rows + (size_t)i * K, K)) {
          if (!uniq) atomicOr(err, 2u);
          continue;
        }
        if (w != i)
          for (int j = 0; j < K; ++j) rows[(size_t)w * K + j] = rows[(size_t)i * K + j];
        ++w;
      }
      if (uniq) uniq[a0 + a] = w - first;
    }
    return;
  }
  for (unsigned i = threadIdx.x; i < cnt * K; i += kCtThreads) s_row[i % K][i / K] = rows[(size_t)lo * K + i];
  __syncthreads();
  // -1, 0, 1: row x against row y of the same bucket
  auto order = [&](unsigned x, unsigned y) {
#pragma unroll
    for (int j = 1; j < K; ++j)
      if (s_row[j][x] != s_row[j][y]) return s_row[j][x] < s_row[j][y] ? -1 : 1;
    return 0;
  };
  if (uniq) {
    for (unsigned i = threadIdx.x; i < cnt; i += kCtThreads) {
      const unsigned a = s_row[0][i] - a0;
      bool first = true;
      for (unsigned y = s_off[a] - lo; y < i && first; ++y) first = order(y, i) != 0;
      s_first[i] = first;
      if (first) atomicAdd(&s_uniq[a], 1u);
    }
    __syncthreads();
  }
  for (unsigned i = threadIdx.x; i < cnt; i += kCtThreads) {
    if (uniq && !s_first[i]) continue;
    const unsigned a = s_row[0][i] - a0, first = s_off[a] - lo, last = s_off[a + 1] - lo;
    unsigned below = 0;
    for (unsigned y = first; y < last; ++y) {
      const int o = order(y, i);
      if (o < 0 && (!uniq || s_first[y])) ++below;
      if (!uniq && o == 0 && y < i) {  // keeps the rows distinct places
        atomicOr(err, 2u);
        ++below;
      }
    }
    const size_t dst = (size_t)lo + first + below;
    if constexpr (K == 4) {
      reinterpret_cast<uint4*>(rows)[dst] = make_uint4(s_row[0][i], s_row[1][i], s_row[2][i], s_row[3][i]);
    } else {
#pragma unroll
      for (int j = 0; j < K; ++j) rows[dst * K + j] = s_row[j][i];
    }
  }
  if (uniq && threadIdx.x < na) uniq[a0 + threadIdx.x] = s_uniq[threadIdx.x];
}

void launch_bucket_sort(unsigned* rows, const unsigned* boff, unsigned n, int k, unsigned* err, unsigned* uniq,
                        cudaStream_t st) {
  if (n == 0) return;
  auto kernel = k == 4 ? ct_bucket_sort_kernel<4> : ct_bucket_sort_kernel<3>;
  kernel<<<(n + kSortNodes - 1) / kSortNodes, kCtThreads, 0, st>>>(rows, boff, n, err, uniq);
}

// unique rows of every bucket to their place in the output (uoff: scanned
// unique counts)
__global__ void ct_bucket_compact_kernel(const unsigned* __restrict__ rows, const unsigned* __restrict__ boff,
                                         const unsigned* __restrict__ uoff, unsigned n, int k,
                                         unsigned* __restrict__ out) {
  for (unsigned a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
    const unsigned lo = boff[a], cnt = uoff[a + 1] - uoff[a], dst = uoff[a];
    for (unsigned i = 0; i < cnt; ++i)
      for (int j = 0; j < k; ++j) out[(size_t)(dst + i) * k + j] = rows[(size_t)(lo + i) * k + j];
  }
}

// Exclusive scan of n counters in place (n up to 2^32 - 1): per-block scans
// of 2048 entries with their totals, a scan of the totals, the block offsets
// added back.
constexpr int kScanPer = 8;  // entries per thread
__global__ void ct_scan_blocks_kernel(unsigned* __restrict__ a, unsigned n, unsigned* __restrict__ tot) {
  __shared__ unsigned btot;
  const unsigned long long b0 = (unsigned long long)blockIdx.x * kCtThreads * kScanPer;
  const unsigned long long t0 = b0 + (unsigned long long)threadIdx.x * kScanPer;
  unsigned v[kScanPer], sum = 0;
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    v[j] = t0 + j < n ? a[t0 + j] : 0u;
    sum += v[j];
  }
  unsigned run = ct_block_scan(sum, &btot);
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    if (t0 + j < n) a[t0 + j] = run;
    run += v[j];
  }
  if (threadIdx.x == 0) tot[blockIdx.x] = btot;
}

__global__ void ct_scan_add_kernel(unsigned* __restrict__ a, unsigned n, const unsigned* __restrict__ tot) {
  const unsigned long long b0 = (unsigned long long)blockIdx.x * kCtThreads * kScanPer;
  const unsigned add = tot[blockIdx.x];
  for (int j = threadIdx.x; j < kCtThreads * kScanPer; j += kCtThreads)
    if (b0 + j < n) a[b0 + j] += add;
}

unsigned grid_of(unsigned long long work, int threads, unsigned long long max_blocks) {
  unsigned long long b = (work + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (unsigned)b;
}

ftk2b_status cfail(ftk2b_ctx* ctx, ftk2b_status st, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  ctx->err = buf;
  return st;
}

#define C_TRY(call)                                                                             \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess)                                                                      \
      return cfail(ctx, e_ == cudaErrorMemoryAllocation ? FTK2B_OOM : FTK2B_CUDA_ERROR,          \
                   "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

enum {
  kBufField = 0, kBufPos, kBufMask, kBufBlk, kBufVoff, kBufSimp, kBufLam, kBufBary, kBufFirst, kBufParent,
  kBufCells, kBufKey0, kBufKey1, kBufVal0, kBufVal1, kBufHist, kBufCellsOut, kBufTrack, kBufCount, kBufList,
  kBufField2, kBufUpOff, kBufUpNbr, kBufBaseCells,
  // fiber surfaces on extruded meshes
  kBufFeTris, kBufFeEdges, kBufFeSimp, kBufFeLam, kBufFeBary, kBufFePhase, kBufFeDisc, kBufFeFlag, kBufFeHi,
  kBufFeLo, kBufCount_
};

template <typename T>
ftk2b_status run_contour(ftk2b_ctx* ctx, const CtGeom& g, const void* field, T thr, double q,
                         ftk2b_contour_result* res) {
  cudaStream_t st = ctx->stream;
  DevBuf* B = ctx->contour;
  const int d = g.d;
  const unsigned long long nblk = (g.nv + kCtBlock - 1) / kCtBlock;
  C_TRY(B[kBufPos].ensure(4 * ct_words(g)));
  C_TRY(B[kBufMask].ensure(2 * g.nv));
  C_TRY(B[kBufVoff].ensure(4 * g.nv));
  C_TRY(B[kBufBlk].ensure(4 * (nblk + 1)));
  C_TRY(B[kBufCount].ensure(64));
  auto* pos = static_cast<unsigned*>(B[kBufPos].p);
  auto* mask = static_cast<unsigned short*>(B[kBufMask].p);
  auto* voff = static_cast<unsigned*>(B[kBufVoff].p);
  auto* blk = static_cast<unsigned*>(B[kBufBlk].p);
  auto* counts = static_cast<unsigned*>(B[kBufCount].p);  // [0] n, [1] cells, [2] roots, [3] err
  auto* total64 = reinterpret_cast<unsigned long long*>(counts + 8);
  auto* cell64 = reinterpret_cast<unsigned long long*>(counts + 10);  // manifold cells (64-bit)
  const T* a = static_cast<const T*>(field);
  const unsigned sms = (unsigned)ctx->num_sms;

  // the mixed hypercubes, once: every later stage walks this list
  C_TRY(B[kBufList].ensure(8 * (g.ncube ? g.ncube : 1)));
  auto* list = static_cast<unsigned long long*>(B[kBufList].p);
  unsigned* list_cnt = counts + 4;

  C_TRY(cudaMemsetAsync(counts, 0, 64, st));
  C_TRY(cudaEventRecord(ctx->ev0, st));
  ct_sign_kernel<T><<<grid_of(g.nv, 4 * 256, 32ull * sms), 256, 0, st>>>(g, a, thr, q, pos);
  ct_mask_kernel<<<(unsigned)nblk, kCtThreads, 0, st>>>(g, pos, mask, blk, total64, list, list_cnt);
  C_TRY(launch_scan(blk, (unsigned)nblk, counts + 0, nullptr, st));
  ctx->launches += 3;
  unsigned long long n64 = 0;
  C_TRY(cudaMemcpyAsync(&n64, total64, 8, cudaMemcpyDeviceToHost, st));
  C_TRY(ctx->sync());
  // features are indexed with 32 bits
  if (n64 >= 0xFFFFFFF0ull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^32 - 16 crossing edges");
  const unsigned n = (unsigned)n64;
  const size_t ncap = n ? n : 1;
  C_TRY(B[kBufSimp].ensure(16 * ncap));
  C_TRY(B[kBufLam].ensure(16 * ncap));
  C_TRY(B[kBufBary].ensure(8 * ncap));
  C_TRY(B[kBufParent].ensure(4 * ncap));
  C_TRY(B[kBufTrack].ensure(8 * ncap));
  if (d == 3) C_TRY(B[kBufFirst].ensure(8 * ncap));
  auto* simp = static_cast<unsigned long long*>(B[kBufSimp].p);
  auto* lam = static_cast<double*>(B[kBufLam].p);
  auto* bary = static_cast<float*>(B[kBufBary].p);
  auto* parent = static_cast<unsigned*>(B[kBufParent].p);
  auto* track = static_cast<unsigned long long*>(B[kBufTrack].p);
  auto* first = d == 3 ? static_cast<unsigned long long*>(B[kBufFirst].p) : nullptr;
  ct_emit_kernel<T><<<(unsigned)nblk, kCtThreads, 0, st>>>(g, a, thr, mask, blk, voff, simp, lam, bary, parent);
  if (n && g.ncube) {
    const unsigned long long most = kCtPer * ((1ull << d) - 1);  // one item a thread
    const dim3 grid((unsigned)nblk, (unsigned)std::min(most, (kJoinBlocks * sms + nblk - 1) / nblk));
    if (n >= kCtHooked) {
      const unsigned fgrid = grid_of(n, 256, 8ull * sms);
      ct_hook_kernel<<<(unsigned)nblk, kCtThreads, 0, st>>>(g, mask, voff, parent);
      uf_flatten_kernel<<<fgrid, 256, 0, st>>>(parent, n);
      ct_join_kernel<<<grid, kCtThreads, 0, st>>>(g, mask, voff, parent, counts + 3, true);
      uf_flatten_kernel<<<fgrid, 256, 0, st>>>(parent, n);
      ctx->launches += 4;
    }
    ct_join_kernel<<<grid, kCtThreads, 0, st>>>(g, mask, voff, parent, counts + 3, false);
    ctx->launches += 1;
  }
  ctx->launches += 1;
  const unsigned wgrid = 16u * sms;  // 8 warps per block
  if (d == 3 && n) {
    ct_fill_u64_kernel<<<grid_of(n, 256, 8ull * sms), 256, 0, st>>>(first, ~0ull, n);
    ct_first_kernel<<<wgrid, 256, 0, st>>>(g, list, list_cnt, mask, voff, first);
    ctx->launches += 2;
  }

  // manifold cells: a few per feature (about 2 per node on 2D+t, 4 to 6 on
  // 3D+t), grown once to the exact count if short
  unsigned cap = (unsigned)std::min<unsigned long long>(
      0x7FFFFFFFull, std::max<unsigned long long>(1024ull, (d == 4 ? 8ull : 4ull) * n));
  unsigned ncell = 0;
  const int kc = d;  // entries per cell: 3 (triangles) or 4 (tets)
  const unsigned nb = n + 1;  // bucket offsets, the last one the total
  C_TRY(B[kBufKey0].ensure(4ull * nb));  // counts of the leading nodes, then offsets
  auto* boff = static_cast<unsigned*>(B[kBufKey0].p);
  for (int attempt = 0; attempt < 2; ++attempt) {
    C_TRY(B[kBufCells].ensure((size_t)4 * kc * cap));
    auto* cells = static_cast<unsigned*>(B[kBufCells].p);
    C_TRY(cudaMemsetAsync(cell64, 0, 8, st));
    C_TRY(cudaMemsetAsync(boff, 0, 4ull * nb, st));
    auto cells_kernel = d == 3 ? ct_cells_kernel<3> : ct_cells_kernel<4>;
    cells_kernel<<<wgrid, 256, 0, st>>>(g, list, list_cnt, mask, voff, first, n, cells, cell64, cap, boff);
    ctx->launches += 1;
    unsigned long long nc64 = 0;
    C_TRY(cudaMemcpyAsync(&nc64, cell64, 8, cudaMemcpyDeviceToHost, st));
    C_TRY(ctx->sync());
    if (nc64 >= 0x7FFFFFFFull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^31 - 1 manifold cells");
    ncell = (unsigned)nc64;
    if (ncell <= cap) break;
    cap = ncell;
  }
  auto* cells = static_cast<unsigned*>(B[kBufCells].p);

  // lexicographic order of the cells: buckets by leading node, then each
  // bucket's rows sorted
  const unsigned ccap = ncell ? ncell : 1;
  const unsigned sblocks = (unsigned)((nb + kCtThreads * kScanPer - 1) / (kCtThreads * kScanPer));
  C_TRY(B[kBufKey1].ensure(4ull * nb));            // scatter cursors
  C_TRY(B[kBufVal0].ensure(4ull * (sblocks + 1)));  // scan block totals
  C_TRY(B[kBufCellsOut].ensure(4ull * kc * ccap));
  auto* bcur = static_cast<unsigned*>(B[kBufKey1].p);
  auto* btot = static_cast<unsigned*>(B[kBufVal0].p);
  auto* cells_out = static_cast<unsigned*>(B[kBufCellsOut].p);
  const unsigned cg = grid_of(ccap, 256, 16ull * sms);
  if (ncell) {
    C_TRY(cudaMemsetAsync(bcur, 0, 4ull * nb, st));
    ct_scan_blocks_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    C_TRY(launch_scan(btot, sblocks, nullptr, nullptr, st));
    ct_scan_add_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    ct_bucket_scatter_kernel<<<cg, 256, 0, st>>>(cells, ncell, kc, boff, bcur, cells_out);
    launch_bucket_sort(cells_out, boff, n, kc, counts + 3, nullptr, st);
    ctx->launches += 5;
  }
  if (n) {
    C_TRY(launch_uf_label(parent, counts + 0, n, track, counts + 2, st));
    ctx->launches += 1;
  }
  C_TRY(cudaEventRecord(ctx->ev1, st));

  // results to the host
  unsigned hc[4] = {0, 0, 0, 0};
  C_TRY(cudaMemcpyAsync(hc, counts, 16, cudaMemcpyDeviceToHost, st));
  res->n_features = n;
  res->cell_dim = d - 1;
  res->n_cells = ncell;
  res->simplices = static_cast<uint64_t*>(host_alloc(16 * ncap));
  res->lambda = static_cast<double*>(host_alloc(16 * ncap));
  res->barycentric = static_cast<float*>(host_alloc(8 * ncap));
  res->track_id = static_cast<uint64_t*>(host_alloc(8 * ncap));
  res->scalar = static_cast<float*>(host_alloc(4 * ncap));
  res->cells = static_cast<uint32_t*>(host_alloc(4ull * kc * ccap));
  if (!res->simplices || !res->lambda || !res->barycentric || !res->track_id || !res->scalar || !res->cells)
    return cfail(ctx, FTK2B_OOM, "host result allocation failed");
  C_TRY(ctx->sync());
  C_TRY(copy_to_host(ctx, {{res->simplices, simp, 16ull * n},
                           {res->lambda, lam, 16ull * n},
                           {res->barycentric, bary, 8ull * n},
                           {res->track_id, track, 8ull * n},
                           {res->cells, cells_out, 4ull * kc * ncell}}));
  if (hc[3] & 1u) return cfail(ctx, FTK2B_CUDA_ERROR, "union-find did not settle");
  if (hc[3] & 2u) return cfail(ctx, FTK2B_CUDA_ERROR, "duplicate manifold cell");
  const float sc = (float)thr;
  host_parallel(n, 4ull * n, [&](size_t b, size_t e) { std::fill(res->scalar + b, res->scalar + e, sc); });
  res->n_tracks = hc[2];
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  res->device_ms = ms;
  return FTK2B_OK;
}

// ---------------------------------------------------------------------------
// Fiber surfaces: FiberPredicate<T> on a regular 3D+t mesh (predicate.hpp:
// 341-362; form_general_manifold_patches with k = 2, engine.hpp:1341-1418).
// Features are the mesh triangles where both fields minus their thresholds
// have the origin inside (simulation of simplicity, 2-D).  Every triangle of
// the Freudenthal mesh is (c, c + a, c + b) for corner masks 0 < a < b, a a
// subset of b (50 types in a 4-cube), so triangles in simplex order are
// (c, a, b) in vertex order, then a, then b as binary numbers: ranks again
// come from per-vertex masks and a scan.  The reference's node code
// (v_min << 24 | a << 4 | b, mesh.hpp:736-749) orders triangles the same way,
// so its star centres are the smallest ranks.

struct FsTables {
  unsigned char ta[50], tb[50];  // corner masks of the second and third vertex, by type
  unsigned char idx[16][16];     // type of (a, b), 255 where (a, b) is no triangle
};

// four bit planes, interleaved by word: of component j, plane 2j positive
// (quantised >= 1) and plane 2j + 1 negative (<= -1); zero leaves both clear
template <typename T>
__global__ void fs_class_kernel(CtGeom g, const T* __restrict__ f0, const T* __restrict__ f1, T t0, T t1,
                                double q, uint4* __restrict__ cls) {
  const unsigned lane = threadIdx.x & 31;
  T v[4][2];
  ct_each_word(
      g.nv,
      [&](unsigned long long i, int j) {
        const unsigned long long k = ct_index(g, i);
        v[j][0] = __ldg(f0 + k);
        v[j][1] = __ldg(f1 + k);
      },
      [&](unsigned long long w, int j) {
        const bool in = 32 * w + lane < g.nv;
        unsigned p[4];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const T y = fp<T>::sub(v[j][k], k ? t1 : t0);
          const double x = in ? __dadd_rn(__dmul_rn((double)y, q), y > T(0) ? 0.5 : -0.5) : 0.0;
          p[2 * k] = __ballot_sync(0xffffffffu, x >= 1.0);
          p[2 * k + 1] = __ballot_sync(0xffffffffu, x <= -1.0);
        }
        if (lane == 0) cls[w] = make_uint4(p[0], p[1], p[2], p[3]);
      });
}

template <typename T>
__device__ __forceinline__ void fs_values(const CtGeom& g, const T* f0, const T* f1, T t0, T t1,
                                          unsigned long long ai, unsigned long long gid, int a, int b, T v[3][2]) {
  const unsigned long long ao[3] = {0ull, g.aoff[a], g.aoff[b]}, go[3] = {0ull, g.goff[a], g.goff[b]};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    v[i][0] = ct_adj(g, f0, ai + ao[i], gid + go[i], t0);
    v[i][1] = ct_adj(g, f1, ai + ao[i], gid + go[i], t1);
  }
}

// Per vertex: bit t of the 50-bit mask = triangle type t from this vertex is a
// feature.  One component of one strict sign at all three vertices keeps the
// origin outside whatever the ties (exact pre-test); the rest go through the
// exact 2-D test.
//
// A warp takes 32 consecutive vertices; lanes e and 16 + e hold the planes of
// the two components at their corners e.  What all corners share every
// triangle shares, so most warps are done after an AND over the lanes; in the
// others a lane takes a triangle type and finds the vertices where its corners
// share nothing, and these triangles are listed in shared memory and tested by
// full warps.  Vertices whose hypercube is left after the first step are listed
// for the cells.  96^3 x 8 double: 507 us with two class loads per triangle and
// vertex and the exact test where it came up, 128 with the sixteen classes in a
// register, now 95.
template <typename T>
__global__ void __launch_bounds__(kCtThreads) fs_mask_kernel(
    CtGeom g, FsTables tb, const T* __restrict__ f0, const T* __restrict__ f1, T t0, T t1, double q,
    const uint4* __restrict__ cls, unsigned long long* __restrict__ mask, unsigned* __restrict__ blk,
    unsigned long long* __restrict__ total64, unsigned* __restrict__ cand, unsigned* __restrict__ cand_cnt) {
  __shared__ unsigned n_list[kCtPer], s_at;
  __shared__ unsigned long long s_mask[kCtThreads], s_gid[kCtThreads], s_ai[kCtThreads];
  __shared__ unsigned short s_list[kCtThreads * 50];  // vertex of the share << 6 | triangle type
  __shared__ unsigned char s_ab[64];                  // corners a << 4 | b of a triangle type
  const unsigned tid = threadIdx.x, lane = tid & 31, full = 0xffffffffu;
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock + tid;
  if (tid < 64) s_ab[tid] = tid < 50 ? (unsigned char)(tb.ta[tid] << 4 | tb.tb[tid]) : 0;
  if (tid < kCtPer) n_list[tid] = 0;
  const unsigned e = lane & 15u;
  unsigned n0[kCtPer], n1[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long w0 = i0 - lane + j * kCtThreads;
    n0[j] = n1[j] = full;
    if (w0 < g.nv) {
      const unsigned long long o = w0 + ct_corner_step(g, e);
      const uint2* p = reinterpret_cast<const uint2*>(cls + o / 32) + (lane >> 4);
      const uint2 lo = p[0], hi = p[2];
      n0[j] = __funnelshift_r(lo.x, hi.x, (unsigned)o & 31u);
      n1[j] = __funnelshift_r(lo.y, hi.y, (unsigned)o & 31u);
    }
  }
  __syncthreads();
  unsigned rank[kCtPer], cube = 0;  // feature triangles, listed cubes << 16
#pragma unroll 1
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long i = i0 + j * kCtThreads;
    unsigned x0 = n0[0], x1 = n1[0];
#pragma unroll
    for (int k = 1; k < kCtPer; ++k)
      if (j == k) x0 = n0[k], x1 = n1[k];
    // vertices that share a sign with all corners `out` does not excuse
    auto sharing = [&](unsigned out) {
      unsigned x = x0 | out, y = x1 | out;
#pragma unroll
      for (int s = 8; s; s >>= 1) {
        x &= __shfl_xor_sync(full, x, s);
        y &= __shfl_xor_sync(full, y, s);
      }
      x |= y;
      return x | __shfl_xor_sync(full, x, 16);
    };
    unsigned left = ~sharing(0u) & __ballot_sync(full, i < g.nv);
    s_mask[tid] = 0;
    if (left) {
      unsigned long long c[4];
      ct_coords(g, i, c);
      const unsigned inb = i < g.nv ? ct_inbounds(g, c) : 0u;
      unsigned in[4], in_e = full;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        in[k] = __ballot_sync(full, (inb >> k) & 1u);
        if ((e >> k) & 1u) in_e &= in[k];
      }
      left &= ~sharing(~in_e);
      if ((left >> lane) & 1u) {
        if (inb == 15u) cube |= 1u << j;
        s_gid[tid] = ct_gid(g, c);
        s_ai[tid] = ct_aidx(g, c);
      }
      const unsigned c0 = __shfl_sync(full, x0, 0), c1 = __shfl_sync(full, x1, 0);
      const unsigned c2 = __shfl_sync(full, x0, 16), c3 = __shfl_sync(full, x1, 16);
      for (unsigned t = lane; t < 64; t += 32) {
        const unsigned a = s_ab[t] >> 4, b = s_ab[t] & 15u;
        unsigned common = c0 & __shfl_sync(full, x0, a) & __shfl_sync(full, x0, b);
        common |= c1 & __shfl_sync(full, x1, a) & __shfl_sync(full, x1, b);
        common |= c2 & __shfl_sync(full, x0, 16 + a) & __shfl_sync(full, x0, 16 + b);
        common |= c3 & __shfl_sync(full, x1, 16 + a) & __shfl_sync(full, x1, 16 + b);
        unsigned open = t < 50 ? left & ~common : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((b >> k) & 1u) open &= in[k];
        if (open) {
          unsigned at = atomicAdd(&n_list[j], (unsigned)__popc(open));
          for (; open; open &= open - 1) s_list[at++] = (unsigned short)((tid - lane + __ffs(open) - 1) << 6 | t);
        }
      }
    }
    __syncthreads();
    const unsigned n = n_list[j];
    unsigned long long m = 0;
    if (n) {  // uniform over the block
      for (unsigned k = tid; k < n; k += kCtThreads) {
        const unsigned x = s_list[k] >> 6, t = s_list[k] & 63u;
        T v[3][2];
        fs_values(g, f0, f1, t0, t1, s_ai[x], s_gid[x], s_ab[t] >> 4, s_ab[t] & 15u, v);
        if (sos_inside2<T>(v, q)) atomicOr(&s_mask[x], 1ull << t);
      }
      __syncthreads();
      m = s_mask[tid];
    }
    if (i < g.nv) mask[i] = m;
    const unsigned r = (unsigned)__popcll(m) | ((cube >> j) & 1u) << 16;
#pragma unroll
    for (int k = 0; k < kCtPer; ++k)
      if (j == k) rank[k] = r;
  }
  const unsigned n = ct_block_ranks(rank);
  if (tid == 0) {
    blk[blockIdx.x] = n & 0xFFFFu;
    if (n & 0xFFFFu) atomicAdd(total64, (unsigned long long)(n & 0xFFFFu));
    if (n >> 16) s_at = atomicAdd(cand_cnt, n >> 16);
  }
  if (n >> 16 == 0) return;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kCtPer; ++j)
    if ((cube >> j) & 1u) cand[s_at + (rank[j] >> 16)] = (unsigned)(i0 + j * kCtThreads);
}

// The feature triangles of a block's vertices, a thread per triangle, listed
// in rank order in shared memory first.  voff (first rank) is written where a
// vertex has triangles.
template <typename T>
__global__ void __launch_bounds__(kCtThreads) fs_emit_kernel(
    CtGeom g, FsTables tb, const T* __restrict__ f0, const T* __restrict__ f1, T t0, T t1,
    const unsigned long long* __restrict__ mask, const unsigned* __restrict__ blk_off, unsigned* __restrict__ voff,
    unsigned long long* __restrict__ simp, double* __restrict__ lam, float* __restrict__ bary) {
  __shared__ unsigned short s_list[kCtThreads * 50];  // vertex of the share << 6 | triangle type
  __shared__ unsigned s_end[kCtPer];
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kCtBlock;
  const unsigned base = blk_off[blockIdx.x];
  unsigned long long m[kCtPer];
  unsigned rank[kCtPer], cnt[kCtPer];
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned long long i = i0 + j * kCtThreads + threadIdx.x;
    m[j] = i < g.nv ? mask[i] : 0ull;
    rank[j] = cnt[j] = (unsigned)__popcll(m[j]);
  }
  if (ct_block_ranks(rank) == 0) return;
#pragma unroll
  for (int j = 0; j < kCtPer; ++j)
    if (threadIdx.x == kCtThreads - 1) s_end[j] = rank[j] + cnt[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kCtPer; ++j) {
    const unsigned lo = j ? s_end[j - 1] : 0u, hi = s_end[j];
    if (lo == hi) continue;  // uniform over the block
    if (m[j]) voff[i0 + j * kCtThreads + threadIdx.x] = base + rank[j];
    unsigned w = rank[j] - lo;
    for (unsigned long long x = m[j]; x; x &= x - 1)
      s_list[w++] = (unsigned short)(threadIdx.x << 6 | (__ffsll(x) - 1));
    __syncthreads();
    for (unsigned k = threadIdx.x; k < hi - lo; k += kCtThreads) {
      const unsigned t = s_list[k] & 63u;
      const int a = tb.ta[t], b = tb.tb[t];
      unsigned long long c[4];
      ct_coords(g, i0 + j * kCtThreads + (s_list[k] >> 6), c);
      const unsigned long long gid = ct_gid(g, c);
      T v[3][2];
      fs_values(g, f0, f1, t0, t1, ct_aidx(g, c), gid, a, b, v);
      T l[3];
      if (!solve_exact<2, T>(v, l))  // FiberPredicate keeps the centroid: (T)1.0 / 3.0
        for (int z = 0; z < 3; ++z) l[z] = (T)((double)(T)1.0 / 3.0);
      const size_t r = (size_t)base + lo + k;
      simp[3 * r] = gid;
      simp[3 * r + 1] = gid + g.goff[a];
      simp[3 * r + 2] = gid + g.goff[b];
      for (int z = 0; z < 3; ++z) {
        lam[3 * r + z] = (double)l[z];
        bary[3 * r + z] = (float)l[z];
      }
    }
    __syncthreads();
  }
}

// hypercubes with a feature triangle at one of their lower corners (a
// superset of the cubes whose pentatopes hold features), among the cubes the
// class pre-test left
__global__ void fs_list_kernel(CtGeom g, const unsigned long long* __restrict__ mask,
                               const unsigned* __restrict__ cand, const unsigned* __restrict__ cand_cnt,
                               unsigned long long* __restrict__ list, unsigned* __restrict__ cnt) {
  const unsigned lane = threadIdx.x & 31, n = *cand_cnt;
  const unsigned step = gridDim.x * blockDim.x;
  for (unsigned long long k0 = blockIdx.x * blockDim.x; k0 < n; k0 += step) {
    const unsigned long long k = k0 + threadIdx.x;
    const unsigned long long base = k < n ? cand[k] : 0u;
    bool any = false;
    if (k < n)
#pragma unroll
      for (int e = 0; e < 15; ++e) any |= mask[base + g.loff[e]] != 0ull;
    const unsigned bal = __ballot_sync(0xffffffffu, any);
    unsigned wbase = 0;
    if (lane == 0 && bal) wbase = atomicAdd(cnt, (unsigned)__popc(bal));
    wbase = __shfl_sync(0xffffffffu, wbase, 0);
    if (any) list[wbase + __popc(bal & ((1u << lane) - 1u))] = base;
  }
}

// One pentatope per lane (24 per listed cube): its feature triangles in rank
// order (the reference's code order), the star centre h_S = the first; per
// tet face (path vertex i left out), the face's feature triangles in order,
// h_T the first, and a triangle {h_S, h_T, n} for every later n, unless h_S is
// h_T or n (engine.hpp:1388-1413).  Two passes: count, reserve per warp, write.
__global__ void fs_cells_kernel(CtGeom g, FsTables tb, const unsigned long long* __restrict__ list,
                                const unsigned* list_cnt, const unsigned long long* __restrict__ mask,
                                const unsigned* __restrict__ voff, unsigned* __restrict__ cells,
                                unsigned long long* cnt, unsigned cap, unsigned* parent, unsigned* err) {
  const int lane = threadIdx.x & 31;
  const unsigned nl = *list_cnt;
  const unsigned long long warp = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  // triangle z of pentatope `lane`: its lowest corner's step and its type
  __shared__ unsigned long long s_off[10][24];
  __shared__ unsigned char s_type[10][24];
  if (threadIdx.x < 24) {
    int pe[5], z = 0;
    pe[0] = 0;
    for (int i = 0; i < 4; ++i) pe[i + 1] = pe[i] | (1 << g.perm[threadIdx.x][i]);
    for (int i = 0; i < 3; ++i)
      for (int j = i + 1; j < 4; ++j)
        for (int k = j + 1; k < 5; ++k, ++z) {
          s_off[z][threadIdx.x] = g.loff[pe[i]];
          s_type[z][threadIdx.x] = tb.idx[pe[j] ^ pe[i]][pe[k] ^ pe[i]];
        }
  }
  __syncthreads();
  for (unsigned long long it = warp; it < nl; it += nwarps) {
    unsigned rank[10], vset[10];
    int nn = 0;
    if (lane < 24) {
      const unsigned long long base = list[it];
      int z = 0;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i + 1; j < 4; ++j)
#pragma unroll
          for (int k = j + 1; k < 5; ++k, ++z) {
            const unsigned t = s_type[z][lane];
            const unsigned long long v = base + s_off[z][lane];
            const unsigned long long mv = __ldg(mask + v);
            if (!((mv >> t) & 1ull)) continue;
            unsigned rk = __ldg(voff + v) + (unsigned)__popcll(mv & ((1ull << t) - 1ull));
            unsigned vs = (1u << i) | (1u << j) | (1u << k);
            int p = nn++;
            while (p > 0 && rank[p - 1] > rk) {
              rank[p] = rank[p - 1];
              vset[p] = vset[p - 1];
              --p;
            }
            rank[p] = rk;
            vset[p] = vs;
          }
    }
    // pass 1: count
    unsigned mine = 0;
    if (nn >= 2) {
      const unsigned hs = rank[0];
      for (int f = 0; f < 5; ++f) {
        int seen = 0;
        unsigned ht = 0;
        for (int x = 0; x < nn; ++x) {
          if (vset[x] & (1u << f)) continue;
          if (seen++ == 0) {
            ht = rank[x];
            continue;
          }
          if (hs != ht && hs != rank[x]) ++mine;
        }
      }
    }
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const unsigned wtot = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long wbase = 0;
    if (lane == 31 && wtot) wbase = atomicAdd(cnt, (unsigned long long)wtot);
    wbase = __shfl_sync(0xffffffffu, wbase, 31);
    unsigned long long slot = wbase + incl - mine;
    // pass 2: write and join
    if (mine) {
      const unsigned hs = rank[0];
      for (int f = 0; f < 5; ++f) {
        int seen = 0;
        unsigned ht = 0;
        for (int x = 0; x < nn; ++x) {
          if (vset[x] & (1u << f)) continue;
          if (seen++ == 0) {
            ht = rank[x];
            continue;
          }
          if (hs == ht || hs == rank[x]) continue;
          unsigned tri[3] = {hs, ht, rank[x]};
          ct_sort4(tri, 3);
          if (slot < cap)
            for (int k = 0; k < 3; ++k) cells[(size_t)slot * 3 + k] = tri[k];
          ++slot;
          uf_unite_flat(parent, tri[0], tri[1], err);
          uf_unite_flat(parent, tri[0], tri[2], err);
        }
      }
    }
  }
}

template <typename T>
ftk2b_status run_fiber_surface(ftk2b_ctx* ctx, const CtGeom& g, const FsTables& tb, const void* fa,
                               const void* fb, T t0, T t1, double q, ftk2b_fiber_surface_result* res) {
  cudaStream_t st = ctx->stream;
  DevBuf* B = ctx->contour;
  const unsigned long long nblk = (g.nv + kCtBlock - 1) / kCtBlock;
  if (nblk >= 0xFFFFFFF0ull) return cfail(ctx, FTK2B_UNSUPPORTED, "mesh too large");
  C_TRY(B[kBufPos].ensure(16 * ct_words(g)));
  C_TRY(B[kBufHist].ensure(8 * g.nv));
  C_TRY(B[kBufVoff].ensure(4 * g.nv));
  C_TRY(B[kBufBlk].ensure(4 * (nblk + 1)));
  C_TRY(B[kBufCount].ensure(64));
  auto* cls = static_cast<uint4*>(B[kBufPos].p);
  auto* mask = static_cast<unsigned long long*>(B[kBufHist].p);
  auto* voff = static_cast<unsigned*>(B[kBufVoff].p);
  auto* blk = static_cast<unsigned*>(B[kBufBlk].p);
  auto* counts = static_cast<unsigned*>(B[kBufCount].p);  // [0] n, [1] cells, [2] roots, [3] err, [4] cubes
  auto* total64 = reinterpret_cast<unsigned long long*>(counts + 8);
  auto* cell64 = reinterpret_cast<unsigned long long*>(counts + 10);  // manifold cells (64-bit)
  const T* a0 = static_cast<const T*>(fa);
  const T* a1 = static_cast<const T*>(fb);
  const unsigned sms = (unsigned)ctx->num_sms;
  C_TRY(cudaMemsetAsync(counts, 0, 64, st));
  C_TRY(cudaEventRecord(ctx->ev0, st));
  C_TRY(B[kBufCells].ensure(4 * (g.ncube ? g.ncube : 1)));
  auto* cand = static_cast<unsigned*>(B[kBufCells].p);  // until the cells come
  fs_class_kernel<T><<<grid_of(g.nv, 4 * 256, 32ull * sms), 256, 0, st>>>(g, a0, a1, t0, t1, q, cls);
  fs_mask_kernel<T><<<(unsigned)nblk, kCtThreads, 0, st>>>(g, tb, a0, a1, t0, t1, q, cls, mask, blk, total64, cand,
                                                           counts + 5);
  C_TRY(launch_scan(blk, (unsigned)nblk, counts + 0, nullptr, st));  // counts[0]: feature count (labels)
  ctx->launches += 3;
  unsigned long long n64 = 0;
  C_TRY(cudaMemcpyAsync(&n64, total64, 8, cudaMemcpyDeviceToHost, st));
  C_TRY(ctx->sync());
  if (n64 >= 0xFFFFFFF0ull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^32 - 16 feature triangles");
  const unsigned n = (unsigned)n64;
  const size_t ncap = n ? n : 1;
  C_TRY(B[kBufSimp].ensure(24 * ncap));
  C_TRY(B[kBufLam].ensure(24 * ncap));
  C_TRY(B[kBufBary].ensure(12 * ncap));
  C_TRY(B[kBufParent].ensure(4 * ncap));
  C_TRY(B[kBufTrack].ensure(8 * ncap));
  auto* simp = static_cast<unsigned long long*>(B[kBufSimp].p);
  auto* lam = static_cast<double*>(B[kBufLam].p);
  auto* bary = static_cast<float*>(B[kBufBary].p);
  auto* parent = static_cast<unsigned*>(B[kBufParent].p);
  auto* track = static_cast<unsigned long long*>(B[kBufTrack].p);
  fs_emit_kernel<T><<<(unsigned)nblk, kCtThreads, 0, st>>>(g, tb, a0, a1, t0, t1, mask, blk, voff, simp, lam, bary);
  C_TRY(B[kBufList].ensure(8 * (g.ncube ? g.ncube : 1)));
  auto* list = static_cast<unsigned long long*>(B[kBufList].p);
  unsigned* list_cnt = counts + 4;
  fs_list_kernel<<<grid_of(g.ncube, 256, 8ull * sms), 256, 0, st>>>(g, mask, cand, counts + 5, list, list_cnt);
  ctx->launches += 2;

  unsigned cap = (unsigned)std::min<unsigned long long>(0x7FFFFFFFull, std::max<unsigned long long>(1024ull, 4ull * n));
  unsigned ncell = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    C_TRY(B[kBufCells].ensure((size_t)12 * cap));
    auto* cells = static_cast<unsigned*>(B[kBufCells].p);
    C_TRY(cudaMemsetAsync(counts + 1, 0, 12, st));
    C_TRY(cudaMemsetAsync(cell64, 0, 8, st));
    if (n) ct_iota_kernel<<<grid_of(n, 256, 8ull * sms), 256, 0, st>>>(parent, n);
    fs_cells_kernel<<<16u * sms, 256, 0, st>>>(g, tb, list, list_cnt, mask, voff, cells, cell64, cap, parent,
                                              counts + 3);
    ctx->launches += 2;
    unsigned long long nc64 = 0;
    C_TRY(cudaMemcpyAsync(&nc64, cell64, 8, cudaMemcpyDeviceToHost, st));
    C_TRY(ctx->sync());
    if (nc64 >= 0x7FFFFFFFull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^31 - 1 manifold triangles");
    ncell = (unsigned)nc64;
    if (ncell <= cap) break;
    cap = ncell;
  }
  auto* cells = static_cast<unsigned*>(B[kBufCells].p);

  // sorted, unique triangles: buckets by leading node, each sorted and made
  // unique, compacted
  const unsigned ccap = ncell ? ncell : 1;
  const unsigned nb = n + 1;
  const unsigned sblocks = (unsigned)((nb + kCtThreads * kScanPer - 1) / (kCtThreads * kScanPer));
  C_TRY(B[kBufKey0].ensure(4ull * nb));
  C_TRY(B[kBufKey1].ensure(4ull * nb));
  C_TRY(B[kBufVal0].ensure(4ull * (sblocks + 1)));
  C_TRY(B[kBufVal1].ensure(4ull * nb));
  C_TRY(B[kBufCellsOut].ensure(12ull * ccap));
  C_TRY(B[kBufMask].ensure(12ull * ccap));
  auto* boff = static_cast<unsigned*>(B[kBufKey0].p);
  auto* bcur = static_cast<unsigned*>(B[kBufKey1].p);
  auto* btot = static_cast<unsigned*>(B[kBufVal0].p);
  auto* uoff = static_cast<unsigned*>(B[kBufVal1].p);
  auto* rows = static_cast<unsigned*>(B[kBufCellsOut].p);
  auto* cells_out = static_cast<unsigned*>(B[kBufMask].p);
  const unsigned cg = grid_of(ccap, 256, 16ull * sms);
  unsigned nuniq = 0;
  if (ncell) {
    C_TRY(cudaMemsetAsync(boff, 0, 4ull * nb, st));
    C_TRY(cudaMemsetAsync(bcur, 0, 4ull * nb, st));
    C_TRY(cudaMemsetAsync(uoff, 0, 4ull * nb, st));
    ct_bucket_count_kernel<<<cg, 256, 0, st>>>(cells, ncell, 3, boff);
    ct_scan_blocks_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    C_TRY(launch_scan(btot, sblocks, nullptr, nullptr, st));
    ct_scan_add_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    ct_bucket_scatter_kernel<<<cg, 256, 0, st>>>(cells, ncell, 3, boff, bcur, rows);
    launch_bucket_sort(rows, boff, n, 3, counts + 3, uoff, st);
    ct_scan_blocks_kernel<<<sblocks, kCtThreads, 0, st>>>(uoff, nb, btot);
    C_TRY(launch_scan(btot, sblocks, nullptr, nullptr, st));
    ct_scan_add_kernel<<<sblocks, kCtThreads, 0, st>>>(uoff, nb, btot);
    ct_bucket_compact_kernel<<<grid_of(n, 128, 32ull * sms), 128, 0, st>>>(rows, boff, uoff, n, 3, cells_out);
    ctx->launches += 10;
    C_TRY(cudaMemcpyAsync(&nuniq, uoff + n, 4, cudaMemcpyDeviceToHost, st));
  }
  if (n) {
    C_TRY(launch_uf_label(parent, counts + 0, n, track, counts + 2, st));
    ctx->launches += 1;
  }
  C_TRY(cudaEventRecord(ctx->ev1, st));
  unsigned hc[4] = {0, 0, 0, 0};
  C_TRY(cudaMemcpyAsync(hc, counts, 16, cudaMemcpyDeviceToHost, st));
  C_TRY(ctx->sync());
  res->n_features = n;
  res->n_cells = nuniq;
  res->simplices = static_cast<uint64_t*>(host_alloc(24 * ncap));
  res->lambda = static_cast<double*>(host_alloc(24 * ncap));
  res->barycentric = static_cast<float*>(host_alloc(12 * ncap));
  res->track_id = static_cast<uint64_t*>(host_alloc(8 * ncap));
  res->scalar = static_cast<float*>(std::calloc(ncap, 4));
  res->cells = static_cast<uint32_t*>(host_alloc(12ull * (nuniq ? nuniq : 1)));
  if (!res->simplices || !res->lambda || !res->barycentric || !res->track_id || !res->scalar || !res->cells)
    return cfail(ctx, FTK2B_OOM, "host result allocation failed");
  C_TRY(copy_to_host(ctx, {{res->simplices, simp, 24ull * n},
                           {res->lambda, lam, 24ull * n},
                           {res->barycentric, bary, 12ull * n},
                           {res->track_id, track, 8ull * n},
                           {res->cells, cells_out, 12ull * nuniq}}));
  if (hc[3] & 1u) return cfail(ctx, FTK2B_CUDA_ERROR, "union-find did not settle");
  res->n_tracks = hc[2];
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  res->device_ms = ms;
  return FTK2B_OK;
}

// ---------------------------------------------------------------------------
// Level sets on ExtrudedSimplicialMesh(UnstructuredSimplicialMesh, L)
// (mesh.hpp:542-599): vertex ids v = s + t * S (S base vertices, layers
// t = 0 .. L), the field per vertex.  The mesh's edges from a lower vertex
// a + tS, in id order, are its spatial edges to b + tS (base edges a < b),
// its vertical edge to a + (t + 1)S and the prism diagonals to b + (t + 1)S
// (the Kuhn split of a prism over a sorted base cell joins v_a at t to v_b at
// t + 1 only for a < b), so ranks again come from a per-vertex mask over
// 2 deg(a) + 1 candidates and a scan.  The reference's first pass visits the
// spatial and vertical edges only (iterate_simplices(1)); the diagonals it
// meets while marching over the cells, which it visits by layer, base cell
// (in stored order, each sorted) and Kuhn index j (vertices v_0..v_j at t,
// v_j..v_k at t + 1), one worker at a time.

// One simplex of the sweep: path corners and signs.
struct CtSimplex {
  int pe[5];      // corner of path vertex i
  unsigned ps;    // bit i: path vertex i positive
  int npos;
};

// The crossing edges of a 1-vs-rest or 2D+t 2-2 split in the order the
// reference's marching functions meet them, as path-vertex pairs: the lone
// vertex with the others in order; positives outer, others inner.
__device__ __forceinline__ int ct_crossings(const CtSimplex& x, int nvtx, int* ea, int* eb) {
  int ne = 0;
  if (x.npos == 1 || x.npos == nvtx - 1) {
    const bool lone_pos = x.npos == 1;
    int lone = 0;
    for (int i = 0; i < nvtx; ++i)
      if ((((x.ps >> i) & 1u) != 0) == lone_pos) lone = i;
    for (int o = 0; o < nvtx; ++o)
      if (o != lone) {
        ea[ne] = lone;
        eb[ne] = o;
        ++ne;
      }
  } else {
    for (int a = 0; a < nvtx; ++a) {
      if (!((x.ps >> a) & 1u)) continue;
      for (int b = 0; b < nvtx; ++b) {
        if ((x.ps >> b) & 1u) continue;
        ea[ne] = a;
        eb[ne] = b;
        ++ne;
      }
    }
  }
  return ne;
}

struct CeGeom {
  int d;                       // spacetime dims: 3 (triangle base) or 4 (tet base)
  unsigned long long S, L;     // base vertices, layers
  unsigned long long nv;       // S * (L + 1)
  unsigned long long ncell;    // base cells
  const unsigned* up_off;      // CSR of base neighbours b > a: up_nbr[up_off[a] .. up_off[a + 1])
  const unsigned* up_nbr;
  const unsigned* cells;       // ncell * d sorted base vertex ids
};

__device__ __forceinline__ int ce_nbr_index(const CeGeom& g, unsigned a, unsigned b) {
  const unsigned lo = g.up_off[a], hi = g.up_off[a + 1];
  for (unsigned i = lo; i < hi; ++i)
    if (g.up_nbr[i] == b) return (int)(i - lo);
  return -1;
}

// mask bit of the edge (x, y), x < y, in x's candidate order
__device__ __forceinline__ int ce_bit(const CeGeom& g, unsigned long long x, unsigned long long y) {
  const unsigned long long t = x / g.S;
  const unsigned a = (unsigned)(x - t * g.S);
  const int deg = (int)(g.up_off[a + 1] - g.up_off[a]);
  if (y < (t + 1) * g.S) return ce_nbr_index(g, a, (unsigned)(y - t * g.S));
  if (y == x + g.S) return deg;
  return deg + 1 + ce_nbr_index(g, a, (unsigned)(y - (t + 1) * g.S));
}

__device__ __forceinline__ unsigned ce_node(const CeGeom& g, const unsigned long long* __restrict__ mask,
                                            const unsigned* __restrict__ voff, unsigned long long x,
                                            unsigned long long y) {
  const int bit = max(ce_bit(g, x, y), 0);  // every cell pair is a base edge, so the index exists
  return voff[x] + (unsigned)__popcll(mask[x] & ((1ull << bit) - 1ull));
}

template <typename T>
__global__ void ce_sign_kernel(CeGeom g, const T* __restrict__ a, T thr, double q, unsigned char* __restrict__ pos) {
  for (unsigned long long v = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; v < g.nv;
       v += (unsigned long long)gridDim.x * blockDim.x)
    pos[v] = ct_positive(fp<T>::sub(__ldg(a + v), thr), v, q) ? 1 : 0;
}

__global__ void ce_mask_kernel(CeGeom g, const unsigned char* __restrict__ pos, unsigned long long* __restrict__ mask,
                               unsigned* __restrict__ blk, unsigned long long* __restrict__ total64) {
  __shared__ unsigned tot;
  const unsigned long long v = blockIdx.x * (unsigned long long)kCtThreads + threadIdx.x;
  unsigned long long m = 0;
  if (v < g.nv) {
    const unsigned long long t = v / g.S;
    const unsigned a = (unsigned)(v - t * g.S);
    const unsigned lo = g.up_off[a], hi = g.up_off[a + 1];
    const int deg = (int)(hi - lo);
    const unsigned char p = pos[v];
    for (unsigned i = lo; i < hi; ++i)
      if (pos[g.up_nbr[i] + t * g.S] != p) m |= 1ull << (i - lo);
    if (t < g.L) {
      if (pos[v + g.S] != p) m |= 1ull << deg;
      for (unsigned i = lo; i < hi; ++i)
        if (pos[g.up_nbr[i] + (t + 1) * g.S] != p) m |= 1ull << (deg + 1 + (int)(i - lo));
    }
    mask[v] = m;
  }
  ct_block_scan((unsigned)__popcll(m), &tot);
  if (threadIdx.x == 0) {
    blk[blockIdx.x] = tot;
    atomicAdd(total64, (unsigned long long)tot);
  }
}

template <typename T>
__global__ void ce_emit_kernel(CeGeom g, const T* __restrict__ a, T thr, const unsigned long long* __restrict__ mask,
                               const unsigned* __restrict__ blk_off, unsigned* __restrict__ voff,
                               unsigned long long* __restrict__ simp, double* __restrict__ lam,
                               float* __restrict__ bary) {
  __shared__ unsigned tot;
  const unsigned long long v = blockIdx.x * (unsigned long long)kCtThreads + threadIdx.x;
  const unsigned long long m = v < g.nv ? mask[v] : 0ull;
  const unsigned base = blk_off[blockIdx.x] + ct_block_scan((unsigned)__popcll(m), &tot);
  if (v >= g.nv) return;
  voff[v] = base;
  if (!m) return;
  const unsigned long long t = v / g.S;
  const unsigned aa = (unsigned)(v - t * g.S);
  const unsigned lo = g.up_off[aa];
  const int deg = (int)(g.up_off[aa + 1] - lo);
  const T a0 = fp<T>::sub(__ldg(a + v), thr);
  unsigned r = base;
  for (int bit = 0; bit < 2 * deg + 1; ++bit) {
    if (!((m >> bit) & 1ull)) continue;
    unsigned long long y;
    if (bit < deg) y = g.up_nbr[lo + bit] + t * g.S;
    else if (bit == deg) y = v + g.S;
    else y = g.up_nbr[lo + bit - deg - 1] + (t + 1) * g.S;
    const T a1 = fp<T>::sub(__ldg(a + y), thr);
    T l0, l1;
    ct_solve(a0, a1, &l0, &l1);
    simp[2 * (size_t)r] = v;
    simp[2 * (size_t)r + 1] = y;
    lam[2 * (size_t)r] = (double)l0;
    lam[2 * (size_t)r + 1] = (double)l1;
    bary[2 * (size_t)r] = (float)l0;
    bary[2 * (size_t)r + 1] = (float)l1;
    ++r;
  }
}

// vertices (global ids, ascending) and signs of spacetime cell q = (t, c, j)
__device__ __forceinline__ void ce_cell(const CeGeom& g, const unsigned char* pos, unsigned long long q,
                                        unsigned long long* vid, unsigned* ps, int* npos) {
  const int d = g.d;
  const unsigned long long j = q % d, tc = q / d, c = tc % g.ncell, t = tc / g.ncell;
  const unsigned* cv = g.cells + c * d;
  int k = 0;
  for (int l = 0; l <= (int)j; ++l) vid[k++] = cv[l] + t * g.S;
  for (int l = (int)j; l < d; ++l) vid[k++] = cv[l] + (t + 1) * g.S;
  unsigned s = 0;
  int np = 0;
  for (int i = 0; i <= d; ++i) {
    const unsigned b = pos[vid[i]];
    s |= b << i;
    np += (int)b;
  }
  *ps = s;
  *npos = np;
}

__device__ __forceinline__ bool ce_late(const CeGeom& g, unsigned long long x, unsigned long long y) {
  // a diagonal: its ends lie on consecutive layers and it is not vertical
  return y >= (x / g.S + 1) * g.S && y != x + g.S;
}

// (2D+t) first meeting of every diagonal node: (cell order, marching position)
__global__ void ce_first_kernel(CeGeom g, const unsigned char* __restrict__ pos,
                                const unsigned long long* __restrict__ mask, const unsigned* __restrict__ voff,
                                unsigned long long* __restrict__ first) {
  const unsigned long long nsc = g.L * g.ncell * 3ull;
  for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; q < nsc;
       q += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long vid[5];
    unsigned ps;
    int npos;
    ce_cell(g, pos, q, vid, &ps, &npos);
    if (npos == 0 || npos == 4) continue;
    CtSimplex x;
    x.ps = ps;
    x.npos = npos;
    int ea[4], eb[4];
    const int ne = ct_crossings(x, 4, ea, eb);
    for (int k = 0; k < ne; ++k) {
      const unsigned long long lo = vid[min(ea[k], eb[k])], hi = vid[max(ea[k], eb[k])];
      if (!ce_late(g, lo, hi)) continue;
      atomicMin(first + ce_node(g, mask, voff, lo, hi), q * 4ull + (unsigned long long)k);
    }
  }
}

// marching on every spacetime cell, one per thread; slots reserved per warp
__global__ void ce_cells_kernel(CeGeom g, const unsigned char* __restrict__ pos,
                                const unsigned long long* __restrict__ mask, const unsigned* __restrict__ voff,
                                const unsigned long long* __restrict__ first, unsigned n,
                                unsigned* __restrict__ cells, unsigned long long* cnt, unsigned cap,
                                unsigned* parent, unsigned* err) {
  const int d = g.d, kc = d;
  const int lane = threadIdx.x & 31;
  const unsigned long long nsc = g.L * g.ncell * (unsigned long long)d;
  for (unsigned long long q0 = blockIdx.x * (unsigned long long)blockDim.x; q0 < nsc;
       q0 += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long q = q0 + threadIdx.x;
    unsigned cell[3][4];
    unsigned nodes[6];
    int nn = 0, ncell = 0;
    if (q < nsc) {
      unsigned long long vid[5];
      unsigned ps;
      int npos;
      ce_cell(g, pos, q, vid, &ps, &npos);
      CtSimplex x;
      x.ps = ps;
      x.npos = npos;
      auto node = [&](int i, int j) { return ce_node(g, mask, voff, vid[min(i, j)], vid[max(i, j)]); };
      if (npos != 0 && npos != d + 1) {
        if (npos == 1 || npos == d || d == 3) {
          int ea[6], eb[6];
          const int ne = ct_crossings(x, d + 1, ea, eb);
          for (int k = 0; k < ne; ++k) nodes[k] = node(ea[k], eb[k]);
          nn = ne;
          if (ne == d) {
            for (int k = 0; k < d; ++k) cell[0][k] = nodes[k];
            ncell = 1;
          } else {
            unsigned nd[4];
            unsigned long long key[4];
            for (int k = 0; k < 4; ++k) {
              nd[k] = nodes[k];
              const unsigned long long f = first[nd[k]];
              key[k] = f == ~0ull ? (unsigned long long)nd[k] : (unsigned long long)n + f;
            }
            for (int i = 1; i < 4; ++i)
              for (int j = i; j > 0 && key[j - 1] > key[j]; --j) {
                const unsigned long long kx = key[j - 1];
                key[j - 1] = key[j];
                key[j] = kx;
                const unsigned nx = nd[j - 1];
                nd[j - 1] = nd[j];
                nd[j] = nx;
              }
            cell[0][0] = nd[0], cell[0][1] = nd[1], cell[0][2] = nd[2];
            cell[1][0] = nd[0], cell[1][1] = nd[2], cell[1][2] = nd[3];
            ncell = 2;
          }
        } else {
          const bool two_pos = npos == 2;
          int two[2], three[3], n2 = 0, n3 = 0;
          for (int i = 0; i < 5; ++i) {
            if ((((ps >> i) & 1u) != 0) == two_pos) two[n2++] = i;
            else three[n3++] = i;
          }
          unsigned T0[3], T1[3];
          for (int t = 0; t < 3; ++t) {
            T0[t] = node(two[0], three[t]);
            T1[t] = node(two[1], three[t]);
          }
          cell[0][0] = T0[0], cell[0][1] = T0[1], cell[0][2] = T0[2], cell[0][3] = T1[2];
          cell[1][0] = T0[0], cell[1][1] = T0[1], cell[1][2] = T1[1], cell[1][3] = T1[2];
          cell[2][0] = T0[0], cell[2][1] = T1[0], cell[2][2] = T1[1], cell[2][3] = T1[2];
          for (int t = 0; t < 3; ++t) nodes[t] = T0[t], nodes[3 + t] = T1[t];
          nn = 6;
          ncell = 3;
        }
      }
    }
    unsigned incl = (unsigned)ncell;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const unsigned wtot = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long wbase = 0;
    if (lane == 31 && wtot) wbase = atomicAdd(cnt, (unsigned long long)wtot);
    wbase = __shfl_sync(0xffffffffu, wbase, 31);
    unsigned long long slot = wbase + incl - (unsigned)ncell;
    for (int c = 0; c < ncell; ++c, ++slot) {
      ct_sort4(cell[c], kc);
      if (slot < cap)
        for (int k = 0; k < kc; ++k) cells[(size_t)slot * kc + k] = cell[c][k];
    }
    for (int k = 1; k < nn; ++k) uf_unite(parent, nodes[0], nodes[k], err);
  }
}

template <typename T>
ftk2b_status run_contour_extruded(ftk2b_ctx* ctx, CeGeom g, const void* field, T thr, double q,
                                  ftk2b_contour_result* res) {
  cudaStream_t st = ctx->stream;
  DevBuf* B = ctx->contour;
  const int d = g.d, kc = d;
  const unsigned long long nblk = (g.nv + kCtThreads - 1) / kCtThreads;
  if (nblk >= 0xFFFFFFF0ull) return cfail(ctx, FTK2B_UNSUPPORTED, "mesh too large");
  C_TRY(B[kBufPos].ensure(g.nv));
  C_TRY(B[kBufHist].ensure(8 * g.nv));
  C_TRY(B[kBufVoff].ensure(4 * g.nv));
  C_TRY(B[kBufBlk].ensure(4 * (nblk + 1)));
  C_TRY(B[kBufCount].ensure(64));
  auto* pos = static_cast<unsigned char*>(B[kBufPos].p);
  auto* mask = static_cast<unsigned long long*>(B[kBufHist].p);
  auto* voff = static_cast<unsigned*>(B[kBufVoff].p);
  auto* blk = static_cast<unsigned*>(B[kBufBlk].p);
  auto* counts = static_cast<unsigned*>(B[kBufCount].p);  // [0] n, [2] roots, [3] err
  auto* total64 = reinterpret_cast<unsigned long long*>(counts + 8);
  auto* cell64 = reinterpret_cast<unsigned long long*>(counts + 10);
  const T* a = static_cast<const T*>(field);
  const unsigned sms = (unsigned)ctx->num_sms;
  C_TRY(cudaMemsetAsync(counts, 0, 64, st));
  C_TRY(cudaEventRecord(ctx->ev0, st));
  ce_sign_kernel<T><<<grid_of(g.nv, 256, 32ull * sms), 256, 0, st>>>(g, a, thr, q, pos);
  ce_mask_kernel<<<(unsigned)nblk, kCtThreads, 0, st>>>(g, pos, mask, blk, total64);
  C_TRY(launch_scan(blk, (unsigned)nblk, counts + 0, nullptr, st));
  ctx->launches += 3;
  unsigned long long n64 = 0;
  C_TRY(cudaMemcpyAsync(&n64, total64, 8, cudaMemcpyDeviceToHost, st));
  C_TRY(ctx->sync());
  if (n64 >= 0xFFFFFFF0ull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^32 - 16 crossing edges");
  const unsigned n = (unsigned)n64;
  const size_t ncap = n ? n : 1;
  C_TRY(B[kBufSimp].ensure(16 * ncap));
  C_TRY(B[kBufLam].ensure(16 * ncap));
  C_TRY(B[kBufBary].ensure(8 * ncap));
  C_TRY(B[kBufParent].ensure(4 * ncap));
  C_TRY(B[kBufTrack].ensure(8 * ncap));
  C_TRY(B[kBufFirst].ensure(8 * ncap));
  auto* simp = static_cast<unsigned long long*>(B[kBufSimp].p);
  auto* lam = static_cast<double*>(B[kBufLam].p);
  auto* bary = static_cast<float*>(B[kBufBary].p);
  auto* parent = static_cast<unsigned*>(B[kBufParent].p);
  auto* track = static_cast<unsigned long long*>(B[kBufTrack].p);
  auto* first = static_cast<unsigned long long*>(B[kBufFirst].p);
  ce_emit_kernel<T><<<(unsigned)nblk, kCtThreads, 0, st>>>(g, a, thr, mask, blk, voff, simp, lam, bary);
  ctx->launches += 1;
  const unsigned long long nsc = g.L * g.ncell * (unsigned long long)d;
  if (n) ct_fill_u64_kernel<<<grid_of(n, 256, 8ull * sms), 256, 0, st>>>(first, ~0ull, n);
  if (d == 3 && n) {
    ce_first_kernel<<<grid_of(nsc, 256, 64ull * sms), 256, 0, st>>>(g, pos, mask, voff, first);
    ctx->launches += 2;
  }
  unsigned cap = (unsigned)std::min<unsigned long long>(
      0x7FFFFFFFull, std::max<unsigned long long>(1024ull, (d == 4 ? 8ull : 4ull) * n));
  unsigned ncell = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    C_TRY(B[kBufCells].ensure((size_t)4 * kc * cap));
    auto* cells = static_cast<unsigned*>(B[kBufCells].p);
    C_TRY(cudaMemsetAsync(counts + 1, 0, 12, st));
    C_TRY(cudaMemsetAsync(cell64, 0, 8, st));
    if (n) ct_iota_kernel<<<grid_of(n, 256, 8ull * sms), 256, 0, st>>>(parent, n);
    ce_cells_kernel<<<grid_of(nsc, 256, 64ull * sms), 256, 0, st>>>(g, pos, mask, voff, first, n, cells, cell64,
                                                                    cap, parent, counts + 3);
    ctx->launches += 2;
    unsigned long long nc64 = 0;
    C_TRY(cudaMemcpyAsync(&nc64, cell64, 8, cudaMemcpyDeviceToHost, st));
    C_TRY(ctx->sync());
    if (nc64 >= 0x7FFFFFFFull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^31 - 1 manifold cells");
    ncell = (unsigned)nc64;
    if (ncell <= cap) break;
    cap = ncell;
  }
  auto* cells = static_cast<unsigned*>(B[kBufCells].p);
  const unsigned ccap = ncell ? ncell : 1;
  const unsigned nb = n + 1;
  const unsigned sblocks = (unsigned)((nb + kCtThreads * kScanPer - 1) / (kCtThreads * kScanPer));
  C_TRY(B[kBufKey0].ensure(4ull * nb));
  C_TRY(B[kBufKey1].ensure(4ull * nb));
  C_TRY(B[kBufVal0].ensure(4ull * (sblocks + 1)));
  C_TRY(B[kBufCellsOut].ensure(4ull * kc * ccap));
  auto* boff = static_cast<unsigned*>(B[kBufKey0].p);
  auto* bcur = static_cast<unsigned*>(B[kBufKey1].p);
  auto* btot = static_cast<unsigned*>(B[kBufVal0].p);
  auto* cells_out = static_cast<unsigned*>(B[kBufCellsOut].p);
  const unsigned cg = grid_of(ccap, 256, 16ull * sms);
  if (ncell) {
    C_TRY(cudaMemsetAsync(boff, 0, 4ull * nb, st));
    C_TRY(cudaMemsetAsync(bcur, 0, 4ull * nb, st));
    ct_bucket_count_kernel<<<cg, 256, 0, st>>>(cells, ncell, kc, boff);
    ct_scan_blocks_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    C_TRY(launch_scan(btot, sblocks, nullptr, nullptr, st));
    ct_scan_add_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    ct_bucket_scatter_kernel<<<cg, 256, 0, st>>>(cells, ncell, kc, boff, bcur, cells_out);
    launch_bucket_sort(cells_out, boff, n, kc, counts + 3, nullptr, st);
    ctx->launches += 6;
  }
  if (n) {
    C_TRY(launch_uf_label(parent, counts + 0, n, track, counts + 2, st));
    ctx->launches += 1;
  }
  C_TRY(cudaEventRecord(ctx->ev1, st));
  unsigned hc[4] = {0, 0, 0, 0};
  C_TRY(cudaMemcpyAsync(hc, counts, 16, cudaMemcpyDeviceToHost, st));
  C_TRY(ctx->sync());
  res->n_features = n;
  res->cell_dim = d - 1;
  res->n_cells = ncell;
  res->simplices = static_cast<uint64_t*>(host_alloc(16 * ncap));
  res->lambda = static_cast<double*>(host_alloc(16 * ncap));
  res->barycentric = static_cast<float*>(host_alloc(8 * ncap));
  res->track_id = static_cast<uint64_t*>(host_alloc(8 * ncap));
  res->scalar = static_cast<float*>(host_alloc(4 * ncap));
  res->cells = static_cast<uint32_t*>(host_alloc(4ull * kc * ccap));
  if (!res->simplices || !res->lambda || !res->barycentric || !res->track_id || !res->scalar || !res->cells)
    return cfail(ctx, FTK2B_OOM, "host result allocation failed");
  C_TRY(copy_to_host(ctx, {{res->simplices, simp, 16ull * n},
                           {res->lambda, lam, 16ull * n},
                           {res->barycentric, bary, 8ull * n},
                           {res->track_id, track, 8ull * n},
                           {res->cells, cells_out, 4ull * kc * ncell}}));
  if (hc[3] & 1u) return cfail(ctx, FTK2B_CUDA_ERROR, "union-find did not settle");
  if (hc[3] & 2u) return cfail(ctx, FTK2B_CUDA_ERROR, "duplicate manifold cell");
  const float sc = (float)thr;
  host_parallel(n, 4ull * n, [&](size_t b, size_t e) { std::fill(res->scalar + b, res->scalar + e, sc); });
  res->n_tracks = hc[2];
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  res->device_ms = ms;
  return FTK2B_OK;
}

// Level sets on an extruded mesh: base cells sorted, the CSR of base edges by
// lower vertex, the field (one value per vertex id) staged.
ftk2b_status contour_extruded(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, const ftk2b_field_desc* field,
                              double threshold, double sos_q, ftk2b_contour_result** out) {
  const int cd = mesh->base_cell_dim;
  if (cd != 2 && cd != 3) return cfail(ctx, FTK2B_UNSUPPORTED, "extruded base cells are triangles or tets");
  if (!mesh->base_cells || !mesh->n_base_cells || !mesh->n_base_verts || mesh->n_layers < 1)
    return cfail(ctx, FTK2B_INVALID_ARG, "extruded mesh needs base cells, vertices and at least one layer");
  const unsigned long long S = mesh->n_base_verts, L = mesh->n_layers, nv = S * (L + 1);
  if (S >= 0xFFFFFFFFull || nv >= (1ull << 40)) return cfail(ctx, FTK2B_UNSUPPORTED, "mesh too large");
  if (field->nd != 1 || field->dims[0] < nv)
    return cfail(ctx, FTK2B_INVALID_ARG, "extruded meshes read a per-vertex array of at least %llu values", nv);
  const int d = cd + 1;
  const unsigned long long nc = mesh->n_base_cells;
  std::vector<unsigned> cells(nc * d);
  std::vector<unsigned long long> pairs;
  pairs.reserve(nc * d * (d - 1) / 2);
  for (unsigned long long c = 0; c < nc; ++c) {
    unsigned v[4];
    for (int k = 0; k < d; ++k) {
      const uint64_t x = mesh->base_cells[c * d + k];
      if (x >= S) return cfail(ctx, FTK2B_INVALID_ARG, "base cell %llu names vertex %llu of %llu", c,
                               (unsigned long long)x, S);
      v[k] = (unsigned)x;
    }
    std::sort(v, v + d);
    for (int k = 0; k < d; ++k) cells[c * d + k] = v[k];
    for (int i = 0; i < d; ++i)
      for (int j = i + 1; j < d; ++j) pairs.push_back(((unsigned long long)v[i] << 32) | v[j]);
  }
  std::sort(pairs.begin(), pairs.end());
  pairs.erase(std::unique(pairs.begin(), pairs.end()), pairs.end());
  std::vector<unsigned> up_off(S + 1, 0), up_nbr(pairs.size());
  for (unsigned long long p : pairs) ++up_off[(p >> 32) + 1];
  for (unsigned long long a = 0; a < S; ++a) {
    if (up_off[a + 1] > 31) return cfail(ctx, FTK2B_UNSUPPORTED, "base vertex with more than 31 higher neighbours");
    up_off[a + 1] += up_off[a];
  }
  for (size_t i = 0; i < pairs.size(); ++i) up_nbr[i] = (unsigned)(pairs[i] & 0xFFFFFFFFu);
  if (cudaSetDevice(ctx->device) != cudaSuccess) return cfail(ctx, FTK2B_CUDA_ERROR, "cudaSetDevice failed");
  DevBuf* B = ctx->contour;
  C_TRY(B[kBufUpOff].ensure(4 * up_off.size()));
  C_TRY(B[kBufUpNbr].ensure(4 * (up_nbr.size() + 1)));
  C_TRY(B[kBufBaseCells].ensure(4 * cells.size()));
  C_TRY(cudaMemcpyAsync(B[kBufUpOff].p, up_off.data(), 4 * up_off.size(), cudaMemcpyHostToDevice, ctx->stream));
  if (!up_nbr.empty())
    C_TRY(cudaMemcpyAsync(B[kBufUpNbr].p, up_nbr.data(), 4 * up_nbr.size(), cudaMemcpyHostToDevice, ctx->stream));
  C_TRY(cudaMemcpyAsync(B[kBufBaseCells].p, cells.data(), 4 * cells.size(), cudaMemcpyHostToDevice, ctx->stream));
  const size_t es = field->dtype == FTK2B_F64 ? 8 : 4;
  const void* dev = field->comp[0];
  if (field->location != FTK2B_DEVICE) {
    C_TRY(B[kBufField].ensure(nv * es));
    C_TRY(cudaMemcpyAsync(B[kBufField].p, field->comp[0], nv * es, cudaMemcpyHostToDevice, ctx->stream));
    dev = B[kBufField].p;
  }
  CeGeom g;
  std::memset(&g, 0, sizeof(g));
  g.d = d;
  g.S = S;
  g.L = L;
  g.nv = nv;
  g.ncell = nc;
  g.up_off = static_cast<const unsigned*>(B[kBufUpOff].p);
  g.up_nbr = static_cast<const unsigned*>(B[kBufUpNbr].p);
  g.cells = static_cast<const unsigned*>(B[kBufBaseCells].p);
  auto* res = new (std::nothrow) ftk2b_contour_result;
  if (!res) return cfail(ctx, FTK2B_OOM, "result allocation failed");
  std::memset(res, 0, sizeof(*res));
  const unsigned long long E = pairs.size();
  res->n_simplices = E * (L + 1) + S * L + E * L;  // spatial, vertical, diagonal edges
  // the upload of the host vectors must finish before they go out of scope
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
    ftk2b_contour_result_free(res);
    return cfail(ctx, FTK2B_CUDA_ERROR, "mesh upload failed");
  }
  const ftk2b_status st = field->dtype == FTK2B_F64
                              ? run_contour_extruded<double>(ctx, g, dev, (double)threshold, sos_q, res)
                              : run_contour_extruded<float>(ctx, g, dev, (float)threshold, sos_q, res);
  if (st != FTK2B_OK) {
    ftk2b_contour_result_free(res);
    return st;
  }
  *out = res;
  return FTK2B_OK;
}

// ---------------------------------------------------------------------------
// Fiber surfaces on ExtrudedSimplicialMesh(UnstructuredSimplicialMesh(tets), L)
// (FiberPredicate<T>, predicate.hpp:341-362; the mesh, mesh.hpp:542-712;
// form_general_manifold_patches with k = 2, engine.hpp:1342-1417).  Vertex ids
// s + t S, two fields per vertex.  The triangles of the 4-D mesh are
//   spatial   every base triangle at every layer t = 0 .. L
//   lateral   the two Kuhn pieces over every base edge a < b between layers
//             t and t + 1: {a@t, a@t+1, b@t+1}, {a@t, b@t, b@t+1}
//   interior  the two triangles inside the prism over every base triangle
//             a < b < c: {a@t, b@t+1, c@t+1}, {a@t, b@t, c@t+1}
// The reference's phase 1 iterates the spatial and lateral ones (node ids in
// simplex order); the interior ones it finds while patching, numbered in the
// order it meets them: pentatopes by layer, base tet (stored order) and prism
// piece j, each pentatope's triangles in find_m_subsimplices order
// (engine.hpp:1645-1652) -- the order of its run on one worker.  Pipeline:
//   fe_test   one thread per candidate triangle: the 2-D origin test and the
//             solve with its centroid fallback, accepted ones compacted
//   sort      two stable radix sorts (third vertex, then the first two) give
//             the canonical order
//   fe_disc   one thread per pentatope: the first meeting position of every
//             accepted interior triangle (atomic minimum)
//   fe_fan    one thread per pentatope: its active triangles by node order,
//             the star-fan triangles {h_S, h_T, n}, union-find hooks
//   buckets   the fan triangles sorted and made unique; track ids

struct FeGeom {
  unsigned long long S, L, nv;      // base vertices, layers, S (L + 1)
  unsigned long long ntet, ntri, nedge;
  const unsigned* tets;              // 4 per base tet, ascending, stored order
  const unsigned* tris;              // unique base triangles, simplex order
  const unsigned* edges;             // unique base edges, simplex order
};

// candidate c: its vertex ids (ascending) and 1 when it lies inside a prism
__device__ __forceinline__ int fe_candidate(const FeGeom& g, unsigned long long c, unsigned long long v[3]) {
  const unsigned long long nsp = (g.L + 1) * g.ntri, nlat = 2 * g.L * g.nedge;
  if (c < nsp) {
    const unsigned long long t = c / g.ntri, i = c - t * g.ntri;
    for (int k = 0; k < 3; ++k) v[k] = g.tris[3 * i + k] + t * g.S;
    return 0;
  }
  c -= nsp;
  if (c < nlat) {
    const unsigned long long j = c & 1, q = c >> 1, t = q / g.nedge, e = q - t * g.nedge;
    const unsigned long long a = g.edges[2 * e], b = g.edges[2 * e + 1];
    v[0] = a + t * g.S;
    v[1] = j == 0 ? a + (t + 1) * g.S : b + t * g.S;
    v[2] = b + (t + 1) * g.S;
    return 0;
  }
  c -= nlat;
  const unsigned long long k = c & 1, q = c >> 1, t = q / g.ntri, i = q - t * g.ntri;
  const unsigned long long a = g.tris[3 * i], b = g.tris[3 * i + 1], cc = g.tris[3 * i + 2];
  v[0] = a + t * g.S;
  v[1] = b + (k == 0 ? t + 1 : t) * g.S;
  v[2] = cc + (t + 1) * g.S;
  return 1;
}

template <typename T>
__global__ void fe_test_kernel(FeGeom g, const T* __restrict__ f0, const T* __restrict__ f1, T t0, T t1, double q,
                               unsigned long long ncand, unsigned long long* __restrict__ simp,
                               double* __restrict__ lam, float* __restrict__ bary, unsigned* __restrict__ phase,
                               unsigned* cnt, unsigned cap) {
  const int lane = threadIdx.x & 31;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < ncand; base += stride) {
    const unsigned long long c = base + threadIdx.x;
    bool acc = false;
    unsigned long long v[3] = {0, 0, 0};
    int ph = 0;
    T l[3];
    if (c < ncand) {
      ph = fe_candidate(g, c, v);
      T val[3][2];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        val[k][0] = fp<T>::sub(__ldg(f0 + v[k]), t0);  // values[i][j] - thresholds[j]
        val[k][1] = fp<T>::sub(__ldg(f1 + v[k]), t1);
      }
      if (sos_inside2<T>(val, q)) {
        acc = true;
        if (!solve_exact<2, T>(val, l))  // FiberPredicate keeps the centroid: (T)1.0 / 3.0
          for (int k = 0; k < 3; ++k) l[k] = (T)((double)(T)1.0 / 3.0);
      }
    }
    const unsigned ball = __ballot_sync(0xFFFFFFFFu, acc);
    if (!ball) continue;
    unsigned b0 = 0;
    if (lane == 0) b0 = atomicAdd(cnt, (unsigned)__popc(ball));
    b0 = __shfl_sync(0xFFFFFFFFu, b0, 0);
    if (!acc) continue;
    const unsigned r = b0 + __popc(ball & ((1u << lane) - 1u));
    if (r >= cap) continue;
    for (int k = 0; k < 3; ++k) {
      simp[3 * (size_t)r + k] = v[k];
      lam[3 * (size_t)r + k] = (double)l[k];
      bary[3 * (size_t)r + k] = (float)l[k];
    }
    phase[r] = (unsigned)ph;
  }
}

__global__ void fe_set_kernel(unsigned* p, unsigned v) { *p = v; }

__global__ void fe_key_lo_kernel(const unsigned long long* __restrict__ simp, unsigned n,
                                 unsigned long long* __restrict__ key, unsigned* __restrict__ val) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    key[i] = simp[3 * (size_t)i + 2];
    val[i] = i;
  }
}

// keys of the first two vertices in the order of perm (the sort by the
// third vertex), written over that sort's keys
__global__ void fe_key_hi_kernel(const unsigned long long* __restrict__ simp, const unsigned* __restrict__ perm,
                                 unsigned n, unsigned long long* __restrict__ key) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned p = perm[i];
    key[i] = (simp[3 * (size_t)p] << 32) | simp[3 * (size_t)p + 1];
  }
}

// canonical order: features gathered by perm, lookup keys, vertex flags,
// first-meeting positions reset, union-find parents
__global__ void fe_gather_kernel(const unsigned* __restrict__ perm, unsigned n,
                                 const unsigned long long* __restrict__ simp_u, const double* __restrict__ lam_u,
                                 const float* __restrict__ bary_u, const unsigned* __restrict__ phase_u,
                                 unsigned long long* __restrict__ simp, double* __restrict__ lam,
                                 float* __restrict__ bary, unsigned* __restrict__ phase,
                                 unsigned long long* __restrict__ hi, unsigned* __restrict__ lo,
                                 unsigned char* __restrict__ vflag, unsigned long long* __restrict__ disc,
                                 unsigned* __restrict__ parent) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned p = perm[i];
    unsigned long long v[3];
    for (int k = 0; k < 3; ++k) {
      v[k] = simp_u[3 * (size_t)p + k];
      simp[3 * (size_t)i + k] = v[k];
      lam[3 * (size_t)i + k] = lam_u[3 * (size_t)p + k];
      bary[3 * (size_t)i + k] = bary_u[3 * (size_t)p + k];
      vflag[v[k]] = 1;
    }
    phase[i] = phase_u[p];
    hi[i] = (v[0] << 32) | v[1];
    lo[i] = (unsigned)v[2];
    disc[i] = ~0ull;
    parent[i] = i;
  }
}

__device__ __forceinline__ long long fe_find(const unsigned long long* __restrict__ hi,
                                             const unsigned* __restrict__ lo, unsigned n, unsigned long long h,
                                             unsigned l) {
  unsigned a = 0, b = n;
  while (a < b) {
    const unsigned mid = (a + b) >> 1;
    const unsigned long long hm = hi[mid];
    const unsigned lm = lo[mid];
    if (hm == h && lm == l) return mid;
    if (hm < h || (hm == h && lm < l)) a = mid + 1;
    else b = mid;
  }
  return -1;
}

// Pentatope p of the reference's iteration order: layer t, base tet c, prism
// piece j; its vertex ids (ascending), the spatial id and layer of each.
__device__ __forceinline__ void fe_pentatope(const FeGeom& g, unsigned long long p, unsigned long long cell[5],
                                             unsigned sp[5], int lay[5]) {
  const unsigned long long t = p / (4 * g.ntet), r = p - t * 4 * g.ntet, c = r >> 2;
  const int j = (int)(r & 3);
  const unsigned* w = g.tets + 4 * c;
  int k = 0;
  for (int l = 0; l <= j; ++l, ++k) {
    sp[k] = w[l];
    lay[k] = 0;
    cell[k] = w[l] + t * g.S;
  }
  for (int l = j; l <= 3; ++l, ++k) {
    sp[k] = w[l];
    lay[k] = 1;
    cell[k] = w[l] + (t + 1) * g.S;
  }
}

__global__ void fe_disc_kernel(FeGeom g, unsigned long long npent, const unsigned char* __restrict__ vflag,
                               const unsigned long long* __restrict__ hi, const unsigned* __restrict__ lo,
                               unsigned n, unsigned long long* __restrict__ disc) {
  for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < npent;
       p += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long cell[5];
    unsigned sp[5];
    int lay[5];
    fe_pentatope(g, p, cell, sp, lay);
    int nf = 0;
    for (int k = 0; k < 5; ++k) nf += vflag[cell[k]];
    if (nf < 3) continue;
    int pos = 0;
    for (int a = 0; a < 5; ++a)
      for (int b = a + 1; b < 5; ++b)
        for (int c = b + 1; c < 5; ++c, ++pos) {
          // inside a prism: three distinct base vertices over both layers
          if (sp[a] == sp[b] || sp[b] == sp[c] || lay[a] == lay[c]) continue;
          const long long idx = fe_find(hi, lo, n, (cell[a] << 32) | cell[b], (unsigned)cell[c]);
          if (idx >= 0) atomicMin(&disc[idx], p * 16 + (unsigned long long)pos);
        }
  }
}

__global__ void fe_fan_kernel(FeGeom g, unsigned long long npent, const unsigned char* __restrict__ vflag,
                              const unsigned long long* __restrict__ hi, const unsigned* __restrict__ lo, unsigned n,
                              const unsigned* __restrict__ phase, const unsigned long long* __restrict__ disc,
                              unsigned* __restrict__ cells, unsigned long long* cnt, unsigned cap,
                              unsigned* parent, unsigned* err) {
  for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < npent;
       p += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long cell[5];
    unsigned sp[5];
    int lay[5];
    fe_pentatope(g, p, cell, sp, lay);
    int nf = 0;
    for (int k = 0; k < 5; ++k) nf += vflag[cell[k]];
    if (nf < 3) continue;
    unsigned node[10], vs[10];
    unsigned long long ord[10];
    int nn = 0;
    for (int a = 0; a < 5; ++a)
      for (int b = a + 1; b < 5; ++b)
        for (int c = b + 1; c < 5; ++c) {
          const long long idx = fe_find(hi, lo, n, (cell[a] << 32) | cell[b], (unsigned)cell[c]);
          if (idx < 0) continue;
          // node order: phase-1 triangles in simplex order, then the others
          // by the position at which patching first met them
          const unsigned long long o = phase[idx] ? ((1ull << 63) | disc[idx]) : (unsigned long long)idx;
          int w = nn++;
          while (w > 0 && ord[w - 1] > o) {
            ord[w] = ord[w - 1];
            node[w] = node[w - 1];
            vs[w] = vs[w - 1];
            --w;
          }
          ord[w] = o;
          node[w] = (unsigned)idx;
          vs[w] = (1u << a) | (1u << b) | (1u << c);
        }
    if (nn < 2) continue;
    const unsigned hs = node[0];
    unsigned mine = 0;
    for (int f = 0; f < 5; ++f) {
      int seen = 0;
      unsigned ht = 0;
      for (int x = 0; x < nn; ++x) {
        if (vs[x] & (1u << f)) continue;
        if (seen++ == 0) {
          ht = node[x];
          continue;
        }
        if (hs != ht && hs != node[x]) ++mine;
      }
    }
    if (!mine) continue;
    unsigned long long slot = atomicAdd(cnt, (unsigned long long)mine);
    for (int f = 0; f < 5; ++f) {
      int seen = 0;
      unsigned ht = 0;
      for (int x = 0; x < nn; ++x) {
        if (vs[x] & (1u << f)) continue;
        if (seen++ == 0) {
          ht = node[x];
          continue;
        }
        if (hs == ht || hs == node[x]) continue;
        unsigned tri[3] = {hs, ht, node[x]};
        ct_sort4(tri, 3);
        if (slot < cap)
          for (int k = 0; k < 3; ++k) cells[(size_t)slot * 3 + k] = tri[k];
        ++slot;
        uf_unite(parent, tri[0], tri[1], err);
        uf_unite(parent, tri[0], tri[2], err);
      }
    }
  }
}

template <typename T>
ftk2b_status run_fiber_surface_extruded(ftk2b_ctx* ctx, const FeGeom& g, const void* fa, const void* fb, T t0, T t1,
                                        double q, ftk2b_fiber_surface_result* res) {
  cudaStream_t st = ctx->stream;
  DevBuf* B = ctx->contour;
  const unsigned sms = (unsigned)ctx->num_sms;
  const unsigned long long ncand = (g.L + 1) * g.ntri + 2 * g.L * g.nedge + 2 * g.L * g.ntri;
  const unsigned long long npent = 4 * g.L * g.ntet;
  C_TRY(B[kBufCount].ensure(64));
  auto* counts = static_cast<unsigned*>(B[kBufCount].p);  // [0] n, [1] accepted, [2] roots, [3] err
  auto* cell64 = reinterpret_cast<unsigned long long*>(counts + 10);
  const T* a0 = static_cast<const T*>(fa);
  const T* a1 = static_cast<const T*>(fb);
  C_TRY(cudaMemsetAsync(counts, 0, 64, st));
  C_TRY(cudaEventRecord(ctx->ev0, st));
  // 1. every candidate triangle, accepted ones compacted (capacity grows once)
  unsigned cap = ctx->fe_cap ? ctx->fe_cap : (1u << 18);
  unsigned n = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    C_TRY(B[kBufSimp].ensure(24ull * cap));
    C_TRY(B[kBufLam].ensure(24ull * cap));
    C_TRY(B[kBufBary].ensure(12ull * cap));
    C_TRY(B[kBufVoff].ensure(4ull * cap));
    C_TRY(cudaMemsetAsync(counts + 1, 0, 4, st));
    fe_test_kernel<T><<<grid_of(ncand, 256, 64ull * sms), 256, 0, st>>>(
        g, a0, a1, t0, t1, q, ncand, static_cast<unsigned long long*>(B[kBufSimp].p),
        static_cast<double*>(B[kBufLam].p), static_cast<float*>(B[kBufBary].p), static_cast<unsigned*>(B[kBufVoff].p),
        counts + 1, cap);
    ctx->launches += 1;
    C_TRY(cudaMemcpyAsync(ctx->h_counters, counts + 1, 4, cudaMemcpyDeviceToHost, st));
    C_TRY(ctx->sync());
    n = ctx->h_counters[0];
    if (n <= cap) break;
    if (n >= 0x7FFFFFF0u) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^31 feature triangles");
    cap = n + n / 8 + 1024;
    ctx->fe_cap = cap;
  }
  const size_t ncap = n ? n : 1;
  auto* simp_u = static_cast<unsigned long long*>(B[kBufSimp].p);
  // 2. canonical order
  C_TRY(B[kBufKey0].ensure(8 * ncap));
  C_TRY(B[kBufKey1].ensure(8 * ncap));
  C_TRY(B[kBufVal0].ensure(4 * ncap));
  C_TRY(B[kBufVal1].ensure(4 * ncap));
  const int sgrid = ctx->sort_grid((unsigned)ncap);
  C_TRY(B[kBufHist].ensure(4ull * 256 * sgrid));
  auto* k0 = static_cast<unsigned long long*>(B[kBufKey0].p);
  auto* k1 = static_cast<unsigned long long*>(B[kBufKey1].p);
  auto* v0 = static_cast<unsigned*>(B[kBufVal0].p);
  auto* v1 = static_cast<unsigned*>(B[kBufVal1].p);
  auto* hist = static_cast<unsigned*>(B[kBufHist].p);
  int vb = 1;
  while (vb < 64 && (g.nv >> vb) != 0) ++vb;
  fe_set_kernel<<<1, 1, 0, st>>>(counts + 0, n);
  fe_key_lo_kernel<<<grid_of(ncap, 256, 16ull * sms), 256, 0, st>>>(simp_u, n, k0, v0);
  unsigned long long nl = 0;
  const bool alt1 = radix_sort(k0, v0, k1, v1, counts + 0, (unsigned)ncap, vb, hist, sgrid, st, &nl);
  unsigned long long* kr = alt1 ? k1 : k0;
  unsigned* vr = alt1 ? v1 : v0;
  fe_key_hi_kernel<<<grid_of(ncap, 256, 16ull * sms), 256, 0, st>>>(simp_u, vr, n, kr);
  const bool alt2 = radix_sort(kr, vr, alt1 ? k0 : k1, alt1 ? v0 : v1, counts + 0, (unsigned)ncap, 32 + vb, hist,
                               sgrid, st, &nl);
  const unsigned* perm = alt2 ? (alt1 ? v0 : v1) : vr;
  ctx->launches += nl + 3;
  C_TRY(B[kBufFeSimp].ensure(24 * ncap));
  C_TRY(B[kBufFeLam].ensure(24 * ncap));
  C_TRY(B[kBufFeBary].ensure(12 * ncap));
  C_TRY(B[kBufFePhase].ensure(4 * ncap));
  C_TRY(B[kBufFeDisc].ensure(8 * ncap));
  C_TRY(B[kBufFeHi].ensure(8 * ncap));
  C_TRY(B[kBufFeLo].ensure(4 * ncap));
  C_TRY(B[kBufFeFlag].ensure(g.nv));
  C_TRY(B[kBufParent].ensure(4 * ncap));
  C_TRY(B[kBufTrack].ensure(8 * ncap));
  auto* simp = static_cast<unsigned long long*>(B[kBufFeSimp].p);
  auto* lam = static_cast<double*>(B[kBufFeLam].p);
  auto* bary = static_cast<float*>(B[kBufFeBary].p);
  auto* phase = static_cast<unsigned*>(B[kBufFePhase].p);
  auto* disc = static_cast<unsigned long long*>(B[kBufFeDisc].p);
  auto* hi = static_cast<unsigned long long*>(B[kBufFeHi].p);
  auto* lo = static_cast<unsigned*>(B[kBufFeLo].p);
  auto* vflag = static_cast<unsigned char*>(B[kBufFeFlag].p);
  auto* parent = static_cast<unsigned*>(B[kBufParent].p);
  auto* track = static_cast<unsigned long long*>(B[kBufTrack].p);
  C_TRY(cudaMemsetAsync(vflag, 0, g.nv, st));
  fe_gather_kernel<<<grid_of(ncap, 256, 16ull * sms), 256, 0, st>>>(
      perm, n, simp_u, static_cast<const double*>(B[kBufLam].p), static_cast<const float*>(B[kBufBary].p),
      static_cast<const unsigned*>(B[kBufVoff].p), simp, lam, bary, phase, hi, lo, vflag, disc, parent);
  // 3. first meeting positions of the interior triangles
  fe_disc_kernel<<<grid_of(npent, 256, 64ull * sms), 256, 0, st>>>(g, npent, vflag, hi, lo, n, disc);
  ctx->launches += 2;
  // 4. star-fan triangles
  unsigned ccap = (unsigned)std::min<unsigned long long>(0x7FFFFFFFull, std::max<unsigned long long>(1024ull, 4ull * n));
  unsigned ncell = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    C_TRY(B[kBufCells].ensure((size_t)12 * ccap));
    C_TRY(cudaMemsetAsync(cell64, 0, 8, st));
    if (attempt) ct_iota_kernel<<<grid_of(ncap, 256, 8ull * sms), 256, 0, st>>>(parent, n);
    fe_fan_kernel<<<grid_of(npent, 256, 64ull * sms), 256, 0, st>>>(g, npent, vflag, hi, lo, n, phase, disc,
                                                                    static_cast<unsigned*>(B[kBufCells].p), cell64,
                                                                    ccap, parent, counts + 3);
    ctx->launches += 1;
    unsigned long long nc64 = 0;
    C_TRY(cudaMemcpyAsync(&nc64, cell64, 8, cudaMemcpyDeviceToHost, st));
    C_TRY(ctx->sync());
    if (nc64 >= 0x7FFFFFFFull) return cfail(ctx, FTK2B_UNSUPPORTED, "more than 2^31 - 1 manifold triangles");
    ncell = (unsigned)nc64;
    if (ncell <= ccap) break;
    ccap = ncell;
  }
  auto* cells = static_cast<unsigned*>(B[kBufCells].p);
  // 5. sorted, unique triangles: buckets by leading node
  const unsigned nb = n + 1;
  const unsigned sblocks = (unsigned)((nb + kCtThreads * kScanPer - 1) / (kCtThreads * kScanPer));
  const unsigned cc = ncell ? ncell : 1;
  C_TRY(B[kBufKey0].ensure(4ull * nb));
  C_TRY(B[kBufKey1].ensure(4ull * nb));
  C_TRY(B[kBufVal0].ensure(4ull * (sblocks + 1)));
  C_TRY(B[kBufVal1].ensure(4ull * nb));
  C_TRY(B[kBufCellsOut].ensure(12ull * cc));
  C_TRY(B[kBufMask].ensure(12ull * cc));
  auto* boff = static_cast<unsigned*>(B[kBufKey0].p);
  auto* bcur = static_cast<unsigned*>(B[kBufKey1].p);
  auto* btot = static_cast<unsigned*>(B[kBufVal0].p);
  auto* uoff = static_cast<unsigned*>(B[kBufVal1].p);
  auto* rows = static_cast<unsigned*>(B[kBufCellsOut].p);
  auto* cells_out = static_cast<unsigned*>(B[kBufMask].p);
  const unsigned cg = grid_of(cc, 256, 16ull * sms);
  unsigned nuniq = 0;
  if (ncell) {
    C_TRY(cudaMemsetAsync(boff, 0, 4ull * nb, st));
    C_TRY(cudaMemsetAsync(bcur, 0, 4ull * nb, st));
    C_TRY(cudaMemsetAsync(uoff, 0, 4ull * nb, st));
    ct_bucket_count_kernel<<<cg, 256, 0, st>>>(cells, ncell, 3, boff);
    ct_scan_blocks_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    C_TRY(launch_scan(btot, sblocks, nullptr, nullptr, st));
    ct_scan_add_kernel<<<sblocks, kCtThreads, 0, st>>>(boff, nb, btot);
    ct_bucket_scatter_kernel<<<cg, 256, 0, st>>>(cells, ncell, 3, boff, bcur, rows);
    launch_bucket_sort(rows, boff, n, 3, counts + 3, uoff, st);
    ct_scan_blocks_kernel<<<sblocks, kCtThreads, 0, st>>>(uoff, nb, btot);
    C_TRY(launch_scan(btot, sblocks, nullptr, nullptr, st));
    ct_scan_add_kernel<<<sblocks, kCtThreads, 0, st>>>(uoff, nb, btot);
    ct_bucket_compact_kernel<<<grid_of(n, 128, 32ull * sms), 128, 0, st>>>(rows, boff, uoff, n, 3, cells_out);
    ctx->launches += 10;
    C_TRY(cudaMemcpyAsync(&nuniq, uoff + n, 4, cudaMemcpyDeviceToHost, st));
  }
  if (n) {
    C_TRY(launch_uf_label(parent, counts + 0, n, track, counts + 2, st));
    ctx->launches += 1;
  }
  C_TRY(cudaEventRecord(ctx->ev1, st));
  unsigned hc[4] = {0, 0, 0, 0};
  C_TRY(cudaMemcpyAsync(hc, counts, 16, cudaMemcpyDeviceToHost, st));
  C_TRY(ctx->sync());
  res->n_features = n;
  res->n_cells = nuniq;
  res->simplices = static_cast<uint64_t*>(host_alloc(24 * ncap));
  res->lambda = static_cast<double*>(host_alloc(24 * ncap));
  res->barycentric = static_cast<float*>(host_alloc(12 * ncap));
  res->track_id = static_cast<uint64_t*>(host_alloc(8 * ncap));
  res->scalar = static_cast<float*>(std::calloc(ncap, 4));
  res->cells = static_cast<uint32_t*>(host_alloc(12ull * (nuniq ? nuniq : 1)));
  if (!res->simplices || !res->lambda || !res->barycentric || !res->track_id || !res->scalar || !res->cells)
    return cfail(ctx, FTK2B_OOM, "host result allocation failed");
  C_TRY(copy_to_host(ctx, {{res->simplices, simp, 24ull * n},
                           {res->lambda, lam, 24ull * n},
                           {res->barycentric, bary, 12ull * n},
                           {res->track_id, track, 8ull * n},
                           {res->cells, cells_out, 12ull * nuniq}}));
  if (hc[3] & 1u) return cfail(ctx, FTK2B_TIMEOUT, "union-find retry bound reached");
  res->n_tracks = hc[2];
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  res->device_ms = ms;
  return FTK2B_OK;
}

// Fiber surfaces on an extruded mesh over tets: base tets sorted, the unique
// base triangles and edges in simplex order, both fields (one value per
// vertex id) staged.
ftk2b_status fiber_surface_extruded(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, const ftk2b_field_desc* field,
                                    const double thr[2], double sos_q, ftk2b_fiber_surface_result** out) {
  if (mesh->base_cell_dim != 3 || mesh->ndims != 4)
    return cfail(ctx, FTK2B_UNSUPPORTED, "fiber surfaces on extruded meshes need tet base cells (ndims 4)");
  if (!mesh->base_cells || !mesh->n_base_cells || !mesh->n_base_verts || mesh->n_layers < 1)
    return cfail(ctx, FTK2B_INVALID_ARG, "extruded mesh needs base cells, vertices and at least one layer");
  const unsigned long long S = mesh->n_base_verts, L = mesh->n_layers, nv = S * (L + 1);
  if (S >= 0xFFFFFFFFull || nv >= 0xFFFFFFFFull) return cfail(ctx, FTK2B_UNSUPPORTED, "mesh too large");
  if ((field->layout != FTK2B_LAYOUT_SEPARATE && field->layout != FTK2B_LAYOUT_PER_VERTEX) || field->nd != 1 ||
      field->dims[0] < nv)
    return cfail(ctx, FTK2B_INVALID_ARG, "extruded meshes read two per-vertex arrays of at least %llu values", nv);
  const unsigned long long nc = mesh->n_base_cells;
  std::vector<unsigned> tets(nc * 4);
  std::vector<unsigned long long> tri_keys, edge_keys;
  tri_keys.reserve(nc * 4);
  edge_keys.reserve(nc * 6);
  for (unsigned long long c = 0; c < nc; ++c) {
    unsigned v[4];
    for (int k = 0; k < 4; ++k) {
      const uint64_t x = mesh->base_cells[c * 4 + k];
      if (x >= S) return cfail(ctx, FTK2B_INVALID_ARG, "base cell %llu names vertex %llu of %llu", c,
                               (unsigned long long)x, S);
      v[k] = (unsigned)x;
    }
    std::sort(v, v + 4);
    for (int k = 0; k < 4; ++k) tets[c * 4 + k] = v[k];
    for (int r = 0; r < 4; ++r) {
      unsigned w[3];
      int k = 0;
      for (int i = 0; i < 4; ++i)
        if (i != r) w[k++] = v[i];
      // 21 bits per id when they fit, else the rows are sorted as triples
      tri_keys.push_back(((unsigned long long)w[0] << 42) | ((unsigned long long)w[1] << 21) | w[2]);
    }
    for (int i = 0; i < 4; ++i)
      for (int j = i + 1; j < 4; ++j) edge_keys.push_back(((unsigned long long)v[i] << 32) | v[j]);
  }
  std::vector<unsigned> tris;
  if (S < (1ull << 21)) {
    std::sort(tri_keys.begin(), tri_keys.end());
    tri_keys.erase(std::unique(tri_keys.begin(), tri_keys.end()), tri_keys.end());
    tris.resize(3 * tri_keys.size());
    for (size_t i = 0; i < tri_keys.size(); ++i) {
      tris[3 * i] = (unsigned)(tri_keys[i] >> 42);
      tris[3 * i + 1] = (unsigned)((tri_keys[i] >> 21) & 0x1FFFFF);
      tris[3 * i + 2] = (unsigned)(tri_keys[i] & 0x1FFFFF);
    }
  } else {
    std::vector<std::array<unsigned, 3>> t3;
    t3.reserve(nc * 4);
    for (unsigned long long c = 0; c < nc; ++c)
      for (int r = 0; r < 4; ++r) {
        std::array<unsigned, 3> w;
        int k = 0;
        for (int i = 0; i < 4; ++i)
          if (i != r) w[k++] = tets[c * 4 + i];
        t3.push_back(w);
      }
    std::sort(t3.begin(), t3.end());
    t3.erase(std::unique(t3.begin(), t3.end()), t3.end());
    tris.resize(3 * t3.size());
    for (size_t i = 0; i < t3.size(); ++i)
      for (int k = 0; k < 3; ++k) tris[3 * i + k] = t3[i][k];
  }
  std::sort(edge_keys.begin(), edge_keys.end());
  edge_keys.erase(std::unique(edge_keys.begin(), edge_keys.end()), edge_keys.end());
  std::vector<unsigned> edges(2 * edge_keys.size());
  for (size_t i = 0; i < edge_keys.size(); ++i) {
    edges[2 * i] = (unsigned)(edge_keys[i] >> 32);
    edges[2 * i + 1] = (unsigned)(edge_keys[i] & 0xFFFFFFFFu);
  }
  if (cudaSetDevice(ctx->device) != cudaSuccess) return cfail(ctx, FTK2B_CUDA_ERROR, "cudaSetDevice failed");
  DevBuf* B = ctx->contour;
  C_TRY(B[kBufBaseCells].ensure(4 * tets.size()));
  C_TRY(B[kBufFeTris].ensure(4 * tris.size()));
  C_TRY(B[kBufFeEdges].ensure(4 * edges.size()));
  C_TRY(cudaMemcpyAsync(B[kBufBaseCells].p, tets.data(), 4 * tets.size(), cudaMemcpyHostToDevice, ctx->stream));
  C_TRY(cudaMemcpyAsync(B[kBufFeTris].p, tris.data(), 4 * tris.size(), cudaMemcpyHostToDevice, ctx->stream));
  C_TRY(cudaMemcpyAsync(B[kBufFeEdges].p, edges.data(), 4 * edges.size(), cudaMemcpyHostToDevice, ctx->stream));
  const size_t es = field->dtype == FTK2B_F64 ? 8 : 4;
  const void* dev[2] = {field->comp[0], field->comp[1]};
  if (field->location != FTK2B_DEVICE) {
    const int slot[2] = {kBufField, kBufField2};
    for (int j = 0; j < 2; ++j) {
      C_TRY(B[slot[j]].ensure(nv * es));
      C_TRY(cudaMemcpyAsync(B[slot[j]].p, field->comp[j], nv * es, cudaMemcpyHostToDevice, ctx->stream));
      dev[j] = B[slot[j]].p;
    }
  }
  // the upload of the host vectors must finish before they go out of scope
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return cfail(ctx, FTK2B_CUDA_ERROR, "mesh upload failed");
  FeGeom g;
  std::memset(&g, 0, sizeof(g));
  g.S = S;
  g.L = L;
  g.nv = nv;
  g.ntet = nc;
  g.ntri = tris.size() / 3;
  g.nedge = edges.size() / 2;
  g.tets = static_cast<const unsigned*>(B[kBufBaseCells].p);
  g.tris = static_cast<const unsigned*>(B[kBufFeTris].p);
  g.edges = static_cast<const unsigned*>(B[kBufFeEdges].p);
  auto* res = new (std::nothrow) ftk2b_fiber_surface_result;
  if (!res) return cfail(ctx, FTK2B_OOM, "result allocation failed");
  std::memset(res, 0, sizeof(*res));
  res->n_simplices = (L + 1) * g.ntri + 2 * L * g.nedge + 2 * L * g.ntri;
  const ftk2b_status st =
      field->dtype == FTK2B_F64
          ? run_fiber_surface_extruded<double>(ctx, g, dev[0], dev[1], thr[0], thr[1], sos_q, res)
          : run_fiber_surface_extruded<float>(ctx, g, dev[0], dev[1], (float)thr[0], (float)thr[1], sos_q, res);
  if (st != FTK2B_OK) {
    ftk2b_fiber_surface_result_free(res);
    return st;
  }
  *out = res;
  return FTK2B_OK;
}

}  // namespace

// Geometry of a regular mesh and its scalar array(s) for the level-set and
// fiber-surface pipelines; *nelem receives the element count of one array.
static ftk2b_status ct_geometry(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, const ftk2b_field_desc* field,
                                CtGeom& g, size_t* nelem_out);

extern "C" ftk2b_status ftk2b_contour_extract(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh,
                                              const ftk2b_field_desc* field, double threshold, double sos_q,
                                              ftk2b_contour_result** out) {
  ftk2b::NvtxRange nvtx_range("ftk2b_contour_extract");
  if (!ctx) return FTK2B_INVALID_ARG;
  if (!mesh || !field || !out) return cfail(ctx, FTK2B_INVALID_ARG, "null argument");
  *out = nullptr;
  if (field->dtype != FTK2B_F32 && field->dtype != FTK2B_F64)
    return cfail(ctx, FTK2B_INVALID_ARG, "dtype must be FTK2B_F32 or FTK2B_F64");
  if (field->ncomp != 1 || !field->comp[0] ||
      (field->layout != FTK2B_LAYOUT_SEPARATE && field->layout != FTK2B_LAYOUT_PER_VERTEX))
    return cfail(ctx, FTK2B_INVALID_ARG, "level sets read one scalar array (ncomp 1, layout SEPARATE)");
  if (!(sos_q > 0)) return cfail(ctx, FTK2B_INVALID_ARG, "sos_q must be positive");
  if (mesh->kind == FTK2B_MESH_EXTRUDED) return contour_extruded(ctx, mesh, field, threshold, sos_q, out);
  if (mesh->kind != FTK2B_MESH_REGULAR) return cfail(ctx, FTK2B_INVALID_ARG, "unknown mesh kind %d", mesh->kind);
  const int d = mesh->ndims;
  if (d != 3 && d != 4) return cfail(ctx, FTK2B_UNSUPPORTED, "regular meshes have 3 or 4 dims (got %d)", d);
  CtGeom g;
  size_t nelem = 1;
  {
    const ftk2b_status gs = ct_geometry(ctx, mesh, field, g, &nelem);
    if (gs != FTK2B_OK) return gs;
  }
  const size_t es = field->dtype == FTK2B_F64 ? 8 : 4;
  const unsigned long long nv = g.nv;
  if (cudaSetDevice(ctx->device) != cudaSuccess) return cfail(ctx, FTK2B_CUDA_ERROR, "cudaSetDevice failed");
  const void* dev = field->comp[0];
  if (field->location != FTK2B_DEVICE) {
    C_TRY(ctx->contour[kBufField].ensure(nelem * es));
    C_TRY(cudaMemcpyAsync(ctx->contour[kBufField].p, field->comp[0], nelem * es, cudaMemcpyHostToDevice,
                          ctx->stream));
    dev = ctx->contour[kBufField].p;
  }
  (void)nv;
  auto* res = new (std::nothrow) ftk2b_contour_result;
  if (!res) return cfail(ctx, FTK2B_OOM, "result allocation failed");
  std::memset(res, 0, sizeof(*res));
  unsigned long long edges = 0;
  for (int e = 1; e < (1 << d); ++e) {
    unsigned long long c = 1;
    for (int k = 0; k < d; ++k) c *= ((e >> k) & 1) ? g.L[k] - 1 : g.L[k];
    edges += c;
  }
  res->n_simplices = edges;
  const ftk2b_status st =
      field->dtype == FTK2B_F64
          ? run_contour<double>(ctx, g, dev, (double)threshold, sos_q, res)
          : run_contour<float>(ctx, g, dev, (float)threshold, sos_q, res);
  if (st != FTK2B_OK) {
    ftk2b_contour_result_free(res);
    return st;
  }
  *out = res;
  return FTK2B_OK;
}

static ftk2b_status ct_geometry(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh, const ftk2b_field_desc* field,
                                CtGeom& g, size_t* nelem_out) {
  const int d = mesh->ndims;
  std::memset(&g, 0, sizeof(g));
  g.d = d;
  unsigned long long nv = 1, ncube = 1, gstride = 1;
  for (int k = 0; k < d; ++k) {
    const unsigned long long L = mesh->local_dims[k], G = mesh->global_dims[k], O = mesh->offset[k];
    if (L < 1) return cfail(ctx, FTK2B_INVALID_ARG, "local dim %d is 0", k);
    if (G < O + L) return cfail(ctx, FTK2B_INVALID_ARG, "dim %d: offset + local exceeds the global dim", k);
    g.L[k] = L;
    g.gs[k] = gstride;
    g.g0 += O * gstride;
    gstride *= G;
    nv *= L;
    ncube *= L - 1;
  }
  g.nv = nv;
  g.ncube = ncube;
  size_t nelem = 1;
  if (field->nd == 1) {
    g.per_vertex = 1;
    nelem = field->dims[0];
    if (nelem < gstride) return cfail(ctx, FTK2B_INVALID_ARG, "per-vertex array shorter than the global vertex count");
  } else {
    if (field->nd != d) return cfail(ctx, FTK2B_INVALID_ARG, "the scalar array needs nd == mesh dims (or 1)");
    unsigned long long s = 1;
    for (int k = 0; k < d; ++k) {
      if (field->dims[k] < g.L[k]) return cfail(ctx, FTK2B_INVALID_ARG, "array dim %d smaller than the local dim", k);
      g.as[k] = s;
      s *= field->dims[k];
    }
    nelem = s;
  }
  if (nv >= (1ull << 40)) return cfail(ctx, FTK2B_UNSUPPORTED, "mesh too large");
  unsigned long long ls = 1, lstr[4] = {0, 0, 0, 0};
  for (int k = 0; k < d; ++k) {
    lstr[k] = ls;
    ls *= g.L[k];
  }
  for (int k = 0; k < d; ++k) g.lstr[k] = lstr[k];
  // axis order of the p-th Kuhn simplex as the CPU mesh decodes it
  // (mesh.hpp:407-409): successive swaps p[i] <-> p[i + j], j = p % (d - i)
  const int np = d == 3 ? 6 : 24;
  for (int p = 0; p < np; ++p) {
    int ax[4] = {0, 1, 2, 3}, t = p;
    for (int i = 0; i < d; ++i) {
      const int j = t % (d - i);
      std::swap(ax[i], ax[i + j]);
      t /= d - i;
    }
    for (int i = 0; i < 4; ++i) g.perm[p][i] = (unsigned char)ax[i];
  }
  for (int e = 0; e < (1 << d); ++e)
    for (int k = 0; k < d; ++k)
      if ((e >> k) & 1) {
        g.loff[e] += lstr[k];
        g.goff[e] += g.gs[k];
        g.aoff[e] += g.as[k];
      }
  g.linear = !g.per_vertex;
  for (int k = 0; k < d; ++k) g.linear &= g.L[k] == 1 || g.as[k] == lstr[k];
  g.small = nv < (1ull << 31);
  for (int k = 0; g.small && k < d; ++k) {
    int l = 0;
    while ((1ull << l) < g.L[k]) ++l;
    g.shf[k] = 31 + l;
    g.mul[k] = (unsigned)(((1ull << g.shf[k]) + g.L[k] - 1) / g.L[k]);
  }
  *nelem_out = nelem;
  return FTK2B_OK;
}

extern "C" ftk2b_status ftk2b_fiber_surface_extract(ftk2b_ctx* ctx, const ftk2b_mesh_desc* mesh,
                                                    const ftk2b_field_desc* field, const double thresholds[2],
                                                    double sos_q, ftk2b_fiber_surface_result** out) {
  ftk2b::NvtxRange nvtx_range("ftk2b_fiber_surface_extract");
  if (!ctx) return FTK2B_INVALID_ARG;
  if (!mesh || !field || !thresholds || !out) return cfail(ctx, FTK2B_INVALID_ARG, "null argument");
  *out = nullptr;
  if (field->dtype != FTK2B_F32 && field->dtype != FTK2B_F64)
    return cfail(ctx, FTK2B_INVALID_ARG, "dtype must be FTK2B_F32 or FTK2B_F64");
  if (!(sos_q > 0)) return cfail(ctx, FTK2B_INVALID_ARG, "sos_q must be positive");
  if (mesh->kind == FTK2B_MESH_EXTRUDED) {
    if (field->ncomp != 2 || !field->comp[0] || !field->comp[1])
      return cfail(ctx, FTK2B_INVALID_ARG, "fiber surfaces read two scalar arrays (ncomp 2)");
    return fiber_surface_extruded(ctx, mesh, field, thresholds, sos_q, out);
  }
  if (mesh->kind != FTK2B_MESH_REGULAR || mesh->ndims != 4)
    return cfail(ctx, FTK2B_UNSUPPORTED, "fiber surfaces run on 3D+t meshes (ndims 4)");
  if (field->ncomp != 2 || field->layout != FTK2B_LAYOUT_SEPARATE || !field->comp[0] || !field->comp[1])
    return cfail(ctx, FTK2B_INVALID_ARG, "fiber surfaces read two scalar arrays (ncomp 2, layout SEPARATE)");
  CtGeom g;
  size_t nelem = 1;
  {
    const ftk2b_status gs = ct_geometry(ctx, mesh, field, g, &nelem);
    if (gs != FTK2B_OK) return gs;
  }
  if (g.nv >= 0xFFFFFFF0ull) return cfail(ctx, FTK2B_UNSUPPORTED, "mesh too large for fiber surfaces");
  // triangle types of a 4-cube: corner masks 0 < a < b with a a subset of b,
  // in (a, b) order
  FsTables tb;
  std::memset(&tb, 255, sizeof(tb));
  int nt = 0;
  for (int a = 1; a < 16; ++a)
    for (int b = a + 1; b < 16; ++b)
      if ((a & b) == a) {
        tb.ta[nt] = (unsigned char)a;
        tb.tb[nt] = (unsigned char)b;
        tb.idx[a][b] = (unsigned char)nt;
        ++nt;
      }
  if (nt != 50) return cfail(ctx, FTK2B_CUDA_ERROR, "triangle table has %d types", nt);
  const size_t es = field->dtype == FTK2B_F64 ? 8 : 4;
  if (cudaSetDevice(ctx->device) != cudaSuccess) return cfail(ctx, FTK2B_CUDA_ERROR, "cudaSetDevice failed");
  const void* dev[2] = {field->comp[0], field->comp[1]};
  if (field->location != FTK2B_DEVICE) {
    const int slot[2] = {kBufField, kBufField2};
    for (int j = 0; j < 2; ++j) {
      C_TRY(ctx->contour[slot[j]].ensure(nelem * es));
      C_TRY(cudaMemcpyAsync(ctx->contour[slot[j]].p, field->comp[j], nelem * es, cudaMemcpyHostToDevice,
                            ctx->stream));
      dev[j] = ctx->contour[slot[j]].p;
    }
  }
  auto* res = new (std::nothrow) ftk2b_fiber_surface_result;
  if (!res) return cfail(ctx, FTK2B_OOM, "result allocation failed");
  std::memset(res, 0, sizeof(*res));
  // triangles of the mesh: for each type, the corners c with c + b inside
  unsigned long long tris = 0;
  for (int t = 0; t < 50; ++t) {
    unsigned long long c = 1;
    for (int k = 0; k < 4; ++k) c *= ((tb.tb[t] >> k) & 1) ? g.L[k] - 1 : g.L[k];
    tris += c;
  }
  res->n_simplices = tris;
  const ftk2b_status st =
      field->dtype == FTK2B_F64
          ? run_fiber_surface<double>(ctx, g, tb, dev[0], dev[1], (double)thresholds[0], (double)thresholds[1],
                                      sos_q, res)
          : run_fiber_surface<float>(ctx, g, tb, dev[0], dev[1], (float)thresholds[0], (float)thresholds[1], sos_q,
                                     res);
  if (st != FTK2B_OK) {
    ftk2b_fiber_surface_result_free(res);
    return st;
  }
  *out = res;
  return FTK2B_OK;
}

extern "C" void ftk2b_fiber_surface_result_free(ftk2b_fiber_surface_result* r) {
  if (!r) return;
  std::free(r->simplices);
  std::free(r->lambda);
  std::free(r->barycentric);
  std::free(r->track_id);
  std::free(r->scalar);
  std::free(r->cells);
  delete r;
}

extern "C" void ftk2b_contour_result_free(ftk2b_contour_result* r) {
  if (!r) return;
  std::free(r->simplices);
  std::free(r->lambda);
  std::free(r->barycentric);
  std::free(r->track_id);
  std::free(r->scalar);
  std::free(r->cells);
  delete r;
}
