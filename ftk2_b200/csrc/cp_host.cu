#include "cp_host.h"

#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <memory>
#include <new>
#include <thread>

#include "cp_api_internal.h"

namespace ftk2b {

namespace {

size_t host_threads(size_t bytes) {
  const size_t cores = std::thread::hardware_concurrency();
  return std::max<size_t>(1, std::min({kHostThreads, cores / 2, bytes / kHostThreadBytes}));
}

// runs body(0) .. body(k - 1), all but the first on threads of their own while
// those can be started
template <typename F>
void run_threads(size_t k, F body) {
  std::thread th[kHostThreads];
  size_t started = 1;
  try {
    for (; started < k; ++started) th[started] = std::thread(body, started);
  } catch (const std::exception&) {  // no thread, or no memory for one
  }
  body(0);
  for (size_t i = started; i < k; ++i) body(i);
  for (size_t i = 1; i < started; ++i) th[i].join();
}

}  // namespace

void host_parallel(size_t n, size_t bytes, void (*f)(void*, size_t, size_t), void* arg) {
  const size_t k = std::min(host_threads(bytes), std::max<size_t>(n, 1));
  if (k <= 1) {
    f(arg, 0, n);
    return;
  }
  run_threads(k, [&](size_t i) { f(arg, n * i / k, n * (i + 1) / k); });
}

void* host_alloc(size_t bytes) {
  constexpr size_t kHuge = size_t(2) << 20;
  if (bytes < 2 * kHuge) return std::malloc(bytes ? bytes : 1);
  void* p = nullptr;
  const size_t n = (bytes + kHuge - 1) / kHuge * kHuge;
  if (posix_memalign(&p, kHuge, n) != 0) return nullptr;
  madvise(p, n, MADV_HUGEPAGE);
  return p;
}

HostWords::~HostWords() { std::free(p_); }

bool HostWords::alloc(size_t n) {
  std::free(p_);
  n_ = 0;
  p_ = n <= SIZE_MAX / 16 ? static_cast<uint64_t*>(host_alloc(8 * n)) : nullptr;
  if (p_) n_ = n;
  return p_ != nullptr;
}

namespace {

// Blocks of 32,768 words are hashed apart (by any thread) in four interleaved
// chains, each a multiply per word: one chain over everything is bound by the
// multiplier's latency (27 ms for the 9.2 million words of a 100 x 100 x 40
// tet mesh).
constexpr size_t kHashBlock = 32768;

inline uint64_t mix(uint64_t h, uint64_t x) {
  h ^= x + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2);
  return h * 0xBF58476D1CE4E5B9ull;
}

uint64_t hash_block(const uint64_t* p, size_t n) {
  uint64_t h[4] = {1, 2, 3, 4};
  size_t i = 0;
  for (; i + 4 <= n; i += 4)
    for (int j = 0; j < 4; ++j) h[j] = mix(h[j], p[i + j]);
  for (; i < n; ++i) h[0] = mix(h[0], p[i]);
  return mix(mix(mix(h[0], h[1]), h[2]), h[3]);
}

uint64_t hash_blocks(size_t n, const uint64_t* src, uint64_t* copy_to, const void* copy_from) {
  const size_t nb = (n + kHashBlock - 1) / kHashBlock;
  auto block = [&](size_t b) {
    const size_t lo = b * kHashBlock, m = std::min(kHashBlock, n - lo);
    if (copy_to) std::memcpy(copy_to + lo, static_cast<const char*>(copy_from) + 8 * lo, 8 * m);
    return hash_block((copy_to ? copy_to : src) + lo, m);
  };
  std::unique_ptr<uint64_t[]> hb(new (std::nothrow) uint64_t[nb ? nb : 1]);
  if (hb)
    host_parallel(nb, 8 * n, [&](size_t b0, size_t b1) {
      for (size_t b = b0; b < b1; ++b) hb[b] = block(b);
    });
  uint64_t h = 0x9E3779B97F4A7C15ull ^ n;
  for (size_t b = 0; b < nb; ++b) h = mix(h, hb ? hb[b] : block(b));
  return h;
}

}  // namespace

uint64_t hash_words(const uint64_t* p, size_t n) { return hash_blocks(n, p, nullptr, nullptr); }

uint64_t copy_hash_words(uint64_t* dst, const void* src, size_t n) { return hash_blocks(n, nullptr, dst, src); }

namespace {
constexpr size_t kRingChunk = size_t(1) << 20;
constexpr size_t kRingChunks = 16;
static_assert(kRingChunks == sizeof(ftk2b_ctx::d2h_ev) / sizeof(cudaEvent_t), "an event per chunk of the ring");
}  // namespace

cudaError_t copy_to_host(ftk2b_ctx* ctx, std::initializer_list<HostCopy> copies) {
  size_t sum = 0;
  for (const HostCopy& c : copies) sum += (c.bytes + 15) & ~size_t(15);
  if (sum <= ctx->pin.bytes - 256) {  // the context's own pinned block holds everything
    ctx->pack_ready = false;
    char* p = static_cast<char*>(ctx->pin.h) + 256;
    cudaError_t e = cudaSuccess;
    size_t o = 0;
    for (const HostCopy& c : copies) {
      if (c.bytes && !e) e = cudaMemcpyAsync(p + o, c.src, c.bytes, cudaMemcpyDeviceToHost, ctx->stream);
      o += (c.bytes + 15) & ~size_t(15);
    }
    const cudaError_t se = cudaStreamSynchronize(ctx->stream);
    if (e || se) return e ? e : se;
    o = 0;
    for (const HostCopy& c : copies) {
      if (c.bytes) std::memcpy(c.dst, p + o, c.bytes);
      o += (c.bytes + 15) & ~size_t(15);
    }
    return cudaSuccess;
  }
  if (!ctx->d2h_ring.h && ctx->d2h_ring.alloc(kRingChunk * kRingChunks) != cudaSuccess) {
    // no memory to pin: the driver's own copies
    cudaError_t e = cudaSuccess;
    for (const HostCopy& c : copies)
      if (c.bytes && !e) e = cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, ctx->stream);
    const cudaError_t se = cudaStreamSynchronize(ctx->stream);
    return e ? e : se;
  }
  for (cudaEvent_t& ev : ctx->d2h_ev)
    if (!ev) {
      const cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
      if (e) {
        ev = nullptr;
        return e;
      }
    }
  size_t total = 0, np = 0;
  for (const HostCopy& c : copies) {
    total += c.bytes;
    np += (c.bytes + kRingChunk - 1) / kRingChunk;
  }
  // piece i of the copies, each cut into chunks
  auto piece = [&copies](size_t i) {
    for (const HostCopy& c : copies) {
      const size_t n = (c.bytes + kRingChunk - 1) / kRingChunk, o = i * kRingChunk;
      if (i < n)
        return HostCopy{static_cast<char*>(c.dst) + o, static_cast<const char*>(c.src) + o,
                        std::min(kRingChunk, c.bytes - o)};
      i -= n;
    }
    return HostCopy{nullptr, nullptr, 0};
  };
  char* ring = static_cast<char*>(ctx->d2h_ring.h);
  // piece i uses chunk i % kRingChunks; whoever empties a chunk queues the
  // next piece into it, so no thread waits for a free chunk
  std::atomic<size_t> next{0};
  std::atomic<int> err{0};
  auto queue = [&](size_t i) {
    const size_t s = i % kRingChunks;
    const HostCopy c = piece(i);
    cudaError_t e = cudaMemcpyAsync(ring + s * kRingChunk, c.src, c.bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (!e) e = cudaEventRecord(ctx->d2h_ev[s], ctx->stream);
    if (e) err.store((int)e);
    return e == cudaSuccess;
  };
  // queued[s]: one past the last piece queued into chunk s
  std::atomic<size_t> queued[kRingChunks];
  for (auto& q : queued) q.store(0);
  for (size_t i = 0; i < std::min(np, kRingChunks); ++i) {
    if (!queue(i)) break;
    queued[i].store(i + 1);
  }
  const int device = ctx->device;
  run_threads(total < kCopyThreadBytes ? 1 : std::min(host_threads(total), np), [&](size_t t) {
    if (t && cudaSetDevice(device) != cudaSuccess) {
      err.store((int)cudaErrorUnknown);
      return;
    }
    for (;;) {
      const size_t i = next.fetch_add(1);
      if (i >= np) return;
      const size_t s = i % kRingChunks;
      // piece i is queued by the thread that empties piece i - kRingChunks
      while (queued[s].load(std::memory_order_acquire) != i + 1) {
        if (err.load()) return;
        std::this_thread::yield();
      }
      const cudaError_t e = cudaEventSynchronize(ctx->d2h_ev[s]);
      if (e) {
        err.store((int)e);
        return;
      }
      const HostCopy c = piece(i);
      std::memcpy(c.dst, ring + s * kRingChunk, c.bytes);
      if (i + kRingChunks < np) {
        if (!queue(i + kRingChunks)) return;
        queued[s].store(i + kRingChunks + 1, std::memory_order_release);
      }
    }
  });
  const cudaError_t se = cudaStreamSynchronize(ctx->stream);
  return err.load() ? (cudaError_t)err.load() : se;
}

}  // namespace ftk2b
