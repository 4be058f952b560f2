// Host memory traffic of the calls that move many megabytes: allocation,
// copies and content hashes by several threads.
//
// One core touches new memory at a few GB/s (a page fault per 4 KB) and copies
// at about 10, far below the 50 GB/s the device delivers over PCIe, so from
// kHostThreadBytes on the work is shared by up to kHostThreads threads that
// live for the call.  Below that, starting them (about 20 us each) costs more
// than it saves.
#pragma once

#include <cstddef>
#include <cstdint>
#include <initializer_list>

#include <cuda_runtime.h>

struct ftk2b_ctx;

namespace ftk2b {

constexpr size_t kHostThreads = 8;
constexpr size_t kHostThreadBytes = size_t(2) << 20;  // per thread, at least
// Copies from the device take several threads from here on: a thread that
// calls the driver costs 0.1 to 0.6 ms to start and end, and which it is varies
// from call to call.  Level sets of 4.3 and 9 MB: 485 to 800 and 530 to 1,060 us
// a call with several threads, 577 and 774 with one; of 20 MB 1,340 against 1,545.
constexpr size_t kCopyThreadBytes = size_t(16) << 20;

// f(begin, end) over [0, n) in contiguous shares, one per thread; `bytes` is
// the memory the whole range touches.  A thread that cannot be started leaves
// its share to the caller.  None of this file's functions throws or needs memory
// of its own to succeed: they are called below C entry points.
void host_parallel(size_t n, size_t bytes, void (*f)(void* arg, size_t begin, size_t end), void* arg);
template <typename F>
void host_parallel(size_t n, size_t bytes, F f) {
  host_parallel(n, bytes, [](void* arg, size_t begin, size_t end) { (*static_cast<F*>(arg))(begin, end); }, &f);
}

// Memory for a large array, released with free(); from 4 MB on aligned and
// advised for 2 MB pages, which fault once per 2 MB instead of once per 4 KB.
void* host_alloc(size_t bytes);

// 64-bit content hash of n words (any change to how it is formed is a change
// of the checkpoint format: a blob holds it).
uint64_t hash_words(const uint64_t* p, size_t n);

// Uninitialised array of 64-bit words of host_alloc memory.
class HostWords {
 public:
  HostWords() = default;
  HostWords(const HostWords&) = delete;
  HostWords& operator=(const HostWords&) = delete;
  ~HostWords();
  bool alloc(size_t n);
  uint64_t* data() const { return p_; }
  size_t size() const { return n_; }
  bool empty() const { return n_ == 0; }

 private:
  uint64_t* p_ = nullptr;
  size_t n_ = 0;
};

// Copies src (any alignment) to dst and returns the words' hash.
uint64_t copy_hash_words(uint64_t* dst, const void* src, size_t n);

struct HostCopy {
  void* dst;
  const void* src;  // device
  size_t bytes;
};

// Device arrays to pageable host memory through a ring of pinned chunks of the
// context: the host threads empty chunks while the next ones arrive.  Waits
// for the copies (and all work queued on the stream before).
cudaError_t copy_to_host(ftk2b_ctx* ctx, std::initializer_list<HostCopy> copies);

}  // namespace ftk2b
