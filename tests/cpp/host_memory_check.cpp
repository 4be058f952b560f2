// The threaded host functions below the C entry points when memory runs out:
// the results of a run with memory, and nothing thrown.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "../../ftk2_b200/csrc/cp_host.h"

static bool no_memory = false;

void* operator new(std::size_t n) {
  void* p = no_memory ? nullptr : std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main() {
  const size_t n = (size_t(5) << 20) + 17;  // 40 MB: several threads
  std::vector<uint64_t> a(n), b(n), c(n);
  for (size_t i = 0; i < n; ++i) a[i] = i * 0x9E3779B97F4A7C15ull;
  const uint64_t h = ftk2b::hash_words(a.data(), n);
  const char* odd = reinterpret_cast<const char*>(a.data()) + 3;
  const uint64_t g = ftk2b::copy_hash_words(b.data(), odd, n - 1);
  no_memory = true;
  bool ok = ftk2b::hash_words(a.data(), n) == h && ftk2b::copy_hash_words(c.data(), odd, n - 1) == g;
  size_t calls = 0;
  if (ok && std::getenv("HASH_ONLY") == nullptr) {
    ftk2b::host_parallel(n, 8 * n, [&](size_t lo, size_t hi) {
      for (size_t i = lo; i < hi; ++i) b[i] = i;
      ++calls;  // no thread could be started: all on this one
    });
    for (size_t i = 0; i < n; ++i) ok = ok && b[i] == i;
    ok = ok && calls > 0;
    ftk2b::HostWords w;
    ok = ok && !w.alloc(SIZE_MAX / 4) && w.empty() && w.alloc(3);
  }
  no_memory = false;
  std::puts(ok ? "ok" : "wrong");
  return ok ? 0 : 1;
}
