// Loaded ahead of libftk2b.so, this takes the place of its cull: the real one
// runs (its candidates are queued) and, when asked to, the error word is set
// as a block does whose bounded copy wait ran out.  Nothing fails on the GPU.
#include <dlfcn.h>

#include "../../ftk2_b200/csrc/cp_internal.h"

namespace {
void* library = nullptr;
int failures = 0;
}  // namespace

extern "C" int failing_cull_library(const char* path) {
  library = dlopen(path, RTLD_NOW | RTLD_NOLOAD);
  return library != nullptr;
}
extern "C" void failing_cull_next(int n) { failures = n; }

namespace ftk2b {

cudaError_t launch_extract_regular(int f64, const RegularMesh& mesh, const FieldAccess& fa, const ExtractConfig& cfg,
                                   const CandidateQueue& cq, unsigned* err, cudaStream_t st, bool allow_tma,
                                   int* used_tma, int* launches) {
  Dl_info self;
  if (!library || !dladdr(reinterpret_cast<void*>(&launch_extract_regular), &self)) return cudaErrorUnknown;
  auto real = reinterpret_cast<decltype(&launch_extract_regular)>(dlsym(library, self.dli_sname));
  if (!real || real == &launch_extract_regular) return cudaErrorUnknown;
  const cudaError_t e = real(f64, mesh, fa, cfg, cq, err, st, allow_tma, used_tma, launches);
  if (e || failures == 0) return e;
  --failures;
  return cudaMemsetAsync(err, 2, 1, st);  // the low byte: bit 1
}

}  // namespace ftk2b
