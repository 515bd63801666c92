// Harness of tests/test_round_buffers.py: the set-up of a device's round buffers while
// the runtime's call number `fail` (counted from 1 over all calls of make) fails.
// Prints the failed attempt's status, which parts it left, what is still allocated,
// then the same after a second attempt that nothing disturbs.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "round_buffers.h"

static int fail_at, calls;
static std::set<void*> live;
static cudaError_t last = cudaSuccess;

static cudaError_t make(void** p, size_t n) {
  if (++calls == fail_at) {
    *p = reinterpret_cast<void*>(16);  // a failed call may leave anything there
    return last = cudaErrorMemoryAllocation;
  }
  live.insert(*p = std::malloc(n));
  return cudaSuccess;
}
static cudaError_t drop(void* p) {
  if (!live.erase(p)) std::abort();
  std::free(p);
  return cudaSuccess;
}

extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make(reinterpret_cast<void**>(s), 1); }
cudaError_t cudaMalloc(void** p, size_t n) { return make(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return make(p, n); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
cudaError_t cudaFree(void* p) { return drop(p); }
cudaError_t cudaFreeHost(void* p) { return drop(p); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
}

int main(int, char** argv) {
  fail_at = std::atoi(argv[1]);
  mccfr::RoundParts r;
  for (int attempt = 0; attempt < 2; ++attempt) {
    const cudaError_t e = r.make(100, 20);
    std::printf("%d %d %zu %d\n", (int)e, (r.stream != nullptr) + (r.h_up != nullptr) + (r.d_up != nullptr) +
                (r.h_err != nullptr) + (r.d_err != nullptr), live.size(), (int)last);
  }
  r.free_all();
  r.free_all();
  std::printf("%zu\n", live.size());
}
