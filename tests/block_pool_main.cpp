// Harness of tests/test_block_pool.py: the library's block pool over an allocator that
// holds at most `room` bytes.  Arguments: room, then requests (blocks of 100 bytes, 28
// behind them); "r<bytes>" changes the room.  Prints, per request, the status, the
// blocks got and the allocations tried so far; at the end what is still allocated.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "block_pool.h"

static size_t room, used;
static int tries;
static std::map<void*, size_t> live;
static cudaError_t last = cudaSuccess;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  ++tries;
  if (used + n > room) return last = cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  live[*p] = n;
  used += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  used -= live.at(p);
  live.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
}

int main(int argc, char** argv) {
  room = std::strtoull(argv[1], nullptr, 10);
  mccfr::BlockPool pool;
  for (int i = 2; i < argc; ++i) {
    if (argv[i][0] == 'r') {
      room = std::strtoull(argv[i] + 1, nullptr, 10);
      continue;
    }
    const int want = std::atoi(argv[i]);
    const cudaError_t e = pool.holds(want) ? cudaSuccess : pool.take(want, 100, 28);
    std::printf("%d %d %d\n", (int)e, pool.blocks, tries);
  }
  pool.free();
  std::printf("%zu %d\n", used, (int)last);
}
