// block_pool.h — device memory that comes in equal blocks, and may be less than wanted.
//
// Host code over the CUDA runtime's allocator alone, so that a test can put an
// allocator that fails in its place.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>

namespace mccfr {

// Up to `want` blocks of `per_block` bytes and `extra` bytes behind them, in one
// allocation.  Fewer blocks are tried while the device is short of memory, and what
// a request got is kept for it: a later one of no more blocks neither frees nor
// allocates, whatever it got.
struct BlockPool {
  void* p = nullptr;
  int blocks = 0;  // that there is room for
  int asked = 0;   // the largest request answered

  bool holds(int want) const { return p && want <= asked; }

  cudaError_t take(int want, size_t per_block, size_t extra) {
    free();
    for (int n = want;; n = (n + 1) / 2) {
      const cudaError_t e = cudaMalloc(&p, n * per_block + extra);
      if (e == cudaSuccess) {
        blocks = n;
        asked = want;
        return e;
      }
      p = nullptr;
      cudaGetLastError();  // clear the allocation error
      if (e != cudaErrorMemoryAllocation || n <= 1) return e;
    }
  }

  void free() {
    if (p) cudaFree(p);
    p = nullptr;
    blocks = asked = 0;
  }
};

}  // namespace mccfr
