// round_buffers.h — what every round of a device needs before its first launch.
//
// Host code over the CUDA runtime alone, so that a test can let any of its calls fail.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>

namespace mccfr {

// A stream, an upload block and error flags, each pinned and on the device.  Made
// all together or not at all: a call that fails half-way gives back what it made, so
// the next one starts over and none meets a missing part.
struct RoundParts {
  cudaStream_t stream = nullptr;
  void *h_up = nullptr, *d_up = nullptr;
  void *h_err = nullptr, *d_err = nullptr;

  cudaError_t make(size_t up_bytes, size_t err_bytes) {
    if (stream) return cudaSuccess;
    cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) stream = nullptr;
    const auto part = [&e](void*& p, cudaError_t (*alloc)(void**, size_t), size_t bytes) {
      if (e != cudaSuccess) return;
      void* q = nullptr;
      e = alloc(&q, bytes);
      if (e == cudaSuccess) p = q;
    };
    const auto device = [](void** p, size_t n) { return cudaMalloc(p, n); };
    const auto pinned = [](void** p, size_t n) { return cudaMallocHost(p, n); };
    part(d_up, device, up_bytes);
    part(h_up, pinned, up_bytes);
    part(d_err, device, err_bytes);
    part(h_err, pinned, err_bytes);
    if (e != cudaSuccess) {
      free_all();
      cudaGetLastError();  // clear the allocation error
    }
    return e;
  }

  void free_all() {
    if (stream) cudaStreamDestroy(stream);
    if (h_up) cudaFreeHost(h_up);
    if (d_up) cudaFree(d_up);
    if (h_err) cudaFreeHost(h_err);
    if (d_err) cudaFree(d_err);
    stream = nullptr;
    h_up = d_up = h_err = d_err = nullptr;
  }
};

}  // namespace mccfr
