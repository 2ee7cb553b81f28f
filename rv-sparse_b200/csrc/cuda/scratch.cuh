// Device scratch of the Matrix Market passes, out of a pool (k_coo.cu).
#pragma once

#include <cuda_runtime.h>

namespace rvsp {

// The current device's pool, or nullptr when it could not be made.
cudaMemPool_t scratch_pool();

// Device scratch of one call, from the pool (cudaMalloc when the pool could
// not be made), released in stream order when the call returns.
struct Scratch {
  static constexpr int kSlots = 16;
  void *p[kSlots] = {};
  int n = 0;
  cudaStream_t s = nullptr;
  cudaMemPool_t pool = nullptr;
  explicit Scratch(cudaStream_t st) : s(st), pool(scratch_pool()) {}
  cudaError_t alloc(void **out, size_t bytes) {
    if (n >= kSlots) return cudaErrorMemoryAllocation;  // more buffers than slots
    const size_t b = bytes ? bytes : 1;
    cudaError_t e = pool ? cudaMallocFromPoolAsync(out, b, pool, s) : cudaMalloc(out, b);
    if (e == cudaSuccess) p[n++] = *out;
    return e;
  }
  ~Scratch() {
    for (int i = 0; i < n; ++i) {
      if (pool) cudaFreeAsync(p[i], s);
      else cudaFree(p[i]);
    }
  }
};

}  // namespace rvsp
