// work_pool.h -- work buffers of one call, allocated and freed in stream order.
#pragma once

#include <cuda_runtime.h>

namespace qgb
{

// A work buffer of the device's pool (capi.cu); when the device has run out, tried again without the library's idle
// memory.
cudaError_t work_alloc(void** p, size_t bytes, cudaStream_t st);
// Returns the pool's unused memory to the device; adds the bytes to *released.
void trim_work_pool(int64_t* released);
// cudaMalloc with that second try.
cudaError_t alloc_or_release(void** p, size_t bytes);

// A buffer of the work pool, freed in stream order when it goes out of scope.
// Each call owns its buffers, so calls of several threads share none.
struct WorkBuf {
  void* p = nullptr;
  cudaStream_t st = nullptr;
  WorkBuf() = default;
  WorkBuf(const WorkBuf&) = delete;
  WorkBuf& operator=(const WorkBuf&) = delete;
  ~WorkBuf()
  {
    if (p) cudaFreeAsync(p, st);
  }
  cudaError_t alloc(size_t bytes, cudaStream_t stream)
  {
    st = stream;
    return work_alloc(&p, bytes, stream);
  }
};

}  // namespace qgb
