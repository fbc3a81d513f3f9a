// work_pool.h -- work buffers of one call, allocated and freed in stream order.
#pragma once

#include <cuda_runtime.h>

namespace qgb
{

// The device's pool for work buffers (capi.cu).  It keeps at most 1 GiB from
// call to call; beyond that the memory goes back to the device when a stream
// is next synchronised.
cudaError_t work_pool(cudaMemPool_t* out);

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
    cudaMemPool_t pool = nullptr;
    cudaError_t e = work_pool(&pool);
    st = stream;
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&p, bytes > 0 ? bytes : 1, pool, stream);
    if (e != cudaSuccess) p = nullptr;
    return e;
  }
};

}  // namespace qgb
