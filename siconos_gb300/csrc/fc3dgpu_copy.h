// Host to device on the stream whose kernels read the data.  A plain cudaMemcpy
// from pageable memory returns when small data is staged, before it has
// arrived, and the contexts' streams do not wait for the default stream it runs
// on: a kernel launched right behind it could read what was there before.
#pragma once
#include <cuda_runtime.h>

static inline cudaError_t copy_to_device(void* d, const void* h, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return cudaSuccess;
  const cudaError_t e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s);
  return e == cudaSuccess ? cudaStreamSynchronize(s) : e;  // the host buffer is the caller's again
}
