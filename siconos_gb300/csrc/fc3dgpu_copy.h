// Host to device on the stream whose kernels read the data.  A plain cudaMemcpy
// from pageable memory returns when small data is staged, before it has
// arrived, and the contexts' streams do not wait for the default stream it runs
// on: a kernel launched right behind it could read what was there before.
// The way back is on that stream too: a copy on the default stream had no turn for
// as long as two other threads kept cooperative launches queued (none in 3 s
// beside a 2D and a 3D solver in a loop).
#pragma once
#include <cuda_runtime.h>

static inline cudaError_t copy_to_device(void* d, const void* h, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return cudaSuccess;
  const cudaError_t e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s);
  return e == cudaSuccess ? cudaStreamSynchronize(s) : e;  // the host buffer is the caller's again
}

static inline cudaError_t copy_to_host(void* h, const void* d, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return cudaSuccess;
  const cudaError_t e = cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, s);
  return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}
