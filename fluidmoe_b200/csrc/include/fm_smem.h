// A kernel's limit of dynamic shared memory.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace fm {

// Raises a kernel's limit, which belongs to the device, once for each of the first 64 devices and at every launch for others;
// `done` is a static of the launcher.
inline cudaError_t allow_smem(const void* kernel, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

}  // namespace fm
