// Host-side helper of the kernel launchers.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace ma {

// The opt-in to more than 48 KB of dynamic shared memory is per function and per device; it is
// made once for each (the reference does it at import, flash_attention.cu:140-147), not on every
// launch.  `done` holds one bit per device ordinal.
inline cudaError_t allow_dynamic_smem(const void* kern, int bytes, std::atomic<unsigned long long>* done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool tracked = dev >= 0 && dev < 64;
  if (tracked && ((done->load(std::memory_order_acquire) >> dev) & 1ull)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && tracked) done->fetch_or(1ull << dev, std::memory_order_release);
  return e;
}

}  // namespace ma
