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

// Launch with programmatic stream serialization: the kernel's set-up (barriers, TMEM, descriptors) overlaps
// the tail of the kernel before it; the kernel calls grid_dep_wait() before it touches global memory.
// A launch after a launch costs 1 to 2 us less for it (measured back to back: N = 512, 2 x 8 heads 11.6 ->
// 11.2 us; D = 64, N = 1024, 4 x 12 heads causal 20.5 -> 18.6; decode of 16 x 4001 keys 50.5 -> 48.7).
template <typename Kernel, typename... Args>
inline cudaError_t launch_overlapped(Kernel kern, dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                                     const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace ma
