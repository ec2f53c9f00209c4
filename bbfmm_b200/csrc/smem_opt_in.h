// Dynamic shared memory above 48 KB needs an opt-in per kernel and device.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace bbfmm {

// Opts Kernel into `bytes` on the current device, once per device of the process (a solver may be made
// on each). Safe with several threads: the call may be repeated, never left out.
template <auto Kernel>
cudaError_t smem_opt_in(int bytes) {
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute((const void *)Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace bbfmm
