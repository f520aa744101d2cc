// Host side of kernel launches.
#pragma once
#include <atomic>
#include <cuda_runtime_api.h>

extern "C" void msb_set_error(const char* fmt, ...);

namespace msb {
// Lets `kern` be launched with `bytes` of dynamic shared memory on the current device.  The limit belongs to the device, so it is
// stated once per device of the process; `stated` is the launcher's own record (a bit per device, static).
inline int allow_smem(const void* kern, int bytes, const char* what, std::atomic<unsigned long long>& stated) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;      // devices past the record are told every time
  if (e == cudaSuccess && (stated.load(std::memory_order_relaxed) & bit)) return 0;
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) {
    msb_set_error("%s: cannot set %d bytes of dynamic shared memory: %s", what, bytes, cudaGetErrorString(e));
    return 1;
  }
  stated.fetch_or(bit, std::memory_order_relaxed);
  return 0;
}
}  // namespace msb
