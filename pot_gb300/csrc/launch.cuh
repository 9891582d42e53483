// Host-side launch helpers.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace otg {

// Lets kernel `k` be launched with `smem` bytes of dynamic shared memory.  The
// limit belongs to the kernel, not to the launch: set to what one call needs,
// it failed the launch of another thread that had just set it to more.  It is
// only ever raised, to all that the device gives.
inline bool allow_smem(const void* k, size_t smem) {
  cudaFuncAttributes a;
  int dev = 0, most = 0;
  if (cudaFuncGetAttributes(&a, k) != cudaSuccess) { cudaGetLastError(); return false; }
  if ((size_t)a.maxDynamicSharedSizeBytes >= smem) return true;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  most -= (int)a.sharedSizeBytes;
  if (most > 0 && (size_t)most >= smem &&
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}

}  // namespace otg
