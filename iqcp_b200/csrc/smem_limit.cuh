// Dynamic shared memory beyond the default limit.
#pragma once
#include <cuda_runtime.h>

namespace iqcp {

// Lets `kernel` be launched with `smem` bytes of dynamic shared memory on the
// current device.  The limit is one value per function, shared by every host
// thread, so it is always raised to the device's own (less the kernel's static
// arrays), never to one call's size: a thread that sets a smaller size between
// another's setting and launch makes that launch fail.
template <typename K>
cudaError_t allow_dynamic_smem(K kernel, size_t smem) {
  if (smem <= 32 * 1024) return cudaSuccess;  // within the default 48 KB beside the static arrays
  int dev = 0, optin = 0;
  cudaFuncAttributes fa;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
  if (e != cudaSuccess) return e;
  if (smem + fa.sharedSizeBytes > (size_t)optin) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

}  // namespace iqcp
