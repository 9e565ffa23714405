// The limit of a kernel's dynamic shared memory on the current device.
#pragma once
#include <cuda_runtime.h>

#include "../core/per_device.h"

namespace amem {

// Allows `kernel` `bytes` of dynamic shared memory on the current device; `done` remembers where that was said already.
template <typename K>
cudaError_t allow_smem(OncePerDevice& done, K* kernel, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  return done(dev, [&] { return cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
}

}  // namespace amem
