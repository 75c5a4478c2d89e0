// Leave for a kernel to take a launch's dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace esl {

// The limit belongs to the kernel on the device, for every thread of the
// process: set to each launch's own size, one thread's could fall between
// another's call here and its launch, which then failed. So it is always set
// to all that a CTA may have beside the kernel's static shared memory.
template <class K>
inline cudaError_t allow_smem(K* kernel, size_t bytes) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess) return e;
  const size_t most = size_t(227) * 1024 - a.sharedSizeBytes;
  if (bytes > most) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most));
}

}  // namespace esl
