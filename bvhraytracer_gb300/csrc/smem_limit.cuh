// Dynamic shared memory above the default 48 KB per block.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace bvhgpu {
namespace dev {

// Prepares a launch of `kernel` with `bytes` of dynamic shared memory. The
// limit is a property of the kernel, not of a launch: set to what each launch
// takes, a thread's launch of less would undercut another thread's of more
// between its two calls. So it is always set to all that a block may have.
template <typename K>
inline cudaError_t allow_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              227 * 1024 - (int)a.sharedSizeBytes);
}

}  // namespace dev
}  // namespace bvhgpu
