// Dynamic shared memory of kernels whose size follows the grid.
//
// The limit set by cudaFuncSetAttribute belongs to the kernel for the whole
// process, not to the context that set it: a limit fitted to one grid refuses
// the launches of a larger grid that was set up before it.  So these kernels
// get the largest limit the device allows, which no later call lowers; what a
// launch takes is its own argument.  (Kernels of a compile-time length always
// set the same value.)
#pragma once
#include <cuda_runtime.h>

namespace sb {

constexpr int SMEM_BLOCK_MAX = 227 * 1024;  // per block, static and dynamic (sm_100)

template <class K>
inline cudaError_t smem_max(K kernel) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              SMEM_BLOCK_MAX - (int)a.sharedSizeBytes);
}

}  // namespace sb
