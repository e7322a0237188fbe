// Kernel launches inside one call: the kernels of a call run back to back on one stream and each depends on the one
// before it. A programmatic dependent launch lets the next kernel's blocks start while the last ones of the current
// kernel drain; pdl_wait() is where a kernel first touches what the kernels before it wrote (it returns when they have
// completed and their writes are visible), pdl_trigger() lets the next one be scheduled. The trigger stands at a kernel's
// end: given at its start, blocks of the next kernel sat in slots that the current one still needed (a [1,24,4608,128]
// call took 207 us, 195 without dependent launches, 188 like this). Without the launch attribute both are no-ops.
// No block leaves a kernel in front of pdl_wait() by a return: if all of them did, the kernel would end before the one it
// depends on, and what follows on the stream (the next user of the workspace) waits for this one only.
// A kernel with a pdl_wait() takes no `const T* __restrict__`: that promises data which nothing writes while the kernel runs,
// so that loads may go through the non-coherent path and in front of the wait, and the kernel before it still writes.
#pragma once
#include <cuda_runtime.h>

namespace sparge {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool dependent, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
  if (e != cudaSuccess) cudaGetLastError();   // reported by the caller's status: the next check of this thread is not about it
  return e;
}

}  // namespace sparge
