// tlr_pdl.cuh -- programmatic dependent launch of the triangular solves.
#pragma once

#include <cuda_runtime.h>

namespace tlr {

// Programmatic dependent launch: a solve kernel lets the next one launch
// right away (launch_dependents) and waits for its predecessor's results
// only where it reads them (wait); loads of factor data go out before the
// wait.  Both are no-ops for a kernel launched without the attribute.
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// launch, with programmatic stream serialisation when pdl (captured into
// the graph as a programmatic dependency on the previous kernel)
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl_smem(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                            size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st,
                       Args... args) {
  return launch_pdl_smem(pdl, kernel, grid, block, 0, st, args...);
}

}  // namespace tlr
