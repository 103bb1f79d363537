// Programmatic dependent launch (PDL): a kernel chained to its predecessor on
// a stream may be scheduled while that one drains.  It does what does not
// depend on the predecessor (index arithmetic, constant tables), waits for
// the predecessor's results with wait_for_predecessor(), and lets its own
// successor come up with release_successor().  The wait returns only when the
// predecessor has completed and its writes are visible, so the order of
// results is that of plain launches.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace lbmc {

__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_successor() { asm volatile("griddepcontrol.launch_dependents;"); }

template <class... Args>
inline cudaError_t launch_chained(void (*kernel)(Args...), dim3 grid, dim3 block, cudaStream_t stream,
                                  typename std::common_type<Args>::type... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace lbmc
