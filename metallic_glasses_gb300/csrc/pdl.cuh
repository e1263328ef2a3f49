// pdl.cuh -- programmatic dependent launch. A kernel launched by launch_pdl may
// be scheduled while the previous kernel of its stream finishes; its threads
// read nothing that a kernel writes before pdl_wait, which waits for the
// previous kernel and its writes. pdl_release lets the next one be scheduled
// once every block has reached it (or returned).
#pragma once
#include <cuda_runtime.h>

namespace stz {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `early` 0: an ordinary launch.
template <typename... A, typename... B>
void launch_pdl(void (*kern)(A...), dim3 grid, int threads, size_t smem, cudaStream_t st, int early, B&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, static_cast<A>(args)...);
}

}  // namespace stz
