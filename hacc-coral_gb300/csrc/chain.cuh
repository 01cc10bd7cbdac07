// chain.cuh -- kernels that follow one another in a stream, each on the last
// one's results: launched so that the next grid's blocks are set up while the
// last one still runs (programmatic dependent launch).
//
// A kernel launched with launch_chained calls chain_enter() first, in every
// thread and before any return: it waits until the grid before it has ended
// and its writes are visible, then lets the grid after it be set up.  (A block
// that skipped the wait would let its grid end, and the next one start, before
// the grid two back is done.)  A kernel launched the usual way may stand
// anywhere between.
#pragma once

#include <cuda_runtime.h>

namespace hsr {

#if defined(__CUDACC__)
__device__ __forceinline__ void chain_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                           cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace hsr
