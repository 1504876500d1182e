// launch.hpp -- launches of the step's kernel chains.
#pragma once
#include <cuda_runtime.h>

namespace h3c {

// Launches a kernel that starts with chain_begin() (fv_kernels.cuh) so that
// its set-up overlaps the kernel before it on the stream; captured into a
// graph, the edge between the two becomes a programmatic one.
template <class... P, class... A>
inline void launch_chain(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace h3c
