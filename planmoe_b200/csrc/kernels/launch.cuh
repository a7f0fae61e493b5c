// Kernel launches that follow one another without the gap that a full stop between them leaves.
#pragma once

#include <cuda_runtime.h>

namespace planmoe {

// Launches `kern`, which calls chain_begin() before it touches global memory, so that its blocks may take their places while the
// kernel before it ends (programmatic dependent launch).  Without that, 2.5 us lie between one kernel's end and the next one's
// work, in a pass of up to eighteen launches.  Only grids of at most one block per SM: blocks of a larger one would crowd onto
// the SMs that come free first, and a kernel that is one wave of the chip then lasts as long as the fullest SM (16384 tokens,
// 16 experts, with the row kernels chained too: 569 us a pass, without 546).
constexpr unsigned kChainedBlocks = 148;

template <class... Params, class... Args>
cudaError_t launch_chained(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (unsigned long long)grid.x * grid.y * grid.z <= kChainedBlocks ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

}  // namespace planmoe
