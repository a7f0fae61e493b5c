// Kernel launches that follow one another without the gap that a full stop between them leaves.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace planmoe {

// Lets `kern` have `bytes` of dynamic shared memory.  The limit is the present device's, not the process's: `done`, a static of the
// call's place, has a bit for each device that has been told (one beyond the 64th is told every time).
template <class Kern>
cudaError_t allow_smem(Kern* kern, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

// Launches `kern`, which calls chain_begin() before it touches global memory, so that its blocks may take their places while the
// kernel before it ends (programmatic dependent launch).  Without that, 2.5 us lie between one kernel's end and the next one's
// work, in a pass of up to eighteen launches.  Only grids of at most one block per SM: blocks of a larger one may crowd onto the
// SMs that come free first, and nothing is gained (three runs each, us a pass as it is and with the row kernels chained too:
// inference of 16384 tokens with 16 experts 583 - 591 and 588 - 595, training on 8192 tokens with two 778 - 790 and 788 - 802).
// The GEMM kernels of one rank, whose grids are resident at once, set the attribute themselves.
// Kernels that deal with other ranks are neither launched so nor let the next one start early (chain_begin); others may be in a
// pass of several ranks, too: gates, column sums, weight gradients.
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
