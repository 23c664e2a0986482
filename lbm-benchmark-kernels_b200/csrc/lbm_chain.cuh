// lbm_chain.cuh -- back-to-back step kernels of one stream without the launch
// gap (programmatic dependent launch).
//
// A kernel launched with launch_chained may start while its predecessor in the
// stream drains: its blocks are set up, and what never changes (items, run
// records) is fetched, before chain_wait(), which returns once the predecessor
// has completed and its writes are visible. Every thread calls chain_wait()
// before it reads or writes anything that another kernel writes, and before
// any return, so that a kernel never completes before its predecessor.
// chain_next() lets the successor start; it does so once every block of this
// kernel has called it or ended, so waiting blocks of the successor never keep
// out blocks of this one.
#pragma once
#include <cuda_runtime.h>

namespace lbm {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Grids of fewer than about 4 blocks per SM (of 148) leave it to the blocks' ends: the
// successor's blocks, placed beside theirs, would crowd on the SMs that free up
// first. us per step, plain launches / from the start / at the ends: list pull
// 172 tiles 6.2 / 5.4 / 4.1, 408 tiles 8.2 / 5.8 / 5.2, 3274 tiles 53.0 / 49.0 /
// 50.7; batch FP32 of 82 tiles 2.8 / 3.1 / 2.4, 850 tiles 6.9 / 6.0 / 6.5.
constexpr unsigned kChainEarlyBlocks = 592;
__device__ __forceinline__ void chain_next() {
  if (gridDim.x >= kChainEarlyBlocks) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// A launch whose blocks are all resident at once (they wait for one another).
template <class... P, class... A>
void launch_together(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace lbm
