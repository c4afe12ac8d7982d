// Launches that overlap their predecessor in the stream (programmatic stream
// serialization), so that a chain of short kernels does not pay for a launch
// between each two: about 2.5 us a kernel.  The transpose and the normalisation
// launched so: 64 x 64 x 200 frames 266 -> 247 us a run, 512 x 512 x 1,000
// 430 -> 403 us, 512 x 512 x 5,000 streamed in blocks of 512 2.84 -> 2.61 ms.
#pragma once

#include "xpcs_internal.h"

namespace xg {

// A launch whose kernel may start before the one before it in the stream is
// complete, also as part of a captured graph.  The kernel itself waits for what
// it needs: overlap_after, or overlap_begin / overlap_end.
template <typename... Params, typename... Args>
void launch_overlapped(void (*kernel)(Params...), dim3 grid, int block, size_t smem,
                       cudaStream_t st, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  XG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
  XG_CHECK_LAUNCH();
}

// First in a kernel of a chain: waits until the kernel before is complete and its
// writes are visible, then lets the next one's blocks take their places as soon as
// all of this one's have theirs.  Each kernel of a chain waits, so each is
// complete only after all before it.
__device__ __forceinline__ void overlap_after() {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
}

// Kernels that need nothing from one another, the first launched plainly: each
// begins with overlap_begin (the next may start once every block of this one has)
// and ends with overlap_end (this kernel is complete only when the one before is,
// so that what follows in the stream waits for all of them).
__device__ __forceinline__ void overlap_begin() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void overlap_end() {
  if (blockIdx.x == 0 && threadIdx.x == 0) cudaGridDependencySynchronize();
}

}  // namespace xg
