// Launches that overlap their set-up with the end of the kernel before them in the stream
// (programmatic dependent launch).  A kernel launched by launchAfter() begins with gridWait(): its
// blocks may be placed on the SMs while the kernel before it still runs, and touch memory only once
// that kernel has finished and its writes are visible.  Every kernel that calls gridWait() lets the
// next one be placed as soon as all its own blocks run; since each kernel of a chain waits for the
// one before it before it ends, the order of the whole chain is kept.  After a kernel or a copy
// that gives no such signal the launch is an ordinary one.
//
// Taken by the tiled path, whose evaluation of one chain is eight short kernels in a row, and by
// the clearing and conversion kernels (one 2,500-atom chain with copies 116 -> 98 us; 1,024
// molecules, through the latter alone, 389 -> 380).  Not by the fused evaluation, whose large units
// come first and are then placed on the SMs that happen to be free (1,024 molecules 389 -> 436 us),
// the FP64 passes (128 molecules 206 -> 216) or the line-search kernels.  The graph minimizer's
// captured cycle begins with the clearing kernel, to which nothing in the graph is a predecessor,
// and holds the tiled passes of molecules on the tiled path as programmatic edges; its fused
// evaluations and line-search steps are ordinary nodes (all of them launched this way: one
// molecule, 60 cycles 4.38 -> 4.59 ms).
#ifndef STORMM_B200_LAUNCH_CUH
#define STORMM_B200_LAUNCH_CUH

#include <cuda_runtime.h>

#include <utility>

namespace sb {

__device__ __forceinline__ void gridWait() {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
}

template <class... Params, class... Args>
cudaError_t launchAfter(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem,
                        cudaStream_t stream, Args &&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace sb

#endif
