// Programmatic dependent launch: a kernel launched through launch_pdl may start while the kernel before it in the stream
// still runs.  What it does before pdl_wait() (barriers, descriptors, index arithmetic) then hides behind the end of that kernel,
// as does the launch itself: 2 to 3 us per link of a chain of small kernels.
//
// The rules that every kernel launched this way keeps:
//  * all its threads that touch global memory call pdl_wait() before they do, in every CTA.  It returns when the kernels
//    before this one have completed and their writes are visible, so that chains of such kernels stay ordered;
//  * tensor memory is allocated after pdl_wait(): CTAs that wait must not hold what the kernel before them needs.  Sharing an
//    SM, the two would wait for each other;
//  * no thread waits for another kernel's CTA.
// A kernel that wants its CTAs on SMs of their own, but is small enough for two of them on one, is launched plainly: early CTAs
// gather on the SMs that are free first (the Cholesky inverse in an optimizer step of the 8B shape: 8142 us, launched early 8192).
// Newton-Schulz of one 256 x 256 matrix as 17 kernels 130 -> 103 us (it is one kernel now), a Muon step on ragged matrices (61)
// 992 -> 910, logits of 8 x 777 tokens (100) 1842 -> 1708.
// pdl_trigger() lets the next kernel of the stream start as soon as every CTA of this one has called it (or exited).
#pragma once

#include <cuda_runtime.h>

namespace dion {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cluster: CTAs per cluster along x (0: none)
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, unsigned cluster,
                       const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 0 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace dion
