// Launching a kernel so that its start overlaps the end of the kernel before it on the stream
// (programmatic dependent launch).
//
// A small layer is some forty kernels of 2 to 10 us, and between two of them the device idles while
// the last blocks drain, the next grid is scheduled and its prologue runs (barriers, tensor memory,
// descriptor fetches: about 2 us for a GEMM).  A kernel launched with launch_overlapped may be
// scheduled as soon as every block of its predecessor has called allow_next_kernel() or left; it must
// call wait_previous_kernel() - which returns when the predecessor has completed and its writes are
// visible - in every thread before that thread touches global memory.  Kernels call
// allow_next_kernel() late, when a block has no more work to start: called early, the next kernel's
// blocks would sit on the SMs for the whole length of this one and keep the optimizer's kernel, which
// runs beside the products of the backward pass, out.  Both calls do nothing in a kernel launched the
// ordinary way, and a predecessor that never calls allow_next_kernel() (ATen's kernels, copies) is
// simply waited for.
#pragma once
#include <cuda_runtime.h>

namespace ft {

__device__ __forceinline__ void wait_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next_kernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cluster: blocks of a cluster along x (1: none)
template <typename... Params, typename... Args>
inline cudaError_t launch_overlapped(void (*kern)(Params...), dim3 grid, unsigned block, size_t smem, cudaStream_t s,
                                     int cluster, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

}  // namespace ft
