// Launching a kernel so that its start overlaps the end of the kernel before it on the stream
// (programmatic dependent launch).
//
// A small layer is some forty kernels of 2 to 10 us, and between two of them the device idles while
// the last blocks drain, the next grid is scheduled and its prologue runs (barriers, tensor memory,
// descriptor fetches: about 2 us for a GEMM).  Measured, ordinary -> overlapped launches, medians of four runs
// in turn on one box: a forward block of 3 x 1000 tokens and width 1600 290 -> 271 us, a GPT-2 small of 2 x 512
// tokens, forward + backward, 5.29 -> 5.12 ms; blocks of 2048 tokens and more do not tell them apart (Llama-2-7B
// 5.01 -> 4.99, Llama-3-70B 9.90 -> 9.95 ms, runs 3 % apart).  A kernel launched with launch_overlapped may be
// scheduled as soon as every block of its predecessor has called allow_next_kernel() or left; it must
// call wait_previous_kernel() - which returns when the predecessor has completed and its writes are
// visible - in every thread before that thread touches global memory.  Its pointer arguments carry no
// __restrict__ (nor __ldg): to the compiler that means memory nobody writes while the kernel runs, and lets it
// load before the wait or through a cache that keeps what the predecessor has overwritten since.  Where that
// leaves loads behind stores or barriers, the kernels order them by hand.  Kernels call
// allow_next_kernel() late, when a block has no more work to start: called early, the next kernel's
// blocks would sit on the SMs for the whole length of this one and keep the optimizer's kernel, which
// runs beside the products of the backward pass, out.  Both calls do nothing in a kernel launched the
// ordinary way, and a predecessor that never calls allow_next_kernel() (ATen's kernels, copies) is
// simply waited for.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace ft {

__device__ __forceinline__ void wait_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next_kernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Where a kernel may start under its predecessor: only a short one, by the bytes it moves or the operations
// it does.  Two microseconds are nothing to a kernel of hundreds, and early blocks can only be in the way of the
// optimizer's kernel on the other stream.  The limits lie above everything that was seen to gain (up to 210 MB and
// 0.08 TFLOP in the two workloads above) and below the kernels of a Llama-2-13B training step of 32768 tokens (from
// 670 MB and 1.7 TFLOP), whose time does not depend on them: no launch overlapped 3552 ms, with these limits 3560,
// all overlapped 3562, medians of four runs each in turn on one box, 3547 to 3567 in all.
inline bool overlap_bytes(int64_t bytes) { return bytes <= (384LL << 20); }
inline bool overlap_product(int64_t m, int64_t n, int64_t k) { return 2.0 * m * n * k <= 1e12; }

// More than 48 KB of dynamic shared memory are granted to one kernel on one device.  One object per kernel
// (a static beside its launch) asks once for each device of the process.
class DynamicSmem {
 public:
  template <typename Kern>
  void grant(Kern kern, int bytes) {
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev < 64 ? uint64_t(1) << dev : 0;
    if (granted_.load(std::memory_order_relaxed) & bit) return;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
      granted_.fetch_or(bit, std::memory_order_relaxed);
  }

 private:
  std::atomic<uint64_t> granted_{0};
};

// cluster: blocks of a cluster along x (1: none)
template <typename... Params, typename... Args>
inline cudaError_t launch_overlapped(void (*kern)(Params...), dim3 grid, unsigned block, size_t smem, cudaStream_t s,
                                     int cluster, bool overlap, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (overlap) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

}  // namespace ft
