// Kernels that follow one another on a stream (programmatic dependent launch).
//
// A kernel launched with launch_chained may start while the previous kernel of its stream is
// still running, so that its launch and prologue overlap that kernel's end (2 to 3 us per launch
// for a GEMM, about 1 us for a small kernel).  In return grid_wait() comes before every access that
// it makes to global memory: that returns once the previous kernel has completed and its writes are
// visible.  A thread with such accesses calls it itself, or makes them only after one that has
// called it (the GEMM kernels: the threads that load wait, all else follows from what they load).
// Every CTA of every kernel launched so waits, on all paths, which makes the order transitive.
// grid_launch_next() lets the next kernel of the stream start, as far as it was launched so, once
// every CTA has called it; in a kernel launched in the ordinary way both cost nothing.
#pragma once
#include <cuda_runtime.h>

namespace psdev {

__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_launch_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches `k`; clusters of `cluster` CTAs along x.
template <typename... P, typename... A>
inline int launch_chained(void (*k)(P...), unsigned grid, unsigned block, size_t smem,
                          cudaStream_t s, int cluster, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

}  // namespace psdev
