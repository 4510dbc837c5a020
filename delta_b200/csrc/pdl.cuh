// Programmatic dependent launch for the kernels of the replayed time step.
//
// A kernel launched with launch_dep(true, ...) may start while the kernel before it on
// the stream is still running (the launch attribute cudaLaunchAttributeProgrammatic-
// StreamSerialization; under stream capture it becomes a programmatic edge of the graph).
// Every such kernel calls dep_sync() as its first statement: griddepcontrol.wait returns
// once the previous kernel has completed and its memory operations are visible, so nothing
// the kernel reads or writes is touched before then; griddepcontrol.launch_dependents then
// lets the next kernel's launch begin.  What overlaps is the launch and block scheduling of
// a kernel with the end of the one before it.  Launched without the attribute (the stepped
// path), dep_sync() returns at once.
//
// CTAs of a dependent kernel that are resident early cannot hold up the kernel before it: they
// become resident only when all of that kernel's CTAs have issued launch_dependents, so each
// of them runs already.  A kernel of launch_dep waits on no other CTA of its own either; one
// whose CTAs do is one cluster (launch_dep_cluster), which the hardware starts as a whole, and
// its dependents start only when all of its CTAs have issued launch_dependents.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace delta {

__device__ __forceinline__ void dep_sync() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// kernel<<<grid, block, smem, st>>>(args...), as a programmatic dependent launch when dep.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(bool dep, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args &&...args) {
  if (!dep) {
    kernel<<<grid, block, smem, st>>>(std::forward<Args>(args)...);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// kernel as one cluster of `ctas` CTAs, a programmatic dependent launch; its CTAs may wait on
// one another.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep_cluster(void (*kernel)(KArgs...), unsigned ctas, unsigned block, cudaStream_t st,
                                      Args &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = ctas;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace delta
