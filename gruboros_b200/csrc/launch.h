// Kernel launches with programmatic stream serialisation.
//
// The kernels of a pass depend on one another one by one, and for small shapes the time between two of them (grid launch,
// barrier and tensor-memory set-up, about 2 us) is as long as their work.  A kernel launched here may become resident
// while its predecessor on the stream still runs: it sets itself up, calls pdl_wait() before its first access to memory
// that an earlier kernel writes (or still reads), and lets its own successor start with pdl_trigger().  pdl_wait() returns
// when the predecessor has finished and its writes are visible; since the predecessor waited for its own, everything
// before it has finished too.  Only kernels in which every block calls pdl_wait() may be launched this way.
#pragma once
#include <cuda_runtime.h>

namespace grb {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename Kern, typename... Args>
inline int launch_pdl(Kern kern, dim3 grid, int threads, size_t smem, cudaStream_t st, int cluster, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess ? 0 : -5;
}

}  // namespace grb
