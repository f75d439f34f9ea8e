// pcg_launch.cuh -- the launch of every kernel of a translation unit.
#pragma once

#include <cuda_runtime.h>

namespace PCG_TU {

// Launches k over `grid` blocks (clusters of `cluster`). With kOverlapPrevious in
// a.overlap the launch may start while the previous launch of the stream still runs (see
// await_previous; the host's overlap_launch decides).
template <class A>
static cudaError_t launch_kernel(void (*k)(A), unsigned grid, unsigned threads, unsigned cluster, const A& a,
                                 cudaStream_t s) {
  cudaLaunchAttribute at[2] = {};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cfg.attrs = at;
  if (a.overlap & pcg::kOverlapPrevious) {
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[cfg.numAttrs].val.clusterDim.x = cluster;
    at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, a);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}
template <class A>
static cudaError_t launch_kernel(void (*k)(A), unsigned grid, const A& a, cudaStream_t s) {
  return launch_kernel(k, grid, 128u, 1u, a, s);
}

}  // namespace PCG_TU
