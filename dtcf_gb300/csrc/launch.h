// Launches whose start overlaps the end of the kernel before (programmatic
// dependent launch): the next kernel's CTAs are placed as its predecessor's
// last ones exit, and wait there for its memory, instead of being placed
// after that.  Every kernel launched so calls begin_dependent() before it
// touches memory another kernel may write: it returns when all earlier work
// of the stream is complete and visible, as at a plain kernel's start.  No
// kernel lets its successor start earlier than its own end: placed early, the
// waiting CTAs cost more than they gain.  Measured, plain / so / with the
// successor started at the kernel's own start: CCSD at o = 8, v = 24, per
// iteration of 69 kernels, in a graph 309 / 297 / 324 us, launched one by one
// 462 / 309 / 338; the CCD residual table (o = 12, v = 36) 1224 / 1126 / 1333;
// a permute of 47 x 53 x 61 x 39 after another 20.5 / 15.4 / 16.0; the split
// GEMMs alone plain / so: a plan of M = N = K = 400 at 4 slices 35.3 / 33.5.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "common.h"

namespace gbx {

#ifdef __CUDACC__
__device__ __forceinline__ void begin_dependent() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// cluster: CTAs of a cluster (1: none); smem: dynamic shared memory.
template <class... P, class... A>
cudaError_t try_launch_dependent(void (*kernel)(P...), unsigned grid, unsigned threads, cudaStream_t st,
                                 unsigned cluster, size_t smem, A&&... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(a)...);
}

template <class... P, class... A>
int launch_dependent(void (*kernel)(P...), unsigned grid, unsigned threads, cudaStream_t st, unsigned cluster,
                     size_t smem, A&&... a) {
  GBX_CUDA(try_launch_dependent(kernel, grid, threads, st, cluster, smem, std::forward<A>(a)...));
  return GBX_OK;
}

template <class... P, class... A>
int launch(void (*kernel)(P...), unsigned grid, unsigned threads, cudaStream_t st, A&&... a) {
  return launch_dependent(kernel, grid, threads, st, 1u, 0, std::forward<A>(a)...);
}
#endif

}  // namespace gbx
