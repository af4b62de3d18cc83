// Launch helpers: kernels that may start while their predecessor in the stream is still draining
// (programmatic dependent launch), and kernels whose blocks wait on one another (cooperative launch).
#pragma once

#include <cuda_runtime.h>

#include "../common.h"

namespace bagua {
namespace kernels {

// A kernel launched with launch_overlapped() calls this before it touches memory: it returns once every
// kernel in front of it in the stream has finished and its stores are visible.  Where the launch was an
// ordinary one it returns at once.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel of the stream be scheduled as soon as this grid leaves room for it.
__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The kernel's blocks are scheduled, and run up to wait_for_predecessor(), while the kernel in front
// of it ends: about 1 us less between two short kernels.
template <typename... P, typename... A>
inline void launch_overlapped_shared(void (*kernel)(P...), dim3 grid, dim3 block, size_t shared, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = shared;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BAGUA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

template <typename... P, typename... A>
inline void launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A... args) {
  launch_overlapped_shared(kernel, grid, block, 0, s, args...);
}

// `clusters` clusters of `blocks` blocks each, which may start while the kernel in front of them ends.  More than 8 blocks need
// cudaFuncAttributeNonPortableClusterSizeAllowed.
template <typename... P, typename... A>
inline void launch_clusters(void (*kernel)(P...), int clusters, int blocks, dim3 block, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)blocks;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * blocks));
  cfg.blockDim = block;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  BAGUA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

// All blocks of the grid are resident together, or the launch fails.
template <typename... P, typename... A>
inline void launch_cooperative(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BAGUA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

inline int sm_count() {
  static int counts[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (counts[dev] == 0) {
    int n = 0;
    counts[dev] = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
  }
  return counts[dev];
}

}  // namespace kernels
}  // namespace bagua
