// Launch of a kernel as a programmatic dependent of the kernel before it in the stream.
//
// The launch may begin while that kernel's last blocks still run: barriers, tensor memory and descriptors are set up and the
// first weight tiles are prefetched into L2 under its tail, and every thread then executes griddepcontrol.wait
// (dependency_wait), which returns when the kernel before it has completed and its writes are visible.  Rules for the
// kernels launched this way:
//   * before dependency_wait nothing is read or written but launch parameters; the weights are only PREFETCHED into L2,
//     which is right whoever wrote them last;
//   * what a predecessor may have written is read with ordinary loads (or TMA / cp.async) after dependency_wait, never through
//     the read-only path (__ldg, ld.global.nc, const __restrict__): that is for data nobody writes while the kernel runs, and
//     this kernel is running while its predecessor writes;
//   * dependency_trigger comes after dependency_wait, so a kernel that starts early finds everything up to the kernel two
//     before it complete: at most two kernels of a stream overlap;
//   * every block executes dependency_wait, so the completion of the kernel implies that of its predecessors.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "kernels.h"

namespace sfb200 {

// cluster = 0: as compiled (none, or __cluster_dims__).  dependent = false: the kernel starts when the one before it has completed.
template <class... P, class... A>
int launch_kernel(bool dependent, void (*kernel)(P...), dim3 grid, int block, size_t smem, int cluster, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(block), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = dependent ? 1 : 0;
  if (cluster > 0) {
    cudaLaunchAttribute& c = attr[cfg.numAttrs++];
    c.id = cudaLaunchAttributeClusterDimension;
    c.val.clusterDim.x = static_cast<unsigned>(cluster);
    c.val.clusterDim.y = 1;
    c.val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  if (cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...) != cudaSuccess) {
    cudaGetLastError();
    return kErrCuda;
  }
  return kOk;
}

template <class... P, class... A>
int launch_dependent(void (*kernel)(P...), dim3 grid, int block, size_t smem, int cluster, cudaStream_t stream, A&&... args) {
  return launch_kernel(true, kernel, grid, block, smem, cluster, stream, std::forward<A>(args)...);
}

}  // namespace sfb200
