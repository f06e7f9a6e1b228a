// Programmatic dependent launch: a kernel launched with `launch` may become resident while the kernel before it on the
// stream still runs, so that its set-up (barriers, tensor memory, first weight loads) is over when its inputs are there.
//
// Two rules keep the order of a stream's memory operations what it was:
//   * every thread of a kernel launched here calls `wait` before it touches memory that an earlier kernel may write or
//     read; what it touches before are model weights and its own shared memory only;
//   * a kernel calls `release` after its own `wait` and after its tensor memory is allocated, so a kernel that has started
//     early never overlaps anything but its direct predecessor, whose CTAs all hold what they need to finish.
// Kernels that never release hold back their successor until they end, as an ordinary launch does.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace xpool {
namespace pdl {

__device__ __forceinline__ void wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// For kernels whose CTAs last about a microsecond (a row's gather, norm or rotation). The GPU takes about a nanosecond for each CTA
// that releases, and the successor can become resident with a grid's last CTAs only, so a grid of more CTAs than the GPU holds leaves
// it to their ends. A gather of 512 elements a row, a CTA a row, us without release / with: 592 rows 1.28 / 1.30, 1000 rows 1.52 / 1.48,
// 2000 rows 2.04 / 2.55, 8192 rows 5.30 / 9.09. (Where CTAs last longer the nanoseconds are hidden and the early start counts:
// decode attention of 7 requests loses 0.3 us a launch without it.)
__device__ __forceinline__ void release_short() {
  if (gridDim.x * gridDim.y * gridDim.z <= 148 * 8) release();
}

// cluster > 1: CTAs of consecutive x index form clusters of that many
template <typename... K, typename... A>
inline cudaError_t launch(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace pdl
}  // namespace xpool
