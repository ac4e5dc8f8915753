// Launch of a kernel as a programmatic dependent of the one before it in the stream.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include <utility>

namespace rb {

// The kernel's CTAs may be set up while the last ones of its predecessor still run, where that one says so (griddep_launch); the kernel
// itself calls griddep_wait before it touches global memory. A CTA says so once it holds its tensor memory - a successor that took it
// first would wait for a CTA that waits for it - and where its last load has been issued.
// For kernels of one or two CTAs an SM, the copy of rows and the sum of K ranges. Other passes over memory, many small blocks, are launched the
// plain way: set up early they crowd onto the SMs that are free first, and blocks that only wait slow the ones at work (a permutation behind a sum
// of K ranges 13 -> 21 us; f32 planes of 1664 x 1216 x 349 19.3 -> 20.0 a call).
template <typename... P, typename... A>
cudaError_t launch_after(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, unsigned cluster, A&&... args) {
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3(grid, 1, 1);
  lc.blockDim = dim3(block, 1, 1);
  lc.dynamicSmemBytes = smem;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    lc.numAttrs = 2;
  }
  lc.attrs = attr;
  return cudaLaunchKernelEx(&lc, kern, std::forward<A>(args)...);
}

}  // namespace rb
