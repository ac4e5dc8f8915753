// Launch of a kernel as a programmatic dependent of the one before it in the stream.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include <utility>

namespace rb {

// The kernel's CTAs may be set up while the last ones of its predecessor still run, where that one says so (griddep_launch); the kernel
// itself calls griddep_wait before it touches global memory. A CTA says so once it holds its tensor memory - a successor that took it
// first would wait for a CTA that waits for it - and where its last load has been issued; the GEMM kernel not always (GemmParams::early).
// Without that word, too, such a launch follows its predecessor in a stream 1 to 2.5 us sooner than a plain one: 300^3 f32, operand pass and product,
// 15.9 -> 13.8 us a call, 137 x 384 x 1600 f32 18.4 -> 15.8, 64 images 128 -> 128, 28x28, 3x3 f32 96 -> 89.
// For kernels of one or two CTAs an SM, the operand passes and the sum of K ranges. Other passes over memory, many small blocks, are launched the
// plain way: behind kernels that do say so they crowd onto the SMs that are free first, and blocks that only wait slow the ones at work (a permutation
// behind a sum of K ranges 13 -> 21 us). The products behind operand passes and before sums do not say so.
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
