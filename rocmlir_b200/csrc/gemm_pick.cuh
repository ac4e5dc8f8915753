// The instantiations of gemm_tcgen05_kernel: those of one tail (GemmTail) in a source file of their own, so that they compile side by side
// and without the host code.
#pragma once
#include "gemm_sm100.cuh"

namespace rb {

typedef void (*GemmKernel)(const GemmTensorMaps, const GemmParams);

GemmKernel gemm_kernel_plain(int kind, bool a_mn, bool b_mn, int ctas);    // gemm_plain_sm100.cu
GemmKernel gemm_kernel_fused(int kind, bool a_mn, bool b_mn, int ctas);    // gemm_fused_sm100.cu
GemmKernel gemm_kernel_copied(int kind, bool a_mn, bool b_mn, int ctas);   // gemm_copied_sm100.cu
GemmKernel gemm_kernel_halves(int ctas, int tail);                          // gemm_halves_sm100.cu

template <int KIND, int CTAS, int TAIL>
GemmKernel pick_major(bool a_mn, bool b_mn) {
  if (!a_mn && !b_mn) return gemm_tcgen05_kernel<KIND, false, false, CTAS, TAIL>;
  if (!a_mn && b_mn) return gemm_tcgen05_kernel<KIND, false, true, CTAS, TAIL>;
  if (a_mn && !b_mn) return gemm_tcgen05_kernel<KIND, true, false, CTAS, TAIL>;
  return gemm_tcgen05_kernel<KIND, true, true, CTAS, TAIL>;
}
template <int CTAS, int TAIL>
GemmKernel pick_kind(int kind, bool a_mn, bool b_mn) {
  switch (kind) {
    case kKindF16: return pick_major<kKindF16, CTAS, TAIL>(a_mn, b_mn);
    case kKindTF32: return gemm_tcgen05_kernel<kKindTF32, false, false, CTAS, TAIL>;  // f32 operands are made K-major first
    case kKindI8: return pick_major<kKindI8, CTAS, TAIL>(a_mn, b_mn);
    default: return pick_major<kKindF8, CTAS, TAIL>(a_mn, b_mn);
  }
}
template <int TAIL>
GemmKernel pick_kernel(int kind, bool a_mn, bool b_mn, int ctas) {
  return ctas == 2 ? pick_kind<2, TAIL>(kind, a_mn, b_mn) : pick_kind<1, TAIL>(kind, a_mn, b_mn);
}

}  // namespace rb
