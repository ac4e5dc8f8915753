// gemm_tcgen05_kernel for f32 operands as two f16 planes each.
#include "gemm_pick.cuh"

namespace rb {
namespace {
template <int CTAS>
GemmKernel pick_halves(int tail) {
  return tail == kTailCopied  ? gemm_tcgen05_kernel<kKindHalves, false, false, CTAS, kTailCopied>
         : tail == kTailFused ? gemm_tcgen05_kernel<kKindHalves, false, false, CTAS, kTailFused>
                              : gemm_tcgen05_kernel<kKindHalves, false, false, CTAS, kTailNone>;
}
}  // namespace
GemmKernel gemm_kernel_halves(int ctas, int tail) { return ctas == 2 ? pick_halves<2>(tail) : pick_halves<1>(tail); }
}  // namespace rb
