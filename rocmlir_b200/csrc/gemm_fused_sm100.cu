// gemm_tcgen05_kernel for fused elementwise tails.
#include "gemm_pick.cuh"

namespace rb {
GemmKernel gemm_kernel_fused(int kind, bool a_mn, bool b_mn, int ctas) { return pick_kernel<kTailFused>(kind, a_mn, b_mn, ctas); }
}  // namespace rb
