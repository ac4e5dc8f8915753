// gemm_tcgen05_kernel for results that are converted and stored.
#include "gemm_pick.cuh"

namespace rb {
GemmKernel gemm_kernel_plain(int kind, bool a_mn, bool b_mn, int ctas) { return pick_kernel<kTailNone>(kind, a_mn, b_mn, ctas); }
}  // namespace rb
