// gemm_tcgen05_kernel for rows of C that are copied out of the staging tile.
#include "gemm_pick.cuh"

namespace rb {
GemmKernel gemm_kernel_copied(int kind, bool a_mn, bool b_mn, int ctas) { return pick_kernel<kTailCopied>(kind, a_mn, b_mn, ctas); }
}  // namespace rb
