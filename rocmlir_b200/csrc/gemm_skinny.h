// GEMM with at most 64 rows against a weight matrix stored out x in (csrc/gemm_skinny_sm100.cu).
#pragma once
#include "../../include/rocmlir_b200.h"
#include "epilogue.cuh"

namespace rb {
// Whether the product is one of this kernel's, and faster there than on the general kernel.
bool gemm_skinny_applicable(const RbGemmProblem* p, uint32_t epi_flags);
// The operands, formats and epilogue as gemm_run has validated them; no workspace.
RbStatus gemm_skinny_run(const RbGemmProblem* p, const EpiParams& epi, const void* a, const void* b, void* c, int kind, uint32_t fmt_a,
                         uint32_t fmt_b, uint32_t cfmt, long long wait_cycles, int stall, void* stream);
}  // namespace rb
