// What the attention kernels share: tile extents, kernel parameters, element conversions.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "epilogue.cuh"
#include "lib_state.h"
#include "ptx.cuh"

namespace rb {

constexpr int kQT = 128;    // query rows per CTA
constexpr int kKT = 128;    // keys per block
constexpr float kLog2e = 1.4426950408889634f;

struct AttMaps {
  CUtensorMap q, k, v, o;
};

struct AttParams {
  int G, Sq, Sk, D, Dv;
  int trans_k;       // K stored [G][Sk][D] (K-major) instead of [G][D][Sk]
  int is_bf16;
  int causal;
  int q_tiles;
  float scale_log2;  // scale * log2(e)
  const void* bias;  // optional additive [G][Sq][Sk], element type
  const void* scale_t;  // optional multiplicative [G][Sq][Sk], element type (applied before the bias)
  const int8_t* mask;  // optional [G][Sq][Sk]: score kept where mask != 0, else mask_fill
  float mask_fill;
  long long mask_bytes;   // size of the mask
  uint32_t idesc_s, idesc_pv;
  uint32_t* status;
  const void* quant_bias;      // first-GEMM-quantised form: device pointers to one i8 and one f16 (else null)
  const void* quant_scale;
  unsigned long long* trace;   // optional [CTAs][16] cycle counters (two-tile kernel), see rbSetTraceBuffer
  int splits;        // single-tile kernel: CTAs of a cluster that divide a query tile's key blocks (1, 2, 4 or 8)
  void* o;           //   result [G][Sq][o_cols] and its row length, written directly when splits > 1
  int o_cols;
  int linear;        // GEMM+GEMM: P = S rounded to the element type (no scale, no softmax, no division by a row sum)
};

__device__ __forceinline__ float load_elem(const void* p, long long i, int is_bf16) {
  return is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i])
                 : __half2float(reinterpret_cast<const __half*>(p)[i]);
}
__device__ __forceinline__ uint32_t pack2(float a, float b, int is_bf16) {
  if (is_bf16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two query tiles per CTA, without side tensors, scale above zero (attention_prefill_sm100.cu).
constexpr int kPrefillThreads = 384;
RbStatus attention_prefill_launch(const AttMaps& maps, const AttParams& p, cudaStream_t stream);

}  // namespace rb
