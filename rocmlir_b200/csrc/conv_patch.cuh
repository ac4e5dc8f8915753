// What the two kernels for images of few channels share (conv_patch_sm100.cu, conv_window_sm100.cu): the copies of image rows into
// shared memory and the stores of finished pixels.
#pragma once
#include "epilogue.cuh"
#include "ptx.cuh"

namespace rb {

__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int gran, int bytes) {
  if (gran == 8) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  else if (gran == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shared memory by byte offset from the start of the dynamic allocation: plain loads and stores that the compiler knows to be
// in shared memory (through an aligned-up pointer they are generic ones) and may schedule freely between barriers.
extern __shared__ __align__(16) uint8_t smem_raw[];
template <typename T>
__device__ __forceinline__ T lds(uint32_t off) {
  return *reinterpret_cast<const T*>(smem_raw + off);
}

// Up to 32 output channels (from n on, `ncols` of them) of this lane's pixel, whose first element lies at `pix`: from tensor memory
// to the result, through the fused tail with EPI. All lanes of the warp call it; those without a pixel pass valid = false.
template <bool EPI, typename Params>
__device__ __forceinline__ void store_pixel(const Params& p, bool valid, long long pix, uint32_t taddr, int n, int ncols,
                                            const float* vec_scale, const float* vec_bias) {
  uint32_t v[32];
  tmem_ld32(taddr, v);
  tmem_ld_wait();
  const long long o = pix + (long long)n * p.o_k;
  if constexpr (!EPI) {
    uint32_t h[16];
    pack_row16<32>(v, h, p.is_bf16 != 0);
    if (valid) {
      uint16_t* d = static_cast<uint16_t*>(p.out) + o;
      if (p.wide && ncols == 32) {
        st_global_v8(d, h);
        st_global_v8(d + 16, h + 8);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < ncols) d[j * p.o_k] = (uint16_t)(h[j / 2] >> (16 * (j & 1)));
      }
    }
  } else {
    float x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
    EpiRow er;
    if ((p.epi.flags & RB_EPI_BIAS) && (p.epi.flags & RB_EPI_BIAS_SCALAR)) er.row_bias = load_bias(p.epi.bias, p.epi.bias_type, 0);
    er.res_stride = p.o_k;
    er.ncols = ncols;
    er.res = (valid && (p.epi.flags & RB_EPI_RESIDUAL))
                 ? static_cast<const uint8_t*>(p.epi.residual) + (p.epi.res_type == RB_F32 ? 4 : 2) * o
                 : nullptr;
    epi_apply32(x, p.epi, vec_scale, vec_bias, er);
    if (valid) {
      if (p.wide && ncols == 32) {
        uint4 w4[8];
        const int nw = pack_row32(x, p.out_type, w4, p.epi.out_zero);
        uint4* d = reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.out) + o * dtype_size(p.out_type));
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < nw) d[i] = w4[i];
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < ncols) store_elem(p.out, o + j * p.o_k, x[j], p.out_type, p.epi.out_zero);
      }
    }
  }
}

}  // namespace rb
