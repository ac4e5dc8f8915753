// Host side of rbGemm: validates a rock.gemm problem, prepares operands that TMA cannot address
// directly (row pitch not a multiple of 16 bytes -> padded copy in the caller's workspace; f32 ->
// TF32 hi/lo split), encodes the tensor maps and launches the persistent tcgen05 kernel.
#include "gemm_pick.cuh"

#include <atomic>
#include <cstdio>
#include <mutex>

#include "gemm_skinny.h"
#include "launch.cuh"
#include "lib_state.h"

namespace rb {
namespace {

thread_local int t_variant = 0;
thread_local long long t_wait_cycles = kWaitCycles;   // rbSetWaitLimit
thread_local int t_stall_launches = 0;                // rbInjectStall: GEMM launches left to stall
// Chained pair (rbGemmGemm with equal inner extents): the G = 2 problem handed to gemm_run has group 0 = (a, b, c) and
// group 1 = (c of group 0, b2, c2); gemm_run builds tensor maps whose group stride is the distance between the two
// tensors and lets the kernel order the groups through flags (GemmParams::chain_flags).
struct GemmChain {
  const void* b2;
  void* c2;
  unsigned int* flags;
  size_t flags_bytes;
};
thread_local const GemmChain* t_chain = nullptr;

// ---- auxiliary kernels ---------------------------------------------------------------------------
// Operands whose rows do not start on 16-byte boundaries are copied into rows that do (both of a product in one launch):
// rows of row_bytes bytes become rows of pitch_bytes bytes, the rest of a row zero.
struct PadJob {
  const uint8_t* src;
  uint8_t* dst;
  unsigned long long rows;
  unsigned row_bytes, pitch_bytes;
};
struct PadJobs {
  PadJob job[2];
  unsigned long long first[3];   // vectors of 16 bytes before each job
};

// Bytes [at, at + 16) of the source row that starts at `row` (any alignment), zeros from byte `n` on: the aligned 32-bit
// words around them, shifted into place. A word is read whole only where all of it lies inside [row, row + n).
__device__ __forceinline__ uint4 load_row16(const uint8_t* row, unsigned at, unsigned n) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(row) + at;
  const unsigned shift = (unsigned)(a & 3) * 8;
  const unsigned lead = (unsigned)(a & 3);
  uint32_t w[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const long long o = (long long)at - lead + 4 * i;   // offset of the word inside the row
    w[i] = 0u;
    if (o >= 0 && o + 4 <= (long long)n) {
      w[i] = __ldg(reinterpret_cast<const uint32_t*>(row + o));
    } else if (o + 4 > 0 && o < (long long)n && (i < 4 || lead)) {
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (o + b >= 0 && o + b < (long long)n) w[i] |= (uint32_t)__ldg(row + o + b) << (8 * b);
    }
  }
  return make_uint4(__funnelshift_r(w[0], w[1], shift), __funnelshift_r(w[1], w[2], shift), __funnelshift_r(w[2], w[3], shift),
                    __funnelshift_r(w[3], w[4], shift));
}

// One 16-byte vector of the destination per thread and step: bound by the one read and one write of the operand, and at these
// sizes by the launch. 3 x 1024 x 769 f16 (4.7 MB): 4.4 us; with one byte and one 64-bit division per thread the whole call of
// the 3 x 1024 x 1024 x 769 product took 28.7 us, now 16.4.
__global__ void pad_rows_kernel(const PadJobs p) {
  griddep_launch();   // the product is set up meanwhile
  griddep_wait();
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < p.first[2];
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const bool second = i >= p.first[1];
    const PadJob j = second ? p.job[1] : p.job[0];
    const unsigned long long v = i - (second ? p.first[1] : 0ull);
    const unsigned per_row = j.pitch_bytes / 16;
    const unsigned long long r = (v >> 32) ? v / per_row : (unsigned)v / per_row;
    const unsigned at = (unsigned)(v - r * per_row) * 16;
    *reinterpret_cast<uint4*>(j.dst + v * 16) = load_row16(j.src + r * j.row_bytes, at, j.row_bytes);
  }
}

// f32 operands are re-laid into K-major planes in the workspace before the TF32 MMA: an MN-major
// operand is transposed (the 32-bit MN-major shared-memory layout needs a different swizzle mode, so
// the kernel keeps a single K-major path for TF32), rows are pitched to a multiple of 16 bytes, and with
// SPLIT the value is separated into x = hi + lo (+ O(2^-22 |x|)) with hi and lo both exactly
// representable in TF32 (low 13 mantissa bits zero), so that hi*hi + hi*lo + lo*hi carries fp32-class
// accuracy whatever the tensor core does with the low bits.
//   src: [G][R][C] row-major.  TRANSPOSE = false: out [G][R][pitch] (pitch >= C)
//                              TRANSPOSE = true : out [G][C][pitch] (pitch >= R)
__device__ __forceinline__ float tf32_round(float x) {
  const uint32_t xb = __float_as_uint(x);
  if ((xb & 0x7F800000u) == 0x7F800000u) return x;  // inf / nan
  return __uint_as_float((xb + 0x1000u) & 0xFFFFE000u);
}
// Up to two operands per launch, dealt out in 64 x 64 tiles. Bound by one read and `planes` writes of the operand, so both
// sides move 16 bytes per thread (the read element by element where the rows of the source do not allow it). Two operands of
// 4096 x 4096: 61 us, 6.6 TB/s.
template <typename T>
struct PlaneJob {
  const float* src;
  T* hi;
  T* lo;                  // nullptr (f32 planes only): one plane, the value itself
  int R, C, pitch;        // src [G][R][C]; out [G][R][pitch], or with transpose [G][C][pitch]
  int transpose;
  int tiles_x, tiles_y;   // tiles of the output-padded extent along C and R
};
// The tiles of both jobs, a block per tile: seen() gets a thread's sixteen values as they lie, store() four neighbours along K of one row of the
// planes at offset o, after() the tile's place when it is done.
template <typename T, typename Seen, typename Store, typename After>
__device__ __forceinline__ void plane_tiles(const PlaneJob<T>* jobs, const long long* first, Seen&& seen, Store&& store, After&& after) {
  __shared__ float tile[64][65];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 vectors of four x 16 rows
  for (long long t = blockIdx.x; t < first[2]; t += gridDim.x) {
    const bool second = t >= first[1];
    const PlaneJob<T> j = second ? jobs[1] : jobs[0];
    const long long lt = t - (second ? first[1] : 0), per_g = (long long)j.tiles_x * j.tiles_y;
    const long long g = lt / per_g;
    const int rem = (int)(lt - g * per_g);
    const int c0 = (rem % j.tiles_x) * 64, r0 = (rem / j.tiles_x) * 64;
    const float* s = j.src + g * (long long)j.R * j.C;
    const bool vec = j.C % 4 == 0 && (reinterpret_cast<uintptr_t>(j.src) & 15) == 0;
    float x[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // all four reads in flight
      const int r = r0 + ty + 16 * i, c = c0 + tx * 4;
      const float* q = s + (long long)r * j.C + c;
      if (vec && r < j.R && c < j.C) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(q));
        x[i][0] = v.x; x[i][1] = v.y; x[i][2] = v.z; x[i][3] = v.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[i][e] = (r < j.R && c + e < j.C) ? __ldg(q + e) : 0.0f;
      }
    }
    seen(second, x);
    if (!j.transpose) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + ty + 16 * i, c = c0 + tx * 4;
        if (r < j.R && c < j.pitch) store(j, (g * j.R + r) * (long long)j.pitch + c, x[i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) tile[ty + 16 * i][tx * 4 + e] = x[i][e];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int oc = c0 + ty + 16 * i, orr = r0 + tx * 4;   // output row = source column, output column = source row
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = tile[tx * 4 + e][ty + 16 * i];
        if (oc < j.C && orr < j.pitch) store(j, (g * j.C + oc) * (long long)j.pitch + orr, y);
      }
      __syncthreads();
    }
    after(j, s, r0 + ty, c0 + tx * 4);
  }
}
// The grid covers the padded extent of whichever dimension becomes the output row (zeros past the source's extent).
template <typename T>
PlaneJob<T> plane_job(const float* src, T* hi, T* lo, int R, int C, int pitch, bool transpose) {
  PlaneJob<T> j;
  j.src = src; j.hi = hi; j.lo = lo; j.R = R; j.C = C; j.pitch = pitch; j.transpose = transpose ? 1 : 0;
  j.tiles_x = ((transpose ? C : pitch) + 63) / 64;
  j.tiles_y = ((transpose ? pitch : R) + 63) / 64;
  return j;
}
typedef PlaneJob<float> F32Job;
struct F32Jobs {
  F32Job job[2];
  long long first[3];     // tiles before each job
};
__device__ __forceinline__ void store_planes4(const F32Job& j, long long o, const float* x) {
  if (j.lo) {
    float h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      h[e] = tf32_round(x[e]);
      l[e] = isfinite(h[e]) ? tf32_round(x[e] - h[e]) : 0.0f;
    }
    *reinterpret_cast<float4*>(j.hi + o) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(j.lo + o) = make_float4(l[0], l[1], l[2], l[3]);
  } else {
    *reinterpret_cast<float4*>(j.hi + o) = make_float4(x[0], x[1], x[2], x[3]);
  }
}
__global__ void __launch_bounds__(256) f32_prepare_kernel(const F32Jobs p, const unsigned int* gate) {
  griddep_launch();   // the product is set up meanwhile
  griddep_wait();
  if (gate && *reinterpret_cast<const volatile unsigned int*>(gate) == 0u) return;   // f16 planes will do
  plane_tiles(p.job, p.first, [](bool, const float (*)[4]) {}, [](const F32Job& j, long long o, const float* x) { store_planes4(j, o, x); },
              [](const F32Job&, const float*, int, int) {});
}
RbStatus launch_f32_jobs(F32Jobs& jobs, int count, long long groups, int sms, cudaStream_t stream, const unsigned int* gate = nullptr) {
  jobs.first[0] = 0;
  for (int i = 0; i < 2; ++i)
    jobs.first[i + 1] = jobs.first[i] + (i < count ? groups * (long long)jobs.job[i].tiles_x * jobs.job[i].tiles_y : 0);
  const unsigned grid = (unsigned)std::min<long long>(jobs.first[2], (long long)sms * (gate ? 8 : 32));   // (one wave of blocks that may have to end at once)
  RB_CUDA_TRY(launch_after(f32_prepare_kernel, grid, 256, 0, stream, 1, jobs, gate));
  count_launch();
  return RB_SUCCESS;
}

// ---- f32 operands as f16 planes (see kMaxPlanes) -----------------------------------------------------------------------------
// Scales of the two operands, from 512 runs of 32 elements of each: a power of two that brings the largest to 2^13 (1 where all are zero), and the flag,
// which stands when no such scales exist. One block, a warp per run, the loads in flight together: single elements, 16384 lines of each operand, took 20
// us from L2 and 117 from memory.
// Values of |y| < kHalfFull, y = scale * x, have fewer bits in f16 planes (steps of 2^-36) than in TF32 ones: kHalfLeast has 18 of 22.
constexpr float kHalfFull = 1.0f / 16384, kHalfLeast = kHalfFull / 16;
struct HalvesState {
  float scale[2], out_scale;
  unsigned int flag;        // not zero: an operand does not fit, TF32 planes it is
};
struct HalvesSample {
  const float* src[2];
  long long n[2];
  HalvesState* state;
};
__global__ void __launch_bounds__(1024) halves_scale_kernel(const HalvesSample p) {
  __shared__ float top[2][32];
  __shared__ int low_runs;
  griddep_launch();
  griddep_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float v[2][16];
  if (threadIdx.x == 0) low_runs = 0;
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    // an odd number of runs apart, so that rows of any length are met in all their columns (small operands: the runs overlap)
    const long long runs = p.n[o] / 512 / 32, step = runs > 1 ? ((runs - 1) | 1) * 32 : p.n[o] / 512;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const long long at = (i * 32 + warp) * step + lane;
      v[o][i] = at < p.n[o] ? fabsf(__ldg(p.src[o] + at)) : 0.0f;
    }
  }
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, v[o][i]);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if (lane == 0) top[o][warp] = m;
  }
  __syncthreads();
  int e[2];
  bool fits = true;
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    float m = top[o][lane];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    const int x = (int)(__float_as_uint(m) >> 23);   // the biased exponent: 0 for zeros and subnormal numbers, 255 for infinities
    fits = fits && x < 255;
    e[o] = x == 0 ? 0 : 140 - x;                     // 2^e * m lies in [2^13, 2^14)
    fits = fits && e[o] <= 126 && e[o] >= -126;
    // values that will not fit, seen here already: two in a run, or one below the least
    const float scale = e[o] <= 126 && e[o] >= -126 ? __uint_as_float((uint32_t)(127 + e[o]) << 23) : 1.0f;
    float least = kHalfFull;
#pragma unroll
    for (int i = 0; i < 16; ++i) least = fminf(least, v[o][i] != 0.0f ? v[o][i] * scale : kHalfFull);
    bool low = false;
    if (__any_sync(0xffffffffu, least < kHalfFull)) {
      low = __any_sync(0xffffffffu, least < kHalfLeast);
#pragma unroll
      for (int i = 0; i < 16; ++i) low = low || __popc(__ballot_sync(0xffffffffu, v[o][i] != 0.0f && v[o][i] * scale < kHalfFull)) > 1;
    }
    if (low && lane == 0) low_runs = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int sum = -(e[0] + e[1]);
    fits = fits && sum <= 126 && sum >= -126;
    p.state->scale[0] = fits ? __uint_as_float((uint32_t)(127 + e[0]) << 23) : 1.0f;
    p.state->scale[1] = fits ? __uint_as_float((uint32_t)(127 + e[1]) << 23) : 1.0f;
    p.state->out_scale = fits ? __uint_as_float((uint32_t)(127 + sum) << 23) : 1.0f;
    p.state->flag = fits && low_runs == 0 ? 0u : 1u;
  }
}
// The planes: hi = f16(y), lo = f16((y - hi) * kLoFactor) of y = scale * x, K-major like the TF32 ones. |y| >= 65504 does not fit. From kHalfFull up
// they are off by 2^-23 of y at most, as TF32 planes are (2^-22 where the residual is half a step of the largest numbers). Nothing is lost to a value below, wherever it stands, because it raises the flag: what
// selects it in the other operand - a diagonal, a few rows that are not zero - is not known here. The one exception keeps ordinary data on this form, where
// one value in 3e7 is that small (normal ones; 4096 x 4096 of them have such a value in 4 cases of 10): one value of kHalfLeast or more in all
// tiles of a block, among three others at least that are not zero in its 64 of a row and in its 64 of a column. Zeros are exact and count for nothing.
// Bound by one read and one write of the operand. 4096^3, both operands: TF32 planes 62 us, these 46, with the sample 53.
typedef PlaneJob<__half> HalvesJob;   // pitch: a multiple of eight
struct HalvesJobs {
  HalvesJob job[2];
  long long first[3];
  HalvesState* state;
};
// Whether the values below kHalfFull among a thread's sixteen (rows r, r + 16, ..., columns c ... c + 3 of a source of R x C) may stay in f16
// planes (see above); lows counts those of the block.
__device__ __noinline__ bool low_values_fit(const float* s, int R, int C, int r, int c, float scale, int* lows) {
  bool fit = true;
#pragma unroll 1
  for (int e = 0; e < 16 && fit; ++e) {
    const int rr = r + 16 * (e >> 2), cc = c + (e & 3);
    if (rr >= R || cc >= C) continue;
    const float v = s[(long long)rr * C + cc], y = fabsf(v * scale);
    if (v == 0.0f || y >= kHalfFull) continue;
    fit = y >= kHalfLeast && atomicAdd(lows, 1) == 0;
    if (!fit) break;
    int in_row = 0, in_col = 0;
#pragma unroll 1
    for (int i = 0; i < 64; ++i) {
      const int ri = (rr & ~63) + i, ci = (cc & ~63) + i;
      in_row += ci < C && s[(long long)rr * C + ci] != 0.0f ? 1 : 0;
      in_col += ri < R && s[(long long)ri * C + cc] != 0.0f ? 1 : 0;
    }
    fit = in_row >= 4 && in_col >= 4;
  }
  return fit;
}
__global__ void __launch_bounds__(256, 5) f32_halves_kernel(const HalvesJobs p) {
  __shared__ int lows;      // values below kHalfFull
  griddep_launch();
  griddep_wait();
  if (threadIdx.x == 0) lows = 0;
  // other blocks may raise the flag at any time: one thread reads it for the block
  if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<const volatile unsigned int*>(&p.state->flag) != 0u)) return;
  bool bad = false, low = false;
  float scale = 1.0f;
  plane_tiles(
      p.job, p.first,
      [&](bool second, const float (*x)[4]) {
        scale = p.state->scale[second ? 1 : 0];
        low = false;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float v = x[i >> 2][i & 3], y = fabsf(v * scale);
          bad = bad || !(y < 65504.0f);
          low = low || (y < kHalfFull && v != 0.0f);
        }
      },
      [&](const HalvesJob& j, long long o, const float* x) {
        __half h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float y = x[e] * scale;
          h[e] = __float2half_rn(y);
          // (a residual of 16, half a step of the largest numbers, would round up to infinity)
          l[e] = __float2half_rn(fminf(fmaxf((y - __half2float(h[e])) * kLoFactor, -65504.0f), 65504.0f));
        }
        *reinterpret_cast<uint2*>(j.hi + o) = *reinterpret_cast<const uint2*>(h);
        *reinterpret_cast<uint2*>(j.lo + o) = *reinterpret_cast<const uint2*>(l);
      },
      [&](const HalvesJob& j, const float* s, int r, int c) {
        if (low && !bad) bad = !low_values_fit(s, j.R, j.C, r, c, scale, &lows);
      });
  if (__syncthreads_or(bad ? 1 : 0) && threadIdx.x == 0) p.state->flag = 1u;
}

// Zeros for a C that both K ranges of an f32 product are added to; a kernel and not a memset, which does not start before its predecessor has
// ended nor let its successor be set up. us a call, planes and their sum / memset / this: 512 x 576 x 640 24.7 / 26.7 / 22.6, 1536 x 1536 x 4096
// 110.9 / 109.6 / 103.8, 2048 x 1024 x 2304 71.6 / 70.2 / 63.6, 4096 x 4096 x 2304 406 / 376 / 380.
__global__ void zero_kernel(float4* c, long long n4) {
  griddep_launch();
  griddep_wait();   // what runs before may read C (an operand in the same memory)
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) c[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// ---- tile configuration -----------------------------------------------------------------------
// The measured tile-shape table of this library, in the role of rocMLIR's perf_config heuristics
// (mlir/lib/Dialect/Rock/Tuning/GridwiseGemmParams.cpp:384-417): tile width from N, CTA pairs whenever
// the operand layout allows them, the deepest ring that fits, and a K split when the output has too few
// tiles to fill the GPU (the role of split-K in mlir/lib/Dialect/Rock/Transforms/GemmToGridwise.cpp:268-394,
// here with f32 partial planes and a fixed-order reduction instead of atomics).
// Planning uses the SM count of the current device when one is present (148 on a B200) and 148 otherwise, so that
// the configuration queries answer the same on a build machine without a GPU.
int planned_sms() { return planning_sm_count(); }

struct GemmConfig {
  int ctas, bn, stages, splits;
  int kpr;                 // K blocks per barrier round (see GemmParams::kpr)
  bool plain_stores;
  int dp_tiles, sk_tiles;  // stream-K tail (see GemmParams); sk_tiles == 0: every tile is computed whole
};

// TF32 planes per operand (see kMaxPlanes)
int gemm_planes(const RbGemmProblem* p) { return p->ab_type == RB_F32 && p->f32_mode == 0 ? 2 : 1; }

// Products that gain from f16 planes: two more passes and the launches of a form that is not taken, 8 to 10 us, against half of the tensor core's
// time - and of the im2col loads of a convolution, where filters of several taps gain from a quarter of the size on. us, f16 and TF32 planes:
// 1536^3 46 and 43, 2048 x 2048 x 1024 44 and 46, 1800^3 61 and 74, 2500^3 124 and 173; 3x3, 128 -> 128, 28x28, 10 images 40 and 43, 24 images 47
// and 58, 64 images 88 and 125; pointwise 128 -> 256, 28x28, 64 images 63 and 60. Explicit variants keep the TF32 form.
bool halves_pay(const RbGemmProblem* p, bool conv) {
  return p->ab_type == RB_F32 && p->f32_mode == 0 && 2.0 * p->g * p->m * (double)p->n * p->k >= (conv && p->k >= 512 ? 2e9 : 8e9);
}

// Tile and K split of a plain product by an estimate of its time, where nobody has asked for one. A launch costs `fixed`; a CTA (or
// pair) then walks its tiles, K block by K block: at least `block` (operand fetch and issue of its MMAs), and no faster than all
// CTAs together draw operands through the L2 -> SM fabric; a tile shorter than the store of the tile before it waits for that; the
// last store is exposed. A K split adds the planes and the pass that sums them. Constants in microseconds, fitted to every tile of 1600 products (f16,
// bf16, fp8, i8; up to three waves of the rule's tiles, with and without K ranges; replayed graphs; 7 % off on average, on others too), for f32 to six
// products, operand passes included. The rule before - 256 columns in pairs whatever the size, a K split as soon as half of the pairs idle - lost most
// where a product is a wave of tiles or less, us before and by the estimate: 1024^3 f16 15.0 / 8.9 (64 columns, no split), 1536^3 bf16 22.5 / 12.7,
// 2048 x 1024 x 2048 f16 21.7 / 14.5, 364 x 1344 x 1792 i8 15.2 / 9.7. Beyond three waves of its tiles the rule stays, such products being bound by memory
// or by power. Of 2831 products, 700 of them new to the fit, 15 are more than 2 % slower than by the rule (1536 x 448 x 4736 f16 18.1 -> 19.2 the most),
// of 600 more two, and the mean is 0.86 of its time, 1.005 of the fastest tile's. An estimate that took the store of every tile for the exposed one had to be beaten by
// 15 % and made 34 slower, narrow tiles in many waves above all (3 x 180 x 7720 x 213 bf16 18.0 -> 20.9, 896 x 6016 x 1024 i8 20.4 -> 22.1).
// The chained pair of rbGemmGemm goes by the same estimate: 12 sizes from 128 x 256 x 256 to 2048 x 2048 x 2048, f16 and bf16, take 0.71 to 1.02 of the
// rule's time.
struct TileCost {
  int ctas, bn;
  double fixed, block, kb_per_block;   // kb_per_block: KB a CTA fetches per K block
};
struct StoreCost {
  double last, tile, column, ragged, margin;   // a column of the exposed store; a tile and a column of the others; rows off 16 bytes; what an estimate must beat
  double ragged_tile;                          // rows off 16 bytes in the others
};
constexpr TileCost kTileCosts[] = {{1, 64, 4.75, 0.239, 24}, {1, 128, 4.35, 0.311, 32}, {2, 128, 5.68, 0.233, 24}, {1, 256, 3.50, 0.446, 48}, {2, 256, 4.91, 0.324, 32}};
constexpr StoreCost kStoreCost = {0.0087, 0.84, 0.0084, 2.58, 0.97, 2.58};
// f32 with two TF32 planes: fitted to 131000 tiles and K ranges of 18000 products of 12 to 4096 rows and columns, K of 64 to 8192, alone and in groups
// of three, 5 % off on average (the pass over the operands, the same for all of them, left out here). Of 959
// products new to the fit one is more than 5 % slower than by the estimate before (fitted to six products, no K ranges) and 23 more than 2 %, the mean is 0.95:
// 64 x 246 x 2019 29.8 -> 17.2 us, 128 x 1739 x 620 35.4 -> 21.1, 3 x 64 x 650 x 595 33.3 -> 19.4; 27 x 192 x 64 7.9 -> 8.1.
// Fitted apart, from 35 products of several waves: rows off 16 bytes cost a tile that is not the last twice an aligned one's store, where the common
// factor of 11.9, that of the exposed store, chose 256 columns for 704 x 3098 x 128 (17.0 -> 21.6 us) and 64 for 2304 x 2157 x 384 (37.7 -> 48.6); and beyond three
// waves tiles of 64 columns are 4 to 13 % slower than estimated.
constexpr TileCost kTileCostsF32[] = {{1, 64, 7.47, 0.518, 48}, {1, 128, 7.37, 0.608, 64}, {2, 128, 8.24, 0.526, 48}, {1, 256, 7.60, 1.069, 96}, {2, 256, 8.65, 0.818, 64}};
constexpr StoreCost kStoreCostF32 = {0.0031, 0.58, 0.037, 11.9, 0.97, 2.0};

// *ctas and *bn come in as the rule gives them and stay unless another tile, or fewer K ranges, is estimated faster by the margin. K is not cut where
// the rule does not cut it: such a product needs no planes in its workspace and can be handed out as one kernel. An f32 result keeps
// accumulation chains no longer than the rule's: the tensor core truncates what it adds, and of two chains in place of one the error of f16 and
// fp8 products against 64 bits is half (1.2e-6 -> 0.6e-6 at K = 1024; values of one sign 6.1e-6 -> 2.8e-6). In a 16-bit result its rounding hides that
// (2.067e-4 both ways). whole: only all of K at once, whatever the result, where that is no slower than the rule (see choose_one_kernel).
// f32 operands: where the rule cuts K (for speed, or to keep chains to 2048 elements), as many ranges as any tile gains by, down to eight blocks each;
// with whole, and for what f16 planes may take over, the rule.
void estimate_tile(const RbGemmProblem* p, bool b_mn, int che, long long kblocks, int sms, bool whole, int* ctas, int* bn, int* splits) {
  const bool f32 = p->ab_type == RB_F32;
  const int need = f32 ? (int)((p->k + 2047LL) / 2048) : 1;   // (see choose_config)
  const TileCost* const costs = f32 ? kTileCostsF32 : kTileCosts;
  const StoreCost& sc = f32 ? kStoreCostF32 : kStoreCost;
  const int es_c = (int)dtype_bytes(p->c_type);
  // an 8-bit result is requantised, 4-byte ones (and planes) are two staged rows for one; rows off 16 bytes are copied out by the warps
  const double words = f32 ? 1.0 : 1.45;
  const bool off16 = (long long)p->n * es_c % 16 != 0;
  const double width = (p->c_type == RB_I8 ? 2.76 : es_c == 4 ? words : 1.0) * (off16 ? sc.ragged : 1.0);
  // *s comes in as the ranges wanted, 0 for the rule's
  auto estimate = [&](const TileCost& t, long long* s, long long* waves) {
    const long long tiles = (long long)p->g * ((p->m + kBM * t.ctas - 1) / (kBM * t.ctas)) * ((p->n + t.bn - 1) / t.bn);
    const long long units = sms / t.ctas;
    if (*s == 0) *s = tiles * 2 <= units && kblocks >= 16 ? std::max<long long>(1, std::min<long long>(std::min(units / tiles, kblocks / 8), 128)) : 1;
    *s = std::min<long long>(std::max<long long>(*s, need), kblocks);
    const long long items = tiles * *s, kb = (kblocks + *s - 1) / *s;
    *waves = (items + units - 1) / units;
    const double busy = (double)std::min(items, units) * t.ctas;
    const double block = std::max(t.block, busy * t.kb_per_block / 12500.0);
    // (a byte per element in 64 columns: half of a staged row, copied out by the warps)
    const double columns = (f32 ? std::min(t.bn, (int)p->n) : t.bn) * (*s > 1 ? words : t.bn == 64 && es_c == 1 ? 1.52 * width : width);
    const double others = off16 && *s == 1 ? columns / sc.ragged * sc.ragged_tile : columns;
    double us = t.fixed + std::max(kb * block, sc.tile + sc.column * others) * (double)(*waves - 1) + kb * block + sc.last * columns;
    const double plane_mb = (double)p->g * p->m * p->n * 4 / 1e6;
    if (f32 && *s > 1) us += *s == 2 && p->n % 4 == 0 ? 0.88 + plane_mb * 0.368 : 1.51 + (double)*s * plane_mb * 0.298;   // (two: see add_ranges)
    if (!f32 && *s > 1) us += 2.13 + (double)*s * plane_mb * 0.265;
    return us;
  };
  const int rule_ctas = *ctas, rule_bn = *bn;
  double best = 0;
  long long s = 0, waves = 1;
  for (int i = 0; i < 5; ++i) {
    const TileCost& t = costs[i];
    if (t.ctas == rule_ctas && t.bn == rule_bn) best = (whole ? 1.0 : sc.margin) * estimate(t, &s, &waves);
  }
  if (best == 0 || waves > 3 || (f32 && s > 1 && (whole || halves_pay(p, false)))) return;   // (s and waves are those of the rule's tile)
  const long long rule_splits = whole ? 1 : s;
  const long long chain = p->c_type == RB_F32 && p->ab_type != RB_I8 && !whole ? (kblocks + s - 1) / s : kblocks;   // longest accumulation chain allowed
  for (int i = 0; i < 5; ++i) {
    const TileCost& t = costs[i];
    if ((b_mn && (t.bn / t.ctas) % che != 0) || (f32 && t.bn > 64 && t.bn >= 2 * p->n)) continue;
    if (t.ctas == 2 && (p->m <= kBM || kblocks <= 2)) continue;   // (see choose_config)
    const long long tiles = (long long)p->g * ((p->m + kBM * t.ctas - 1) / (kBM * t.ctas)) * ((p->n + t.bn - 1) / t.bn);
    const long long most = f32 && rule_splits > 1 ? std::max<long long>(rule_splits, std::min<long long>(std::min(sms / t.ctas / tiles, kblocks / 8), 128)) : 1;
    for (long long want = f32 ? rule_splits : 1; want <= (f32 || rule_splits == 1 ? most : 2); ++want) {   // (f32: fewer than the rule's have longer chains)
      s = f32 || want == 1 ? want : 0;
      double us = estimate(t, &s, &waves);
      if (s > 1 && !f32) us *= 1.08;   // (K ranges other than the rule's are the less certain ones)
      if (f32 && t.bn == 64 && waves > 3) continue;   // (see kStoreCostF32)
      if (us < best && (kblocks + s - 1) / s <= chain) { best = us; *ctas = t.ctas; *bn = t.bn; *splits = (int)s; }
    }
  }
}

GemmConfig choose_config(const RbGemmProblem* p, int variant, bool epi_vec = false, bool implicit = false, bool whole = false) {
  GemmConfig c;
  const int asked = variant;
  if (variant == 0) variant = (int)tuned_variant_gemm(p);   // the measured table, when it knows the problem
  const int es = (int)dtype_bytes(p->ab_type);
  const bool b_mn = p->ab_type != RB_F32 && p->trans_b == 0;
  const int che = kRowBytes / es;
  const int bn_code = (variant >> 12) & 0xF;
  c.bn = bn_code == 1 ? 64 : bn_code == 2 ? 128 : bn_code == 3 ? 256 : (p->n <= 64 ? 64 : p->n <= 128 ? 128 : 256);
  const int planes = gemm_planes(p);
  // Two TF32 planes of 256 columns fill tensor memory with one buffer, so a tile's epilogue is exposed; with a short K that is
  // most of the tile, and where there are more tiles than CTA pairs 128 columns with two buffers win (us, f32): 4096 x 4096 x 128
  // 40.3 -> 36.9, x 256 56.3 -> 49.2, 2048 x 8192 x 64 30.9 -> 27.4. At K = 1024 148 against 155, and with one wave 8192 x 512 x 256
  // 20.5 against 22.0.
  if (bn_code == 0 && c.bn == 256 && planes == 2 && p->k <= 256 &&
      (long long)p->g * ((p->m + 2 * kBM - 1) / (2 * kBM)) * ((p->n + 255) / 256) > planned_sms() / 2)
    c.bn = 128;
  if (b_mn && c.bn < che) c.bn = che;                       // an MN-major B tile is loaded in whole 128-byte chunks
  c.ctas = ((variant & 0xF) == 1) ? 1 : 2;
  if (b_mn && (c.bn / 2) % che != 0) c.ctas = 1;
  if (p->m <= kBM && (variant & 0xF) != 2) c.ctas = 1;      // a pair would compute 128 empty rows
  {
    // a main loop of one or two K blocks leaves the epilogue exposed, and the epilogue of a pair is the slower one
    // (measured at K = 64, 256 columns: 134 us paired, 86 us unpaired, the HBM floor being 79 us)
    const long long kb = (p->k + kRowBytes / es - 1) / (kRowBytes / es);
    if (kb <= 2 && (variant & 0xF) != 2) c.ctas = 1;
  }
  if (c.bn == 64 && (variant & 0xF) != 2) c.ctas = 1;        // measured: 64-column tiles run faster unpaired (345 vs 324 TFLOP/s)
  int est_splits = 0;
  if (variant == 0 && !implicit && (p->ab_type != RB_F32 || planes == 2))
    estimate_tile(p, b_mn, che, (p->k + kRowBytes / es - 1) / (kRowBytes / es), planned_sms(), whole, &c.ctas, &c.bn, &est_splits);
  c.stages = (variant >> 4) & 0xF;
  const int max_stages = c.ctas == 2 ? GemmSmemLayout<2>::max_stages(c.bn, epi_vec, planes) : GemmSmemLayout<1>::max_stages(c.bn, epi_vec, planes);
  if (c.stages <= 0 || c.stages > max_stages) c.stages = max_stages;
  // K blocks per barrier round. One round costs the issuing thread about 310 + 44 n cycles for n MMAs (measured),
  // which four 128x256x16 MMAs (512 cycles) barely hide and four narrower ones do not. Measured: two blocks per
  // round at 256 columns (4096^3 f16 1100 -> 1290 TFLOP/s with this producer loop), four at 128 and 64 columns.
  // Variant bits 28-29: 1, 2, 3 = 1, 2, 4 blocks; 0 = this rule.
  // (two TF32 planes: a K block is twelve MMAs, a round of its own)
  const int kpr_code = planes == 2 ? 1 : (variant >> 28) & 3;
  c.kpr = kpr_code == 1 ? 1 : kpr_code == 2 ? 2 : kpr_code == 3 ? 4 : (c.bn <= 128 ? 4 : 2);
  while (c.kpr > 1 && c.stages < 2 * c.kpr) c.kpr /= 2;   // at least two rounds in flight
  c.stages = c.stages / c.kpr * c.kpr;
  c.plain_stores = ((variant >> 8) & 1) != 0;
  const int bke = kRowBytes / es;
  const long long kblocks = (p->k + bke - 1) / bke;
  const long long tiles = (long long)p->g * ((p->m + kBM * c.ctas - 1) / (kBM * c.ctas)) * ((p->n + c.bn - 1) / c.bn);
  const long long units = planned_sms() / c.ctas;
  c.splits = est_splits ? est_splits : (variant >> 16) & 0xFF;
  if (c.splits == 0) {
    c.splits = 1;
    if (tiles * 2 <= units && kblocks >= 16) {
      long long want = units / tiles;
      long long cap = kblocks / 8;  // at least 8 K blocks per range
      c.splits = (int)std::max<long long>(1, std::min<long long>(std::min(want, cap), 128));
    }
  }
  // f32 in accurate mode: the tensor core adds each MMA's products into the f32 accumulator with truncation, a bias
  // of about -2^-24 per 8-element step that grows linearly with the length of one accumulation chain (measured:
  // relative error 7.5e-9 x K on same-sign data; 1.9e-4 at K = 25088, where the sequential f32 loop of the reference
  // has 1e-5). Chains are therefore kept to 2048 elements; the partial planes are added with round-to-nearest.
  if (p->ab_type == RB_F32 && p->f32_mode == 0) {   // also under an explicit variant: shorter chains only
    const long long need = std::min<long long>(((long long)p->k + 2047) / 2048, 255);
    if (need > c.splits) c.splits = (int)need;
  }
  if (c.splits > kblocks) c.splits = (int)kblocks;
  // every range must be non-empty with ceil-division ranges
  // (also of the blocks of 64 that f16 planes have: 29 ranges of K = 50176 are 28 of them, and the sum read a plane that nobody had written)
  const bool both = halves_pay(p, implicit) && (asked == 0 || ((variant >> 16) & 0xFF) == 0);
  auto empty = [&](long long blocks) { return (c.splits - 1) * ((blocks + c.splits - 1) / c.splits) >= blocks; };
  while (c.splits > 1 && (empty(kblocks) || (both && empty((p->k + 63LL) / 64)))) --c.splits;
  // Stream-K tail (variant bit 9 switches it ON): when the last wave of whole tiles would leave more than 5 % of the
  // GPU idle, the tiles of the last full wave plus the remainder are dealt out by K blocks instead. Measured on
  // B200 it does not pay for the shapes tried (4096^3 f16: 1090 vs 1120 TFLOP/s sustained; 2048x11008x4096 i8:
  // 2000 vs 2300 TOP/s): the GPU runs at its power cap, idle SMs in the last wave let the busy ones clock higher,
  // and the short partial items expose their epilogues. It stays available for tuning.
  c.dp_tiles = (int)tiles;
  c.sk_tiles = 0;
  if (c.splits == 1 && tiles > units && ((variant >> 9) & 1) && kblocks >= 8) {
    const long long rem = tiles % units;
    const long long waves = (tiles + units - 1) / units;
    if (rem != 0 && (double)(units - rem) / (double)(waves * units) > 0.05) {
      c.sk_tiles = (int)(rem + units);
      c.dp_tiles = (int)(tiles - c.sk_tiles);
    }
  }
  return c;
}

// The configuration of a launch that is to be one kernel, or has no room for the planes of K ranges: ranges that only keep the sums of an
// f32 result short, or gain little, are left out; others stay.
GemmConfig choose_one_kernel(const RbGemmProblem* p, int variant, bool epi_vec = false, bool implicit = false) {
  const GemmConfig c = choose_config(p, variant, epi_vec, implicit);
  if (c.splits == 1) return c;
  const GemmConfig whole = choose_config(p, variant, epi_vec, implicit, true);
  return whole.splits == 1 || p->ab_type == RB_F32 ? whole : c;
}

// Sums the partial planes of a K split in a fixed order (range 0, 1, 2, ...), applies the epilogue and
// writes C. One thread per VEC consecutive columns of a row, the reads of up to eight planes in flight together: the pass
// is bound by reading the planes (they are in L2), and a result of few rows has few threads to hide that latency with.
// VEC = 4 needs rows of a multiple of four columns, C stored row-major and its rows on boundaries of four elements.
template <int VEC>
__global__ void splitk_reduce_kernel(const void* __restrict__ partial, int splits, long long plane, int G, int M, int N,
                                     void* __restrict__ c, int c_type, int trans_c, int acc_is_int, EpiParams epi) {
  const long long total = (long long)G * M * N / VEC;
  griddep_wait();
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < total; i0 += (long long)gridDim.x * blockDim.x) {
    const long long i = i0 * VEC;
    const long long gm = (i >> 32) ? i / N : (long long)((unsigned)i / (unsigned)N);
    const int n = (int)(i - gm * N);
    const long long g = (gm >> 32) ? gm / M : (long long)((unsigned)gm / (unsigned)M);
    const int m = (int)(gm - g * M);
    const long long o = trans_c ? (g * N + n) * (long long)M + m : i;
    uint32_t acc[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] = 0u;
    for (int s0 = 0; s0 < splits; s0 += 8) {
      uint32_t v[8][VEC];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        if (s0 + s < splits) {
          const uint32_t* q = reinterpret_cast<const uint32_t*>(partial) + (s0 + s) * plane + i;
          if constexpr (VEC == 4) {
            const uint4 u = __ldcg(reinterpret_cast<const uint4*>(q));
            v[s][0] = u.x; v[s][1] = u.y; v[s][2] = u.z; v[s][3] = u.w;
          } else {
            v[s][0] = __ldcg(q);
          }
        }
      }
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s0 + s < splits) {
#pragma unroll
          for (int e = 0; e < VEC; ++e)
            acc[e] = acc_is_int ? acc[e] + v[s][e] : __float_as_uint(__fadd_rn(__uint_as_float(acc[e]), __uint_as_float(v[s][e])));
        }
    }
    if (acc_is_int && c_type == RB_I32 && epi.flags == 0) {
      if constexpr (VEC == 4) *reinterpret_cast<uint4*>(static_cast<uint32_t*>(c) + o) = make_uint4(acc[0], acc[1], acc[2], acc[3]);
      else static_cast<uint32_t*>(c)[o] = acc[0];
      continue;
    }
    float x[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      x[e] = acc_is_int ? __int2float_rn((int)acc[e]) : __uint_as_float(acc[e]);
      if (epi.flags) x[e] = epi_apply(x[e], epi, n + e, m, o + e);
    }
    if constexpr (VEC == 4) {
      if (c_type == RB_F32) {
        *reinterpret_cast<float4*>(static_cast<float*>(c) + o) = make_float4(x[0], x[1], x[2], x[3]);
      } else if (c_type == RB_F16) {
        __half2 h[2] = {__floats2half2_rn(x[0], x[1]), __floats2half2_rn(x[2], x[3])};
        *reinterpret_cast<uint2*>(static_cast<__half*>(c) + o) = *reinterpret_cast<uint2*>(h);
      } else if (c_type == RB_BF16) {
        __nv_bfloat162 h[2] = {__floats2bfloat162_rn(x[0], x[1]), __floats2bfloat162_rn(x[2], x[3])};
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(c) + o) = *reinterpret_cast<uint2*>(h);
      } else {
#pragma unroll
        for (int e = 0; e < VEC; ++e) store_elem(c, o + e, x[e], c_type, epi.out_zero);
      }
    } else {
      store_elem(c, o, x[0], c_type, epi.out_zero);
    }
  }
}

struct OperandPlan {
  bool src_mn_major;    // as stored by the caller: contiguous dimension is M/N (not K)
  bool mn_major;        // as the kernel sees it (after a transposing copy, if any)
  int src_rows, src_cols;  // stored matrix per batch
  long long rows;       // rows per batch as the kernel sees it
  int cols;             // contiguous extent as the kernel sees it
  int pitch;            // elements per row as the kernel sees it
  bool needs_copy;      // operand goes through the workspace
};

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

OperandPlan plan_operand(bool mn_major, int mn, int k, size_t es, bool is_f32, bool split) {
  OperandPlan o;
  o.src_mn_major = mn_major;
  o.src_rows = mn_major ? k : mn;
  o.src_cols = mn_major ? mn : k;
  o.mn_major = is_f32 ? false : mn_major;
  o.rows = o.mn_major ? k : mn;
  o.cols = o.mn_major ? mn : k;
  const int elems16 = (int)(16 / es);
  o.pitch = (o.cols + elems16 - 1) / elems16 * elems16;
  o.needs_copy = o.pitch != o.cols || (is_f32 && (split || mn_major));
  return o;
}

bool valid_ab(int t) {
  return t == RB_F32 || t == RB_F16 || t == RB_BF16 || t == RB_I8 || (t >= RB_F8E4M3 && t <= RB_F8E5M2_E4M3);
}
bool valid_c(int t) { return t >= RB_F32 && t <= RB_F8E4M3; }

RbStatus check_problem(const RbGemmProblem* p) {
  if (!p) return fail(RB_INVALID_PARAM, "problem is NULL");
  if (p->g <= 0 || p->m <= 0 || p->n <= 0 || p->k <= 0) return fail(RB_INVALID_PARAM, "g, m, n, k must be positive");
  if (!valid_ab(p->ab_type) || !valid_c(p->c_type)) return fail(RB_INVALID_PARAM, "unknown element type");
  return RB_SUCCESS;
}

size_t halves_state_at(size_t total) { return align_up(total, 256); }
size_t halves_workspace(size_t total) { return halves_state_at(total) + 256; }

struct Workspace {
  size_t a_off[2], b_off[2];  // [0] = copy / hi, [1] = lo
  size_t partial_off;         // K-split partial planes
  size_t sk_off, sk_flags_off;  // stream-K partial tiles and their arrival counters
  size_t total;
};

Workspace plan_workspace(const RbGemmProblem* p, const OperandPlan& oa, const OperandPlan& ob, const GemmConfig& cfg) {
  Workspace w{};
  const size_t es = dtype_bytes(p->ab_type);
  const bool split = p->ab_type == RB_F32 && p->f32_mode == 0;
  size_t off = 0;
  const size_t a_bytes = align_up((size_t)p->g * oa.rows * oa.pitch * es, 256);
  const size_t b_bytes = align_up((size_t)p->g * ob.rows * ob.pitch * es, 256);
  if (oa.needs_copy) { w.a_off[0] = off; off += a_bytes; }
  if (split && oa.needs_copy) { w.a_off[1] = off; off += a_bytes; }
  if (ob.needs_copy) { w.b_off[0] = off; off += b_bytes; }
  if (split && ob.needs_copy) { w.b_off[1] = off; off += b_bytes; }
  if (cfg.splits > 1) {
    w.partial_off = off;
    off += align_up((size_t)cfg.splits * p->g * p->m * p->n * 4, 256);
  }
  if (cfg.sk_tiles > 0) {
    const size_t units = planned_sms() / cfg.ctas;
    w.sk_off = off;
    off += align_up(units * (size_t)(kBM * cfg.ctas) * cfg.bn * 4, 256);
    w.sk_flags_off = off;
    off += align_up(units * 8 * sizeof(unsigned int), 256);
  }
  w.total = off;
  return w;
}


}  // namespace
}  // namespace rb

using namespace rb;

extern "C" void rbSetGemmVariant(int variant) { t_variant = variant; }
extern "C" int rbGetGemmVariant(void) { return t_variant; }
extern "C" void rbSetWaitLimit(uint64_t sm_cycles) {
  t_wait_cycles = sm_cycles == 0 ? kWaitCycles : (long long)std::min<uint64_t>(sm_cycles, (uint64_t)1 << 40);
}
extern "C" void rbInjectStall(int launches) { t_stall_launches = launches > 0 ? launches : 0; }

size_t rb::gemm_workspace_bytes(const RbGemmProblem* p, int implicit_operand, bool least) {
  if (check_problem(p) != RB_SUCCESS) return 0;
  const size_t es = dtype_bytes(p->ab_type);
  const bool f32 = p->ab_type == RB_F32, split = f32 && p->f32_mode == 0;
  OperandPlan oa = plan_operand(p->trans_a != 0, p->m, p->k, es, f32, split);
  OperandPlan ob = plan_operand(p->trans_b == 0, p->n, p->k, es, f32, split);
  if (implicit_operand == 0) oa.needs_copy = false;
  if (implicit_operand == 1) ob.needs_copy = false;
  const size_t total = plan_workspace(p, oa, ob, (least ? choose_one_kernel(p, t_variant, false, implicit_operand >= 0)
                                                        : choose_config(p, t_variant, false, implicit_operand >= 0))).total;
  return !least && implicit_operand <= 0 && halves_pay(p, implicit_operand == 0) ? halves_workspace(total) : total;
}

extern "C" size_t rbGemmWorkspaceSize(const RbGemmProblem* p) { return rb::gemm_workspace_bytes(p, -1); }

RbStatus rb::f32_planes(const float* src, float* hi, float* lo, int groups, int R, int C, int pitch, bool transpose,
                        bool split, void* stream_v) {
  // the pass stores 16 bytes at a time (and the tensor maps over the planes ask for the same start)
  if (reinterpret_cast<uintptr_t>(hi) % 16 || (split && reinterpret_cast<uintptr_t>(lo) % 16) || pitch % 4)
    return fail(RB_UNSUPPORTED, "f32 planes: the workspace must be 16-byte aligned");
  const DeviceInfo* dev = device_info();
  if (!dev) return RB_CUDA_ERROR;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  F32Jobs jobs;
  memset(&jobs, 0, sizeof(jobs));
  jobs.job[0] = plane_job(src, hi, split ? lo : nullptr, R, C, pitch, transpose);
  return launch_f32_jobs(jobs, 1, groups, dev->sm_count, stream);
}

extern "C" RbStatus rbGemmGetConfig(const RbGemmProblem* p, RbGemmConfigInfo* out) { return rb::gemm_config(p, -1, out); }

RbStatus rb::gemm_config(const RbGemmProblem* p, int implicit_operand, RbGemmConfigInfo* out, bool one_kernel) {
  RbStatus st = check_problem(p);
  if (st != RB_SUCCESS) return st;
  if (!out) return fail(RB_INVALID_PARAM, "out is NULL");
  const auto choose = [&](bool epi_vec) {
    return one_kernel ? choose_one_kernel(p, t_variant, epi_vec, implicit_operand >= 0) : choose_config(p, t_variant, epi_vec, implicit_operand >= 0);
  };
  const GemmConfig c = choose(false);
  const int es = (int)dtype_bytes(p->ab_type);
  const long long tiles = (long long)p->g * ((p->m + kBM * c.ctas - 1) / (kBM * c.ctas)) * ((p->n + c.bn - 1) / c.bn);
  const long long items = tiles * c.splits;
  const long long units = planned_sms() / c.ctas;
  memset(out, 0, sizeof(*out));
  out->tile_m = kBM * c.ctas;
  out->tile_n = c.bn;
  out->tile_k = kRowBytes / es;
  out->ctas = c.ctas;
  out->stages = c.stages;
  out->splits = c.splits;
  out->stream_k = c.sk_tiles > 0 ? 1 : 0;
  out->grid = (uint32_t)(c.ctas * std::min<long long>(items, units));
  out->block = kGemmThreads;
  out->dynamic_smem = (uint32_t)(c.ctas == 2 ? GemmSmemLayout<2>::total(c.stages, c.bn, false, gemm_planes(p))
                                              : GemmSmemLayout<1>::total(c.stages, c.bn, false, gemm_planes(p)));
  // with per-column epilogue vectors (bias / column scales) the ring may be one stage shorter and the staging single
  {
    const GemmConfig ce = choose(true);
    out->stages_epi_vec = ce.stages;
    out->dynamic_smem_epi_vec = (uint32_t)(ce.ctas == 2 ? GemmSmemLayout<2>::total(ce.stages, ce.bn, true, gemm_planes(p))
                                                        : GemmSmemLayout<1>::total(ce.stages, ce.bn, true, gemm_planes(p)));
  }
  out->kpr = c.kpr;
  const int bn_code = c.bn == 64 ? 1 : c.bn == 128 ? 2 : 3;
  const int kpr_code = c.kpr == 1 ? 1 : c.kpr == 2 ? 2 : 3;
  out->variant = (uint32_t)c.ctas | ((uint32_t)c.stages << 4) | (c.plain_stores ? 1u << 8 : 0u) |
                 (c.sk_tiles > 0 ? 1u << 9 : 0u) | ((uint32_t)bn_code << 12) | ((uint32_t)c.splits << 16) |
                 ((uint32_t)kpr_code << 28);
  return RB_SUCCESS;
}

extern "C" RbStatus rbGemm(const RbGemmProblem* p, const RbEpilogue* epi, const void* a, const void* b, void* c,
                           void* workspace, size_t workspace_bytes, void* stream_v) {
  return rb::gemm_run(p, epi, a, b, c, workspace, workspace_bytes, stream_v, nullptr);
}

// Name of an instantiation of gemm_tcgen05_kernel inside the cubin image (Itanium mangling of
// rb::gemm_tcgen05_kernel<KIND, A_MN, B_MN, CTAS, TAIL>(GemmTensorMaps, GemmParams)).
static std::string kernel_symbol(int kind, bool a_mn, bool b_mn, int ctas, int tail) {
  return "_ZN2rb19gemm_tcgen05_kernelILi" + std::to_string(kind) + "ELb" + (a_mn ? "1" : "0") + "ELb" + (b_mn ? "1" : "0") +
         "ELi" + std::to_string(ctas) + "ELi" + std::to_string(tail) + "EEEvNS_14GemmTensorMapsENS_10GemmParamsE";
}

RbStatus rb::check_epilogue(const RbEpilogue* epi, int c_type) {
  if (!epi) return RB_SUCCESS;
  const uint32_t flags = epi->flags;
  if ((flags & RB_EPI_COL_SCALE) && !epi->col_scale) return fail(RB_INVALID_PARAM, "col_scale is NULL");
  if ((flags & RB_EPI_BIAS) && !epi->bias) return fail(RB_INVALID_PARAM, "bias is NULL");
  if ((flags & RB_EPI_BIAS) && !(epi->bias_type == RB_F32 || epi->bias_type == RB_F16 || epi->bias_type == RB_BF16))
    return fail(RB_INVALID_PARAM, "bias_type must be f32, f16 or bf16");
  if ((flags & RB_EPI_BIAS_ROW) && (flags & RB_EPI_BIAS_SCALAR)) return fail(RB_INVALID_PARAM, "bias is per row or scalar, not both");
  if ((epi->flags & RB_EPI_RESIDUAL) && !epi->residual) return fail(RB_INVALID_PARAM, "residual is NULL");
  if ((epi->flags & RB_EPI_RESIDUAL) && !(epi->res_type == RB_F32 || epi->res_type == RB_F16 || epi->res_type == RB_BF16))
    return fail(RB_INVALID_PARAM, "res_type must be f32, f16 or bf16");
  if ((epi->flags & RB_EPI_UNARY) && (epi->unary <= RB_UNARY_NONE || epi->unary > RB_UNARY_TANH))
    return fail(RB_INVALID_PARAM, "unary must name one of the RbUnary functions");
  if ((flags & RB_EPI_CLIP) && !(epi->clip_lo <= epi->clip_hi)) return fail(RB_INVALID_PARAM, "clip needs lo <= hi");
  if ((flags & RB_EPI_ZP_OUT) && c_type != RB_I8) return fail(RB_INVALID_PARAM, "an output zero point needs an i8 result");
  return RB_SUCCESS;
}

RbStatus rb::gemm_run(const RbGemmProblem* p, const RbEpilogue* epi, const void* a, const void* b, void* c,
                      void* workspace, size_t workspace_bytes, void* stream_v, const ConvAOperand* conva,
                      RbKernelLaunch* capture) {
  RbStatus st = check_problem(p);
  if (st != RB_SUCCESS) return st;
  const bool conv_a = conva && conva->operand == 0, conv_b = conva && conva->operand == 1;
  if (conva) {
    const bool f32_ok = conv_a && (p->f32_mode != 0 || conva->tensor_lo);   // TF32 planes prepared by the caller
    if (p->g != 1 || (conv_a && p->trans_a) || (conv_b && p->trans_b) || (p->ab_type == RB_F32 && !f32_ok) || !conva->tensor)
      return fail(RB_UNSUPPORTED, "implicit operand: one group, A K-major or B stored K x N (f32: A only, as TF32 planes)");
    if (conv_a) a = conva->tensor;
    else b = conva->tensor;
  }
  if (!a || !b || !c) return fail(RB_INVALID_PARAM, "a, b and c must be device pointers");
  const DeviceInfo* dev = device_info();
  if (!dev) return RB_CUDA_ERROR;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

  const int abt = p->ab_type;
  const size_t es = dtype_bytes(abt);
  const bool is_int = abt == RB_I8;
  const uint32_t flags = (epi ? epi->flags : 0u) | (p->store_method == 1 ? (uint32_t)RB_EPI_RESIDUAL : 0u);
  if (is_int && flags == 0 && p->c_type != RB_I32)
    return fail(RB_UNSUPPORTED, "i8 x i8 without an epilogue produces i32 (rocmlir-gen: -t i8 implies an i32 result)");
  if (!is_int && p->c_type == RB_I32) return fail(RB_UNSUPPORTED, "float inputs cannot produce an i32 result");
  if (p->store_method != 0 && p->store_method != 1) return fail(RB_INVALID_PARAM, "store_method must be 0 (set) or 1 (add)");
  if (p->store_method == 1) {
    // C += A.B (rock.gemm with store_method = atomic_add, RockOps.td:136-181): the fused residual step reading C itself
    if (!(p->c_type == RB_F32 || p->c_type == RB_F16 || p->c_type == RB_BF16))
      return fail(RB_UNSUPPORTED, "store_method add exists for f32, f16 and bf16 results");
    if (epi && (epi->flags & RB_EPI_RESIDUAL)) return fail(RB_UNSUPPORTED, "store_method add cannot be combined with a residual operand");
  }
  st = check_epilogue(epi, p->c_type);
  if (st != RB_SUCCESS) return st;

  int kind;
  uint32_t fmt, fmt_b = 0xffffffffu, cfmt = 1;   // fmt_b: B's format when it differs from A's
  switch (abt) {
    case RB_F16: kind = kKindF16; fmt = 0; break;
    case RB_BF16: kind = kKindF16; fmt = 1; break;
    case RB_F32: kind = kKindTF32; fmt = 2; break;
    case RB_I8: kind = kKindI8; fmt = 1; cfmt = 2; break;
    case RB_F8E5M2: kind = kKindF8; fmt = 1; break;               // f8f6f4 kind: 0 = e4m3, 1 = e5m2
    case RB_F8E4M3_E5M2: kind = kKindF8; fmt = 0; fmt_b = 1; break;
    case RB_F8E5M2_E4M3: kind = kKindF8; fmt = 1; fmt_b = 0; break;
    default: kind = kKindF8; fmt = 0; break;
  }

  const bool is_f32 = abt == RB_F32;
  const bool split = is_f32 && p->f32_mode == 0;
  OperandPlan oa = plan_operand(p->trans_a != 0 /* A stored G x K x M */, p->m, p->k, es, is_f32, split);
  if (conv_a) {  // fetched in place by im2col loads: never copied, never padded
    oa.needs_copy = false;
    oa.pitch = oa.cols;
  }
  OperandPlan ob = plan_operand(p->trans_b == 0 /* B stored G x K x N */, p->n, p->k, es, is_f32, split);
  if (conv_b) {
    ob.needs_copy = false;
    ob.pitch = ob.cols;
  }
  const bool a_mn = oa.mn_major, b_mn = ob.mn_major;
  const bool epi_vec = epi_needs_col_vectors(flags);
  GemmConfig cfg = choose_config(p, t_variant, epi_vec, conva != nullptr);
  Workspace ws = plan_workspace(p, oa, ob, cfg);
  if (cfg.splits > 1 && (capture || !workspace || workspace_bytes < ws.total)) {
    cfg = choose_one_kernel(p, t_variant, epi_vec, conva != nullptr);
    ws = plan_workspace(p, oa, ob, cfg);
  }
  if (cfg.sk_tiles > 0 && (!workspace || workspace_bytes < ws.total)) {
    // the stream-K tail is an optimisation: without room for its partial tiles every tile is computed whole
    cfg.sk_tiles = 0;
    ws = plan_workspace(p, oa, ob, cfg);
  }
  const GemmChain* chain = t_chain;
  // group 1 of a chained pair: A is group 0's C, B and C are the chain's; base = lower address, stride = distance
  const void* chain_ptr[3][2] = {{a, c}, {b, chain ? chain->b2 : nullptr}, {c, chain ? chain->c2 : nullptr}};
  uint64_t chain_stride[3] = {0, 0, 0};
  int chain_flip = 0;
  if (chain) {
    if (p->g != 2 || oa.needs_copy || ob.needs_copy || cfg.splits != 1 || conva || epi || capture || p->trans_c ||
        p->store_method != 0 || p->c_type != abt || p->k != p->n)
      return fail(RB_UNSUPPORTED, "this pair of products does not run as one chained launch");
    if (cfg.sk_tiles > 0) { cfg.sk_tiles = 0; ws = plan_workspace(p, oa, ob, cfg); }
    for (int i = 0; i < 3; ++i) {
      const uintptr_t x0 = reinterpret_cast<uintptr_t>(chain_ptr[i][0]), x1 = reinterpret_cast<uintptr_t>(chain_ptr[i][1]);
      const uintptr_t d = x1 > x0 ? x1 - x0 : x0 - x1;
      if (d == 0 || d % 16 || x0 % 16 || d >= ((uintptr_t)1 << 40))
        return fail(RB_UNSUPPORTED, "chained launch: the two tensors of an operand must be distinct, 16-byte aligned and within 2^40 bytes");
      chain_stride[i] = (uint64_t)d;
      if (x1 < x0) chain_flip |= 1 << i;
    }
  }
  if (capture && (oa.needs_copy || ob.needs_copy || cfg.splits > 1))
    return fail(RB_UNSUPPORTED, "this problem runs as several kernels (operand copy, TF32 planes or a K split): it has no "
                                "single-kernel binary; launch it through the library");
  if (ws.total > 0) {
    if (!workspace || workspace_bytes < ws.total)
      return fail(RB_WORKSPACE_TOO_SMALL, "workspace of " + std::to_string(ws.total) + " bytes required");
    if (reinterpret_cast<uintptr_t>(workspace) % 16) return fail(RB_INVALID_PARAM, "workspace must be 16-byte aligned");
  }
  if ((reinterpret_cast<uintptr_t>(a) % 16 && !oa.needs_copy) || (reinterpret_cast<uintptr_t>(b) % 16 && !ob.needs_copy))
    return fail(RB_UNSUPPORTED, "operand base addresses must be 16-byte aligned");

  EpiParams ep;
  memset(&ep, 0, sizeof(ep));
  if (epi) {
    ep.flags = epi->flags; ep.alpha = epi->alpha; ep.out_recip = epi->out_recip;
    ep.mid_type = epi->mid_type; ep.bias_type = epi->bias_type;
    ep.col_scale = epi->col_scale; ep.bias = epi->bias;
    ep.clip_lo = epi->clip_lo; ep.clip_hi = epi->clip_hi;
    ep.in_zero = epi->in_zero; ep.out_zero = (epi->flags & RB_EPI_ZP_OUT) ? epi->out_zero : 0;
    ep.residual = epi->residual; ep.res_type = epi->res_type;
    ep.unary = (epi->flags & RB_EPI_UNARY) ? epi->unary : 0;
  }
  if (p->store_method == 1) {
    // the kernel's result is rounded to C's type and added to what C holds, like an atomic add of the stored value
    ep.flags |= RB_EPI_RESIDUAL;
    ep.residual = c; ep.res_type = p->c_type;
    if (!(ep.flags & RB_EPI_ROUND_MID)) { ep.flags |= RB_EPI_ROUND_MID; ep.mid_type = p->c_type; }
  }

  // few rows against weights stored N x K: the tile turned round (an explicit variant keeps this kernel)
  if (!capture && !chain && !conva && t_variant == 0 && gemm_skinny_applicable(p, ep.flags) && tuned_variant_gemm(p) == 0) {
    const int stall = t_stall_launches > 0 ? 1 : 0;
    t_stall_launches -= stall;
    return gemm_skinny_run(p, ep, a, b, c, kind, fmt, fmt_b == 0xffffffffu ? fmt : fmt_b, cfmt, t_wait_cycles, stall, stream_v);
  }

  // Two K ranges of an f32 product in full accuracy: both are added to a C of zeros by TMA reductions instead of going through planes and a
  // pass that sums them. 0 + x + y and 0 + y + x are the same number, so the result does not depend on which comes first; of three
  // ranges it would. Subnormal partial sums and results are kept (tests/test_gemm_f32_ranges_gpu.py). 4096^3: 678 us -> 657 in all.
  // C is cleared right before the launch: by then both operands have been read into their planes (hence full accuracy only; a single TF32
  // pass may read them in place), so C may lie over one of them as with any other number of ranges. The workspace query knows neither C's
  // address nor the epilogue and counts the planes all the same.
  const bool add_ranges = cfg.splits == 2 && split && p->c_type == RB_F32 && ep.flags == 0 && !p->trans_c && !cfg.plain_stores && !chain &&
                          p->n % 4 == 0 && reinterpret_cast<uintptr_t>(c) % 16 == 0;

  // without room for their state, or as a part of something else, TF32 planes
  const bool conv_src = conv_a && conva->src != nullptr;
  const bool halves = halves_pay(p, conv_a) && t_variant == 0 && !capture && !chain && (!conva || (conv_src && conva->tensor_lo && conva->C % 64 == 0)) &&
                      (oa.needs_copy || conv_src) && ob.needs_copy && workspace && workspace_bytes >= halves_workspace(ws.total);

  uint8_t* wsb = static_cast<uint8_t*>(workspace);
  HalvesState* const state = halves ? reinterpret_cast<HalvesState*>(wsb + halves_state_at(ws.total)) : nullptr;
  const int half_pitch = (int)align_up((size_t)p->k, 8);
  const void* a_half[2] = {nullptr, nullptr};
  const void* b_half[2] = {nullptr, nullptr};
  const void* a_src[2] = {a, nullptr};
  const void* b_src[2] = {b, nullptr};
  if (is_f32) {
    F32Jobs jobs;
    memset(&jobs, 0, sizeof(jobs));
    int nj = 0;
    auto add = [&](const void* src, const OperandPlan& o, const size_t* off, const void** planes) {
      float* hi = reinterpret_cast<float*>(wsb + off[0]);
      float* lo = split ? reinterpret_cast<float*>(wsb + off[1]) : nullptr;
      jobs.job[nj++] = plane_job(static_cast<const float*>(src), hi, lo, o.src_rows, o.src_cols, o.pitch, o.src_mn_major);
      planes[0] = hi;
      planes[1] = lo;
    };
    if (oa.needs_copy) add(a, oa, ws.a_off, a_src);
    if (ob.needs_copy) add(b, ob, ws.b_off, b_src);
    if (halves) {
      // the f16 planes lie where the TF32 ones would: whichever form is not taken is never read
      HalvesSample sample;
      sample.src[0] = conv_src ? conva->src : static_cast<const float*>(a); sample.src[1] = static_cast<const float*>(b);
      sample.n[0] = conv_src ? (long long)conva->src_groups * conva->src_rows * conva->src_cols : (long long)p->g * p->m * p->k;
      sample.n[1] = (long long)p->g * p->k * p->n;
      sample.state = state;
      HalvesJobs hj;
      memset(&hj, 0, sizeof(hj));
      hj.state = state;
      auto add_half = [&](int i, const void* src, const OperandPlan& o, const size_t* off, const void** planes) {
        __half* hi = reinterpret_cast<__half*>(wsb + off[0]);
        __half* lo = hi + align_up((size_t)p->g * o.rows * half_pitch, 128);
        hj.job[i] = plane_job(static_cast<const float*>(src), hi, lo, o.src_rows, o.src_cols, half_pitch, o.src_mn_major);
        hj.first[i + 1] = hj.first[i] + p->g * (long long)hj.job[i].tiles_x * hj.job[i].tiles_y;
        planes[0] = hi;
        planes[1] = lo;
      };
      if (conv_src) {
        hj.job[0] = plane_job(conva->src, reinterpret_cast<__half*>(const_cast<void*>(conva->tensor)),
                               reinterpret_cast<__half*>(const_cast<void*>(conva->tensor_lo)), conva->src_rows, conva->src_cols, conva->C,
                               conva->src_transpose);
        hj.first[1] = conva->src_groups * (long long)hj.job[0].tiles_x * hj.job[0].tiles_y;
      } else {
        add_half(0, a, oa, ws.a_off, a_half);
      }
      add_half(1, b, ob, ws.b_off, b_half);
      RB_CUDA_TRY(launch_after(halves_scale_kernel, 1, 1024, 0, stream, 1, sample));
      RB_CUDA_TRY(launch_after(f32_halves_kernel, (unsigned)std::min<long long>(hj.first[2], (long long)dev->sm_count * 32), 256, 0, stream, 1, hj));
      count_launch(2);
    }
    if (conv_src) {
      F32Jobs image;
      memset(&image, 0, sizeof(image));
      image.job[0] = plane_job(conva->src, static_cast<float*>(const_cast<void*>(conva->tensor)), static_cast<float*>(const_cast<void*>(conva->tensor_lo)),
                             conva->src_rows, conva->src_cols, conva->C, conva->src_transpose);
      st = launch_f32_jobs(image, 1, conva->src_groups, dev->sm_count, stream, halves ? &state->flag : nullptr);
      if (st != RB_SUCCESS) return st;
    }
    if (nj > 0) st = launch_f32_jobs(jobs, nj, p->g, dev->sm_count, stream, halves ? &state->flag : nullptr);
    if (st != RB_SUCCESS) return st;
  } else {
    PadJobs pj;
    memset(&pj, 0, sizeof(pj));
    int nj = 0;
    auto add = [&](const void* src, const OperandPlan& o, size_t off) {
      PadJob& j = pj.job[nj];
      j.src = static_cast<const uint8_t*>(src);
      j.dst = wsb + off;
      j.rows = (unsigned long long)p->g * o.rows;
      j.row_bytes = (unsigned)(o.cols * es);
      j.pitch_bytes = (unsigned)(o.pitch * es);
      pj.first[nj + 1] = pj.first[nj] + j.rows * (j.pitch_bytes / 16);
      ++nj;
    };
    if (oa.needs_copy) { add(a, oa, ws.a_off[0]); a_src[0] = wsb + ws.a_off[0]; }
    if (ob.needs_copy) { add(b, ob, ws.b_off[0]); b_src[0] = wsb + ws.b_off[0]; }
    if (nj > 0) {
      if (nj == 1) pj.first[2] = pj.first[1];
      const int pb = (int)std::min<unsigned long long>((pj.first[2] + 255) / 256, (unsigned long long)dev->sm_count * 8);
      RB_CUDA_TRY(launch_after(pad_rows_kernel, pb, 256, 0, stream, 1, pj));
      count_launch();
    }
  }
  RB_CUDA_TRY(cudaGetLastError());   // launch errors of the preparation kernels

  // Variant word (rbSetGemmVariant): bits 0-3: 1 = single CTA per tile, 2 = CTA pair (0 = automatic);
  // bits 4-7 ring depth; bit 8 plain stores instead of TMA stores; bits 12-15 tile width code (1 = 64,
  // 2 = 128, 3 = 256); bits 16-23 K-split count. Zero fields mean "choose" (see choose_config).
  const int ctas = cfg.ctas, bn = cfg.bn, stages = cfg.stages, splits = cfg.splits;

  const size_t es_c = dtype_bytes(p->c_type);
  void* partial = splits > 1 ? static_cast<void*>(wsb + ws.partial_off) : nullptr;

  // f32 products that may run on f16 planes are launched in both forms; the operands' state says on the device which one works
  for (int form = halves ? 0 : 1; form < 2; ++form) {
    const bool half = form == 0;
    const size_t es_op = half ? 2 : es;                    // of the planes that this form reads
    const int bke = (int)(kRowBytes / es_op);
    GemmTensorMaps maps;
    memset(&maps, 0, sizeof(maps));
    CUtensorMapDataType dt = abt == RB_F16 || half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                             : abt == RB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                             : abt == RB_F32  ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                              : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    // An MN-major tile is 128-byte chunks of M/N x K rows; when the extent is a whole number of chunks the chunk
    // index becomes a tensor dimension of its own and one 4-D box fetches the whole tile of a stage.
    const bool a_fused = oa.mn_major && oa.cols % bke == 0 && oa.pitch == oa.cols;
    const bool b_fused = ob.mn_major && ob.cols % bke == 0 && ob.pitch == ob.cols;
    auto encode_operand = [&](CUtensorMap* m, const void* base, const OperandPlan& o, int box_rows_kmajor,
                              std::string* err) {
      const bool fused = (&o == &oa) ? a_fused : b_fused;
      const int ci = (&o == &oa) ? 0 : 1;
      const uint64_t pitch = (uint64_t)(half ? half_pitch : o.pitch) * es_op;
      const uint64_t gstride = chain ? chain_stride[ci] : (uint64_t)o.rows * pitch;
      if (chain) base = (chain_flip >> ci) & 1 ? chain_ptr[ci][1] : chain_ptr[ci][0];
      if (fused) {
        const uint64_t dims[4] = {(uint64_t)bke, (uint64_t)o.rows, (uint64_t)(o.cols / bke), (uint64_t)p->g};
        const uint64_t strides[3] = {pitch, (uint64_t)kRowBytes, gstride};
        const uint32_t box[4] = {(uint32_t)bke, (uint32_t)bke, (uint32_t)(box_rows_kmajor / bke), 1u};
        return encode_tiled(m, dt, 4, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, err);
      }
      const uint64_t dims[3] = {(uint64_t)o.cols, (uint64_t)o.rows, (uint64_t)p->g};
      const uint64_t strides[2] = {pitch, gstride};
      // K-major: box = BKE k-elements x tile rows. MN-major: box = one 128-byte chunk of MN x BKE k-rows.
      const uint32_t box[3] = {(uint32_t)bke, (uint32_t)(o.mn_major ? bke : box_rows_kmajor), 1u};
      return encode_tiled(m, dt, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, err);
    };
    std::string err;
    const int planes = gemm_planes(p);   // [0] hi (or the operand itself), [1] lo
    if (conva) {
      const ConvAOperand& cv = *conva;
      const int che = bke;                   // elements per 128-byte run of channels
      if (cv.C % che != 0) return fail(RB_UNSUPPORTED, "implicit operand: channels must be a multiple of 128 bytes");
      const long long pixels = (long long)cv.N * cv.P * cv.Q, taps = (long long)cv.Y * cv.X * cv.C;
      if (conv_a ? (pixels != p->m || taps != p->k) : (pixels != p->k || taps != p->n))
        return fail(RB_INVALID_PARAM, "implicit operand does not match the GEMM extents");
      const uint64_t dims[4] = {(uint64_t)cv.C, (uint64_t)cv.W, (uint64_t)cv.H, (uint64_t)cv.N};
      const uint64_t strides[3] = {(uint64_t)cv.C * es_op, (uint64_t)cv.W * cv.C * es_op, (uint64_t)cv.H * cv.W * cv.C * es_op};
      // bounding box of the base pixel: from -pad to (extent - 1) + upper corner, so that stepping by the stride
      // visits exactly P x Q positions (CUTLASS states the same rule for its fprop maps)
      const int lower[2] = {-cv.pad_w, -cv.pad_h};
      const int upper[2] = {cv.pad_w_hi - (cv.X - 1) * cv.dil_w, cv.pad_h_hi - (cv.Y - 1) * cv.dil_h};
      const uint32_t trav[2] = {(uint32_t)cv.stride_w, (uint32_t)cv.stride_h};
      // A: a tile is 128 pixels (rows) x one K block of channels. B: a chunk is one K block of pixels x 64 channels.
      for (int sg = 0; sg < (conv_a ? planes : 1); ++sg) {
        const void* plane = sg == 1 ? cv.tensor_lo : cv.tensor;
        if (!encode_im2col_nhwc(conv_a ? &maps.a[sg] : &maps.b[0], dt, plane, dims, strides, lower, upper, (uint32_t)che,
                                (uint32_t)(conv_a ? kBM : bke), trav, &err))
          return fail(RB_UNSUPPORTED, "implicit operand (im2col): " + err);
      }
    }
    // An A of fewer rows than a tile: no others are asked for (what the stage then holds there goes into rows of the sum that nothing reads).
    // Rows beyond the tensor cost a TMA load more than rows of it do - us a call, fp8, K = 1344: 42 x 6560 9.8 -> 8.8, 42 x 8192 10.7 -> 8.8, 128 rows
    // 8.8 and 8.9 - where every CTA's tile has them; in the last row of tiles alone they are not seen.
    const int a_box = ctas == 1 && !conv_a && !chain && !oa.mn_major && p->m < kBM ? (int)(p->m + 7) / 8 * 8 : kBM;
    for (int s = 0; s < planes; ++s) {
      if (!conv_a && !encode_operand(&maps.a[s], half ? a_half[s] : a_src[s], oa, a_box, &err)) return fail(RB_UNSUPPORTED, "A: " + err);
      if (!conv_b && !encode_operand(&maps.b[s], half ? b_half[s] : b_src[s], ob, bn / ctas, &err)) return fail(RB_UNSUPPORTED, "B: " + err);
    }

    GemmParams kp;
    memset(&kp, 0, sizeof(kp));
    kp.G = p->g; kp.M = p->m; kp.N = p->n; kp.K = p->k;
    kp.bn = bn;
    kp.splits = splits;
    kp.tiles_m = (p->m + kBM * ctas - 1) / (kBM * ctas);
    kp.tiles_n = (p->n + bn - 1) / bn;
    kp.kblocks = (p->k + bke - 1) / bke;
    kp.planes = planes;
    kp.stage_tx = (ctas == 2 ? GemmSmemLayout<2>::stage_bytes(bn, planes) : GemmSmemLayout<1>::stage_bytes(bn, planes)) - planes * (kBM - a_box) * (int)kRowBytes;
    const uint32_t fmt_op = half ? 0u : fmt;
    kp.idesc = make_idesc(cfmt, fmt_op, fmt_b == 0xffffffffu ? fmt_op : fmt_b, a_mn ? 1u : 0u, b_mn ? 1u : 0u, (uint32_t)(kBM * ctas), (uint32_t)bn);
    kp.acc_is_int = is_int ? 1 : 0;
    if (splits > 1 && conva && conva->c_rows_per_img > 0)
      return fail(RB_UNSUPPORTED, "a channel-major result cannot be combined with a K split");
    if (splits > 1 && !add_ranges) {
      // every K range writes raw accumulators into its own plane; the reduction applies the epilogue
      kp.c = partial;
      kp.c_type = is_int ? RB_I32 : RB_F32;
      kp.c_stride_m = p->n; kp.c_stride_n = 1;
      kp.c_stride_g = (long long)p->m * p->n;
      kp.split_stride = (long long)p->g * p->m * p->n;
      kp.vec_ok = (p->n % 4 == 0) ? 1 : 0;
      kp.c_tma = cfg.plain_stores ? 0 : kp.vec_ok ? 1 : 2;   // planes are stored like a C of splits * g groups
    } else {
      kp.c = c;
      kp.c_type = p->c_type;
      if (p->trans_c) { kp.c_stride_m = 1; kp.c_stride_n = p->m; } else { kp.c_stride_m = p->n; kp.c_stride_n = 1; }
      kp.c_stride_g = (long long)p->m * p->n;
      if (chain)   // signed distance from group 0's result to group 1's, in elements
        kp.c_stride_g = (reinterpret_cast<intptr_t>(chain->c2) - reinterpret_cast<intptr_t>(c)) / (intptr_t)es_c;
      kp.vec_ok = (!p->trans_c && ((size_t)p->n * es_c) % 16 == 0 && reinterpret_cast<uintptr_t>(c) % 16 == 0) ? 1 : 0;
      // rows off 16-byte boundaries: staged like the others, copied out by the warps (us, element stores from the registers before): 3 x 640 x
      // 2279, K = 768, bf16 with bias and ReLU 179 -> 30; 2000 x 3001 x 640 95 -> 29; 4096 x 4095 x 4096 f16 243 -> 149; f32 768 x 1043 x 3648
      // 98 -> 64
      // (and so is an 8-bit result in tiles of 64 columns: the box of the store map is a staged row, 128 of them)
      kp.c_tma = cfg.plain_stores || p->trans_c ? 0 : kp.vec_ok && bn * es_c >= (size_t)kRowBytes ? 1 : 2;
      if (conva && conva->c_rows_per_img > 0) {   // NKHW result: strided element stores, coalesced along the pixels
        kp.c_rows_per_img = conva->c_rows_per_img;
        kp.c_img_stride = conva->c_img_stride;
        kp.c_stride_m = 1;
        kp.c_stride_n = conva->c_col_stride;
        kp.vec_ok = 0;
        kp.c_tma = 0;
      }
      kp.epi = ep;
    }
    if (kp.c_tma == 1) {
      const int st_type = kp.c_type;                      // what the kernel stores: C's type, or raw planes
      const size_t es_st = dtype_bytes(st_type);
      const CUtensorMapDataType cdt = st_type == RB_F16    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                      : st_type == RB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                      : st_type == RB_F32  ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                      : st_type == RB_I32  ? CU_TENSOR_MAP_DATA_TYPE_INT32
                                                           : CU_TENSOR_MAP_DATA_TYPE_UINT8;
      const uint64_t cdims[3] = {(uint64_t)p->n, (uint64_t)p->m, (uint64_t)p->g * (add_ranges ? 1 : splits)};
      const uint64_t cstrides[2] = {(uint64_t)p->n * es_st, chain ? chain_stride[2] : (uint64_t)p->m * p->n * es_st};
      const uint32_t cbox[3] = {(uint32_t)(kRowBytes / es_st), 32u, 1u};
      void* cbase = (chain && (chain_flip & 4)) ? chain->c2 : kp.c;
      if (!encode_tiled(&maps.c, cdt, 3, cbase, cdims, cstrides, cbox, CU_TENSOR_MAP_SWIZZLE_128B, &err))
        return fail(RB_UNSUPPORTED, "C: " + err);
    }
    kp.c_add = add_ranges ? 1 : 0;
    kp.status = dev->status_word;
    kp.stages = stages;
    kp.kpr = cfg.kpr;
    kp.probe = kProbeBuild ? (t_variant >> 24) & 7 : 0;
    kp.wait_cycles = t_wait_cycles;
    if (t_stall_launches > 0) { kp.stall = 1; t_stall_launches -= form; }
    // Set up early, a successor overlaps its launch with this kernel's tail; between launches of a stream the early start itself costs 0.4 to 0.8 us, which
    // is not always won back. us a call in a stream, early and not: 1791 x 1024 x 2944 i8 13.6 / 13.8, 2048^3 f16 19.2 / 19.7, 13 images 512 -> 128, 35x35,
    // pointwise, stride 2, 8.4 / 9.0. Not where
    // * the call has other launches, small blocks that wait beside the CTAs at work (300 x 700 x 4096, K in ranges, 15.5 / 15.2, 64 x 246 x 2019 f32
    //   19.6 / 18.6, 543 x 768 x 365 x 3, rows copied, 12.9 / 11.8, 3 x 1024 x 1024 x 769 14.7 / 14.3) - but the launch of the form that is not taken;
    // * few rows draw a large B, which is what bounds them, on more than half of the SMs, so that a successor's CTAs have to wait for one (45 x 6080 x 3392
    //   fp8 12.4 / 11.9, 256 x 4096 x 4096 i8 13.9 / 13.4, 164 x 2848 x 2688 fp8 10.9 / 10.4; 66 x 4336 x 1920 fp8, 68 CTAs, 8.9 / 9.3);
    // * single CTAs work on several short tiles each, the next tile's loads under way behind a tile's stores (171 images 64 -> 256, 44x44, input gradient,
    //   47.1 / 45.7, 148 images 64 -> 128, 45x45, input gradient, 32.6 / 31.9, 21 images 512 -> 64, 39x39 10.7 / 10.2; ten K blocks gain, 755 x 6416 x 1280 i8
    //   17.2 / 17.5, and so do pairs, 10 images 256 -> 512, 55x55, 19.4 / 20.0).
    const long long own = (long long)p->g * kp.tiles_m * kp.tiles_n * ctas;   // CTAs, were there one for every tile
    const bool streams_b = p->m <= 3 * kBM && (double)p->n * p->k * es >= 7e6 && 2 * own > dev->sm_count;
    const bool several = ctas == 1 && kp.kblocks <= 8 && own > dev->sm_count;
    kp.early = halves || !(splits > 1 || oa.needs_copy || ob.needs_copy || streams_b || several) ? 1 : 0;
    if (halves) {
      kp.gate = &state->flag;
      kp.gate_want = half ? 0u : 1u;
      kp.halves_scale = &state->out_scale;
    }
    if (conva) {
      kp.conva.enabled = conv_a ? 1 : 2; kp.conva.P = conva->P; kp.conva.Q = conva->Q; kp.conva.X = conva->X;
      kp.conva.cchunks = conva->C / bke;
      kp.conva.stride_h = conva->stride_h; kp.conva.stride_w = conva->stride_w;
      kp.conva.dil_h = conva->dil_h; kp.conva.dil_w = conva->dil_w; kp.conva.pad_h = conva->pad_h; kp.conva.pad_w = conva->pad_w;
    }
    kp.a_fused = a_fused ? 1 : 0;
    kp.b_fused = b_fused ? 1 : 0;

    if (chain) {
      if ((size_t)kp.tiles_m * kp.tiles_n * ctas * 4 * sizeof(unsigned int) > chain->flags_bytes)
        return fail(RB_UNSUPPORTED, "chained launch: too many tiles for the flag words");
      static std::atomic<unsigned int> next_chain_token{0xc4a10001u};
      kp.chain_flags = chain->flags;
      kp.chain_token = next_chain_token.fetch_add(1, std::memory_order_relaxed);
      kp.chain_flip = chain_flip;
    }
    const long long num_tiles = (long long)kp.G * kp.tiles_m * kp.tiles_n;
    const long long num_items = num_tiles * splits;
    if (num_items > 0x7fffffffLL) return fail(RB_UNSUPPORTED, "too many tiles");
    // the stream-K split was planned for a B200's SM count; on anything else every tile is computed whole
    const bool use_sk = cfg.sk_tiles > 0 && dev->sm_count == planned_sms();
    kp.dp_tiles = use_sk ? cfg.dp_tiles : (int)num_tiles;
    kp.sk_tiles = use_sk ? cfg.sk_tiles : 0;
    if (use_sk) {
      kp.sk_partial = wsb + ws.sk_off;
      kp.sk_flags = reinterpret_cast<unsigned int*>(wsb + ws.sk_flags_off);
      static std::atomic<unsigned int> next_token{0x5eed0001u};
      kp.sk_token = next_token.fetch_add(1, std::memory_order_relaxed);
    }

    // fused elementwise code and copied rows only in launches that have such work (see GemmTail)
    const int tail = kp.c_tma == 2 ? kTailCopied : kp.epi.flags != 0 ? kTailFused : kTailNone;
    const GemmKernel kern = half                 ? gemm_kernel_halves(ctas, tail)
                            : tail == kTailCopied  ? gemm_kernel_copied(kind, a_mn, b_mn, ctas)
                            : tail == kTailFused ? gemm_kernel_fused(kind, a_mn, b_mn, ctas)
                                                 : gemm_kernel_plain(kind, a_mn, b_mn, ctas);
    const bool kernel_epi_vec = splits == 1 && epi_vec;  // with a K split the reduction kernel applies the epilogue
    const int smem = ctas == 2 ? GemmSmemLayout<2>::total(stages, bn, kernel_epi_vec, planes) : GemmSmemLayout<1>::total(stages, bn, kernel_epi_vec, planes);
    {
      const RbStatus sst = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
      if (sst != RB_SUCCESS) return sst;
    }

    cudaLaunchConfig_t lc;
    memset(&lc, 0, sizeof(lc));
    lc.blockDim = dim3(kGemmThreads, 1, 1);
    lc.dynamicSmemBytes = (size_t)smem;
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    lc.attrs = attr;
    attr[lc.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[lc.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++lc.numAttrs;
    if (ctas == 2) {
      attr[lc.numAttrs].id = cudaLaunchAttributeClusterDimension;
      attr[lc.numAttrs].val.clusterDim.x = 2; attr[lc.numAttrs].val.clusterDim.y = 1; attr[lc.numAttrs].val.clusterDim.z = 1;
      ++lc.numAttrs;
      const int pairs = dev->sm_count / 2;
      lc.gridDim = dim3((unsigned)(2 * (int)std::min<long long>(num_items, pairs)), 1, 1);
    } else {
      lc.gridDim = dim3((unsigned)std::min<long long>(num_items, dev->sm_count), 1, 1);
    }
    if (capture) {
      static_assert(sizeof(GemmTensorMaps) + sizeof(GemmParams) + 64 <= sizeof(capture->params), "parameter block too small");
      memset(capture, 0, sizeof(*capture));
      const std::string sym = kernel_symbol(kind, kind == kKindTF32 ? false : a_mn, kind == kKindTF32 ? false : b_mn, ctas, tail);
      snprintf(capture->symbol, sizeof(capture->symbol), "%s", sym.c_str());
      capture->grid = lc.gridDim.x;
      capture->block = kGemmThreads;
      capture->cluster = (uint32_t)ctas;
      capture->dynamic_smem = (uint32_t)smem;
      capture->param_count = 2;
      capture->param_offset[0] = 0;
      capture->param_size[0] = (uint32_t)sizeof(GemmTensorMaps);
      capture->param_offset[1] = (uint32_t)((sizeof(GemmTensorMaps) + 63) / 64 * 64);
      capture->param_size[1] = (uint32_t)sizeof(GemmParams);
      kp.trace = nullptr;
      memcpy(capture->params + capture->param_offset[0], &maps, sizeof(maps));
      memcpy(capture->params + capture->param_offset[1], &kp, sizeof(kp));
      return RB_SUCCESS;
    }
    kp.trace = trace_buffer((size_t)lc.gridDim.x * 16);
    if (add_ranges && (half || !halves)) {
      const long long n4 = (long long)p->g * p->m * p->n / 4;
      cudaLaunchConfig_t zc;
      memset(&zc, 0, sizeof(zc));
      zc.gridDim = dim3((unsigned)std::min<long long>((n4 + 1023) / 1024, (long long)dev->sm_count * 4), 1, 1);
      zc.blockDim = dim3(256, 1, 1);
      zc.stream = stream;
      zc.attrs = attr;   // (the first is the programmatic launch)
      zc.numAttrs = 1;
      RB_CUDA_TRY(cudaLaunchKernelEx(&zc, zero_kernel, static_cast<float4*>(c), n4));
      count_launch();
    }
    RB_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, maps, kp));
    count_launch();
  }
  if (splits > 1 && !add_ranges) {
    const long long total = (long long)p->g * p->m * p->n;
    const bool vec = p->n % 4 == 0 && !p->trans_c && reinterpret_cast<uintptr_t>(c) % (4 * es_c) == 0;
    const long long threads = total / (vec ? 4 : 1);
    const int blocks = (int)std::min<long long>((threads + 127) / 128, (long long)dev->sm_count * 16);
    if (vec)
      RB_CUDA_TRY(launch_after(splitk_reduce_kernel<4>, blocks, 128, 0, stream, 1, partial, splits, total, p->g, p->m, p->n, c, p->c_type,
                               p->trans_c ? 1 : 0, is_int ? 1 : 0, ep));
    else
      RB_CUDA_TRY(launch_after(splitk_reduce_kernel<1>, blocks, 128, 0, stream, 1, partial, splits, total, p->g, p->m, p->n, c, p->c_type,
                               p->trans_c ? 1 : 0, is_int ? 1 : 0, ep));
    count_launch();
  }
  return RB_SUCCESS;
}

// ---- the kernels as a loadable binary --------------------------------------------------------------------------------
// The image is the cubin that nvcc makes of csrc/cubin/gemm_kernels.cu (every instantiation of gemm_tcgen05_kernel
// for sm_100a), linked into the library as data.
extern "C" const unsigned char rb_gemm_cubin_start[];
extern "C" const unsigned char rb_gemm_cubin_end[];

extern "C" RbStatus rbGetKernelBinary(const void** image, size_t* size) {
  if (!image && !size) return rb::fail(RB_INVALID_PARAM, "image and size are both NULL");
  if (image) *image = rb_gemm_cubin_start;
  if (size) *size = (size_t)(rb_gemm_cubin_end - rb_gemm_cubin_start);
  return RB_SUCCESS;
}

extern "C" RbStatus rbGemmEncodeLaunch(const RbGemmProblem* p, const RbEpilogue* epi, const void* a, const void* b, void* c,
                                       RbKernelLaunch* out) {
  if (!out) return rb::fail(RB_INVALID_PARAM, "out is NULL");
  return rb::gemm_run(p, epi, a, b, c, nullptr, 0, nullptr, nullptr, out);
}

// ---- rbGemmNoAlloc ------------------------------------------------------------------------------------
// Scratch for callers that may not allocate device memory: one fixed array inside the library image. Every GPU
// that loads the library carries it until the process exits; all calls share it.
namespace {
constexpr size_t kNoAllocScratchBytes = RB_NO_ALLOC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 16;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kNoAllocMaxDevices];   // nullptr until a lookup on that device has succeeded
}  // namespace

extern "C" RbStatus rbGemmNoAlloc(const RbGemmProblem* p, const RbEpilogue* epi, const void* a, const void* b, void* c,
                                  void* stream) {
  RbStatus st = rb::check_problem(p);
  if (st != RB_SUCCESS) return st;
  size_t need = rbGemmWorkspaceSize(p);
  if (need > kNoAllocScratchBytes) need = rb::gemm_workspace_bytes(p, -1, true);
  if (need > kNoAllocScratchBytes)
    return rb::fail(RB_WORKSPACE_TOO_SMALL,
                    "rbGemmNoAlloc: this problem needs " + std::to_string(need) + " bytes of scratch, the built-in "
                    "scratch holds " + std::to_string(kNoAllocScratchBytes) + "; use rbGemm with a caller workspace");
  int dev = 0;
  RB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return rb::fail(RB_CUDA_ERROR, "device index out of range");
  // In host code the array's name is only a handle for the runtime, not a device address: the address the kernels
  // get is looked up per device, with that device current. Only a successful lookup is remembered; a failed one
  // (for instance a first call made while a stream capture was open) is reported and tried again by the next call.
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
      void* ptr = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if (e != cudaSuccess || !ptr)
        return rb::fail(RB_CUDA_ERROR, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
      g_noalloc_ptr[dev] = ptr;
    }
    scratch = g_noalloc_ptr[dev];
  }
  return rbGemm(p, epi, a, b, c, need ? scratch : nullptr, need ? kNoAllocScratchBytes : 0, stream);
}

// ---- rbGemmGemm -------------------------------------------------------------------------------------------
// O = (A . B1) . B2 with the intermediate rounded to the element type: what rocMLIR's attention skeleton computes
// with the softmax removed (mlir/lib/Dialect/Rock/Transforms/GridwiseGemmToBlockwise.cpp:1790-1813, 2162-2165).
// With k1 and n2 at most 128 (the shapes of that skeleton) it runs on the attention kernel in one launch: S = A . B1
// in tensor memory, rounded to the element type in place, second product straight from there; no workspace. Larger
// inner extents do not fit the SM (O alone would be 128 x n2 f32 in TMEM): the intermediate (M x N1, element type)
// goes through the caller's workspace, small enough to stay in L2 - as one chained launch of the GEMM kernel when
// k1 = n1 = n2 (see below), else as two launches. Variant bit 27 forces the two-launch form.
// Flag words of the chained form: four per (128-row block, tile of columns), for tiles of 32 columns or more.
static size_t chain_flag_bytes(int m, int n1) {
  return rb::align_up((size_t)((m + 127) / 128) * ((n1 + 31) / 32) * 4 * sizeof(unsigned int), 256);
}

extern "C" size_t rbGemmGemmWorkspaceSize(int32_t g, int32_t m, int32_t k1, int32_t n1, int32_t n2, int32_t data_type) {
  if (g <= 0 || m <= 0 || k1 <= 0 || n1 <= 0 || n2 <= 0 || !rb::dtype_bytes(data_type)) return 0;
  // (the one-launch form needs none of it; the size is reported for the two-launch form so that a caller who sized
  // its buffer once can switch forms with the variant word)
  RbGemmProblem p1 = {g, m, n1, k1, 0, 0, 0, data_type, data_type, 0};
  RbGemmProblem p2 = {g, m, n2, n1, 0, 0, 0, data_type, data_type, 0};
  const size_t mid = rb::align_up((size_t)g * m * n1 * rb::dtype_bytes(data_type), 256);
  return mid + std::max(rbGemmWorkspaceSize(&p1), rbGemmWorkspaceSize(&p2)) + chain_flag_bytes(m, n1);
}

extern "C" RbStatus rbGemmGemm(int32_t g, int32_t m, int32_t k1, int32_t n1, int32_t n2, int32_t data_type,
                               const void* a, const void* b1, const void* b2, void* o, void* workspace,
                               size_t workspace_bytes, void* stream) {
  if (!(data_type == RB_F16 || data_type == RB_BF16 || data_type == RB_F32))
    return rb::fail(RB_UNSUPPORTED, "gemm+gemm exists for f16, bf16 and f32");
  const size_t need = rbGemmGemmWorkspaceSize(g, m, k1, n1, n2, data_type);
  if (need == 0) return rb::fail(RB_INVALID_PARAM, "sizes must be positive");
  if (rb::gemm_gemm_on_chip_applicable(k1, n1, n2, data_type) && !((rbGetGemmVariant() >> 27) & 1))
    return rb::gemm_gemm_on_chip(g, m, k1, n1, n2, data_type, a, b1, b2, o, stream);
  if (!workspace || workspace_bytes < need)
    return rb::fail(RB_WORKSPACE_TOO_SMALL, "workspace of " + std::to_string(need) + " bytes required");
  RbGemmProblem p1 = {g, m, n1, k1, 0, 0, 0, data_type, data_type, 0};
  RbGemmProblem p2 = {g, m, n2, n1, 0, 0, 0, data_type, data_type, 0};
  const size_t mid = rb::align_up((size_t)g * m * n1 * rb::dtype_bytes(data_type), 256);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  // Equal inner extents (k1 = n1 = n2), one group, 16-bit: ONE launch of the GEMM kernel over a two-group problem whose
  // second group reads the first group's result; the tiles of the second product start as soon as the row block of the
  // intermediate they read is complete, so there is no drain and refill between the products. Variant bit 27 keeps
  // the two-launch form; shapes or pointers the chained form does not take fall through to it.
  if (g == 1 && k1 == n1 && n1 == n2 && data_type != RB_F32 && !((rbGetGemmVariant() >> 27) & 1)) {
    const size_t fb = chain_flag_bytes(m, n1);
    RbGemmProblem pc = {2, m, n1, k1, 0, 0, 0, data_type, data_type, 0};
    rb::GemmChain ch = {b2, o, reinterpret_cast<unsigned int*>(ws + need - fb), fb};
    rb::t_chain = &ch;
    const RbStatus cst = rbGemm(&pc, nullptr, a, b1, ws, nullptr, 0, stream);
    rb::t_chain = nullptr;
    if (cst != RB_UNSUPPORTED) return cst;
  }
  RbStatus st = rbGemm(&p1, nullptr, a, b1, ws, ws + mid, workspace_bytes - mid, stream);
  if (st != RB_SUCCESS) return st;
  return rbGemm(&p2, nullptr, ws, b2, o, ws + mid, workspace_bytes - mid, stream);
}
