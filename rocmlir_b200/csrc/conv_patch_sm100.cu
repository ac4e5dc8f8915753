// Forward convolution of an image with few channels (16-bit types, one group): the im2col tile is built by the SM itself.
//
// rocMLIR's implicit GEMM (ConvRewritePattern, mlir/lib/Dialect/Rock/Transforms/ConvToGemm.cpp:1133-1400) reads the image
// through its pad -> embed -> merge coordinate map element by element, whatever the channel count. The TMA forms of this
// library (conv_halo_sm100.cu, the im2col loads of gemm_sm100.cuh) move whole 128-byte runs of channels, so an image whose
// pixel is not a multiple of 128 bytes - the first layer of every image network has three channels - used to be
// expanded into an im2col matrix in memory: Y * X copies of the image written, read, padded to 16-byte rows and read
// again. This kernel keeps that matrix on the chip:
//
//   * a tile is R x Qt output pixels of one image (at most 128), whose input window - a few KB - is copied once into
//     shared memory by cp.async, zeros outside the image, one tile ahead of its use;
//   * the 128 x K operand is gathered from the window into 128-byte-swizzled K-major blocks. A warp owns 32 pixels, a
//     step is the same eight k values for all of them, so the offsets are warp-uniform and the reads of neighbouring
//     pixels fall into different banks. Runs of 2, 4 or 8 channels are read as one word; a filter row of an odd channel
//     count is a contiguous run of the window as well (7 x 3 elements), and where padding k to whole steps per run costs
//     little, eight of its elements are five aligned words and a shift;
//   * the filter stays in shared memory in the same form for all tiles of the persistent CTA, tcgen05.mma accumulates
//     into one of two TMEM buffers, and the previous tile's result is stored while the tensor core works.
//
// (Images of up to 24 channels that start on 16 bytes take conv_window_sm100.cu where its estimate is the lower one.)
//
// Bound: the gather (one 2-byte read per element of the operand for three channels), then HBM writes of the result. Two
// CTAs per SM overlap one's gather with the other's stores and waits. N = 64, 3 -> 64 channels, 224 x 224, 7 x 7 stride 2,
// f16 channels last: 1826 us through the im2col matrix, 102 here. (152 with 64-bit tile arithmetic and element reads: the kernel
// issued 9600 warp instructions per tile, which ncu showed as its limit. 384 threads instead of 256: 111 us.)
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <numeric>
#include <string>

#include "conv_patch.cuh"
#include "lib_state.h"
#include "launch.cuh"

namespace rb {
namespace {

constexpr int kPatchThreads = 256;
constexpr int kABlockBytes = 128 * 128;   // 128 pixels x 64 k values
constexpr int kMaxNt = 128;               // output channels per CTA: two TMEM buffers of two CTAs fit 512 columns

struct PatchParams {
  const uint16_t* in;
  const uint16_t* fil;
  void* out;
  long long i_n, i_c, i_h;          // image strides in elements; a row is (w, c) contiguous, or w contiguous (planar)
  long long f_k;                    // filter strides in elements
  int f_c, f_y, f_x;
  long long o_n, o_k, o_p, o_q;     // result strides in elements
  int N, H, W, C, P, Q, Y, X, Kout;
  int stride_h, stride_w, dil_h, dil_w, pad_h, pad_w;
  int planar;                       // 0: channels last, k = (y, x, c); 1: channel planes, k = (c, y, x)
  int unit;                         // elements per image column of a row: C, or 1 when planar
  int R, Qt, tiles_p, tiles_q;      // tile raster
  int num_tiles;
  int rows, planes, pitch;          // window: planes x rows x pitch elements
  int gran;                         // elements per window copy: 8, 4 or 2 (cp.async), 1 = plain loads
  int run, run_pad;                 // k is runs of `run` elements, each padded to run_pad; run_pad == run: k is dense
  int kelems, ksteps, kblocks;      // k extent (padding included), MMA steps of 16, blocks of 64
  int nbuf;                         // blocks of the operand in shared memory
  int nt, passes;                   // output channels per CTA and CTAs groups that share a tile
  uint32_t idesc, tmem_cols;
  int is_bf16, out_type;
  int wide;                         // plain result, channels contiguous: 32-byte stores
  EpiParams epi;
  uint32_t* status;
  long long wait_cycles;
};

struct PatchTile {
  int n, p0, q0;
  __device__ PatchTile(const PatchParams& p, unsigned tile) {   // 32-bit: a 64-bit division is two hundred instructions
    const unsigned r = tile / (unsigned)p.tiles_q;
    n = (int)(r / (unsigned)p.tiles_p);
    p0 = (int)(r - (unsigned)n * (unsigned)p.tiles_p) * p.R;
    q0 = (int)(tile - r * (unsigned)p.tiles_q) * p.Qt;
  }
  // position of the window's first column inside its copy granule: the copy starts on a granule of the image row
  __device__ int skew(const PatchParams& p) const { return ((q0 * p.stride_w - p.pad_w) * p.unit) & (p.gran - 1); }
};

// Copies the input window of `tile` into `win` ([planes][rows][pitch]), zeros outside the image.
__device__ __forceinline__ void load_window(const PatchParams& p, const PatchTile& t, uint16_t* win) {
  const int e0 = (t.q0 * p.stride_w - p.pad_w) * p.unit;   // first element of the window inside its image row
  const int lo0 = e0 - t.skew(p);                          // a multiple of the copy granule
  const int h0 = t.p0 * p.stride_h - p.pad_h;
  const int row_elems = p.W * p.unit;
  const int gran = p.gran, per_row = p.pitch / gran;
  const uint16_t* img = p.in + (long long)t.n * p.i_n;
  // a warp per window row: consecutive lanes copy consecutive granules
  for (int pr = threadIdx.x >> 5; pr < p.planes * p.rows; pr += kPatchThreads / 32) {
    const int pl = p.planes == 1 ? 0 : pr / p.rows, h = h0 + pr - pl * p.rows;
    const bool row_ok = h >= 0 && h < p.H;
    const uint16_t* row = img + (long long)pl * p.i_c + (long long)h * p.i_h;
    uint16_t* dst = win + pr * p.pitch;
    for (int v = threadIdx.x & 31; v < per_row; v += 32) {
      const int lo = lo0 + v * gran;
      const int valid = (row_ok && lo >= 0) ? min(gran, max(0, row_elems - lo)) : 0;
      const uint16_t* src = valid > 0 ? row + lo : p.in;
      if (gran > 1) cp_async(smem_u32(dst + v * gran), src, gran, 2 * valid);
      else dst[v] = valid > 0 ? __ldg(src) : (uint16_t)0;
    }
  }
}

// Eight k values of one pixel from the window (`px`: where the pixel lies in shared memory; `offs`: where the step's eight
// entries of the offset table lie), in runs of VEC elements at warp-uniform offsets. VEC = 0: all eight lie in one run from entry 0 on,
// and entries 4 to 7 mask what is padding (it must be zero whatever the window holds there). The instruction count of this
// function is what bounds the kernel.
template <int VEC>
__device__ __forceinline__ uint4 gather8(uint32_t px, uint32_t offs, int left) {
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  if constexpr (VEC == 0) {
    const uint4 mask = lds<uint4>(offs + 16);
    const uint32_t a = px + lds<uint32_t>(offs), shift = (a & 2u) * 8u;
    const uint32_t b = a & ~3u;
    uint32_t r[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) r[i] = lds<uint32_t>(b + 4 * i);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(r[i], r[i + 1], shift);
    w[0] &= mask.x; w[1] &= mask.y; w[2] &= mask.z; w[3] &= mask.w;
  } else if constexpr (VEC == 1) {
    const uint4 x = lds<uint4>(offs), y = lds<uint4>(offs + 16);
    const uint32_t o[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    if (left >= 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = (uint32_t)lds<uint16_t>(px + o[2 * i]) | ((uint32_t)lds<uint16_t>(px + o[2 * i + 1]) << 16);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < left) w[i / 2] |= (uint32_t)lds<uint16_t>(px + o[i]) << (16 * (i & 1));
    }
  } else if constexpr (VEC == 2) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (2 * i < left) w[i] = lds<uint32_t>(px + lds<uint32_t>(offs + 8 * i));
  } else if constexpr (VEC == 4) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (4 * i < left) {
        const uint2 u = lds<uint2>(px + lds<uint32_t>(offs + 16 * i));
        w[2 * i] = u.x; w[2 * i + 1] = u.y;
      }
  } else {
    if (left > 0) return lds<uint4>(px + lds<uint32_t>(offs));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <bool EPI>
__device__ __forceinline__ void store_tile(const PatchParams& p, const PatchTile& t, int rr, int qq, uint32_t taddr, int n0,
                                           const float* vec_scale, const float* vec_bias) {
  const int warp = threadIdx.x >> 5;
  const bool valid = rr < p.R && t.p0 + rr < p.P && t.q0 + qq < p.Q;
  const long long pix = (long long)t.n * p.o_n + (long long)(t.p0 + rr) * p.o_p + (long long)(t.q0 + qq) * p.o_q;
  for (int c = (warp >> 2) * 32; c < p.nt; c += 64) {
    const int ncols = min(32, p.Kout - n0 - c);
    if (ncols <= 0) break;   // warp-uniform
    store_pixel<EPI>(p, valid, pix, taddr + ((uint32_t)((warp & 3) * 32) << 16) + c, n0 + c, ncols, vec_scale + c, vec_bias + c);
  }
}

template <int VEC, bool EPI>
__global__ void __launch_bounds__(kPatchThreads, 2)
conv_patch_kernel(const PatchParams p) {
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // [operand blocks][filter blocks][two windows][k offsets][per-channel vectors][barrier, TMEM address]
  uint8_t* a_smem = smem;
  uint8_t* b_smem = a_smem + p.nbuf * kABlockBytes;
  uint16_t* win = reinterpret_cast<uint16_t*>(b_smem + (size_t)p.kblocks * p.nt * 128);
  const int win_elems = p.planes * p.rows * p.pitch;
  int* offs = reinterpret_cast<int*>(win + 2 * win_elems);
  float* vec_scale = reinterpret_cast<float*>(offs + p.ksteps * 16);
  float* vec_bias = vec_scale + p.nt;
  uint64_t* bar = reinterpret_cast<uint64_t*>(vec_bias + p.nt);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bar + 1);

  const int warp = warp_id_uniform(), lane = threadIdx.x & 31;
  const int n0 = (int)(blockIdx.x % p.passes) * p.nt;
  const int step = (int)(gridDim.x / p.passes);
  int tile = (int)(blockIdx.x / p.passes);

  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc<1>(tmem_holder, p.tmem_cols);
    tmem_relinquish<1>();
  }
  griddep_wait();   // nothing above touches what an earlier kernel of the stream reads or writes
  load_window(p, PatchTile(p, tile), win);   // (the grid has no more CTAs per pass than there are tiles)
  // offsets of every k inside a window, and (in the operand area, which is not in use yet) inside a filter row
  int* foffs = reinterpret_cast<int*>(a_smem);
  for (int k = threadIdx.x; k < p.ksteps * 16; k += kPatchThreads) {
    const int nrun = k / p.run_pad, in_run = k - nrun * p.run_pad;
    const int kk = nrun * p.run + in_run;        // position in the dense order (y, x, c), or (c, y, x) when planar
    int c, y, x;
    if (p.planar) { x = kk % p.X; const int r = kk / p.X; y = r % p.Y; c = r / p.Y; }
    else { c = kk % p.C; const int r = kk / p.C; x = r % p.X; y = r / p.X; }
    const bool ok = k < p.kelems && in_run < p.run;
    int o = !ok ? 0 : p.planar ? (c * p.rows + y * p.dil_h) * p.pitch + x * p.dil_w : y * p.dil_h * p.pitch + x * p.dil_w * p.C + c;
    foffs[k] = ok ? c * p.f_c + y * p.f_y + x * p.f_x : -1;
    o *= 2;
    if (VEC == 0 && (k & 4)) {   // valid halves of word (k & 3) of the step
      const int first = (k & ~7) + 2 * (k & 3), left = (k & ~7) < p.kelems ? p.run - (in_run - (k & 7)) - (first - (k & ~7)) : 0;
      o = left >= 2 ? -1 : left == 1 ? 0xffff : 0;
    }
    offs[k] = o;
  }
  if constexpr (EPI) {
    for (int j = threadIdx.x; j < p.nt; j += kPatchThreads) {
      const int n = min(n0 + j, p.Kout - 1);
      vec_scale[j] = (p.epi.flags & RB_EPI_COL_SCALE) ? __ldg(p.epi.col_scale + n) : 1.0f;
      vec_bias[j] = epi_col_bias(p.epi.flags) ? load_bias(p.epi.bias, p.epi.bias_type, n) : 0.0f;
    }
  }
  __syncthreads();
  // the filter: row = output channel, 16-byte pieces swizzled like a TMA load would leave them, zeros past its extents
  {
    const int pieces = p.kblocks * 8, have = p.ksteps * 2;
    for (int i = threadIdx.x; i < p.nt * pieces; i += kPatchThreads) {
      const int j = i % pieces, n = i / pieces;
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (j < have && n0 + n < p.Kout) {
        const uint16_t* f = p.fil + (long long)(n0 + n) * p.f_k;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (foffs[8 * j + e] >= 0) w[e / 2] |= (uint32_t)__ldg(f + foffs[8 * j + e]) << (16 * (e & 1));
      }
      *reinterpret_cast<uint4*>(b_smem + (size_t)(j >> 3) * p.nt * 128 + n * 128 + (((j & 7) ^ (n & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  // this thread's pixel (operand row), the same for every tile: rows past the tile's pixels repeat pixel 0
  const int m = (warp & 3) * 32 + lane;
  const int rr = m / p.Qt, qq = m - rr * p.Qt;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t px = smem_u32(win) - raw + 2u * (uint32_t)(rr < p.R ? rr * p.stride_h * p.pitch + qq * p.stride_w * p.unit : 0);
  const uint32_t a_row = smem_u32(a_smem) - raw + m * 128, a_swz = (uint32_t)(m & 7) << 4, offs_at = smem_u32(offs) - raw;
  const uint32_t a_lo0 = smem_desc_lo(smem_u32(a_smem), 16), b_lo0 = smem_desc_lo(smem_u32(b_smem), 16);
  const uint32_t desc_hi = smem_desc_hi(1024);

  bool ok = true;
  uint32_t groups = 0;       // operand groups handed to the tensor core so far: phase of the barrier
  uint32_t t = 0;
  PatchTile cur(p, tile), prev = cur;
  for (; tile < p.num_tiles; tile += step, ++t) {
    const uint32_t tmem_d = tmem_base + (t & 1u) * p.nt;
    cp_async_wait_all();
    const uint32_t w = px + 2u * ((t & 1u) * (uint32_t)win_elems + (uint32_t)cur.skew(p));
    for (int kb0 = 0; kb0 < p.kblocks; kb0 += p.nbuf) {
      // the MMAs of the previous group have read the operand blocks (and, at a tile's start, finished the last tile)
      if (groups > 0) ok = mbar_wait_warp(bar, (groups - 1) & 1u, p.status, kStatusTimeoutMma, p.wait_cycles);
      if (!__syncthreads_and(ok)) { ok = false; break; }
      const int steps = min(p.nbuf * 4, p.ksteps - kb0 * 4);   // MMA steps of this group
      for (int j0 = warp >> 2; j0 < steps * 2; j0 += 8) {   // four steps in flight: all their reads before the first write
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = kb0 * 64 + (j0 + 2 * u) * 8;
          if (j0 + 2 * u < steps * 2) v[u] = gather8<VEC>(w, offs_at + 4 * k, p.kelems - k);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + 2 * u;
          if (j < steps * 2)
            *reinterpret_cast<uint4*>(smem_raw + a_row + (j >> 3) * kABlockBytes + (((uint32_t)(j & 7) << 4) ^ a_swz)) = v[u];
        }
      }
      fence_proxy_async();
      tc_fence_before();   // this thread's TMEM reads of the buffer that is about to be overwritten
      __syncthreads();
      if (threadIdx.x == 0) {
        tc_fence_after();
        for (int s = 0; s < steps; ++s) {
          const uint32_t blk = (uint32_t)s >> 2, in = ((uint32_t)s & 3u) * 2u;
          umma_ss<kKindF16, 1>(tmem_d, desc64(a_lo0 + blk * (kABlockBytes >> 4) + in, desc_hi),
                               desc64(b_lo0 + (kb0 + blk) * (uint32_t)(p.nt * 8) + in, desc_hi), p.idesc, (kb0 | s) ? 1u : 0u);
        }
        tc_commit<1>(bar);
      }
      ++groups;
    }
    if (!ok) break;
    const PatchTile next(p, tile + step < p.num_tiles ? tile + step : tile);
    if (tile + step < p.num_tiles) load_window(p, next, win + ((t + 1) & 1u) * win_elems);
    if (t > 0) {   // the previous tile's result, while the tensor core works on this one
      tc_fence_after();
      store_tile<EPI>(p, prev, rr, qq, tmem_base + ((t - 1) & 1u) * p.nt, n0, vec_scale, vec_bias);
    }
    prev = cur;
    cur = next;
  }
  griddep_launch();   // the last load is under way
  cp_async_wait_all();
  if (ok && t > 0) {
    ok = mbar_wait(bar, (groups - 1) & 1u, p.status, kStatusTimeoutEpilogue, p.wait_cycles);
    if (__syncthreads_and(ok)) {
      tc_fence_after();
      store_tile<EPI>(p, prev, rr, qq, tmem_base + ((t - 1) & 1u) * p.nt, n0, vec_scale, vec_bias);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, p.tmem_cols);
  }
}

struct PatchShape {
  int R, Qt, rows, planes, pitch, nbuf, nt, passes, ctas_per_sm, smem;
  int run, run_pad, kelems;
};

// Tile, operand blocks and output channels per CTA that fit. Fewest passes over the output channels first (each pass
// gathers the operand again), then two CTAs per SM before one.
bool choose_shape(const PatchConv& c, PatchShape* s) {
  // contiguous runs of the window: a filter row over all channels (one channel plane when planar). Padding them to steps of
  // eight is worth a fifth more k (7 x 7 x 3: 168 instead of 147); words of two or more channels need no padding.
  s->run = c.planar ? c.X : c.X * c.C;
  s->run_pad = (s->run + 7) / 8 * 8;
  if (c.dil_w != 1 || s->run_pad * 5 > s->run * 6 || (!c.planar && c.C % 2 == 0)) s->run_pad = s->run;
  s->kelems = c.Y * c.X * c.C / s->run * s->run_pad;
  const int kelems = s->kelems, kblocks = (kelems + 63) / 64, ksteps = (kelems + 15) / 16;
  const int unit = c.planar ? 1 : c.C;
  s->planes = c.planar ? c.C : 1;
  const int cols = (c.Q + 127) / 128;
  s->Qt = (c.Q + cols - 1) / cols;
  for (int passes = (c.Kout + kMaxNt - 1) / kMaxNt; passes <= 4; ++passes) {
    s->passes = passes;
    s->nt = ((c.Kout + passes - 1) / passes + 31) / 32 * 32;
    if ((long long)s->nt * (passes - 1) >= c.Kout) continue;   // a pass without channels
    for (s->ctas_per_sm = 2; s->ctas_per_sm >= 1; --s->ctas_per_sm) {
      const int limit = s->ctas_per_sm == 2 ? 115712 - 1024 : 232448;
      for (s->R = std::min(128 / s->Qt, c.P); s->R >= 1; s->R /= 2) {
        s->rows = (s->R - 1) * c.stride_h + (c.Y - 1) * c.dil_h + 1;
        s->pitch = ((((s->Qt - 1) * c.stride_w + (c.X - 1) * c.dil_w + 1) * unit + 7) + 7) / 8 * 8;
        const long long fixed = (long long)kblocks * s->nt * 128 + 4LL * s->planes * s->rows * s->pitch + ksteps * 64LL + s->nt * 8LL + 64 + 1024;
        for (s->nbuf = std::min(kblocks, 4); s->nbuf >= std::min(kblocks, 2); --s->nbuf) {
          // (the operand area also holds the filter offsets while the filter is loaded)
          if (fixed + (long long)s->nbuf * kABlockBytes <= limit && ksteps * 64LL <= (long long)s->nbuf * kABlockBytes) {
            s->smem = (int)(fixed + (long long)s->nbuf * kABlockBytes);
            return true;
          }
        }
      }
    }
  }
  return false;
}

// Runs of channels that can be read as one word (channels last: k walks the channels of a tap); 0: padded runs, by single elements.
int gather_run(const PatchConv& c, const PatchShape& s) {
  return s.run_pad != s.run ? 0 : c.planar ? 1 : c.C % 8 == 0 ? 8 : c.C % 4 == 0 ? 4 : c.C % 2 == 0 ? 2 : 1;
}

}  // namespace

// Device times of the forms in microseconds, replayed graphs. The product of an im2col matrix: fitted to 396 convolutions (1 to 384 channels, 16 to
// 512 output channels, 7 x 7 to 224 x 224, filters 1, 3, 5, 7, strides 1 and 2, both layouts, 5 to 2500 us), 9 % off on average. This kernel and
// the window kernel: fitted to 1900 of 1 to 96 channels and 1 to 256 output channels, strides to 4, images of 5 x 5 to 224 x 300, 11 and 8 % off.
// A tile gathers 128 x k elements however few pixels it has, once per group of 128 output channels, copies a window, by single elements where
// image rows start on any even byte, and every CTA brings the filter over element by element first; so taking this kernel
// wherever it fits made a third of the convolutions slower, a pointwise layer of 512 -> 512 channels (64 channels-first images of 7 x 7) 32 -> 497 us:
//   64 x 224 x 224 x 3 -> 64, 7 x 7 stride 2: 102 us here, 1830 there;  32 x 28 x 28 x 24 -> 64, 3 x 3: 13.5 / 16.4
//   16 x 14 x 14 x 96 -> 192, 3 x 3: 64 / 16;  channels first 32 x 28 x 28 x 128 -> 128, 3 x 3 stride 2: 299 / 75
// An image off 16 bytes can not take the window kernel and goes by the other two estimates (*off16: whether to this kernel).
bool conv_patch_pays(PatchConv* conv, bool wide_gather, bool result_direct, int out_bytes, bool* off16) {
  const PatchConv& c = *conv;
  *off16 = false;
  PatchShape s;
  if (!choose_shape(c, &s)) return false;
  const double sms = planning_sm_count(), pixels = 1e-6 * c.N * c.P * c.Q, k = (double)c.Y * c.X * c.C;
  const double tiles = (double)c.N * ((c.P + s.R - 1) / s.R) * ((c.Q + s.Qt - 1) / s.Qt), rows = (double)s.planes * s.rows;
  const double ctas = std::min(tiles, std::floor(sms * s.ctas_per_sm / s.passes));
  const double on_one_sm = std::min<double>(s.ctas_per_sm, std::max(1.0, ctas * s.passes / sms));   // they share its issue slots
  // result: whole groups of 32 columns (in the last group of a row, all columns where rows are off 32 bytes, or in channel planes one by one)
  const double columns = std::min(c.Kout, s.nt), fill = std::min(1.0, s.R * s.Qt / 128.0);
  const double one_by_one = c.o_k != 1 ? 0.004 * columns : fill * ((c.Kout * out_bytes) % 32 ? 0.124 * columns : 0.093 * (c.Kout % 32));
  const long long starts = (long long)c.W * (c.planar ? 1 : c.C) | c.i_h | c.i_n | (c.planar ? c.i_c : 0);
  const double row = starts % 4 == 0 ? 0.033 + 8e-5 * s.pitch : starts % 2 == 0 ? 0.030 + 2.1e-4 * s.pitch : 0.025 + 8.6e-4 * s.pitch;
  // pixels of a warp that fall into the same banks: `ways` of the lanes that shared memory serves at a time
  const int word = 2 * gather_run(c, s) < 4 ? 4 : 2 * gather_run(c, s), step = c.stride_w * (c.planar ? 1 : c.C) * 2;
  const double ways = (128.0 / word) / std::min(128.0 / word, std::max(1.0, 128.0 / std::gcd(step, 128)));
  const double tile = 0.225 + 0.0047 * s.kelems * (1 + 0.07 * (ways - 1)) + 0.0077 * std::max(0, s.kelems - 400) + 0.0047 * s.nt + rows * row + one_by_one;
  const double here = 4.4 + on_one_sm * (std::ceil(tiles / ctas) * tile + 0.0140 * s.nt * ((s.kelems + 63) / 64));
  // im2col matrix (a vector or an element per thread), its rows padded to 16 bytes, product (rows of it off 16 bytes are copied out),
  // permutation of the result
  double there = 8.1 + pixels * (117 + 2 * k * (wide_gather ? 0.386 : 3.42)) + 0.0039 * pixels * std::max(c.Kout, 64) * k + 0.0042 * k;
  if ((c.Y * c.X * c.C) % 8 != 0) there += 1.3 + pixels * 2 * k * 0.364;
  if (!result_direct) there += 4.1 + pixels * 2 * c.Kout * 1.56;
  if ((c.Kout * out_bytes) % 16) there += 2.6 + pixels * (54 + 2.0 * c.Kout);
  const int variant = rbGetGemmVariant();
  const double window = ((variant >> 10) & 1) ? -1.0 : conv_window_plan(conv);
  if (window < 0 || (((variant >> 30) & 1) == 0 && window > 0.95 * here)) conv->win_q = 0;
  *off16 = here * 1.05 < there;
  return (conv->win_q ? std::min(here, window) : here) * 1.05 < there;
}

bool conv_patch_applicable(const PatchConv& c) {
  // offsets inside the window, the filter and an image row are 32-bit
  if (c.dil_h > 4096 || c.dil_w > 4096 || c.stride_h > 4096 || c.stride_w > 4096 || c.Y > 4096 || c.X > 4096) return false;
  if ((long long)c.N * c.P * c.Q >= (1LL << 30)) return false;
  const long long row = ((long long)c.W + c.pad_w + c.pad_w_r) * (c.planar ? 1 : c.C);
  const long long kelems = (long long)c.Y * c.X * c.C;
  if (kelems > 4096 || row >= (1LL << 30) || (long long)c.H + c.pad_h + c.pad_h_r >= (1LL << 30)) return false;
  if (c.f_c * c.C + c.f_y * c.Y + c.f_x * c.X >= (1LL << 30)) return false;
  const long long win_cols = ((std::min(c.Q, 128) - 1LL) * c.stride_w + (c.X - 1LL) * c.dil_w + 1) * (c.planar ? 1 : c.C);
  const long long win_rows = 127LL * c.stride_h + (c.Y - 1LL) * c.dil_h + 1;
  if (win_cols > (1 << 20) || win_rows > (1 << 20)) return false;
  PatchShape s;
  return choose_shape(c, &s);
}

RbStatus conv_patch_run(const PatchConv& c, const void* image, const void* filter, void* out, int out_type, const RbEpilogue* epi,
                        void* stream_v) {
  // the kernel takes its tensors element by element where they lie off wider boundaries, but not off those of an element
  if ((reinterpret_cast<uintptr_t>(image) | reinterpret_cast<uintptr_t>(filter)) % 2 || reinterpret_cast<uintptr_t>(out) % dtype_bytes(out_type))
    return fail(RB_UNSUPPORTED, "tensors must start on a multiple of their element size");
  if (c.win_q > 0 && reinterpret_cast<uintptr_t>(image) % 16 == 0) return conv_window_run(c, image, filter, out, out_type, epi, stream_v);
  const DeviceInfo* dev = device_info();
  if (!dev) return RB_CUDA_ERROR;
  PatchShape s;
  if (!conv_patch_applicable(c) || !choose_shape(c, &s)) return fail(RB_UNSUPPORTED, "convolution outside the reach of the patch kernel");
  PatchParams p;
  memset(&p, 0, sizeof(p));
  p.in = static_cast<const uint16_t*>(image);
  p.fil = static_cast<const uint16_t*>(filter);
  p.out = out;
  p.i_n = c.i_n; p.i_c = c.planar ? c.i_c : 0; p.i_h = c.i_h;
  p.f_k = c.f_k; p.f_c = (int)c.f_c; p.f_y = (int)c.f_y; p.f_x = (int)c.f_x;
  p.o_n = c.o_n; p.o_k = c.o_k; p.o_p = c.o_p; p.o_q = c.o_q;
  p.N = c.N; p.H = c.H; p.W = c.W; p.C = c.C; p.P = c.P; p.Q = c.Q; p.Y = c.Y; p.X = c.X; p.Kout = c.Kout;
  p.stride_h = c.stride_h; p.stride_w = c.stride_w; p.dil_h = c.dil_h; p.dil_w = c.dil_w; p.pad_h = c.pad_h; p.pad_w = c.pad_w;
  p.planar = c.planar ? 1 : 0;
  p.unit = c.planar ? 1 : c.C;
  p.R = s.R; p.Qt = s.Qt; p.rows = s.rows; p.planes = s.planes; p.pitch = s.pitch;
  p.tiles_p = (c.P + s.R - 1) / s.R; p.tiles_q = (c.Q + s.Qt - 1) / s.Qt;
  p.num_tiles = c.N * p.tiles_p * p.tiles_q;
  // the widest copy that every image row starts on: rows, images and the base address at multiples of it
  p.gran = 8;
  while (p.gran > 1 && (((long long)c.W * p.unit) % p.gran || c.i_h % p.gran || c.i_n % p.gran || p.i_c % p.gran ||
                        reinterpret_cast<uintptr_t>(image) % (2 * p.gran)))
    p.gran /= 2;
  p.run = s.run; p.run_pad = s.run_pad;
  p.kelems = s.kelems; p.ksteps = (p.kelems + 15) / 16; p.kblocks = (p.kelems + 63) / 64;
  p.nbuf = s.nbuf; p.nt = s.nt; p.passes = s.passes;
  const uint32_t fmt = c.is_bf16 ? 1u : 0u;
  p.idesc = make_idesc(1, fmt, fmt, 0, 0, 128, (uint32_t)s.nt);
  p.tmem_cols = 32;
  while ((int)p.tmem_cols < 2 * s.nt) p.tmem_cols *= 2;
  p.is_bf16 = c.is_bf16;
  p.out_type = out_type;
  const bool with_epi = (epi && epi->flags) || out_type != (c.is_bf16 ? RB_BF16 : RB_F16);
  const long long wide_bytes = with_epi ? 16 : 32, es_o = (long long)dtype_bytes(out_type);
  p.wide = c.o_k == 1 && reinterpret_cast<uintptr_t>(out) % wide_bytes == 0 && (c.o_n * es_o) % wide_bytes == 0 &&
           (c.o_p * es_o) % wide_bytes == 0 && (c.o_q * es_o) % wide_bytes == 0;
  if (epi && epi->flags) {
    p.epi.flags = epi->flags; p.epi.alpha = epi->alpha; p.epi.out_recip = epi->out_recip; p.epi.mid_type = epi->mid_type;
    p.epi.bias_type = epi->bias_type; p.epi.col_scale = epi->col_scale; p.epi.bias = epi->bias;
    p.epi.clip_lo = epi->clip_lo; p.epi.clip_hi = epi->clip_hi; p.epi.in_zero = epi->in_zero;
    p.epi.out_zero = (epi->flags & RB_EPI_ZP_OUT) ? epi->out_zero : 0;
    p.epi.residual = epi->residual; p.epi.res_type = epi->res_type;
    p.epi.unary = (epi->flags & RB_EPI_UNARY) ? epi->unary : 0;
  }
  p.status = dev->status_word;
  p.wait_cycles = kWaitCycles;
  const int vec = gather_run(c, s);
  typedef void (*Kernel)(const PatchParams);
  const Kernel kern = with_epi ? (vec == 8 ? conv_patch_kernel<8, true> : vec == 4 ? conv_patch_kernel<4, true>
                                  : vec == 2 ? conv_patch_kernel<2, true> : vec == 1 ? conv_patch_kernel<1, true> : conv_patch_kernel<0, true>)
                               : (vec == 8 ? conv_patch_kernel<8, false> : vec == 4 ? conv_patch_kernel<4, false>
                                  : vec == 2 ? conv_patch_kernel<2, false> : vec == 1 ? conv_patch_kernel<1, false> : conv_patch_kernel<0, false>);
  RbStatus st = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), s.smem);
  if (st != RB_SUCCESS) return st;
  const long long per_pass = std::max<long long>(1, (long long)dev->sm_count * s.ctas_per_sm / s.passes);
  const int grid = (int)std::min<long long>((long long)p.num_tiles, per_pass) * s.passes;
  RB_CUDA_TRY(launch_after(kern, grid, kPatchThreads, s.smem, static_cast<cudaStream_t>(stream_v), 1, p));
  count_launch();
  return RB_SUCCESS;
}

}  // namespace rb
