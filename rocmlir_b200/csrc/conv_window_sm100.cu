// Forward convolution of an image with few channels (16-bit types, one group) whose tensor-core operand is the input window itself.
//
// conv_patch_sm100.cu writes the 128 x K im2col tile of every 128 output pixels: each input element is gathered once per filter
// tap that reads it, and that gather bounds it (7 x 7 stride 2: 12 times). Here an input row is prepared once, and the tensor core
// reads it through descriptors, shifted, for every filter row (and, with five or more channels, every tap) that needs it:
//
//   * shared memory holds entries of 16 bytes, eight k values of one raster position; neighbouring positions lie 16 bytes apart.
//     That is a K-major operand without swizzle whose rows are 16 bytes apart: eight rows make a core matrix of 128
//     contiguous bytes (stride byte offset 128), and the second eight k values of an instruction lie wherever the leading
//     byte offset says. A k step is therefore any two entry columns of the window, each at its own start address. (68 cycles for
//     128 x 64 x 16 with sixteen warps at work beside it; the 128-byte-swizzled form measures 60 in the halo kernel.)
//   * runs (up to four channels): a filter row is a run of X * C elements; entry (h, q, j) holds elements 8 j .. 8 j + 7 of the run
//     that output column q reads in input row h, zeros past the run. Filter rows share it.
//   * pixels (five channels and more): entry (h, w, j) holds channels 8 j .. 8 j + 7 of pixel w, zeros past the last channel; filter
//     rows and taps share it. With a stride the pixels are kept by phase, w = stride * i + f, so that output columns are
//     neighbours again. Images channels last with whole groups of eight channels need no preparation: cp.async puts them there.
//   * input rows are kept by phase of the vertical stride too, so a tile's raster (R output rows of Wp positions) is contiguous for
//     every filter row. Rows of an instruction past the raster read whatever follows; their results are not stored.
//   * Bound: what the sixteen warps do for an item, one after the other: of 9360 cycles (with clocks read in between) for four tiles of 64 channels
//     3340 go into preparation, 3260 into stores, 1560 into copies and 990 into waits, beside 2980 of products. us, the gathering form before:
//     N = 64, 3 -> 64 channels, 224 x 224, 7 x 7 stride 2 100 -> 71; 30 x 7 -> 32 channels, 184 x 184, 7 x 7 stride 2 82 -> 25; 20 x 16 -> 32,
//     223 x 223, 3 x 3 116 -> 39; 109 x 8 -> 64, 62 x 62, 5 x 5 54 -> 31; 36 x 3 -> 32, 195 x 195, 3 x 3 stride 2 107 -> 19 (rows that start on any
//     even byte). Of 1000 convolutions
//     that the estimates in conv_patch_pays were not fitted to, they take a form more than 6 % slower than the fastest in 80, and 15 are
//     more than 5 % slower than without this kernel (the worst 14.2 -> 18.3 us).
//   * sixteen warps prepare item i + 1 and store item i - 1 while the seventeenth issues item i: two windows, two sets of
//     accumulators in tensor memory, the raw rows of the next item on their way by cp.async meanwhile.
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <string>

#include "conv_patch.cuh"
#include "lib_state.h"
#include "launch.cuh"

namespace rb {
namespace {

constexpr int kWorkers = 512;                  // threads that prepare and store
constexpr int kWindowThreads = kWorkers + 32;  // + the issuing warp
constexpr int kMaxChunks = 128;                // 16-byte columns of k
constexpr int kMaxPlanes = 32;                 // entry columns per input row
constexpr int kMaxPhases = 8;
constexpr int kWindowMaxC = 24;
constexpr int kWindowMaxNt = 128;
constexpr int kWindowSmem = 232448;
constexpr int kTableBytes = 32 * kMaxPlanes + 8 * kWindowMaxNt + 64;   // (see the kernel)
constexpr int kZeroBytes = 128 * 16;           // the second half of an odd last k step

// How an entry gets its eight values from the raw rows: as a run of elements at any even address (shifted words), at multiples of 4
// or 8 bytes, element by element through a table, or directly from the image by cp.async (no raw rows)
enum Fetch { kShifted, kWords, kPairs, kElements, kDirect };

struct WindowParams {
  const uint16_t* in;
  const uint16_t* fil;
  void* out;
  long long i_n, i_c, i_h;
  long long f_k;
  int f_c, f_y, f_x;
  long long o_n, o_k, o_p, o_q;
  int N, H, W, C, P, Q, X, Kout;
  int stride_h, stride_w, dil_w, pad_h, pad_w;
  int planar, unit;                 // elements per image column of a row: C, or 1 with channel planes
  int pixels;                       // entries of pixels, else of runs
  int R, Qt, tiles_p, tiles_q, num_items;
  int Wp, mtiles;                   // raster pitch of an item, 128-row tiles of it
  int planes, phases, rows_ph;      // window [planes][phases][rows_ph][Wp] entries
  int raw_planes, raw_rows, raw_pitch;         // raw rows, in elements
  int segs, tasks;                  // 32 entries of a row of the window: a warp's task
  int estep;                        // raw elements between neighbouring entries
  int chunks, mmas;
  int nt, passes;
  int win_off, zero_off, fil_off, raw_off, tab_off, task_off;   // shared memory, bytes from the aligned start
  int win_bytes;
  uint32_t idesc, tmem_cols;
  int is_bf16, out_type, wide;
  EpiParams epi;
  uint32_t* status;
  long long wait_cycles;
  short phase_row[kMaxPhases];      // input row of a phase's first entry row
  short plane_off[kMaxPlanes];      // first raw element of an entry, from its raster position on
  short plane_col[kMaxPlanes];      // pixels: phase of the column
  unsigned char plane_n[kMaxPlanes];   // valid values of an entry
  uint32_t steps[kMaxChunks / 2];      // k step: entry where its first half starts | distance to its second half << 16
  unsigned char chunk_y[kMaxChunks], chunk_x[kMaxChunks], chunk_j[kMaxChunks];   // filter row, tap (pixels) and group of eight of a k column
};

struct Item {
  int n, p0, q0;
  __device__ Item(const WindowParams& p, unsigned item) {
    const unsigned r = item / (unsigned)p.tiles_q;
    n = (int)(r / (unsigned)p.tiles_p);
    p0 = (int)(r - (unsigned)n * (unsigned)p.tiles_p) * p.R;
    q0 = (int)(item - r * (unsigned)p.tiles_q) * p.Qt;
  }
};

// Raw rows: the 16-byte granules of the image that hold them, each row where it lies inside its first granule, zeros outside the
// image row. A granule that begins before the image row brings what lies there; clear_row_heads takes that out again.
struct RawRow {
  long long at;     // element of the image where the window's row starts (may lie before the image row)
  int skew;         // its position inside its granule
  int e0;           // the same element, counted from the start of the image row
  bool ok;          // a row of the image
  __device__ RawRow(const WindowParams& p, const Item& t, int pr) {
    const int pl = p.raw_planes == 1 ? 0 : pr / p.raw_rows, h = t.p0 * p.stride_h - p.pad_h + pr - pl * p.raw_rows;
    e0 = (t.q0 * p.stride_w - p.pad_w) * p.unit;
    at = (long long)t.n * p.i_n + (long long)pl * p.i_c + (long long)h * p.i_h + e0;
    skew = (int)at & 7;
    ok = h >= 0 && h < p.H;
  }
};
__device__ __forceinline__ void load_raw(const WindowParams& p, const Item& t, uint32_t raw) {
  const int row_elems = p.W * p.unit, per_row = p.raw_pitch / 8, lane = threadIdx.x & 31;
  for (int pr = threadIdx.x >> 5; pr < p.raw_planes * p.raw_rows; pr += kWorkers / 32) {   // a warp per row
    const RawRow r(p, t, pr);
    const long long first = r.at - r.skew;
    const uint32_t dst = smem_u32(smem_raw) + raw + 2u * (uint32_t)(pr * p.raw_pitch);
    const int lo0 = r.e0 - r.skew;
#pragma unroll 4
    for (int v = lane; v < per_row; v += 32) {
      const int lo = lo0 + 8 * v;
      const int bytes = r.ok && lo > -8 ? max(0, min(16, 2 * (row_elems - lo))) : 0;
      cp_async(dst + 16u * (uint32_t)v, p.in + (bytes ? first + 8 * v : 0), 8, bytes);
    }
  }
}
// (by the lane that copied the granule, once its copies have arrived)
__device__ __forceinline__ void clear_row_heads(const WindowParams& p, const Item& t, uint32_t raw) {
  if (t.q0 * p.stride_w >= p.pad_w) return;   // what lies before the row is not part of the window
  for (int pr = threadIdx.x >> 5; pr < p.raw_planes * p.raw_rows; pr += kWorkers / 32) {
    const RawRow r(p, t, pr);
    const int head = r.skew - r.e0, v = head >> 3, n = head & 7;
    if (n && v < p.raw_pitch / 8 && (int)(threadIdx.x & 31) == (v & 31)) {
      uint16_t* d = reinterpret_cast<uint16_t*>(smem_raw + raw + 2u * (uint32_t)(pr * p.raw_pitch) + 16u * (uint32_t)v);
      for (int i = 0; i < n; ++i) d[i] = 0;
    }
  }
}

// Pixels of whole groups of eight channels, channels last on 16-byte boundaries: entries straight from the image.
__device__ __forceinline__ void load_direct(const WindowParams& p, const Item& t, uint32_t win) {
  const int rows = p.phases * p.rows_ph, h0 = t.p0 * p.stride_h - p.pad_h, w0 = t.q0 * p.stride_w - p.pad_w;
  for (int u = threadIdx.x >> 5; u < p.planes * rows; u += kWorkers / 32) {
    const int j = u / rows, r = u - j * rows, ph = r / p.rows_ph;
    const int h = h0 + p.phase_row[ph] + (r - ph * p.rows_ph) * p.stride_h;
    const bool row_ok = h >= 0 && h < p.H;
    const int f = p.plane_col[j];
    const long long row = (long long)t.n * p.i_n + (long long)h * p.i_h + (p.plane_off[j] - f * p.unit);
    for (int e = threadIdx.x & 31; e < p.Wp; e += 32) {
      const int w = w0 + e * p.stride_w + f;
      const bool ok = row_ok && w >= 0 && w < p.W;
      cp_async(smem_u32(smem_raw) + win + (uint32_t)(u * p.Wp + e) * 16u, p.in + (ok ? row + (long long)w * p.C : 0), 8, ok ? 16 : 0);
    }
  }
}

// One entry from the raw rows. a: shared-memory offset of its first element; n: its valid values (warp-uniform).
template <int FETCH>
__device__ __forceinline__ uint4 fetch8(uint32_t a, int n) {
  uint32_t w[4];
  if constexpr (FETCH == kShifted) {
    const uint32_t shift = (a & 2u) * 8u, b = a & ~3u;
    uint32_t r[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) r[i] = lds<uint32_t>(b + 4 * i);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(r[i], r[i + 1], shift);
  } else if constexpr (FETCH == kWords) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = lds<uint32_t>(a + 4 * i);
  } else {
    const uint2 x = lds<uint2>(a), y = lds<uint2>(a + 8);
    w[0] = x.x; w[1] = x.y; w[2] = y.x; w[3] = y.y;
  }
  if (n < 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] &= n >= 2 * i + 2 ? 0xffffffffu : n == 2 * i + 1 ? 0xffffu : 0u;
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// The same element by element: offs holds (byte offset << 3 | what the element's plane adds to the row's position in its granule).
__device__ __forceinline__ uint4 fetch8_elements(uint32_t a, uint32_t offs, int n, uint32_t skew) {
  const uint4 o0 = lds<uint4>(offs), o1 = lds<uint4>(offs + 16);
  const uint32_t o[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t lo = 0u, hi = 0u;
    if (2 * i < n) lo = lds<uint16_t>(a + (o[2 * i] >> 3) + 2u * ((skew + o[2 * i]) & 7u));
    if (2 * i + 1 < n) hi = lds<uint16_t>(a + (o[2 * i + 1] >> 3) + 2u * ((skew + o[2 * i + 1]) & 7u));
    w[i] = lo | (hi << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Entries of an item from its raw rows, a task of 32 at a time, several tasks in flight. A task: {offset of its first element in the
// raw rows, of its first entry in the window, valid values | entries << 8 | plane << 16, what its row adds to the position in a granule}.
template <int FETCH>
__device__ __forceinline__ void prepare(const WindowParams& p, const Item& t, uint32_t raw, uint32_t win, uint32_t tasks, uint32_t eoffs) {
  const int lane = threadIdx.x & 31;
  const uint32_t step = 2u * (uint32_t)(p.estep * lane);
  const uint32_t skew = (uint32_t)t.n * (uint32_t)p.i_n + (uint32_t)(t.p0 * p.stride_h - p.pad_h) * (uint32_t)p.i_h +
                        (uint32_t)((t.q0 * p.stride_w - p.pad_w) * p.unit);   // modulo 8
  constexpr int kFlight = FETCH == kElements ? 2 : 4;
  for (int k0 = threadIdx.x >> 5; k0 < p.tasks; k0 += kFlight * (kWorkers / 32)) {
    uint4 v[kFlight];
    uint32_t dst[kFlight];
#pragma unroll
    for (int i = 0; i < kFlight; ++i) {
      const int k = k0 + i * (kWorkers / 32);
      dst[i] = 0xffffffffu;
      v[i] = make_uint4(0u, 0u, 0u, 0u);
      if (k < p.tasks) {
        const uint4 task = lds<uint4>(tasks + 16u * (uint32_t)k);
        const int n = (int)(task.z & 0xffu);
        if (lane < (int)((task.z >> 8) & 0xffu)) {
          dst[i] = win + task.y + 16u * (uint32_t)lane;
          const uint32_t at = raw + task.x + step, sk = skew + task.w;
          if constexpr (FETCH == kElements) v[i] = fetch8_elements(at, eoffs + 32u * (task.z >> 16), n, sk);
          else v[i] = fetch8<FETCH>(at + 2u * (sk & 7u), n);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kFlight; ++i)
      if (dst[i] != 0xffffffffu) *reinterpret_cast<uint4*>(smem_raw + dst[i]) = v[i];
  }
}

// The result of an item: a unit is 32 channels of 32 raster positions of one quarter of a tile.
template <bool EPI>
__device__ __forceinline__ void store_item(const WindowParams& p, const Item& t, uint32_t tmem, int n0, const float* vec_scale,
                                           const float* vec_bias) {
  const int warp = threadIdx.x >> 5, quarter = warp & 3, lane = threadIdx.x & 31, groups = p.nt / 32;
  for (int u = warp >> 2; u < p.mtiles * groups; u += kWorkers / 128) {
    const int tile = u / groups, c = (u - tile * groups) * 32;
    const int ncols = min(32, p.Kout - n0 - c);
    if (ncols <= 0) continue;   // warp-uniform
    const unsigned m = (unsigned)(tile * 128 + quarter * 32 + lane), r = m / (unsigned)p.Wp, q = m - r * (unsigned)p.Wp;
    const bool valid = (int)r < p.R && t.p0 + (int)r < p.P && (int)q < p.Qt && t.q0 + (int)q < p.Q;
    const long long pix = (long long)t.n * p.o_n + (long long)(t.p0 + (int)r) * p.o_p + (long long)(t.q0 + (int)q) * p.o_q;
    store_pixel<EPI>(p, valid, pix, tmem + tile * p.nt + ((uint32_t)(quarter * 32) << 16) + c, n0 + c, ncols, vec_scale + c, vec_bias + c);
  }
}

template <int FETCH, bool EPI>
__global__ void __launch_bounds__(kWindowThreads, 1) conv_window_kernel(const __grid_constant__ WindowParams p) {
  const uint32_t base = (128u - (smem_u32(smem_raw) & 127u)) & 127u;   // aligned start inside the allocation
  const uint32_t win = base + p.win_off, fil = base + p.fil_off, raw = base + p.raw_off, tab = base + p.tab_off;
  // tables: [element offsets: 8 per plane][scale, bias][barriers][tensor-memory address]; [tasks]
  const uint32_t eoffs = tab, tasks = base + p.task_off;
  float* vec_scale = reinterpret_cast<float*>(smem_raw + eoffs + 32u * kMaxPlanes);
  float* vec_bias = vec_scale + kWindowMaxNt;
  uint64_t* full = reinterpret_cast<uint64_t*>(vec_bias + kWindowMaxNt);   // [2]: the window is prepared
  uint64_t* done = full + 2;                                               // [2]: its products are in tensor memory
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done + 2);

  const int warp = warp_id_uniform(), lane = threadIdx.x & 31;
  const bool worker = warp < kWorkers / 32;
  const int n0 = (int)(blockIdx.x % p.passes) * p.nt;
  const int step = (int)(gridDim.x / p.passes);
  const int first = (int)(blockIdx.x / p.passes);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full[i], kWorkers / 32);
      mbar_init(&done[i], 1);
    }
    fence_mbar_init();
  }
  if (warp == kWorkers / 32) {
    tmem_alloc<1>(tmem_holder, p.tmem_cols);
    tmem_relinquish<1>();
    for (int i = lane; i < kZeroBytes / 16; i += 32) *reinterpret_cast<uint4*>(smem_raw + base + p.zero_off + 16 * i) = make_uint4(0u, 0u, 0u, 0u);
  }
  if (worker) {   // (the grid has no more CTAs per pass than there are items)
    if constexpr (FETCH == kElements) {
      for (int i = threadIdx.x; i < p.planes * 8; i += kWorkers) {
        const int j = i / 8, t = i & 7;
        int c, x;   // channel plane and column of the value (x in image columns)
        if (p.pixels) { c = p.plane_off[j] + t; x = p.plane_col[j]; }
        else { const int r = 8 * j + t; x = r / p.C; c = r - x * p.C; x *= p.dil_w; }
        const int o = p.planar ? c * p.raw_rows * p.raw_pitch + x : x * p.C + c;
        const uint32_t add = p.planar ? (uint32_t)c * (uint32_t)p.i_c : 0u;
        *reinterpret_cast<uint32_t*>(smem_raw + eoffs + 4 * i) = t < p.plane_n[j] ? ((uint32_t)(2 * o) << 3) | (add & 7u) : 0u;
      }
    }
    if constexpr (FETCH != kDirect) {
      const int rows = p.phases * p.rows_ph;
      for (int k = threadIdx.x; k < p.tasks; k += kWorkers) {
        const int u = k / p.segs, seg = k - u * p.segs, j = u / rows, r = u - j * rows, ph = r / p.rows_ph;
        const int hr = p.phase_row[ph] + (r - ph * p.rows_ph) * p.stride_h;
        uint4 task;
        task.x = 2u * (uint32_t)(hr * p.raw_pitch + (FETCH == kElements ? 0 : p.plane_off[j]) + seg * 32 * p.estep);
        task.y = 16u * (uint32_t)(u * p.Wp + seg * 32);
        task.z = (uint32_t)p.plane_n[j] | ((uint32_t)min(32, p.Wp - seg * 32) << 8) | ((uint32_t)j << 16);
        task.w = (uint32_t)hr * (uint32_t)p.i_h;
        *reinterpret_cast<uint4*>(smem_raw + tasks + 16u * (uint32_t)k) = task;
      }
    }
    griddep_wait();   // nothing above touches what an earlier kernel of the stream reads or writes
    if constexpr (FETCH == kDirect) load_direct(p, Item(p, first), win);
    else load_raw(p, Item(p, first), raw);
    if constexpr (EPI) {
      for (int j = threadIdx.x; j < p.nt; j += kWorkers) {
        const int n = min(n0 + j, p.Kout - 1);
        vec_scale[j] = (p.epi.flags & RB_EPI_COL_SCALE) ? __ldg(p.epi.col_scale + n) : 1.0f;
        vec_bias[j] = epi_col_bias(p.epi.flags) ? load_bias(p.epi.bias, p.epi.bias_type, n) : 0.0f;
      }
    }
    // the filter, k column by k column: an entry per output channel, zeros past its extents
    for (int i = threadIdx.x; i < p.mmas * 2 * p.nt; i += kWorkers) {
      const int k = i / p.nt, n = i - k * p.nt;
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (k < p.chunks && n0 + n < p.Kout) {
        const uint16_t* f = p.fil + (long long)(n0 + n) * p.f_k + (long long)p.chunk_y[k] * p.f_y;
        const int j = p.chunk_j[k];
        int c = p.pixels ? 8 * j : (8 * j) % p.C, x = p.pixels ? p.chunk_x[k] : (8 * j) / p.C;
        const int left = p.pixels ? p.C - 8 * j : p.X * p.C - 8 * j;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (e < left) w[e / 2] |= (uint32_t)__ldg(f + (long long)c * p.f_c + (long long)x * p.f_x) << (16 * (e & 1));
          if (++c == p.C) { c = 0; ++x; }
        }
      }
      *reinterpret_cast<uint4*>(smem_raw + fil + 16u * (uint32_t)i) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t buf_cols = (uint32_t)(p.mtiles * p.nt);
  const uint32_t smem0 = smem_u32(smem_raw);

  if (!worker) {
    // ------------------------------ issuing warp ------------------------------
    // (all lanes run the loop, one elected lane issues: the descriptors stay warp-uniform)
    const bool leader = elect_one();
    const uint32_t hi = smem_desc_hi_plain(128), idesc = p.idesc;
    const uint32_t b0 = smem_desc_lo(smem0 + fil, 16u * (uint32_t)p.nt), b_step = 2u * (uint32_t)p.nt;
    const uint32_t zero = (smem0 + base + p.zero_off) >> 4, win16 = (smem0 + win) >> 4, win_step = (uint32_t)p.win_bytes >> 4;
    const int whole = p.chunks / 2, num_items = p.num_items, mtiles = p.mtiles, nt = p.nt;
    const bool odd = (p.chunks & 1) != 0;
    uint32_t t = 0;
    for (int item = first; item < num_items; item += step, ++t) {
      if (!mbar_wait_warp(&full[t & 1u], (t >> 1) & 1u, p.status, kStatusTimeoutMma, p.wait_cycles)) break;
      tc_fence_after();
      uint32_t a16 = win16 + (t & 1u) * win_step, d = tmem_base + (t & 1u) * buf_cols;
      for (int tile = 0; tile < mtiles; ++tile, a16 += 128u, d += (uint32_t)nt) {
        uint32_t b = b0;
#pragma unroll 4
        for (int i = 0; i < whole; ++i, b += b_step) {
          const uint32_t a = p.steps[i] + a16;
          if (leader) umma_ss<kKindF16, 1>(d, desc64(a, hi), desc64(b, hi), idesc, i ? 1u : 0u);
        }
        if (odd) {
          const uint32_t a = (p.steps[whole] + a16) & 0x3FFFu;
          if (leader) umma_ss<kKindF16, 1>(d, desc64(a | ((zero - a) << 16), hi), desc64(b, hi), idesc, whole ? 1u : 0u);
        }
      }
      if (leader) tc_commit<1>(&done[t & 1u]);
    }
  } else {
    // ------------------------------ preparing and storing warps ------------------------------
    bool ok = true;   // after a wait ran out the loop goes on without work or waits: the warps meet in every step
    uint32_t t = 0;
    Item cur(p, first), prev = cur;
    for (int item = first; item < p.num_items; item += step, ++t) {
      const uint32_t w = win + (t & 1u) * (uint32_t)p.win_bytes;
      cp_async_wait_all();
      if constexpr (FETCH != kDirect) {
        clear_row_heads(p, cur, raw);
        named_barrier(1, kWorkers);   // every thread's copies are there
        prepare<FETCH>(p, cur, raw, w, tasks, eoffs);   // (the products of item t - 2 have read this window: they were stored a step ago)
      }
      fence_proxy_async();
      tc_fence_before();   // this warp's reads of the accumulators that are about to be overwritten
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[t & 1u]);
      const bool more = item + step < p.num_items;
      const Item next(p, (unsigned)(more ? item + step : item));
      if constexpr (FETCH != kDirect) {
        named_barrier(1, kWorkers);   // the raw rows have been read
        if (more) load_raw(p, next, raw);
      }
      if (t > 0) {
        if (ok) ok = mbar_wait_warp(&done[(t - 1u) & 1u], ((t - 1u) >> 1) & 1u, p.status, kStatusTimeoutEpilogue, p.wait_cycles);
        // (every warp copies only after its own wait: the products of item t - 1 have read the window)
        if (FETCH == kDirect && more && ok) load_direct(p, next, win + ((t + 1u) & 1u) * (uint32_t)p.win_bytes);
        tc_fence_after();
        if (ok) store_item<EPI>(p, prev, tmem_base + ((t - 1u) & 1u) * buf_cols, n0, vec_scale, vec_bias);
      } else if (FETCH == kDirect && more) {
        load_direct(p, next, win + (uint32_t)p.win_bytes);
      }
      prev = cur;
      cur = next;
    }
    griddep_launch();   // the last load is under way
    cp_async_wait_all();
    if (t > 0 && ok && mbar_wait_warp(&done[(t - 1u) & 1u], ((t - 1u) >> 1) & 1u, p.status, kStatusTimeoutEpilogue, p.wait_cycles)) {
      tc_fence_after();
      store_item<EPI>(p, prev, tmem_base + ((t - 1u) & 1u) * buf_cols, n0, vec_scale, vec_bias);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kWorkers / 32) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, p.tmem_cols);
  }
}

struct WindowShape {
  bool pixels;
  int fetch;
  int planes, phases, rows_ph, col_phases, groups;   // groups: entries per pixel or run
  int halo, raw_rows, raw_span;                      // entry columns beyond Qt; raw elements of a row beyond the entries' step
  int chunks, mmas, nt, passes;
  int R, Qt, Wp, mtiles;
  int segs, tasks;
  int raw_pitch, win_bytes, smem;
  int max_ctas;
  double store_cycles, tensor_cycles;   // of a tile of 128 raster positions
  double us;   // estimated time
};

// What does not depend on the tile (rows_ph and raw_rows without the tile's rows).
bool window_operand(const PatchConv& c, WindowShape* s) {
  if (c.stride_h > kMaxPhases || c.stride_w > kMaxPhases || c.Y > 32 || c.X > 32 || c.C > kWindowMaxC) return false;
  const int unit = c.planar ? 1 : c.C;
  // runs waste the last entry of a filter row, pixels the last entry of a pixel
  s->pixels = c.C > 4;
  if (s->pixels) {
    int phases = 0;
    for (int f = 0; f < c.stride_w; ++f) {
      bool used = false;
      for (int x = 0; x < c.X; ++x) used = used || (x * c.dil_w) % c.stride_w == f;
      phases += used;
    }
    s->col_phases = phases;
    s->groups = (c.C + 7) / 8;
    s->planes = phases * s->groups;
    s->halo = (c.X - 1) * c.dil_w / c.stride_w;
    s->chunks = c.Y * c.X * s->groups;
    s->raw_span = (c.stride_w - 1) * unit + (c.planar ? 1 : c.C);
  } else {
    s->col_phases = 1;
    s->groups = (c.X * c.C + 7) / 8;
    s->planes = s->groups;
    s->halo = 0;
    s->chunks = c.Y * s->groups;
    s->raw_span = ((c.X - 1) * c.dil_w + 1) * unit;
  }
  if (s->planes > kMaxPlanes || s->chunks > kMaxChunks || s->halo > 1024 || s->raw_span > (1 << 15)) return false;
  s->passes = (c.Kout + kWindowMaxNt - 1) / kWindowMaxNt;
  s->nt = ((c.Kout + s->passes - 1) / s->passes + 31) / 32 * 32;
  if (s->passes > 8 || (long long)s->nt * (s->passes - 1) >= c.Kout) return false;   // (no pass without channels)
  s->mmas = (s->chunks + 1) / 2;
  s->max_ctas = std::max(1, planning_sm_count() / s->passes);
  s->store_cycles = 4.0 * (s->nt / 32) * 130 * (c.o_k == 1 && c.Kout % 32 == 0 ? 1 : 1.6);
  s->tensor_cycles = (double)s->mmas * (4096 + 32 * s->nt) / 90.0;
  s->phases = 0;
  int last_row = 0;
  for (int f = 0; f < c.stride_h; ++f) {
    bool used = false;
    for (int y = 0; y < c.Y; ++y) used = used || (y * c.dil_h) % c.stride_h == f;
    if (used) { ++s->phases; last_row = f; }
  }
  s->rows_ph = (c.Y - 1) * c.dil_h / c.stride_h;
  s->raw_rows = last_row + 1 - c.stride_h;
  const int whole = c.i_h % 8 == 0 && c.i_n % 8 == 0 ? 8 : c.i_h % 4 == 0 && c.i_n % 4 == 0 ? 4 : c.i_h % 2 == 0 && c.i_n % 2 == 0 ? 2 : 1;
  if (s->pixels && !c.planar && c.C % 8 == 0 && whole == 8) s->fetch = kDirect;
  else if (c.planar || (!s->pixels && c.dil_w != 1)) s->fetch = kElements;
  else s->fetch = c.C % 4 == 0 && whole >= 4 ? kPairs : c.C % 2 == 0 && whole >= 2 ? kWords : kShifted;
  return true;
}

// The kernel on tiles of R x Qt output pixels: whether it fits, and an estimate of its time: the longer of an item's two sides, the
// products and what the sixteen warps do meanwhile, times the items of a CTA. (A tile that cannot be faster than `limit` microseconds by the
// products and stores alone is not looked at further: most of a search ends there, and its 1 us is a tenth of a small call.)
bool window_tile(const PatchConv& c, const WindowShape& operand, int Qt, int R, double limit, WindowShape* out) {
  const unsigned mtiles = (unsigned)(R * (Qt + operand.halo) + 127) / 128;
  const unsigned items = (unsigned)c.N * ((unsigned)(c.P + R - 1) / (unsigned)R) * ((unsigned)(c.Q + Qt - 1) / (unsigned)Qt);   // (at most N x P x Q < 2^30)
  const unsigned ctas = std::min(items, (unsigned)operand.max_ctas);
  const double per_cta = (double)((items + ctas - 1) / ctas);
  const double store = mtiles * operand.store_cycles, tensor = mtiles * operand.tensor_cycles + 250;
  if (4.5 + per_cta * std::max(tensor, store / 1.2 + 1200) / 1900 >= limit) return false;
  WindowShape s = operand;
  const int unit = c.planar ? 1 : c.C, raw_planes = c.planar ? c.C : 1;
  s.Qt = Qt;
  s.R = R;
  s.Wp = Qt + s.halo;
  s.mtiles = (int)mtiles;
  s.rows_ph += R;
  s.raw_rows += s.rows_ph * c.stride_h;
  const long long entries = (long long)s.planes * s.phases * s.rows_ph * s.Wp;
  if (2 * s.mtiles * s.nt > 512 || entries > 0x3fff || (long long)s.raw_rows * raw_planes > 4096) return false;
  s.win_bytes = (int)entries * 16;
  s.segs = (s.Wp + 31) / 32;
  s.tasks = s.fetch == kDirect ? 0 : s.planes * s.phases * s.rows_ph * s.segs;
  if (s.tasks > 2048) return false;
  s.raw_pitch = (7 + (s.Wp - 1) * c.stride_w * unit + s.raw_span + 10 + 7) / 8 * 8;
  const long long raw = s.fetch == kDirect ? 0 : 2LL * raw_planes * s.raw_rows * s.raw_pitch;
  // the products of a raster's last rows read up to 127 + halo entries past the second window
  const long long total = 128 + 2LL * s.win_bytes + kZeroBytes + 32LL * s.mmas * s.nt + kTableBytes + 16LL * s.tasks + std::max(raw, 16LL * (128 + s.halo));
  if (total > kWindowSmem) return false;
  s.smem = (int)total;
  const double lanes = (double)s.planes * s.phases * s.rows_ph * s.segs;   // warp steps of the preparation
  const double prep = lanes * (s.fetch == kDirect ? 14 : s.fetch == kElements ? 44 : s.fetch == kShifted ? 26 : 18) +
                      (s.fetch == kDirect ? 0.0 : (double)raw_planes * s.raw_rows * (30 + s.raw_pitch / 256.0 * 16));
  const double item = std::max(tensor, (prep + store) / 1.2 + 1200);
  s.us = 4.5 + (s.fetch == kElements ? 1.0 : 0.0) + (per_cta * item + tensor + 6.0 * s.mmas * s.nt) / 1900;   // + the filter
  *out = s;
  return true;
}

// The fastest tile by that estimate among a few: columns cut evenly, as many rows as one to all of the accumulators hold.
bool window_shape(const PatchConv& c, WindowShape* best) {
  WindowShape s, t;
  memset(&s, 0, sizeof(s));
  if (!window_operand(c, &s)) return false;
  bool found = false;
  const int max_tiles = 256 / s.nt;
  for (int cols = (c.Q + 255) / 256, tries = 0; cols <= c.Q && tries < 6; ++cols, ++tries) {
    const int Qt = (c.Q + cols - 1) / cols;
    if (tries && Qt < 8) break;
    for (int tiles = max_tiles, last = 0; tiles >= 1; --tiles) {
      const int R = std::min(c.P, tiles * 128 / (Qt + s.halo));
      if (R < 1) break;
      if (R == last) continue;   // (a low image: the same tile again)
      last = R;
      if (window_tile(c, s, Qt, R, found ? best->us : 1e30, &t) && (!found || t.us < best->us)) { *best = t; found = true; }
    }
  }
  return found;
}

// The kernel's time with that tile, for the choice between kernels. (The estimate above ranks the tiles of one convolution; between
// convolutions it was up to five times too low: it knew nothing of what results off 32 bytes, element by element, and filters by channel planes
// cost, and rows of single channels by element.) Cycles fitted to 1500 convolutions.
double window_time(const PatchConv& c, const WindowShape& s) {
  static const double kEntries[] = {23, 14, 14, 65, 46};   // of 32 entries, by Fetch
  const double columns = std::min(c.Kout, s.nt), units = 4.0 * s.mtiles, fill = s.R * s.Qt / (128.0 * s.mtiles);
  const double prep = (double)s.planes * s.phases * s.rows_ph * s.segs * kEntries[s.fetch] +
                      (s.fetch == kDirect ? 0.0 : 58.0 * (c.planar ? c.C : 1) * s.raw_rows);
  const double store = units * (c.o_k != 1 ? 5.2 * columns : c.Kout % 16 ? 62 * fill * columns : 99 * std::floor(columns / 32) + 62 * fill * (c.Kout % 32));
  const double tensor = (double)s.mtiles * s.mmas * (4096 + 32 * s.nt) / 75.0 + 250, entries = (double)s.mmas * s.nt;
  // a filter whose channels are not neighbours comes element by element, from L2 once it no longer fits what is left of the L1
  const double filter = c.f_c == 1 ? 5.8 * entries : 7.0 * entries + 26 * std::max(0.0, entries - 3000);
  const double items = (double)c.N * ((c.P + s.R - 1) / s.R) * ((c.Q + s.Qt - 1) / s.Qt);
  const double ctas = std::min(items, (double)s.max_ctas);
  return 4.0 + (std::ceil(items / ctas) * std::max(tensor, prep + store + 1820) + tensor + filter) / 1900;
}

}  // namespace

double conv_window_plan(PatchConv* c) {
  WindowShape s;
  c->win_q = c->win_r = 0;
  if (!window_shape(*c, &s)) return -1.0;
  c->win_q = s.Qt;
  c->win_r = s.R;
  return window_time(*c, s);
}

RbStatus conv_window_run(const PatchConv& c, const void* image, const void* filter, void* out, int out_type, const RbEpilogue* epi,
                         void* stream_v) {
  const DeviceInfo* dev = device_info();
  if (!dev) return RB_CUDA_ERROR;
  const bool with_epi = (epi && epi->flags) || out_type != (c.is_bf16 ? RB_BF16 : RB_F16);
  WindowShape s;
  memset(&s, 0, sizeof(s));
  // (raw rows are copied by the image's 16-byte granules)
  if (c.win_q <= 0 || reinterpret_cast<uintptr_t>(image) % 16 || !window_operand(c, &s) || !window_tile(c, s, c.win_q, c.win_r, 1e30, &s))
    return fail(RB_UNSUPPORTED, "convolution outside the reach of the window kernel");
  WindowParams p;
  memset(&p, 0, sizeof(p));
  p.in = static_cast<const uint16_t*>(image);
  p.fil = static_cast<const uint16_t*>(filter);
  p.out = out;
  p.i_n = c.i_n; p.i_c = c.planar ? c.i_c : 0; p.i_h = c.i_h;
  p.f_k = c.f_k; p.f_c = (int)c.f_c; p.f_y = (int)c.f_y; p.f_x = (int)c.f_x;
  p.o_n = c.o_n; p.o_k = c.o_k; p.o_p = c.o_p; p.o_q = c.o_q;
  p.N = c.N; p.H = c.H; p.W = c.W; p.C = c.C; p.P = c.P; p.Q = c.Q; p.X = c.X; p.Kout = c.Kout;
  p.stride_h = c.stride_h; p.stride_w = c.stride_w; p.dil_w = c.dil_w; p.pad_h = c.pad_h; p.pad_w = c.pad_w;
  p.planar = c.planar ? 1 : 0;
  p.unit = c.planar ? 1 : c.C;
  p.pixels = s.pixels ? 1 : 0;
  p.R = s.R; p.Qt = s.Qt; p.tiles_p = (c.P + s.R - 1) / s.R; p.tiles_q = (c.Q + s.Qt - 1) / s.Qt;
  p.num_items = c.N * p.tiles_p * p.tiles_q;
  p.Wp = s.Wp; p.mtiles = s.mtiles;
  p.planes = s.planes; p.phases = s.phases; p.rows_ph = s.rows_ph;
  p.raw_planes = c.planar ? c.C : 1; p.raw_rows = s.raw_rows; p.raw_pitch = s.raw_pitch;
  p.estep = c.stride_w * p.unit;
  p.segs = s.segs; p.tasks = s.tasks;
  p.chunks = s.chunks; p.mmas = s.mmas;
  p.nt = s.nt; p.passes = s.passes;
  int nph = 0, row_phase[kMaxPhases] = {}, ncol = 0, col_phase[kMaxPhases] = {};
  for (int f = 0; f < c.stride_h; ++f)
    for (int y = 0; y < c.Y; ++y)
      if ((y * c.dil_h) % c.stride_h == f) { row_phase[f] = nph; p.phase_row[nph++] = (short)f; break; }
  if (s.pixels) {
    for (int f = 0; f < c.stride_w; ++f) {
      bool used = false;
      for (int x = 0; x < c.X; ++x) used = used || (x * c.dil_w) % c.stride_w == f;
      if (!used) continue;
      col_phase[f] = ncol++;
      for (int j = 0; j < s.groups; ++j) {
        const int pl = col_phase[f] * s.groups + j;
        p.plane_off[pl] = (short)(s.fetch == kElements ? 8 * j : f * p.unit + 8 * j);
        p.plane_col[pl] = (short)f;
        p.plane_n[pl] = (unsigned char)std::min(8, c.C - 8 * j);
      }
    }
  } else {
    for (int j = 0; j < s.groups; ++j) {
      p.plane_off[j] = (short)(8 * j);
      p.plane_n[j] = (unsigned char)std::min(8, c.X * c.C - 8 * j);
    }
  }
  // the columns of k in the order of their addresses: the second half of a step lies behind the first
  struct Column { int at, y, x, j; };
  Column cols[kMaxChunks];
  int n = 0;
  for (int y = 0; y < c.Y; ++y)
    for (int x = 0; x < (s.pixels ? c.X : 1); ++x)
      for (int j = 0; j < s.groups; ++j) {
        const int yd = y * c.dil_h, xd = x * c.dil_w;
        const int pl = s.pixels ? col_phase[xd % c.stride_w] * s.groups + j : j;
        cols[n++] = {((pl * s.phases + row_phase[yd % c.stride_h]) * s.rows_ph + yd / c.stride_h) * s.Wp + (s.pixels ? xd / c.stride_w : 0), y, x, j};
      }
  std::sort(cols, cols + n, [](const Column& a, const Column& b) { return a.at < b.at; });
  for (int i = 0; i < n; ++i) {
    if (i % 2 == 0) p.steps[i / 2] = (uint32_t)cols[i].at | (i + 1 < n ? (uint32_t)(cols[i + 1].at - cols[i].at) << 16 : 0u);
    p.chunk_y[i] = (unsigned char)cols[i].y; p.chunk_x[i] = (unsigned char)cols[i].x; p.chunk_j[i] = (unsigned char)cols[i].j;
  }
  p.win_bytes = s.win_bytes;
  p.win_off = 0;
  p.zero_off = 2 * s.win_bytes;
  p.fil_off = p.zero_off + kZeroBytes;
  p.tab_off = p.fil_off + 32 * s.mmas * s.nt;
  p.task_off = p.tab_off + kTableBytes;
  p.raw_off = p.task_off + 16 * s.tasks;
  const uint32_t fmt = c.is_bf16 ? 1u : 0u;
  p.idesc = make_idesc(1, fmt, fmt, 0, 0, 128, (uint32_t)s.nt);
  p.tmem_cols = 32;
  while ((int)p.tmem_cols < 2 * s.mtiles * s.nt) p.tmem_cols *= 2;
  p.is_bf16 = c.is_bf16;
  p.out_type = out_type;
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
  typedef void (*Kernel)(const WindowParams);
  static const Kernel kernels[5][2] = {{conv_window_kernel<kShifted, false>, conv_window_kernel<kShifted, true>},
                                       {conv_window_kernel<kWords, false>, conv_window_kernel<kWords, true>},
                                       {conv_window_kernel<kPairs, false>, conv_window_kernel<kPairs, true>},
                                       {conv_window_kernel<kElements, false>, conv_window_kernel<kElements, true>},
                                       {conv_window_kernel<kDirect, false>, conv_window_kernel<kDirect, true>}};
  const Kernel kern = kernels[s.fetch][with_epi ? 1 : 0];
  RbStatus st = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), s.smem);
  if (st != RB_SUCCESS) return st;
  const long long per_pass = std::max<long long>(1, dev->sm_count / s.passes);
  const int grid = (int)std::min<long long>((long long)p.num_items, per_pass) * s.passes;
  RB_CUDA_TRY(launch_after(kern, grid, kWindowThreads, s.smem, static_cast<cudaStream_t>(stream_v), 1, p));
  count_launch();
  return RB_SUCCESS;
}

}  // namespace rb
