// GEMM with few rows (the tokens of a generation step against a weight matrix stored out x in): C^T = B . A^T.
//
// The general kernel (gemm_sm100.cuh) makes the rows of A the 128 rows of the tensor-core tile, so with eight tokens 15
// of 16 rows of every A tile are zeros that are written to shared memory and multiplied, its tiles are 256 columns wide
// (16 for a 4096-wide layer), and filling the GPU takes a K split whose f32 planes a second launch adds up. Here the
// weights are the 128-row operand and the tokens, padded to 16, 32 or 64, the narrow one:
//   * a K block is 16 KB of weights and 2 to 8 KB of tokens, a tile is 128 output columns, two CTAs share an SM;
//   * the CTAs of a cluster divide a tile's K blocks and add their accumulators through distributed shared memory, in
//     rank order, so the result is deterministic and there is no plane in memory and no second launch;
//   * a thread of the epilogue owns an output column: its bias and scale are one load each.
// Bound: reading the weights once from HBM, and below about 10 us the launch itself. 8 x 4096 x 4096 f16 with bias: 18.4 us a call
// through the general kernel and its reduction, 9.8 here (32 MB of weights need 5.1 from HBM). Where the line to the general
// kernel lies: gemm_skinny_applicable. 64 rows are the widest operand the two CTAs of an SM have room for.
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <string>

#include "epilogue.cuh"
#include "gemm_skinny.h"
#include "lib_state.h"
#include "ptx.cuh"

namespace rb {
namespace {

constexpr int kSkinnyThreads = 192;    // producer, MMA issuer (and TMEM), four epilogue warps
constexpr int kTileN = 128;            // output columns (weight rows) per tile
constexpr int kWBytes = kTileN * 128;  // one K block of weights: 128 rows of 128 bytes
constexpr int kSkinnyMaxStages = 8;
constexpr int kSkinnyMaxSplits = 8;    // portable cluster size

struct SkinnyMaps {
  CUtensorMap w, x;   // weights [g][N][K], tokens [g][M][K]; boxes of 128 bytes x 128 (nt) rows
};

struct SkinnyParams {
  int M, N, G;
  int nt;                  // tokens padded to 16, 32 or 64: columns of the accumulator
  int kblocks, splits, tiles_n, stages;
  uint32_t idesc, tmem_cols;
  int acc_is_int;
  void* c;
  int c_type;
  EpiParams epi;
  uint32_t* status;
  long long wait_cycles;
  int stall;
};

__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

template <int KIND>
__global__ void __launch_bounds__(kSkinnyThreads, 2)
gemm_skinny_kernel(const __grid_constant__ SkinnyMaps maps, const SkinnyParams p) {
  constexpr int BKE = KIND == kKindF16 ? 64 : 128;   // K elements per block
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = kWBytes + p.nt * 128;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* empty_bar = full_bar + kSkinnyMaxStages;
  uint64_t* done_bar = empty_bar + kSkinnyMaxStages;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done_bar + 1);

  const int warp = threadIdx.x >> 5, lane = lane_id();
  const int splits = p.splits;
  const int part = splits > 1 ? (int)cluster_ctarank() : 0;
  const int tile = blockIdx.x / splits;
  const int g = tile / p.tiles_n, n0 = (tile - g * p.tiles_n) * kTileN;
  // an even share of the K blocks: every part has at least one
  const int kb0 = (int)((long long)p.kblocks * part / splits), kb1 = (int)((long long)p.kblocks * (part + 1) / splits);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    fence_mbar_init();
    prefetch_tmap(&maps.w);
    prefetch_tmap(&maps.x);
  }
  if (warp == 1) {
    tmem_alloc<1>(tmem_holder, p.tmem_cols);
    tmem_relinquish<1>();
    griddep_launch();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  griddep_wait();   // nothing above touches what an earlier kernel of the stream reads or writes

  uint32_t* part_smem = reinterpret_cast<uint32_t*>(smem);   // [nt][128] accumulators of this part, after the main loop
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      uint32_t s = 0, ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[s], ph ^ 1u, p.status, kStatusTimeoutProducer + s, p.wait_cycles)) break;
        if (!p.stall) {   // (rbInjectStall: the stage is never filled)
          uint8_t* sw = smem + s * stage_bytes;
          mbar_expect_tx(&full_bar[s], (uint32_t)stage_bytes);
          tma_load_3d(sw, &maps.w, &full_bar[s], kb * BKE, n0, g);
          tma_load_3d(sw + kWBytes, &maps.x, &full_bar[s], kb * BKE, 0, g);
        }
        if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t s = 0, ph = 0;
      const uint32_t hi = smem_desc_hi(1024);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full_bar[s], ph, p.status, kStatusTimeoutMma + s, p.wait_cycles)) { ok = false; break; }
        const uint32_t a = smem_desc_lo(smem_u32(smem + s * stage_bytes), 16), b = a + (kWBytes >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)   // 32 bytes of K per MMA
          umma_ss<KIND, 1>(tmem_base, desc64(a + 2 * k, hi), desc64(b + 2 * k, hi), p.idesc, (kb > kb0 || k) ? 1u : 0u);
        tc_commit<1>(&empty_bar[s]);
        if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
      }
      if (ok) tc_commit<1>(done_bar);
    }
  } else {
    const int q = warp & 3;                 // TMEM lanes 32 q .. 32 q + 31 = output columns of this warp
    const int col = q * 32 + lane, n = n0 + col;
    if (mbar_wait_warp(done_bar, 0, p.status, kStatusTimeoutEpilogue, p.wait_cycles)) {
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
      for (int m0 = 0; m0 < p.nt; m0 += 16) {
        if (m0 >= p.M) break;
        uint32_t v[16];
        tmem_ld16(taddr + m0, v);
        tmem_ld_wait();
        if (splits > 1) {   // the ring is idle: every MMA has completed
#pragma unroll
          for (int j = 0; j < 16; ++j) part_smem[(m0 + j) * kTileN + col] = v[j];
        } else if (n < p.N) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (m0 + j < p.M) {
              const long long o = ((long long)g * p.M + m0 + j) * p.N + n;
              if (p.acc_is_int && p.c_type == RB_I32 && p.epi.flags == 0) {
                static_cast<uint32_t*>(p.c)[o] = v[j];
              } else {
                float x = p.acc_is_int ? __int2float_rn((int)v[j]) : __uint_as_float(v[j]);
                if (p.epi.flags) x = epi_apply(x, p.epi, n, m0 + j, o);
                store_elem(p.c, o, x, p.c_type, p.epi.out_zero);
              }
            }
          }
        }
      }
    }
  }
  if (splits > 1) {
    cluster_sync();
    // token m is added up by the CTA m mod splits, thread = output column, parts in rank order
    for (int i = threadIdx.x; i < kTileN * ((p.M - part + splits - 1) / splits); i += kSkinnyThreads) {
      const int m = part + i / kTileN * splits, col = i % kTileN, n = n0 + col;
      const uint32_t addr = smem_u32(part_smem + m * kTileN + col);
      uint32_t v[kSkinnyMaxSplits];
#pragma unroll
      for (int s = 0; s < kSkinnyMaxSplits; ++s)
        if (s < splits) v[s] = ld_cluster_u32(mapa_u32(addr, s));
      uint32_t acc = 0u;
#pragma unroll
      for (int s = 0; s < kSkinnyMaxSplits; ++s)
        if (s < splits) acc = p.acc_is_int ? acc + v[s] : __float_as_uint(__fadd_rn(__uint_as_float(acc), __uint_as_float(v[s])));
      if (n < p.N) {
        const long long o = ((long long)g * p.M + m) * p.N + n;
        if (p.acc_is_int && p.c_type == RB_I32 && p.epi.flags == 0) {
          static_cast<uint32_t*>(p.c)[o] = acc;
        } else {
          float x = p.acc_is_int ? __int2float_rn((int)acc) : __uint_as_float(acc);
          if (p.epi.flags) x = epi_apply(x, p.epi, n, m, o);
          store_elem(p.c, o, x, p.c_type, p.epi.out_zero);
        }
      }
    }
    cluster_sync();   // nobody leaves while its shared memory is being read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, p.tmem_cols);
  }
}

}  // namespace

namespace {
// Parts of K: as many CTAs as fit two to an SM, at least four K blocks each (a part's fixed cost is about that of streaming
// four blocks).
int skinny_splits(const RbGemmProblem* p, long long tiles, int kblocks, int sms) {
  return (int)std::max<long long>(1, std::min<long long>({(long long)kSkinnyMaxSplits, 2LL * sms / tiles, (long long)kblocks / 4}));
}
}  // namespace

// Which of the two kernels takes a product with few rows. Here an output column is one thread's, so a row costs every CTA
// about 0.15 us (0.05 where i32 sums are stored as they are) divided by the parts of K, while the general kernel stores a
// tile of any height in about a microsecond (twice that where rows of C do not start on 16-byte boundaries), but needs a second launch
// when it divides K. Measured, us here / there, device time of repeated calls, f16:
//   parts of K   (16..64) x 4096 x 4096: 9.6..12.1 / 14.7..16.2;  64 x 1024 x 1024: 8.9 / 8.4;  33 x 11008 x 4096: 21.5 / 26.4
//   two parts    16 x 4096 x 512: 6.6 / 7.1;  33: 9.6 / 7.1;  64: 13.7 / 7.0
//   one part     16 x 1024 x 256: 6.4 / 5.9;  33: 9.0 / 6.0;  64: 12.8 / 6.0;  K of two blocks, 16 x 64 x 128 in 32 groups: 6.2 / 5.5
//   long K       64 x 32000 x 4096, one part: 52.7 / 50.7;  33: 50.2 / 50.4
//   few tiles, K cut into more ranges there than a cluster has: 16 x 128 x 8192: 8.1 / 11.1;  x 32768: 22.2 / 13.7
//   clusters that fill the SMs to the last slot do not pack: 33 x 4096 x 4096 in 3 groups (96 clusters of 3): 29.1 / 28.2
//   several CTAs per slot, one tile each where the general kernel is persistent: 64 x 4096 x 128 in 64 groups: 90.7 / 22.9,
//                16: 40.8 / 22.0;  16 x 128256 x 4096: 165 / 183;  1 x 64 x 64 in 512 groups: 8.0 / 11.5
//   C off 16 bytes, one part, short K: 35 x 10245 x 64: 8.6 / 10.0;  64 x 1023 x 256: 12.2 / 8.5;  64 x 4095 x 128 in 64 groups: 90.5 / 83
// Of 600 products of up to 64 rows on 16 bytes, one is more than 5 % slower by these lines than on the general kernel (48 x 224 x 992 i8, 9.1 / 6.8).
// Of 400 off 16 bytes five are (59 x 2246 x 2288 fp8 in 57 groups 90 / 75); taking this kernel for all of them, 42 of 700 were more than 6 %
// slower.
bool gemm_skinny_applicable(const RbGemmProblem* p, uint32_t epi_flags) {
  const long long es = (long long)dtype_bytes(p->ab_type);
  if (p->m > 64 || p->trans_a || !p->trans_b || p->trans_c || p->ab_type == RB_F32 || (p->k * es) % 16) return false;
  const int sms = planning_sm_count(), kblocks = (int)((p->k * es + 127) / 128);
  const long long slots = 2LL * sms, tiles = (long long)p->g * ((p->n + kTileN - 1) / kTileN);
  const int rows = p->c_type == RB_I32 && epi_flags == 0 ? (p->m + 2) / 3 : p->m;
  // Rows of C off 16 bytes are stored element by element here and copied out of a staging tile there, K in one part up to eight blocks. us
  // of 131, 1030 and 10245 columns, K = 256, 16 rows: 6.3 / 6.6, 6.4 / 6.6, 6.8 / 9.0; 24: 7.3 / 6.7, 7.5 / 6.8, 7.7 / 9.1; 48: 10.3 / 6.7, 10.5 / 7.0, 10.8 / 9.3.
  if ((p->n * (long long)dtype_bytes(p->c_type)) % 16)
    return rows <= (kblocks > 4 ? 26 : 20) + (tiles > 64 ? 14 : 0) || kblocks > 8 || skinny_splits(p, tiles, kblocks, sms) > 1;
  if (tiles > slots) return (kblocks >= 8 && 2 * rows <= kblocks) || (tiles <= 2 * slots && rows <= 6);
  const int splits = skinny_splits(p, tiles, kblocks, sms);
  if (splits == 1) return rows <= (kblocks >= 4 ? std::max(16, kblocks / 2) : 12);
  if (kblocks >= 32 * splits && tiles * splits < sms) return false;
  const bool packs = tiles * splits * 10 <= slots * 9;
  if (rows <= (packs ? 8 : 4) * splits) return true;
  const bool divided_there = kblocks >= 16 && 2LL * p->g * ((p->n + 255) / 256) <= sms;
  return packs && rows <= 16 * splits && (splits >= 3 || divided_there);
}

RbStatus gemm_skinny_run(const RbGemmProblem* p, const EpiParams& epi, const void* a, const void* b, void* c, int kind, uint32_t fmt_a,
                         uint32_t fmt_b, uint32_t cfmt, long long wait_cycles, int stall, void* stream_v) {
  const DeviceInfo* dev = device_info();
  if (!dev) return RB_CUDA_ERROR;
  const int es = (int)dtype_bytes(p->ab_type), bke = 128 / es;
  SkinnyParams kp;
  memset(&kp, 0, sizeof(kp));
  kp.M = p->m; kp.N = p->n; kp.G = p->g;
  kp.nt = p->m <= 16 ? 16 : p->m <= 32 ? 32 : 64;
  kp.kblocks = (p->k + bke - 1) / bke;
  kp.tiles_n = (p->n + kTileN - 1) / kTileN;
  const long long tiles = (long long)p->g * kp.tiles_n;
  kp.splits = skinny_splits(p, tiles, kp.kblocks, dev->sm_count);
  const int stage_bytes = kWBytes + kp.nt * 128;
  kp.stages = std::min(kSkinnyMaxStages, (115712 - 1024 - 512) / stage_bytes);   // two CTAs per SM
  kp.idesc = make_idesc(cfmt, fmt_b, fmt_a, 0, 0, (uint32_t)kTileN, (uint32_t)kp.nt);
  kp.tmem_cols = kp.nt < 32 ? 32 : kp.nt;
  kp.acc_is_int = p->ab_type == RB_I8;
  kp.c = c;
  kp.c_type = p->c_type;
  kp.epi = epi;
  kp.status = dev->status_word;
  kp.wait_cycles = wait_cycles;
  kp.stall = stall;
  const CUtensorMapDataType dt = p->ab_type == RB_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                 : p->ab_type == RB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  SkinnyMaps maps;
  std::string err;
  const uint64_t pitch[1] = {(uint64_t)p->k * es};
  {
    const uint64_t dims[3] = {(uint64_t)p->k, (uint64_t)p->n, (uint64_t)p->g};
    const uint64_t strides[2] = {pitch[0], pitch[0] * p->n};
    const uint32_t box[3] = {(uint32_t)bke, (uint32_t)kTileN, 1u};
    if (!encode_tiled(&maps.w, dt, 3, b, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, &err)) return fail(RB_UNSUPPORTED, "B: " + err);
  }
  {
    const uint64_t dims[3] = {(uint64_t)p->k, (uint64_t)p->m, (uint64_t)p->g};
    const uint64_t strides[2] = {pitch[0], pitch[0] * p->m};
    const uint32_t box[3] = {(uint32_t)bke, (uint32_t)kp.nt, 1u};
    if (!encode_tiled(&maps.x, dt, 3, a, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, &err)) return fail(RB_UNSUPPORTED, "A: " + err);
  }
  typedef void (*Kernel)(const SkinnyMaps, const SkinnyParams);
  const Kernel kern = kind == kKindF16 ? gemm_skinny_kernel<kKindF16> : kind == kKindI8 ? gemm_skinny_kernel<kKindI8> : gemm_skinny_kernel<kKindF8>;
  const int smem = kp.stages * stage_bytes + 512 + 1024;
  RbStatus st = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
  if (st != RB_SUCCESS) return st;
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)(tiles * kp.splits), 1, 1);
  lc.blockDim = dim3(kSkinnyThreads, 1, 1);
  lc.dynamicSmemBytes = (size_t)smem;
  lc.stream = static_cast<cudaStream_t>(stream_v);
  cudaLaunchAttribute attr[2];
  lc.attrs = attr;
  attr[lc.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[lc.numAttrs].val.programmaticStreamSerializationAllowed = 1;
  ++lc.numAttrs;
  if (kp.splits > 1) {
    attr[lc.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[lc.numAttrs].val.clusterDim.x = (unsigned)kp.splits; attr[lc.numAttrs].val.clusterDim.y = 1; attr[lc.numAttrs].val.clusterDim.z = 1;
    ++lc.numAttrs;
  }
  RB_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, maps, kp));
  count_launch();
  return RB_SUCCESS;
}

}  // namespace rb
