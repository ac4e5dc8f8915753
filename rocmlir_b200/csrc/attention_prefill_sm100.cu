// rock.attention over more than one query tile, no side tensors, a scale above zero: two 128-row query tiles per CTA, each with a softmax group and an
// issuing warp of its own, so that one tile's products run while the other tile's scores become probabilities.
//
// 384 threads: warp 0 producer (TMA loads, work items), warps 1 and 3 MMA issuers of tile A and B, warp 2 TMEM allocator, warps 4-7
// softmax of tile A, warps 8-11 softmax of tile B (thread = query row = TMEM lane). TMEM: S_A, S_B (P over their first 64 columns),
// O_A, O_B = 512 columns. A tile's MMAs come from one thread and execute in order: PV(j) S(j+1) PV(j+1) ..., so S(j+1) may overwrite
// P(j), and the arrival of S(j+1) tells that O holds PV(j). The two issuers take turns, one block of one tile each: left to themselves
// both tiles fall into step, and then both want the exponentials, or the tensor core, at once (512 heads x 2048, causal 541 -> 607 us,
// all keys 0.90 -> 1.10 ms).
//
// A CTA works on one item (group, pair of query tiles) after another. The first is its own index, the following ones are those
// of CTAs that have not started yet (cluster launch control): items of uneven length - causal ones - go to whichever SM is free,
// without a counter in memory. The stream of blocks does not stop between items: the scores of the next item's first block are
// issued behind the last products of this one, and the softmax warps write O while they are computed.
//
// 512 heads x 2048 x 128, f16, twenty launches in a row: causal 776 -> 529 us, all keys 1135 -> 885; D = 64 735 -> 450 and 1072 -> 713;
// 64 heads x 1000, causal 50.6 -> 32.5 (one CTA per item, one issuing lane, scores read twice). The clock settles at 1.59 GHz under this kernel (1.76 at
// D = 64) from the first launch on: it is bound by power next to the chain of a tile's block (scores out 100 cycles, exponentials
// 1450, products and next scores 900 of a period of 3150). What the issuing warps cost was the code itself: with one copy of the
// products for each tile and K layout in a kernel of 77 KB every stretch of a round took 100 to 200 cycles to be fetched between the
// softmax warps' loops (period 3650); the whole warp runs the loop on uniform values, one lane issues (a lane alone: 4500).
// Every fourth exponential by a polynomial on the FMA pipe: 541 and 541 us, D = 64 735 and 713, not worth its error.
#include <algorithm>

#include "attention.cuh"
#include "launch.cuh"

namespace rb {
namespace {

struct PrefillSmem {
  static constexpr int kStages = 2;
  static constexpr int kTile = kQT * 256;               // a tile of Q, K or V, up to D = 128
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + 2 * kTile;
  static constexpr int kV = kK + kStages * kTile;
  static constexpr int kO = kV + kStages * kTile;       // eight warps x 32 rows x 64 columns of a result on its way out
  static constexpr int kBars = kO + 8 * 32 * 128;
  static constexpr int kTotal = kBars + 512 + 1024;
};

// Registers of a thread after the split: 256 x 208 + 128 x 88 = 384 x 168, what the block is launched with. A row's 128 scores stay in registers.
constexpr int kSoftmaxRegs = 208, kIssueRegs = 88;

// Group, first row and key blocks of the two tiles (0: the tile lies past the last query) of item idx; causal: longest first among as
// many groups as their K and V share the L2 cache (batch), so that the last items of a launch are short ones and a group's keys are
// still read from L2 by its next tile.
__device__ __forceinline__ int4 item_of(const AttParams& p, int batch, int idx) {
  const int pair_tiles = (p.q_tiles + 1) / 2;
  int g, pt;
  if (p.causal) {
    const int first = idx / (batch * pair_tiles) * batch, r = idx % (batch * pair_tiles);
    const int n = min(batch, p.G - first);
    pt = pair_tiles - 1 - r / n;
    g = first + r % n;
  } else {
    g = idx / pair_tiles;
    pt = idx % pair_tiles;
  }
  const int q0 = pt * (2 * kQT), blocks = (p.Sk + kKT - 1) / kKT;
  int nb[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int tq0 = q0 + t * kQT;
    nb[t] = tq0 >= p.Sq ? 0 : p.causal ? min(blocks, (min(tq0 + kQT, p.Sq) - 1) / kKT + 1) : blocks;
  }
  return make_int4(g, q0, nb[0], nb[1]);
}

template <int FROM, int TO>
__device__ __forceinline__ float row_max(const uint32_t* v, float start) {
  float m[4] = {start, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int i = FROM; i < TO; i += 8)
#pragma unroll
    for (int c = 0; c < 4; ++c) m[c] = fmaxf(fmaxf(m[c], __uint_as_float(v[i + 2 * c])), __uint_as_float(v[i + 2 * c + 1]));
  return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// KSTEPS: 16-element steps of a head's dimension; TRANS_K: K stored [G][Sk][D].
template <bool BF16, int KSTEPS, bool TRANS_K>
__global__ void __launch_bounds__(kPrefillThreads, 1) attention_prefill_kernel(const __grid_constant__ AttMaps maps, const AttParams p,
                                                                               const int batch) {
  constexpr int NS = PrefillSmem::kStages, kTile = PrefillSmem::kTile;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  int4* items = reinterpret_cast<int4*>(smem + PrefillSmem::kBars);        // [2] work items; a negative group: no more
  uint8_t* answer = smem + PrefillSmem::kBars + 32;                        // 16 bytes
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + PrefillSmem::kBars + 48);
  uint64_t* q_full = bars;                 // [2 tiles]
  uint64_t* q_empty = q_full + 2;          // [2 tiles]
  uint64_t* kv_full = q_empty + 2;         // [NS] V of a round's block and K of the next
  uint64_t* kv_empty = kv_full + NS;       // [NS]
  uint64_t* s_full = kv_empty + NS;        // [2 tiles]
  uint64_t* p_part = s_full + 2;           // [2 tiles] first 96 keys of P
  uint64_t* p_full = p_part + 2;           // [2 tiles]
  uint64_t* o_full = p_full + 2;           // [2 tiles] last product of an item
  uint64_t* item_full = o_full + 2;        // [2]
  uint64_t* item_empty = item_full + 2;    // [2]
  uint64_t* turn = item_empty + 2;         // [2 tiles] the tile's issuer may go on
  uint64_t* answered = turn + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(answered + 1);

  const int warp = warp_id_uniform();
  const int lane = lane_id();

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_part[i], 4);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_full[i], 1);
      mbar_init(&turn[i], 1);
      mbar_init(&item_full[i], 1);
      mbar_init(&item_empty[i], 2 + 8);   // issuers and softmax warps
    }
    for (int i = 0; i < NS; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 2);
    }
    mbar_init(answered, 1);
    fence_mbar_init();
  }
  if (warp == 2) {
    tmem_alloc<1>(tmem_holder, 512);
    tmem_relinquish<1>();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&maps.q);
    prefetch_tmap(&maps.k);
    prefetch_tmap(&maps.v);
    prefetch_tmap(&maps.o);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;   // S_A 0, S_B 128, O_A 256, O_B 384
  griddep_wait();   // nothing above touches what an earlier kernel of the stream reads or writes

  // Item n of this CTA, the same in all lanes; nothing when the wait has run out.
  auto read_item = [&](int n, uint32_t code, bool& ok) -> int4 {
    ok = mbar_wait_all(&item_full[n & 1], (uint32_t)(n >> 1) & 1u, p.status, code);
    int4 it = items[n & 1];
    if (!ok) it.x = -1;
    it.x = __shfl_sync(0xffffffffu, it.x, 0);
    it.y = __shfl_sync(0xffffffffu, it.y, 0);
    it.z = __shfl_sync(0xffffffffu, it.z, 0);
    it.w = __shfl_sync(0xffffffffu, it.w, 0);
    if (lane == 0) mbar_arrive(&item_empty[n & 1]);
    return it;
  };

  if (warp < 4) {
    regs_dec<kIssueRegs>();
    if (warp == 0 && lane == 0) {
      // ------------------------------ producer ------------------------------
      // Round by round what the issuer works on: V of block j and K of the block whose scores follow, the next one or the first of the
      // next item. The first round has no products, the last no scores.
      const uint32_t kd_bytes = kQT * KSTEPS * 32, v_bytes = (uint32_t)kKT * p.Dv * 2;
      int s = 0;
      uint32_t par = 0, q_par = 0;
      bool ok = true, asked = false;
      int idx = blockIdx.x;
      int4 it = make_int4(-1, 0, 0, 0);
      int blocks = 0, j = -1;
      for (int n = 0; ok;) {
        const bool last = j + 1 >= blocks;
        int4 nx = it;
        if (last) {
          if (asked) {
            if (!mbar_wait(answered, (uint32_t)(n - 1) & 1u, p.status, kStatusTimeoutProducer + 17)) break;
            idx = cta_answer(answer);
            fence_proxy_async();   // the answer is written through the async proxy again
          }
          nx = make_int4(-1, 0, 0, 0);
          if (idx >= 0) nx = item_of(p, batch, idx);
          if (!mbar_wait(&item_empty[n & 1], ((uint32_t)(n >> 1) & 1u) ^ 1u, p.status, kStatusTimeoutProducer + 16)) break;
          items[n & 1] = nx;
          mbar_arrive(&item_full[n & 1]);
          ++n;
          if (idx >= 0) {
            mbar_expect_tx(answered, 16);
            cta_request(answer, answered);
            asked = true;
          }
        }
        const bool more = !last || idx >= 0;
        const int sj = last ? 0 : j + 1;
        if (!mbar_wait(&kv_empty[s], par ^ 1u, p.status, kStatusTimeoutProducer + s)) break;
        mbar_expect_tx(&kv_full[s], (j >= 0 ? v_bytes : 0u) + (more ? kd_bytes : 0u));
        if (j >= 0) {
#pragma unroll 1
          for (int c = 0; c < p.Dv / 64; ++c)
            tma_load_3d(smem + PrefillSmem::kV + s * kTile + c * (kKT * 128), &maps.v, &kv_full[s], c * 64, j * kKT, it.x);
        }
        if (!more) break;
        {
          uint8_t* kd = smem + PrefillSmem::kK + s * kTile;
          if constexpr (TRANS_K) {
#pragma unroll 1
            for (int a = 0; a < KSTEPS / 4; ++a) tma_load_3d(kd + a * (kKT * 128), &maps.k, &kv_full[s], a * 64, sj * kKT, nx.x);
          } else {
#pragma unroll 1
            for (int c = 0; c < kKT / 64; ++c) tma_load_3d(kd + c * (KSTEPS * 2048), &maps.k, &kv_full[s], sj * kKT + c * 64, 0, nx.x);
          }
        }
        if (last) {   // the queries of a new item, when a tile's last scores have been computed; rows past the end arrive as zeros
#pragma unroll 1
          for (int t = 0; t < 2; ++t) {
            if ((t ? nx.w : nx.z) == 0) continue;
            if (!(ok = mbar_wait(&q_empty[t], ((q_par >> t) & 1u) ^ 1u, p.status, kStatusTimeoutProducer + 18 + t))) break;
            q_par ^= 1u << t;
            mbar_expect_tx(&q_full[t], kd_bytes);
#pragma unroll 1
            for (int a = 0; a < KSTEPS / 4; ++a)
              tma_load_3d(smem + PrefillSmem::kQ + t * kTile + a * (kQT * 128), &maps.q, &q_full[t], a * 64, nx.y + t * kQT, nx.x);
          }
          it = nx;
          blocks = max(it.z, it.w);
        }
        j = sj;
        if (++s == NS) { s = 0; par ^= 1u; }
      }
      griddep_launch();   // the last load is under way
    } else if (warp == 1 || warp == 3) {
      // ------------------------------ MMA issuer of one tile ------------------------------
      const int t = warp >> 1;
      // The whole warp runs the loop, on values that the compiler knows to be the same in all lanes, and one lane issues.
      const bool leader = elect_one();
      const uint32_t hi = smem_desc_hi(1024);
      const uint32_t q_lo0 = smem_desc_lo(smem_u32(smem + PrefillSmem::kQ), 16);
      const uint32_t k_lo0 = smem_desc_lo(smem_u32(smem + PrefillSmem::kK), TRANS_K ? 16u : (uint32_t)KSTEPS * 2048);
      const uint32_t v_lo0 = smem_desc_lo(smem_u32(smem + PrefillSmem::kV), kKT * 128);
      const uint32_t idesc_s = p.idesc_s, idesc_pv = p.idesc_pv;
      const bool trace = p.trace != nullptr && t == 0;
      long long w_p = 0, w_kv = 0, w_turn = 0;
      unsigned long long rounds = 0;
      const long long t_begin = trace ? clock64() : 0;
      auto timed = [&](long long& sum, uint64_t* bar, uint32_t parity, uint32_t code) -> bool {
        const long long t0 = trace ? clock64() : 0;
        const bool r = mbar_wait_all(bar, parity, p.status, kStatusTimeoutMma + code);
        if (trace) sum += clock64() - t0;
        return r;
      };
      int nb = 0, blocks = 0, n = 0;   // the tile's key blocks and those of the item under way (none yet)
      int j = -1;                      // the round's block
      int s = 0;                       // ring position
      uint32_t par = 0, q_par = 0, p_par = 0, turn_par = t ? 0u : 1u;   // tile A begins
      bool ok = true;
      const uint32_t tmem_p = tmem_base + t * 128, tmem_o = tmem_base + 256 + t * 128, q_lo = q_lo0 + t * (kTile >> 4);
      for (;;) {
        // products of block j, then scores of block sj: the next one, or the first of the next item
        const bool last = j + 1 >= blocks;
        int sj = j + 1, sb = nb, sblocks = blocks;
        bool more = true;
        if (last) {
          const int4 nx = read_item(n, kStatusTimeoutMma + 24, ok);
          if (!ok) break;
          ++n;
          more = nx.x >= 0;
          sj = 0;
          sb = more ? (t ? nx.w : nx.z) : 0;
          sblocks = max(nx.z, nx.w);
        }
        if (!(ok = timed(w_kv, &kv_full[s], par, s))) break;
        tc_fence_after();
        if (!(ok = timed(w_turn, &turn[t], turn_par, 26 + t))) break;
        turn_par ^= 1u;
        if (j >= 0 && j < nb) {
          const uint32_t v_lo = v_lo0 + s * (kTile >> 4);
          // the first 96 keys, then the others, as soon as their probabilities are written
          if (!(ok = timed(w_p, &p_part[t], p_par, 20 + t))) break;
          tc_fence_after();
          if (leader) {
#pragma unroll
            for (int kk = 0; kk < 6; ++kk)
              umma_ts<kKindF16>(tmem_o, tmem_p + kk * 8, desc64(v_lo + ((kk * 2048) >> 4), hi), idesc_pv, kk ? 1u : (j ? 1u : 0u));
          }
          if (!(ok = timed(w_p, &p_full[t], p_par, 22 + t))) break;
          p_par ^= 1u;
          tc_fence_after();
          if (leader) {
#pragma unroll
            for (int kk = 6; kk < 8; ++kk)
              umma_ts<kKindF16>(tmem_o, tmem_p + kk * 8, desc64(v_lo + ((kk * 2048) >> 4), hi), idesc_pv, 1u);
            if (j + 1 == nb) tc_commit<1>(&o_full[t]);
          }
        }
        if (sj < sb) {
          const uint32_t k_lo = k_lo0 + s * (kTile >> 4);
          if (sj == 0) {
            if (!(ok = mbar_wait_all(&q_full[t], q_par, p.status, kStatusTimeoutMma + 8 + t))) break;
            q_par ^= 1u;
            tc_fence_after();
          }
          if (leader) {
#pragma unroll
            for (int kk = 0; kk < KSTEPS; ++kk) {
              const uint32_t k_major = ((kk >> 2) * (kQT * 128) + (kk & 3) * 32) >> 4;
              umma_ss<kKindF16, 1>(tmem_p, desc64(q_lo + k_major, hi), desc64(k_lo + (TRANS_K ? k_major : (kk * 2048) >> 4), hi), idesc_s, kk ? 1u : 0u);
            }
            tc_commit<1>(&s_full[t]);
            if (sj + 1 == sb) tc_commit<1>(&q_empty[t]);
          }
        }
        if (leader) mbar_arrive(&turn[t ^ 1]);
        if (!more) break;
        if (leader) tc_commit<1>(&kv_empty[s]);
        if (++s == NS) { s = 0; par ^= 1u; }
        nb = sb;
        blocks = sblocks;
        j = sj;
        ++rounds;
      }
      if (trace && leader) {
        unsigned long long* tr = p.trace + (size_t)blockIdx.x * 16;
        tr[0] = (unsigned long long)(clock64() - t_begin);   // issuer of tile A: total
        tr[1] = (unsigned long long)w_kv;                    //   waiting for K and V tiles
        tr[2] = (unsigned long long)w_p;                     //   waiting for P
        tr[3] = rounds;
        tr[4] = (unsigned long long)w_turn;                  //   waiting for its turn
      }
    }
  } else {
    // ------------------------------ softmax and result of one tile ------------------------------
    regs_inc<kSoftmaxRegs>();
    const int t = (warp - 4) >> 2;
    const int wq = warp & 3;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_base + t * 128;
    const uint32_t tmem_o = tmem_base + lane_base + 256 + t * 128;
    const uint64_t scale2 = pair_f32(p.scale_log2, p.scale_log2);
    uint8_t* stg = smem + PrefillSmem::kO + (warp - 4) * (32 * 128);
    uint32_t s_par = 0, o_par = 0;
    long long sm_wait = 0, sm_busy = 0;
    bool ok = true;
    int4 it = read_item(0, kStatusTimeoutEpilogue + 8, ok);
    for (int n = 1; ok && it.x >= 0; ++n) {
      const int nb = t ? it.w : it.z;
      const int tq0 = it.y + t * kQT;
      float m_ref = -INFINITY, l = 0.0f;   // maximum that the exponentials are taken against, row sum
#pragma unroll 1
      for (int j = 0; j < nb; ++j) {
        const long long ts0 = p.trace ? clock64() : 0;
        if (!(ok = mbar_wait_all(&s_full[t], s_par, p.status, kStatusTimeoutEpilogue + t))) break;
        s_par ^= 1u;
        const long long ts1 = p.trace ? clock64() : 0;
        sm_wait += ts1 - ts0;
        tc_fence_after();
        const int key0 = j * kKT;
        uint32_t v[128];
        tmem_ld64(tmem_s, v);
        tmem_ld64(tmem_s + 64, v + 64);
        tmem_ld_wait();
        if (key0 + kKT > p.Sk || (p.causal && key0 + kKT - 1 > tq0)) {   // end of the keys, or the diagonal
          const int limit = min(p.Sk, p.causal ? tq0 + wq * 32 + lane + 1 : p.Sk) - key0;
#pragma unroll
          for (int i = 0; i < kKT; ++i) v[i] = i < limit ? v[i] : 0xff800000u;
        }
        // P of keys 32c .. 32c + 31, over columns of scores that are in registers by now, and the four sums
        uint64_t la = 0, lb = 0;
        uint32_t w[16];
        auto chunk = [&](int c, uint64_t neg_m) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int e = c * 32 + 2 * i;
            const float2 x = unpair_f32(fma_f32x2(pair_f32(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), scale2, neg_m));
            const float p0 = ex2(x.x), p1 = ex2(x.y);
            if (i & 1) lb = add_f32x2(lb, pair_f32(p0, p1));
            else la = add_f32x2(la, pair_f32(p0, p1));
            w[i] = pack2(p0, p1, BF16);
          }
        };
        // The exponentials are taken against m_ref, which moves only when the maximum has outgrown it by 2^8. From the second block on it
        // seldom does, so the first 96 keys are worked on while the maximum is found, and once more where m_ref had to move.
        float alpha = 1.0f;
        bool sure = false;
        if (j == 0) {
          const float mb = row_max<0, kKT>(v, -INFINITY) * p.scale_log2;   // the scale is positive
          m_ref = mb > -INFINITY ? mb : -INFINITY;
          sure = true;
        }
        uint64_t neg_m;
        for (;;) {
          const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;
          neg_m = pair_f32(-m_use, -m_use);
          la = lb = 0;
          chunk(0, neg_m);
          tmem_st16(tmem_s + 0, w);
          float mx = row_max<0, 48>(v, -INFINITY);
          chunk(1, neg_m);
          tmem_st16(tmem_s + 16, w);
          mx = row_max<48, 96>(v, mx);
          chunk(2, neg_m);
          tmem_st16(tmem_s + 32, w);
          mx = row_max<96, kKT>(v, mx);
          if (sure) break;
          const float mb = mx * p.scale_log2;
          const bool moved = mb > m_ref + 8.0f || (m_ref == -INFINITY && mb > -INFINITY);
          if (!__any_sync(0xffffffffu, moved)) break;
          if (moved) {
            alpha = ex2(m_ref - mb);
            m_ref = mb;
          }
#pragma unroll 1
          for (int c = 0; c < p.Dv / 16; ++c) {   // S(j) is there, so PV(j - 1) is in O
            uint32_t o[16];
            tmem_ld16(tmem_o + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st16(tmem_o + c * 16, o);
          }
          sure = true;
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_part[t]);
        chunk(3, neg_m);
        tmem_st16(tmem_s + 48, w);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t]);
        const float2 l01 = unpair_f32(la), l23 = unpair_f32(lb);
        l = l * alpha + ((l01.x + l01.y) + (l23.x + l23.y));
        if (p.trace) sm_busy += clock64() - ts1;
      }
      if (!ok) break;
      const int g = it.x;
      it = read_item(n, kStatusTimeoutEpilogue + 8, ok);   // while the last product runs
      if (!ok) break;
      if (nb > 0) {
        if (!(ok = mbar_wait_all(&o_full[t], o_par, p.status, kStatusTimeoutEpilogue + 6 + t))) break;
        o_par ^= 1u;
        tc_fence_after();
        const float inv = (l > 0.0f) ? 1.0f / l : 0.0f;
        const bool rows = tq0 + wq * 32 < p.Sq;
#pragma unroll 1
        for (int c = 0; c < p.Dv / 64; ++c) {
          uint32_t o[64];
          tmem_ld64(tmem_o + c * 64, o);
          tmem_ld_wait();
          if (lane == 0) bulk_wait_read<0>();   // the last box has left the staging rows
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
              w[k] = pack2(__uint_as_float(o[8 * i + 2 * k]) * inv, __uint_as_float(o[8 * i + 2 * k + 1]) * inv, BF16);
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0 && rows) {   // rows and columns past the end are clipped
            tma_store_3d(&maps.o, stg, c * 64, tq0 + wq * 32, g);
            bulk_commit();
          }
        }
        // O has been read: the next P announced by this warp lets the next item's products overwrite it
        __syncwarp();
        tc_fence_before();
      }
    }
    if (lane == 0) bulk_wait<0>();
    __syncwarp();
    if (p.trace && wq == 0 && lane == 0) {
      p.trace[(size_t)blockIdx.x * 16 + 8 + 2 * t] = (unsigned long long)sm_wait;   // softmax group t: waiting for S
      p.trace[(size_t)blockIdx.x * 16 + 9 + 2 * t] = (unsigned long long)sm_busy;   //   busy (incl. rescale)
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

template <bool BF16, int KSTEPS>
RbStatus launch(const AttMaps& maps, const AttParams& p, int batch, int items, cudaStream_t stream) {
  void (*const kern)(const AttMaps, const AttParams, const int) =
      p.trans_k ? attention_prefill_kernel<BF16, KSTEPS, true> : attention_prefill_kernel<BF16, KSTEPS, false>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), PrefillSmem::kTotal) != RB_SUCCESS) return RB_CUDA_ERROR;
  RB_CUDA_TRY(launch_after(kern, (unsigned)items, kPrefillThreads, PrefillSmem::kTotal, stream, 1, maps, p, batch));
  return RB_SUCCESS;
}

}  // namespace

RbStatus attention_prefill_launch(const AttMaps& maps, const AttParams& p, cudaStream_t stream) {
  const long long group_bytes = 2LL * p.Sk * (p.D + p.Dv);
  const int batch = (int)std::max(1LL, std::min((long long)p.G, (32LL << 20) / group_bytes));
  const int items = p.G * ((p.q_tiles + 1) / 2);
  if (p.D == 64) return p.is_bf16 ? launch<true, 4>(maps, p, batch, items, stream) : launch<false, 4>(maps, p, batch, items, stream);
  return p.is_bf16 ? launch<true, 8>(maps, p, batch, items, stream) : launch<false, 8>(maps, p, batch, items, stream);
}

}  // namespace rb
