// Causal online-softmax (flash) attention forward for sm_100a, GQA-aware.
//
// One persistent CTA per SM owns TWO 128-row query tiles of one head at a time.  Q and the K / V tiles (128 rows each, a
// ring) come in by TMA (local memory, no multicast).  For query tile w: S_w = Q_w K^T is a tcgen05.mma into tensor
// memory; 128 softmax threads (one query row each, so row max / row sum need no shuffles) read S_w, keep the running
// max and sum in the log2 domain and write P_w as bf16 back over S_w's columns; O_w += P_w V takes P_w straight from
// tensor memory.  While one tile's threads work on exponentials the tensor core runs the other tile's two products:
//
//   tensor core : S0(j) | PV1(j-1) S1(j) | PV0(j) S0(j+1) | PV1(j) S1(j+1) | ...
//   softmax 0   :        P0(j)           |      ...       |   P0(j+1)
//   softmax 1   :   ...  |    P1(j)                       |   ...
//
// O_w is only rescaled when the running max grew by more than 2^8 (the final division by the row sum makes the result
// exact either way); the softmax threads do it themselves, with a tcgen05.ld / tcgen05.st round trip.
//
// The schedule (two query tiles in turn, rescaling only beyond 2^8, the second product started before all of P is there) is
// that of the published FlashAttention-4.
//
// What bounds it: per 128 x 128 scores at head_dim 128 the tensor core needs 1024 clocks and the exponentials also 1024
// (16 a clock and SM); at head_dim 64 512 against 1024.  At head_dim 128 and T 8191 both units run at about 66 %
// of a CTA's time (ncu): a tile's chain of loading, maximum, exponentials and its two products is what is left over.  (2^x on
// the FMA pipe for a quarter of the scores changed nothing, for more of them it was slower.)  One query tile per CTA with P
// through shared memory, two CTAs per SM (attention_fwd_tile.cuh, which short launches still take), makes P's round trip and
// the wait for its product part of every tile's chain.  That kernel -> this one, launches repeated, SM clock under load beside it:
//   B 8, H 32, T 4096, D 128        1484 ->  937 us in short bursts, 1572 (1837 MHz) -> 1092 us (1537 MHz) for seconds under
//                                   the power cap (741 -> 1174 and 699 -> 1007 TFLOP/s)
//   B 1, H 24 / 8, T 8191, D 128     466 ->  317 us, 502 (1792 MHz) -> 368 us (1575 MHz)
//   B 4, H 32 / 4, T 2048, D 64      125 ->  105 us (1965 MHz)
//   B 8, H 12, T 1024, D 64         32.9 -> 28.6 us (1965 MHz), 43 -> 36 us with a cold L2
//
// The reference has no attention kernel in use: its CPU path materialises softmax(QK^T s + mask) V
// (crates/incin-backends/src/cpu/ops/shape_ops.rs:1245-1269) and CUDA reports SDPA as unsupported;
// flash_attention_lite.cu there is dead code with one thread per query row.
#include "ptx.cuh"
#include "launch.cuh"
#include "../../include/incin_b200.h"
#include <math_constants.h>

namespace incin {

int make_operand_map(CUtensorMap* out, const void* ptr, long long inner, long long rows, long long ld,
                     long long batch_lo, long long stride_lo, long long batch_hi, long long stride_hi, int box_inner,
                     int box_rows);
int device_sm_count();

constexpr int FA_BM = 128;        // rows of one query tile and of one K / V tile
constexpr int FA_THREADS = 384;   // warp 0: TMA, warp 1: tcgen05 issue, warps 4-7 / 8-11: softmax of query tile 0 / 1
// Registers: 384 threads are launched with 168 each (64512 of the SM's 65536).  The first warpgroup gives back all but 88
// and the two softmax warpgroups take 208, enough to hold a whole row of scores: 128 x (88 + 208 + 208) = 64512.
constexpr int FA_REGS_ISSUE = 88, FA_REGS_SOFTMAX = 208;

template <int D>
struct FaCfg {
  static constexpr int TILE_BYTES = FA_BM * D * 2;      // one Q, K or V tile
  static constexpr int STAGES = D == 128 ? 5 : 8;       // ring of K_0 V_0 K_1 V_1 ... tiles
  static constexpr int OFF_RING = 2 * TILE_BYTES;       // behind the two query tiles
  static constexpr int OFF_BAR = OFF_RING + STAGES * TILE_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
  // tensor memory: S_w (P_w in its first 64 columns) at [128 w, 128 w + 128), O_w at 256 + D w
  static constexpr int TMEM_COLS = 512, COL_O = 256;
  // columns of P_w after which the first products of O_w += P_w V are let go: against none of them 96 of 128 took 5 % off
  // head_dim 128 (B 1, H 24 / 8, T 8191) and 3 % off head_dim 64 (B 4, H 32 / 4, T 2048); 64 is no better
  static constexpr int PART = 96;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared-memory plan");
};

struct FaParams {
  int T, Hq, Hkv, B;
  int n_pairs;       // pairs of query tiles per head
  float scale_log2;  // softmax scale * log2(e)
  __nv_bfloat16* O;
  long long o_stride_b, o_stride_t, o_stride_h;
  float* lse;  // [B, Hq, Tpad], log2 domain; rows in [T, Tpad) are written as +inf
  int Tpad;
  int* status;
  int pair_major;   // 1: all heads' heaviest pairs come first in the item list, 0: the pairs of one head are neighbours
};

template <int D>
__global__ void __launch_bounds__(FA_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const FaParams p) {
  using Cfg = FaCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sRing = smem + Cfg::OFF_RING;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* full = bars;            // [STAGES <= 8] a K or V tile has landed
  uint64_t* empty = bars + 8;       // [STAGES <= 8] the products that read it have finished
  uint64_t* q_full = bars + 16;     // [2] query tile w has landed
  uint64_t* q_empty = bars + 18;    // [2] the last score product of query tile w has finished
  uint64_t* s_full = bars + 20;     // [2] S_w is in tensor memory (and every earlier product has finished)
  uint64_t* p_full = bars + 22;     // [2] P_w is in tensor memory, O_w rescaled (one arrival per softmax warp)
  uint64_t* o_full = bars + 24;     // [2] O_w of this item is complete
  uint64_t* p_part = bars + 26;     // [2] the first PART columns of P_w are in tensor memory, O_w rescaled
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_heads = p.Hq * p.B;
  const int n_items = p.n_pairs * n_heads;
  // Item list, walked in snake order (round r of CTA c: item r G + c, in odd rounds (r + 1) G - 1 - c), so that a CTA
  // which got a long item in one round gets a short one in the next.  When K / V of all heads together fit L2
  // (pair_major), the pair is the slowest index: all heads' heaviest pairs come first and the light ones fill the gaps
  // at the end.  Otherwise a head's pairs are neighbours, so that its K / V are read from DRAM once.
  auto item_of = [&](int r, int& q0, int& hq, int& b) -> bool {
    const int G = (int)gridDim.x, c = (int)blockIdx.x;
    const int idx = (r & 1) ? (r + 1) * G - 1 - c : r * G + c;
    if (idx >= n_items) return false;
    const int pair = p.pair_major ? idx / n_heads : idx % p.n_pairs;
    const int hb = p.pair_major ? idx % n_heads : idx / p.n_pairs;
    q0 = (p.n_pairs - 1 - pair) * (2 * FA_BM);
    hq = hb % p.Hq;
    b = hb / p.Hq;
    return true;
  };
  // K / V tiles that query tile w of the item sees (causal); 0 when the tile lies beyond the sequence
  auto kv_tiles = [&](int q0, int w) -> int {
    const int first = q0 + w * FA_BM;
    return first >= p.T ? 0 : min(first + FA_BM - 1, p.T - 1) / FA_BM + 1;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int w = 0; w < 2; ++w) {
      mbar_init(&q_full[w], 1);
      mbar_init(&q_empty[w], 1);
      mbar_init(&s_full[w], 1);
      mbar_init(&p_full[w], 4);
      mbar_init(&o_full[w], 1);
      mbar_init(&p_part[w], 4);
    }
    *abort_flag = 0;
    mbar_init_fence();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();   // tensor memory is held; a successor may be scheduled as CTAs retire
  pdl_wait();                // no global memory was touched above

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FA_REGS_ISSUE));
  if (warp == 0) {
    // producer: the whole warp walks the loop (warp-uniform waits and address arithmetic), one elected lane issues
    const bool leader = elect_one() != 0;
    int stage = 0;
    uint32_t phase = 0, q_phase[2] = {0, 0};
    bool ok = true;
    int q0, hq, b;
    for (int r = 0; ok && item_of(r, q0, hq, b); ++r) {
      const int hkv = hq / (p.Hq / p.Hkv);
      const int n1 = kv_tiles(q0, 1), n = max(kv_tiles(q0, 0), n1);
      auto load_q = [&](int w) -> bool {
        if (!mbar_wait(&q_empty[w], q_phase[w] ^ 1, abort_flag, p.status, kStatusTimeoutEmpty)) return false;
        q_phase[w] ^= 1;
        if (leader) {
          mbar_expect_tx(&q_full[w], Cfg::TILE_BYTES);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(smem + w * Cfg::TILE_BYTES + c * (FA_BM * 128), &tmQ, &q_full[w], c * 64, q0 + w * FA_BM, hq, b);
        }
        __syncwarp();
        return true;
      };
      auto load_kv = [&](const CUtensorMap* tm, int j) -> bool {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status, kStatusTimeoutEmpty)) return false;
        if (leader) {
          mbar_expect_tx(&full[stage], Cfg::TILE_BYTES);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(sRing + stage * Cfg::TILE_BYTES + c * (FA_BM * 128), tm, &full[stage], c * 64, j * FA_BM, hkv, b);
        }
        __syncwarp();
        if (++stage == Cfg::STAGES) {
          stage = 0;
          phase ^= 1;
        }
        return true;
      };
      ok = load_q(0) && load_kv(&tmK, 0) && (n1 == 0 || load_q(1)) && load_kv(&tmV, 0);
      for (int j = 1; j < n && ok; ++j) ok = load_kv(&tmK, j) && load_kv(&tmV, j);
    }
  } else if (warp == 1) {
    // issuer: the whole warp walks the loop, one elected lane executes the tcgen05 instructions.  S_w(j+1) follows
    // O_w += P_w(j) V_j directly although it overwrites P_w: products of one issuing thread run in order.  (PTX states that
    // for products of one accumulator and shape; for these two it is what the published kernels of this schedule rely on,
    // and tests/test_attention_edges_gpu.py repeats the forward pass to the bit to catch an exception.)
    const bool leader = elect_one() != 0;
    constexpr uint32_t idesc_s = make_idesc_bf16(FA_BM, FA_BM, false, false);
    constexpr uint32_t idesc_o = make_idesc_bf16(FA_BM, D, false, true);
    constexpr uint32_t kDescHi = ((1024u >> 4) & 0x3FFF) | (1u << 14) | (2u << 29);   // SBO 1024, version, SWIZZLE_128B
    constexpr uint32_t kLoK = (16u >> 4) << 16;                                       // K-major: LBO 16
    constexpr uint32_t kLoMN = ((uint32_t)(FA_BM * 128) >> 4) << 16;                  // MN-major V: 64-column chunks 16 KB apart
    auto desc = [&](uint32_t lo) -> uint64_t { return (static_cast<uint64_t>(kDescHi) << 32) | lo; };
    const uint32_t q16 = (smem_u32(smem) & 0x3FFFF) >> 4, ring16 = (smem_u32(sRing) & 0x3FFFF) >> 4;
    uint32_t q_phase[2] = {0, 0}, p_phase[2] = {0, 0};
    int stage = 0;          // ring position of the next tile to be consumed
    uint32_t phase = 0;
    bool ok = true;
    auto scores = [&](int w, int k_stage) {   // S_w = Q_w K^T
      const uint32_t a = q16 + w * (Cfg::TILE_BYTES >> 4), bk = ring16 + k_stage * (Cfg::TILE_BYTES >> 4);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = (kk >> 2) * (FA_BM * 128 >> 4) + (kk & 3) * 2;
        if (leader) umma_f16_ss(tmem_base + w * FA_BM, desc(a + off + kLoK), desc(bk + off + kLoK), idesc_s, kk > 0 ? 1u : 0u);
      }
      if (leader) umma_commit(&s_full[w]);
      __syncwarp();
    };
    auto take = [&](int& my_stage) -> bool {   // next tile of the ring
      if (!mbar_wait(&full[stage], phase, abort_flag, p.status, kStatusTimeoutFull)) return false;
      my_stage = stage;
      if (++stage == Cfg::STAGES) {
        stage = 0;
        phase ^= 1;
      }
      return true;
    };
    auto wait_q = [&](int w) -> bool {
      if (!mbar_wait(&q_full[w], q_phase[w], abort_flag, p.status, kStatusTimeoutFull)) return false;
      q_phase[w] ^= 1;
      return true;
    };
    int q0, hq, b;
    for (int r = 0; ok && item_of(r, q0, hq, b); ++r) {
      const int n_w[2] = {kv_tiles(q0, 0), kv_tiles(q0, 1)};
      const int n = max(n_w[0], n_w[1]);
      int k_stage = 0, v_stage = 0;
      ok = take(k_stage);
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        if (!ok || n_w[w] == 0) continue;
        ok = wait_q(w);
        if (!ok) continue;
        tc_fence_after();
        scores(w, k_stage);
        if (leader && n_w[w] == 1) umma_commit(&q_empty[w]);
      }
      if (ok && leader) umma_commit(&empty[k_stage]);
      for (int j = 0; j < n && ok; ++j) {
        ok = take(v_stage);
        if (ok && j + 1 < n) ok = take(k_stage);
        if (!ok) break;
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          if (!ok || j >= n_w[w]) continue;
          const uint32_t bv = ring16 + v_stage * (Cfg::TILE_BYTES >> 4);
          // O_w += P_w V: 16 kv rows per product, P_w from tensor memory, the first products before all of P_w is there
          ok = mbar_wait(&p_part[w], p_phase[w], abort_flag, p.status, kStatusTimeoutTmemFull);
          if (!ok) continue;
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < FA_BM / 16; ++kk) {
            if (kk == Cfg::PART / 16) {
              ok = mbar_wait(&p_full[w], p_phase[w], abort_flag, p.status, kStatusTimeoutTmemFull);
              if (!ok) break;
              tc_fence_after();
            }
            if (leader) umma_f16_ts(tmem_base + Cfg::COL_O + w * D, tmem_base + w * FA_BM + kk * 8, desc(bv + kk * 128 + kLoMN),
                                    idesc_o, (j > 0 || kk > 0) ? 1u : 0u);
          }
          if (!ok) continue;
          p_phase[w] ^= 1;
          if (j + 1 < n_w[w]) {
            scores(w, k_stage);
            if (leader && j + 2 == n_w[w]) umma_commit(&q_empty[w]);
          } else if (leader) {
            umma_commit(&o_full[w]);
          }
          __syncwarp();
        }
        if (ok && leader) {
          umma_commit(&empty[v_stage]);
          if (j + 1 < n) umma_commit(&empty[k_stage]);
        }
        __syncwarp();
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FA_REGS_SOFTMAX));
    // ------------------------------------------------------------------ softmax / rescale / epilogue of query tile w
    const int w = (warp >> 2) - 1;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;  // row inside the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_S = tmem_base + w * FA_BM + lane_addr, tmem_O = tmem_base + Cfg::COL_O + w * D + lane_addr;
    uint32_t s_phase = 0, o_phase = 0;
    bool ok = true;
    int q0, hq, b;
    for (int r_item = 0; ok && item_of(r_item, q0, hq, b); ++r_item) {
      const int n = kv_tiles(q0, w);
      if (n == 0) continue;
      const int q_idx = q0 + w * FA_BM + row;
      float m_ref = -CUDART_INF_F;
      float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      for (int j = 0; j < n; ++j) {
        if (!mbar_wait(&s_full[w], s_phase, abort_flag, p.status, kStatusTimeoutTmemFull)) { ok = false; break; }
        s_phase ^= 1;
        tc_fence_after();
        // whole S row into registers with back-to-back TMEM loads and a single wait
        uint32_t s[FA_BM];
#pragma unroll
        for (int c = 0; c < FA_BM / 32; ++c) tmem_ld_32x32(tmem_S + c * 32, reinterpret_cast<uint32_t(&)[32]>(s[c * 32]));
        tmem_ld_wait();
        if (j == n - 1) {   // the diagonal tile is the last one; masked scores become -inf
          const int last = min(q_idx, p.T - 1) - j * FA_BM;
#pragma unroll
          for (int i = 0; i < FA_BM; ++i)
            if (i > last) s[i] = __float_as_uint(-CUDART_INF_F);
        }
        float mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};   // four chains, three-input maxima
#pragma unroll
        for (int i = 0; i < FA_BM; i += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            mx4[e] = fmaxf(fmaxf(mx4[e], __uint_as_float(s[i + e * 2])), __uint_as_float(s[i + e * 2 + 1]));
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
        // lazy rescale: only move the reference when the maximum grew by more than 2^8
        const bool need = mx > m_ref + 8.0f;
        if (__any_sync(0xffffffffu, need)) {
          const float alpha = need ? exp2f(m_ref - mx) : 1.0f;   // 0 on the first tile
          if (need) m_ref = mx;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            l2[e].x *= alpha;
            l2[e].y *= alpha;
          }
          if (j > 0) {   // s_full covers O_w += P_w(j-1) V_{j-1}: O_w is at rest
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32(tmem_O + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32(tmem_O + c * 32, o);
            }
          }
        }
        // P = exp2(s * scale - m_ref) as packed bf16 over the first half of S_w's columns, row sums in fp32
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), nm2 = make_float2(-m_ref, -m_ref);
#pragma unroll
        for (int c = 0; c < FA_BM / 32; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = fma2(make_float2(__uint_as_float(s[c * 32 + i]), __uint_as_float(s[c * 32 + i + 1])), sc2, nm2);
            const float2 e = make_float2(exp2f(x.x), exp2f(x.y));
            l2[(i >> 1) & 1] = add2(l2[(i >> 1) & 1], e);
            pk[i >> 1] = pack_bf16x2(e.x, e.y);
          }
          tmem_st_32x16(tmem_S + c * 16, pk);
          if ((c + 1) * 32 == Cfg::PART) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_part[w]);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();                        // every lane's stores and fences precede the single arrival of its warp
        if (lane == 0) mbar_arrive(&p_full[w]);
      }
      if (!ok || !mbar_wait(&o_full[w], o_phase, abort_flag, p.status, kStatusTimeoutTmemFull)) { ok = false; break; }
      o_phase ^= 1;
      tc_fence_after();
      const float l_sum = (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
      const float inv = 1.0f / l_sum;
      const bool live_row = q_idx < p.T;
      __nv_bfloat16* orow = p.O + (long long)b * p.o_stride_b + (long long)q_idx * p.o_stride_t +
                            (long long)hq * p.o_stride_h;
      const bool wide = aligned32(orow);
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_O + c * 32, o);
        tmem_ld_wait();
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack_bf16x2(__uint_as_float(o[e * 2]) * inv, __uint_as_float(o[e * 2 + 1]) * inv);
        if (live_row && wide) {   // 32 bytes per store: whole sectors of the row
          st_global_b256(orow + c * 32, reinterpret_cast<uint32_t(&)[8]>(pk[0]));
          st_global_b256(orow + c * 32 + 16, reinterpret_cast<uint32_t(&)[8]>(pk[8]));
        } else if (live_row) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            *reinterpret_cast<uint4*>(orow + c * 32 + u * 8) = make_uint4(pk[u * 4], pk[u * 4 + 1], pk[u * 4 + 2], pk[u * 4 + 3]);
        }
        __syncwarp();
      }
      p.lse[((long long)b * p.Hq + hq) * p.Tpad + q_idx] = live_row ? m_ref + log2f(l_sum) : CUDART_INF_F;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

}  // namespace incin

#include "attention_fwd_tile.cuh"

namespace incin {

// Whether the kernel with one query tile per CTA is the faster one.  Measured over head_dim 64 and 128, 6 to 32 heads (grouped
// and not), B 1 to 64, T 16 to 2048 (560 launches; the pairs alone are up to 1.8 times as slow at these, single tiles alone up
// to 1.9 times at length).  Pairs | single tiles, in us:
// - No more pairs than SMs: a pair takes longer than its two tiles side by side.  head_dim 128, B 1, H 8: T 64 5.6 | 4.3,
//   T 192 8.7 | 6.1, T 300 9.4 | 8.1, T 384 9.5 | 9.9, T 448 12.0 | 10.5, T 1000 18.5 | 21.0.  At head_dim 64 only an even
//   number of tiles loses (H 6: T 256 7.4 | 6.6, T 384 7.4 | 7.9, T 1000 15.8 | 14.2).  Where the single tiles do not fit
//   the SMs at once either, the two are even, except at head_dim 128 up to T 192.
// - More: both go in rounds, of a pair per SM and of two tiles per SM.  A pair of which only one tile exists counts as much
//   as two, so with one or three tiles a head the rounds decide (H 12, D 64, T 128: B 16 8.3 | 7.1 in 2 | 1 rounds, B 32
//   10.7 | 11.5 in 3 | 2); with two or five, how full the last one is (D 128, H 24 / 8, T 256: B 8 16.6 | 13.6 at 65 %,
//   B 16 23.5 | 24.5 at 86 %).  At head_dim 128 single tiles stop after 64 keys: up to T 64 they always win (B 64, H 32:
//   44.8 | 37.5), and gain more up to T 192 and T 320.
static bool one_tile_per_cta(const incin_attn_desc* d, int sms) {
  const int tiles = (d->T + FA_BM - 1) / FA_BM;
  if (d->Hq > 65535 || d->B > 65535 || tiles > 65535) return false;   // its grid
  const long long heads = (long long)d->Hq * d->B, pairs = (tiles + 1) / 2 * heads;
  const bool wide = d->D == 128;
  if (pairs <= sms) {
    const bool half = pairs * 2 <= sms, third = pairs * 3 <= sms;
    if (!wide) return tiles % 2 == 0 && (tiles <= 4 ? half : third);
    return d->T <= 192 || (d->T <= 320 && half) || (d->T > 384 && d->T <= 448 && third);
  }
  if (wide && d->T <= 64) return true;
  const long long rounds = (pairs + sms - 1) / sms, single_rounds = (tiles * heads + 2 * sms - 1) / (2 * sms);
  auto emptier = [&](int percent) { return pairs * 100 < rounds * sms * percent; };   // than that, on average over the rounds
  switch (tiles) {
    case 1: return rounds <= 6 && rounds == 2 * single_rounds;
    case 2: return wide && emptier(d->T <= 192 ? 87 : 75);
    case 3: return 2 * rounds >= 3 * single_rounds || (wide && d->T <= 320 && emptier(87));
    case 5: return emptier(75);
    default: return false;
  }
}

template <int D>
static int launch_fwd(const incin_attn_desc* d, cudaStream_t stream) {
  using Cfg = FaCfg<D>;
  CUtensorMap tq, tk, tv;
  int rc = make_operand_map(&tq, d->q, D, d->T, d->q_stride_t, d->Hq, d->q_stride_h, d->B, d->q_stride_b, 64, FA_BM);
  if (rc) return rc;
  rc = make_operand_map(&tk, d->k, D, d->T, d->k_stride_t, d->Hkv, d->k_stride_h, d->B, d->k_stride_b, 64, FA_BM);
  if (rc) return rc;
  rc = make_operand_map(&tv, d->v, D, d->T, d->v_stride_t, d->Hkv, d->v_stride_h, d->B, d->v_stride_b, 64, FA_BM);
  if (rc) return rc;
  auto kern = flash_fwd_kernel<D>;
  static PerDeviceFlags attr;
  if (!ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, attr)) return INCIN_ERR_LAUNCH;
  const int n_q_tiles = (d->T + FA_BM - 1) / FA_BM;
  FaParams p;
  p.T = d->T;
  p.Hq = d->Hq;
  p.Hkv = d->Hkv;
  p.B = d->B;
  p.n_pairs = (n_q_tiles + 1) / 2;
  p.scale_log2 = d->scale * 1.4426950408889634f;
  p.O = (__nv_bfloat16*)d->o;
  p.o_stride_b = d->o_stride_b;
  p.o_stride_t = d->o_stride_t;
  p.o_stride_h = d->o_stride_h;
  p.lse = d->lse;
  p.Tpad = n_q_tiles * FA_BM;
  p.status = (int*)d->status;
  // K and V of every (batch, KV head) within 48 MB, about 40 % of L2: the line measured for the kernel with one tile per CTA
  // (heaviest tiles first cost it 19 % at 512 MB).  For this one, all heads' heaviest pairs first | head by head, us: 24 MB
  // (B 8, H 12, T 1024, D 64) 28.6 | 33.9, 32 MB (B 1, H 24 / 8, T 8191, D 128) 315 | 428, 96 MB (H 24) 335 | 441, 128 MB
  // (B 2, H 32, T 4096) 250 | 265, 192 MB (B 6, H 24 / 8, T 8191) 2055 | 1983, 256 MB (B 8, H 32, T 2048) 297 | 277, 512 MB
  // (T 4096) 1102 | 931: it lies nearer to 128 MB.
  p.pair_major = ((long long)d->B * d->Hkv * d->T * D * 2 * 2 <= (48ll << 20)) ? 1 : 0;
  const long long items = (long long)p.n_pairs * d->Hq * d->B;
  if (items > (1ll << 30)) return INCIN_ERR_TOO_LARGE;   // the kernel counts items in 32 bits
  const int sms = device_sm_count();
  const dim3 grid((unsigned)(items < sms ? items : sms));
  if (launch_pdl<true>(kern, grid, dim3(FA_THREADS), Cfg::SMEM_BYTES, stream, tq, tk, tv, p) != cudaSuccess) return INCIN_ERR_LAUNCH;
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

}  // namespace incin

extern "C" int incin_flash_attn_fwd(const incin_attn_desc* d, void* stream) {
  if (!d || !d->q || !d->k || !d->v || !d->o || !d->lse || d->B <= 0 || d->T <= 0 || d->Hq <= 0 || d->Hkv <= 0 ||
      d->Hq % d->Hkv != 0)
    return INCIN_ERR_ARGUMENT;
  if ((d->o_stride_t % 8) || (d->o_stride_h % 8) || (d->o_stride_b % 8) || (reinterpret_cast<uintptr_t>(d->o) & 15))
    return INCIN_ERR_ALIGNMENT;
  if (d->D != 64 && d->D != 128) return INCIN_ERR_UNSUPPORTED;
  const cudaStream_t s = (cudaStream_t)stream;
  if (incin::one_tile_per_cta(d, incin::device_sm_count()))
    return d->D == 64 ? incin::launch_fwd_tile<64, 128>(d, s) : incin::launch_fwd_tile<128, 64>(d, s);
  return d->D == 64 ? incin::launch_fwd<64>(d, s) : incin::launch_fwd<128>(d, s);
}
