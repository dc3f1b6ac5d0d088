// Triple-dot-product trittention forward on Blackwell tensor cores (tcgen05 + TMEM + TMA).
//
// Formulation.  For one query q and a tile of 128 K2 rows, the 128 "pair rows" r = (q, k)
// carry the pre-scaled operand  A[r,h] = alpha*log2(e) * Q[q,h] * K2[k,h].  With it the
// score slab is an ordinary GEMM, S[r,j] = sum_h A[r,h] K1[j,h], and the walk over j is
// exactly a flash-attention inner loop with K1 as keys and SiLU(V1) as values:
//     acc[r,h] = sum_j exp2(S[r,j] - m_r) SiLU(V1)[j,h]          (online soft-max per row)
// The V2 factor and the soft-max over k are applied when the tile is folded into the
// query's running output:  O[q,h] = sum_r w_r acc[r,h] V2[k_r,h] / sum_r w_r l_r.
// (The reference's Blackwell Triton kernel uses the same (q,k)-row arrangement,
// b200/fwd_b200.py:217-220,253,317-321, with 16x16 query/key tiles; its generic kernel
// builds K1 x K2 outer products per tile, triple_dot_product/kernels/fwd.py:160-164.)
//
// One CTA (persistent, 512 threads) processes a pair of queries (qa, qb) of the same 128-row
// block as two row tiles that share every K1 / SiLU(V1) tile and take turns on the tensor pipe:
//   warp 0       TMA producer: the K2 tile of each k-tile, then a ring of 128-row K1 / SiLU(V1) tiles
//   warp 1       issues tcgen05.mma: S_x = A_x*K1^T (128x128 fp32 slab in TMEM, one per tile) and
//                acc_x += P_x*SiLU(V1) with P_x read from TMEM (it overlays S_x) and the value tile used
//                row-major (MN-major descriptor).  128-column slabs keep every accumulation chain at
//                8 instructions of 128x128x16, the shape the pipe runs at full rate.
//   warps 4-11   two soft-max warpgroups (one row per thread); they also form A_a, A_b.  Where a head-wide bound on
//                the scores is small (per-head statistics from a small kernel before this one) every row has the same
//                soft-max reference and the warpgroups work on the same slab, tile a then
//                tile b, 64 of its 128 columns each: one pass, exp2, P written back to TMEM as 16-bit over the
//                first half of the columns just read.  Otherwise warpgroup x owns tile x and a thread its whole
//                row: row maximum, exp2 with lazy rescaling of the accumulator, P over the first 64 columns of S_x
//   warps 12-15  fold warpgroup: when a k-tile is finished, folds acc_x (times V2, soft-max over k) into
//                the queries' running (max, sum, output) while the other warps start the next k-tile; with one reference for
//                a head the sums just add up in registers, without exchanges between threads
// What bounds it: the exponentials (66 % of the special-function unit's time at head dimension 64, 58 % at 128, where the products
// take as long), the rest of the soft-max stage of a slab around them and the change of k-tiles.  A time trace of the form before had
// 1300 cycles a stage against 1024 of exponentials, and 3300 to 4100 a change, 2000 of them the operands.  Operands with a thread on
// one column of every 16th or 32nd row, norms only where a row's bound is asked for, and the fold without exchanges: T=512 D=64 bf16
// 32 heads 1034 -> 900 us, T=4096 D=64 4 heads 33.6 -> 33.1 ms, T=2048 D=128 16 heads 23.1 -> 22.6 ms; with row maxima T=512 D=128
// fp16 16 heads 812 -> 740 us, T=2048 D=64 4 heads 5.33 ms, same.  The code size matters: with the stages unrolled by tile and mode
// (165 to 235 KB for 115 to 140) the same changes were 4 to 15 % slower than before them.
// Causal structure: for a fixed query the mask is "j <= q" on columns and "k <= q" on rows, so
// whole slabs above q are never visited, only the last slab is masked (by a column bound that
// is uniform over the rows), and rows with k > q get weight zero in the fold.
#include "tritt_common.cuh"
#include "tritt_sm100.cuh"
#include "tritt_sm100_tdp_diag.cuh"

#include <type_traits>

namespace tritt {
namespace {
using namespace sm100;

constexpr int kThreads = 512;
constexpr int kBJ = 128;            // key columns per slab
constexpr float kRescaleGap = 8.f;  // rescale the accumulator only when the row max grew by more than 2^8

template <int D> struct FwdCfg {
  static constexpr int kTileA = 128 * D * 2;    // bytes of one 128-row tile (operand, K1 or SiLU(V1))
  static constexpr int kStages = 4;
  static constexpr int kOffAa = 0;
  static constexpr int kOffAb = kTileA;
  static constexpr int kOffRing = 2 * kTileA;
  static constexpr int kOffStats = kOffRing + kStages * kTileA;  // [2 parities][2 tiles][128][4] fp32: row (reference, two partial sums, -)
  static constexpr int kOffRed = kOffStats + 2 * 2 * 128 * 4 * 4;  // [2 tiles][4 warps][D] fp32 column sums
  static constexpr int kOffFstat = kOffRed + 2 * 4 * D * 4;        // [2 tiles][8] fp32 warp max / sum
  static constexpr int kOffNorm = kOffFstat + 2 * 8 * 4;            // [2 tiles][128] fp32: |A_row|^2
  static constexpr int kOffBars = kOffNorm + 2 * 128 * 4;
  static constexpr int kSmem = kOffBars + 256;
  static constexpr int kTmemO = 256;  // S_a | S_b | acc_a | acc_b
};

struct FwdParams {
  void* out;
  float* lse;
  const void *q, *v2;
  int T, BN, nq, q_mod, q_rem, causal, n_pairs;
  int k1w, k2w, kkl, kkr;  // windows of the causal mask (T or more = unbounded)
  float scale2;  // alpha * log2(e)
  const float* k1_norm2_max;  // [BN] largest squared row norm of K1 per head, or null (no score bound available)
  const float* q_norm2_max;   // [BN] largest squared row norm of Q per head (with k1_norm2_max)
  const float* k2_elem2_max;  // [BN] largest squared element of K2 per head (with k1_norm2_max)
  float bound_limit;          // rows whose score bound is below this skip the row-maximum pass
  int* status;
};

struct FwdBarriers {
  uint64_t ring_full[4], ring_empty[4];
  uint64_t k2_full, a_ready, a_free;
  uint64_t s_ready[2], p_ready[2];               // per tile, one phase per slab
  // Per k-tile hand-offs with the fold warpgroup.  stats_ready is doubled by k-tile parity: with one slab per k-tile
  // (short sequences, narrow windows) the soft-max warps can hand over the next k-tile's statistics before the fold
  // warpgroup, still storing the previous item, has looked at this one's, and a barrier two phases ahead of its waiter
  // reads as not ready for ever.
  uint64_t o_done[2], o_free[2], stats_ready[2][2];
  uint64_t fold_sync;
  uint32_t tmem_base;
  int abort_flag;
};

// A row's columns among 32, as a bit mask or as bounds.  The mask takes one instruction per element instead of two: forward
// at head dimension 64, T=512 1067 -> 1033 us, with the row-maximum pass 658 -> 621 us, T=4096 34.2 -> 33.6 ms.  At 128
// the bounds are the better form (T=2048 24.1 against 24.4 ms).
template <bool MASK> struct Columns {
  int lo, hi;
  uint32_t mask;
  __device__ __forceinline__ Columns(int l, int h) : lo(l), hi(h), mask(MASK ? column_mask(l, h) : 0u) {}
  __device__ __forceinline__ bool has(int c) const { return MASK ? (mask >> c & 1u) != 0 : c >= lo && c <= hi; }
};

// Fraction of the soft-max reference that all rows of a head with a small score bound share: -log2(29 / 32).  Scores near zero
// are the usual case, and their P, near 2^-reference, is then near 29 / 32 of a power of two: on the 16-bit grid, so that scores of
// zero are not rounded at all, and where the grid's step is small against the value.  At a power of two it is twice as coarse:
// error of the output against fp64 (bf16 T=64 D=64 / T=333 D=128) 2.90e-3 / 2.91e-3 with whole numbers, 2.57e-3 / 2.59e-3 with
// this or with each row's own bound as the reference.
constexpr float kReferenceFraction = 0.142019f;

template <int D, typename T16>
__global__ void __launch_bounds__(kThreads, 1)
tdp_fwd_kernel(const __grid_constant__ CUtensorMap tmK1, const __grid_constant__ CUtensorMap tmK2,
               const __grid_constant__ CUtensorMap tmSV1, FwdParams p) {
  using Cfg = FwdCfg<D>;
  constexpr int NS = Cfg::kStages;
  constexpr int KH = D / 64;  // 64-column halves per row
  extern __shared__ __align__(1024) uint8_t smem[];
  static_assert(sizeof(FwdBarriers) <= 256, "barrier block too large");
  FwdBarriers& bars = *reinterpret_cast<FwdBarriers*>(smem + Cfg::kOffBars);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (smem_u32(smem) & 1023u) {
    // swizzled tiles need 1024-byte alignment; uniform over the CTA, so every thread leaves here
    if (tid == 0 && p.status) atomicOr(p.status, 8);
    return;
  }

  if (tid == 0) {
    bars.abort_flag = 0;
    for (int i = 0; i < NS; ++i) {
      mbar_init(&bars.ring_full[i], 1);
      mbar_init(&bars.ring_empty[i], 1);
    }
    mbar_init(&bars.k2_full, 1);
    mbar_init(&bars.a_ready, 256);
    mbar_init(&bars.a_free, 256);
    for (int x = 0; x < 2; ++x) {
      mbar_init(&bars.s_ready[x], 1);
      mbar_init(&bars.p_ready[x], 256);
      mbar_init(&bars.o_free[x], 128);
      mbar_init(&bars.stats_ready[0][x], 256);
      mbar_init(&bars.stats_ready[1][x], 256);
      mbar_init(&bars.o_done[x], 1);
    }
    mbar_init(&bars.fold_sync, 128);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&bars.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;

  const int T = p.T;
  const long n_items = (long)p.n_pairs * p.BN;

  // Work item -> (head, query pair).  Items are ordered by decreasing cost (late queries first).
  auto decode = [&](long item, int& bh, int& qa, int& qb) {
    const int pr = p.n_pairs - 1 - (int)(item / p.BN);
    bh = (int)(item % p.BN);
    const int ia = 2 * pr, ib = min(2 * pr + 1, p.nq - 1);
    qa = p.q_rem + ia * p.q_mod;
    qb = p.q_rem + ib * p.q_mod;
  };
  // Tiles a query pair visits (qa <= qb).  Causal mask: j <= q <= j + k1w, k <= q <= k + k2w, k - kkl <= j <= k + kkr.
  // k-tiles: rows k in [max(0, qa - k2w, qa - k1w - kkr), qb]  (rows below the third bound see no column at all);
  // slabs of k-tile kt: columns j in [max(0, qa - k1w, k_first - kkl), min(qb, k_last + kkr)], never empty.
  auto k_range = [&](int qa, int qb, int& kt0, int& nkt) {
    if (!p.causal) {
      kt0 = 0;
      nkt = (T + 127) / 128;
      return;
    }
    const int klo = max(0, max(qa - p.k2w, qa - p.k1w - p.kkr));
    kt0 = klo / 128;
    nkt = qb / 128 - kt0 + 1;
  };
  auto j_range = [&](int qa, int qb, int kt, int& jt0, int& njt) {
    if (!p.causal) {
      jt0 = 0;
      njt = (T + kBJ - 1) / kBJ;
      return;
    }
    const int klo = max(0, max(qa - p.k2w, qa - p.k1w - p.kkr));
    const int ka = max(kt * 128, klo), kb = min(kt * 128 + 127, qb);
    const int ja = max(0, max(qa - p.k1w, ka - p.kkl)), jb = min(qb, kb + p.kkr);
    jt0 = ja / kBJ;
    njt = jb / kBJ - jt0 + 1;
  };
  // Attended columns of k-tile kt (union over its rows): [ja, jb].  A slab whose attended columns all lie in one
  // 64-column half (halves() = 1: the lower, 2: the upper, 0: both) runs as 128 x 64 score products and a 64-deep
  // value product.
  auto col_span = [&](int qa, int qb, int kt, int& ja, int& jb) {
    ja = 0;
    jb = T - 1;
    if (p.causal) {
      const int klo = max(0, max(qa - p.k2w, qa - p.k1w - p.kkr));
      const int ka = max(kt * 128, klo), kb = min(kt * 128 + 127, qb);
      ja = max(0, max(qa - p.k1w, ka - p.kkl));
      jb = min(qb, kb + p.kkr);
    }
  };
  auto halves = [](int ja, int jb, int j0) { return jb < j0 + 64 ? 1 : (ja >= j0 + 64 ? 2 : 0); };
  // How the soft-max warps divide a head's work.  Every score of the head is bounded by
  // |s| max_q |Q_q| max |K2 element| max_j |K1_j|  (|A_row|^2 = s^2 sum_h Q_h^2 K2_h^2 <= s^2 max_h K2_h^2 |Q_q|^2).
  // Where that is below the limit, all rows of the head have one soft-max reference (head_reference: one pass, nothing to agree on
  // between threads, nothing to merge between tiles) and the two warpgroups split every slab's columns; otherwise each warpgroup
  // owns one tile and a thread its whole row (maximum pass, rescaling).  Uniform over a work item, read by every role.
  auto head_bound = [&](int bh) -> float {
    if (!p.k1_norm2_max) return INFINITY;
    return fabsf(p.scale2) * sqrtf(__ldg(p.q_norm2_max + bh)) * sqrtf(__ldg(p.k2_elem2_max + bh)) * sqrtf(__ldg(p.k1_norm2_max + bh));
  };
  auto head_split = [&](int bh) -> bool { return head_bound(bh) <= p.bound_limit; };
  // From the head's own bound: with the limit for all heads P of small scores would be 2^-40 in bf16, and the fold's products of
  // it with values of 1e-13 below fp32's smallest normal number.
  auto head_reference = [&](int bh) -> float { return ceilf(head_bound(bh)) + kReferenceFraction; };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // (the whole warp walks the schedule converged, one elected lane issues the copies)
    {
      const bool leader = elect_one();
      if (leader) {
        tma_prefetch_desc(&tmK1);
        tma_prefetch_desc(&tmK2);
        tma_prefetch_desc(&tmSV1);
      }
      uint32_t kt_count = 0, pos = 0;
      bool alive = true;
      auto load_stage = [&](const CUtensorMap* tm, int row0, int bh) -> bool {
        const int st = pos % NS;
        if (!__all_sync(0xffffffffu, mbar_wait(&bars.ring_empty[st], ((pos / NS) & 1) ^ 1, abort_flag))) return false;
        if (leader) {
          mbar_arrive_expect_tx(&bars.ring_full[st], Cfg::kTileA);
          for (int hh = 0; hh < KH; ++hh)
            tma_load_3d(smem + Cfg::kOffRing + st * Cfg::kTileA + hh * 16384, tm, &bars.ring_full[st], hh * 64, row0, bh);
        }
        ++pos;
        return true;
      };
      for (long item = blockIdx.x; item < n_items && alive; item += gridDim.x) {
        int bh, qa, qb, kt0, nkt;
        decode(item, bh, qa, qb);
        k_range(qa, qb, kt0, nkt);
        for (int kt = kt0; kt < kt0 + nkt && alive; ++kt, ++kt_count) {
          int jt0, njt;
          j_range(qa, qb, kt, jt0, njt);
          // the first K1 tile does not depend on the previous k-tile: fetch it before waiting for the operand buffer
          alive = load_stage(&tmK1, jt0 * kBJ, bh);
          if (!alive || !__all_sync(0xffffffffu, mbar_wait(&bars.a_free, (kt_count & 1) ^ 1, abort_flag))) {
            alive = false;
            break;
          }
          if (leader) {
            mbar_arrive_expect_tx(&bars.k2_full, Cfg::kTileA);
            for (int hh = 0; hh < KH; ++hh)
              tma_load_3d(smem + Cfg::kOffAa + hh * 16384, &tmK2, &bars.k2_full, hh * 64, kt * 128, bh);
          }
          // ring order: K1(0), V(0), K1(1), V(1), ...
          for (int jt = jt0; jt < jt0 + njt && alive; ++jt) {
            alive = load_stage(&tmSV1, jt * kBJ, bh);
            if (alive && jt + 1 < jt0 + njt) alive = load_stage(&tmK1, (jt + 1) * kBJ, bh);
          }
        }
      }
      if (!alive) {
        // give copies still in flight a bounded chance to land before the CTA retires
        const uint32_t first = pos > (uint32_t)NS ? pos - NS : 0;
        for (uint32_t q2 = first; q2 < pos; ++q2) {
          const long long t0 = clock64();
          while (!mbar_try_wait(&bars.ring_full[q2 % NS], (q2 / NS) & 1) && clock64() - t0 < kWaitTicks / 8) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the schedule in step and one elected lane issues: with converged control flow the
    // descriptor arithmetic stays on the uniform datapath, where a lone thread needs a register-to-uniform move per
    // operand and loses its issue slots to the busy warps of its scheduler.
    {
      const bool leader = elect_one();
      // (every lane waits; the vote keeps the warp converged whatever a lane's wait returned)
      auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
      };
      auto commit = [&](uint64_t* bar) {
        if (leader) mma_commit(bar);
      };
      constexpr int kFmt = std::is_same<T16, __nv_bfloat16>::value ? 1 : 0;
      constexpr uint32_t idesc_s = make_idesc_f16(128, kBJ, kFmt, false, false);
      constexpr uint32_t idesc_pv = make_idesc_f16(128, D, kFmt, false, true);
      // descriptor low words; per instruction only a constant (in 16-byte units) is added
      constexpr uint32_t kHi = desc_hi(1024);
      constexpr uint32_t kTile16 = Cfg::kTileA >> 4;
      const uint32_t aLo[2] = {desc_lo(smem_u32(smem + Cfg::kOffAa), 16), desc_lo(smem_u32(smem + Cfg::kOffAb), 16)};
      const uint32_t ringK = desc_lo(smem_u32(smem + Cfg::kOffRing), 16);      // K-major view of a stage
      const uint32_t ringMN = desc_lo(smem_u32(smem + Cfg::kOffRing), 16384);  // row-major (MN-major) view
      uint32_t kt_count = 0, base = 0, n = 0;  // n: slabs finished so far (same for both tiles)
      bool alive = true;
      auto wait_full = [&](uint32_t pos) {
        return wait_all(&bars.ring_full[pos % NS], (pos / NS) & 1);
      };
      auto release = [&](uint32_t pos) { commit(&bars.ring_empty[pos % NS]); };
      // S_x = A_x * K1tile^T  (one chain of D/16 instructions); hm != 0: only 64 rows of the key tile (the lower
      // or the upper ones), scores in the first 64 columns of S_x
      constexpr uint32_t idesc_s64 = make_idesc_f16(128, 64, kFmt, false, false);
      auto issue_s = [&](int x, uint32_t pos, int hm) {
        const uint32_t bLo = ringK + (pos % NS) * kTile16;
        if (hm == 0) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t kk = (k >> 2) * (16384 >> 4) + (k & 3) * 2;
            if (leader) mma_ss_lo(tmem + x * kBJ, aLo[x] + kk, bLo + kk, kHi, idesc_s, k > 0);
          }
        } else {
          const uint32_t bRow = bLo + (hm == 2 ? (64 * 128) >> 4 : 0);   // rows 64.. of a 128-byte-pitch block
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t kk = (k >> 2) * (16384 >> 4) + (k & 3) * 2;
            if (leader) mma_ss_lo(tmem + x * kBJ, aLo[x] + kk, bRow + kk, kHi, idesc_s64, k > 0);
          }
        }
        commit(&bars.s_ready[x]);
      };
      // acc_x (+)= P_x * SiLU(V1)tile  (one chain of 8 instructions; P_x overlays the first 64 columns of S_x);
      // hm != 0: P_x has 64 columns (4 instructions) and meets the lower or upper 64 rows of the value tile
      // (split: P of a warpgroup's columns sits over the first half of them; otherwise over the first 64 columns of S_x)
      auto issue_pv = [&](int x, uint32_t pos, uint32_t acc, int hm, bool split) {
        const uint32_t bLo = ringMN + (pos % NS) * kTile16;
        if (hm == 0) {
#pragma unroll
          for (int k = 0; k < kBJ / 16; ++k)
            if (leader)
              mma_ts_lo(tmem + Cfg::kTmemO + x * D, tmem + x * kBJ + (split ? (k >> 2) * 64 + (k & 3) * 8 : k * 8),
                      bLo + k * (2048 >> 4), kHi, idesc_pv, k > 0 ? 1u : acc);
        } else {
          const uint32_t bRow = bLo + (hm == 2 ? (4 * 2048) >> 4 : 0);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (leader)
              mma_ts_lo(tmem + Cfg::kTmemO + x * D, tmem + x * kBJ + (split ? (k >> 1) * 32 + (k & 1) * 8 : k * 8),
                      bRow + k * (2048 >> 4), kHi, idesc_pv, k > 0 ? 1u : acc);
        }
      };

      // Each tile's end is told to the fold warps as it comes (head dimension 128: T=1024 fp16 8 heads 3.54 ms against 3.56 with both
      // at the end of the k-tile, T=2048 16 heads 22.6 against 22.7), or both at the end (64: the loop over the slabs is shorter by
      // it, T=2048 with large scores 5.33 against 5.42 ms, fp16 6.03 against 6.14, T=512 32 heads 900 against 911 us).
      constexpr bool kDoneByTile = D == 128;
      for (long item = blockIdx.x; item < n_items && alive; item += gridDim.x) {
        int bh, qa, qb, kt0, nkt;
        decode(item, bh, qa, qb);
        k_range(qa, qb, kt0, nkt);
        const bool split = head_split(bh);
        for (int kt = kt0; kt < kt0 + nkt && alive; ++kt, ++kt_count) {
          int jt0, njt;
          j_range(qa, qb, kt, jt0, njt);
          if (!wait_all(&bars.a_ready, kt_count & 1)) { alive = false; break; }
          tc_fence_after();
          if (!wait_full(base)) { alive = false; break; }
          int ja, jb;
          col_span(qa, qb, kt, ja, jb);
          int hm = halves(ja, jb, jt0 * kBJ);
          issue_s(0, base, hm);
          issue_s(1, base, hm);
          release(base);
          for (int jt = 0; jt < njt && alive; ++jt, ++n) {
            const uint32_t pv = base + 2 * jt + 1, pk = base + 2 * jt + 2;
            const bool more = jt + 1 < njt;
            const int hm_next = more ? halves(ja, jb, (jt0 + jt + 1) * kBJ) : 0;
            for (int x = 0; x < 2 && alive; ++x) {
              if (!wait_all(&bars.p_ready[x], n & 1)) { alive = false; break; }
              if (jt == 0) {
                // the fold warpgroup must have drained the previous k-tile's accumulator of this tile
                if (!wait_all(&bars.o_free[x], (kt_count & 1) ^ 1)) { alive = false; break; }
              }
              tc_fence_after();
              if (x == 0 && !wait_full(pv)) { alive = false; break; }
              issue_pv(x, pv, jt > 0, hm, split);
              if (kDoneByTile && !more) commit(&bars.o_done[x]);
              if (x == 1) release(pv);
              if (more) {
                if (x == 0 && !wait_full(pk)) { alive = false; break; }
                issue_s(x, pk, hm_next);
                if (x == 1) release(pk);
              }
            }
            hm = hm_next;
          }
          if (!kDoneByTile && alive) {
            commit(&bars.o_done[0]);
            commit(&bars.o_done[1]);
          }
          base += 2 * njt;
        }
      }
    }
  } else if (warp >= 4 && warp < 12) {
    // ------------------------------------------------------------------ soft-max warpgroups
    // Both warpgroups work on the same slab, tile a first, then tile b: warpgroup `wg` takes the slab's columns
    // [wg * 64, wg * 64 + 64) (32 of a half-width slab's 64), one row per thread, and writes P over the first half of
    // the columns it has read.  While they are on one tile, the tensor pipe runs the other tile's two products.
    const int wg = (warp - 4) >> 2;         // column half of every slab
    const int wq = warp & 3;                // TMEM lane quadrant of this warp
    const int row = wq * 32 + lane;         // row of both tiles owned by this thread
    const int st = tid - 128;               // 0..255 over both warpgroups
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    float* stats = (float*)(smem + Cfg::kOffStats);
    float* norms = (float*)(smem + Cfg::kOffNorm);
    uint32_t kt_count = 0, n = 0;
    bool alive = true;

    // largest score of this thread's NC columns at TMEM address tS ([lo, hi]: the columns the row may see)
    auto row_max = [&](auto nc, uint32_t tS, bool full, int lo, int hi) -> float {
      constexpr int NC = decltype(nc)::value;
      uint32_t sr[NC];
      if constexpr (NC == 64) tmem_ld64(tS, sr); else tmem_ld32(tS, sr);
      tmem_wait_ld();
      float mx = -INFINITY;
      if (full) {
        // four independent chains instead of one NC-deep dependency
        float m0 = __uint_as_float(sr[0]), m1 = __uint_as_float(sr[1]), m2 = __uint_as_float(sr[2]),
              m3 = __uint_as_float(sr[3]);
#pragma unroll
        for (int c = 4; c < NC; c += 4) {
          m0 = fmaxf(m0, __uint_as_float(sr[c]));
          m1 = fmaxf(m1, __uint_as_float(sr[c + 1]));
          m2 = fmaxf(m2, __uint_as_float(sr[c + 2]));
          m3 = fmaxf(m3, __uint_as_float(sr[c + 3]));
        }
        mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      } else {
#pragma unroll
        for (int c32 = 0; c32 < NC; c32 += 32) {
          const Columns<D == 64> cols(lo - c32, hi - c32);
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (cols.has(c)) mx = fmaxf(mx, __uint_as_float(sr[c32 + c]));
        }
      }
      return mx;
    };
    // P = exp2(S - m) of this thread's NC columns, packed to 16 bits over the first NC / 2 of them; returns their sum
    // (written at tP, which lies within columns this thread has read)
    auto form_p = [&](auto nc, uint32_t tS, uint32_t tP, bool full, int lo, int hi, float m) -> float {
      constexpr int NC = decltype(nc)::value;
      uint32_t sr[NC];
      if constexpr (NC == 64) tmem_ld64(tS, sr); else tmem_ld32(tS, sr);
      tmem_wait_ld();
      uint32_t pk[NC / 2];
      float ps0 = 0.f, ps1 = 0.f;
      if (full) {
        // packed fp32 pairs: one subtraction and one addition per two scores
        const float2 nm = make_float2(-m, -m);
        float2 pa = make_float2(0.f, 0.f), pb = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < NC; c += 4) {
          const float2 x0 = __fadd2_rn(make_float2(__uint_as_float(sr[c]), __uint_as_float(sr[c + 1])), nm);
          const float2 x1 = __fadd2_rn(make_float2(__uint_as_float(sr[c + 2]), __uint_as_float(sr[c + 3])), nm);
          const float2 e0 = make_float2(exp2f(x0.x), exp2f(x0.y));
          const float2 e1 = make_float2(exp2f(x1.x), exp2f(x1.y));
          pa = __fadd2_rn(pa, e0);
          pb = __fadd2_rn(pb, e1);
          pk[c >> 1] = pack2<T16>(e0.x, e0.y);
          pk[(c >> 1) + 1] = pack2<T16>(e1.x, e1.y);
        }
        ps0 = pa.x + pb.x;
        ps1 = pa.y + pb.y;
      } else {
        // (a row with no valid column so far has m = -inf and selects 0 everywhere)
        const float2 nm = make_float2(-m, -m);
        float2 pa = make_float2(0.f, 0.f);
#pragma unroll
        for (int c32 = 0; c32 < NC; c32 += 32) {
          const Columns<D == 64> cols(lo - c32, hi - c32);
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            const float2 x =
                __fadd2_rn(make_float2(__uint_as_float(sr[c32 + c]), __uint_as_float(sr[c32 + c + 1])), nm);
            const float2 e = make_float2(cols.has(c) ? exp2f(x.x) : 0.f, cols.has(c + 1) ? exp2f(x.y) : 0.f);
            pa = __fadd2_rn(pa, e);
            pk[(c32 + c) >> 1] = pack2<T16>(e.x, e.y);
          }
        }
        ps0 = pa.x;
        ps1 = pa.y;
      }
      tmem_st(tP, pk);
      return ps0 + ps1;
    };

    for (long item = blockIdx.x; item < n_items && alive; item += gridDim.x) {
      int bh, qa, qb, kt0, nkt;
      decode(item, bh, qa, qb);
      k_range(qa, qb, kt0, nkt);
      const T16* Qg = (const T16*)p.q + (size_t)bh * T * D;
      // largest K1 row norm of this head: with |A_row| it bounds every score of the row (Cauchy-Schwarz)
      const float k1_max = p.k1_norm2_max ? sqrtf(__ldg(p.k1_norm2_max + bh)) : INFINITY;
      // The item's k-tiles, one copy of the code for each organisation: with one copy for both, neither had the registers and the
      // schedule of its own (T=512 D=64 32 heads 928 us against 900, T=557 fp16 not causal with large scores 3.70 ms against 3.60).
      auto walk = [&](auto split_c) {
        constexpr bool kSplit = decltype(split_c)::value;
        // (every lane has the same value; the reduction leaves it in a uniform register)
        const float reference = kSplit ? __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(head_reference(bh)))) : 0.f;
        for (int kt = kt0; kt < kt0 + nkt && alive; ++kt, ++kt_count) {
          int jt0, njt, ja, jb;
          j_range(qa, qb, kt, jt0, njt);
          col_span(qa, qb, kt, ja, jb);
          // Columns this row may see, per tile: [c_lo, c_hi].  A row outside the k range of its query (its weight in
          // the fold is zero) keeps the query's own column range so that it never sees an empty one by construction;
          // a row inside can still see none in a slab, or at all: its maximum then stays -inf and its P zero.
          int c_lo[2] = {0, 0}, c_hi[2] = {T - 1, T - 1};
          if (p.causal) {
            const int k_r = kt * 128 + row;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int qx = x == 0 ? qa : qb;
              const bool in_k = k_r <= qx && qx - k_r <= p.k2w;
              c_lo[x] = max(qx - p.k1w, in_k ? k_r - p.kkl : 0);
              c_hi[x] = in_k ? min(qx, k_r + p.kkr) : qx;
            }
          }
          // ---- operand formation: A_a = s*Q[qa] (.) K2tile (in place), A_b = s*Q[qb] (.) K2tile
          constexpr int kCols = D / 8, kRowStep = 256 / kCols;
          const int col = st % kCols;
          const uint32_t off0 = (col >> 3) * 16384 + swz128(st / kCols, col & 7);
          float2 qv[2][4];   // this thread's columns of the two queries
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(Qg + (size_t)(x ? qb : qa) * D + col * 8));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) qv[x][e] = unpack2<T16>(w[e]);
          }
          alive = __all_sync(0xffffffffu, mbar_wait(&bars.k2_full, kt_count & 1, abort_flag));
          if (!alive) break;
          // A thread has one 16-byte column of every (256 / kCols)-th row.  (The backward forms the same products in the same
          // order for large scores, where a rounding the other way would show.)
          {
#pragma unroll 2
            for (int i = 0; i < 128 / kRowStep; ++i) {
              const uint32_t off = off0 + i * kRowStep * 128;
              const uint4 kv = *reinterpret_cast<const uint4*>(smem + Cfg::kOffAa + off);
              const uint32_t w[4] = {kv.x, kv.y, kv.z, kv.w};
              uint32_t a[2][4];
              float nr[2] = {0.f, 0.f};   // this thread's share of |A_a[r]|^2 and |A_b[r]|^2
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 f = __fmul2_rn(unpack2<T16>(w[e]), make_float2(p.scale2, p.scale2));
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                  const float2 g = __fmul2_rn(f, qv[x][e]);
                  a[x][e] = pack2<T16>(g.x, g.y);
                  if constexpr (!kSplit) nr[x] = fmaf(g.x, g.x, fmaf(g.y, g.y, nr[x]));
                }
              }
              *reinterpret_cast<uint4*>(smem + Cfg::kOffAa + off) = make_uint4(a[0][0], a[0][1], a[0][2], a[0][3]);
              *reinterpret_cast<uint4*>(smem + Cfg::kOffAb + off) = make_uint4(a[1][0], a[1][1], a[1][2], a[1][3]);
              if constexpr (!kSplit) {
                // (read by the owner of the row after its first s_ready wait of this k-tile, which this thread's
                //  a_ready arrival below precedes; rewritten only after it has passed a_free)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
#pragma unroll
                  for (int o = kCols / 2; o >= 1; o >>= 1) nr[x] += __shfl_xor_sync(0xffffffffu, nr[x], o);
                  if (col == 0) norms[x * 128 + st / kCols + i * kRowStep] = nr[x];
                }
              }
            }
          }
          fence_async_smem();   // generic-proxy stores above -> visible to the tensor core's reads
          mbar_arrive(&bars.a_ready);

          if constexpr (kSplit) {
            // ---- walk over the slabs, both warpgroups on the same slab: tile a, then tile b; warpgroup `wg` takes the
            // slab's columns [wg * 64, wg * 64 + 64) (32 of a half-width slab's 64).  The reference of every row is the head's: with
            // a bound b of the scores P stays within [2^-(2 b + 1.15), 1], representable in the 16-bit type, and no row maximum is
            // needed.
            // (The head's own bound instead of a launch parameter costs 1 to 2 % at head dimension 128, T=2048 16
            // heads 22.4 -> 22.7 ms, and nothing at 64.)
            float l_sum[2] = {0.f, 0.f};
            for (int jt = 0; jt < njt && alive; ++jt, ++n) {
              // A slab with attended columns in one 64-column half only was computed for that half alone: its scores
              // are in the first 64 columns of S_x and stand for the slab's columns [coff, coff + 64).
              const int hm = halves(ja, jb, (jt0 + jt) * kBJ);
              const int nh = hm ? 1 : 2, coff = hm == 2 ? 64 : 0;
              const int cw = 32 * nh;                                  // columns of this warpgroup in this slab
              const int j0 = (jt0 + jt) * kBJ + coff + wg * cw;      // its first column
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                alive = __all_sync(0xffffffffu, mbar_wait(&bars.s_ready[x], n & 1, abort_flag));
                if (!alive) break;
                tc_fence_after();
                // the last score product of this k-tile has read A_a and A_b
                if (x == 1 && jt == njt - 1) mbar_arrive(&bars.a_free);
                const uint32_t tS = tmem + lane_base + x * kBJ + wg * cw;
                // this row's valid columns among the warpgroup's: [lo, hi]; the warp takes the unmasked code when all
                // its rows see all of them
                const int lo = c_lo[x] - j0, hi = c_hi[x] - j0;
                const bool full = __all_sync(0xffffffffu, lo <= 0 && hi >= cw - 1);
                // P over the first half of the columns this thread has read
                l_sum[x] += nh == 2 ? form_p(std::integral_constant<int, 64>{}, tS, tS, full, lo, hi, reference)
                                    : form_p(std::integral_constant<int, 32>{}, tS, tS, full, lo, hi, reference);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bars.p_ready[x]);
              }
            }
            if (!alive) break;
            // ---- hand this k-tile's row sums to the fold warpgroup
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              stats[(((kt_count & 1) * 2 + x) * 128 + row) * 4 + 1 + wg] = l_sum[x];
              mbar_arrive(&bars.stats_ready[kt_count & 1][x]);
            }
          } else {
            // ---- walk over the slabs, one warpgroup per tile (warpgroup 0: tile a), one whole row per thread: row
            // maximum, exp2 with lazy rescaling of the accumulator.  A warp whose rows all have a score bound below the
            // limit still uses the bound as reference and skips the maximum pass.  (Arrivals count twice: the barriers
            // expect both warpgroups.)
            const int x = wg;
            const int c_lo_x = x ? c_lo[1] : c_lo[0], c_hi_x = x ? c_hi[1] : c_hi[0];
            const uint32_t tS = tmem + lane_base + x * kBJ;
            float m_used = -INFINITY, l_sum = 0.f;
            bool fast = false;
            for (int jt = 0; jt < njt && alive; ++jt, ++n) {
              alive = __all_sync(0xffffffffu, mbar_wait(&bars.s_ready[x], n & 1, abort_flag));
              if (!alive) break;
              tc_fence_after();
              if (jt == 0) {
                const float bound = sqrtf(norms[x * 128 + row]) * k1_max;
                fast = __all_sync(0xffffffffu, bound <= p.bound_limit);
                if (fast) m_used = bound;
              }
              if (jt == njt - 1) mbar_arrive(&bars.a_free);  // the last score product of this k-tile has read A_x
              const int hm = halves(ja, jb, (jt0 + jt) * kBJ);
              const int nh = hm ? 1 : 2, coff = hm == 2 ? 64 : 0;
              const int j0 = (jt0 + jt) * kBJ + coff;
              const int lo = c_lo_x - j0, hi = c_hi_x - j0;
              const bool full = __all_sync(0xffffffffu, lo <= 0 && hi >= 64 * nh - 1);
              using N64 = std::integral_constant<int, 64>;
              if (!fast) {
                // pass 1: row maximum
                float mx = row_max(N64{}, tS, full, lo, hi);
                if (nh == 2) mx = fmaxf(mx, row_max(N64{}, tS + 64, full, lo - 64, hi - 64));
                if (jt == 0) {
                  m_used = mx;  // nothing accumulated yet in this k-tile
                } else {
                  const bool grow = mx > m_used + kRescaleGap;
                  if (__any_sync(0xffffffffu, grow)) {
                    // some row of this warp moved its max up noticeably: rescale accumulator rows (factor 1 for the
                    // rows that did not move)
                    const float corr = grow ? exp2f(m_used - mx) : 1.f;
                    if (grow) {
                      m_used = mx;
                      l_sum *= corr;
                    }
                    // (s_ready of this slab was committed after the previous P*V, so that product has landed)
                    const uint32_t tO = tmem + lane_base + Cfg::kTmemO + x * D;
#pragma unroll
                    for (int ch = 0; ch < D / 32; ++ch) {
                      uint32_t o[32];
                      tmem_ld32(tO + ch * 32, o);
                      tmem_wait_ld();
#pragma unroll
                      for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                      tmem_st32(tO + ch * 32, o);
                    }
                  }
                }
              }
              // pass 2: P = exp2(S - m), packed to 16 bits over the columns already consumed
              l_sum += form_p(N64{}, tS, tS, full, lo, hi, m_used);
              if (nh == 2) l_sum += form_p(N64{}, tS + 64, tS + 32, full, lo - 64, hi - 64, m_used);
              tmem_wait_st();
              tc_fence_before();
              mbar_arrive_n(&bars.p_ready[x], 2);
            }
            if (!alive) break;
            // ---- hand this k-tile's row statistics to the fold warpgroup
            float* srow = stats + (((kt_count & 1) * 2 + x) * 128 + row) * 4;
            srow[0] = m_used;
            srow[1] = l_sum;
            srow[2] = 0.f;
            mbar_arrive_n(&bars.stats_ready[kt_count & 1][x], 2);
          }
        }
      };
      if (head_split(bh)) walk(std::true_type{});
      else walk(std::false_type{});
      if (!alive) break;
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ fold warpgroup
    // After the last P*V of a k-tile: O[q_x,h] accumulates sum_r w_r acc_x[r,h] V2[k_r,h] with
    // w_r = 2^(m_r - M) over the valid rows, merged into the query's running (max, sum, output).
    const int wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const float* stats = (const float*)(smem + Cfg::kOffStats);
    float* red = (float*)(smem + Cfg::kOffRed);      // [2][4][D]
    float* fstat = (float*)(smem + Cfg::kOffFstat);  // [2][8]
    uint32_t kt_count = 0, sync_phase = 0;
    bool alive = true;
    auto fold_sync = [&]() -> bool {
      mbar_arrive(&bars.fold_sync);
      const bool ok = mbar_wait(&bars.fold_sync, sync_phase & 1, abort_flag);
      ++sync_phase;
      return __all_sync(0xffffffffu, ok);
    };
    for (long item = blockIdx.x; item < n_items && alive; item += gridDim.x) {
      int bh, qa, qb, kt0, nkt;
      decode(item, bh, qa, qb);
      k_range(qa, qb, kt0, nkt);
      const T16* V2g = (const T16*)p.v2 + (size_t)bh * T * D;
      if (head_split(bh)) {
        // ---- every row has the same reference, so the k-tiles' sums just add up: sum_r acc_x[r,h] V2[k_r,h] over the rows a
        // thread reads as 16 x 256-bit fragments (rows lane / 4 + 8 i, column pairs 2 (lane % 4) + 8 g), kept in registers to the
        // end of the item: no exchange between threads per k-tile.  (One copy of the code for both tiles: their sums change
        // places after each.)
        float2 o[D / 8], other[D / 8];
        float l = 0.f, l_other = 0.f;
        auto swap_tiles = [&]() {
#pragma unroll
          for (int i = 0; i < D / 8; ++i) {
            const float2 keep = o[i];
            o[i] = other[i];
            other[i] = keep;
          }
          const float keep = l;
          l = l_other;
          l_other = keep;
        };
#pragma unroll
        for (int i = 0; i < D / 8; ++i) o[i] = other[i] = make_float2(0.f, 0.f);
        auto valid = [&](int k, int q) { return p.causal ? k <= q && q - k <= p.k2w : k < T; };
        for (int kt = kt0; kt < kt0 + nkt && alive; ++kt, ++kt_count) {
          const uint32_t par = kt_count & 1;
#pragma unroll 1
          for (int x = 0; x < 2; ++x) {
            const int qx = x ? qb : qa;
            // V2 rows (r: 16-row half, row of the pair); a row outside the query's range counts as zero
            const T16* v2r[4];
            bool ok[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const int k = kt * 128 + wq * 32 + (r >> 1) * 16 + (r & 1) * 8 + (lane >> 2);
              ok[r] = valid(k, qx);
              v2r[r] = V2g + (size_t)min(k, T - 1) * D + 2 * (lane & 3);
            }
            constexpr int kC = 16;   // columns whose V2 words are fetched together, ahead of the accumulator
            uint32_t v2w[kC / 8][4];
            auto fetch = [&](int c0) {
#pragma unroll
              for (int g = 0; g < kC / 8; ++g)
#pragma unroll
                for (int r = 0; r < 4; ++r) v2w[g][r] = __ldg(reinterpret_cast<const uint32_t*>(v2r[r] + c0 + g * 8));
            };
            fetch(0);
            alive = __all_sync(0xffffffffu, mbar_wait(&bars.o_done[x], par, abort_flag));
            if (!alive) break;
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < D; c0 += kC) {
              uint32_t d[kC / 16][2][8];
#pragma unroll
              for (int c16 = 0; c16 < kC / 16; ++c16)
#pragma unroll
                for (int hl = 0; hl < 2; ++hl)
                  tmem_ld_16x256b_x2(tmem + lane_base + ((uint32_t)(hl * 16) << 16) + Cfg::kTmemO + x * D + c0 + c16 * 16, d[c16][hl]);
              float2 v[kC / 8][4];
#pragma unroll
              for (int g = 0; g < kC / 8; ++g)
#pragma unroll
                for (int r = 0; r < 4; ++r) v[g][r] = unpack2<T16>(ok[r] ? v2w[g][r] : 0u);
              if (c0 + kC < D) fetch(c0 + kC);
#pragma unroll
              for (int c16 = 0; c16 < kC / 16; ++c16) tmem_wait_ld(d[c16][0], d[c16][1]);
#pragma unroll
              for (int g = 0; g < kC / 8; ++g)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                  const uint32_t* f = d[g >> 1][r >> 1] + (g & 1) * 4 + (r & 1) * 2;
                  float2& a = o[c0 / 8 + g];
                  a = __ffma2_rn(make_float2(__uint_as_float(f[0]), __uint_as_float(f[1])), v[g][r], a);
                }
            }
            alive = __all_sync(0xffffffffu, mbar_wait(&bars.stats_ready[par][x], (kt_count >> 1) & 1, abort_flag));
            if (!alive) break;
            const float* srow = stats + ((par * 2 + x) * 128 + row) * 4;
            if (valid(kt * 128 + row, qx)) l += srow[1] + srow[2];
            // accumulator and statistics have been read: both may be overwritten (the statistics two k-tiles on, whose scores
            // follow the next k-tile's values)
            tc_fence_before();
            mbar_arrive(&bars.o_free[x]);
            swap_tiles();
          }
        }
        if (!alive) break;
        // ---- sums over the warp's rows (a tree over lane / 4) and over the warps, then the two output rows
#pragma unroll 1
        for (int x = 0; x < 2; ++x) {
          float z[D / 4];
#pragma unroll
          for (int i = 0; i < D / 8; ++i) {
            z[2 * i] = o[i].x;
            z[2 * i + 1] = o[i].y;
          }
#pragma unroll
          for (int b = 16, half = D / 8; b >= 4; b >>= 1, half >>= 1) {
            const bool upper = lane & b;
#pragma unroll
            for (int i = 0; i < half; ++i) {
              const float keep = upper ? z[i + half] : z[i], send = upper ? z[i] : z[i + half];
              z[i] = keep + __shfl_xor_sync(0xffffffffu, send, b);
            }
          }
          // z[i]: element f = (lane bits 4, 3, 2) * D / 32 + i of the thread's columns 8 (f / 2) + 2 (lane % 4) + f % 2
#pragma unroll
          for (int i = 0; i < D / 32; i += 2) {
            const int f = (((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)) * (D / 32) + i;
            *reinterpret_cast<float2*>(red + (x * 4 + wq) * D + 8 * (f >> 1) + 2 * (lane & 3)) = make_float2(z[i], z[i + 1]);
          }
#pragma unroll
          for (int b = 16; b >= 1; b >>= 1) l += __shfl_xor_sync(0xffffffffu, l, b);
          if (lane == 0) fstat[x * 8 + wq] = l;
          swap_tiles();
        }
        if (!fold_sync()) { alive = false; break; }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float L = fstat[x * 8] + fstat[x * 8 + 1] + fstat[x * 8 + 2] + fstat[x * 8 + 3];
          const int qx = x == 0 ? qa : qb;
          if (row < D) {
            const float O = red[(x * 4) * D + row] + red[(x * 4 + 1) * D + row] + red[(x * 4 + 2) * D + row] + red[(x * 4 + 3) * D + row];
            ((T16*)p.out)[((size_t)bh * T + qx) * D + row] = from_f<T16>(O / L);
          }
          if (row == 0) p.lse[(size_t)bh * T + qx] = (head_reference(bh) + log2f(L)) * kLn2;
        }
        if (!fold_sync()) { alive = false; break; }  // red / fstat are rewritten by the next item
        continue;
      }
      // running state per tile; thread `row` (< D) owns output column h = row
      float M_run[2] = {-INFINITY, -INFINITY}, L_run[2] = {0.f, 0.f}, O_run[2] = {0.f, 0.f};
      for (int kt = kt0; kt < kt0 + nkt && alive; ++kt, ++kt_count) {
        const int k_r = kt * 128 + row;
        const uint32_t par = kt_count & 1;
        // row statistics of both tiles
        float m_r[2], l_r[2];
        bool valid[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          alive = alive && __all_sync(0xffffffffu, mbar_wait(&bars.stats_ready[par][x], (kt_count >> 1) & 1, abort_flag));
          if (!alive) break;
          const float* srow = stats + ((par * 2 + x) * 128 + row) * 4;
          m_r[x] = srow[0];
          l_r[x] = srow[1] + srow[2];
          const int qx = x == 0 ? qa : qb;
          valid[x] = p.causal ? (k_r <= qx && qx - k_r <= p.k2w) : (k_r < T);
          float wm = valid[x] ? m_r[x] : -INFINITY;
#pragma unroll
          for (int o = 16; o >= 1; o >>= 1) wm = fmaxf(wm, __shfl_xor_sync(0xffffffffu, wm, o));
          if (lane == 0) fstat[x * 8 + wq] = wm;
        }
        if (!alive) break;
        if (!fold_sync()) { alive = false; break; }
        float Mt[2], w[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          // -inf when no row of this tile saw a valid column for this query (possible under narrow windows): the
          // tile then contributes nothing; a single such row has m_r = -inf and gets weight 0
          Mt[x] = fmaxf(fmaxf(fstat[x * 8], fstat[x * 8 + 1]), fmaxf(fstat[x * 8 + 2], fstat[x * 8 + 3]));
          w[x] = (valid[x] && m_r[x] > -INFINITY) ? exp2f(m_r[x] - Mt[x]) : 0.f;
          float lw = w[x] * l_r[x];
#pragma unroll
          for (int o = 16; o >= 1; o >>= 1) lw += __shfl_xor_sync(0xffffffffu, lw, o);
          if (lane == 0) fstat[x * 8 + 4 + wq] = lw;
        }
        // accumulators: the last P*V of both tiles must have landed
        alive = __all_sync(0xffffffffu, mbar_wait(&bars.o_done[0], par, abort_flag)) &&
                __all_sync(0xffffffffu, mbar_wait(&bars.o_done[1], par, abort_flag));
        if (!alive) break;
        tc_fence_after();
        const bool in_range = k_r < T;
#pragma unroll 1
        for (int ch = 0; ch < D / 32; ++ch) {
          // this row's V2 values for the chunk (shared by both tiles)
          float v2f[32];
#pragma unroll
          for (int i4 = 0; i4 < 4; ++i4) {
            const uint4 vv = in_range ? __ldg(reinterpret_cast<const uint4*>(V2g + (size_t)k_r * D + ch * 32 + i4 * 8))
                                      : make_uint4(0, 0, 0, 0);
            const uint32_t wv[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = unpack2<T16>(wv[e]);
              v2f[i4 * 8 + 2 * e] = f.x;
              v2f[i4 * 8 + 2 * e + 1] = f.y;
            }
          }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            uint32_t o[32];
            tmem_ld32(tmem + lane_base + Cfg::kTmemO + x * D + ch * 32, o);
            tmem_wait_ld();
            if (ch == D / 32 - 1) {
              // last chunk of this tile's accumulator is in registers: it may be overwritten
              tc_fence_before();
              mbar_arrive(&bars.o_free[x]);
            }
            float v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(o[i]) * (w[x] * v2f[i]);
            const float colsum = warp_transpose_sum(v, lane);
            red[(x * 4 + wq) * D + ch * 32 + lane] = colsum;
          }
        }
        if (!fold_sync()) { alive = false; break; }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          if (!(Mt[x] > -INFINITY)) continue;   // nothing valid in this tile for this query
          const float Lt = fstat[x * 8 + 4] + fstat[x * 8 + 5] + fstat[x * 8 + 6] + fstat[x * 8 + 7];
          const float Mn = fmaxf(M_run[x], Mt[x]);
          const float ca = exp2f(M_run[x] - Mn), cb = exp2f(Mt[x] - Mn);
          if (row < D) {
            const float Ot = red[(x * 4) * D + row] + red[(x * 4 + 1) * D + row] + red[(x * 4 + 2) * D + row] +
                             red[(x * 4 + 3) * D + row];
            O_run[x] = O_run[x] * ca + Ot * cb;
          }
          L_run[x] = L_run[x] * ca + Lt * cb;
          M_run[x] = Mn;
        }
        if (!fold_sync()) { alive = false; break; }  // red / fstat are rewritten by the next k-tile
      }
      if (!alive) break;
      // ---- store the two output rows and their log-sum-exp
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int qx = x == 0 ? qa : qb;
        if (row < D) ((T16*)p.out)[((size_t)bh * T + qx) * D + row] = from_f<T16>(O_run[x] / L_run[x]);
        if (row == 0) p.lse[(size_t)bh * T + qx] = (M_run[x] + log2f(L_run[x])) * kLn2;
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && bars.abort_flag && p.status) atomicOr(p.status, 2);
}

// What the forward kernels need before they start, in one pass over the tensors: SiLU(V1) in the inputs' type and, when
// `stats` is not null, the per-head statistics behind the score bounds,
//   stats[bh] = max_j |K1[bh, j, :]|^2,  stats[BN + bh] = max_q |Q[bh, q, :]|^2,  stats[2 BN + bh] = max element^2 of K2[bh],
// and, for a call that the kernel over diagonals is asked for (DIAG), fp16: the largest |element| of K1, K2, V1 and V2 in four more
// arrays.  DIAG: that kernel's counters are zeroed; a head with an element that is not finite has an infinite max_q |Q|^2, and so no
// bound on its scores: the maxima pass over a NaN, and an infinite or NaN value reaches, as 0 * W, every query of two tiles there.
// A cluster of blocks takes one head: the maxima meet in the first block's shared memory, so that no launch has to
// zero anything and no atomics are needed.  8 elements per thread and pass; a row is held by D / 8 neighbouring lanes.
// Bound by latency: a pass waits for its reads (1 us), a block for the cluster twice and for its launch.  So a head has as many blocks
// (eight, the portable cluster size, at most) as the chip holds, each with a pass of work, and larger ones where that leaves many
// passes (prepare_fwd).  us, blocks of 256 threads, eight a head -> the present ones: 16 heads T=1200 D=64 6.4 -> 5.8, T=2048
// 8.7 -> 7.0, T=8192 30 -> 18, one head T=8192 25 -> 11, 1024 heads T=200 37 -> 24, 4096 heads T=140 131 -> 65.  DIAG with more reads
// under way and half as many threads on an SM: T=1200 9.2 -> 5.6 in 32 and 64 registers.
constexpr int kPrepThreads = 256, kPrepMost = 1024, kPrepMostDiag = 512, kStats = 7;
template <typename T16, bool DIAG>
__global__ void __launch_bounds__(DIAG ? kPrepMostDiag : kPrepMost, 2)
fwd_prepare_kernel(const T16* __restrict__ v1, const T16* __restrict__ k1, const T16* __restrict__ q,
                   const T16* __restrict__ k2, const T16* __restrict__ v2, T16* __restrict__ sv1, float* __restrict__ stats, int head_elems,
                   int D, int BN, int blocks, unsigned* __restrict__ counters, int n_counters) {
  constexpr int COUNT = DIAG && std::is_same<T16, __half>::value ? kStats : 3;
  __shared__ float red[8][COUNT];      // [block of the cluster]; used in the first block
  __shared__ float wred[kPrepMost / 32][COUNT];
  const int bh = blockIdx.x / blocks, part = blockIdx.x % blocks;
  const size_t base = (size_t)bh * head_elems;
  const int lanes = D / 8;
  float m[COUNT] = {};
  if constexpr (DIAG) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_counters; i += gridDim.x * blockDim.x) counters[i] = 0;
  }
  uint32_t top_k1 = 0, top_k2 = 0, top_q = 0, top_v1 = 0, top_v2 = 0;   // largest |element|, of either half (DIAG: NaN if there is one)
  // (the bound is the same for all lanes of a row: head_elems is a multiple of D)
  for (int i = (part * blockDim.x + threadIdx.x) * 8; i < head_elems; i += blocks * blockDim.x * 8) {
    // (all reads of a pass together: it waits for memory)
    const uint4 v = *reinterpret_cast<const uint4*>(v1 + base + i);
    uint4 x, a, b, c;
    if (DIAG) x = *reinterpret_cast<const uint4*>(v2 + base + i);
    if (stats) {
      a = *reinterpret_cast<const uint4*>(k1 + base + i);
      b = *reinterpret_cast<const uint4*>(q + base + i);
      c = *reinterpret_cast<const uint4*>(k2 + base + i);
    }
    const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack2<T16>(wv[e]);
      o[e] = pack2<T16>(silu_f(f.x), silu_f(f.y));
    }
    *reinterpret_cast<uint4*>(sv1 + base + i) = make_uint4(o[0], o[1], o[2], o[3]);
    if constexpr (DIAG) {
      grow_abs<T16, true>(top_v1, v);
      grow_abs<T16, true>(top_v2, x);
    }
    if (stats) {
      const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
      grow_abs<T16, DIAG>(top_k2, c);
      if constexpr (DIAG) {
        grow_abs<T16, true>(top_k1, a);
        grow_abs<T16, true>(top_q, b);
      }
      float n1 = 0.f, nq = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 y = unpack2<T16>(wa[e]), z = unpack2<T16>(wb[e]);
        n1 = fmaf(y.x, y.x, fmaf(y.y, y.y, n1));
        nq = fmaf(z.x, z.x, fmaf(z.y, z.y, nq));
      }
      // (the lanes of a row are all here or all gone; which lanes of the warp are is not the same everywhere)
      const uint32_t row_lanes = ((lanes == 32 ? 0u : 1u << lanes) - 1u) << ((threadIdx.x & 31) / lanes * lanes);
      for (int o2 = lanes / 2; o2 >= 1; o2 >>= 1) {
        n1 += __shfl_xor_sync(row_lanes, n1, o2);
        nq += __shfl_xor_sync(row_lanes, nq, o2);
      }
      m[0] = fmaxf(m[0], n1);
      m[1] = fmaxf(m[1], nq);
    }
  }
  if (!stats) return;
  auto larger_half = [](uint32_t v) {
    const float2 f = unpack2<T16>(v);
    return fmaxf(f.x, f.y);
  };
  m[2] = larger_half(top_k2);
  if constexpr (COUNT == kStats) {
    m[3] = larger_half(top_k1);
    m[5] = larger_half(top_v1);
    m[6] = larger_half(top_v2);
  }
  if constexpr (DIAG) {
    const uint32_t bad = not_finite<T16>(top_k1) | not_finite<T16>(top_k2) | not_finite<T16>(top_q) | not_finite<T16>(top_v1) | not_finite<T16>(top_v2);
    if (bad & 0x80008000u) m[1] = INFINITY;
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
    for (int e = 0; e < COUNT; ++e) m[e] = fmaxf(m[e], __shfl_xor_sync(0xffffffffu, m[e], o));
  if constexpr (COUNT == kStats) m[4] = m[2];
  m[2] *= m[2];
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int e = 0; e < COUNT; ++e) wred[threadIdx.x >> 5][e] = m[e];
  }
  cluster_sync_all();   // every block of the cluster runs: its shared memory may be written (a block barrier as well)
  if (threadIdx.x < COUNT) {
    float v = 0.f;
    for (int w = 0; w < blockDim.x / 32; ++w) v = fmaxf(v, wred[w][threadIdx.x]);
    uint32_t dst;   // the first block's red[part][.]
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_u32(&red[part][threadIdx.x])), "r"(0));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(v) : "memory");
  }
  cluster_sync_all();
  if (part == 0 && threadIdx.x < COUNT) {
    float v = 0.f;
    for (int c = 0; c < blocks; ++c) v = fmaxf(v, red[c][threadIdx.x]);
    stats[(size_t)threadIdx.x * BN + bh] = v;
  }
}

// SiLU(V1) at the head of the workspace and, when the workspace has the optional tail, the statistics (the returned pointer is to the
// first of its arrays of B*N values, the K1 row norms); `diag`: the kernel over diagonals is asked.
template <typename T16>
int prepare_fwd(const TdpArgs& a, const DiagParams* diag, T16** sv1_out, float** k1n_out) {
  const int BN = a.B * a.N;
  const size_t n = (size_t)BN * a.T * a.D, tail = align_up(n * 2, 256);
  T16* sv1 = (T16*)a.workspace;
  float* k1n = nullptr;
  if (a.workspace_bytes >= tail + (diag ? kStats : 3) * (size_t)BN * sizeof(float)) k1n = reinterpret_cast<float*>((char*)a.workspace + tail);
  const int head_elems = a.T * a.D;
  // Blocks of 256 threads that an SM holds; a head's blocks; and the passes of one.  us with 1 / 2 / 4 / 8 blocks a head: 256 heads T=512
  // 19.1 / 13.0 / 11.7 / 13.5 (diag 19.1 / 13.2 / 16.6 / 21.2), 1024 heads T=200 24.5 / 26.8 / 29.9 / 36.8.
  const long resident = (long)num_sms() * (diag ? 4 : 8);
  int blocks = 1;
  while (blocks < 8 && blocks * kPrepThreads * 8 < head_elems && 2L * BN * blocks <= resident) blocks *= 2;
  const int passes = (head_elems - 1) / (blocks * kPrepThreads * 8) + 1;
  // Larger blocks where passes are many and SMs free.  us with 256 / 512 / 1024 threads (diag 256 / 512), inputs in L2, and in HBM in
  // brackets: 8 heads, 4 passes 5.3 / 4.1 / 4.3 [8.4 / 5.8 / 4.8] (4.7 / 4.0 [6.6 / 5.0]); 16 heads, 2 passes 4.0 / 3.8 / 5.7 [5.6 / 4.4 / 6.0]
  // (3.8 / 4.1 [4.8 / 4.6]), 5 passes 6.3 / 6.0 / 7.3 [10.2 / 8.0 / 8.1] (5.7 / 6.1 [8.2 / 7.5]), 8 passes 8.7 / 7.1 / 7.7 [14.8 / 9.8 / 8.5]
  // (7.7 / 7.3 [11.4 / 8.9]), 32 passes 31 / 20 / 18 [50 / 30 / 21]; 32 heads, 3 passes 4.9 / 5.0 / 6.0 [8.0 / 7.0 / 6.5] (4.6 / 5.3 [7.0 / 6.8]),
  // 7 passes 8.1 / 7.3 / 7.8 [14.7 / 11.2 / 9.6] (7.4 / 7.4 [12.1 / 10.6]); 64 heads, 4 passes 7.1 / 7.6 / 10.8 [11.5 / 10.0 / 12.6] (7.5 / 10.0 [11.0 / 13.1]).
  const long grid = (long)BN * blocks, sms = num_sms();
  const bool few = 2 * grid <= sms;
  int threads = kPrepThreads;
  if (passes >= (few || !diag ? 2 : 4) && 2 * grid <= resident) threads = 512;
  if (!diag && passes >= (few ? 4 : 6) && grid <= 2 * sms) threads = kPrepMost;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = blocks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(BN * blocks), 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.stream = a.stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TRITT_CUDA_OK(cudaLaunchKernelEx(&cfg, diag ? fwd_prepare_kernel<T16, true> : fwd_prepare_kernel<T16, false>, (const T16*)a.v1,
                                   (const T16*)a.k1, (const T16*)a.q, (const T16*)a.k2, (const T16*)a.v2, sv1, k1n, head_elems, a.D, BN,
                                   blocks, diag ? diag->arrived : nullptr, diag ? diag->g.grid * kDiagArrivals : 0));
  count_launch();
  *sv1_out = sv1;
  *k1n_out = k1n;
  return 0;
}

template <int D, typename T16>
int launch_fwd(const TdpArgs& a) {
  using Cfg = FwdCfg<D>;
  const int BN = a.B * a.N;
  T16* sv1 = nullptr;
  float* k1n = nullptr;
  const bool band = sm100_tdp_fwd_band_applies(a.T, a.mask);
  const size_t diag_offset = align_up(align_up((size_t)BN * a.T * D * 2, 256) + kStats * (size_t)BN * sizeof(float), 256);
  DiagParams diag;
  const bool by_diagonals =
      band && a.workspace_bytes > diag_offset &&
      sm100_tdp_fwd_diag_plan(a, (char*)a.workspace + diag_offset, a.workspace_bytes - diag_offset, diag);
  int rc = prepare_fwd<T16>(a, by_diagonals ? &diag : nullptr, &sv1, &k1n);
  if (rc) return rc;
  diag.stats = k1n;
  if (by_diagonals && (rc = sm100_tdp_fwd_diag(a, diag))) return rc;
  if (band) return sm100_tdp_fwd_band(a, sv1, k1n, by_diagonals ? &diag : nullptr);
  CUtensorMap tmK1, tmK2, tmSV1;
  if ((rc = make_tmap_3d(&tmK1, a.k1, 2, D, a.T, BN, 64, 128))) return rc;
  if ((rc = make_tmap_3d(&tmSV1, sv1, 2, D, a.T, BN, 64, 128))) return rc;
  if ((rc = make_tmap_3d(&tmK2, a.k2, 2, D, a.T, BN, 64, 128))) return rc;
  FwdParams p{};
  p.out = a.out_o;
  p.lse = a.out_lse;
  p.q = a.q;
  p.v2 = a.v2;
  p.T = a.T;
  p.BN = BN;
  p.q_mod = a.q_mod;
  p.q_rem = a.q_rem;
  p.nq = a.q_rem < a.T ? (a.T - a.q_rem + a.q_mod - 1) / a.q_mod : 0;
  p.n_pairs = (p.nq + 1) / 2;
  p.causal = a.mask.causal;
  p.k1w = a.mask.k1w;
  p.k2w = a.mask.k2w;
  p.kkl = a.mask.kkl;
  p.kkr = a.mask.kkr;
  p.scale2 = a.alpha * kLog2e;
  p.k1_norm2_max = k1n;
  p.q_norm2_max = k1n ? k1n + BN : nullptr;
  p.k2_elem2_max = k1n ? k1n + 2 * BN : nullptr;
  // P = exp2(S - reference) lies in [2^-(2 limit + 1.15), 1]: normal numbers of the 16-bit type (bf16 2^-126, fp16 2^-14)
  p.bound_limit = std::is_same<T16, __nv_bfloat16>::value ? 40.f : 6.f;
  p.status = a.status_word;
  if (p.nq == 0) return 0;
  auto kern = tdp_fwd_kernel<D, T16>;
  TRITT_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
  const long items = (long)p.n_pairs * BN;
  const int grid = (int)(items < num_sms() ? items : num_sms());
  kern<<<grid, kThreads, Cfg::kSmem, a.stream>>>(tmK1, tmK2, tmSV1, p);
  count_launch();
  TRITT_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace


bool sm100_tdp_supported(int op, int T, int D, int dtype, const TdpMask& m) {
  if (op != TRITT_OP_TDP_FWD && op != TRITT_OP_TDP_BWD) return false;
  if (dtype != TRITT_BF16 && dtype != TRITT_F16) return false;
  if (D != 64 && D != 128) return false;
  (void)m;  // every window of the causal mask is handled
  return T >= 1;
}

// Extra bytes behind the forward's SiLU(V1) copy that enable the score bound (the forward runs without them too).
size_t sm100_tdp_fwd_optional_workspace(int B, int N, int T, int D, int dtype, const TdpMask* m, int q_mod) {
  if (dtype != TRITT_BF16 && dtype != TRITT_F16) return 0;
  const size_t n = (size_t)B * N * T * D;
  const size_t diag = sm100_tdp_fwd_diag_workspace(B, N, T, D, m, q_mod);
  return align_up(n * 2, 256) - n * 2 + align_up((diag ? kStats : 3) * (size_t)B * N * sizeof(float), 256) + align_up(diag, 256);
}

size_t sm100_tdp_workspace(int op, int B, int N, int T, int D, int dtype) {
  if (dtype != TRITT_BF16 && dtype != TRITT_F16) return 0;
  if (op == TRITT_OP_TDP_FWD) return (size_t)B * N * T * D * 2;
  if (op == TRITT_OP_TDP_BWD) return sm100_tdp_bwd_workspace(B, N, T, D);
  return 0;
}

int sm100_tdp_fwd(const TdpArgs& a) {
  // general kernel: the two queries of a pair must fall in the same 128-row block (the band kernel has no such rule)
  if (!sm100_tdp_fwd_band_applies(a.T, a.mask) && (a.q_mod < 1 || a.q_mod > 64 || (a.q_mod & (a.q_mod - 1)))) {
    set_error("tensor-core path needs a power-of-two query shard count <= 64 (got %d)", a.q_mod);
    return -30;
  }
  if (a.dtype == TRITT_BF16) return a.D == 128 ? launch_fwd<128, __nv_bfloat16>(a) : launch_fwd<64, __nv_bfloat16>(a);
  return a.D == 128 ? launch_fwd<128, __half>(a) : launch_fwd<64, __half>(a);
}

}  // namespace tritt
