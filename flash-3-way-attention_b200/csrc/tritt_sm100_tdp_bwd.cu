// Triple-dot-product trittention backward on Blackwell tensor cores (tcgen05 + TMEM + TMA).
//
// The score S[q,j,k] = alpha sum_h Q[q,h] K1[j,h] K2[k,h] and the gated value are trilinear, so any of the three
// indices can be the one that is stepped over.  Here it is k: for one k the (q, j) plane is an ordinary attention
// backward whose key and value operands carry the k-th rows of K2 and V2,
//     A [j,h] = K1[j,h] * K2[k,h]      A'[j,h] = SiLU(V1)[j,h] * V2[k,h]
//     S  = alpha*log2(e) * Q A^T (for large scores R K1^T with R [q,h] = alpha*log2(e) * Q[q,h] * K2[k,h])
//                         P  = exp2(S - lse2[q])       (recomputed from the saved lse)
//     dP = dO A'^T        dS = P * (dP - Dq[q]),       Dq = sum_h dO O
// and all five gradients follow from three more products:
//     dQ[q,:] += dS A                                  (accumulated over k in tensor memory)
//     G = dS^T Q:   dK1[j,h] += alpha K2[k,h] G[j,h],   dK2[k,h] += alpha sum_j K1[j,h] G[j,h]
//     U = P^T dO:   dSV1[j,h] += V2[k,h] U[j,h],        dV2[k,h] += sum_j SiLU(V1)[j,h] U[j,h]
// Five products per (q-tile, j-tile, k) where stepping over q needs six (and needed eight with every key-side
// gradient owned by rows), and one exponential per attended triple instead of two.
// (The reference runs one Triton kernel per gradient, recomputing P five times:
// triple_dot_product/kernels/bwd_dq.py, bwd_dk1.py, bwd_dk2.py, bwd_dv1.py, bwd_dv2.py.)
//
// A work item is a tile of 128 queries x JT rows j with its range of k; the item's Q, dO, K1 and SiLU(V1) tiles stay
// in shared memory for the whole range, dQ in tensor memory, dK1 and dSiLU(V1) in the registers of the fold
// warpgroups; per step only the two rows K2[k], V2[k] come in and two rows of dK2, dV2 go out (vector reductions into
// fp32 sums that stay in L2).  All steps of a call are laid out in one line and cut in equal parts, one per CTA
// (every sum is a reduction, so an item may be cut anywhere): no last wave.
//
// What bounds it: no unit, but the chains of tensor-memory reads, shared-memory accesses and waits of the soft-max and fold warps,
// while the tensor cores' operand reads keep shared memory busy.  A step takes 2760 cycles at head dimension 128 and 3790 at 64;
// 16 heads of T=768: issue slots 60 / 63 % busy, tensor pipe 49 / 37 %, shared memory 30 / 37 % by the warps and 47 / 38 % by the
// tensor cores.
// Operands formed by one 16-bit product per pair instead of fp32 products and conversions, the products issued by three warps
// instead of one, A' doubled, exponentials beside the arithmetic of dS, looks at barriers ahead of the waits, and waits that seldom
// read the clock, backward of T=2048 D=128 bf16 16 heads 70.9 -> 64.1 ms, T=4096 D=64 4 heads 79.9 -> 78.1, T=512 D=64 32 heads 1.80 ->
// 1.70, not causal fp16 16 heads 1.83 -> 1.78, windows 128/128/32/32 at T=2048 1.22 -> 1.14, T=333 D=128 4 heads 189 -> 169 us.
// Against a query and 128 rows of one key tensor per tile (eight products, exponentials twice), same call, training
// steps: T=2048 D=128 bf16 16 heads 114.5 -> 94.9 ms, T=4096 D=64 4 heads 140.5 -> 113.8 ms, T=512 D=64 fp16 16 heads 2.37
// -> 1.59 ms, windows 128/128/32/32 at T=2048 4.54 -> 1.77 ms.
//
// Narrow bands (kk_left + kk_right <= 72, head dimension 64, small scores): tdp_bwd_diag_kernel, the same kernel with steps over the
// diagonals d = k - j.  On a diagonal A [j,h] = K1[j,h] K2[j+d,h] and A' alike, all else as above, except that row j of G and U
// belongs to one row k = j + d of dK2 and dV2: nothing is summed over rows, and a step adds two tiles of 128 x 64 to the fp32 sums
// (vector reductions; the SMs together take 5.8 TB/s of them, twice what a step asks for) where stepping over k adds two rows.  All
// 128 x 128 of an item's cells lie in the band, of which a step over k has a band's width.  What bounds it: the fold warps, 4800
// cycles a step (operands 1500, fold 3100) whose spills and exchanges between lanes count most.  us per backward, steps over k ->
// diagonals: 16 heads T=2048 fp16 windows 128/128/32/32 951 -> 606, 256/256/40/20 1378 -> 808, 8/8/4/4 529 -> 150, 400/400/36/36
// 1818 -> 1366; without windows, band 32/32 T=1024 1094 -> 690, 16/16 T=512 322 -> 133.  A head is this kernel's or the one's over k
// (diag_head), as its scores and elements are.
//
// Tile shapes: the accumulators S | dP | G | U | dQ have to fit 512 columns of tensor memory.  Head dimension 64:
// JT = 128, G and U as [j x h] (128 + 128 + 64 + 64 + 64).  Head dimension 128: JT = 64 and G, U transposed,
// [h x j], so that their M extent is 128 (64 + 64 + 64 + 64 + 128); a JT of 128 would need 640 columns.
//
// CTA: 20 warps (both kernels).  0-3 and 4-7: soft-max warpgroups (half of a step's columns each, one query per thread); 8-11: forms
// A and folds G; 12-15: forms A' and folds U; 16, 18, 19: issue the products S and dP, U, dQ and G (large scores: 16 all five,
// 18 and 19 form R); 17: TMA and the K2 / V2 rows.  P and dS are written to shared memory, where both the transposed (U, G) and the plain (dQ) product can read them.
#include "tritt_sm100_tdp.cuh"

#include <atomic>
#include <type_traits>

namespace tritt {
namespace {
using namespace sm100;

constexpr int kBwdThreads = 640;
// Registers per thread: 640 threads are launched with 96 each (480 per lane of the five warpgroups) and split them anew.  The
// shares are tight: the two bodies spill 420 to 520 bytes a thread together, the one over diagonals 280 to 350, most of it what an item
// or a step reads once or twice.  (80 / 128 / 64 or 96 / 120 / 48 for soft-max, fold and service warps in the small-score body: 5 to 8 % slower, as their
// loops spill.)
constexpr int kRegsLaunch = 96;
// (88 / 136 / 32 for large scores at head dimension 64, where R's warps spill then: fp16 16 heads T=512 916 -> 927 us, bf16 T=2048 4 heads
// 10.45 -> 10.50 ms, windows 16/16/8/8 T=1200 380 -> 386, 128/128/0/0 T=2048 984 -> 989.  Small scores: 1687 us -> 1750 at 32 heads of T=512.)
// (Diagonals: the fold warps need more, what the service warps can spare.  Band 128/128/32/32 at T=2048, soft-max / fold / service:
// 88 / 128 / 48 757 us, 88 / 136 / 32 671, 80 / 136 / 48 731, 80 / 144 / 32 748; twice as many fold warps of 72 registers 930.)
// (Large scores at head dimension 128 have the service warps form 32 KB of R per step, and soft-max warps that hold half as many
// columns as at 64: with 48 registers those service warps spill, 1.60 -> 1.90 ms at 16 heads of T=512.)
template <int D, bool LARGE, bool DIAG> struct BwdRegs {
  static constexpr int kSoftmax = D == 128 && LARGE ? 80 : 88, kFold = DIAG ? 136 : 128,
                       kService = DIAG ? 32 : D == 128 && LARGE ? 64 : 48;
  static_assert(2 * kSoftmax + 2 * kFold + kService <= 5 * kRegsLaunch, "more registers than the launch has");
};
constexpr int kVecBatch = 4;     // K2 / V2 rows per hand-over
constexpr int kVecSlots = 4;     // batches in flight
// S = Q A^T rounds the product K1 K2 where the forward rounds R = Q K2, so that P does not match the saved log-sum-exp and no
// longer sums to one; and the rounding of A is also dQ's.  Where scores are of order 1 or more and few pairs carry a query,
// the gradients were up to 2.4 times further from fp64 than with the forward's operand (scores of order 3, not causal, T=200:
// dQ 2.0 to 2.4 times, dV2 1.5 to 2.3; of order 1, D=128, bf16: dQ 1.33).  CTAs with such heads form S = R K1^T, from
// the rows that the forward formed: 0.5 to 1.06 times there, dV2 1.00.  R is 128 x D for any JT and is formed by two warps, so
// this costs speed (B200, against S = Q A^T, the same inputs): T=512 D=64 16 heads 0.87 -> 0.91 ms, T=4096 D=64 4 heads 78.3 -> 81.8,
// T=2048 D=128 16 heads 64.1 -> 74.9, T=1024 9.3 -> 11.1.  Hence the bound, on |Q row| |K1 row| max|K2| in log2 units: Gaussian inputs with
// a bound of 21 to 82 (their scores are 1/60 to 1/80 of it) show no excess with A (dQ 0.85 to 1.0), aligned inputs come
// closer to their bound.
constexpr float kScoreBound = 16.f;
constexpr int kStatParts = 32, kStatFloats = 8;
// Rows of a window of K2 or V2 (128 + kk_left + kk_right at most): what shared memory has left beside one A' instead of two and without the K1
// and SiLU(V1) tiles.
constexpr int kDiagRows = 200;
constexpr int kPartHeads = 512;   // heads of a CTA's part, at most, where the kernel over diagonals is asked

template <int D, bool DIAG = false> struct BwdCfg {
  static constexpr int JT = D == 64 ? 128 : 64;       // rows j of an item
  static constexpr int CW = JT / 2;                   // columns of one soft-max thread
  static constexpr int kTileQ = 128 * D * 2;          // Q, dO
  static constexpr int kTileJ = JT * D * 2;           // K1, SiLU(V1), A, A'  (16 KiB for both head dimensions)
  static constexpr int kTileP = 128 * JT * 2;         // P, dS
  static constexpr int kOffQ = 0;
  static constexpr int kOffDO = kOffQ + kTileQ;
  static constexpr int kOffK1 = kOffDO + kTileQ;      // K1 | SiLU(V1)
  // DIAG: windows of K2 and V2 rows instead (K1 and SiLU(V1) go straight to the registers that keep them)
  static constexpr int kWindow = kDiagRows * D * 2;
  static constexpr int kOffA = kOffK1 + (DIAG ? 2 * kWindow : 2 * kTileJ);   // A (two buffers) | A'
  static constexpr int kOffP = kOffA + 3 * kTileJ;    // P | dS (two buffers)
  // R (see tdp_bwd_body), in blocks of 64 columns: over the SiLU(V1) tile, and behind P | dS
  static constexpr int kOffR0 = kOffK1 + kTileJ, kOffR1 = kOffP + 3 * kTileP;
  static constexpr int kOffVec = kOffR1 + (D / 64 - 1) * 16384;  // [slot][K2 rows | V2 rows][row of the batch][D], 16-bit
  static constexpr int kVecPart = kVecBatch * D * 2;  // bytes of a batch of rows of one tensor
  static constexpr int kOffBars = kOffVec + (DIAG ? 0 : kVecSlots * 2 * kVecPart);
  static constexpr int kOffHeads = kOffBars + 512;    // PartHeads' marks
  static constexpr int kSmem = kOffHeads + (D == 64 ? kPartHeads : 0);
  static constexpr int kTmemS = 0, kTmemDP = JT, kTmemG = 2 * JT, kTmemU = kTmemG + 64, kTmemDQ = kTmemU + 64;
  static constexpr int kTmemQ = kTmemDQ + D, kTmemDO = kTmemQ + D / 2;   // 16-bit, two elements a column
  static_assert(kTmemDO + D / 2 <= 512 && kSmem <= 232448, "tensor / shared memory");
};

// The steps (q-tile, j-tile, k) of a call in the order they are cut: heads, q-tiles, j-tiles, k.  Causal mask
// j <= q <= j + k1w,  k <= q <= k + k2w,  k - kkl <= j <= k + kkr:  a q-tile [qa, qb] meets the j-tiles of rows
// [qa - k1w, qb], and a pair of tiles the k in [max(qa - k2w, ja - kkr), min(qb, jb + kkl)].
// The j-tiles lie side by side (stride = JT, lead = 0), or, for a narrow band, overlap: tile jt belongs to the k in
// [jt stride, jt stride + stride) and has all the rows j that these see, stride + kkl + kkr = JT of them (lead = kkl).  Then a k
// meets one j-tile per q-tile, instead of (JT + kkl + kkr) / JT on average.
struct BwdGeometry {
  int T, nq, q_mod, q_rem, causal;
  int k1w, k2w, kkl, kkr;  // windows of the causal mask (T or more = unbounded)
  int JT;                  // rows of a j-tile
  int stride, lead;        // tile jt has the rows from jt * stride - lead on
  bool diagonals;          // steps are the diagonals d = k - j, counted from -kkr
  __host__ __device__ int q_tiles() const { return (nq + 127) / 128; }
  __host__ __device__ int first_q(int qt) const { return q_rem + qt * 128 * q_mod; }
  __host__ __device__ int last_q(int qt) const {
    const int i = qt * 128 + 127;
    return q_rem + (i < nq ? i : nq - 1) * q_mod;
  }
  __host__ __device__ bool overlapping() const { return stride != JT; }
  __host__ __device__ int j_row(int jt) const { return jt * stride - lead; }
  // rows [lo, hi) of j-tile jt, counted from its first, that the q-tile's sums may take: of an overlapping tile those that a query of
  // the q-tile sees
  __host__ __device__ void j_rows(int qt, int jt, int& lo, int& hi) const {
    lo = 0;
    hi = T - j_row(jt);
    if (!overlapping()) return;
    const int a = first_q(qt) - k1w;
    lo = (a > 0 ? a : 0) - j_row(jt);
    hi = last_q(qt) + 1 - j_row(jt);
  }
  __host__ __device__ int k_first(int qa) const {   // of the k that a query from qa on sees
    const int reach = k2w < k1w + kkr ? k2w : k1w + kkr;
    return qa > reach ? qa - reach : 0;
  }
  __host__ __device__ int j_first(int qt) const {
    if (overlapping()) return k_first(first_q(qt)) / stride;
    if (diagonals) {
      const int reach = k1w < k2w + kkl ? k1w : k2w + kkl, qa = first_q(qt);
      return qa > reach ? (qa - reach) / JT : 0;
    }
    const int lo = first_q(qt) - k1w;
    return causal && lo > 0 ? lo / JT : 0;
  }
  __host__ __device__ int j_last(int qt) const { return (causal ? last_q(qt) : T - 1) / stride; }
  __host__ __device__ int k_range(int qt, int jt, int& k0) const {   // number of steps of a pair of tiles
    k0 = 0;
    if (!causal) return T;
    const int qa = first_q(qt), qb = last_q(qt);
    if (overlapping()) {
      const int a = k_first(qa), b = jt * stride;
      k0 = a > b ? a : b;
      const int k1 = qb < b + stride - 1 ? qb : b + stride - 1;
      return k1 >= k0 ? k1 - k0 + 1 : 0;
    }
    const int ja = jt * JT, jb = ja + JT - 1;
    if (diagonals) {   // 0 <= j + d <= q,  q - k2w <= j + d
      int d0 = qa - k2w - jb, d1 = qb - ja;
      if (d0 < -jb) d0 = -jb;
      if (d0 < -kkr) d0 = -kkr;
      if (d1 > kkl) d1 = kkl;
      k0 = d0 + kkr;
      return d1 >= d0 ? d1 - d0 + 1 : 0;
    }
    if (qa - k2w > k0) k0 = qa - k2w;
    if (ja - kkr > k0) k0 = ja - kkr;
    const int k1 = qb < jb + kkl ? qb : jb + kkl;
    return k1 >= k0 ? k1 - k0 + 1 : 0;
  }
};

struct BwdParams {
  const void *q, *d_o, *k2, *v2, *k1, *sv1;
  const float *lse, *drow;
  const float* stats;      // [BN][stat_parts][kStatFloats] (see tdp_bwd_prepare_kernel), or null
  int stat_parts;
  float *dq, *dk1, *dk2, *dsv1, *dv2;   // fp32 sums, zero on entry
  BwdGeometry g;
  int BN;
  int i_first;             // query rows (of the shard) before this one are not this kernel's
  long head_steps;         // steps of one head
  float alpha;
  bool diag_asked;         // the heads that are diag_head() are the kernel's that steps over diagonals, the others the one's over k
  int* status;
};

struct BwdItem {
  int bh, qt, jt, k0, len, flags;   // len 0: no more items
  int ea, eb;                       // A and A' carry factors 2^ea and 2^eb (range_shift), R 2^er (product_shift)
  int er, pad_[3];
};
enum {
  kFirstOfQ = 1, kLastOfQ = 2,   // the first / last item of a run over the j-tiles of one q-tile
  kShiftBits = 8                 // (flags >> kShiftBits: dS carries a factor 2^that, beside P's)
};
constexpr int kItemSlots = 4;               // (an item is read before its successor but one is written)

struct BwdBarriers {
  alignas(16) BwdItem items[kItemSlots];
  uint64_t tile_full, tile_free;            // Q, dO, K1, SiLU(V1) of an item
  uint64_t vec_full[kVecSlots], vec_empty[kVecSlots];
  uint64_t a_ready[2], a_free[2], ap_ready[2], ap_free[2], r_ready;  // doubled by step parity (a producer may be two steps ahead)
  // (ds_ready: warp 16 lets the soft-max warps go on to the next step's dS before warp 19 has looked at this one's, and a barrier
  // two phases ahead of its waiter reads as not ready for ever)
  uint64_t s_ready, s_free, p_ready, dp_ready, ds_ready[2], ds_free[2];
  uint64_t acc_done[2], acc_free[2];         // G, U
  uint64_t qdo_ready, dq_done, dq_free;
  uint32_t tmem_base;
  int abort_flag;
};

// the steps [s0, s1) of the line that are this CTA's
__device__ __forceinline__ void cta_part(const BwdParams& p, long& s0, long& s1) {
  const long H = p.head_steps;
  const long total = H * p.BN, c = gridDim.x;
  s0 = total / c * blockIdx.x + total % c * blockIdx.x / c;
  s1 = total / c * (blockIdx.x + 1) + total % c * (blockIdx.x + 1) / c;
}

// fp16 only: the recomputed probabilities of a query that attends n pairs are ~1/n, which for late rows lies below
// fp16's normal range (6e-5; 1/n = 2e-7 at q = 2048).  P and dS are therefore formed times 2^e, e = min(10, log2 of the
// attended pairs' count bound), and the folds divide it out.  2^10 keeps a probability of 1 times a dP - Dq below 63
// finite (dS has a further power of two where dP is small: ds_shift).  One e per q-tile, since G and U sum over its queries:
// that of the first query the kernel takes there, which has the fewest pairs (without windows 8 or 10 in the first tile, as
// the exact first queries leave none below 289 or 1089 pairs, and 10 in the others).
// bf16 has fp32's exponent range: e = 0.
template <typename T16>
__device__ __forceinline__ int prob_shift(int q, int causal, int T, int k1w, int k2w) {
  if constexpr (std::is_same<T16, __half>::value) {
    const int n1 = causal ? min(q, k1w) + 1 : T, n2 = causal ? min(q, k2w) + 1 : T;
    return min(10, (31 - __clz(n1)) + (31 - __clz(n2)));
  }
  return 0;
}

// A's power without statistics: as large as alpha log2(e), so that keys of 300 under an alpha of 1/64 do not overflow, and at most
// 1; 2^-17 keeps every product of two fp16 numbers finite.
__device__ __forceinline__ int alpha_shift(float alpha) {
  return min(0, max(-17, (int)(__float_as_uint(fabsf(alpha * kLog2e)) >> 23) - 127));
}
// The power of R = alpha log2(e) Q K2, which is formed in fp32: the bound on the products is brought to [2^14, 2^15).
template <typename T16> __device__ __forceinline__ int product_shift(float bound) {
  if constexpr (std::is_same<T16, __half>::value) {
    if (!(bound > 0.f) || !isfinite(bound)) return 0;
    return min(80, max(-80, 14 - ((__float_as_int(bound) >> 23) - 127)));
  }
  return 0;
}

// fp16 only: the further power of two of dS = P (dP - Dq), from a bound on |dP|, which holds for |Dq| (a mean of dP) as well:
// with P's 2^10 the product stays below 2^15.  0 where the bound leaves no room, that is from 8 on (as a bound it is far above
// what occurs: values of order 1 run without it).
template <typename T16> __device__ __forceinline__ int ds_shift(float bound) {
  if constexpr (std::is_same<T16, __half>::value) {
    if (!(bound > 0.f) || !isfinite(bound)) return 0;
    return min(24, max(0, 3 - ((__float_as_int(bound) >> 23) - 127)));
  }
  return 0;
}

__device__ __forceinline__ void red_add(float* p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void red_add2(float* p, float a, float b) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// The statistics of a head over its parts, in every lane (zeros without them).
struct BwdStats {
  float k1, k2, sv1, v2;    // largest element of K1, K2, SiLU(V1), V2
  float k1_row, q_row, do_row, sv1_row;   // largest squared norm of a row
  bool finite;              // all elements of Q, K1, K2, V1, V2 and dO are (the maxima pass over a NaN)
};
__device__ __forceinline__ BwdStats head_stats(const BwdParams& p, int bh, int lane) {
  float m[kStatFloats] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (p.stats && lane < p.stat_parts) {
    const float4* src = reinterpret_cast<const float4*>(p.stats + ((size_t)bh * p.stat_parts + lane) * kStatFloats);
    const float4 x = __ldg(src), y = __ldg(src + 1);
    m[0] = x.x; m[1] = x.y; m[2] = x.z; m[3] = x.w; m[4] = y.x; m[5] = y.y; m[6] = y.z; m[7] = y.w;
  }
  const bool finite = !__any_sync(0xffffffffu, __float_as_int(m[5]) < 0);   // (q_row's sign: see the preparation)
  m[5] = fabsf(m[5]);
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
    for (int i = 0; i < kStatFloats; ++i) m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
  return BwdStats{m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7], finite};
}

// Whether the head may have large scores: |S| <= |Q row| |K1 row| max|K2|, in log2 units, as S is.  (Not >: inf * 0 is large as well.
// Rounded one by one, so that whoever asks gets the same answer.)
__device__ __forceinline__ bool large_head(const BwdParams& p, const BwdStats& st) {
  const float q = __fsqrt_rn(__fmul_rn(st.k1_row, st.q_row));
  return !(__fmul_rn(__fmul_rn(fabsf(__fmul_rn(p.alpha, kLog2e)), q), st.k2) <= kScoreBound);
}
// Whether the head is the kernel's that steps over diagonals, if that is asked: small scores and finite elements.  (On a diagonal a row
// of K2 or V2 meets all queries of a tile that a row j = k - d meets, the tile before its own included.)
__device__ __forceinline__ bool diag_head(const BwdParams& p, const BwdStats& st) { return st.finite && !large_head(p, st); }

// What the heads of this CTA's part are, the same for every thread.  (Only its own: a look at all heads of a call, by every CTA of
// both kernels, took 5 % of a backward of 4096 heads of T=140.)
struct PartHeads {
  bool large;   // one may have large scores (without statistics: yes)
  bool diag;    // one is diag_head()
  bool others;  // one is not
};
template <int D, bool DIAG> __device__ __forceinline__ PartHeads part_heads(const BwdParams& p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* const marks = smem + BwdCfg<D, DIAG>::kOffHeads;   // of head bh: diag_head()
  long s0, s1;
  cta_part(p, s0, s1);
  PartHeads h{!p.stats, false, false};
  const int last = (int)((s1 - 1) / p.head_steps);
  for (int bh = (int)(s0 / p.head_steps) + (threadIdx.x >> 5); bh <= last && p.stats; bh += kBwdThreads / 32) {
    const BwdStats st = head_stats(p, bh, threadIdx.x & 31);
    const bool diag = diag_head(p, st);
    h.large |= large_head(p, st);
    h.diag |= diag;
    h.others |= !diag;
    if (p.diag_asked) marks[bh % kPartHeads] = diag;
  }
  h.large = __syncthreads_or(h.large);
  if (p.diag_asked) {
    h.diag = __syncthreads_or(h.diag);
    h.others = __syncthreads_or(h.others);
  }
  return h;
}

// One CTA's part of the line of steps, item by item (walked by the loader warp, which hands the items to the others).
// `marks` (null: all are): only those heads of the part that are (DIAG) or are not marked (part_heads).
template <bool DIAG> struct BwdWalk {
  const BwdGeometry& g;
  const uint8_t* marks;
  long left;                    // steps of this CTA not handed out yet
  int bh, qt, jt, k0, len;      // next item (len 0: none)

  __device__ void step() {
    if (++jt > g.j_last(qt)) {
      if (++qt == g.q_tiles()) {
        qt = 0;
        ++bh;
      }
      jt = g.j_first(qt);
    }
  }
  __device__ void find(long skip) {   // first item with steps, from (bh, qt, jt) on, less `skip` steps
    while (left > 0) {
      const int n = g.k_range(qt, jt, k0);
      if (n > skip) {
        k0 += (int)skip;
        len = n - (int)skip < left ? n - (int)skip : (int)left;
        left -= len;
        if (!marks || (marks[bh % kPartHeads] != 0) == DIAG) return;
        skip = 0;
      } else {
        skip -= n;
      }
      step();
    }
    len = 0;
  }
  __device__ BwdWalk(const BwdParams& p, const uint8_t* marks) : g(p.g), marks(marks) {
    long s0, s1;
    const long H = p.head_steps;
    cta_part(p, s0, s1);
    left = s1 - s0;
    bh = (int)(s0 / H);
    qt = 0;
    jt = g.j_first(0);
    find(s0 % H);
  }
  // hands out the item found last and looks for the one after it
  __device__ BwdItem next(const BwdItem& prev) {
    BwdItem it{bh, qt, jt, k0, len, 0, 0, 0, 0, {0, 0, 0}};
    if (len == 0) return it;
    if (bh != prev.bh || qt != prev.qt) it.flags |= kFirstOfQ;
    step();
    find(0);
    if (len == 0 || bh != it.bh || qt != it.qt) it.flags |= kLastOfQ;
    return it;
  }
};

// LARGE: S = R K1^T with R [q,h] = alpha*log2(e) * Q[q,h] * K2[k,h] instead of S = Q A^T (see kScoreBound).
template <int D, typename T16, bool LARGE, bool DIAG = false>
__device__ __forceinline__ void tdp_bwd_body(const CUtensorMap& tmQ, const CUtensorMap& tmDO, const CUtensorMap& tmK1,
                                             const CUtensorMap& tmSV1, const BwdParams& p) {
  using Cfg = BwdCfg<D, DIAG>;
  constexpr int JT = Cfg::JT, CW = Cfg::CW;
  constexpr bool kOneAp = LARGE || DIAG;   // a single buffer of A'
  static_assert(!DIAG || (D == 64 && !LARGE), "steps over diagonals: head dimension 64, small scores");
  extern __shared__ __align__(1024) uint8_t smem[];
  static_assert(sizeof(BwdBarriers) <= 512, "barrier block too large");
  BwdBarriers& bars = *reinterpret_cast<BwdBarriers*>(smem + Cfg::kOffBars);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (smem_u32(smem) & 1023u) {
    // swizzled tiles need 1024-byte alignment; uniform over the CTA, so every thread leaves here
    if (tid == 0 && p.status) atomicOr(p.status, 8);
    return;
  }
  if (tid == 0) {
    bars.abort_flag = 0;
    mbar_init(&bars.tile_full, 1);
    mbar_init(&bars.tile_free, (LARGE ? 1 : 3) + 8);   // the item's last products, and the fold warps (they read K1, SiLU(V1))
    for (int i = 0; i < kVecSlots; ++i) {
      mbar_init(&bars.vec_full[i], 1);
      mbar_init(&bars.vec_empty[i], 8);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars.a_ready[i], 4);
      mbar_init(&bars.a_free[i], 1);
      mbar_init(&bars.ap_ready[i], 4);
      mbar_init(&bars.ap_free[i], 1);
      mbar_init(&bars.ds_ready[i], 8);
      mbar_init(&bars.ds_free[i], 1);
    }
    mbar_init(&bars.r_ready, 2);
    mbar_init(&bars.s_ready, 1);
    mbar_init(&bars.s_free, 8);
    mbar_init(&bars.p_ready, 8);
    mbar_init(&bars.dp_ready, 1);
    mbar_init(&bars.acc_done[1], 1);
    mbar_init(&bars.acc_free[1], 4);
    mbar_init(&bars.acc_done[0], 1);
    mbar_init(&bars.acc_free[0], 4);
    mbar_init(&bars.qdo_ready, 8);
    mbar_init(&bars.dq_done, 1);
    mbar_init(&bars.dq_free, 8);
    fence_barrier_init();
  }
  if (warp == 16) {
    tmem_alloc(&bars.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;
  const BwdGeometry& g = p.g;
  const int T = g.T;
  // (every lane waits; the vote keeps the warp converged whatever a lane's wait returned)
  auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
    return __all_sync(0xffffffffu, LARGE ? mbar_wait(bar, parity, abort_flag) : mbar_wait_looks(bar, parity, abort_flag));
  };
  // the same for two barriers at once: half of the lanes look at each
  auto wait_two = [&](uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1) -> bool {
    const bool ok = wait_all(lane & 1 ? b1 : b0, lane & 1 ? p1 : p0);
    __syncwarp();
    return ok;
  };
  auto test_two = [&](uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1) -> bool {
    return mbar_test(lane & 1 ? b1 : b0, lane & 1 ? p1 : p0);
  };
  // one arrival per warp, after the caller's fences
  auto arrive_warp = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };

  // The item of phase `items` of tile_full; false: there is none, or the wait ran out (`alive` is then cleared).
  auto next_item = [&](uint32_t items, BwdItem& it, bool& alive) -> bool {
    alive = wait_all(&bars.tile_full, items & 1);
    if (!alive) return false;
    const int4 a = *reinterpret_cast<const int4*>(&bars.items[items % kItemSlots]);
    const int4 b = *reinterpret_cast<const int4*>(&bars.items[items % kItemSlots].len);
    // (every lane has the same; the reductions tell the compiler so, which keeps what follows from them on the uniform datapath:
    // with large scores 16 heads T=512 D=64 fp16 936 -> 927 us, 4 heads T=300 123 -> 122; with small ones less than runs differ)
    auto uniform = [](int v) -> int { return __reduce_max_sync(0xffffffffu, v); };
    it.bh = uniform(a.x); it.qt = uniform(a.y); it.jt = uniform(a.z); it.k0 = uniform(a.w);
    it.len = uniform(b.x); it.flags = uniform(b.y); it.ea = uniform(b.z); it.eb = uniform(b.w);
    if (LARGE) it.er = bars.items[items % kItemSlots].er;
    return it.len > 0;
  };

  if (warp < 8) {
    set_regs<kRegsLaunch, BwdRegs<D, LARGE, DIAG>::kSoftmax>();
    // ------------------------------------------------------------------ soft-max warpgroups
    const int wg = warp >> 2, wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    uint8_t* const prow = smem + Cfg::kOffP + (JT == 128 ? wg * 16384 : 0);
    const int ch0 = JT == 128 ? 0 : wg * 4;    // first 16-byte chunk of this thread's columns in its 128-byte row
    uint32_t n = 0, runs = 0, items = 0;
    bool alive = true;
    BwdItem it;
    int q = 0;
    bool q_ok = false, single = false, s_seen = false;
    float lse2 = 0.f, drow = 0.f, dq_scale = 0.f;
    // S and dP carry factors: in fp16 powers of two, and S = Q A^T lacks alpha * log2(e), which R carries
    constexpr bool kScaled = !LARGE || std::is_same<T16, __half>::value;
    constexpr int H = CW / 2;
    while (alive && next_item(items, it, alive)) {
      ++items;
      if (it.flags & kFirstOfQ) {
        const int i = it.qt * 128 + row;
        q_ok = i < g.nq && i >= p.i_first;
        q = g.q_rem + (q_ok ? i : 0) * g.q_mod;
        const int e = prob_shift<T16>(g.q_rem + max(it.qt * 128, p.i_first) * g.q_mod, g.causal, T, g.k1w, g.k2w);
        // (a row that is not this kernel's has P = 0 and a zero row of Q and dO, and needs Dq = 0 as well: 0 * (dP - Dq)
        // of another query's infinite or NaN Dq would be NaN, which G sums into every key the tile meets)
        lse2 = q_ok ? __ldg(p.lse + (size_t)it.bh * T + q) * kLog2e - (float)e : 0.f;
        const int f = it.flags >> kShiftBits;
        drow = q_ok ? __ldg(p.drow + (size_t)it.bh * T + q) * pow2i<T16>(f) : 0.f;
        dq_scale = pow2i<T16>(-e - it.ea - f) * p.alpha;
        // A query that attends a single pair has P = 1 and a score gradient of exactly zero (TdpMask::single_pair):
        // P (dP - Dq) has two terms that are equal only up to the 16-bit rounding of the stored output, so its dS
        // is set to zero.
        {
          // this query's row of Q (warpgroup 0) or dO (warpgroup 1) as the score products' operand in tensor memory
          // (the previous run's products have all run: its dq_done was waited for)
          const T16* src = (const T16*)(wg == 0 ? p.q : p.d_o) + ((size_t)it.bh * T + q) * D;
#pragma unroll
          for (int c = 0; c < D; c += 32) {
            uint32_t v[16];
#pragma unroll
            for (int e4 = 0; e4 < 4; ++e4) {
              const uint4 x = q_ok ? __ldg(reinterpret_cast<const uint4*>(src + c + e4 * 8)) : make_uint4(0, 0, 0, 0);
              v[e4 * 4] = x.x;
              v[e4 * 4 + 1] = x.y;
              v[e4 * 4 + 2] = x.z;
              v[e4 * 4 + 3] = x.w;
            }
            tmem_st16(tmem + lane_base + (wg == 0 ? Cfg::kTmemQ : Cfg::kTmemDO) + c / 2, v);
          }
          tmem_wait_st();
          tc_fence_before();
          arrive_warp(&bars.qdo_ready);
        }
        single = TdpMask{g.causal, T, g.k1w, g.k2w, g.kkl, g.kkr}.single_pair(q);
      }
      const bool any_single = __any_sync(0xffffffffu, single);
      const float2 nlse = make_float2(-lse2, -lse2);
      const float2 ndq = kScaled && single ? make_float2(0.f, 0.f) : make_float2(-drow, -drow);
      // (R carries alpha * log2(e), A does not)
      const float sa = LARGE ? pow2i<T16>(-it.er) : pow2i<T16>(-it.ea) * (p.alpha * kLog2e);
      const float sb = single ? 0.f : pow2i<T16>((it.flags >> kShiftBits) - it.eb);
      // v * scale + add; without the scale where it is 1
      auto scaled = [](uint32_t v0, uint32_t v1, float scale, float2 add) {
        const float2 v = make_float2(__uint_as_float(v0), __uint_as_float(v1));
        return kScaled ? __ffma2_rn(v, make_float2(scale, scale), add) : __fadd2_rn(v, add);
      };
      const int j0 = g.j_row(it.jt) + wg * CW;
      for (int i = 0; i < it.len; ++i, ++n) {
        const int k = it.k0 + i;
        // columns this query sees at this k, relative to the thread's first: [lo, hi] (empty: hi < lo)
        int lo = -j0, hi = T - 1 - j0;
        if (DIAG) {   // (k counts diagonals from -kkr)
          const int d = k - g.kkr;
          lo = max(max(q - g.k1w, q - d - g.k2w), max(0, -d)) - j0;
          hi = min(q, q - d) - j0;
        } else if (g.causal) {
          lo = max(max(q - g.k1w, k - g.kkl), 0) - j0;   // (an overlapping tile may begin ahead of row 0)
          hi = k <= q && q - k <= g.k2w ? min(q, k + g.kkr) - j0 : lo - 1;
        }
        if (!q_ok) hi = lo - 1;
        alive = __all_sync(0xffffffffu, s_seen) || wait_all(&bars.s_ready, n & 1);
        if (!alive) break;
        tc_fence_after();
        uint8_t* const dsrow = prow + (1 + (n & 1)) * Cfg::kTileP;
        const bool full = __all_sync(0xffffffffu, lo <= 0 && hi >= CW - 1);
        if constexpr (LARGE) {
          // 32 columns at a time: S -> P, then dP and P (still in fp32) -> dS.  (What the other body does, half of the columns beside
          // the other half, gains nothing behind one issuing warp, and spills: 944 against 920 us at 16 heads of T=512 D=64 fp16,
          // 5460 against 5320 at T=1024 D=128 8 heads.)
#pragma unroll 1
          for (int c0 = 0; c0 < CW; c0 += 32) {
            uint32_t s[32];
            tmem_ld32(tmem + lane_base + Cfg::kTmemS + wg * CW + c0, s);
            tmem_wait_ld();
            if (c0 + 32 == CW) {
              // the scores are in registers: the next step's product may overwrite them
              tc_fence_before();
              arrive_warp(&bars.s_free);
            }
            if (full) {
#pragma unroll
              for (int c = 0; c < 32; c += 2) {
                const float2 x = scaled(s[c], s[c + 1], sa, nlse);
                s[c] = __float_as_uint(exp2f(x.x));
                s[c + 1] = __float_as_uint(exp2f(x.y));
              }
            } else {
#pragma unroll
              for (int c = 0; c < 32; ++c)
                s[c] = c0 + c >= lo && c0 + c <= hi ? __float_as_uint(exp2f(fmaf(__uint_as_float(s[c]), sa, -lse2))) : 0u;
            }
            if (c0 == 0) {
              // the previous step's U has read P
              alive = wait_all(&bars.acc_done[1], (n & 1) ^ 1);
              if (!alive) break;
            }
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e)
                w[e] = pack2<T16>(__uint_as_float(s[c + 2 * e]), __uint_as_float(s[c + 2 * e + 1]));
              *reinterpret_cast<uint4*>(prow + swz128(row, ch0 + ((c0 + c) >> 3))) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            if (c0 + 32 == CW) {
              fence_async_smem();
              arrive_warp(&bars.p_ready);
            }
            if (any_single) {
#pragma unroll
              for (int c = 0; c < 32; ++c) s[c] = single ? 0u : s[c];
            }
            if (c0 == 0) {
              alive = wait_all(&bars.dp_ready, n & 1);
              if (alive) alive = wait_all(&bars.ds_free[n & 1], ((n >> 1) & 1) ^ 1);
              if (!alive) break;
              tc_fence_after();
            }
#pragma unroll
            for (int c1 = 0; c1 < 32; c1 += 16) {
              uint32_t dp[16];
              tmem_ld16(tmem + lane_base + Cfg::kTmemDP + wg * CW + c0 + c1, dp);
              tmem_wait_ld();
#pragma unroll
              for (int c = 0; c < 16; c += 8) {
                uint32_t w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 d = scaled(dp[c + 2 * e], dp[c + 2 * e + 1], sb, ndq);
                  const float2 ds = __fmul2_rn(
                      make_float2(__uint_as_float(s[c1 + c + 2 * e]), __uint_as_float(s[c1 + c + 2 * e + 1])), d);
                  w[e] = pack2<T16>(ds.x, ds.y);
                }
                *reinterpret_cast<uint4*>(dsrow + swz128(row, ch0 + ((c0 + c1 + c) >> 3))) = make_uint4(w[0], w[1], w[2], w[3]);
              }
            }
          }
          if (!alive) break;
        } else {
          // Half of the columns S -> P; then, eight columns at a time, the other half S -> P beside dP and P (still in fp32) ->
          // dS of the first, so that exponentials and arithmetic overlap within a warp; then dS of the second half.
          bool seen = false;   // (looks at barriers ahead of their waits)
          const uint32_t tS = tmem + lane_base + Cfg::kTmemS + wg * CW, tDP = tmem + lane_base + Cfg::kTmemDP + wg * CW;
          constexpr int SN = D == 128 ? H : 8;   // (head dimension 64 has no registers for all of them)
          uint32_t s[H], sn[SN], dp[8];   // scores, then P; scores of the second half; dP
          // (most steps over a diagonal are masked: a bit of a mask is one instruction, two comparisons are two)
          uint32_t mask[2] = {0, 0};
          if constexpr (DIAG) {
            mask[0] = column_mask(lo, hi);
            mask[1] = column_mask(lo - 32, hi - 32);
          }
          // columns c.. of S -> P
          auto to_p = [&](int c, uint32_t* v, const uint32_t* x) {
            if (full) {
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                const float2 y = scaled(x[e], x[e + 1], sa, nlse);
                v[e] = __float_as_uint(exp2f(y.x));
                v[e + 1] = __float_as_uint(exp2f(y.y));
              }
            } else if constexpr (DIAG) {
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                const uint32_t m = mask[c >> 5] >> ((c + e) & 31);
                const float2 y = scaled(x[e], x[e + 1], sa, nlse);
                v[e] = m & 1u ? __float_as_uint(exp2f(y.x)) : 0u;
                v[e + 1] = m & 2u ? __float_as_uint(exp2f(y.y)) : 0u;
              }
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e)
                v[e] = c + e >= lo && c + e <= hi ? __float_as_uint(exp2f(fmaf(__uint_as_float(x[e]), sa, -lse2))) : 0u;
            }
          };
          auto put = [&](uint8_t* row_base, int c, const uint32_t* v) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = pack2<T16>(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
            *reinterpret_cast<uint4*>(row_base + swz128(row, ch0 + (c >> 3))) = make_uint4(w[0], w[1], w[2], w[3]);
          };
          // columns c..: P in v and dP in dp -> dS
          auto to_ds = [&](int c, const uint32_t* v) {
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              float2 pv = make_float2(__uint_as_float(v[e]), __uint_as_float(v[e + 1]));
              if (!kScaled && any_single) pv = single ? make_float2(0.f, 0.f) : pv;
              const float2 ds = __fmul2_rn(pv, scaled(dp[e], dp[e + 1], sb, ndq));
              w[e] = __float_as_uint(ds.x);
              w[e + 1] = __float_as_uint(ds.y);
            }
            put(dsrow, c, w);
          };
          tmem_ld(tS, s);
          tmem_wait_ld(s);
          seen = mbar_test(&bars.acc_done[1], (n & 1) ^ 1);
          tmem_ld(tS + H, sn);
#pragma unroll
          for (int c = 0; c < H; c += 8) to_p(c, s + c, s + c);
          // the previous step's U has read P
          alive = __all_sync(0xffffffffu, seen) || wait_all(&bars.acc_done[1], (n & 1) ^ 1);
          if (!alive) break;
          seen = test_two(&bars.dp_ready, n & 1, &bars.ds_free[n & 1], ((n >> 1) & 1) ^ 1);
#pragma unroll
          for (int c = 0; c < H; c += 8) put(prow, c, s + c);
          alive = __all_sync(0xffffffffu, seen) || wait_two(&bars.dp_ready, n & 1, &bars.ds_free[n & 1], ((n >> 1) & 1) ^ 1);
          if (!alive) break;
          tc_fence_after();
          tmem_ld(tDP, dp);
#pragma unroll
          for (int c = 0; c < H; c += 8) {
            tmem_wait_ld(sn, dp);
            if (SN == H ? c == 0 : c + 8 == H) {
              // the scores are in registers: the next step's product may overwrite them
              tc_fence_before();
              arrive_warp(&bars.s_free);
            }
            uint32_t x[8];
            to_ds(c, s + c);
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = sn[SN == H ? c + e : e];
            tmem_ld(tDP + c + 8, dp);
            if constexpr (SN == 8) {
              if (c + 8 < H) tmem_ld(tS + H + c + 8, sn);
            }
            to_p(H + c, s + c, x);
            put(prow, H + c, s + c);
          }
          fence_async_smem();
          arrive_warp(&bars.p_ready);
          s_seen = mbar_test(&bars.s_ready, (n + 1) & 1);
#pragma unroll
          for (int c = 0; c < H; c += 8) {
            tmem_wait_ld(dp);
            to_ds(H + c, s + c);
            if (c + 8 < H) tmem_ld(tDP + H + c + 8, dp);
          }
        }
        tc_fence_before();
        fence_async_smem();
        arrive_warp(&bars.ds_ready[n & 1]);
      }
      if (!alive) break;
      if ((it.flags & kLastOfQ)) {
        // ---- dQ of this q-tile (over the j-tiles this CTA had of it): half of the columns per warpgroup
        alive = wait_all(&bars.dq_done, runs & 1);
        if (!alive) break;
        tc_fence_after();
        float* dst = p.dq + ((size_t)it.bh * T + q) * D + wg * (D / 2);
#pragma unroll
        for (int c0 = 0; c0 < D / 2; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(tmem + lane_base + Cfg::kTmemDQ + wg * (D / 2) + c0, v);
          tmem_wait_ld();
          if (q_ok) {
#pragma unroll
            for (int c = 0; c < 32; c += 4)
              red_add4(dst + c0 + c, __uint_as_float(v[c]) * dq_scale, __uint_as_float(v[c + 1]) * dq_scale,
                       __uint_as_float(v[c + 2]) * dq_scale, __uint_as_float(v[c + 3]) * dq_scale);
          }
        }
        tc_fence_before();
        arrive_warp(&bars.dq_free);
        ++runs;
      }
    }
  } else if (warp < 16) {
    set_regs<kRegsLaunch, BwdRegs<D, LARGE, DIAG>::kFold>();
    // ------------------------------------------------------------------ operand / fold warpgroups
    // role 0: forms A two steps ahead, folds G into dK1 (registers) and dK2;  role 1: forms A' two steps ahead (large scores: one), folds
    // U into dSiLU(V1) and dV2.  The fold reads the accumulator as 16 x 256-bit fragments (thread t: rows t / 4 + 8 i,
    // columns 8 g + 2 (t % 4) and the next), which is also how ldmatrix hands out the K1 / SiLU(V1) tile: the sums
    // over the 32 rows of a warp are four rows within a thread and a 7-shuffle tree per 32 columns.
    // (the role is a run-time value: one copy of the code for both warpgroups halves what the instruction caches have to
    // hold of it)
    const int role = (warp - 8) >> 2, w = warp & 3;
    const T16* const vec = reinterpret_cast<const T16*>(smem + Cfg::kOffVec + role * Cfg::kVecPart);
    // row of step i of an item whose first batch is vb0
    auto vec_row = [&](uint32_t vb0, int i) {
      return vec + ((vb0 + i / kVecBatch) % kVecSlots * 2 * kVecBatch + i % kVecBatch) * D;
    };
    const uint32_t tacc = tmem + ((uint32_t)(w * 32) << 16) + (role ? Cfg::kTmemU : Cfg::kTmemG);
    const int ahead = kOneAp ? 2 - role : 2;   // (A' has a second buffer, over the SiLU(V1) tile, where R does not need that)
    // address of this lane's row of the four 8 x 8 blocks of (16-column group c16, 16-lane half hl) within a tile
    auto frag = [&](int c16, int hl) -> uint32_t {
      if constexpr (D == 64) {
        // (j 0-7, h 0-7), (j 8-15, h 0-7), (j 0-7, h 8-15), (j 8-15, h 8-15)
        return swz128(w * 32 + hl * 16 + (lane & 15), c16 * 2 + (lane >> 4));
      } else {
        // (h 0-7, j 0-7), (h 8-15, j 0-7), (h 0-7, j 8-15), (h 8-15, j 8-15), transposed
        const int ch = w * 4 + hl * 2 + ((lane >> 3) & 1), j = c16 * 16 + (lane >> 4) * 8 + (lane & 7);
        return (ch >> 3) * (JT * 128) + swz128(j, ch & 7);
      }
    };
    // (DIAG: row j of the tile meets row k = j + n - kkr on diagonal n, which is row j + n of the window)
    const uint32_t window_u = smem_u32(smem + Cfg::kOffK1 + role * Cfg::kWindow);
    auto window_frag = [&](int n, int c16, int hl) -> uint32_t {
      return window_u + swz128(w * 32 + hl * 16 + (lane & 15) + n, c16 * 2 + (lane >> 4));
    };
    const uint32_t raw_u = smem_u32(smem + Cfg::kOffK1 + role * Cfg::kTileJ);
    const uint32_t formed_u = smem_u32(smem + Cfg::kOffA + role * 2 * Cfg::kTileJ);
    uint32_t n = 0, items = 0, vb0 = 0;
    bool alive = true;
    BwdItem it;
    while (alive && next_item(items, it, alive)) {
      float2 acc[32];   // [16-column group c16][16-lane half][8-column group][row of the pair]
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = make_float2(0.f, 0.f);
      uint32_t x[4][2][4];   // this thread's elements of the K1 / SiLU(V1) tile, [c16][hl][8 x 8 block]
#pragma unroll
      for (int c16 = 0; c16 < 4; ++c16)
#pragma unroll
        for (int hl = 0; hl < 2; ++hl) {
          if constexpr (DIAG) {
            const T16* src = (const T16*)(role ? p.sv1 : p.k1) + (size_t)it.bh * T * D + c16 * 16 + 2 * (lane & 3);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const int j = it.jt * JT + w * 32 + hl * 16 + (b & 1) * 8 + (lane >> 2);
              x[c16][hl][b] = j < T ? __ldg(reinterpret_cast<const uint32_t*>(src + (size_t)j * D + (b >> 1) * 8)) : 0u;
            }
          } else if constexpr (D == 64) ldmatrix_x4(x[c16][hl], raw_u + frag(c16, hl));
          else ldmatrix_x4_trans(x[c16][hl], raw_u + frag(c16, hl));
        }
      if (!DIAG) arrive_warp(&bars.tile_free);
      int j_lo, j_hi;
      if (!DIAG && g.overlapping()) {
        g.j_rows(it.qt, it.jt, j_lo, j_hi);
        // (rows beyond those that a query of the tile sees, which tiles side by side end with, would bring 0 * inf to its sums)
#pragma unroll
        for (int c16 = 0; c16 < 4; ++c16)
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            uint32_t& v = x[c16][b >> 2][b & 3];
            if constexpr (D == 64) {
              const int r = w * 32 + (b >> 2) * 16 + (b & 1) * 8 + (lane >> 2);
              v = r >= j_lo && r < j_hi ? v : 0u;
            } else {
              const int r = c16 * 16 + (b >> 1 & 1) * 8 + 2 * (lane & 3);
              v &= (r >= j_lo && r < j_hi ? 0xffffu : 0u) | (r + 1 >= j_lo && r + 1 < j_hi ? 0xffff0000u : 0u);
            }
          }
      }
      const int ex = role ? it.eb : it.ea;   // (x carries 2^ex from here on)
      if (std::is_same<T16, __half>::value) {
        const float2 m = make_float2(pow2i<T16>(ex), pow2i<T16>(ex));
#pragma unroll
        for (int c16 = 0; c16 < 4; ++c16)
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const float2 f = __fmul2_rn(unpack2<T16>(x[c16][b >> 2][b & 3]), m);
            x[c16][b >> 2][b & 3] = pack2<T16>(f.x, f.y);
          }
      }
      const int len = it.len;
      const int e = prob_shift<T16>(g.q_rem + max(it.qt * 128, p.i_first) * g.q_mod, g.causal, T, g.k1w, g.k2w);
      const float unshift = pow2i<T16>(-e);
      const float unshift_ds = unshift * pow2i<T16>(-(it.flags >> kShiftBits));
      const float jscale = role ? unshift : unshift_ds * p.alpha;
      const float zscale = jscale * pow2i<T16>(-ex);
      float* zrow = (role ? p.dv2 : p.dk2) + ((size_t)it.bh * T + it.k0) * D;
      // (DIAG: only rows k that a query of the tile sees: the others' products are zero, or NaN beside an infinite row)
      int k_row0 = 0;
      unsigned k_rows = 0;
      if (DIAG) {
        const int k_lo = max(0, it.qt * 128 - g.k2w);
        k_row0 = it.jt * JT - g.kkr + it.k0 + w * 32 + (lane >> 2) - k_lo;
        k_rows = (unsigned)(min(it.qt * 128 + 128, T) - k_lo);
      }
      if (DIAG) zrow += (ptrdiff_t)(it.jt * JT - g.kkr + w * 32 + (lane >> 2)) * D + ((lane & 1) << 3) + ((lane & 2) << 1);
      auto form = [&](int i) -> bool {
        const uint32_t m = n + i;
        // The operand's buffer: the product of its last step has run (A: two steps before, through dQ; A': dP, two steps before,
        // or with a single buffer the step before).  At the first row of a batch half of the lanes look whether it is there.
        const uint32_t mb = kOneAp && role ? m - 1 : m, vb = vb0 + i / kVecBatch;
        uint64_t* const bar = role ? &bars.ap_free[mb & 1] : &bars.a_free[mb & 1];
        const uint32_t parity = ((mb >> 1) & 1) ^ (kOneAp && role ? 0 : 1);
        const bool first = !DIAG && (i & (kVecBatch - 1)) == 0;
        if (!wait_two(bar, parity, first ? &bars.vec_full[vb % kVecSlots] : bar, first ? (vb / kVecSlots) & 1 : parity)) return false;
        const T16* v = vec_row(vb0, i);
        const uint32_t dst = role == 0 ? formed_u + (m & 1) * Cfg::kTileJ : kOneAp || !(m & 1) ? formed_u : raw_u;
        uint32_t vr[4];   // head dimension 128: twice the element of row r
        if constexpr (D == 128) {
#pragma unroll
          for (int r = 0; r < 4; ++r)
            vr[r] = __byte_perm(*reinterpret_cast<const uint16_t*>(v + w * 32 + r * 8 + (lane >> 2)), 0, 0x1010);
        }
        if constexpr (DIAG) {
          // (two fragments at a time, or each read waits for the store before; four spill)
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            uint32_t a[2][4];
#pragma unroll
            for (int e = 0; e < 2; ++e) ldmatrix_x4(a[e], window_frag(it.k0 + i, (c + e) >> 1, (c + e) & 1));
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int c16 = (c + e) >> 1, hl = (c + e) & 1;
#pragma unroll
              for (int b = 0; b < 4; ++b) a[e][b] = mul2<T16>(x[c16][hl][b], a[e][b]);
              stmatrix_x4(dst + frag(c16, hl), a[e]);
            }
          }
        } else
#pragma unroll
        for (int c16 = 0; c16 < 4; ++c16) {
          uint32_t v0 = 0, v1 = 0;
          if constexpr (D == 64) {
            v0 = *reinterpret_cast<const uint32_t*>(v + c16 * 16 + 2 * (lane & 3));
            v1 = *reinterpret_cast<const uint32_t*>(v + c16 * 16 + 8 + 2 * (lane & 3));
          }
#pragma unroll
          for (int hl = 0; hl < 2; ++hl) {
            uint32_t a[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) a[b] = mul2<T16>(x[c16][hl][b], D == 64 ? (b < 2 ? v0 : v1) : vr[hl * 2 + (b & 1)]);
            if constexpr (D == 64) stmatrix_x4(dst + frag(c16, hl), a);
            else stmatrix_x4_trans(dst + frag(c16, hl), a);
          }
        }
        fence_async_smem();
        arrive_warp(role ? &bars.ap_ready[kOneAp ? 0 : m & 1] : &bars.a_ready[m & 1]);
        return true;
      };
      // (one loop, so that there is one copy of each of the two stages: step i0 forms operand i0, folds step i0 - ahead)
      for (int i0 = 0; i0 < len + ahead && alive; ++i0) {
        const int i = i0 - ahead;
        // (keeps the compiler from unpacking x once, outside the loop, into twice the registers)
#pragma unroll
        for (int c16 = 0; c16 < 4; ++c16)
#pragma unroll
          for (int b = 0; b < 8; ++b) asm volatile("" : "+r"(x[c16][b >> 2][b & 3]));
        bool seen = false;   // (a look ahead of the wait)
        if (i >= 0) seen = mbar_test(&bars.acc_done[role], (n + i) & 1);
        if (i0 < len) {
          alive = form(i0);
          if (!alive) break;
        }
        if (i < 0) continue;
        alive = __all_sync(0xffffffffu, seen) || wait_all(&bars.acc_done[role], (n + i) & 1);
        if (!alive) break;
        tc_fence_after();
        const T16* v = vec_row(vb0, i);
        if constexpr (DIAG) {
          // Lanes are rows j, columns are h; row k = j + d of dK2 / dV2 gets K1 G / SiLU(V1) U.  Pairs of lanes swap halves, so that
          // a reduction takes four columns of a thread (with two of them, without exchanges, 820 us where this took 757).  Eight
          // rows by 16 columns at a time: with 16 by 16 the registers in flight spill (671 us for 642).
          const int k = k_row0 + i;   // from the first row that a query of the tile sees
          const bool odd = lane & 1;
          const float2 zs = make_float2(zscale, zscale);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int c16 = c >> 1, hl = c & 1;
            uint32_t d[8], vw[4];
            tmem_ld_16x256b_x2(tacc + ((uint32_t)(hl * 16) << 16) + c16 * 16, d);
            ldmatrix_x4(vw, window_frag(it.k0 + i, c16, hl));
            tmem_wait_ld();
            if (c == 7) {
              tc_fence_before();
              arrive_warp(&bars.acc_free[role]);
            }
            // (all exchanges ahead of the reductions: one waits for the other's answer else)
            float2 z0[2], z1[2], other[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const float2 g0 = make_float2(__uint_as_float(d[2 * r]), __uint_as_float(d[2 * r + 1]));
              const float2 g1 = make_float2(__uint_as_float(d[4 + 2 * r]), __uint_as_float(d[5 + 2 * r]));
              z0[r] = __fmul2_rn(__fmul2_rn(g0, unpack2<T16>(x[c16][hl][r])), zs);
              z1[r] = __fmul2_rn(__fmul2_rn(g1, unpack2<T16>(x[c16][hl][2 + r])), zs);
              other[r].x = __shfl_xor_sync(0xffffffffu, odd ? z0[r].x : z1[r].x, 1);
              other[r].y = __shfl_xor_sync(0xffffffffu, odd ? z0[r].y : z1[r].y, 1);
              float2& a0 = acc[c16 * 8 + hl * 4 + r];
              float2& a1 = acc[c16 * 8 + hl * 4 + 2 + r];
              a0 = __ffma2_rn(g0, unpack2<T16>(vw[r]), a0);
              a1 = __ffma2_rn(g1, unpack2<T16>(vw[2 + r]), a1);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const float2 o = other[r], u = z0[r], v = z1[r];
              if ((unsigned)(k + hl * 16 + r * 8) < k_rows)
                red_add4(zrow + (hl * 16 + r * 8) * D + c16 * 16, odd ? o.x : u.x, odd ? o.y : u.y, odd ? v.x : o.x, odd ? v.y : o.y);
            }
          }
        } else if constexpr (D == 64) {
          // lanes are rows j, columns are h
          float z2[8];
#pragma unroll
          for (int c16 = 0; c16 < 4; ++c16) {
            uint32_t d[2][8];
#pragma unroll
            for (int hl = 0; hl < 2; ++hl) tmem_ld_16x256b_x2(tacc + ((uint32_t)(hl * 16) << 16) + c16 * 16, d[hl]);
            const float2 v0 = unpack2<T16>(*reinterpret_cast<const uint32_t*>(v + c16 * 16 + 2 * (lane & 3)));
            const float2 v1 = unpack2<T16>(*reinterpret_cast<const uint32_t*>(v + c16 * 16 + 8 + 2 * (lane & 3)));
            tmem_wait_ld();
            if (c16 == 3) {
              tc_fence_before();
              arrive_warp(&bars.acc_free[role]);
            }
            float2 z0 = make_float2(0.f, 0.f), z1 = z0;
#pragma unroll
            for (int hl = 0; hl < 2; ++hl) {
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const float2 g0 = make_float2(__uint_as_float(d[hl][2 * r]), __uint_as_float(d[hl][2 * r + 1]));
                const float2 g1 = make_float2(__uint_as_float(d[hl][4 + 2 * r]), __uint_as_float(d[hl][5 + 2 * r]));
                float2& a0 = acc[c16 * 8 + hl * 4 + r];
                float2& a1 = acc[c16 * 8 + hl * 4 + 2 + r];
                a0 = __ffma2_rn(g0, v0, a0);
                a1 = __ffma2_rn(g1, v1, a1);
                z0 = __ffma2_rn(g0, unpack2<T16>(x[c16][hl][r]), z0);
                z1 = __ffma2_rn(g1, unpack2<T16>(x[c16][hl][2 + r]), z1);
              }
            }
            // z0, z1: columns 16 c16 + 2 (lane % 4) and the next, and those 8 further, over this thread's four rows.  The sum
            // over lane / 4 is a tree; its first exchange, here beside the reads, leaves columns 8 g.. with g = lane bit 4
            const bool upper = lane & 16;
            z2[2 * c16] = (upper ? z1.x : z0.x) + __shfl_xor_sync(0xffffffffu, upper ? z0.x : z1.x, 16);
            z2[2 * c16 + 1] = (upper ? z1.y : z0.y) + __shfl_xor_sync(0xffffffffu, upper ? z0.y : z1.y, 16);
          }
          // z2[2 c16 + e]: column 16 c16 + 8 (lane bit 4) + 2 (lane % 4) + e; two more exchanges leave two columns per lane:
          // c16 = 2 (lane bit 3) + (lane bit 2)
#pragma unroll
          for (int half = 4; half >= 2; half >>= 1) {
            const bool upper = lane & (half * 2);
#pragma unroll
            for (int i2 = 0; i2 < half; ++i2) {
              const float keep = upper ? z2[i2 + half] : z2[i2];
              const float send = upper ? z2[i2] : z2[i2 + half];
              z2[i2] = keep + __shfl_xor_sync(0xffffffffu, send, half * 2);
            }
          }
          const int col = ((lane >> 2) & 3) * 16 + (lane >> 4) * 8 + 2 * (lane & 3);
          red_add2(zrow + col, z2[0] * zscale, z2[1] * zscale);
        } else {
          // lanes are columns h of the head, columns are rows j
          float2 z[4];
          float vr[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            z[r] = make_float2(0.f, 0.f);
            vr[r] = to_f(v[w * 32 + r * 8 + (lane >> 2)]);
          }
#pragma unroll
          for (int c16 = 0; c16 < 4; ++c16) {
            uint32_t d[2][8];
#pragma unroll
            for (int hl = 0; hl < 2; ++hl) tmem_ld_16x256b_x2(tacc + ((uint32_t)(hl * 16) << 16) + c16 * 16, d[hl]);
            tmem_wait_ld();
            if (c16 == 3) {
              tc_fence_before();
              arrive_warp(&bars.acc_free[role]);
            }
#pragma unroll
            for (int hl = 0; hl < 2; ++hl) {
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const float2 g0 = make_float2(__uint_as_float(d[hl][2 * r]), __uint_as_float(d[hl][2 * r + 1]));
                const float2 g1 = make_float2(__uint_as_float(d[hl][4 + 2 * r]), __uint_as_float(d[hl][5 + 2 * r]));
                const float2 vv = make_float2(vr[hl * 2 + r], vr[hl * 2 + r]);
                float2& a0 = acc[c16 * 8 + hl * 4 + r];
                float2& a1 = acc[c16 * 8 + hl * 4 + 2 + r];
                a0 = __ffma2_rn(g0, vv, a0);
                a1 = __ffma2_rn(g1, vv, a1);
                float2& zz = z[hl * 2 + r];
                zz = __ffma2_rn(g0, unpack2<T16>(x[c16][hl][r]), zz);
                zz = __ffma2_rn(g1, unpack2<T16>(x[c16][hl][2 + r]), zz);
              }
            }
          }
          // z[r]: h = 32 w + 8 r + lane / 4 over this thread's 16 columns; the tree over lane % 4 leaves row r =
          // 2 (lane bit 1) + (lane bit 0)
          float zr[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) zr[r] = z[r].x + z[r].y;
#pragma unroll
          for (int half = 2; half >= 1; half >>= 1) {
            const bool upper = lane & half;
#pragma unroll
            for (int i2 = 0; i2 < half; ++i2) {
              const float keep = upper ? zr[i2 + half] : zr[i2];
              const float send = upper ? zr[i2] : zr[i2 + half];
              zr[i2] = keep + __shfl_xor_sync(0xffffffffu, send, half);
            }
          }
          red_add(zrow + w * 32 + (lane & 3) * 8 + (lane >> 2), zr[0] * zscale);
        }
        if (!DIAG && ((i & (kVecBatch - 1)) == kVecBatch - 1 || i == len - 1))
          arrive_warp(&bars.vec_empty[(vb0 + i / kVecBatch) % kVecSlots]);
        zrow += D;
      }
      if (!alive) break;
      if (DIAG) arrive_warp(&bars.tile_free);   // (the window has been read)
      n += len;
      vb0 += (len + kVecBatch - 1) / kVecBatch;
      ++items;
      // ---- dK1 / dSiLU(V1) of this item
      p.g.j_rows(it.qt, it.jt, j_lo, j_hi);
      float* const base = (role ? p.dsv1 : p.dk1) + ((ptrdiff_t)it.bh * T + p.g.j_row(it.jt)) * D;
#pragma unroll
      for (int c16 = 0; c16 < 4; ++c16)
#pragma unroll
        for (int hl = 0; hl < 2; ++hl)
#pragma unroll
          for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const float2 a = acc[c16 * 8 + hl * 4 + g * 2 + r];
              const int lr = w * 32 + hl * 16 + r * 8 + (lane >> 2), lc = c16 * 16 + g * 8 + 2 * (lane & 3);
              if constexpr (D == 64) {
                if (lr >= j_lo && lr < j_hi) red_add2(base + lr * D + lc, a.x * jscale, a.y * jscale);
              } else {
                if (lc >= j_lo && lc < j_hi) red_add(base + lc * D + lr, a.x * jscale);
                if (lc + 1 >= j_lo && lc + 1 < j_hi) red_add(base + (lc + 1) * D + lr, a.y * jscale);
              }
            }
    }
  } else {
   set_regs<kRegsLaunch, BwdRegs<D, LARGE, DIAG>::kService>();
   if (warp == 16 || (!LARGE && warp >= 18)) {
    const bool do_rows = warp == 16, do_u = LARGE || warp == 18, do_ds = LARGE || warp == 19;
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the schedule in step and one elected lane issues: with converged control flow the
    // descriptor arithmetic stays on the uniform datapath, where a lone thread needs a register-to-uniform move
    // per operand and loses its issue slots to the busy warps of its scheduler.
    const bool leader = elect_one();
    constexpr int kFmt = std::is_same<T16, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t kHi = desc_hi(1024);
    constexpr uint32_t idesc_s = make_idesc_f16(128, JT, kFmt, false, false);
    constexpr uint32_t idesc_g = make_idesc_f16(128, 64, kFmt, true, true);
    constexpr uint32_t idesc_dq = make_idesc_f16(128, D, kFmt, false, true);
    // (leading-byte offsets: distance of 64-element blocks along M / N of a row-major tile)
    const uint32_t qLo = desc_lo(smem_u32(smem + Cfg::kOffQ), 16384), doLo = desc_lo(smem_u32(smem + Cfg::kOffDO), 16384);
    const uint32_t aLo = desc_lo(smem_u32(smem + Cfg::kOffA), JT * 128);
    const uint32_t a2Lo = desc_lo(smem_u32(smem + Cfg::kOffA + 2 * Cfg::kTileJ), JT * 128);
    const uint32_t sv1Lo = desc_lo(smem_u32(smem + Cfg::kOffK1 + Cfg::kTileJ), JT * 128);
    const uint32_t rLo[2] = {desc_lo(smem_u32(smem + Cfg::kOffR0), 16), desc_lo(smem_u32(smem + Cfg::kOffR1), 16)};
    const uint32_t k1Lo = desc_lo(smem_u32(smem + Cfg::kOffK1), 16);
    const uint32_t pLo = desc_lo(smem_u32(smem + Cfg::kOffP), 16384);
    constexpr uint32_t kTileP16 = Cfg::kTileP >> 4, kTileJ16 = Cfg::kTileJ >> 4;
    auto commit = [&](uint64_t* bar) {
      if (leader) mma_commit(bar);
    };
    // S = Q A^T and dP = dO A'^T: Q / dO from tensor memory, A / A' K-major, D / 16 instructions
    auto issue_rows = [&](uint32_t dcol, uint32_t acol, uint32_t lo_b) {
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
        if (leader)
          mma_ts_lo(tmem + dcol, tmem + acol + k * 8, lo_b + (k >> 2) * ((JT * 128) >> 4) + (k & 3) * 2, kHi, idesc_s, k > 0);
    };
    // G = dS^T Q, U = P^T dO (head dimension 128: the transposes): contraction over the 128 queries, both row-major
    auto issue_fold = [&](uint32_t dcol, uint32_t lo_p, uint32_t lo_q) {
      const uint32_t lo_a = D == 64 ? lo_p : lo_q, lo_b = D == 64 ? lo_q : lo_p;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (leader) mma_ss_lo(tmem + dcol, lo_a + k * (2048 >> 4), lo_b + k * (2048 >> 4), kHi, idesc_g, k > 0);
    };
    // dQ += dS A: contraction over the JT rows j
    auto issue_dq = [&](uint32_t lo_ds, uint32_t lo_a, uint32_t acc) {
#pragma unroll
      for (int k = 0; k < JT / 16; ++k)
        if (leader)
          mma_ss_lo(tmem + Cfg::kTmemDQ, lo_ds + (k >> 2) * (16384 >> 4) + (k & 3) * 2, lo_a + k * (2048 >> 4), kHi, idesc_dq,
                    k > 0 ? 1u : acc);
    };
    uint32_t n = 0, items = 0, runs = 0;
    bool alive = true;
    // Three warps issue: S and dP, U, dQ and G, each as soon as its operands are there.  One warp for all five held them back
    // behind each other's waits: a look at a barrier takes 100 to 200 cycles while the tensor cores read shared memory.  (Large
    // scores: one, as the other two form R.)
    auto issue_s = [&](uint32_t m) -> bool {
      if (!wait_two(LARGE ? &bars.r_ready : &bars.a_ready[m & 1], (LARGE ? m : m >> 1) & 1, &bars.s_free, (m & 1) ^ 1)) return false;
      tc_fence_after();
      if constexpr (LARGE) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          if (leader)
            mma_ss_lo(tmem + Cfg::kTmemS, rLo[k >> 2] + (k & 3) * 2, k1Lo + (k >> 2) * ((JT * 128) >> 4) + (k & 3) * 2, kHi, idesc_s,
                      k > 0);
      } else {
        issue_rows(Cfg::kTmemS, Cfg::kTmemQ, aLo + (m & 1) * kTileJ16);
      }
      commit(&bars.s_ready);
      return true;
    };
    // (the first step of an item has no dP before it that anyone still reads)
    auto issue_dp = [&](uint32_t m, bool after) -> bool {
      uint64_t* const ap = &bars.ap_ready[kOneAp ? 0 : m & 1];
      const uint32_t parity = (kOneAp ? m : m >> 1) & 1;
      if (!wait_two(ap, parity, after ? &bars.ds_ready[(m - 1) & 1] : ap, after ? ((m - 1) >> 1) & 1 : parity)) return false;
      tc_fence_after();
      issue_rows(Cfg::kTmemDP, Cfg::kTmemDO, kOneAp || !(m & 1) ? a2Lo : sv1Lo);
      commit(&bars.dp_ready);
      commit(&bars.ap_free[m & 1]);
      return true;
    };
    BwdItem it;
    while (alive && next_item(items, it, alive)) {
      if (it.flags & kFirstOfQ) {
        alive = wait_all(&bars.qdo_ready, runs & 1);   // (runs: q-tiles finished)
        if (!alive) break;
        tc_fence_after();
      }
      if (do_rows) alive = issue_s(n) && issue_dp(n, false);
      for (int i = 0; i < it.len && alive; ++i, ++n) {
        const bool more = i + 1 < it.len;
        alive = false;
        if (do_rows && more && !(issue_s(n + 1) && (LARGE || issue_dp(n + 1, true)))) break;
        if (do_u) {
          if (!wait_two(&bars.p_ready, n & 1, &bars.acc_free[1], (n & 1) ^ 1)) break;
          tc_fence_after();
          issue_fold(Cfg::kTmemU, pLo, doLo);
          commit(&bars.acc_done[1]);
        }
        if (do_ds) {
          const bool g_free = mbar_test(&bars.acc_free[0], (n & 1) ^ 1);
          if (!wait_all(&bars.ds_ready[n & 1], (n >> 1) & 1)) break;
          tc_fence_after();
          if (LARGE && more && !issue_dp(n + 1, true)) break;
          const bool fresh = i == 0 && (it.flags & kFirstOfQ);
          if (fresh) {
            // the previous q-tile's dQ has been read
            if (!wait_all(&bars.dq_free, (runs & 1) ^ 1)) break;
            tc_fence_after();
          }
          if constexpr (LARGE) {
            if (!wait_all(&bars.a_ready[n & 1], (n >> 1) & 1)) break;
            tc_fence_after();
          }
          const uint32_t ds = pLo + (1 + (n & 1)) * kTileP16;
          issue_dq(ds, aLo + (n & 1) * kTileJ16, fresh ? 0u : 1u);
          commit(&bars.a_free[n & 1]);
          if (!__all_sync(0xffffffffu, g_free) && !wait_all(&bars.acc_free[0], (n & 1) ^ 1)) break;
          tc_fence_after();
          issue_fold(Cfg::kTmemG, ds, qLo);
          commit(&bars.acc_done[0]);
          commit(&bars.ds_free[n & 1]);
        }
        alive = true;
      }
      if (!alive) break;
      commit(&bars.tile_free);
      ++items;
      if ((it.flags & kLastOfQ)) {
        if (do_ds) commit(&bars.dq_done);
        ++runs;
      }
    }
   } else if (warp == 17) {
    // ------------------------------------------------------------------ loader
    const bool leader = elect_one();
    if (leader) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmDO);
      tma_prefetch_desc(&tmK1);
      tma_prefetch_desc(&tmSV1);
    }
    int bh = -1, ea = 0, eb = 0, er = 0, f = 0;
    uint32_t items = 0, vb = 0;
    bool alive = true, in_flight = false;
    BwdWalk<DIAG> walk(p, D == 64 && p.diag_asked ? smem + Cfg::kOffHeads : nullptr);
    BwdItem it{-1, -1, 0, 0, 0, 0, 0, 0, 0, {0, 0, 0}};
    while (alive) {
      it = walk.next(it);
      if (it.len > 0 && it.bh != bh) {
        bh = it.bh;
        const BwdStats st = head_stats(p, bh, lane);
        ea = range_shift<T16>(st.k1, st.k2, alpha_shift(p.alpha));
        eb = range_shift<T16>(st.sv1, st.v2, 0);
        er = product_shift<T16>(fabsf(p.alpha * kLog2e) * sqrtf(st.q_row) * st.k2);
        f = ds_shift<T16>(sqrtf(st.do_row * st.sv1_row) * st.v2);
      }
      it.er = er;
      it.ea = ea;
      it.eb = eb;
      it.flags |= f << kShiftBits;
      alive = wait_all(&bars.tile_free, (items & 1) ^ 1);
      if (!alive) break;
      if (leader) bars.items[items % kItemSlots] = it;
      if (it.len == 0) {
        if (leader) mbar_arrive(&bars.tile_full);
        break;
      }
      if (leader) {
        mbar_arrive_expect_tx(&bars.tile_full, ((it.flags & kFirstOfQ) ? 2 * Cfg::kTileQ : 0) +
                                                   (DIAG ? 2 * (128 + g.kkl + g.kkr) * D * 2 : 2 * Cfg::kTileJ));
#pragma unroll
        for (int b = 0; b < D / 64; ++b) {
          if ((it.flags & kFirstOfQ)) {
            tma_load_3d(smem + Cfg::kOffQ + b * 16384, &tmQ, &bars.tile_full, b * 64, it.qt * 128, it.bh);
            tma_load_3d(smem + Cfg::kOffDO + b * 16384, &tmDO, &bars.tile_full, b * 64, it.qt * 128, it.bh);
          }
          if constexpr (DIAG) {   // (maps of K2 and V2)
            tma_load_3d(smem + Cfg::kOffK1, &tmK1, &bars.tile_full, 0, it.jt * JT - g.kkr, it.bh);
            tma_load_3d(smem + Cfg::kOffK1 + Cfg::kWindow, &tmSV1, &bars.tile_full, 0, it.jt * JT - g.kkr, it.bh);
            continue;
          }
          tma_load_3d(smem + Cfg::kOffK1 + b * JT * 128, &tmK1, &bars.tile_full, b * 64, g.j_row(it.jt), it.bh);
          tma_load_3d(smem + Cfg::kOffK1 + Cfg::kTileJ + b * JT * 128, &tmSV1, &bars.tile_full, b * 64, g.j_row(it.jt), it.bh);
        }
      }
      in_flight = true;
      ++items;
      if (DIAG) continue;
      // K2 / V2 rows, a batch at a time (the last one of an item may be shorter)
      const size_t head = ((size_t)it.bh * T + it.k0) * D;
      for (int i = 0; i < it.len; i += kVecBatch, ++vb) {
        const uint32_t slot = vb % kVecSlots, bytes = min(kVecBatch, it.len - i) * D * 2;
        alive = wait_all(&bars.vec_empty[slot], ((vb / kVecSlots) & 1) ^ 1);
        if (!alive) break;
        if (leader) {
          uint8_t* dst = smem + Cfg::kOffVec + slot * 2 * Cfg::kVecPart;
          const size_t src = head + (size_t)i * D;
          mbar_arrive_expect_tx(&bars.vec_full[slot], 2 * bytes);
          bulk_load(dst, (const T16*)p.k2 + src, bytes, &bars.vec_full[slot]);
          bulk_load(dst + Cfg::kVecPart, (const T16*)p.v2 + src, bytes, &bars.vec_full[slot]);
        }
      }
    }
    if (!alive && in_flight) {
      // give copies still in flight a bounded chance to land before the CTA retires
      const long long t0 = clock64();
      while (!mbar_try_wait(&bars.tile_full, (items - 1) & 1) && clock64() - t0 < kWaitTicks / 8) {
      }
      for (uint32_t b = vb > (uint32_t)kVecSlots ? vb - kVecSlots : 0; b < vb; ++b)
        while (!mbar_try_wait(&bars.vec_full[b % kVecSlots], (b / kVecSlots) & 1) && clock64() - t0 < kWaitTicks / 8) {
        }
    }
   } else if constexpr (LARGE) {
    // ------------------------------------------------------------------ R (warps 18, 19)
    // One step ahead of S, from the Q tile and the step's K2 row, rounded as the forward rounds it.  The first block's buffer
    // is the SiLU(V1) tile, which nothing reads any more once the fold warps have it in registers.  A thread takes one
    // 16-byte column of every kRowStep-th row.
    constexpr int kCols = D / 8, kRowStep = 64 / kCols;
    const int t = tid - 18 * 32, col = t % kCols, row0 = t / kCols;
    const uint8_t* const src = smem + Cfg::kOffQ + (col >> 3) * 16384;
    uint8_t* const dst = smem + (col >> 3 ? Cfg::kOffR1 : Cfg::kOffR0);
    const T16* const vec = reinterpret_cast<const T16*>(smem + Cfg::kOffVec) + col * 8;
    // byte offset of piece e of group g: the swizzle of a row depends on its last three bits, that is on e alone (a group is 8 rows)
    constexpr int kPieces = 8 / kRowStep, kGroups = 128 / 8;
    uint32_t swz[kPieces];
#pragma unroll
    for (int e = 0; e < kPieces; ++e) swz[e] = swz128(row0 + e * kRowStep, col & 7);
    auto at = [&](int g, int e) -> uint32_t { return swz[e] + g * kPieces * kRowStep * 128; };
    uint4 next[kPieces];
    auto fetch = [&](int g) {
#pragma unroll
      for (int e = 0; e < kPieces; ++e) next[e] = *reinterpret_cast<const uint4*>(src + at(g, e));
    };
    uint32_t n = 0, items = 0, vb0 = 0;
    bool alive = true;
    BwdItem it;
    while (alive && next_item(items, it, alive)) {
      ++items;
      fetch(0);
      // (the fold warps have read their tile: they have formed the item's first A')
      alive = wait_all(&bars.ap_ready[0], n & 1);
      for (int i = 0; i < it.len && alive; ++i) {
        if ((i & (kVecBatch - 1)) == 0) {
          const uint32_t vb = vb0 + i / kVecBatch;
          alive = wait_all(&bars.vec_full[vb % kVecSlots], (vb / kVecSlots) & 1);
        }
        // the previous step's S has read the buffer (a second buffer would need a barrier of its own: two S may then have run
        // before this wait, and a barrier two phases ahead of its waiter reads as not ready for ever)
        if (alive && i > 0) alive = wait_all(&bars.s_ready, (n + i - 1) & 1);
        if (!alive) break;
        const uint4 v = *reinterpret_cast<const uint4*>(
            vec + ((vb0 + i / kVecBatch) % kVecSlots * 2 * kVecBatch + i % kVecBatch) * D);
        const float sr = p.alpha * kLog2e * pow2i<T16>(it.er);
        const float2 sr2 = make_float2(sr, sr);
        const float2 m[4] = {__fmul2_rn(unpack2<T16>(v.x), sr2), __fmul2_rn(unpack2<T16>(v.y), sr2),
                             __fmul2_rn(unpack2<T16>(v.z), sr2), __fmul2_rn(unpack2<T16>(v.w), sr2)};
        // (the Q pieces of a group are fetched while the one before is worked on; those of the first, below, from the
        // step before: they do not depend on the step)
#pragma unroll 2
        for (int g = 0; g < kGroups; ++g) {
          uint4 x[kPieces];
#pragma unroll
          for (int e = 0; e < kPieces; ++e) x[e] = next[e];
          fetch((g + 1) % kGroups);
#pragma unroll
          for (int e = 0; e < kPieces; ++e) {
            uint32_t wx[4] = {x[e].x, x[e].y, x[e].z, x[e].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float2 f = __fmul2_rn(unpack2<T16>(wx[c]), m[c]);
              wx[c] = pack2<T16>(f.x, f.y);
            }
            *reinterpret_cast<uint4*>(dst + at(g, e)) = make_uint4(wx[0], wx[1], wx[2], wx[3]);
          }
        }
        fence_async_smem();
        arrive_warp(&bars.r_ready);
      }
      n += it.len;
      vb0 += (it.len + kVecBatch - 1) / kVecBatch;
    }
   }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 16) tmem_dealloc(tmem, 512);
  // what comes after this kernel also reads what the exact first queries, which may still be running, add to the sums
  if (tid == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid == 0 && bars.abort_flag && p.status) atomicOr(p.status, 4);
}

// A CTA that has nothing to do.  As at the body's end the kernel must not end before the one ahead of it, which may be running; one
// block's wait is enough, and the others make room for what comes next (with a wait of all, a kernel over k began when the exact first
// queries had ended: 997 us for 983 at 16 heads of T=2048, windows 128/128/0/0, large scores).
__device__ __forceinline__ void end_without_work() {
  if (blockIdx.x == 0 && threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int D, typename T16>
__global__ void __launch_bounds__(kBwdThreads, 1)
tdp_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
               const __grid_constant__ CUtensorMap tmK1, const __grid_constant__ CUtensorMap tmSV1,
               const __grid_constant__ BwdParams p) {
  const PartHeads heads = part_heads<D, false>(p);
  if (p.diag_asked && !heads.others) {
    end_without_work();
    return;
  }
  if (heads.large) tdp_bwd_body<D, T16, true>(tmQ, tmDO, tmK1, tmSV1, p);
  else tdp_bwd_body<D, T16, false>(tmQ, tmDO, tmK1, tmSV1, p);
}

template <typename T16>
__global__ void __launch_bounds__(kBwdThreads, 1)
tdp_bwd_diag_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                    const __grid_constant__ CUtensorMap tmK2, const __grid_constant__ CUtensorMap tmV2,
                    const __grid_constant__ BwdParams p) {
  asm volatile("griddepcontrol.launch_dependents;");   // (tdp_bwd_kernel, which needs nothing of this one)
  if (part_heads<64, true>(p).diag) tdp_bwd_body<64, T16, false, true>(tmQ, tmDO, tmK2, tmV2, p);
  else end_without_work();
}

// What the kernel needs before it starts, in one pass over the tensors (8 elements per thread and step): zeroed fp32
// sums, SiLU(V1) in the inputs' type, Dq = sum_h dO O per query and, when `stats` is not null, per head the largest
// elements and row norms behind the range shifts and the score bound (BwdStats, kStatFloats floats per head and part) of
// the part's share of the head.  A head has up to kStatParts parts (blocks), which the kernel's loader warp reads one per lane: no
// atomics, and nothing to zero before.
constexpr int kPrepThreads = 256;
template <typename T16>
__global__ void __launch_bounds__(kPrepThreads)
tdp_bwd_prepare_kernel(const T16* __restrict__ v1, const T16* __restrict__ o, const T16* __restrict__ d_o,
                       const T16* __restrict__ q, const T16* __restrict__ k1, const T16* __restrict__ k2,
                       const T16* __restrict__ v2, float* __restrict__ sums, T16* __restrict__ sv1, float* __restrict__ drow, float* __restrict__ stats,
                       size_t n, int head_elems, int D, int parts) {
  __shared__ float wmax[kPrepThreads / 32][kStatFloats];
  const int bh = blockIdx.x / parts, part = blockIdx.x % parts, lanes = D / 8;   // 8 or 16 lanes hold one row
  const uint32_t row_lanes = ((1u << lanes) - 1u) << ((threadIdx.x & 31) / lanes * lanes);
  float k1_max = 0.f, k2_max = 0.f, sv1_max = 0.f, v2_max = 0.f, k1_row = 0.f, q_row = 0.f, do_row = 0.f, sv1_row = 0.f;
  auto words = [](const T16* p, uint32_t (&w)[4]) {
    const uint4 x = *reinterpret_cast<const uint4*>(p);
    w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
  };
  uint32_t bad = 0;   // (see not_finite)
  auto look = [&](const uint32_t (&w)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) bad |= not_finite<T16>(w[e]);
  };
  auto grow = [](float& a, float2 x) { a = fmaxf(a, fmaxf(fabsf(x.x), fabsf(x.y))); };
  // (the lanes of a row are all here or all gone: head_elems is a multiple of D)
  for (int at = (part * kPrepThreads + threadIdx.x) * 8; at < head_elems; at += parts * kPrepThreads * 8) {
    const size_t i = (size_t)bh * head_elems + at;
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      *reinterpret_cast<float4*>(sums + s * n + i) = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(sums + s * n + i + 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    uint32_t wv[4], wa[4], wb[4], r[4];
    words(v1 + i, wv);
    words(o + i, wa);
    words(d_o + i, wb);
    float dot = 0.f, nd = 0.f, ns = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack2<T16>(wv[e]), x = unpack2<T16>(wa[e]), y = unpack2<T16>(wb[e]);
      const float2 g = make_float2(silu_f(f.x), silu_f(f.y));
      r[e] = pack2<T16>(g.x, g.y);
      dot = fmaf(x.x, y.x, fmaf(x.y, y.y, dot));
      const float2 g16 = unpack2<T16>(r[e]);
      grow(sv1_max, g16);
      ns = fmaf(g16.x, g16.x, fmaf(g16.y, g16.y, ns));
      nd = fmaf(y.x, y.x, fmaf(y.y, y.y, nd));
    }
    *reinterpret_cast<uint4*>(sv1 + i) = make_uint4(r[0], r[1], r[2], r[3]);
    for (int s = lanes / 2; s >= 1; s >>= 1) dot += __shfl_xor_sync(row_lanes, dot, s);
    if ((threadIdx.x & (lanes - 1)) == 0) drow[i / D] = dot;
    if (stats) {
      look(wv);
      look(wb);
      words(k1 + i, wv);
      words(k2 + i, wa);
      words(v2 + i, wb);
      look(wv);
      look(wa);
      look(wb);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        grow(k1_max, unpack2<T16>(wv[e]));
        grow(k2_max, unpack2<T16>(wa[e]));
        grow(v2_max, unpack2<T16>(wb[e]));
      }
      words(q + i, wa);
      look(wa);
      float n1 = 0.f, nq = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = unpack2<T16>(wv[e]), y = unpack2<T16>(wa[e]);
        n1 = fmaf(x.x, x.x, fmaf(x.y, x.y, n1));
        nq = fmaf(y.x, y.x, fmaf(y.y, y.y, nq));
      }
      for (int s = lanes / 2; s >= 1; s >>= 1) {
        n1 += __shfl_xor_sync(row_lanes, n1, s);
        nq += __shfl_xor_sync(row_lanes, nq, s);
        nd += __shfl_xor_sync(row_lanes, nd, s);
        ns += __shfl_xor_sync(row_lanes, ns, s);
      }
      do_row = fmaxf(do_row, nd);
      sv1_row = fmaxf(sv1_row, ns);
      k1_row = fmaxf(k1_row, n1);
      q_row = fmaxf(q_row, nq);
    }
  }
  if (!stats) return;
  float w[kStatFloats] = {k1_max, k2_max, sv1_max, v2_max, k1_row, q_row, do_row, sv1_row};
#pragma unroll
  for (int o2 = 16; o2 >= 1; o2 >>= 1)
#pragma unroll
    for (int i = 0; i < kStatFloats; ++i) w[i] = fmaxf(w[i], __shfl_xor_sync(0xffffffffu, w[i], o2));
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int i = 0; i < kStatFloats; ++i) wmax[threadIdx.x >> 5][i] = w[i];
  }
  const bool any_bad = __syncthreads_or(bad & 0x80008000u);
  if (threadIdx.x < kStatFloats) {
    float x = 0.f;
#pragma unroll
    for (int i = 0; i < kPrepThreads / 32; ++i) x = fmaxf(x, wmax[i][threadIdx.x]);
    if (threadIdx.x == 5 && any_bad) x = -x;   // q_row's sign: not all elements are finite
    stats[(size_t)blockIdx.x * kStatFloats + threadIdx.x] = x;
  }
}

// The fp32 sums -> gradients in the inputs' type, SiLU'(V1) applied to dV1 (reference flash_trittention.py:390-391), 8
// elements per thread.  dq_only: just the query rows q_rem + i * q_mod of dQ (a query-sharded call).
template <typename T16>
__global__ void tdp_bwd_finish_kernel(const float* __restrict__ sums, const T16* __restrict__ v1, T16* __restrict__ dq,
                                      T16* __restrict__ dk1, T16* __restrict__ dk2, T16* __restrict__ dv1,
                                      T16* __restrict__ dv2, size_t n, int T, int D, int q_mod, int q_rem, bool dq_only) {
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  auto put = [&](const float* src, T16* dst, const float (*mul)) {
    const float4 a = *reinterpret_cast<const float4*>(src + i), b = *reinterpret_cast<const float4*>(src + i + 4);
    float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    if (mul) {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= mul[e];
    }
    *reinterpret_cast<uint4*>(dst + i) =
        make_uint4(pack2<T16>(f[0], f[1]), pack2<T16>(f[2], f[3]), pack2<T16>(f[4], f[5]), pack2<T16>(f[6], f[7]));
  };
  if ((int)((i / D) % T) % q_mod == q_rem) put(sums + 4 * n, dq, nullptr);
  if (dq_only) return;
  put(sums, dk1, nullptr);
  put(sums + n, dk2, nullptr);
  const uint4 v = *reinterpret_cast<const uint4*>(v1 + i);
  const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
  float g[8];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = unpack2<T16>(wv[e]);
    g[2 * e] = silu_grad_f(f.x);
    g[2 * e + 1] = silu_grad_f(f.y);
  }
  put(sums + 2 * n, dv1, g);
  put(sums + 3 * n, dv2, nullptr);
}

// The register split of the kernel's warpgroups assumes the count it was launched with: setmaxnreg.inc waits without a limit
// for registers that the block does not have, and .dec / .inc in the wrong direction is an illegal instruction.  A build
// that gives the kernel another count is refused instead of being launched.
int check_registers(int launched) {
  if (launched == kRegsLaunch) return 0;
  set_error("the backward kernel was built with %d registers per thread, its split needs %d", launched, kRegsLaunch);
  return -30;
}

template <auto kKernel>
int check_kernel_registers() {
  static std::atomic<int> launched{0};   // (per kernel: a property of the compiled code, the same on every device)
  int n = launched.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaFuncAttributes attr;
    TRITT_CUDA_OK(cudaFuncGetAttributes(&attr, kKernel));
    n = attr.numRegs;
    launched.store(n, std::memory_order_relaxed);
  }
  return check_registers(n);
}

// The first queries of a causal call run in exact fp32 on the CUDA cores.  Their gradients are the largest by far (a query
// attends ~q^2 pairs: its dQ falls like 1/q, and so does what it adds to the first key rows), so their rounding is most of
// the error of the whole result; and in fp16 the first query of a tile sets the tile's range shift (prob_shift).  They are
// a vanishing part of the work on long sequences: a training step's error against fp64 goes from 3.6e-3 to 2.6e-3 at T=2048
// in bf16 with 32 of them.  Short ones take 16: the error is 2 to 10 % higher than with 32, at an eighth of the pairs and
// atomics (160 heads of T=70: 237 against 305 us a call, 204 without any; 4 heads of T=333 D=128: 195, 201, 179).
// (Queries 0 to 31 themselves, not the first 32 rows of a shard: 8 interleaved shards have queries up to 248 among those, with
// 60 times the pairs, and at 64 shards and T=2048 they are the whole shard.)
// Narrow windows leave every query few pairs, W at most, and the first ones are then no larger than the others: their share
// of a gradient's squared norm is about 1.6 (the sum of 1/q^2) against the T / W of the rest.  From T = 8 W on they take no
// path of their own, which costs a call of so little work more than it gives (us per call with / without, 4 heads
// T=2047 D=128 windows 3/2/1/2: fp16 169 / 158, bf16 167 / 156, large scores 186 / 174; the errors are the same to 1 %).

// What a call does, from its arguments alone.
struct BwdPlan {
  BwdGeometry g;
  int i_first;        // query rows (of the shard) that the CUDA cores take, in exact fp32
  long head_steps;    // steps of the kernel per head
  BwdGeometry diag;   // the steps of the kernel that steps over diagonals, if diag_steps > 0
  long diag_steps;
  bool by_queries;    // the kernel that steps over queries instead: every row is its, as items of its own
  long long cells;    // cells (q, j, k) executed per head
};

// A tile's 128 rows of a shard lie q_mod apart, and each of its steps is executed for all of them: at 8 shards the rows of
// a tile span 1024 queries, and one shard of T=1024 executes 0.31 of the whole call's cells instead of 0.125, of T=2048
// 0.21, of T=4096 0.17, of windows 128/128/32/32 0.63.  The kernel that steps over queries executes just a shard's share, at
// a higher price per cell: stepping over k costs 0.66 to 0.77 of it per cell (D=128 0.71; more for large scores).
// ms per call of one of 8 shards, k / queries: T=1024 D=64 16 heads 1.85 / 1.12, T=2048 D=128 16 heads 13.1 / 11.0, T=4096
// D=64 4 heads 13.7 / 13.3, those windows 0.79 / 0.55; of one of 2: 3.38 / 4.34, 35.2 / 45.4, 41.3 / 52.9, 0.97 / 2.09.
constexpr double kCellPrice = 0.8;

// What an item costs beside its steps (its tiles' way in, dK1's and dSiLU(V1)'s out), in steps; and the narrowest stride taken.
// us per backward with tiles side by side / overlapping: 16 heads T=2048 D=64 fp16 windows 128/128/32/32 (stride 64) 1141 / 955,
// 256/256/40/20 (68) 1719 / 1379, 8/8/4/4 (120) 560 / 534; 8 heads T=2000 200/100/48/48 (32) 631 / 482; D=128 16 heads T=2048
// 128/128/16/16 (32 of 64) 1004 / 802.
constexpr long kItemSteps = 3;
constexpr int kMinStride = 8;

// Diagonals are taken where they are fewer by more than a step's higher price and a launch.  Steps and items of a CTA, k / diagonals: us
// with k / diagonals, D=64:  140 / 123: 325 / 350, 74 / 62: 192 / 195, 30 / 25: 98 / 104, 1.4 / 0.3: 75 / 76, 15 / 9: 75 / 77,
// 24 / 9: 87 / 79, 41 / 26: 124 / 110, 31 / 3: 104 / 76, 45 / 9: 135 / 80, 54 / 28: 146 / 114, 449 / 228: 951 / 615, 871 / 548: 1818 / 1400.
// Calls with large scores pay for a kernel that does nothing, without / with it: 16 heads T=2048 windows 128/128/0/0 978 / 983, T=512 band 0/0
// 332 / 334, 8 heads T=633 windows 19/9/2/3 118 / 120.
constexpr double kDiagPrice = 1.3, kDiagGain = 6;

// Steps and items of one head.
long count_steps(const BwdGeometry& g, long& items) {
  long steps = 0;
  items = 0;
  for (int qt = 0; qt < g.q_tiles(); ++qt)
    for (int jt = g.j_first(qt); jt <= g.j_last(qt); ++jt) {
      int k0;
      const int n = g.k_range(qt, jt, k0);
      steps += n;
      items += n > 0;
    }
  return steps;
}

template <int D> BwdPlan make_plan(const TdpArgs& a) {
  BwdPlan p{};
  const int nq = a.q_rem < a.T ? (a.T - a.q_rem + a.q_mod - 1) / a.q_mod : 0;
  constexpr int JT = BwdCfg<D>::JT;
  p.g = BwdGeometry{a.T, nq, a.q_mod, a.q_rem, a.mask.causal, a.mask.k1w, a.mask.k2w, a.mask.kkl, a.mask.kkr, JT, JT, 0, false};
  if (nq == 0) return p;
  const int first = tdp_bwd_first_count(a.T);
  const long long pairs = (min(a.mask.k1w, a.T - 1) + 1LL) * (min(a.mask.k2w, a.T - 1) + 1LL);   // (at most, of any query)
  if (a.mask.causal && a.q_rem < first && pairs * 8 > a.T) {
    p.i_first = (first - a.q_rem + a.q_mod - 1) / a.q_mod;
    if (p.i_first >= nq) {   // nothing left for the kernel
      p.i_first = nq;
      return p;
    }
  }
  long items;
  p.head_steps = count_steps(p.g, items);
  const int stride = JT - a.mask.kkl - a.mask.kkr;
  if (a.mask.causal && stride >= kMinStride) {
    BwdGeometry o = p.g;
    o.stride = stride;
    o.lead = a.mask.kkl;
    long o_items;
    const long o_steps = count_steps(o, o_items);
    if (o_steps + kItemSteps * o_items < p.head_steps + kItemSteps * items) {
      p.g = o;
      p.head_steps = o_steps;
    }
  }
  if (D == 64 && a.mask.causal && a.q_mod == 1 && 128 + a.mask.kkl + a.mask.kkr <= kDiagRows) {
    p.diag = p.g;
    p.diag.stride = JT;
    p.diag.lead = 0;
    p.diag.diagonals = true;
    long d_items, k_items;
    const long d_steps = count_steps(p.diag, d_items);
    count_steps(p.g, k_items);
    const double less = (double)(p.head_steps + kItemSteps * k_items) - kDiagPrice * (double)(d_steps + kItemSteps * d_items);
    if (less * a.B * a.N >= kDiagGain * num_sms()) p.diag_steps = d_steps;
  }
  p.cells = (long long)p.head_steps * 128 * BwdCfg<D>::JT;
  if (a.q_mod > 1) {
    const long long cells = sm100_tdp_bwd_queries_cells(a.T, a.mask, a.q_mod, a.q_rem);
    if (kCellPrice * (double)p.cells > (double)cells) {
      p.by_queries = true;
      p.i_first = 0;
      p.cells = cells;
    }
  }
  return p;
}

// workspace: fp32 sums dK1 | dK2 | dSiLU(V1) | dV2 | dQ, SiLU(V1) in the inputs' type, Dq fp32; and, where the caller's has
// it, the statistics (without them fp16 products are formed without regard to their size)
template <int D, typename T16>
int launch_bwd_sums(const TdpArgs& a, const BwdPlan& plan) {
  using Cfg = BwdCfg<D>;
  const int BN = a.B * a.N;
  const size_t n = (size_t)BN * a.T * a.D;
  float* sums = (float*)a.workspace;
  T16* sv1 = (T16*)(sums + 5 * n);
  float* drow = (float*)(sv1 + n);
  const size_t tail = align_up(sm100_tdp_bwd_workspace(a.B, a.N, a.T, D), 16);
  const bool has_tail = a.workspace_bytes >= tail + (size_t)BN * kStatParts * kStatFloats * sizeof(float);
  float* stats = has_tail ? (float*)((char*)a.workspace + tail) : nullptr;
  const int head_elems = a.T * D, passes = (head_elems + kPrepThreads * 8 - 1) / (kPrepThreads * 8);
  const int parts = passes < kStatParts ? passes : kStatParts;
  tdp_bwd_prepare_kernel<T16><<<(unsigned)(BN * parts), kPrepThreads, 0, a.stream>>>(
      (const T16*)a.v1, (const T16*)a.o, (const T16*)a.d_o, (const T16*)a.q, (const T16*)a.k1, (const T16*)a.k2, (const T16*)a.v2,
      sums, sv1, drow, stats, n, head_elems, D, parts);
  count_launch();
  TRITT_CUDA_OK(cudaGetLastError());
  BwdParams p{};
  p.stats = stats;
  p.stat_parts = parts;
  p.q = a.q; p.d_o = a.d_o; p.k2 = a.k2; p.v2 = a.v2; p.k1 = a.k1; p.sv1 = sv1; p.lse = a.lse_in; p.drow = drow;
  p.dk1 = sums; p.dk2 = sums + n; p.dsv1 = sums + 2 * n; p.dv2 = sums + 3 * n; p.dq = sums + 4 * n;
  p.BN = BN;
  p.alpha = a.alpha;
  const int nq = plan.g.nq;
  if (nq == 0) return 0;
  p.i_first = plan.i_first;
  p.g = plan.g;
  p.head_steps = plan.head_steps;
  p.status = a.status_word;
  if (plan.i_first > 0) {
    const int rc = tdp_bwd_first_queries(a, plan.i_first, sums, drow);
    if (rc) return rc;
  }
  if (p.head_steps == 0) return 0;
  CUtensorMap tmQ, tmDO, tmK1, tmSV1, tmK2, tmV2;
  int rc;
  const size_t shard = (size_t)a.q_rem * D;   // first query row of the shard
  if ((rc = make_tmap_rows(&tmQ, (const T16*)a.q + shard, D, nq, BN, (uint64_t)a.q_mod * D, (uint64_t)a.T * D, 128))) return rc;
  if ((rc = make_tmap_rows(&tmDO, (const T16*)a.d_o + shard, D, nq, BN, (uint64_t)a.q_mod * D, (uint64_t)a.T * D, 128))) return rc;
  if ((rc = make_tmap_3d(&tmK1, a.k1, 2, D, a.T, BN, 64, Cfg::JT))) return rc;
  if ((rc = make_tmap_3d(&tmSV1, sv1, 2, D, a.T, BN, 64, Cfg::JT))) return rc;
  // With exact first queries ahead of it the kernel starts as soon as all their blocks have: it needs the preparation pass,
  // which was done before they began, and nothing of theirs (both add to the sums).  us per backward
  // with this / one after the other: T=333 D=128 4 heads 192 / 198, T=128 D=64 64 heads 171 / 181, T=60 D=64 2 heads 29 / 35.
  auto launch = [&](auto kern, int smem_bytes, long steps, bool early, const CUtensorMap& m2, const CUtensorMap& m3) -> int {
    TRITT_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    const long total = steps * BN, sms = num_sms();   // (equal parts of the whole line of steps)
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(total < sms ? total : sms), 1, 1);
    cfg.blockDim = dim3(kBwdThreads, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = a.stream;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    TRITT_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tmQ, tmDO, m2, m3, p));
    count_launch();
    return 0;
  };
  bool early = plan.i_first > 0;
  if constexpr (D == 64) {
    const long least = plan.diag_steps < plan.head_steps ? plan.diag_steps : plan.head_steps, sms = num_sms();
    if (plan.diag_steps > 0 && stats && BN / (least * BN < sms ? least * BN : sms) + 2 <= kPartHeads) {
      const uint32_t rows = 128 + a.mask.kkl + a.mask.kkr;
      if ((rc = make_tmap_3d(&tmK2, a.k2, 2, D, a.T, BN, 64, rows))) return rc;
      if ((rc = make_tmap_3d(&tmV2, a.v2, 2, D, a.T, BN, 64, rows))) return rc;
      if ((rc = check_kernel_registers<tdp_bwd_diag_kernel<T16>>())) return rc;
      p.diag_asked = true;
      p.g = plan.diag;
      p.head_steps = plan.diag_steps;
      if ((rc = launch(tdp_bwd_diag_kernel<T16>, BwdCfg<D, true>::kSmem, plan.diag_steps, early, tmK2, tmV2))) return rc;
      p.g = plan.g;
      p.head_steps = plan.head_steps;
      early = true;
    }
  }
  if ((rc = check_kernel_registers<tdp_bwd_kernel<D, T16>>())) return rc;
  return launch(tdp_bwd_kernel<D, T16>, Cfg::kSmem, plan.head_steps, early, tmK1, tmSV1);
}

template <typename T16>
int launch_finish(const TdpArgs& a) {
  const size_t n = (size_t)a.B * a.N * a.T * a.D;
  tdp_bwd_finish_kernel<T16><<<(unsigned)((n / 8 + 255) / 256), 256, 0, a.stream>>>(
      (const float*)a.workspace, (const T16*)a.v1, (T16*)a.dq, (T16*)a.dk1, (T16*)a.dk2, (T16*)a.dv1, (T16*)a.dv2, n, a.T,
      a.D, a.q_mod, a.q_rem, (a.flags & TRITT_FLAG_BWD_PARTIAL) != 0);
  count_launch();
  TRITT_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace

size_t sm100_tdp_bwd_workspace(int B, int N, int T, int D) {
  const size_t r = (size_t)B * N * T, n = r * D;
  return 5 * n * sizeof(float) + n * 2 + r * sizeof(float);
}

size_t sm100_tdp_bwd_optional_workspace(int B, int N) { return align_up((size_t)B * N * kStatParts * kStatFloats * sizeof(float) + 16, 256); }

static BwdPlan plan_of(const TdpArgs& a) { return a.D == 128 ? make_plan<128>(a) : make_plan<64>(a); }

static int launch_sums(const TdpArgs& a, const BwdPlan& plan) {
  if (a.dtype == TRITT_BF16)
    return a.D == 128 ? launch_bwd_sums<128, __nv_bfloat16>(a, plan) : launch_bwd_sums<64, __nv_bfloat16>(a, plan);
  return a.D == 128 ? launch_bwd_sums<128, __half>(a, plan) : launch_bwd_sums<64, __half>(a, plan);
}

// (not sharded: the wide path is the only caller)
int sm100_tdp_bwd_sums(const TdpArgs& a) { return launch_sums(a, plan_of(a)); }

void sm100_tdp_bwd_plan(const TdpArgs& a, long long* out) {
  const BwdPlan p = plan_of(a);
  out[0] = p.i_first;
  out[1] = p.cells;
  out[2] = p.by_queries;
}

int sm100_tdp_bwd_check_registers(int launched) { return check_registers(launched); }

int sm100_tdp_bwd(const TdpArgs& a) {
  const BwdPlan plan = plan_of(a);
  if (plan.by_queries) return sm100_tdp_bwd_queries(a);   // (a shard: its key-side sums stay sums)
  const int rc = launch_sums(a, plan);
  if (rc) return rc;
  return a.dtype == TRITT_BF16 ? launch_finish<__nv_bfloat16>(a) : launch_finish<__half>(a);
}

}  // namespace tritt
