// Triple-dot-product trittention forward for narrow (j, k) bands: stepping over the band's diagonals.
//
// For one diagonal d = k - j the score and the gated value are those of an ordinary attention whose key and value rows are
//     A [j,h] = K1[j,h] * K2[j+d,h]        W [j,h] = SiLU(V1)[j,h] * V2[j+d,h]
//     S  = alpha*log2(e) * Q A^T            O += exp2(S - m) W,
// so a tile of 128 queries walks over "keys" (j, d) as flash attention walks over j.  Of a tile of 128 rows j all 128 columns of a
// step lie in the band, and with windows up to 128 a j-tile meets two query tiles, its own and the next: half of those two squares
// is attended.  (Tiles of 4 queries x 32 K2 rows against a slab of 128 columns, tdp_fwd_band_kernel, fill a third of the slab and
// pay for an operand, a fold and two reads of the accumulator per slab.)
//
// It serves calls whose scores are small and whose elements are finite: a bound on every score of a head is the soft-max reference of the
// head's rows.  Other calls are left to tdp_fwd_band_kernel, behind this one, whose operand alpha Q K2 is also what the backward forms for
// large scores; they pay 1 to 3 us for a kernel that ends at once.
//
// A CTA has two slots, each with an accumulator, two soft-max warpgroups (a query per thread, every other 32 of its columns) and every
// other query tile: a step is one d of one j-tile for both.  All steps of a call form one line (heads, j-tiles, d) that is cut in
// equal parts, one per CTA; a query tile whose steps are cut leaves its accumulators in the workspace, which the warp that brings the last
// piece adds up, or in short calls (kMergingBandTiles) the band kernel behind this one.
//
// What bounds it: no single unit.  A step takes 2700 cycles for both slots (160 of 180 us at T=2048; the rest are the preparation, 8, the
// launch, the first loads of items and the pieces); issue slots are 59 % busy, the exponentials' unit 47 %, tensor cores 38 %, and a slot's
// chain (scores, exponentials, P, value product) is not hidden behind the other slot's alone.  One soft-max warpgroup per slot walking all
// 128 columns took 3200 cycles.  Device time of a forward, us, the kernel of 4 queries x 32 rows -> this one: 16 heads T=2048 fp16 windows
// 128/128/32/32 466 -> 180, T=8192 1933 -> 654, T=2048 windows 8/8/4/4 120 -> 43, 8 heads T=1000 117 -> 60, 16 heads T=500 128/128/48/48
// 119 -> 75; fp32 tensors, 8 heads T=2048 254 -> 111.
// Slower: masks of boundary columns by clamped FMAs (194 us for 189), a quarter of the exponentials as polynomials (194), value products
// that start with the first warpgroup's half of P (190).
//
// 28 warps: 0-7 and 8-15: soft-max warpgroups of the slots; 16-23: form A and W, from K1 and SiLU(V1) rows in registers and K2 / V2
// rows in shared memory; 24 and 26 issue the score and the value products; 25: the line of work and all loads.  Three buffers of
// scores are taken in turn, P of 32 columns lies over the first half of their scores: a slot's next scores wait for the other slot's
// last value product, not for its own.
#include "tritt_sm100_tdp_diag.cuh"

#include <atomic>

namespace tritt {
namespace {
using namespace sm100;

constexpr int kDiagThreads = 896;
// Registers per thread: 896 threads are launched with 72 each, and split them anew (set_regs).
constexpr int kDiagRegs = 72, kRegsSoftmax = 72, kRegsFormer = 80, kRegsService = 56;
static_assert(4 * kRegsSoftmax + 2 * kRegsFormer + kRegsService <= 7 * kDiagRegs, "more registers than the launch has");
constexpr int kMaxBand = 96;        // kk_left + kk_right
constexpr int kTile = 128 * kDiagD * 2; // a tile of 128 rows
constexpr int kNB = 3;              // buffers of A and of W
constexpr int kNQ = 4;              // Q tiles
constexpr int kNS = 3;              // buffers of scores
constexpr int kWindow = (128 + kMaxBand) * kDiagD * 2;   // K2 / V2 rows of an item
constexpr int kOffQ = 0, kOffA = kNQ * kTile, kOffW = kOffA + kNB * kTile, kOffK2 = kOffW + kNB * kTile,
              kOffV2 = kOffK2 + kWindow, kOffL = kOffV2 + kWindow, kOffBars = kOffL + 4096, kSmem = kOffBars + 768;
static_assert(kSmem <= 232448 && kOffK2 % 1024 == 0 && kWindow % 1024 == 0, "shared memory");
constexpr int kTmemO = kNS * 128;   // accumulators
constexpr int kItemSlots = 4;

struct alignas(16) DiagItem {
  int bh, jt, n0, len;          // diagonals n0 .. n0 + len - 1, d = n - kkr;  len 0: no more items
  int flags, qn, ea, eb;        // qn: number of the Q tile jt among this CTA's;  A and W carry factors 2^ea and 2^eb
  float sa, reference;
  int pad[2];
};
enum {
  kNewOwn = 1, kNewNext = 2,    // the accumulator of tile jt / jt + 1 starts with this item
  kEndOwn = 4, kEndNext = 8     // ... and ends with it, as far as this CTA goes
};

struct DiagBarriers {
  DiagItem items[kItemSlots];
  uint64_t item_full[kItemSlots], item_free[kItemSlots];
  uint64_t win_full, win_free;
  uint64_t q_full[kNQ], q_free[kNQ];
  uint64_t a_ready[kNB], a_free[kNB], w_ready[kNB], w_free[kNB];
  // (s_ready doubled by the parity of the steps: a slot's next scores do not wait for it to have looked at these)
  uint64_t s_ready[2][2], p_ready[2], pv_done[2], place_free[kNS], l_ready[2];
  uint32_t tmem_base;
  int abort_flag;
};

template <typename T16>
__global__ void __launch_bounds__(kDiagThreads, 1)
tdp_fwd_diag_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK2,
                    const __grid_constant__ CUtensorMap tmV2, const __grid_constant__ DiagParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  static_assert(sizeof(DiagBarriers) <= 768, "barrier block too large");
  DiagBarriers& bars = *reinterpret_cast<DiagBarriers*>(smem + kOffBars);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (smem_u32(smem) & 1023u) {
    // swizzled tiles need 1024-byte alignment; uniform over the CTA, so every thread leaves here
    if (tid == 0 && p.status) atomicOr(p.status, 8);
    return;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (launched ahead of the preparation's end)
  if (!diag_takes(p)) {
    asm volatile("griddepcontrol.launch_dependents;");   // (the band kernel, which waits for this one's end all the same)
    return;
  }
  if (tid == 0) {
    bars.abort_flag = 0;
    for (int i = 0; i < kItemSlots; ++i) {
      mbar_init(&bars.item_full[i], 1);
      mbar_init(&bars.item_free[i], 26);
    }
    mbar_init(&bars.win_full, 1);
    mbar_init(&bars.win_free, 8);
    for (int i = 0; i < kNQ; ++i) {
      mbar_init(&bars.q_full[i], 1);
      mbar_init(&bars.q_free[i], 1);
    }
    for (int i = 0; i < kNB; ++i) {
      mbar_init(&bars.a_ready[i], 8);
      mbar_init(&bars.a_free[i], 1);
      mbar_init(&bars.w_ready[i], 8);
      mbar_init(&bars.w_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars.s_ready[i][0], 1);
      mbar_init(&bars.s_ready[i][1], 1);
      mbar_init(&bars.p_ready[i], 8);
      mbar_init(&bars.l_ready[i], 8);
      mbar_init(&bars.pv_done[i], 1);
    }
    for (int i = 0; i < kNS; ++i) mbar_init(&bars.place_free[i], 1);
    fence_barrier_init();
  }
  if (warp == 24) {
    tmem_alloc(&bars.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;
  const DiagGeometry& g = p.g;
  const int T = g.T;
  // (every lane waits; the vote keeps the warp converged whatever a lane's wait returned)
  auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
    return __all_sync(0xffffffffu, mbar_wait_looks(bar, parity, abort_flag));
  };
  // one arrival per warp, after the caller's fences
  auto arrive_warp = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  // (every lane has the same value; the reduction tells the compiler so)
  auto uniform = [](int v) -> int { return __reduce_max_sync(0xffffffffu, v); };

  if (warp < 16) {
    set_regs<kDiagRegs, kRegsSoftmax>();
    // ------------------------------------------------------------------ soft-max warpgroups
    const int x = warp >> 3, half = warp >> 2 & 1, wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t tB = tmem + ((uint32_t)(wq * 32) << 16), tO = tB + kTmemO + x * kDiagD + half * (kDiagD / 2);
    uint32_t step = 0;        // steps so far
    uint32_t ends = 0;        // query tiles so far
    float l = 0.f;            // sum of this thread's P
    // (sums of the row's two threads, of this query tile and, doubled, the next)
    float* const row_l = reinterpret_cast<float*>(smem + kOffL) + x * 256 + row;
    for (uint32_t items = 0;; ++items) {
      if (!wait_all(&bars.item_full[items % kItemSlots], (items / kItemSlots) & 1)) break;
      const DiagItem& it = bars.items[items % kItemSlots];
      const int len = uniform(it.len);
      if (len == 0) break;
      const int bh = uniform(it.bh), jt = uniform(it.jt), n0 = uniform(it.n0), flags = uniform(it.flags), eb = uniform(it.eb);
      const float sa = it.sa, reference = it.reference;
      arrive_warp(&bars.item_free[items % kItemSlots]);
      const bool own = (jt & 1) == x;
      const int tile = own ? jt : jt + 1, q = tile * 128 + row, j0 = jt * 128;
      if (flags & (own ? kNewOwn : kNewNext)) l = 0.f;
      const float2 sa2 = make_float2(sa, sa), nref = make_float2(-reference, -reference);
      bool alive = true;
      for (int n = n0; n < n0 + len; ++n, ++step) {
        // the columns j that this query sees on diagonal d: j <= q, q - j <= k1w, 0 <= j + d <= q, q - (j + d) <= k2w
        const int d = n - g.kkr;
        const int lo = max(max(q - g.k1w, q - d - g.k2w), max(0, -d)) - j0;
        const int hi = q < T ? min(q, q - d) - j0 : -1;
        const uint32_t turn = 2 * step + x;
        const uint32_t tS = tB + turn % kNS * 128;
        alive = wait_all(&bars.s_ready[x][step & 1], (step >> 1) & 1);
        if (!alive) break;
        tc_fence_after();
        // (every phase of pv_done is looked at, also where nothing waits for it: a barrier a phase behind its waiter reads as ready)
        const bool seen = mbar_test(&bars.pv_done[x], (step & 1) ^ 1);
        float2 sum = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int c0 = 32 * half; c0 < 128; c0 += 64) {
          uint32_t w[16];
          const uint32_t mask = column_mask(lo - c0, hi - c0);
          if (__any_sync(0xffffffffu, mask != 0u)) {
            // (A read is waited for right where it is issued: its registers are written while it is under way, which the compiler
            // does not know of.)
            uint32_t v[32];
            tmem_ld32(tS + c0, v);
            tmem_wait_ld(v);
            if (__all_sync(0xffffffffu, mask == ~0u)) {
#pragma unroll
              for (int c = 0; c < 32; c += 2) {
                const float2 y = __ffma2_rn(make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), sa2, nref);
                const float2 e = make_float2(exp2f(y.x), exp2f(y.y));
                sum = __fadd2_rn(sum, e);
                w[c >> 1] = pack2<T16>(e.x, e.y);
              }
            } else {
#pragma unroll
              for (int c = 0; c < 32; c += 2) {
                const float2 y = __ffma2_rn(make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), sa2, nref);
                const float2 e = make_float2(mask >> c & 1u ? exp2f(y.x) : 0.f, mask >> (c + 1) & 1u ? exp2f(y.y) : 0.f);
                sum = __fadd2_rn(sum, e);
                w[c >> 1] = pack2<T16>(e.x, e.y);
              }
            }
          } else {
#pragma unroll
            for (int c = 0; c < 16; ++c) w[c] = 0u;
          }
          tmem_st16(tS + c0, w);   // over these columns' scores
        }
        l += sum.x + sum.y;
        tmem_wait_st();
        tc_fence_before();
        alive = __all_sync(0xffffffffu, seen) || wait_all(&bars.pv_done[x], (step & 1) ^ 1);
        if (!alive) break;
        arrive_warp(&bars.p_ready[x]);
      }
      if (!alive) break;
      if (!(flags & (own ? kEndOwn : kEndNext)) || tile >= g.tiles()) continue;
      // ---- the tile's output, or this CTA's piece of it
      row_l[(ends & 1) * 512 + half * 128] = l;
      arrive_warp(&bars.l_ready[x]);
      if (!wait_all(&bars.pv_done[x], (step - 1) & 1)) break;
      tc_fence_after();
      if (!wait_all(&bars.l_ready[x], ends & 1)) break;
      const float row_sum = row_l[(ends & 1) * 512] + row_l[(ends & 1) * 512 + 128];
      ++ends;
      int first, pieces;
      g.ctas(bh, tile, first, pieces);
      const float scale = pow2i<T16>(-eb) / row_sum;
      T16* const dst = (T16*)p.out + ((size_t)bh * T + q) * kDiagD + half * (kDiagD / 2);
      auto area_of = [&](int i) -> float* { return diag_area(p, first, i, tile, half) + row; };
      float* const area = area_of((int)blockIdx.x - first);
#pragma unroll 1
      for (int c0 = 0; c0 < kDiagD / 2; c0 += 16) {
        uint32_t t[16];
        tmem_ld16(tO + c0, t);
        tmem_wait_ld(t);
        if (pieces == 1) {
          if (q < T) {
            uint32_t o[8];
#pragma unroll
            for (int c = 0; c < 16; c += 2)
              o[c / 2] = pack2<T16>(__uint_as_float(t[c]) * scale, __uint_as_float(t[c + 1]) * scale);
            *reinterpret_cast<uint4*>(dst + c0) = make_uint4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<uint4*>(dst + c0 + 8) = make_uint4(o[4], o[5], o[6], o[7]);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 16; ++c) area[(c0 + c) * 128] = __uint_as_float(t[c]);
        }
        __syncwarp();   // (the lanes of rows beyond the sequence store nothing; the next read takes the whole warp)
      }
      tc_fence_before();
      if (pieces == 1) {
        if (half == 1 && q < T) p.lse[(size_t)bh * T + q] = (reference + log2f(row_sum)) * kLn2;
        __syncwarp();
        continue;
      }
      area[kDiagD / 2 * 128] = row_sum;
      if (p.band_merges) {
        __syncwarp();
        continue;
      }
      // The warp that brings the last of the tile's pieces adds them up, for its rows and columns, in the order of the CTAs.
      __threadfence();
      __syncwarp();
      unsigned arrived = 0;
      if (lane == 0) arrived = atomicAdd(p.arrived + first * kDiagArrivals + (tile & 1) * 8 + half * 4 + wq, 1u);
      if (__shfl_sync(0xffffffffu, arrived, 0) + 1 != (unsigned)pieces) continue;
      __threadfence();
      float sum = 0.f;
      for (int i = 0; i < pieces; ++i) sum += __ldcg(area_of(i) + kDiagD / 2 * 128);
      const float whole = pow2i<T16>(-eb) / sum;
#pragma unroll 1
      for (int c0 = 0; c0 < kDiagD / 2; c0 += 16) {
        float v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] = 0.f;
        for (int i = 0; i < pieces; i += 2) {   // (two pieces' reads under way)
          const float *const a = area_of(i) + c0 * 128, *const b = area_of(min(i + 1, pieces - 1)) + c0 * 128;
          const float more = i + 1 < pieces ? 1.f : 0.f;
          float x[16], y[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) x[c] = __ldcg(a + c * 128);
#pragma unroll
          for (int c = 0; c < 16; ++c) y[c] = __ldcg(b + c * 128);
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = fmaf(y[c], more, v[c] + x[c]);
        }
        if (q < T) {
          uint32_t o[8];
#pragma unroll
          for (int c = 0; c < 16; c += 2) o[c / 2] = pack2<T16>(v[c] * whole, v[c + 1] * whole);
          *reinterpret_cast<uint4*>(dst + c0) = make_uint4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<uint4*>(dst + c0 + 8) = make_uint4(o[4], o[5], o[6], o[7]);
        }
      }
      if (half == 1 && q < T) p.lse[(size_t)bh * T + q] = (reference + log2f(sum)) * kLn2;
      __syncwarp();
    }
  } else if (warp < 24) {
    set_regs<kDiagRegs, kRegsFormer>();
    // ------------------------------------------------------------------ operands
    // A thread has one 16-byte column of every fourth row of its warp's share.  K1 stays in 16 bits (a product of two 16-bit
    // numbers is rounded once), SiLU(V1) in fp32, so that W is rounded once as well.
    constexpr int NR = 4;
    const int col = lane & 7, row0 = (warp - 16) * 16 + (lane >> 3);
    // (rows row0 + 4 i: the swizzle has two values)
    const uint32_t at[2] = {swz128(row0, col), swz128(row0 + 4, col) - 512};
    uint32_t step = 0;
    bool alive = true;
    for (uint32_t items = 0; alive; ++items) {
      if (!wait_all(&bars.item_full[items % kItemSlots], (items / kItemSlots) & 1)) break;
      const DiagItem& it = bars.items[items % kItemSlots];
      const int len = uniform(it.len);
      const int bh = uniform(it.bh), jt = uniform(it.jt), n0 = uniform(it.n0), ea = uniform(it.ea), eb = uniform(it.eb);
      arrive_warp(&bars.item_free[items % kItemSlots]);
      if (len == 0) break;
      uint32_t a[NR][4];
      float2 s[NR][4];
      {
        const float fa = pow2i<T16>(ea), fb = pow2i<T16>(eb);
        const uint32_t sign = p.alpha < 0.f ? 0x80008000u : 0u;   // (sa is not negative)
        const size_t base = ((size_t)bh * T + jt * 128) * kDiagD + col * 8;
        uint4 ka[NR], va[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const int r = row0 + 4 * i;
          const bool in = jt * 128 + r < T;
          ka[i] = in ? __ldg(reinterpret_cast<const uint4*>((const T16*)p.k1 + base + (size_t)r * kDiagD)) : make_uint4(0, 0, 0, 0);
          va[i] = in ? __ldg(reinterpret_cast<const uint4*>((const T16*)p.v1 + base + (size_t)r * kDiagD)) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const uint32_t kw[4] = {ka[i].x, ka[i].y, ka[i].z, ka[i].w}, vw[4] = {va[i].x, va[i].y, va[i].z, va[i].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (std::is_same<T16, __half>::value) {
              const float2 y = __fmul2_rn(unpack2<T16>(kw[e]), make_float2(fa, fa));
              a[i][e] = pack2<T16>(y.x, y.y) ^ sign;
            } else {
              a[i][e] = kw[e] ^ sign;
            }
            const float2 y = unpack2<T16>(vw[e]);
            s[i][e] = make_float2(silu_f(y.x) * fb, silu_f(y.y) * fb);
          }
        }
      }
      if (!wait_all(&bars.win_full, items & 1)) break;
      for (int n = n0; n < n0 + len; ++n, ++step) {
        const uint32_t buf = step % kNB, parity = ((step / kNB) & 1) ^ 1;
        // row j of the tile meets row k = j + n - kkr, which is row j + n of the window
        const uint32_t from[2] = {swz128(row0 + n, col), swz128(row0 + n + 4, col) - 512};
        alive = wait_all(&bars.a_free[buf], parity);
        if (!alive) break;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const uint4 k2 = *reinterpret_cast<const uint4*>(smem + kOffK2 + from[i & 1] + i * 512);
          *reinterpret_cast<uint4*>(smem + kOffA + buf * kTile + at[i & 1] + i * 512) = make_uint4(
              mul2<T16>(a[i][0], k2.x), mul2<T16>(a[i][1], k2.y), mul2<T16>(a[i][2], k2.z), mul2<T16>(a[i][3], k2.w));
        }
        fence_async_smem();
        arrive_warp(&bars.a_ready[buf]);
        alive = wait_all(&bars.w_free[buf], parity);
        if (!alive) break;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const uint4 v2 = *reinterpret_cast<const uint4*>(smem + kOffV2 + from[i & 1] + i * 512);
          const uint32_t vw[4] = {v2.x, v2.y, v2.z, v2.w};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 z = __fmul2_rn(s[i][e], unpack2<T16>(vw[e]));
            o[e] = pack2<T16>(z.x, z.y);
          }
          *reinterpret_cast<uint4*>(smem + kOffW + buf * kTile + at[i & 1] + i * 512) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        fence_async_smem();
        arrive_warp(&bars.w_ready[buf]);
      }
      if (alive) arrive_warp(&bars.win_free);
    }
  } else {
    set_regs<kDiagRegs, kRegsService>();
    constexpr int kFmt = std::is_same<T16, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t kHi = desc_hi(1024), kTile16 = kTile >> 4;
    constexpr uint32_t idesc_s = make_idesc_f16(128, 128, kFmt, false, false);
    constexpr uint32_t idesc_pv = make_idesc_f16(128, kDiagD, kFmt, false, true);
    const bool leader = elect_one();
    auto commit = [&](uint64_t* bar) {
      if (leader) mma_commit(bar);
    };
    if (warp == 24) {
      // ---------------------------------------------------------------- scores
      const uint32_t qLo = desc_lo(smem_u32(smem + kOffQ), 16), aLo = desc_lo(smem_u32(smem + kOffA), 16);
      uint32_t step = 0, place = 0;
      bool alive = true;
      for (uint32_t items = 0; alive; ++items) {
        if (!wait_all(&bars.item_full[items % kItemSlots], (items / kItemSlots) & 1)) break;
        const DiagItem& it = bars.items[items % kItemSlots];
        const int len = uniform(it.len), jt = uniform(it.jt), flags = uniform(it.flags);
        const uint32_t qn = uniform(it.qn);
        arrive_warp(&bars.item_free[items % kItemSlots]);
        if (len == 0) break;
        for (uint32_t t = qn; t < qn + 2 && alive; ++t) alive = wait_all(&bars.q_full[t % kNQ], (t / kNQ) & 1);
        for (int i = 0; i < len && alive; ++i, ++step) {
          const uint32_t buf = step % kNB, a = aLo + buf * kTile16;
          alive = wait_all(&bars.a_ready[buf], (step / kNB) & 1);
          for (uint32_t x = 0; x < 2 && alive; ++x) {
            const uint32_t turn = 2 * step + x, d = tmem + place * 128;
            const uint32_t q = qLo + (qn + ((jt & 1) == (int)x ? 0 : 1)) % kNQ * kTile16;
            alive = wait_all(&bars.place_free[place], ((turn / kNS) & 1) ^ 1);
            if (!alive) break;
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < kDiagD / 16; ++k)
              if (leader) mma_ss_lo(d, q + k * 2, a + k * 2, kHi, idesc_s, k > 0);
            commit(&bars.s_ready[x][step & 1]);
            place = place + 1 == kNS ? 0 : place + 1;
          }
          commit(&bars.a_free[buf]);
        }
        if (flags & kEndOwn) commit(&bars.q_free[qn % kNQ]);
        if (flags & kEndNext) commit(&bars.q_free[(qn + 1) % kNQ]);
      }
    } else if (warp == 26) {
      // ---------------------------------------------------------------- value products
      const uint32_t wLo = desc_lo(smem_u32(smem + kOffW), 16384);
      uint32_t step = 0, place = 0;
      bool alive = true;
      for (uint32_t items = 0; alive; ++items) {
        if (!wait_all(&bars.item_full[items % kItemSlots], (items / kItemSlots) & 1)) break;
        const DiagItem& it = bars.items[items % kItemSlots];
        const int len = uniform(it.len), jt = uniform(it.jt), flags = uniform(it.flags);
        arrive_warp(&bars.item_free[items % kItemSlots]);
        if (len == 0) break;
        for (int i = 0; i < len && alive; ++i, ++step) {
          const uint32_t buf = step % kNB, w = wLo + buf * kTile16;
          alive = wait_all(&bars.w_ready[buf], (step / kNB) & 1);
          for (uint32_t x = 0; x < 2 && alive; ++x) {
            const bool fresh = i == 0 && (flags & ((jt & 1) == (int)x ? kNewOwn : kNewNext));
            const uint32_t d = tmem + kTmemO + x * kDiagD, a = tmem + place * 128;
            alive = wait_all(&bars.p_ready[x], step & 1);
            if (!alive) break;
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (leader) mma_ts_lo(d, a + (k >> 1) * 32 + (k & 1) * 8, w + k * (2048 >> 4), kHi, idesc_pv, k > 0 || !fresh ? 1u : 0u);
            commit(&bars.place_free[place]);
            commit(&bars.pv_done[x]);
            place = place + 1 == kNS ? 0 : place + 1;
          }
          commit(&bars.w_free[buf]);
        }
      }
    } else if (warp == 25) {
      // ---------------------------------------------------------------- loader
      if (leader) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK2);
        tma_prefetch_desc(&tmV2);
      }
      const int R = g.diagonals(), tiles = g.tiles();
      const uint32_t window = (128 + g.kkl + g.kkr) * kDiagD * 2;
      const long end = g.cut(blockIdx.x + 1);
      long pos = g.cut(blockIdx.x);
      uint32_t items = 0, tiles_loaded = 0;
      int bh = -1;
      bool alive = true, joined = false;   // joined: the item before was the j-tile before of the same head
      DiagItem it{};
      while (true) {
        it.len = 0;
        if (pos < end) {
          const long tile = pos / R;
          const int head = (int)(tile / tiles);
          if (head != bh) {
            bh = head;
            joined = false;
            const float* st = p.stats + head;
            const float bound = head_bound(p.stats, g.BN, head, p.alpha * kLog2e);
            it.ea = range_shift<T16>(__ldg(st + kK1 * g.BN), __ldg(st + kK2 * g.BN), 0);
            it.eb = range_shift<T16>(__ldg(st + kV1 * g.BN), __ldg(st + kV2 * g.BN), 0);
            it.sa = pow2i<T16>(-it.ea) * fabsf(p.alpha * kLog2e);
            it.reference = diag_reference<T16>(bound);
          }
          it.bh = head;
          it.jt = (int)(tile - (long)head * tiles);
          it.n0 = (int)(pos - tile * R);
          it.len = (int)(end - pos < R - it.n0 ? end - pos : R - it.n0);
        }
        if (it.len > 0) {
          const bool last = pos + it.len == end, head_end = it.jt + 1 == tiles;
          it.flags = (joined ? 0 : kNewOwn) | kNewNext | kEndOwn | (last || head_end ? kEndNext : 0);
          it.qn = joined ? tiles_loaded - 1 : tiles_loaded;
        }
        alive = wait_all(&bars.item_free[items % kItemSlots], ((items / kItemSlots) & 1) ^ 1);
        if (!alive) break;
        if (leader) {
          bars.items[items % kItemSlots] = it;
          mbar_arrive(&bars.item_full[items % kItemSlots]);
        }
        if (it.len == 0) break;
        for (int t = joined ? 1 : 0; t < 2 && alive; ++t, ++tiles_loaded) {
          const uint32_t b = tiles_loaded % kNQ;
          alive = wait_all(&bars.q_free[b], ((tiles_loaded / kNQ) & 1) ^ 1);
          if (alive && leader) {
            mbar_arrive_expect_tx(&bars.q_full[b], kTile);
            tma_load_3d(smem + kOffQ + b * kTile, &tmQ, &bars.q_full[b], 0, (it.jt + t) * 128, it.bh);
          }
        }
        if (!alive) break;
        alive = wait_all(&bars.win_free, (items & 1) ^ 1);
        if (!alive) break;
        if (leader) {
          mbar_arrive_expect_tx(&bars.win_full, 2 * window);
          tma_load_3d(smem + kOffK2, &tmK2, &bars.win_full, 0, it.jt * 128 - g.kkr, it.bh);
          tma_load_3d(smem + kOffV2, &tmV2, &bars.win_full, 0, it.jt * 128 - g.kkr, it.bh);
        }
        ++items;
        joined = it.n0 + it.len == R && it.jt + 1 < tiles;
        pos += it.len;
      }
      if (!alive) {
        // give copies still in flight a bounded chance to land before the CTA retires
        const long long t0 = clock64();
        for (uint32_t t = tiles_loaded > 2 ? tiles_loaded - 2 : 0; t < tiles_loaded; ++t)
          while (!mbar_try_wait(&bars.q_full[t % kNQ], (t / kNQ) & 1) && clock64() - t0 < kWaitTicks / 8) {
          }
        if (items > 0)
          while (!mbar_try_wait(&bars.win_full, (items - 1) & 1) && clock64() - t0 < kWaitTicks / 8) {
          }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 24) tmem_dealloc(tmem, 512);
  if (tid == 0 && bars.abort_flag && p.status) atomicOr(p.status, 2);
}

constexpr int kMinSteps = 12;      // of a CTA
size_t area_bytes(int grid) { return (size_t)grid * kDiagAreas * kDiagAreaFloats * sizeof(float); }
size_t scratch_bytes(int grid) { return area_bytes(grid) + (size_t)grid * kDiagArrivals * sizeof(unsigned); }
// This kernel is asked where it costs less than the band kernel, in us: a step 1 (narrow windows, most columns masked) to 1.4, an item (a
// j-tile) 1.3 beside its steps, launch and first item 14, and 3 more, as large scores pay 2 to 3 for the question; a tile of the band kernel
// 1.6 to 2.1.  us of a call with small scores, by the band kernel / here, of CTAs of steps / tiles: 12 / 17 (a diagonal an item) 38 / 42, 12 / 14 32 / 34, 13 / 14 33 / 36, 16 / 15 36 / 38, 36 / 18
// (T=129 128/128/48/48) 36 / 57, 53 / 28 64 / 71, 65 / 42 86 / 88, 70 / 27 59 / 89;  114 / 81 163 / 150, 28 / 68 117 / 60, 42 / 47 96 / 76, 16 / 56 119 / 43,
// 86 / 69 143 / 111, 112 / 280 466 / 179.
constexpr double kStepPrice = 1, kFullStepPrice = 1.4, kItemPrice = 1.3, kLaunchPrice = 17, kTilePrice = 2;
// Tiles of a CTA of tdp_fwd_band_kernel below which that kernel adds up the pieces, launched ahead of this one's end.  A CTA that brings the
// last piece takes 7 us for them, most often at its end, the band kernel 3; in long calls the pieces of many tiles come in between.  us,
// by the band kernel / here: 8 heads T=1000 fp16 61 / 65, 16 heads T=400 128/128/48/48 76.8 / 80.5, T=2048 8/8/4/4 42.6 / 44.8, T=2048
// 128/128/32/32 181 / 179, T=8192 669 / 653, 4096 heads T=140 20/20/4/4 736 / 690.
constexpr long kMergingBandTiles = 128;
// ... and below which it is launched ahead of this one's end.  Large scores, us early / not: 16 heads T=1200 16/16/8/8 81 / 83, T=2048 13/2/12/2
// (56 tiles) 123 / 127; but with inputs that are not in L2 yet, where its CTAs then run slower, 32 heads T=1480 (80) 186 / 181, T=1726 (94) 232 / 208.
constexpr long kEarlyBandTiles = 80;

long diag_steps(int B, int N, int T, int band) { return (long)B * N * ((T + 127) / 128) * (band + 1); }
// Tiles of a CTA of tdp_fwd_band_kernel: the groups of four queries have a block of 32 K2 rows at first, and as many as reach back `reach`
// rows from there on.
double band_tiles_of_cta(long heads, int T, int reach) {
  const int r = min(reach, T - 1), groups = (T + 3) / 4, growing = r / 4;
  const double blocks = growing * (r / 64.0 + 1) + (groups - growing) * (double)((r + 35) / 32);   // of a head
  return (double)((heads * groups + num_sms() - 1) / num_sms()) * blocks / groups;
}
int diag_grid(long steps) { return (int)(steps / kMinSteps < num_sms() ? steps / kMinSteps : num_sms()); }

template <typename T16>
int launch_diag(const TdpArgs& a, const DiagParams& p) {
  const int BN = p.g.BN;
  CUtensorMap tmQ, tmK2, tmV2;
  const uint32_t window = 128 + a.mask.kkl + a.mask.kkr;
  int rc;
  if ((rc = make_tmap_3d(&tmQ, a.q, 2, kDiagD, a.T, BN, 64, 128))) return rc;
  if ((rc = make_tmap_3d(&tmK2, a.k2, 2, kDiagD, a.T, BN, 64, window))) return rc;
  if ((rc = make_tmap_3d(&tmV2, a.v2, 2, kDiagD, a.T, BN, 64, window))) return rc;
  auto kern = tdp_fwd_diag_kernel<T16>;
  // The register split assumes the count the kernel was launched with: see the backward's check.
  static std::atomic<int> registers{0};
  int n = registers.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaFuncAttributes fa;
    TRITT_CUDA_OK(cudaFuncGetAttributes(&fa, kern));
    n = fa.numRegs;
    registers.store(n, std::memory_order_relaxed);
  }
  if (n != kDiagRegs) {
    set_error("the forward kernel for narrow bands was built with %d registers per thread, its split needs %d", n, kDiagRegs);
    return -30;
  }
  TRITT_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)p.g.grid, 1, 1);
  cfg.blockDim = dim3(kDiagThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = a.stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TRITT_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tmQ, tmK2, tmV2, p));
  count_launch();
  return 0;
}

}  // namespace

size_t sm100_tdp_fwd_diag_workspace(int B, int N, int T, int D, const TdpMask* mask, int q_mod) {
  if (D != kDiagD || T <= 128) return 0;
  if (!mask) return scratch_bytes(diag_grid(diag_steps(B, N, T, kMaxBand)));
  const TdpMask& m = *mask;
  // (a query tile meets its own j-tile and the one before: q - j <= min(k1w, k2w + kkl) <= 128)
  if (!m.causal || q_mod != 1 || m.kkl + m.kkr > kMaxBand || (m.k1w > 128 && m.k2w + m.kkl > 128)) return 0;
  const long steps = diag_steps(B, N, T, m.kkl + m.kkr);
  const int grid = diag_grid(steps);
  if (grid < 1) return 0;
  const double R = m.kkl + m.kkr + 1, part = (double)steps / grid;
  const double filled = min(min(m.k1w, m.k2w) + 1, 128) / 128., step = kStepPrice + (kFullStepPrice - kStepPrice) * filled;
  if (step * part + kItemPrice * (part / R + 1) + kLaunchPrice > kTilePrice * band_tiles_of_cta((long)B * N, T, min(m.k2w, m.k1w + m.kkr))) return 0;
  return scratch_bytes(grid);
}

bool sm100_tdp_fwd_diag_plan(const TdpArgs& a, void* workspace, size_t workspace_bytes, DiagParams& p) {
  const TdpMask& m = a.mask;
  const size_t need = sm100_tdp_fwd_diag_workspace(a.B, a.N, a.T, a.D, &m, a.q_mod);
  if (need == 0 || workspace_bytes < need) return false;
  const long steps = diag_steps(a.B, a.N, a.T, m.kkl + m.kkr);
  const int grid = diag_grid(steps);
  p = DiagParams{};
  const double band_tiles = band_tiles_of_cta((long)a.B * a.N, a.T, min(m.k2w, m.k1w + m.kkr));
  p.band_merges = band_tiles < kMergingBandTiles;
  p.early = band_tiles < kEarlyBandTiles;
  p.out = a.out_o;
  p.lse = a.out_lse;
  p.k1 = a.k1;
  p.v1 = a.v1;
  p.areas = (float*)workspace;
  p.arrived = (unsigned*)((char*)workspace + area_bytes(grid));
  p.g = DiagGeometry{a.T, m.k1w, m.k2w, m.kkl, m.kkr, steps, a.B * a.N, grid};
  p.alpha = a.alpha;
  // bf16: up to what the backward takes for small scores; fp16: P = exp2(S - reference) in [2^-12.7, 2^15), normal numbers
  p.bound_limit = a.dtype == TRITT_BF16 ? 16.f : 13.5f;
  p.status = a.status_word;
  return true;
}

int sm100_tdp_fwd_diag(const TdpArgs& a, const DiagParams& p) {
  return a.dtype == TRITT_BF16 ? launch_diag<__nv_bfloat16>(a, p) : launch_diag<__half>(a, p);
}

}  // namespace tritt
