// What the forward kernel that steps over the diagonals of a narrow band (tritt_sm100_tdp_fwd_diag.cu) shares with the one that serves
// such calls otherwise (tritt_sm100_tdp_fwd_band.cu): which of the two does a call, and the pieces of the query tiles that the first one cuts.
#pragma once

#include "tritt_sm100_tdp.cuh"

#include <type_traits>

namespace tritt {

constexpr int kDiagD = 64;                                // head dimension
constexpr int kDiagAreaFloats = 2 * 128 * (kDiagD / 2 + 1);   // of either half of the columns: accumulator [D / 2][128], sums [128]
constexpr int kDiagArrivals = 16;
constexpr int kDiagAreas = 4;   // of a CTA: tiles begun before its part (by the parity of the tile), tiles begun in it
constexpr float kDiagReferenceFraction = 0.142019f;       // (see kReferenceFraction of the general forward kernel)

struct DiagGeometry {
  int T, k1w, k2w, kkl, kkr;
  long steps;      // of the call
  int BN, grid;
  __host__ __device__ int tiles() const { return (T + 127) / 128; }
  __host__ __device__ int diagonals() const { return kkl + kkr + 1; }
  __host__ __device__ long cut(long c) const { return steps * c / grid; }
  __host__ __device__ int cta_of(long step) const { return (int)(((step + 1) * grid + steps - 1) / steps - 1); }   // the last c with cut(c) <= step
  // the CTAs that have steps of query tile t
  __host__ __device__ void ctas(int bh, int t, int& first, int& count) const {
    const long row = (long)bh * tiles(), R = diagonals();
    first = cta_of((row + (t > 0 ? t - 1 : 0)) * R);
    count = cta_of((row + t + 1) * R - 1) - first + 1;
  }
};

struct DiagParams {
  void* out;
  float* lse;
  const void *k1, *v1;
  const float* stats;    // [7][BN] (see fwd_prepare_kernel)
  float* areas;          // [grid][kDiagAreas][kDiagAreaFloats]
  unsigned* arrived;     // [grid][kDiagArrivals], zero: pieces there are of the tiles begun in a CTA's part, by the tile's parity and by warp
  DiagGeometry g;
  float alpha, bound_limit;
  bool band_merges;      // tdp_fwd_band_kernel adds up the pieces
  bool early;            // ... and is launched ahead of this kernel's end
  int* status;
};

// Fills `p` but for the statistics and returns true if that kernel is asked; `workspace`: sm100_tdp_fwd_diag_workspace() bytes of scratch.
// p.arrived[0 .. p.g.grid * kDiagArrivals) has to be zero when it starts.
bool sm100_tdp_fwd_diag_plan(const TdpArgs& a, void* workspace, size_t workspace_bytes, DiagParams& p);
int sm100_tdp_fwd_diag(const TdpArgs& a, const DiagParams& p);
// `sv1`: SiLU(V1) in the inputs' type; `k1n`: per-head largest squared K1 row norm, or null (both prepared by the caller);
// `diag`: what sm100_tdp_fwd_diag() was launched with just before, or null.
int sm100_tdp_fwd_band(const TdpArgs& a, const void* sv1, const float* k1n, const DiagParams* diag);

namespace {

// Statistics of fwd_prepare_kernel: arrays of BN values.
enum { kK1 = 3, kK2 = 4, kV1 = 5, kV2 = 6 };   // largest |element|

// The soft-max reference of all rows of a head, from the bound on its scores: P = exp2(S - reference) is below 2^15 in fp16, 1 in bf16.
template <typename T16> __device__ __forceinline__ float diag_reference(float bound) {
  return ceilf(bound) + kDiagReferenceFraction - (std::is_same<T16, __half>::value ? 15.f : 0.f);
}

// Whether the kernel that steps over diagonals does the call: the scores of all heads are small.  All threads of the block.
__device__ __forceinline__ bool diag_takes(const DiagParams& p) {
  bool large = false;   // (not >: inf * 0 is large as well; a head with an element that is not finite has an infinite bound)
  for (int bh = threadIdx.x; bh < p.g.BN; bh += blockDim.x)
    large |= !(head_bound<true>(p.stats, p.g.BN, bh, p.alpha * kLog2e) <= p.bound_limit);
  return !__syncthreads_or(large);
}

// Piece i of query tile `tile`, whose first one is CTA `first`'s: one half of the columns.
__device__ __forceinline__ float* diag_area(const DiagParams& p, int first, int i, int tile, int half) {
  return p.areas + ((size_t)(first + i) * kDiagAreas + (i == 0 ? 2 : 0) + (tile & 1)) * kDiagAreaFloats + half * (kDiagAreaFloats / 2);
}

// The pieces of the query tiles that are cut -> their outputs.  A thread takes 16 columns of a row at a time.
template <typename T16>
__device__ __forceinline__ void diag_merge(const DiagParams& p) {
  const DiagGeometry& g = p.g;
  const int tiles = g.tiles(), units = g.BN * tiles * (kDiagD / 16), per_block = blockDim.x / 128, row = threadIdx.x % 128;
  for (int u = blockIdx.x * per_block + threadIdx.x / 128; u < units; u += gridDim.x * per_block) {
    const int bh = u / (kDiagD / 16) / tiles, tile = u / (kDiagD / 16) % tiles, c0 = u % (kDiagD / 16) * 16, q = tile * 128 + row;
    int first, pieces;
    g.ctas(bh, tile, first, pieces);
    if (pieces == 1 || q >= g.T) continue;   // (whole: written by its CTA)
    float l = 0.f, v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = 0.f;
#pragma unroll 2
    for (int i = 0; i < pieces; ++i) {
      const float* a = diag_area(p, first, i, tile, c0 / (kDiagD / 2)) + row;
      l += a[kDiagD / 2 * 128];
#pragma unroll
      for (int c = 0; c < 16; ++c) v[c] += a[(c0 % (kDiagD / 2) + c) * 128];
    }
    const float* st = p.stats + bh;
    const float scale = pow2i<T16>(-range_shift<T16>(__ldg(st + kV1 * g.BN), __ldg(st + kV2 * g.BN), 0)) / l;
    T16* dst = (T16*)p.out + ((size_t)bh * g.T + q) * kDiagD + c0;
#pragma unroll
    for (int c = 0; c < 16; c += 8)
      *reinterpret_cast<uint4*>(dst + c) =
          make_uint4(pack2<T16>(v[c] * scale, v[c + 1] * scale), pack2<T16>(v[c + 2] * scale, v[c + 3] * scale),
                     pack2<T16>(v[c + 4] * scale, v[c + 5] * scale), pack2<T16>(v[c + 6] * scale, v[c + 7] * scale));
    if (c0 == 0)
      p.lse[(size_t)bh * g.T + q] = (diag_reference<T16>(head_bound(p.stats, g.BN, bh, p.alpha * kLog2e)) + log2f(l)) * kLn2;
  }
}

}  // namespace
}  // namespace tritt
