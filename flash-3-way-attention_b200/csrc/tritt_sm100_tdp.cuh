// Helpers shared by the tensor-core triple-dot-product forward and backward kernels.
#pragma once

#include "tritt_common.cuh"
#include "tritt_sm100.cuh"

#include <type_traits>

namespace tritt {
namespace {

template <typename T16> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <typename T16> __device__ __forceinline__ float2 unpack2(uint32_t v);
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t v) {
  return __half22float2(*reinterpret_cast<__half2*>(&v));
}

// The products of two pairs, rounded once (a product is exact in fp32, so the same as a multiplication there and a rounding).
template <typename T16> __device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t mul2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t mul2<__half>(uint32_t a, uint32_t b) {
  const __half2 v = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Bit 15 and bit 31 of the result: the low and the high element's exponent is all ones, that is infinite or NaN (no other carries
// out of it).  The other bits mean nothing.
template <typename T16> __device__ __forceinline__ uint32_t not_finite(uint32_t v) {
  return std::is_same<T16, __half>::value ? (v & 0x7c007c00u) + 0x04000400u : (v & 0x7f807f80u) + 0x00800080u;
}

// The larger |element| of each half: of two, or, `NAN_TOO`, NaN if one is.
template <bool NAN_TOO> __device__ __forceinline__ __half2 larger_abs(__half2 m, __half2 v) {
  return NAN_TOO ? __hmax2_nan(m, __habs2(v)) : __hmax2(m, __habs2(v));
}
template <bool NAN_TOO> __device__ __forceinline__ __nv_bfloat162 larger_abs(__nv_bfloat162 m, __nv_bfloat162 v) {
  return NAN_TOO ? __hmax2_nan(m, __habs2(v)) : __hmax2(m, __habs2(v));
}
template <typename T16> struct Pair;
template <> struct Pair<__half> { using type = __half2; };
template <> struct Pair<__nv_bfloat16> { using type = __nv_bfloat162; };
// m's halves grown by the 8 elements of v
template <typename T16, bool NAN_TOO> __device__ __forceinline__ void grow_abs(uint32_t& m, const uint4& v) {
  using P = typename Pair<T16>::type;
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const P x = larger_abs<NAN_TOO>(*reinterpret_cast<const P*>(&m), *reinterpret_cast<const P*>(&w[e]));
    m = *reinterpret_cast<const uint32_t*>(&x);
  }
}

// fp16 only: A = K1 K2 and A' = SiLU(V1) V2 (the forward's W) are products of two small factors (keys of 0.01: 1e-4, against a smallest normal
// value of 6e-5) or of two large ones (beyond 65504 from 256 on), so one factor, x, is taken times a power of two per head:
// the largest that keeps both itself and the largest product the head's elements allow below 2^15.  With the other factor's
// largest element at 1 or above the largest product has 28 binades of normal numbers below it, at 2^-b 28 - b.
// The power is divided out in fp32, of S and dP in the soft-max warps and of the sums.  bf16 has fp32's range: 0.
// Without statistics (or with infinite ones) the power is `otherwise`.
template <typename T16> __device__ __forceinline__ int range_shift(float x, float other, int otherwise) {
  if constexpr (std::is_same<T16, __half>::value) {
    if (!(x > 0.f) || !isfinite(x) || !(other > 0.f) || !isfinite(other)) return otherwise;
    const int a = (__float_as_int(x) >> 23) - 127, b = (__float_as_int(other) >> 23) - 127;
    return 14 - a - max(b + 1, 0);
  }
  return 0;
}
// 2^e for the shifts of fp16 operands, exact, |e| <= 126 (1, without looking at e, for bf16, whose shifts are all 0)
template <typename T16> __device__ __forceinline__ float pow2i(int e) {
  return std::is_same<T16, __half>::value ? __int_as_float((127 + e) << 23) : 1.f;
}

// Bits c of [lo, hi] among 0..31: with a mask of a row's columns a per-element test is one logic instruction (a constant
// bit into a predicate) instead of two comparisons.
__device__ __forceinline__ uint32_t column_mask(int lo, int hi) {
  const uint32_t up = hi < 0 ? 0u : hi >= 31 ? ~0u : (2u << hi) - 1u;
  const uint32_t down = lo <= 0 ? ~0u : lo > 31 ? 0u : ~0u << lo;
  return up & down;
}

// Bound on every score of a head, in log2 units: |s| max_q |Q_q| max |K2 element| max_j |K1_j|, s = alpha log2(e), from the forward's
// statistics (fwd_prepare_kernel).  (Rounded one by one, so that all kernels that ask get the same answer.
// FIRST: reads that the compiler keeps behind a wait for the preparation, as __ldg's need not be.)
template <bool FIRST = false> __device__ __forceinline__ float head_bound(const float* stats, int BN, int bh, float s) {
  auto read = [](const float* p) { return FIRST ? __ldcg(p) : __ldg(p); };
  const float q = __fsqrt_rn(read(stats + BN + bh)), k2 = __fsqrt_rn(read(stats + 2 * BN + bh)), k1 = __fsqrt_rn(read(stats + bh));
  return __fmul_rn(__fmul_rn(__fmul_rn(fabsf(s), q), k2), k1);
}

// Sum of v[0..31] over the 32 lanes of a warp, column-wise: on return lane i holds the
// total of column i.  31 shuffles instead of 32 full reductions.
__device__ __forceinline__ float warp_transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int half = 16; half >= 1; half >>= 1) {
    const bool upper = lane & half;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = upper ? v[i + half] : v[i];
      const float send = upper ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
    }
  }
  return v[0];
}

// SiLU(V1) in the input dtype, computed once per call (the reference does the same as a
// separate PyTorch pass, flash_trittention.py:61-62); the value tiles are then plain TMA loads.
template <typename T16>
__global__ void silu_kernel(const T16* __restrict__ in, T16* __restrict__ out, size_t n) {
  size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i + 8 <= n) {
    const uint4 v = *reinterpret_cast<const uint4*>(in + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack2<T16>(w[e]);
      o[e] = pack2<T16>(silu_f(f.x), silu_f(f.y));
    }
    *reinterpret_cast<uint4*>(out + i) = make_uint4(o[0], o[1], o[2], o[3]);
  } else {
    for (; i < n; ++i) out[i] = from_f<T16>(silu_f(to_f(in[i])));
  }
}

inline int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
  }
  return sms;
}


}  // namespace
}  // namespace tritt
