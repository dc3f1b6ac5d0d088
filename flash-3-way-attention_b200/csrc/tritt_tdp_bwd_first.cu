// The first queries of a causal triple-dot-product backward, in exact fp32 on the CUDA cores: what they add to the sums
// dK1 | dK2 | dSiLU(V1) | dV2, and their dQ.  (Why they are not the tensor-core kernel's: see kFirstQueries there.)
//
// One CTA per (head, query); a query q < 16 (or 32) attends keys 0 .. q, at most 16 x 16 pairs, so everything it needs stays in
// shared memory.  With the rows A[k] = alpha log2(e) Q K2[k] and B[k] = dO V2[k]:
//     S[k,j] = A[k] . K1[j]     P = c exp2(S - max)      dP[k,j] = B[k] . SiLU(V1)[j]     dS = P (dP - Dq)
//     F = dS K1:    dK2[k] += alpha Q F[k],   dQ = alpha sum_k K2[k] F[k]        W = P SiLU(V1):  dV2[k] += dO W[k]
//     G = dS^T A:   dK1[j] += ln(2) G[j]                                         U = P^T B:       dSV1[j] += U[j]
// c brings P to the mass that the forward's scores (A rounded to the inputs' type) have under the saved log-sum-exp, 1 for a
// whole soft-max: exp2(S - lse2) of a query of few pairs and large scores does not sum to one (dV2 1.05 to 1.19 times as
// far from fp64 as with the forward's scores, for scores of order 4 and T=50 to 120), and overflows for scores of order 1e5.
// Dq is the exact sum P dP: dO . O has the forward's rounding of SiLU(V1) and of O, which dP has not, and a query of one
// dominant pair is left with that difference as its dS (16 heads, T=2 to 12, scores of order 3 to 10: dQ 5e-3 to 9e-3 of its
// norm from fp64 in bf16, 6e-4 to 1.3e-3 in fp16; with the exact sum the rounding of the result to 16 bits is what is left,
// 1.7e-3 and 2.1e-4).
// It is latency that counts (it runs ahead of the tensor-core kernel), so every query has a CTA, which adds its share to the
// sums: about 8 us at 4 heads, D=128 and at 16 heads, D=64.  (The general CUDA-core kernel, which walks a query's rows one
// tile after the other, took 60 and 50 us for twice as many queries, this one 12.5 and 18 us for those.)
#include "tritt_common.cuh"
#include "tritt_sm100_tdp.cuh"

namespace tritt {
namespace {

constexpr int kFirstThreads = 256;

template <int D, int NF> struct FirstShared {   // NF: queries below this, and so keys
  static constexpr int kPitch = D + 4;   // (rows 4 banks apart: 8 lanes' 16-byte reads of 8 rows do not conflict)
  float k1[NF][kPitch], s1[NF][kPitch], a[NF][kPitch], b[NF][kPitch];
  float p_kj[NF][NF + 4], ds_kj[NF][NF + 4];   // [k][j], and transposed
  float p_jk[NF][NF + 4], ds_jk[NF][NF + 4];
  float4 mass[kFirstThreads / 32];   // (each warp's largest score, sum of P, of the forward's P, and of P dP)
  float q[D], d_o[D], dq[kFirstThreads / (D / 4)][D];
};

struct FirstParams {
  const void *q, *k1, *k2, *v1, *v2, *d_o;
  const float *lse, *drow;
  float* sums;     // dK1 | dK2 | dSiLU(V1) | dV2 | dQ, n each
  size_t n;
  int T, q_mod, q_rem;
  float alpha;
  TdpMask mask;
};

__device__ __forceinline__ float4 fma4(float s, float4 a, float4 c) {
  return make_float4(fmaf(s, a.x, c.x), fmaf(s, a.y, c.y), fmaf(s, a.z, c.z), fmaf(s, a.w, c.w));
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c))));
}
__device__ __forceinline__ void add_to(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
template <int D, typename T16, int NF>
__global__ void __launch_bounds__(kFirstThreads) tdp_bwd_first_kernel(const __grid_constant__ FirstParams p) {
  extern __shared__ __align__(16) uint8_t raw[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the tensor-core kernel need not wait for this one
  FirstShared<D, NF>& sh = *reinterpret_cast<FirstShared<D, NF>*>(raw);
  const int tid = threadIdx.x, bh = blockIdx.y;
  const int q = p.q_rem + ((int)gridDim.x - 1 - (int)blockIdx.x) * p.q_mod;   // the longest first
  const size_t head = (size_t)bh * p.T * D;
  const float scale2 = p.alpha * kLog2e;
  const int nk = q + 1;   // keys
  auto load8 = [&](const void* base, int row, int h, float (&f)[8]) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>((const T16*)base + head + (size_t)row * D + h));
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 v = unpack2<T16>(w[e]);
      f[2 * e] = v.x;
      f[2 * e + 1] = v.y;
    }
  };
  auto store8 = [](float* dst, const float (&f)[8]) {
    *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
  };
  for (int i = tid; i < nk * (D / 8); i += kFirstThreads) {
    const int row = i / (D / 8), h = i % (D / 8) * 8;
    float f[8], m[8];
    load8(p.k1, row, h, f);
    store8(&sh.k1[row][h], f);
    load8(p.v1, row, h, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = silu_f(f[e]);
    store8(&sh.s1[row][h], f);
    load8(p.k2, row, h, f);
    load8(p.q, q, h, m);
    if (row == 0) store8(&sh.q[h], m);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= scale2 * m[e];
    store8(&sh.a[row][h], f);
    load8(p.v2, row, h, f);
    load8(p.d_o, q, h, m);
    if (row == 0) store8(&sh.d_o[h], m);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= m[e];
    store8(&sh.b[row][h], f);
  }
  __syncthreads();
  // ---- P and dS: one key j and E keys k per thread
  {
    constexpr int E = NF * NF / kFirstThreads;
    const int j = tid % NF, k0 = tid / NF * E;
    const float lse2 = __ldg(p.lse + (size_t)bh * p.T + q) * kLog2e;
    const bool single = p.mask.single_pair(q);   // (its score gradient is exactly zero)
    float s[E], s16[E], dp[E];
#pragma unroll
    for (int e = 0; e < E; ++e) s[e] = s16[e] = dp[e] = 0.f;
    if (j < nk && k0 < nk) {
#pragma unroll 4
      for (int h = 0; h < D; h += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&sh.k1[j][h]), y = *reinterpret_cast<const float4*>(&sh.s1[j][h]);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int k = min(k0 + e, q);
          const float4 a = *reinterpret_cast<const float4*>(&sh.a[k][h]);
          const float2 r0 = unpack2<T16>(pack2<T16>(a.x, a.y)), r1 = unpack2<T16>(pack2<T16>(a.z, a.w));
          s[e] = dot4(x, a, s[e]);
          s16[e] = dot4(x, make_float4(r0.x, r0.y, r1.x, r1.y), s16[e]);
          dp[e] = dot4(y, *reinterpret_cast<const float4*>(&sh.b[k][h]), dp[e]);
        }
      }
    }
    // P: the exact soft-max, with the mass of the forward's scores.  (Not exp2(S - lse2): rounding moves large scores by
    // more than the exponent's range, and an exponential that overflows cannot be scaled back.)
    float top = -INFINITY, sum = 0.f, sum16 = 0.f, sum_dp = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (p.mask.valid(q, j, k0 + e)) top = fmaxf(top, s[e]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const bool ok = p.mask.valid(q, j, k0 + e);
      s[e] = ok ? exp2f(s[e] - top) : 0.f;
      sum += s[e];
      sum16 += ok ? exp2f(s16[e] - lse2) : 0.f;
      if (s[e] != 0.f) sum_dp = fmaf(s[e], dp[e], sum_dp);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      sum16 += __shfl_xor_sync(0xffffffffu, sum16, o);
      sum_dp += __shfl_xor_sync(0xffffffffu, sum_dp, o);
    }
    if ((tid & 31) == 0) sh.mass[tid >> 5] = make_float4(top, sum, sum16, sum_dp);
    __syncthreads();
    float row_top = -INFINITY;
#pragma unroll
    for (int w = 0; w < kFirstThreads / 32; ++w) row_top = fmaxf(row_top, sh.mass[w].x);
    sum = sum16 = sum_dp = 0.f;
#pragma unroll
    for (int w = 0; w < kFirstThreads / 32; ++w) {
      const float4 m = sh.mass[w];
      const float f = m.x == -INFINITY ? 1.f : exp2f(m.x - row_top);   // (a warp without a pair: 0; a NaN stays one)
      sum = fmaf(m.y, f, sum);
      sum16 += m.z;
      if (f != 0.f) sum_dp = fmaf(m.w, f, sum_dp);
    }
    const float c = sum > 0.f ? exp2f(top - row_top) * (sum16 / sum) : 1.f;   // (nothing attended: P is zero; NaN: it stays)
    // Dq = sum P dP where P is the whole soft-max (to 2^-11: its mass has the fp32 rounding of a score in the exponent), else
    // the given dO . O, the sum over all that the log-sum-exp counts
    const float Dq = fabsf(sum16 - 1.f) < 0x1p-11f ? sum_dp / sum : __ldg(p.drow + (size_t)bh * p.T + q);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int k = k0 + e;
      const float pr = s[e] * c;
      const float ds = pr != 0.f && !single ? pr * (dp[e] - Dq) : 0.f;
      sh.p_kj[k][j] = sh.p_jk[j][k] = pr;
      sh.ds_kj[k][j] = sh.ds_jk[j][k] = ds;
    }
  }
  __syncthreads();
  // ---- the four products: 4 columns h of R rows per thread
  constexpr int kChunks = D / 4, kGroups = kFirstThreads / kChunks, R = NF / kGroups;   // NF=16: 8 groups of 2 at D=128, 16 of 1 at 64
  const int h = tid % kChunks * 4, r0 = tid / kChunks * R;
  float4 dq = make_float4(0.f, 0.f, 0.f, 0.f);
  if (r0 < nk) {
    const float4 qv = *reinterpret_cast<const float4*>(&sh.q[h]), dov = *reinterpret_cast<const float4*>(&sh.d_o[h]);
    const float4 aq = make_float4(p.alpha * qv.x, p.alpha * qv.y, p.alpha * qv.z, p.alpha * qv.w);
    const size_t row0 = head + (size_t)r0 * D + h;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    // sum over the pair's other key: two weight matrices (columns of R rows) against two key matrices
    auto products = [&](const float (*wx)[NF + 4], const float (*wy)[NF + 4], const float (*x)[D + 4], const float (*y)[D + 4],
                        float4 (&gx)[R], float4 (&gy)[R]) {
#pragma unroll
      for (int r = 0; r < R; ++r) gx[r] = gy[r] = zero;
#pragma unroll 2
      for (int i = 0; i < nk; ++i) {
        const float4 xv = *reinterpret_cast<const float4*>(&x[i][h]), yv = *reinterpret_cast<const float4*>(&y[i][h]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          gx[r] = fma4(wx[i][r0 + r], xv, gx[r]);   // (R neighbouring floats, the same for the lanes of a row)
          gy[r] = fma4(wy[i][r0 + r], yv, gy[r]);
        }
      }
    };
    float4 f[R], w[R];
    products(sh.ds_jk, sh.p_jk, sh.k1, sh.s1, f, w);   // rows k, summed over j
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = r0 + r;
      if (k < nk) {
        add_to(p.sums + p.n + row0 + (size_t)r * D, mul4(aq, f[r]));
        add_to(p.sums + 3 * p.n + row0 + (size_t)r * D, mul4(dov, w[r]));
        const uint2 kw = __ldg(reinterpret_cast<const uint2*>((const T16*)p.k2 + row0 + (size_t)r * D));
        const float2 lo = unpack2<T16>(kw.x), hi = unpack2<T16>(kw.y);
        dq = make_float4(fmaf(lo.x, f[r].x, dq.x), fmaf(lo.y, f[r].y, dq.y), fmaf(hi.x, f[r].z, dq.z), fmaf(hi.y, f[r].w, dq.w));
      }
    }
    products(sh.ds_kj, sh.p_kj, sh.a, sh.b, f, w);     // rows j, summed over k
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r0 + r < nk) {
        add_to(p.sums + row0 + (size_t)r * D, make_float4(f[r].x * kLn2, f[r].y * kLn2, f[r].z * kLn2, f[r].w * kLn2));
        add_to(p.sums + 2 * p.n + row0 + (size_t)r * D, w[r]);
      }
  }
  *reinterpret_cast<float4*>(&sh.dq[tid / kChunks][h]) = dq;
  __syncthreads();
  if (tid < D) {
    float x = 0.f;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) x += sh.dq[g][tid];
    p.sums[4 * p.n + head + (size_t)q * D + tid] = p.alpha * x;
  }
}

template <int D, typename T16, int NF>
int launch_first_nf(const TdpArgs& a, int queries, float* sums, const float* drow) {
  FirstParams p{};
  p.q = a.q; p.k1 = a.k1; p.k2 = a.k2; p.v1 = a.v1; p.v2 = a.v2; p.d_o = a.d_o;
  p.lse = a.lse_in; p.drow = drow; p.sums = sums; p.n = (size_t)a.B * a.N * a.T * D;
  p.T = a.T; p.q_mod = a.q_mod; p.q_rem = a.q_rem; p.alpha = a.alpha; p.mask = a.mask;
  auto kern = tdp_bwd_first_kernel<D, T16, NF>;
  TRITT_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FirstShared<D, NF>)));
  kern<<<dim3(queries, a.B * a.N), kFirstThreads, sizeof(FirstShared<D, NF>), a.stream>>>(p);
  count_launch();
  TRITT_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int D, typename T16>
int launch_first(const TdpArgs& a, int queries, float* sums, const float* drow) {
  // (the plan takes 16 or 32 queries of the sequence)
  return tdp_bwd_first_count(a.T) == 16 ? launch_first_nf<D, T16, 16>(a, queries, sums, drow)
                                        : launch_first_nf<D, T16, 32>(a, queries, sums, drow);
}

}  // namespace

int tdp_bwd_first_queries(const TdpArgs& a, int queries, float* sums, const float* drow) {
  if (a.dtype == TRITT_BF16)
    return a.D == 128 ? launch_first<128, __nv_bfloat16>(a, queries, sums, drow)
                      : launch_first<64, __nv_bfloat16>(a, queries, sums, drow);
  return a.D == 128 ? launch_first<128, __half>(a, queries, sums, drow) : launch_first<64, __half>(a, queries, sums, drow);
}

}  // namespace tritt
