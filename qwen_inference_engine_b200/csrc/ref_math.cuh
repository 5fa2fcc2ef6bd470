// ref_math.cuh -- device functions that reproduce the reference's arithmetic op for op
// (citations relative to the reference's layers/).  Shared by the per-operator kernels
// (ops_ref_order.cu, gemm_ref_order.cu) and the persistent decode kernel (decode_mega.cu).
// Translation units including this header are compiled with -fmad=false: every fused
// multiply-add that nvcc's default contraction makes of the reference's source expressions is
// spelled __fmaf_rn (which product of a two-product sum it fuses: oracle/fma_contract.cu
// compares outputs), everything else is an explicit _rn intrinsic.
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace qie {

// ------------------------------------------------------------------ quotients by one divisor
// RN(x / b) for several bf16 numerators x: q = RN(x y) with y = RN(1 / b), then one correction q + RN(x - b q) y (Markstein, IBM J. Res. Dev. 34,
// 1990).  For fp32 numerators a second correction makes it exact in general; with 8 significant bits one is enough, which holds for
// every pair of significands (all 2^7 x 2^23 compared with the division).  Three instructions instead of about fifteen.  Magnitudes outside
// quot_ok's range (zero and its sign, subnormals, infinities) take the division.
struct Quot {
  float b, y;
  bool ok;
};
__device__ __forceinline__ Quot quot_of(float b) { return Quot{b, __frcp_rn(b), b >= 0x1p-20f && b <= 0x1p20f}; }
template <int N>
__device__ __forceinline__ void quot16(float (&x)[N], const Quot& d) {
  float lo = fabsf(x[0]), hi = lo;
#pragma unroll
  for (int i = 1; i < N; ++i) lo = fminf(lo, fabsf(x[i])), hi = fmaxf(hi, fabsf(x[i]));
  if (d.ok && lo >= 0x1p-100f && hi <= 0x1p100f) {  // (a NaN among the others passes and stays one)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float q = __fmul_rn(x[i], d.y);
      x[i] = __fmaf_rn(__fmaf_rn(-d.b, q, x[i]), d.y, q);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = __fdiv_rn(x[i], d.b);
  }
}

// The same for fp32 numerators of no matter how many bits: the first correction leaves the quotient or a neighbour of it, the second rounds correctly
// (Markstein).  Zeros are fine where they are positive.
__device__ __forceinline__ bool quot32_ok(float x) { return __float_as_uint(x) == 0u || (fabsf(x) >= 0x1p-100f && fabsf(x) <= 0x1p100f); }
__device__ __forceinline__ float quot32_fast(float x, const Quot& d) {
  float q = __fmul_rn(x, d.y);
  q = __fmaf_rn(__fmaf_rn(-d.b, q, x), d.y, q);
  return __fmaf_rn(__fmaf_rn(-d.b, q, x), d.y, q);
}
__device__ __forceinline__ float quot1(float x, const Quot& d) { return d.ok && quot32_ok(x) ? quot32_fast(x, d) : __fdiv_rn(x, d.b); }
template <int N>
__device__ __forceinline__ void quot32(float (&x)[N], const Quot& d) {
  bool ok = d.ok;
#pragma unroll
  for (int i = 0; i < N; ++i) ok = ok && quot32_ok(x[i]);
  if (ok) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = quot32_fast(x[i], d);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = __fdiv_rn(x[i], d.b);
  }
}

// ------------------------------------------------------------------ products of bf16 pairs
__device__ __forceinline__ void add2(float& a, float& b, float x, float y) {
  asm("{\n\t.reg .b64 u, v;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tadd.rn.f32x2 u, u, v;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "+f"(a), "+f"(b) : "f"(x), "f"(y));
}
// the low and the high products of two words of bf16 pairs, with c and d added before the one rounding each
__device__ __forceinline__ void fma16(float& a, float& b, uint32_t x, uint32_t y, float c, float d) {
  asm("{\n\t.reg .b16 xl, xh, yl, yh;\n\tmov.b32 {xl, xh}, %2;\n\tmov.b32 {yl, yh}, %3;\n\tfma.rn.f32.bf16 %0, xl, yl, %4;\n\tfma.rn.f32.bf16 %1, xh, yh, %5;\n\t}"
      : "=&f"(a), "=f"(b) : "r"(x), "r"(y), "f"(c), "f"(d));
}
// Products of two bf16 numbers between 2^-62 and 2^62 are exact in fp32, so p + q k rounded once is what the product and the sum are; a product
// alone is -0 + q k.
// Lowest and highest magnitude of packed pairs, and whether they leave that range (a zero does: its tiles take products and sums).
struct Magnitudes {
  uint32_t lo = 0x7fff7fffu, hi = 0u;
  __device__ __forceinline__ void see(uint32_t w) {
    w &= 0x7fff7fffu;
    lo = __vminu2(lo, w), hi = __vmaxu2(hi, w);
  }
  __device__ __forceinline__ bool beyond() const {
    return min(lo & 0xffffu, lo >> 16) < (uint32_t)(127 - 62) << 7 || max(hi & 0xffffu, hi >> 16) > (uint32_t)(127 + 62) << 7;
  }
};

// ------------------------------------------------------------------ per-head tree sum
// Lane l holds, for p in [0,NP): elements t = 64p + 2l and 64p + 2l + 1 of a head of
// hd = 64*NP values.  Reproduces  for (stride = hd/2; stride > 0; stride >>= 1)
//   buf[t] += buf[t+stride]  (t < stride)   exactly; the result is valid in lane 0.
template <int NP>
__device__ __forceinline__ float head_tree_sum(float (&v)[NP][2]) {
#pragma unroll
  for (int s = NP / 2; s >= 1; s >>= 1)  // strides >= 64: partners live in the same lane
#pragma unroll
    for (int p = 0; p < s; ++p) {
      v[p][0] = __fadd_rn(v[p][0], v[p + s][0]);
      v[p][1] = __fadd_rn(v[p][1], v[p + s][1]);
    }
  float a = v[0][0], b = v[0][1];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {  // strides 32,16,8,4,2
    a = __fadd_rn(a, __shfl_down_sync(0xffffffffu, a, o));
    b = __fadd_rn(b, __shfl_down_sync(0xffffffffu, b, o));
  }
  return __fadd_rn(a, b);  // stride 1
}

// q/k-norm of one head held in registers (in place, values become the bf16-rounded
// results as floats): qk_norm.cu:46-78.
template <int NP>
__device__ __forceinline__ void head_norm(float (&x)[NP][2], const bf16* __restrict__ w, int lane, float eps = 1e-04f) {
  float sq[NP][2];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    sq[p][0] = __fmul_rn(x[p][0], x[p][0]);
    sq[p][1] = __fmul_rn(x[p][1], x[p][1]);
  }
  float tot = head_tree_sum<NP>(sq);
  float rms = __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)(64 * NP)), eps));
  rms = __shfl_sync(0xffffffffu, rms, 0);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    uint32_t wp = *reinterpret_cast<const uint32_t*>(w + 64 * p + 2 * lane);
    x[p][0] = bf2f(f2bf(__fmul_rn(__fdiv_rn(x[p][0], rms), lo2f(wp))));
    x[p][1] = bf2f(f2bf(__fmul_rn(__fdiv_rn(x[p][1], rms), hi2f(wp))));
  }
}

// RoPE of one head held in registers: RoPE.cu:15-18 (pair j = 32p + lane).
template <int NP>
__device__ __forceinline__ void head_rope(float (&x)[NP][2], const float* __restrict__ cos_row,
                                          const float* __restrict__ sin_row, int lane) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    float c = cos_row[32 * p + lane], s = sin_row[32 * p + lane];
    float x0 = x[p][0], x1 = x[p][1];
    float v1 = __fmaf_rn(x0, c, -__fmul_rn(x1, s));
    float v2 = __fmaf_rn(c, x1, __fmul_rn(x0, s));
    x[p][0] = bf2f(f2bf(v1));
    x[p][1] = bf2f(f2bf(v2));
  }
}

template <int NP>
__device__ __forceinline__ void head_load(float (&x)[NP][2], const bf16* __restrict__ src, int lane) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    uint32_t v = *reinterpret_cast<const uint32_t*>(src + 64 * p + 2 * lane);
    x[p][0] = lo2f(v);
    x[p][1] = hi2f(v);
  }
}
template <int NP>
__device__ __forceinline__ void head_store(const float (&x)[NP][2], bf16* __restrict__ dst, int lane) {
#pragma unroll
  for (int p = 0; p < NP; ++p)
    *reinterpret_cast<uint32_t*>(dst + 64 * p + 2 * lane) = pack2(f2bf(x[p][0]), f2bf(x[p][1]));
}

// SiLU.cu:6-8,19-20:  y = x * (1 / (1 + expf(-x)))
__device__ __forceinline__ float silu_ref(float x) {
  float sg = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x)));
  return __fmul_rn(x, sg);
}


// arg-max candidate order of the reference sampler (logit_decode.cu:15-33,182-223):
// value, then the larger bit-reversed low byte of the index, then the lower index.
struct Cand {
  float val;
  int idx;
};
__device__ __forceinline__ bool cand_better(float va, int ia, float vb, int ib) {
  if (ib < 0) return ia >= 0;
  if (ia < 0) return false;
  if (va > vb) return true;
  if (va < vb) return false;
  unsigned ra = __brev((unsigned)ia << 24), rb = __brev((unsigned)ib << 24);
  if (ra != rb) return ra > rb;
  return ia < ib;
}


}  // namespace qie
