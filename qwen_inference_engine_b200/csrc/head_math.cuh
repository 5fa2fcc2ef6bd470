// head_math.cuh -- head norms (layers/src/qk_norm.cu:43-80) and rotary positions (layers/src/RoPE.cu:6-22) of a head on a few lanes, every result by the
// reference's sequence of IEEE operations (ref_math.cuh).
#pragma once
#include "common.cuh"
#include "ref_math.cuh"

namespace qie {

// 16 bytes; V: the address is a multiple of 16, else of 4
template <bool V>
__device__ __forceinline__ uint4 load16(const void* p) {
  if constexpr (V) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <bool V>
__device__ __forceinline__ void store16(void* p, const uint4& v) {
  if constexpr (V) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    uint32_t* w = reinterpret_cast<uint32_t*>(p);
    w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
  }
}
template <bool V>
__device__ __forceinline__ void load8f(float* f, const bf16* p) {
  const uint4 u = load16<V>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) f[2 * i] = lo2f(w[i]), f[2 * i + 1] = hi2f(w[i]);
}
// a lane's share of a head: elements 8 l .. and HD / 2 + 8 l ..
template <int NP>
struct Head {
  static constexpr int LH = 4 * NP, HALF = 32 * NP;
  float x[16];
  template <bool V>
  __device__ __forceinline__ void load(const bf16* p, int l) {
    load8f<V>(x, p + 8 * l);
    load8f<V>(x + 8, p + HALF + 8 * l);
  }
  template <bool V>
  __device__ __forceinline__ void store(bf16* p, int l) const {
#pragma unroll
    for (int c = 0; c < 16; c += 8)
      store16<V>(p + c / 8 * HALF + 8 * l, make_uint4(pack2f(x[c], x[c + 1]), pack2f(x[c + 2], x[c + 3]), pack2f(x[c + 4], x[c + 5]), pack2f(x[c + 6], x[c + 7])));
  }
  __device__ __forceinline__ void round() {
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const uint32_t p = pack2f(x[i], x[i + 1]);
      x[i] = lo2f(p), x[i + 1] = hi2f(p);
    }
  }
  template <bool V>
  __device__ __forceinline__ void add_bias(const bf16* b, int l) {  // y = bf16(y + b) on the rounded projection output
    Head h;
    h.load<V>(b, l);
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = __fadd_rn(x[i], h.x[i]);
    round();
  }
  // sum of the head's squares: for (stride = hd / 2; stride > 0; stride /= 2) buf[t] += buf[t + stride] for t < stride; every lane of the warp takes part
  __device__ __forceinline__ float squares() const {
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = __fadd_rn(__fmul_rn(x[i], x[i]), __fmul_rn(x[i + 8], x[i + 8]));
#pragma unroll
    for (int m = LH / 2; m >= 1; m >>= 1)
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = __fadd_rn(s[i], __shfl_xor_sync(0xffffffffu, s[i], m));
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1)
#pragma unroll
      for (int i = 0; i < m; ++i) s[i] = __fadd_rn(s[i], s[i + m]);
    return s[0];
  }
  template <bool V>
  __device__ __forceinline__ void norm(float sum, const bf16* w, int l, float eps) {  // qk_norm.cu:46-78 (the division by hd, a power of two, is a product)
    Head h;
    h.load<V>(w, l);
    quot16(x, quot_of(__fsqrt_rn(__fadd_rn(__fmul_rn(sum, 1.f / (64 * NP)), eps))));
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = __fmul_rn(x[i], h.x[i]);
    round();
  }
  template <bool V>
  __device__ __forceinline__ static void load4(float* f, const float* p) {
    const uint4 u = load16<V>(p);
    f[0] = __uint_as_float(u.x), f[1] = __uint_as_float(u.y), f[2] = __uint_as_float(u.z), f[3] = __uint_as_float(u.w);
  }
  template <bool V>
  __device__ __forceinline__ void rope(const float* cos_row, const float* sin_row, int l) {  // RoPE.cu:15-18: pair j is elements 2 j, 2 j + 1
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float co[4], si[4];
      load4<V>(co, cos_row + c * (HALF / 2) + 4 * l);
      load4<V>(si, sin_row + c * (HALF / 2) + 4 * l);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float &x0 = x[8 * c + 2 * i], &x1 = x[8 * c + 2 * i + 1];
        const float v = __fmaf_rn(x0, co[i], -__fmul_rn(x1, si[i]));
        x1 = __fmaf_rn(co[i], x1, __fmul_rn(x0, si[i]));
        x0 = v;
      }
    }
  }
  template <bool V>
  __device__ __forceinline__ void rope_half(const float* cos_row, const float* sin_row, int l) {  // rotate_half: element j pairs with j + hd / 2, table column j
#pragma unroll
    for (int c = 0; c < 8; c += 4) {
      float co[4], si[4];
      load4<V>(co, cos_row + 8 * l + c);
      load4<V>(si, sin_row + 8 * l + c);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float &x0 = x[c + i], &x1 = x[8 + c + i];
        const float v = __fmaf_rn(x0, co[i], -__fmul_rn(x1, si[i]));
        x1 = __fmaf_rn(co[i], x1, __fmul_rn(x0, si[i]));
        x0 = v;
      }
    }
  }
};

}  // namespace qie
