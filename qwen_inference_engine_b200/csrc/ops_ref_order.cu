// ops_ref_order.cu -- the non-GEMM operators of the forward, written so that every
// floating-point result is produced by the same sequence of IEEE operations as the
// reference kernel it replaces (citations relative to the reference's layers/), while
// the work is spread over warps/blocks instead of one thread per token:
//   rmsNorm        src/normalization.cu:5-26   sequential FFMA chain (kept: it IS the spec)
//   qkNorm         src/qk_norm.cu:43-80        shared-memory tree  -> same tree in shuffles
//   RoPE           src/RoPE.cu:6-22            fma(x0,c,-(x1*s)) , fma(c,x1,x0*s)
//   selfattention  src/self_attension.cu:10-149
//   sampling       src/logit_decode.cu:149-274
// This file is compiled with -fmad=false; every fused multiply-add that nvcc's default
// contraction makes of the reference's source expressions is spelled __fmaf_rn here (oracle/fma_contract.cu
// finds the placement from outputs), everything else is an explicit _rn intrinsic.
#include <curand_kernel.h>
#include <math_constants.h>

#include <climits>

#include <algorithm>
#include <type_traits>
#include <map>
#include <mutex>
#include <vector>

#include "cluster.cuh"
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "ref_math.cuh"

namespace qie {

// ------------------------------------------------------------------ embedding
__global__ void embedding_kernel(bf16* __restrict__ out, const bf16* __restrict__ table,
                                 const int* __restrict__ ids, size_t hidden) {
  pdl_wait();
  pdl_trigger();
  const size_t t = blockIdx.x;
  // a sampler that found no finite logit reports -1 (never a valid id); such a row reads row 0 instead of out of bounds
  const bf16* src = table + (size_t)max(ids[t], 0) * hidden;
  bf16* dst = out + t * hidden;
  if ((hidden & 7) == 0) {
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4 = reinterpret_cast<uint4*>(dst);
    for (size_t i = threadIdx.x; i < hidden / 8; i += blockDim.x) d4[i] = s4[i];
  } else {
    for (size_t i = threadIdx.x; i < hidden; i += blockDim.x) dst[i] = src[i];
  }
}

cudaError_t launch_embedding(bf16* out, const bf16* table, const int* ids, size_t hidden, size_t n_tok,
                             cudaStream_t st) {
  if (n_tok == 0) return cudaSuccess;
  return launched(launch_spread<embedding_kernel>(dim3((unsigned)n_tok), dim3(128), 0, st, out, table, ids, hidden));
}

// ------------------------------------------------------------------ a prompt's rows
// The rows of one sequence at consecutive positions: token ids from page-locked memory, positions, slots and the step of the sampled row from arguments; and
// the token back into page-locked memory.  The kernels read and write it across PCIe themselves: copies of four filled arrays in front of a
// forward and one behind it were 4 to 10 us each on the stream (prompts of 512 tokens in reference order 512 -> 494 us).
__global__ void stage_rows_kernel(const volatile int* src, int n, int pos0, int seq, int step, int* __restrict__ ids, int* __restrict__ pos, int* __restrict__ slot,
                                  int* __restrict__ steps) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ids[i] = src[i], pos[i] = pos0 + i, slot[i] = seq;
  if (i == 0) steps[0] = step;
}
__global__ void publish_token_kernel(const int* __restrict__ token, volatile int* dst) {
  pdl_wait();
  pdl_trigger();
  *dst = *token;
}
cudaError_t launch_stage_rows(const int* src, int n, int pos0, int seq, int step, int* ids, int* pos, int* slot, int* steps, cudaStream_t st) {
  return launch_k(stage_rows_kernel, dim3((n + 255) / 256), dim3(256), 0, st, (const volatile int*)src, n, pos0, seq, step, ids, pos, slot, steps);
}
cudaError_t launch_publish_token(const int* token, int* dst, cudaStream_t st) { return launch_k(publish_token_kernel, dim3(1), dim3(1), 0, st, token, (volatile int*)dst); }

// ------------------------------------------------------------------ rmsNorm
// eight elements: RN(x / rms) w, rounded to bf16
__device__ __forceinline__ void norm8(const uint32_t (&x)[4], const uint32_t (&w)[4], const Quot& rms, uint32_t (&o)[4]) {
  float v[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) v[2 * j] = lo2f(x[j]), v[2 * j + 1] = hi2f(x[j]);
  quot16(v, rms);
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j] = pack2f(__fmul_rn(v[2 * j], lo2f(w[j])), __fmul_rn(v[2 * j + 1], hi2f(w[j])));
}

// The reference's sum is a strictly sequential fp32 FFMA chain over the hidden dimension (one thread per token); fp32 addition is not
// associative, so the chain's order is part of the result.  A block takes R rows into shared memory, R lanes of one warp walk a chain each
// side by side, and the block does the rest in parallel.
// What bounds it: the chain, 4 cycles an element (896 wide 1.9 us).  Its loads are 16 bytes and a group of four pieces ahead: single floats read
// inside the loop cost the chain as much again.  us at 1 / 1000 / 4000 rows, before (one row a block, fp32 in shared memory, a division an element) and
// now: 250 wide 2.7 3.3 6.6 and 2.7 3.3 6.7; 896 wide 6.2 6.6 15.7 and 3.8 4.8 9.4; 1536 wide 9.7 10.2 25.3 and 5.3 6.5 13.3; 3584 wide 20.9 21.5 58 and
// 10.1 12.1 26.4.
// VEC: rows (bf16 as they are), weights and results in pieces of 16 bytes.  Other widths and addresses: element by element, one row a block, and the row
// in fp32, so that the chain unpacks nothing: its issue slots bound launches of many rows (1500 rows of 250: 3.9 us, 4.6 from bf16).
// Four rows a block from RMS_MANY rows an SM on (twice as many where a row is narrow): from there more than one chain falls to each of an SM's schedulers,
// and the lanes of one warp share their issue slots.  1 and 4 rows a block, us: 256 wide 1000 rows 2.6 3.2, 1500 3.0 3.3, 2000 4.3 3.4; 640 wide 888 rows 3.9
// 4.2, 1500 5.0 4.5; 896 wide 700 rows 4.6 4.8, 1000 4.8 4.8, 2000 8.6 5.4; 1536 wide 700 rows 6.7 6.6, 1000 7.0 6.6, 2000 13.1 7.3.
constexpr size_t RMS_MANY = 6, RMS_WIDE = 640;
// bytes of a row in shared memory: whole pieces of 16 and one more, so that lanes that walk a row each read different banks
__host__ __device__ inline size_t rms_pitch(size_t hidden, size_t elem) { return ((hidden * elem + 15) / 16 + 1) * 16; }
template <int R, bool VEC>
__global__ void __launch_bounds__(R > 1 ? 256 : 128) rmsnorm_ref_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y, int hidden,
                                                                        size_t x_stride, int n_tok, float eps) {
  static_assert(VEC || R == 1, "one row element by element");
  constexpr int RMS_NT = R > 1 ? 256 : 128;
  using T = std::conditional_t<VEC, bf16, float>;
  constexpr int PIECE = 16 / sizeof(T), GROUP = 4 * PIECE;
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char rms_rows[];
  __shared__ float s_rms[R];
  const int pitch = (int)rms_pitch(hidden, sizeof(T));
  const int row0 = blockIdx.x * R, n = min(R, n_tok - row0), tid = threadIdx.x;
  uint4 w0 = make_uint4(0u, 0u, 0u, 0u);  // this thread's first weights: on their way beside the chain (with four rows the registers would cost a block on the SM)
  if constexpr (VEC) {  // all pieces on their way at once
    const int nv = hidden / 8;
    const uint32_t dst = smem_u32(rms_rows);
    for (int r = 0; r < n; ++r)
      for (int i = tid; i < nv; i += RMS_NT) cp_async16(dst + (uint32_t)(r * pitch + i * 16), x + (size_t)(row0 + r) * x_stride + i * 8);
    cp_async_commit();
    if (R == 1 && tid < nv) w0 = reinterpret_cast<const uint4*>(w)[tid];
    cp_async_wait<0>();
  } else {
    for (int i = tid; i < hidden; i += RMS_NT) reinterpret_cast<float*>(rms_rows)[i] = bf2f(x[(size_t)row0 * x_stride + i]);
  }
  __syncthreads();
  if (tid < n) {
    const uint4* p = reinterpret_cast<const uint4*>(rms_rows + (size_t)tid * pitch);
    float sum = 0.f;
    const int groups = hidden / GROUP, rest = hidden - groups * GROUP;
    uint4 cur[4], nxt[4];
    auto add = [&](const uint4& v, int left) {  // a piece, or the `left` elements that there are of it
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < PIECE; ++j) {
        const float a = !VEC ? __uint_as_float(u[j % 4]) : j & 1 ? hi2f(u[j / 2]) : lo2f(u[j / 2]);
        if (j < left) sum = __fmaf_rn(a, a, sum);
      }
    };
    if (groups > 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) cur[j] = p[j];
    }
#pragma unroll 2
    for (int g = 0; g < groups; ++g) {
      const uint4* q = p + 4 * min(g + 1, groups - 1);
#pragma unroll
      for (int j = 0; j < 4; ++j) nxt[j] = q[j];
#pragma unroll
      for (int j = 0; j < 4; ++j) add(cur[j], PIECE);
#pragma unroll
      for (int j = 0; j < 4; ++j) cur[j] = nxt[j];
    }
    if (rest > 0) {  // up to four more pieces, the last one cut short (never with VEC)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j * PIECE < rest) cur[j] = p[4 * groups + j];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j * PIECE < rest) add(cur[j], VEC ? PIECE : rest - j * PIECE);
    }
    s_rms[tid] = __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)hidden), eps));  // eps 1e-4 in the reference (normalization.cu:9)
  }
  __syncthreads();
  if constexpr (VEC) {
    const int nv = hidden / 8;
    for (int i = tid; i < nv; i += RMS_NT) {
      const uint4 wv = R == 1 && i == tid ? w0 : reinterpret_cast<const uint4*>(w)[i];
      const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r >= n) break;
        const uint4 v = *reinterpret_cast<const uint4*>(rms_rows + (size_t)r * pitch + i * 16);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        uint32_t o[4];
        norm8(u, ww, quot_of(s_rms[r]), o);
        reinterpret_cast<uint4*>(y + (size_t)(row0 + r) * hidden)[i] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  } else {
    const float rms = s_rms[0];
    for (int i = tid; i < hidden; i += RMS_NT)
      y[(size_t)row0 * hidden + i] = f2bf(__fmul_rn(__fdiv_rn(reinterpret_cast<const float*>(rms_rows)[i], rms), bf2f(w[i])));
  }
}

cudaError_t launch_rmsnorm_ref(const bf16* x, const bf16* w, bf16* y, size_t hidden, size_t n_tok, size_t x_stride,
                               cudaStream_t st, float eps) {
  if (n_tok == 0) return cudaSuccess;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const size_t pitch = rms_pitch(hidden, sizeof(bf16)), sms = device_attribute<cudaDevAttrMultiProcessorCount>(dev);
  const bool vec = hidden % 8 == 0 && x_stride % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  if (vec && n_tok >= (hidden < RMS_WIDE ? 2 : 1) * RMS_MANY * sms && 4 * pitch <= 40 * 1024)
    return launched(launch_spread<rmsnorm_ref_kernel<4, true>>(dim3((unsigned)((n_tok + 3) / 4)), dim3(256), 4 * pitch, st, x, w, y, (int)hidden, x_stride, (int)n_tok, eps));
  if (vec)
    return launched(launch_spread<rmsnorm_ref_kernel<1, true>>(dim3((unsigned)n_tok), dim3(128), pitch, st, x, w, y, (int)hidden, x_stride, (int)n_tok, eps));
  static PerDeviceOnce set;  // (12288 elements are a little more than the 48 KB that need no attribute)
  if (set.need()) {
    e = cudaFuncSetAttribute(rmsnorm_ref_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    if (e != cudaSuccess) return e;
    set.done();
  }
  return launched(launch_k(rmsnorm_ref_kernel<1, false>, dim3((unsigned)n_tok), dim3(128), rms_pitch(hidden, sizeof(float)), st, x, w, y, (int)hidden, x_stride, (int)n_tok, eps));
}

// fast-numerics variant: the sum of squares is reduced in parallel (warp shuffles), so it
// differs from the reference's sequential chain in the last fp32 bits.
__global__ void __launch_bounds__(256) rmsnorm_fast_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                            bf16* __restrict__ y, int hidden, size_t x_stride, float eps) {
  pdl_wait();
  pdl_trigger();
  __shared__ float s_part[8];
  const bf16* xr = x + (size_t)blockIdx.x * x_stride;
  bf16* yr = y + (size_t)blockIdx.x * hidden;
  float sum = 0.f;
  for (int i = threadIdx.x * 2; i < hidden; i += 512) {
    uint32_t v = *reinterpret_cast<const uint32_t*>(xr + i);
    float a = lo2f(v), b = hi2f(v);
    sum += a * a + b * b;
  }
  sum = warp_sum(sum);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += s_part[i];
  const float rms = __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)hidden), eps));
  for (int i = threadIdx.x * 2; i < hidden; i += 512) {
    uint32_t v = *reinterpret_cast<const uint32_t*>(xr + i), wv = *reinterpret_cast<const uint32_t*>(w + i);
    *reinterpret_cast<uint32_t*>(yr + i) = pack2(f2bf(__fmul_rn(__fdiv_rn(lo2f(v), rms), lo2f(wv))),
                                                 f2bf(__fmul_rn(__fdiv_rn(hi2f(v), rms), hi2f(wv))));
  }
}
// one WARP per row, 16-byte accesses, no block barrier -- the block-per-row kernel above ran at a quarter of the HBM
// rate on the 4096 rows of a prefill (15.9 us for 25 MB: latency of one tiny block per row); a division an element cost 3 of the 11 us that
// this one then took behind a projection
__global__ void __launch_bounds__(256) rmsnorm_fast_rows_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                                 bf16* __restrict__ y, int hidden, size_t x_stride, float eps,
                                                                 int n_tok) {
  pdl_wait();
  pdl_trigger();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n_tok) return;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * x_stride);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * hidden);
  const int nv = hidden >> 3;
  float sum = 0.f;
  for (int i = lane; i < nv; i += 32) {
    const uint4 v = xr[i];
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = lo2f(u[j]), b = hi2f(u[j]);
      sum += a * a + b * b;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const Quot rms = quot_of(__fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)hidden), eps)));
  for (int i = lane; i < nv; i += 32) {
    const uint4 v = xr[i], wv = wr[i];  // (from L2 where launch_spread's padding leaves L1 less than the SM's rows)
    const uint32_t u[4] = {v.x, v.y, v.z, v.w}, ww[4] = {wv.x, wv.y, wv.z, wv.w};
    uint32_t o4[4];
    norm8(u, ww, rms, o4);
    yr[i] = make_uint4(o4[0], o4[1], o4[2], o4[3]);
  }
}

cudaError_t launch_rmsnorm_fast(const bf16* x, const bf16* w, bf16* y, size_t hidden, size_t n_tok, size_t x_stride,
                                cudaStream_t st, float eps) {
  if (n_tok == 0) return cudaSuccess;
  if (hidden & 1) return cudaErrorInvalidValue;
  // (every row count takes this kernel when the layout allows: a row's result must not depend on how a prompt is chunked)
  if (hidden % 8 == 0 && x_stride % 8 == 0 &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15) == 0) {
    return launched(launch_spread<rmsnorm_fast_rows_kernel>(dim3((unsigned)((n_tok + 7) / 8)), dim3(256), 0, st, x, w, y, (int)hidden, x_stride, eps, (int)n_tok));
  }
  (void)launch_k(rmsnorm_fast_kernel, dim3((unsigned)n_tok), dim3(256), 0, st, x, w, y, (int)hidden, x_stride, eps);
  return cudaGetLastError();
}

// plain K/V scatter (operator-level twin of kv_copy_layer_to_cache_*)
__global__ void kv_store_kernel(KvGeom kv, int layer, const bf16* __restrict__ K, const bf16* __restrict__ V,
                                const int* __restrict__ pos, const int* __restrict__ slot,
                                const int* __restrict__ block_table, int max_pages, int n_tok) {
  pdl_wait();
  pdl_trigger();
  int tok = blockIdx.x;
  int ps = pos[tok];
  int page = block_table[(size_t)slot[tok] * max_pages + ps / kv.page_size];
  int off = ps % kv.page_size;
  int dkv = kv.n_kv * kv.hd;
  for (int i = threadIdx.x; i < dkv; i += blockDim.x) {
    int h = i / kv.hd, d = i % kv.hd;
    kv.chunk(page, layer, 0, h)[(size_t)off * kv.hd + d] = K[(size_t)tok * dkv + i];
    kv.chunk(page, layer, 1, h)[(size_t)off * kv.hd + d] = V[(size_t)tok * dkv + i];
  }
}

cudaError_t launch_kv_store(const KvGeom& kv, int layer, const bf16* K, const bf16* V, const int* pos,
                            const int* slot, const int* block_table, int max_pages, int n_tok, cudaStream_t st) {
  if (n_tok == 0) return cudaSuccess;
  (void)launch_k(kv_store_kernel, dim3(n_tok), dim3(128), 0, st, kv, layer, K, V, pos, slot, block_table, max_pages, n_tok);
  return cudaGetLastError();
}

// K/V rows -> a page list in the reference's layout (kv_copy_layer_to_cache_{prefill,decode}, include_cuda.cu:165-279:
// one cudaMemcpy2D pair per page per layer there; one launch here)
__global__ void kv_store_pagelist_kernel(bf16* const* __restrict__ k_pages, bf16* const* __restrict__ v_pages, int page_size,
                                         int n_layers, int layer, int kv_dim, const bf16* __restrict__ K,
                                         const bf16* __restrict__ V, int pos0, int n_tok) {
  pdl_wait();
  pdl_trigger();
  const int tok = blockIdx.x, pos = pos0 + tok;
  const size_t off = ((size_t)(pos % page_size) * n_layers + layer) * kv_dim;
  bf16* kd = k_pages[pos / page_size] + off;
  bf16* vd = v_pages[pos / page_size] + off;
  for (int i = threadIdx.x; i < kv_dim; i += blockDim.x) {
    kd[i] = K[(size_t)tok * kv_dim + i];
    vd[i] = V[(size_t)tok * kv_dim + i];
  }
}
cudaError_t launch_kv_store_pagelist(bf16* const* k_pages, bf16* const* v_pages, int page_size, int n_layers, int layer, int kv_dim,
                                     const bf16* K, const bf16* V, int pos0, int n_tok, cudaStream_t st) {
  if (n_tok == 0) return cudaSuccess;
  (void)launch_k(kv_store_pagelist_kernel, dim3(n_tok), dim3(128), 0, st, k_pages, v_pages, page_size, n_layers, layer, kv_dim, K, V, pos0, n_tok);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ elementwise
__global__ void silu_kernel(bf16* x, size_t n) {
  pdl_wait();
  pdl_trigger();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    float v = bf2f(x[i]);
    float sg = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-v)));
    x[i] = f2bf(__fmul_rn(v, sg));
  }
}
__global__ void elem_mul_kernel(const bf16* a, const bf16* b, bf16* c, size_t n) {
  pdl_wait();
  pdl_trigger();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) c[i] = f2bf(__fmul_rn(bf2f(a[i]), bf2f(b[i])));
}
__global__ void residual_add_kernel(bf16* a, const bf16* b, size_t n) {
  pdl_wait();
  pdl_trigger();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = f2bf(__fadd_rn(bf2f(a[i]), bf2f(b[i])));
}
cudaError_t launch_silu(bf16* x, size_t n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  (void)launch_k(silu_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, x, n);
  return cudaGetLastError();
}
cudaError_t launch_elem_mul(const bf16* a, const bf16* b, bf16* c, size_t n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  (void)launch_k(elem_mul_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, a, b, c, n);
  return cudaGetLastError();
}
cudaError_t launch_residual_add(bf16* a, const bf16* b, size_t n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  (void)launch_k(residual_add_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, a, b, n);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ attention
// What attn_ref_rows.cu does not take.  grid (q head, token); 256 threads.  Phase 1: one warp per kv position computes the
// score with the reference's 2^k tree over head_dim.  Phase 2: max (order free), expf,
// the reference's sequential sum, p = e/sum.  Phase 3: thread d accumulates
// out[d] = fma(p[k], v[k][d], out[d]) for k ascending (self_attension.cu:112-137).
// Positions > pos[t] contribute exact zeros in the reference (mask -1e9 -> expf = 0 ->
// fma(0, v, o) = o), so stopping at pos[t] is bit-identical.
template <int NP, bool PL>  // PL: page-list addressing (the reference's cache layout)
__global__ void __launch_bounds__(256) attention_ref_kernel(AttnArgs a) {
  pdl_wait();
  pdl_trigger();
  constexpr int hd = 64 * NP;
  extern __shared__ float sm[];
  float* score = sm;                                                   // [kv_len]
  int* pages = reinterpret_cast<int*>(sm + a.max_kv_len);              // [pages used]
  __shared__ float s_red[8];
  __shared__ float s_bcast;

  const int h = blockIdx.x, tok = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (a.tile_rows) {
    const int r0 = tok / a.tile_rows * a.tile_rows, r1 = min(r0 + a.tile_rows, a.n_tok);
    bool one = true;
    for (int i = r0 + 1; i < r1; ++i) one = one && a.slot[i] == a.slot[r0];
    if (one) return;  // attention_ref_rows_kernel has done this row
  }
  const int kv_len = a.pos[tok] + 1;
  const int group = a.n_q / a.kv.n_kv;
  const int kvh = h / group;
  const int psz = a.kv.page_size;
  const int n_pages = (kv_len + psz - 1) / psz;
  if (!PL) {
    const int* bt = a.block_table + (size_t)a.slot[tok] * a.max_pages;
    for (int i = threadIdx.x; i < n_pages; i += blockDim.x) pages[i] = bt[i];
  }
  // row of cache position k: pool chunk [slot][hd], or the reference's page [slot][layer][kv_dim]
  const size_t pl_row = (size_t)a.pl_layers * a.kv.n_kv * hd, pl_off = (size_t)a.layer * a.kv.n_kv * hd + (size_t)kvh * hd;
  auto k_row = [&](int k) -> const bf16* {
    return PL ? a.k_pages[k / psz] + (size_t)(k % psz) * pl_row + pl_off : a.kv.chunk(pages[k / psz], a.layer, 0, kvh) + (size_t)(k % psz) * hd;
  };
  auto v_row = [&](int k) -> const bf16* {
    return PL ? a.v_pages[k / psz] + (size_t)(k % psz) * pl_row + pl_off : a.kv.chunk(pages[k / psz], a.layer, 1, kvh) + (size_t)(k % psz) * hd;
  };

  float q[NP][2];
  head_load<NP>(q, a.q + (size_t)tok * a.n_q * hd + (size_t)h * hd, lane);
  __syncthreads();

  const float inv_den = __fsqrt_rn((float)hd);
  for (int k = warp; k < kv_len; k += 8) {
    const bf16* kp = k_row(k);
    float pr[NP][2];
    head_load<NP>(pr, kp, lane);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      pr[p][0] = __fmul_rn(q[p][0], pr[p][0]);
      pr[p][1] = __fmul_rn(q[p][1], pr[p][1]);
    }
    float dot = head_tree_sum<NP>(pr);
    if (lane == 0) score[k] = __fdiv_rn(dot, inv_den);
  }
  __syncthreads();

  // max
  float m = -1e9f;
  for (int k = threadIdx.x; k < kv_len; k += blockDim.x) m = fmaxf(m, score[k]);
  m = warp_max(m);
  if (lane == 0) s_red[warp] = m;
  __syncthreads();
  m = s_red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) m = fmaxf(m, s_red[i]);
  for (int k = threadIdx.x; k < kv_len; k += blockDim.x) score[k] = expf(__fsub_rn(score[k], m));
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.f;
    int k = 0;
    for (; k + 8 <= kv_len; k += 8) {
      float e0 = score[k], e1 = score[k + 1], e2 = score[k + 2], e3 = score[k + 3];
      float e4 = score[k + 4], e5 = score[k + 5], e6 = score[k + 6], e7 = score[k + 7];
      sum = __fadd_rn(sum, e0);
      sum = __fadd_rn(sum, e1);
      sum = __fadd_rn(sum, e2);
      sum = __fadd_rn(sum, e3);
      sum = __fadd_rn(sum, e4);
      sum = __fadd_rn(sum, e5);
      sum = __fadd_rn(sum, e6);
      sum = __fadd_rn(sum, e7);
    }
    for (; k < kv_len; ++k) sum = __fadd_rn(sum, score[k]);
    s_bcast = sum;
  }
  __syncthreads();
  const float sum = s_bcast;
  for (int k = threadIdx.x; k < kv_len; k += blockDim.x) score[k] = __fdiv_rn(score[k], sum);
  __syncthreads();

  if (threadIdx.x < hd) {
    const int d = threadIdx.x;
    float o = 0.f;
    int k = 0;
    for (; k + 4 <= kv_len; k += 4) {
      float v0 = bf2f(v_row(k)[d]);
      float v1 = bf2f(v_row(k + 1)[d]);
      float v2 = bf2f(v_row(k + 2)[d]);
      float v3 = bf2f(v_row(k + 3)[d]);
      o = __fmaf_rn(score[k], v0, o);
      o = __fmaf_rn(score[k + 1], v1, o);
      o = __fmaf_rn(score[k + 2], v2, o);
      o = __fmaf_rn(score[k + 3], v3, o);
    }
    for (; k < kv_len; ++k) o = __fmaf_rn(score[k], bf2f(v_row(k)[d]), o);
    a.out[(size_t)tok * a.n_q * hd + (size_t)h * hd + d] = f2bf(o);
  }
}

cudaError_t launch_attention_ref(const AttnRefCall& args, cudaStream_t st) {
  if (args.n_tok == 0) return cudaSuccess;
  AttnArgs a = args;
  if (a.kv.hd == 64 || a.kv.hd == 128 || a.kv.hd == 256) {
    int dev = 0, sms = 0, vr = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // Rows of their own, also those of a short prompt: rows, kv heads and parts of a kv head's heads that fill the SMs once are quicker there from 17 positions on
    // (us, attention_ref_rows_kernel and here, 14 heads of 64 on 2: 1 row at 301 positions 14.3 7.9, at 2001 60 24, 32 rows behind 300 15.6 9.1, 64 behind 2000
    // 63 35; 17 rows of a prompt 5.8 5.4; up to 16 positions one block per row and head, 3.5 4.5).  More rows than that share their keys and values here in tiles of several rows,
    // which is worth more the shorter the context: w waves are quicker above 160 w positions with all of six to eight heads in a CTA (96 rows behind 120 15.6 15.1, behind 50
    // 12.5 13.5; 200 behind 300 41 33; 180 behind 300 40 32).  Tiles of several rows with heads of 64: above 250 w (14 heads on 2, 400 rows behind 800 109 115, behind 600 90 97; 8 heads
    // on 1, 640 behind 400 69 80).  Three and more waves of rows on a single kv head, whose keys and values are few: above 180 w (8 heads, 300 behind 200 28.2 30.0, 360 behind 200
    // 35.9 34.3).  A part of a kv head's heads in a CTA: above 225 w (16 heads on 1, 200 behind 2000 166 108, 300 behind 800 90 93), four and more waves of such rows that the tiles take at
    // once above 300 w (240 behind 900 71 80).  One wave above 32 (24 rows of a prompt, 28 heads of 128 on 4 6.7 7.7).  Over 4680 sizes (twelve pairs of head counts, 17 to 700 rows behind 0 to
    // 1500 positions) what is taken is at most 2.7 % slower so, 16 % with 160 w and 225 w alone.  Operator calls with tables beyond attention_ref_rows_kernel's sizes stay with the
    // kernel below.
    int stages = 0;
    const int heads = attention_ref_decode_heads(a, sms, &stages);
    a.tile_rows = attention_ref_tile_rows(a, sms, &vr);
    if (heads) {
      const int G = a.n_q / a.kv.n_kv;
      const long ctas = (long)a.n_tok * a.kv.n_kv * ((G + heads - 1) / heads), waves = (ctas + sms - 1) / sms;
      const auto positions = [&]() -> long {  // from where on rows on their own are quicker than tiles
        if (waves == 1) return heads < 6 ? 0 : 33;
        if (heads < 6) return LONG_MAX;
        if (heads < G) return (waves > 3 && (long)((a.n_tok + a.tile_rows - 1) / a.tile_rows) * a.kv.n_kv <= 2 * sms ? 300 : 225) * waves;
        if (a.kv.hd == 64 && a.tile_rows > 1) return 250 * waves;
        return (a.kv.hd == 64 && a.kv.n_kv == 1 && waves > 2 ? 180 : 160) * waves;
      };
      if (args.decode ? attention_ref_decode_step(a, sms, heads) : a.tile_rows && a.max_kv_len >= positions()) return launch_attention_ref_decode(args, heads, stages, st);
    }
    if (a.tile_rows) {  // (a tile of one row is one sequence's whatever the rows are)
      e = launch_attention_ref_rows(a, a.tile_rows, vr, st);
      if (e != cudaSuccess || a.one_seq || a.tile_rows == 1) return e;
    }
  }
  int max_pages_used = (a.max_kv_len + a.kv.page_size - 1) / a.kv.page_size;
  size_t smem = (size_t)a.max_kv_len * sizeof(float) + (size_t)max_pages_used * sizeof(int);
  dim3 grid(a.n_q, a.n_tok);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
#define QIE_ATTN(NPV)                                                                                              \
  {                                                                                                                \
    /* per-device opt-in to > 48 KiB of dynamic shared memory: set on every launch (cheap), not once per process */ \
    if (a.k_pages) {                                                                                               \
      cudaError_t e = cudaFuncSetAttribute(attention_ref_kernel<NPV, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); \
      if (e != cudaSuccess) return e;                                                                              \
      (void)launch_k(attention_ref_kernel<NPV, true>, dim3(grid), dim3(256), smem, st, a);                          \
    } else {                                                                                                       \
      cudaError_t e = cudaFuncSetAttribute(attention_ref_kernel<NPV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); \
      if (e != cudaSuccess) return e;                                                                              \
      (void)launch_k(attention_ref_kernel<NPV, false>, dim3(grid), dim3(256), smem, st, a);                         \
    }                                                                                                              \
  }
  switch (a.kv.hd) {
    case 64: QIE_ATTN(1); break;
    case 128: QIE_ATTN(2); break;
    case 256: QIE_ATTN(4); break;
    default: return cudaErrorInvalidValue;
  }
#undef QIE_ATTN
  return cudaGetLastError();
}

// ------------------------------------------------------------------ sampling
// The reference runs ONE block of 256 threads and, for each of k rounds, a strided scan
// + shared-memory arg-max whose tie-break is a function of (idx & 255):
// value, then the larger bit-reversed low byte of idx, then the lower idx.  That is a
// total order, so the scan can use any number of threads and still pick the same token.
__global__ void __launch_bounds__(1024) sample_topk_kernel(const bf16* __restrict__ logits, int* __restrict__ out,
                                                            size_t vocab, float temperature, int k, uint64_t seed,
                                                            uint64_t seed_stride, const int* __restrict__ step_ptr,
                                                            unsigned long long subsequence) {
  pdl_wait();
  pdl_trigger();
  __shared__ float topk_vals[256];
  __shared__ int topk_idxs[256];
  __shared__ Cand s_c[32];
  const bf16* row = logits + (size_t)blockIdx.x * vocab;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (k <= 0) {
    if (tid == 0) out[blockIdx.x] = -1;
    return;
  }
  k = min(k, (int)min(vocab, (size_t)256));
  if (!(temperature > 0.0f)) temperature = 1.0f;
  if (tid < 256) {
    topk_vals[tid] = -CUDART_INF_F;
    topk_idxs[tid] = -1;
  }
  __syncthreads();
  for (int sel = 0; sel < k; ++sel) {
    float bv = -CUDART_INF_F;
    int bi = -1;
    for (size_t idx = tid; idx < vocab; idx += blockDim.x) {
      float v = bf2f(row[idx]);
      if (!(v > -CUDART_INF_F)) continue;  // -inf / NaN are never selected (v > local.val fails)
      bool chosen = false;
      for (int t = 0; t < sel; ++t)
        if ((int)idx == topk_idxs[t]) {
          chosen = true;
          break;
        }
      if (!chosen && cand_better(v, (int)idx, bv, bi)) {
        bv = v;
        bi = (int)idx;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (cand_better(ov, oi, bv, bi)) {
        bv = ov;
        bi = oi;
      }
    }
    if (lane == 0) {
      s_c[warp].val = bv;
      s_c[warp].idx = bi;
    }
    __syncthreads();
    if (warp == 0) {
      bv = lane < (blockDim.x >> 5) ? s_c[lane].val : -CUDART_INF_F;
      bi = lane < (blockDim.x >> 5) ? s_c[lane].idx : -1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (cand_better(ov, oi, bv, bi)) {
          bv = ov;
          bi = oi;
        }
      }
      if (lane == 0) {
        topk_vals[sel] = bi >= 0 ? bv : -CUDART_INF_F;
        topk_idxs[sel] = bi;
      }
    }
    __syncthreads();
    if (topk_idxs[sel] == -1) break;
  }
  if (tid == 0) {
    int actual_k = 0;
    for (int i = 0; i < k; ++i) {
      if (topk_idxs[i] != -1)
        actual_k++;
      else
        break;
    }
    if (actual_k == 0) {
      out[blockIdx.x] = -1;
      return;
    }
    if (actual_k == 1) {  // softmax over one candidate is 1; u in (0,1] always selects it
      out[blockIdx.x] = topk_idxs[0];
      return;
    }
    float max_val = __fdiv_rn(topk_vals[0], temperature);
    for (int i = 1; i < actual_k; ++i) {
      float v = __fdiv_rn(topk_vals[i], temperature);
      if (v > max_val) max_val = v;
      topk_vals[i] = v;
    }
    topk_vals[0] = __fdiv_rn(topk_vals[0], temperature);
    float sum = 0.0f;
    for (int i = 0; i < actual_k; ++i) {
      topk_vals[i] = expf(__fsub_rn(topk_vals[i], max_val));
      sum = __fadd_rn(sum, topk_vals[i]);
    }
    curandState rng;
    unsigned long long sd = seed + (unsigned long long)blockIdx.x * seed_stride + (step_ptr ? (unsigned)step_ptr[blockIdx.x] : 0u);
    curand_init(sd, subsequence, 0, &rng);  // logit_decode.cu:256-257: (seed, subsequence, offset 0)
    float u = __fmul_rn(curand_uniform(&rng), sum);
    float cum = 0.0f;
    int picked = topk_idxs[actual_k - 1];
    for (int i = 0; i < actual_k; ++i) {
      cum = __fadd_rn(cum, topk_vals[i]);
      if (u <= cum) {
        picked = topk_idxs[i];
        break;
      }
    }
    out[blockIdx.x] = picked;
  }
}

// Greedy mode (k == 1, what the persistent kernel folds into its lm_head epilogue): the sampled token is the
// arg-max in the reference's total order whatever the random draw, so the row can be scanned by several CTAs with
// 16-byte loads -- the one-block-per-row scan above is latency bound (85 us for 152 k logits, 64 SMs busy at batch
// 64).  Stage 1: CTA (slice, row) reduces its slice to one candidate; stage 2: one warp per row merges the slices.
// Eight logits are one packed maximum, looked at further only where it reaches the thread's best, and few long rows are cut into more slices: one row
// of 151936 behind lm_head 22 us with 8 slices and a comparison in the full order for each, 4.2 now (alone 10.5 and 4.1); 16 rows 12.4 and 5.3, 64 rows 16.7
// and 9.4.  Below 65536 logits 8 slices hold few pieces a thread as they are (32000: 4.8 and 3.7).  Vocabularies of 65536 to 262144, 1 to 256 rows: 0.28 to 0.73
// of the time of 8 slices read value by value, 17 to 48 rows, which keep 8 slices, 0.44 to 0.71.
constexpr int GREEDY_SLICES = 8, GREEDY_MOST = 64;
static int greedy_slices(int n_rows, size_t vocab) { return vocab < 65536 || n_rows > 16 ? GREEDY_SLICES : n_rows > 4 ? 32 : GREEDY_MOST; }
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {  // two bf16 each; a number wins over a NaN
  uint32_t d;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__global__ void __launch_bounds__(256) greedy_slice_kernel(const bf16* __restrict__ logits, Cand* __restrict__ cands, size_t vocab) {
  pdl_wait();
  pdl_trigger();
  __shared__ Cand s_c[8];
  const int slice = blockIdx.x, rowi = blockIdx.y;
  const bf16* row = logits + (size_t)rowi * vocab;
  const size_t nvec = vocab >> 3;  // 8 logits per 16-byte load (rows are 16-byte aligned: vocab % 8 == 0, checked by the launcher)
  const size_t per = (nvec + gridDim.x - 1) / gridDim.x;
  const size_t v0 = (size_t)slice * per, v1 = min(nvec, v0 + per);
  float bv = -CUDART_INF_F;
  int bi = -1;
  constexpr int U = 4;  // loads on their way together
  for (size_t v = v0 + threadIdx.x; v < v1; v += U * 256) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = ld_nc_v4(reinterpret_cast<const uint4*>(row) + min(v + u * 256, v1 - 1));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t w[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
      const uint32_t m = max2(max2(w[0], w[1]), max2(w[2], w[3]));
      const float f = fmaxf(lo2f(m), hi2f(m));
      if (!(v + u * 256 < v1 && f >= bv && f > -CUDART_INF_F)) continue;  // (maxima that are NaN or -inf fail)
      // of those that equal it the first in the reference's order, the largest reversed low bits: 7, 3, 5, 1, 6, 2, 4, 0
      int e = 0;
      if (lo2f(w[2]) == f) e = 4;
      if (lo2f(w[1]) == f) e = 2;
      if (lo2f(w[3]) == f) e = 6;
      if (hi2f(w[0]) == f) e = 1;
      if (hi2f(w[2]) == f) e = 5;
      if (hi2f(w[1]) == f) e = 3;
      if (hi2f(w[3]) == f) e = 7;
      const int i = (int)(v + u * 256) * 8 + e;
      if (cand_better(f, i, bv, bi)) bv = f, bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (cand_better(ov, oi, bv, bi)) bv = ov, bi = oi;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_c[warp] = Cand{bv, bi};
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w2 = 1; w2 < 8; ++w2)
      if (cand_better(s_c[w2].val, s_c[w2].idx, bv, bi)) bv = s_c[w2].val, bi = s_c[w2].idx;
    cands[(size_t)rowi * gridDim.x + slice] = Cand{bv, bi};
  }
}
__global__ void greedy_merge_kernel(const Cand* __restrict__ cands, int* __restrict__ out, int n_rows, int slices) {  // a warp per row
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (r >= n_rows) return;
  float bv = -CUDART_INF_F;
  int bi = -1;
  for (int s2 = lane; s2 < slices; s2 += 32) {
    const Cand c = cands[(size_t)r * slices + s2];
    if (cand_better(c.val, c.idx, bv, bi)) bv = c.val, bi = c.idx;
  }
  for (int o = slices >= 32 ? 16 : 4; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (cand_better(ov, oi, bv, bi)) bv = ov, bi = oi;
  }
  if (lane == 0) out[r] = bi;  // -1 if the row holds no finite logit, like the scan above
}

// Top-k (k > 1) without k scans.  The reference selects by k rounds of "arg-max over everything not chosen yet"
// (logit_decode.cu:182-223), i.e. the k best elements of the row in its total order -- value, then the larger
// bit-reversed low byte of the index, then the lower index (cand_better) -- best first.  That order is the numeric
// order of a 48-bit key [16: order-preserving bf16][8: brev(idx & 255)][24: 0xFFFFFF - idx], all keys distinct, so the
// k-th best key is found by a radix select: six 8-bit digits from the top, one 256-bin shared-memory histogram pass
// over the row per digit (the row is 300 KB and stays in L2), then one pass collects the k keys >= the threshold, a
// bitonic sort orders them, and thread 0 runs the reference's tail (temperature, softmax over k, XORWOW draw, CDF
// scan) unchanged.  7 passes instead of k = 50 (x exclusion-list checks); one block per row.  What the cluster kernel below does not take.
__device__ __forceinline__ unsigned long long topk_key(uint16_t bits, int idx) {
  if (bits == 0x8000u) bits = 0;  // -0.0 == +0.0 in the reference's float compares
  const uint32_t v16 = (bits & 0x8000u) ? (uint32_t)(uint16_t)~bits : (uint32_t)(bits | 0x8000u);
  const uint32_t rev = __brev((unsigned)idx << 24);  // brev of the low byte, in the low byte
  return ((unsigned long long)v16 << 32) | ((unsigned long long)rev << 24) | (unsigned long long)(0xFFFFFFu - (unsigned)idx);
}
__device__ __forceinline__ bool topk_valid(uint16_t b) {  // -inf and NaN are never selected (the reference's v > best fails for both)
  const uint16_t a = b & 0x7fffu;
  return !(a > 0x7f80u) && b != 0xff80u;
}
__global__ void __launch_bounds__(1024) sample_topk_select_kernel(const bf16* __restrict__ logits, int* __restrict__ out, size_t vocab,
                                                                    float temperature, int k, uint64_t seed, uint64_t seed_stride,
                                                                    const int* __restrict__ step_ptr, unsigned long long subsequence) {
  pdl_wait();
  pdl_trigger();
  const int rowi = blockIdx.x;
  __shared__ unsigned hist[256];
  __shared__ unsigned long long sel[256];  // the selected keys, then sorted best first
  __shared__ float topk_vals[256];
  __shared__ int topk_idxs[256];
  __shared__ unsigned long long s_prefix;
  __shared__ int s_need, s_count;
  const uint16_t* row = reinterpret_cast<const uint16_t*>(logits) + (size_t)rowi * vocab;
  const int tid = threadIdx.x;
  if (!(temperature > 0.0f)) temperature = 1.0f;
  k = min(k, (int)min(vocab, (size_t)256));
  // how many candidates exist at all
  unsigned mine = 0;
  for (size_t i = tid; i < vocab; i += blockDim.x) mine += topk_valid(row[i]) ? 1u : 0u;
  if (tid == 0) s_count = 0;
  __syncthreads();
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((tid & 31) == 0 && mine) atomicAdd(&s_count, (int)mine);
  __syncthreads();
  const int actual_k = min(k, s_count);
  if (actual_k <= 0) {
    if (tid == 0) out[rowi] = -1;
    return;
  }
  if (tid == 0) {
    s_prefix = 0ull;
    s_need = actual_k;
  }
  // ---- radix select of the actual_k-th largest key
  for (int d = 5; d >= 0; --d) {
    if (tid < 256) hist[tid] = 0u;
    __syncthreads();
    const unsigned long long prefix = s_prefix;
    const int shift = 8 * d;
    for (size_t i = tid; i < vocab; i += blockDim.x) {
      const uint16_t b = row[i];
      if (!topk_valid(b)) continue;
      const unsigned long long key = topk_key(b, (int)i);
      if (d == 5 || (key >> (shift + 8)) == (prefix >> (shift + 8))) atomicAdd(&hist[(unsigned)(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid == 0) {
      int need = s_need, dig = 255;
      for (; dig > 0; --dig) {  // digits above the threshold digit are taken whole
        if ((int)hist[dig] >= need) break;
        need -= (int)hist[dig];
      }
      s_prefix = prefix | ((unsigned long long)dig << shift);
      s_need = need;
    }
    __syncthreads();
  }
  // ---- collect the keys >= threshold (exactly actual_k: keys are distinct)
  const unsigned long long thr = s_prefix;
  if (tid == 0) s_count = 0;
  if (tid < 256) sel[tid] = 0ull;
  __syncthreads();
  for (size_t i = tid; i < vocab; i += blockDim.x) {
    const uint16_t b = row[i];
    if (!topk_valid(b)) continue;
    const unsigned long long key = topk_key(b, (int)i);
    if (key >= thr) {
      const int slot = atomicAdd(&s_count, 1);
      if (slot < 256) sel[slot] = key;
    }
  }
  __syncthreads();
  // ---- bitonic sort of 256 keys, descending (empty slots are 0 = below every real key)
  for (int size = 2; size <= 256; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (tid < 128) {
        const int lo = 2 * tid - (tid & (stride - 1));
        const int hi = lo + stride;
        const bool desc = (lo & size) == 0;
        const unsigned long long a = sel[lo], b2 = sel[hi];
        if ((a < b2) == desc) {
          sel[lo] = b2;
          sel[hi] = a;
        }
      }
      __syncthreads();
    }
  if (tid < actual_k) {
    const int idx = (int)(0xFFFFFFu - (unsigned)(sel[tid] & 0xFFFFFFull));
    topk_idxs[tid] = idx;
    topk_vals[tid] = bf2f(logits[(size_t)rowi * vocab + idx]);
  }
  __syncthreads();
  if (tid == 0) {  // the reference's tail, logit_decode.cu:225-273 (as in sample_topk_kernel)
    if (actual_k == 1) {
      out[rowi] = topk_idxs[0];
      return;
    }
    float max_val = __fdiv_rn(topk_vals[0], temperature);
    for (int i = 1; i < actual_k; ++i) {
      float v = __fdiv_rn(topk_vals[i], temperature);
      if (v > max_val) max_val = v;
      topk_vals[i] = v;
    }
    topk_vals[0] = __fdiv_rn(topk_vals[0], temperature);
    float sum = 0.0f;
    for (int i = 0; i < actual_k; ++i) {
      topk_vals[i] = expf(__fsub_rn(topk_vals[i], max_val));
      sum = __fadd_rn(sum, topk_vals[i]);
    }
    curandState rng;
    unsigned long long sd = seed + (unsigned long long)rowi * seed_stride + (step_ptr ? (unsigned)step_ptr[rowi] : 0u);
    curand_init(sd, subsequence, 0, &rng);
    float u = __fmul_rn(curand_uniform(&rng), sum);
    float cum = 0.0f;
    int picked = topk_idxs[actual_k - 1];
    for (int i = 0; i < actual_k; ++i) {
      cum = __fadd_rn(cum, topk_vals[i]);
      if (u <= cum) {
        picked = topk_idxs[i];
        break;
      }
    }
    out[rowi] = picked;
  }
}

// 1 < k <= TC_MOST: a cluster of 8, 4 or 2 CTAs per row, each over its part of the row, 16 bytes a load.  The k-th largest of the threads' maxima is a
// bound that at least k values of the slice reach; the values that reach it (about 1.1 k of them) are the slice's candidates.  The first
// CTA gathers the candidates of all slices through distributed shared memory, finds the k-th value by bisection over its 16 bits,
// ranks what is left by counting (all keys differ) and runs the reference's tail: quotients and exponentials by a thread each, the
// two sums in the reference's order.  Where ties (a row of equal logits) leave more candidates than the lists hold, the slice takes four more
// passes to pick its k best, and the first CTA bisects the lower half of the keys.
// One block per row read the row eight times, two bytes a load: k = 50 of 151936, 1 row 369 us, 64 rows 384.  The cluster with both passes over memory,
// every value brought into its order and the gathering CTA by CTA: 18.2 and 39.2.  Now a piece of eight values is one packed maximum and the second pass
// looks into those that reach the bound (a few per cent), the slice is read from memory once, all counts and then all candidates are
// gathered at once, and the draw is compared with the running sums of the one chain: 13.8 and 25.1, with clusters of two for
// many rows 19.4.  The bound is the latency of the steps, not memory (19 MB).  Greedy (k = 1) stays with the two kernels above: 64 rows 9.4 us.
constexpr int TC_CTAS = 8, TC_CAP = 512, TC_MOST = 128;  // TC_CTAS: the largest cluster
// order-preserving 16 bits; 0: never selected
__device__ __forceinline__ uint32_t topk_order16(uint32_t b) {
  if (!topk_valid((uint16_t)b)) return 0u;
  if (b == 0x8000u) b = 0;  // -0.0 == +0.0
  return (b & 0x8000u) ? (uint32_t)(uint16_t)~b : (b | 0x8000u);
}
template <int TC_THREADS>
struct TopkSlice {  // elements in front of the first 16-byte boundary and behind the last whole piece belong to the first slice
  const uint16_t* row;
  size_t v0, v1;
  int head, tail0, loose;
  template <class F>
  __device__ __forceinline__ void each(F&& f) const {  // f(order16, bits, index) for this thread's share of the slice
    const int tid = threadIdx.x;
    constexpr int U = 4;  // loads on their way together, whatever the compiler makes of the loop
    for (size_t v = v0 + tid; v < v1; v += U * TC_THREADS) {
      uint32_t w[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint16_t* p = row + head + min(v + u * TC_THREADS, v1 - 1) * 8;
        asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[u][0]), "=r"(w[u][1]), "=r"(w[u][2]), "=r"(w[u][3]) : "l"(p));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i0 = head + (int)(v + u * TC_THREADS) * 8;
        if (v + u * TC_THREADS < v1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            f(topk_order16(w[u][e] & 0xffffu), w[u][e] & 0xffffu, i0 + 2 * e);
            f(topk_order16(w[u][e] >> 16), w[u][e] >> 16, i0 + 2 * e + 1);
          }
        }
      }
    }
    if (tid < loose) {
      const int i = tid < head ? tid : tail0 + tid - head;
      f(topk_order16(row[i]), (uint32_t)row[i], i);
    }
  }
};
// Every thread's c summed up, one barrier a sum: three counters in turn, the next one cleared in front of the barrier behind which it is added to and
// after all have read what it held.  They start at zero.
struct TopkSums {
  int* cnt;
  int at;
  __device__ __forceinline__ int operator()(int c) {
    const int next = at == 2 ? 0 : at + 1;
    if (threadIdx.x == 0) cnt[next] = 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&cnt[at], c);
    __syncthreads();
    c = cnt[at];
    at = next;
    return c;
  }
};
// Exactly k of a slice of which more than TC_CAP values reach `bound`.  v: the value that the slice's k-th has (the bound itself, unless many large
// values share few threads); of those that equal it the best by the key's lower half: bit-reversed low byte of the index, largest first, then index.
// cls: 256 ints (ties by low byte); tie: indices of one low byte (topk_tie_ints).  Not inlined: beside the kernel's own passes its copies of the loop
// cost those 15 %.
// What `tie` has to hold: a slice is ceil(vocab / 8 / ctas) pieces side by side, of which every 256 consecutive elements hold one of a low byte, and in the first
// slice up to 14 elements more in front of the first and behind the last whole piece of the row: two runs, each with at most one more of the byte.
constexpr size_t topk_tie_ints(size_t vocab, int ctas) { return ((vocab / 8 + ctas - 1) / ctas * 8 + 255) / 256 + 2; }
template <int TC_THREADS>
__device__ __noinline__ void topk_slice_ties(const TopkSlice<TC_THREADS> sl, TopkSums sum, uint32_t mx, uint32_t bound, int k, unsigned long long* cand, int* cls,
                                              int* tie, int* s_n, int* s_tot) {
  const int tid = threadIdx.x;
  auto count = [&](uint32_t t) {  // values that reach t
    int c = 0;
    if (mx >= t) sl.each([&](uint32_t o, uint32_t, int) { c += o >= t; });
    return sum(c);
  };
  uint32_t v = bound;
  int above = count(v + 1);
  if (above >= k) {
    v = 0;
#pragma unroll 1
    for (int bit = 15; bit >= 0; --bit)
      if (count(v | (1u << bit)) >= k) v |= 1u << bit;
    above = count(v + 1);
  }
  int need = k - above;
  if (tid < 256) cls[tid] = 0;
  __syncthreads();
  if (mx >= v) sl.each([&](uint32_t o, uint32_t, int i) { if (o == v) atomicAdd(&cls[i & 255], 1); });
  __syncthreads();
  const int mine = tid < 256 ? cls[__brev((uint32_t)tid << 24)] : 0;  // thread = reversed byte
  uint32_t rv = 0;  // the reversed byte in which the last needed tie lies
#pragma unroll 1
  for (int bit = 7; bit >= 0; --bit)
    if (sum(tid >= (int)(rv | (1u << bit)) ? mine : 0) >= need) rv |= 1u << bit;
  need -= sum(tid > (int)rv ? mine : 0);
  const int byte = (int)__brev(rv << 24);
  if (tid == 0) *s_n = 0;
  __syncthreads();
  if (mx >= v) sl.each([&](uint32_t o, uint32_t, int i) { if (o == v && (i & 255) == byte) tie[atomicAdd(s_n, 1)] = i; });
  __syncthreads();
  const int n_tie = *s_n;
  for (int i = tid; i < n_tie; i += TC_THREADS) {
    int before = 0;
    for (int j = 0; j < n_tie; ++j) before += tie[j] < tie[i];
    if (before == need - 1) *s_tot = tie[i];
  }
  __syncthreads();
  const int last = *s_tot;
  if (tid == 0) *s_n = 0;
  __syncthreads();
  if (mx >= v)
    sl.each([&](uint32_t o, uint32_t b, int i) {
      const uint32_t r = __brev((uint32_t)i << 24);
      if (o > v || (o == v && (r > rv || (r == rv && i <= last)))) cand[atomicAdd(s_n, 1)] = topk_key((uint16_t)b, i);
    });
  __syncthreads();
  if (tid < 3) sum.cnt[tid] = 0;
}
// STAGED: the slice is copied to shared memory once, its two passes read it there; the first CTA's gathered candidates go over it.  In clusters of 8 up
// to TC_STAGE bytes, 48 KB with the 9.6 KB of the rest, so that four CTAs share an SM; in clusters of 4 and 2 twice and four times that, two CTAs and one.
constexpr int TC_STAGE = 38 * 1024;
template <int TC_THREADS, bool STAGED, int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(TC_THREADS)
    sample_topk_cluster_kernel(const bf16* __restrict__ logits, int* __restrict__ out, size_t vocab, float temperature, int k, uint64_t seed,
                               uint64_t seed_stride, const int* __restrict__ step_ptr, unsigned long long subsequence) {
  static_assert(TC_THREADS > TC_MOST && TC_CAP >= TC_MOST, "a thread for every exponential and one for the random number; k candidates fit");
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char tc_buf[];
  __shared__ unsigned long long cand[TC_CAP];             // this slice's candidates
  __shared__ unsigned long long best[TC_CAP];         // first CTA: those that reach the k-th value
  __shared__ __align__(16) float vals[TC_MOST];
  __shared__ float cums[TC_MOST];
  __shared__ int idxs[TC_MOST];
  __shared__ int s_n, s_cnt[3], s_tot, s_ns[CTAS];
  __shared__ float s_u;
  unsigned long long* all = reinterpret_cast<unsigned long long*>(tc_buf);  // first CTA: everybody's
  const int tid = threadIdx.x, slice = blockIdx.x, rowi = blockIdx.y;
  const uint16_t* row = reinterpret_cast<const uint16_t*>(logits) + (size_t)rowi * vocab;
  if (!(temperature > 0.0f)) temperature = 1.0f;
  k = min(k, (int)min(vocab, (size_t)TC_MOST));
  TopkSlice<TC_THREADS> sl;
  sl.row = row;
  sl.head = (int)min((size_t)((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) / 2, vocab);
  const size_t nvec = (vocab - sl.head) / 8, per = (nvec + CTAS - 1) / CTAS;
  sl.v0 = min(nvec, slice * per), sl.v1 = min(nvec, sl.v0 + per);
  sl.tail0 = sl.head + (int)nvec * 8, sl.loose = slice == 0 ? sl.head + (int)vocab - sl.tail0 : 0;
  const bool loose = tid < sl.loose;  // this thread's element in front of the first 16-byte boundary or behind the last whole piece
  const int loose_at = tid < sl.head ? tid : sl.tail0 + tid - sl.head;
  const uint32_t loose_bits = loose ? (uint32_t)row[loose_at] : 0xff80u;
  // f(eight values, the largest of them, index of the first) for this thread's pieces
  auto pieces = [&](auto&& f) {
    constexpr int U = STAGED ? 1 : 4;
    for (size_t v = sl.v0 + tid; v < sl.v1; v += U * TC_THREADS) {
      uint4 q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t at = min(v + u * TC_THREADS, sl.v1 - 1);
        if constexpr (STAGED) q[u] = *reinterpret_cast<const uint4*>(tc_buf + (at - sl.v0) * 16);
        else asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[u].x), "=r"(q[u].y), "=r"(q[u].z), "=r"(q[u].w) : "l"(row + sl.head + at * 8));
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v + u * TC_THREADS < sl.v1) {
          const uint32_t m = max2(max2(q[u].x, q[u].y), max2(q[u].z, q[u].w));
          f(q[u], max2(m, __byte_perm(m, 0, 0x1032)), sl.head + (int)(v + u * TC_THREADS) * 8);
        }
    }
  };
  if constexpr (STAGED) {  // (a thread reads what it has copied)
    const uint32_t dst = smem_u32(tc_buf);
    for (size_t v = sl.v0 + tid; v < sl.v1; v += TC_THREADS) cp_async16(dst + (uint32_t)(v - sl.v0) * 16u, row + sl.head + v * 8);
    cp_async_commit();
    cp_async_wait<0>();
  }
  uint32_t m2 = 0xff80ff80u;  // -inf twice: what stays where there is no number
  pieces([&](const uint4&, uint32_t m, int) { m2 = max2(m2, m); });
  const uint32_t mx = max(topk_order16(m2 & 0xffffu), topk_order16(loose_bits));
  // the largest bound that k maxima reach (1 if fewer threads have a value: then every value is a candidate)
  uint32_t bound = 0;
#pragma unroll 1
  for (int bit = 15; bit >= 0; --bit) {
    const uint32_t t = bound | (1u << bit);
    if (__syncthreads_count(mx >= t) >= k) bound = t;
  }
  bound = max(bound, 1u);
  if (tid == 0) s_n = 0;
  if (tid < 3) s_cnt[tid] = 0;
  __syncthreads();
  if (mx >= bound) {
    auto take = [&](uint32_t b, int i) {
      if (topk_order16(b) < bound) return;
      const int at = atomicAdd(&s_n, 1);
      if (at < TC_CAP) cand[at] = topk_key((uint16_t)b, i);
    };
    pieces([&](const uint4& q, uint32_t m, int i0) {
      if (topk_order16(m & 0xffffu) < bound) return;
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) take(w[e] & 0xffffu, i0 + 2 * e), take(w[e] >> 16, i0 + 2 * e + 1);
    });
    if (loose) take(loose_bits, loose_at);
  }
  __syncthreads();
  if (s_n > TC_CAP) topk_slice_ties<TC_THREADS>(sl, TopkSums{s_cnt, 0}, mx, bound, k, cand, reinterpret_cast<int*>(best), reinterpret_cast<int*>(tc_buf), &s_n, &s_tot);
  cluster_sync_all();
  if (slice == 0) {
    // ---- gather: all counts at once, then all candidates
    if (tid < CTAS) {
      uint32_t an;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(an) : "r"(smem_u32(&s_n)), "r"(tid));
      asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(s_ns[tid]) : "r"(an) : "memory");
    }
    __syncthreads();
    int n = 0;
#pragma unroll
    for (int c = 0; c < CTAS; ++c) {
      uint32_t ac;
      const int cn = s_ns[c];
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ac) : "r"(smem_u32(cand)), "r"(c));
      for (int i = tid; i < cn; i += TC_THREADS) {
        unsigned long long key;
        asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(key) : "r"(ac + 8u * (uint32_t)i));
        all[n + i] = key;
      }
      n += cn;
    }
    __syncthreads();
    const int actual_k = min(k, n);
    // ---- those that reach the actual_k-th value, by bisection over its 16 bits; the actual_k-th key where they are too many
    unsigned long long kth = 0;
    int m = n;  // keys that reach it
    TopkSums sum{s_cnt, 0};
    if (actual_k > 0) {
      uint32_t top = 0;
      uint32_t own[4];  // this thread's values, where they are few
      const bool few = n <= 4 * TC_THREADS;
#pragma unroll
      for (int u = 0; u < 4; ++u) own[u] = tid + u * TC_THREADS < n ? (uint32_t)(all[tid + u * TC_THREADS] >> 32) : 0u;
#pragma unroll 1
      for (int bit = 15; bit >= 0; --bit) {
        const uint32_t t = top | (1u << bit);
        int c = 0;
        if (few) {
#pragma unroll
          for (int u = 0; u < 4; ++u) c += own[u] >= t;
        } else {
          for (int i = tid; i < n; i += TC_THREADS) c += (uint32_t)(all[i] >> 32) >= t;
        }
        c = sum(c);
        if (c >= actual_k) top = t, m = c;
      }
      kth = (unsigned long long)top << 32;
#pragma unroll 1
      for (int bit = 31; bit >= 0 && m > TC_CAP; --bit) {
        const unsigned long long t = kth | (1ull << bit);
        int c = 0;
        for (int i = tid; i < n; i += TC_THREADS) c += all[i] >= t;
        c = sum(c);
        if (c >= actual_k) kth = t, m = c;
      }
      if (tid == 0) s_tot = 0;
      __syncthreads();
      for (int i = tid; i < n; i += TC_THREADS)
        if (all[i] >= kth) best[atomicAdd(&s_tot, 1)] = all[i];
    }
    __syncthreads();
    if (actual_k == 0) {
      if (tid == 0) out[rowi] = -1;
    } else {
      // ---- rank by counting.  A key holds its value, but for the sign of a zero, which no exponential below sees.
      for (int i = tid; i < m; i += TC_THREADS) {
        const unsigned long long key = best[i];
        int rank = 0;
        for (int j = 0; j < m; ++j) rank += best[j] > key;
        if (rank < actual_k) {
          const uint32_t o = (uint32_t)(key >> 32);
          idxs[rank] = (int)(0xFFFFFFu - (unsigned)(key & 0xFFFFFFull));
          vals[rank] = __fdiv_rn(lo2f(o & 0x8000u ? o ^ 0x8000u : ~o & 0xffffu), temperature);
        }
      }
      if (tid == TC_THREADS - 1) {  // (a warp of its own, where it has no key to rank)
        curandState rng;
        const unsigned long long sd = seed + (unsigned long long)rowi * seed_stride + (step_ptr ? (unsigned)step_ptr[rowi] : 0u);
        curand_init(sd, subsequence, 0, &rng);
        s_u = curand_uniform(&rng);
      }
      __syncthreads();
      // ---- the reference's tail, logit_decode.cu:225-273: the best quotient is the largest (division by a positive number keeps the order)
      if (actual_k == 1) {
        if (tid == 0) out[rowi] = idxs[0];  // softmax over one candidate is 1; u in (0,1] always selects it
      } else {
        const float max_val = vals[0];
        __syncthreads();
        if (tid < TC_MOST) vals[tid] = tid < actual_k ? expf(__fsub_rn(vals[tid], max_val)) : 0.f;
        __syncthreads();
        if (tid < 32) {
          // the sum and the running sums that the draw is compared with are the same chain
          if (tid == 0) {
            float sum = 0.0f;
            for (int i = 0; i < actual_k; i += 4) {
              const float4 v = *reinterpret_cast<const float4*>(vals + i);
              cums[i] = sum = __fadd_rn(sum, v.x);
              cums[i + 1] = sum = __fadd_rn(sum, v.y);
              cums[i + 2] = sum = __fadd_rn(sum, v.z);
              cums[i + 3] = sum = __fadd_rn(sum, v.w);
            }
          }
          __syncwarp();
          const float u = __fmul_rn(s_u, cums[actual_k - 1]);
          int at = actual_k - 1;
#pragma unroll
          for (int c = TC_MOST - 32; c >= 0; c -= 32) {
            const uint32_t hit = __ballot_sync(0xffffffffu, c + tid < actual_k && u <= cums[c + tid]);
            if (hit) at = c + __ffs(hit) - 1;
          }
          if (tid == 0) out[rowi] = idxs[at];
        }
      }
    }
  }
  cluster_sync_all();  // nobody leaves while the first CTA reads its candidates
}
template <int TC_THREADS, bool STAGED, int CTAS>
static cudaError_t launch_topk_cluster(const bf16* logits, int* out_tokens, int n_rows, size_t vocab, float temperature, int k, uint64_t seed, uint64_t seed_stride,
                                       const int* step_ptr, unsigned long long subsequence, cudaStream_t st) {
  constexpr size_t all = (size_t)CTAS * TC_CAP * 8;
  const size_t slice = (vocab / 8 + CTAS - 1) / CTAS * 16, tie = topk_tie_ints(vocab, CTAS) * sizeof(int), smem = std::max({STAGED ? slice : 0, all, tie});
  if constexpr (STAGED && CTAS < TC_CTAS) {
    static PerDeviceOnce set;
    if (set.need()) {
      cudaError_t e = cudaFuncSetAttribute(sample_topk_cluster_kernel<TC_THREADS, STAGED, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_STAGE * TC_CTAS / CTAS + 64);
      if (e != cudaSuccess) return e;
      set.done();
    }
  }
  return launch_k(sample_topk_cluster_kernel<TC_THREADS, STAGED, CTAS>, dim3(CTAS, n_rows), dim3(TC_THREADS), smem, st, logits, out_tokens, vocab, temperature, k,
                  seed, seed_stride, step_ptr, subsequence);
}

cudaError_t launch_sample_topk(const bf16* logits, int* out_tokens, int n_rows, size_t vocab, float temperature,
                               int k, uint64_t seed, uint64_t seed_stride, const int* step_ptr, cudaStream_t st,
                               uint64_t subsequence) {
  if (n_rows == 0) return cudaSuccess;
  if (k == 1 && vocab % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && vocab >= 4096) {
    // candidate scratch per stream (engines of one process run on their own streams); buffers are never freed or
    // moved once handed out, because captured CUDA graphs keep their address
    struct Scratch {
      Cand* p = nullptr;
      int cap = 0;
    };
    static std::mutex mu;
    static std::map<std::pair<int, cudaStream_t>, std::vector<Scratch>> pool;  // keyed by (device, stream): a stream handle
                                                                               // value can come back on another device
    Cand* cands = nullptr;
    {
      int dev = 0;
      (void)cudaGetDevice(&dev);
      std::lock_guard<std::mutex> lk(mu);
      std::vector<Scratch>& v = pool[std::make_pair(dev, st)];
      for (const Scratch& sc : v)
        if (sc.cap >= n_rows) cands = sc.p;
      if (!cands) {
        Scratch sc;
        sc.cap = std::max(n_rows, 256);
        cudaError_t e = cudaMalloc(&sc.p, std::max<size_t>(256 * GREEDY_MOST, (size_t)sc.cap * GREEDY_SLICES) * sizeof(Cand));
        if (e != cudaSuccess) return e;
        v.push_back(sc);
        cands = sc.p;
      }
    }
    const int slices = greedy_slices(n_rows, vocab);
    (void)launch_k(greedy_slice_kernel, dim3(slices, n_rows), dim3(256), 0, st, logits, cands, vocab);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    (void)launch_k(greedy_merge_kernel, dim3((n_rows + 3) / 4), dim3(128), 0, st, (const Cand*)cands, out_tokens, n_rows, slices);
    return cudaGetLastError();
  }
  // (slices longer than a candidate list of which fewer than k threads hold a value, vocabularies of 4 to 8 thousand with large k, have no bound to
  // start from: 64 rows of 8000, k = 128, 44 us by the radix select, 86 here)
  if (k > 1 && k <= TC_MOST && vocab <= (1u << 23) && n_rows <= 65535 && (vocab <= (size_t)TC_CTAS * TC_CAP || vocab / (TC_CTAS * 8) > (size_t)k)) {
    // Few rows take all the CTAs they can get; more rows fewer of them, whose first one has fewer candidates to rank and shares its SM with less (us of
    // 151936, k = 50, 8 4 2 CTAs a row: 1 row 14.0 14.9 16.5, 8 14.2 15.4 17.1, 16 17.3 15.6 17.5, 32 17.9 17.3 17.9, 48 24.4 20.8 19.0, 64 25.2 21.9 19.4).  A
    // slice has to hold an eighth more pieces than k: with hardly more, the k-th of their maxima is a bound that most values reach, and the lists are
    // long or overflow (33 rows of 2064, k = 128: 19.9 with eight CTAs, 25.3 with two; from 2304 on two are quicker).  More than 16 rows that stay
    // with eight take 256 threads, so that all clusters are on the chip at once (256 rows of 2056, k = 128: 77 us, 132 with 512).  Against eight CTAs for all
    // (256 threads from 17 rows on, everything read twice from memory), 24 vocabularies of 500 to 262144, 1 to 256 rows, k of 2 to 128: 0.30 to 1.0 of the
    // time; clusters of two near the staging limit, one CTA an SM, 100 to 256 rows of 128256 to 155648 0.51 to 0.64.
    const bool staged = (vocab / 8 + TC_CTAS - 1) / TC_CTAS * 16 <= (size_t)TC_STAGE;
    auto holds = [&](int ctas) { return vocab <= (size_t)ctas * TC_CAP || vocab / (ctas * 8) >= (size_t)k + k / 8; };
    auto launch = staged && n_rows > 32 && holds(2)  ? launch_topk_cluster<512, true, 2>
                  : staged && n_rows > 8 && holds(4) ? launch_topk_cluster<512, true, 4>
                  : n_rows > 16                      ? (staged ? launch_topk_cluster<256, true, 8> : launch_topk_cluster<256, false, 8>)
                                                     : (staged ? launch_topk_cluster<512, true, 8> : launch_topk_cluster<512, false, 8>);
    return launch(logits, out_tokens, n_rows, vocab, temperature, k, seed, seed_stride, step_ptr, subsequence, st);
  }
  // more than TC_MOST candidates, and the above: the radix select; the k-round scan of the reference for vocabularies beyond 2^24 entries, which the
  // 24-bit index field of the key cannot hold, and for k < 1
  if (k > 1 && vocab < (1u << 24))
    (void)launch_k(sample_topk_select_kernel, dim3(n_rows), dim3(1024), 0, st, logits, out_tokens, vocab, temperature, k, seed, seed_stride,
                   step_ptr, (unsigned long long)subsequence);
  else
    (void)launch_k(sample_topk_kernel, dim3(n_rows), dim3(1024), 0, st, logits, out_tokens, vocab, temperature, k, seed, seed_stride, step_ptr,
                   (unsigned long long)subsequence);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ repetition penalty
// apply_repetition_penalty_kernel is declared by the reference (include/layers_include.cuh:33) and never defined; the
// conventional semantics (CTRL / HF RepetitionPenaltyLogitsProcessor) are implemented: every DISTINCT token id of
// a row's context has its logit divided (positive) or multiplied (otherwise) by the penalty.  Row r's context is
// ctx[ctx_row[r] * ctx_stride + 0 .. ctx_len[r]) (ctx_row == nullptr: row r, ctx_len == nullptr: fixed_len).
// One thread per context position; only the first occurrence of a token applies, so no logit is written twice.
__global__ void repetition_penalty_kernel(bf16* __restrict__ logits, const int* __restrict__ ctx, const int* __restrict__ ctx_row,
                                          const int* __restrict__ ctx_len, int len_bias, size_t fixed_len, size_t ctx_stride, int vocab,
                                          float penalty) {
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.y;
  const size_t n = ctx_len ? (size_t)(ctx_len[r] + len_bias) : fixed_len;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int* c = ctx + (size_t)(ctx_row ? ctx_row[r] : r) * ctx_stride;
  const int t = c[i];
  if (t < 0 || t >= vocab) return;
  for (size_t j = 0; j < i; ++j)
    if (c[j] == t) return;
  bf16* p = logits + (size_t)r * vocab + t;
  float v = bf2f(*p);
  v = v > 0.0f ? __fdiv_rn(v, penalty) : __fmul_rn(v, penalty);
  *p = f2bf(v);
}
cudaError_t launch_repetition_penalty(bf16* logits, const int* ctx, const int* ctx_row, const int* ctx_len, int len_bias, size_t fixed_len,
                                      size_t max_len, size_t ctx_stride, int n_rows, int vocab, float penalty, cudaStream_t st) {
  if (n_rows == 0 || max_len == 0) return cudaSuccess;
  (void)launch_k(repetition_penalty_kernel, dim3((unsigned)((max_len + 255) / 256), n_rows), dim3(256), 0, st, logits, ctx, ctx_row, ctx_len,
                 len_bias, fixed_len, ctx_stride, vocab, penalty);
  return cudaGetLastError();
}
// token history of the engine's sequences (only kept while a repetition penalty is set): the input token of every row
// of a forward goes to hist[slot[t]][pos[t]]
__global__ void history_append_kernel(int* __restrict__ hist, size_t stride, const int* __restrict__ ids, const int* __restrict__ pos,
                                      const int* __restrict__ slot, int n) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n && (size_t)pos[t] < stride) hist[(size_t)slot[t] * stride + pos[t]] = ids[t];
}
cudaError_t launch_history_append(int* hist, size_t stride, const int* ids, const int* pos, const int* slot, int n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  (void)launch_k(history_append_kernel, dim3((n + 127) / 128), dim3(128), 0, st, hist, stride, ids, pos, slot, n);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ synthetic weights
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__global__ void synth_fill_kernel(bf16* blob, size_t elem_begin, size_t n, unsigned long long seed, int kind) {
  pdl_wait();
  pdl_trigger();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long g = elem_begin + i;
  unsigned long long a = mix64(seed + (g + 1) * 0x9E3779B97F4A7C15ull);
  unsigned long long b = mix64(a + 0x9E3779B97F4A7C15ull);
  int sum = (int)((a & 0xffff) + ((a >> 16) & 0xffff) + ((a >> 32) & 0xffff) + (a >> 48) + (b & 0xffff) +
                  ((b >> 16) & 0xffff) + ((b >> 32) & 0xffff) + (b >> 48));
  float c = (float)(sum - 262140);
  float v = kind == 0 ? __fmul_rn(c, 0.02f / 53509.92f) : __fadd_rn(1.0f, __fmul_rn(c, 0.05f / 53509.92f));
  blob[g] = f2bf(v);
}
cudaError_t launch_synth_fill(bf16* blob, size_t elem_begin, size_t n_elems, uint64_t seed, int kind,
                              cudaStream_t st) {
  if (!n_elems) return cudaSuccess;
  (void)launch_k(synth_fill_kernel, dim3((unsigned)((n_elems + 255) / 256)), dim3(256), 0, st, blob, elem_begin, n_elems, seed, kind);
  return cudaGetLastError();
}

// fill positions [pos0, pos0+n_pos) of one sequence's KV pages (all layers, K and V) with
// seeded N(0,1)-like values: bench-only stand-in for a long prefill
__global__ void kv_fill_kernel(KvGeom kv, const int* __restrict__ block_row, int pos0, int n_pos,
                               unsigned long long seed) {
  pdl_wait();
  pdl_trigger();
  const size_t per_pos = (size_t)kv.n_layers * 2 * kv.n_kv * kv.hd;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= per_pos * n_pos) return;
  int p = (int)(i / per_pos);
  size_t r = i % per_pos;
  int d = (int)(r % kv.hd);
  r /= kv.hd;
  int head = (int)(r % kv.n_kv);
  r /= kv.n_kv;
  int which = (int)(r % 2);
  int layer = (int)(r / 2);
  int pos = pos0 + p;
  int page = block_row[pos / kv.page_size];
  unsigned long long a = mix64(seed + (i + 1) * 0x9E3779B97F4A7C15ull);
  int sum = (int)((a & 0xffff) + ((a >> 16) & 0xffff) + ((a >> 32) & 0xffff) + (a >> 48));
  float v = __fmul_rn((float)(sum - 131070), 1.0f / 37837.0f);
  kv.chunk(page, layer, which, head)[(size_t)(pos % kv.page_size) * kv.hd + d] = f2bf(v);
}
cudaError_t launch_kv_fill(const KvGeom& kv, const int* block_row, int pos0, int n_pos, uint64_t seed,
                           cudaStream_t st) {
  size_t n = (size_t)kv.n_layers * 2 * kv.n_kv * kv.hd * n_pos;
  if (!n) return cudaSuccess;
  (void)launch_k(kv_fill_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, kv, block_row, pos0, n_pos, seed);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ tensor-parallel arg-max merge
__global__ void tp_cand_make_kernel(const bf16* __restrict__ logits, const int* __restrict__ sampled, TpCand* cand, int n,
                                    size_t vocab_local, int vocab_offset) {
  pdl_wait();
  pdl_trigger();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int li = sampled[i];
  TpCand c;
  c.val = li >= 0 ? bf2f(logits[(size_t)i * vocab_local + li]) : -CUDART_INF_F;
  c.idx = li >= 0 ? li + vocab_offset : -1;
  cand[i] = c;
}
__global__ void tp_cand_merge_kernel(const TpCand* __restrict__ all, int tp, int n, int* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float bv = -CUDART_INF_F;
  int bi = -1;
  for (int r = 0; r < tp; ++r) {
    const TpCand c = all[(size_t)r * n + i];
    if (cand_better(c.val, c.idx, bv, bi)) {
      bv = c.val;
      bi = c.idx;
    }
  }
  out[i] = bi;
}
__global__ void residual_add_f32_kernel(bf16* __restrict__ x, const float* __restrict__ y, size_t n) {
  pdl_wait();
  pdl_trigger();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = f2bf(__fadd_rn(bf2f(x[i]), bf2f(f2bf(y[i]))));
}
cudaError_t launch_residual_add_f32(bf16* x, const float* y, size_t n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  (void)launch_k(residual_add_f32_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, x, y, n);
  return cudaGetLastError();
}
cudaError_t launch_tp_cand_make(const bf16* logits_local, const int* sampled_local, TpCand* cand, int n_rows, size_t vocab_local,
                                int vocab_offset, cudaStream_t st) {
  if (!n_rows) return cudaSuccess;
  (void)launch_k(tp_cand_make_kernel, dim3((n_rows + 127) / 128), dim3(128), 0, st, logits_local, sampled_local, cand, n_rows,
                 vocab_local, vocab_offset);
  return cudaGetLastError();
}
cudaError_t launch_tp_cand_merge(const TpCand* all, int tp, int n_rows, int* out_tokens, cudaStream_t st) {
  if (!n_rows) return cudaSuccess;
  (void)launch_k(tp_cand_merge_kernel, dim3((n_rows + 127) / 128), dim3(128), 0, st, all, tp, n_rows, out_tokens);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ step bookkeeping
__global__ void advance_kernel(int* pos, int* ids, const int* sampled, int n, int* step_ptr) {
  pdl_wait();
  pdl_trigger();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    pos[i] += 1;
    ids[i] = sampled[i];
    if (step_ptr) step_ptr[i] += 1;
  }
}
cudaError_t launch_advance(int* pos, int* ids, const int* sampled, int n, int* step_ptr, cudaStream_t st) {
  if (!n) return cudaSuccess;
  (void)launch_k(advance_kernel, dim3((n + 127) / 128), dim3(128), 0, st, pos, ids, sampled, n, step_ptr);
  return cudaGetLastError();
}

}  // namespace qie
