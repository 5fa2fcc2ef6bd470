// attn_ref_rows.cu -- reference-order attention of many rows of one sequence (prompts), bit for bit what attention_ref_kernel
// (ops_ref_order.cu) and the reference's selfattention (layers/src/self_attension.cu:10-149) compute per row and head.
//
// The order is serial per row and head -- a product tree over the head, a sum of exponentials over the positions, an fma chain per output
// -- but rows and heads are independent of each other.  A CTA takes `rows` consecutive rows times the G query heads of one kv head, up
// to R "virtual rows", one per lane (or per SP = hd / 64 lanes): they share every key and value row, which is widened to fp32 in
// shared memory once and read as a broadcast.
//   scores : lane = (virtual row, key slot); the query sits in 64 registers; 64 products and the tree's 63 sums per score, no shuffles.
//            hd 128 / 256: a lane holds the elements e = c modulo SP, whose strides >= SP are the tree's first levels; the last one or
//            two levels are shuffles.  Scores go to S[position][virtual row] in shared memory.
//   softmax: exponentials and divisions by all threads, the serial sum by one lane per virtual row (R chains side by side)
//   values : lane = (virtual row, group of columns); o = fma(p, v, o) over ascending positions, v broadcast, p one conflict-free read
// What bounds it: fp32 issue (127 + hd instructions per score and value row) and, for the values, shared-memory reads.  One block per
// (row, head) spent its time in single-thread chains and shuffles: 500 rows behind 300 cached positions, 14 heads of 64: 824 us there.
// Positions behind a row's own are never multiplied in (a value there may be infinite).
#include <math_constants.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "ref_math.cuh"

namespace qie {
namespace {

constexpr int NT = 256, NWARP = NT / 32;
constexpr int TILE = 4096;                 // elements of a key or value tile: 64 rows of 64, 32 of 128, 16 of 256
constexpr int TILE_F = 64 * 68;            // floats of a buffer: keys by element class, 64 + 4 floats each
constexpr int MAX_R = 32;

// page ids a CTA keeps in shared memory (a multiple of 4: what follows stays 16-byte aligned)
__host__ __device__ inline int page_ints(const AttnArgs& a) { return a.k_pages ? 0 : ((a.max_kv_len + a.kv.page_size - 1) / a.kv.page_size + 3) & ~3; }
// eight elements; rows off a 16-byte boundary (a caller's own pages, a slice) are read in words
__device__ __forceinline__ uint4 load8(const bf16* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <int NP, int R, bool PL>
__global__ void __launch_bounds__(NT, 2) attention_ref_rows_kernel(AttnArgs a, int rows) {
  pdl_wait();
  pdl_trigger();
  constexpr int HD = 64 * NP, SP = NP, KS = 32 / (R * SP), TK = TILE / HD;
  constexpr int DN = HD * R / (NWARP * 32);  // output columns of a lane
  static_assert(KS >= 1 && DN >= 2, "lanes of a warp");
  extern __shared__ __align__(16) float sm[];
  float* tile = sm;                          // two buffers
  int* pages = reinterpret_cast<int*>(sm + 2 * TILE_F);  // page ids (page lists: read where they are used)
  float* S = sm + 2 * TILE_F + page_ints(a);             // [position][R]
  __shared__ int s_len[MAX_R];
  __shared__ float s_max[NWARP][MAX_R], s_sum[MAX_R];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t = gridDim.x - 1 - blockIdx.x, kvh = blockIdx.y;  // late rows see more positions: they start first
  const int row0 = t * rows, n = min(rows, a.n_tok - row0), G = a.n_q / a.kv.n_kv, psz = a.kv.page_size;
  int slot = 0;
  if (!PL) {
    slot = a.slot[row0];
    if (!a.one_seq)
      for (int i = 1; i < n; ++i)
        if (a.slot[row0 + i] != slot) return;  // rows of several sequences: attention_ref_kernel takes them
  }
  int max_len = 0, min_len = 0x7fffffff;
  for (int i = 0; i < n; ++i) {
    const int l = a.pos[row0 + i] + 1;
    max_len = max(max_len, l), min_len = min(min_len, l);
  }
  if (max_len <= 0) {  // no row sees a position: zeros, and no page to read
    for (int i = tid; i < n * G * HD; i += NT)
      a.out[(size_t)(row0 + i / (G * HD)) * a.n_q * HD + (size_t)kvh * G * HD + i % (G * HD)] = f2bf(0.f);
    return;
  }
  if (tid < R) s_len[tid] = tid < n * G ? a.pos[row0 + tid / G] + 1 : 0;
  if (!PL) {
    const int* bt = a.block_table + (size_t)slot * a.max_pages;
    for (int i = tid; i <= (max_len - 1) / psz; i += NT) pages[i] = bt[i];
    __syncthreads();
  }
  const size_t pl_row = (size_t)a.pl_layers * a.kv.n_kv * HD, pl_off = (size_t)a.layer * a.kv.n_kv * HD + (size_t)kvh * HD;
  const int shift = (psz & (psz - 1)) == 0 ? __ffs(psz) - 1 : -1;
  auto row_of = [&](int k, int is_v) -> const bf16* {
    const int pg = shift >= 0 ? k >> shift : k / psz, off = k - pg * psz;
    if (PL) return (is_v ? a.v_pages : a.k_pages)[pg] + (size_t)off * pl_row + pl_off;
    return a.kv.chunk(pages[pg], a.layer, is_v, kvh) + (size_t)off * HD;
  };
  const int n_tiles = (max_len + TK - 1) / TK;
  uint4 pre[2];  // the next tile's rows: thread = 8 elements twice
  auto fetch = [&](int tl, int is_v) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = (tid + u * NT) * 8, k = min(tl * TK + e / HD, max_len - 1);
      pre[u] = load8(row_of(k, is_v) + e % HD);
    }
  };
  auto put = [&](int buf, int is_v) {
    float* dst = tile + buf * TILE_F;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = (tid + u * NT) * 8, k = e / HD, e0 = e % HD;
      const uint32_t w[4] = {pre[u].x, pre[u].y, pre[u].z, pre[u].w};
      float v[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[2 * i] = lo2f(w[i]), v[2 * i + 1] = hi2f(w[i]);
      if (is_v || SP == 1) {
        float* d = dst + k * (is_v ? HD : 68) + e0;
        *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(d + 4) = make_float4(v[4], v[5], v[6], v[7]);
      } else if (SP == 2) {
        float* d = dst + k * 136 + e0 / 2;
        *reinterpret_cast<float4*>(d) = make_float4(v[0], v[2], v[4], v[6]);
        *reinterpret_cast<float4*>(d + 68) = make_float4(v[1], v[3], v[5], v[7]);
      } else {
        float* d = dst + k * 272 + e0 / 4;
#pragma unroll
        for (int c = 0; c < 4; ++c) *reinterpret_cast<float2*>(d + c * 68) = make_float2(v[c], v[4 + c]);
      }
    }
  };
  // ---- scores
  fetch(0, 0);  // on its way beside the queries
  {
    const int c = lane % SP, r = lane / SP % R, ks = lane / (SP * R);
    float q[64];
    if (r < n * G) {
      const bf16* src = a.q + (size_t)(row0 + r / G) * a.n_q * HD + (size_t)(kvh * G + r % G) * HD;
#pragma unroll
      for (int ch = 0; ch < HD / 8; ++ch) {
        const uint4 x = load8(src + ch * 8);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (SP == 1) q[8 * ch + 2 * i] = lo2f(w[i]), q[8 * ch + 2 * i + 1] = hi2f(w[i]);
          if (SP == 2) q[4 * ch + i] = c ? hi2f(w[i]) : lo2f(w[i]);
          if (SP == 4 && (i & 1) == 0) q[2 * ch + i / 2] = (c & 1) ? hi2f(c & 2 ? w[i + 1] : w[i]) : lo2f(c & 2 ? w[i + 1] : w[i]);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 64; ++j) q[j] = 0.f;
    }
    const float den = __fsqrt_rn((float)HD);
    put(0, 0);
    __syncthreads();
    const int len = s_len[r];
    float mx = -1e9f;
    for (int tl = 0; tl < n_tiles; ++tl) {
      if (tl + 1 < n_tiles) fetch(tl + 1, 0);
      const float* kt = tile + (tl & 1) * TILE_F;
      const int end = min(TK, max_len - tl * TK);  // (a warp's lanes go round together: its first key decides)
#pragma unroll 1
      for (int k0 = warp * KS; k0 < end; k0 += NWARP * KS) {
        const int kk = k0 + ks;
        const float4* kr = reinterpret_cast<const float4*>(kt + (kk * SP + c) * 68);
        // the tree with strides 32 ... 1 over the lane's 64 elements, depth first: part[b] is the sum over the elements b modulo 8
        // folded down to stride 8, with the tree's own pairs
        float part[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float t4[4][8];
#pragma unroll
          for (int m = 0; m < 8; ++m) {  // elements 8 m + 4 h .. + 3
            const float4 kv = kr[2 * m + h];
            t4[0][m] = __fmul_rn(q[8 * m + 4 * h], kv.x);
            t4[1][m] = __fmul_rn(q[8 * m + 4 * h + 1], kv.y);
            t4[2][m] = __fmul_rn(q[8 * m + 4 * h + 2], kv.z);
            t4[3][m] = __fmul_rn(q[8 * m + 4 * h + 3], kv.w);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int s = 4; s >= 1; s >>= 1)  // strides 32, 16, 8
#pragma unroll
              for (int m = 0; m < s; ++m) t4[i][m] = __fadd_rn(t4[i][m], t4[i][m + s]);
            part[4 * h + i] = t4[i][0];
          }
        }
#pragma unroll
        for (int s = 4; s >= 1; s >>= 1)  // strides 4, 2, 1
#pragma unroll
          for (int b = 0; b < s; ++b) part[b] = __fadd_rn(part[b], part[b + s]);
        float dot = part[0];
#pragma unroll
        for (int s = SP / 2; s >= 1; s >>= 1) dot = __fadd_rn(dot, __shfl_xor_sync(0xffffffffu, dot, s));  // the head's last strides
        const float sc = __fdiv_rn(dot, den);
        const int k = tl * TK + kk;
        if (k < len) mx = fmaxf(mx, sc);
        if (c == 0 && k < max_len) S[(size_t)k * R + r] = sc;
      }
      if (tl + 1 < n_tiles) put((tl + 1) & 1, 0);
      __syncthreads();
    }
#pragma unroll
    for (int s = SP * R; s < 32; s <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
    if (lane < SP * R && c == 0) s_max[warp][r] = mx;
    __syncthreads();
  }
  fetch(0, 1);  // (the first values are on their way during the softmax)
  // ---- softmax
  {
    const int r = tid % R, len = s_len[r];
    float m = s_max[0][r];
#pragma unroll
    for (int w = 1; w < NWARP; ++w) m = fmaxf(m, s_max[w][r]);
#pragma unroll 4
    for (int k = tid / R; k < max_len; k += NT / R) S[(size_t)k * R + r] = k < len ? expf(__fsub_rn(S[(size_t)k * R + r], m)) : 0.f;
    __syncthreads();
    if (tid < R) {  // one chain per virtual row; zeros behind a row's positions leave its sum as it is
      float sum = 0.f;
      int k = 0;
      for (; k + 16 <= max_len; k += 16) {
        float e[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) e[i] = S[(size_t)(k + i) * R + tid];
#pragma unroll
        for (int i = 0; i < 16; ++i) sum = __fadd_rn(sum, e[i]);
      }
      for (; k < max_len; ++k) sum = __fadd_rn(sum, S[(size_t)k * R + tid]);
      s_sum[tid] = sum;
    }
    __syncthreads();
    const float sum = s_sum[r];
#pragma unroll 4
    for (int k = tid / R; k < len; k += NT / R) S[(size_t)k * R + r] = __fdiv_rn(S[(size_t)k * R + r], sum);
  }
  // ---- values
  const int r = lane % R, d0 = (warp * (32 / R) + lane / R) * DN, len = s_len[r];
  float o[DN];
#pragma unroll
  for (int i = 0; i < DN; ++i) o[i] = 0.f;
  put(0, 1);
  __syncthreads();
  for (int tl = 0; tl < n_tiles; ++tl) {
    if (tl + 1 < n_tiles) fetch(tl + 1, 1);
    const float* vt = tile + (tl & 1) * TILE_F + d0;
    const float* pt = S + (size_t)tl * TK * R + r;
    auto step = [&](int kk) {
      const float p = pt[kk * R];
      const float* v = vt + kk * HD;
      if constexpr (DN == 2) {
        const float2 x = *reinterpret_cast<const float2*>(v);
        o[0] = __fmaf_rn(p, x.x, o[0]), o[1] = __fmaf_rn(p, x.y, o[1]);
      } else {
#pragma unroll
        for (int i = 0; i < DN; i += 4) {
          const float4 x = *reinterpret_cast<const float4*>(v + i);
          o[i] = __fmaf_rn(p, x.x, o[i]), o[i + 1] = __fmaf_rn(p, x.y, o[i + 1]);
          o[i + 2] = __fmaf_rn(p, x.z, o[i + 2]), o[i + 3] = __fmaf_rn(p, x.w, o[i + 3]);
        }
      }
    };
    if ((tl + 1) * TK <= min_len) {  // every row sees the whole tile
#pragma unroll 8
      for (int kk = 0; kk < TK; ++kk) step(kk);
    } else {
      const int end = min(TK, len - tl * TK);  // (negative for lanes without a row)
      for (int kk = 0; kk < end; ++kk) step(kk);
    }
    if (tl + 1 < n_tiles) put((tl + 1) & 1, 1);
    __syncthreads();
  }
  if (r < n * G) {
    bf16* dst = a.out + (size_t)(row0 + r / G) * a.n_q * HD + (size_t)(kvh * G + r % G) * HD + d0;
#pragma unroll
    for (int i = 0; i < DN; i += 2) {
      if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0) *reinterpret_cast<uint32_t*>(dst + i) = pack2(f2bf(o[i]), f2bf(o[i + 1]));
      else dst[i] = f2bf(o[i]), dst[i + 1] = f2bf(o[i + 1]);
    }
  }
}

template <int NP, int R, bool PL>
cudaError_t launch_rows(const AttnArgs& a, int rows, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(attention_ref_rows_kernel<NP, R, PL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  if (e != cudaSuccess) return e;
  return launch_k(attention_ref_rows_kernel<NP, R, PL>, dim3((a.n_tok + rows - 1) / rows, a.kv.n_kv), dim3(NT), smem, st, a, rows);
}

}  // namespace

// The most virtual rows whose scores leave room for two CTAs on an SM and whose tiles still make two CTAs for every SM, else fewer: a
// tile shares its key and value rows among its virtual rows, but a short launch needs CTAs, and more than 76 KB of scores cost
// the second CTA.  Measured (us, 32 / 16 / 8 virtual rows; one block per row and head): 500 rows behind 300 positions, 14 heads on 2, 64
// wide 128 / 112 / 137; 820.  64 rows behind 800: 98 / 61 / 42; 291.  One row at 801: 89 / 56 / 39; 120.  12 heads on 2, 128 wide, 500
// rows behind 300: - / 185 / 223; 981.
// Up to 16 positions one block per row and head is quicker (16 rows, 12 heads of 128: 6.0, 6.7 here).
int attention_ref_tile_rows(const AttnArgs& a, int num_sms, int* virtual_rows) {
  if (a.max_kv_len <= 16) return 0;
  const int G = a.n_q / a.kv.n_kv, np = a.kv.hd / 64;
  int best = 0;
  for (int R = 32 / np; R >= 8 && R >= G; R /= 2) {
    const size_t s = ((size_t)a.max_kv_len * R + page_ints(a)) * sizeof(float);
    if (s > 180 * 1024) continue;  // (8 virtual rows above 5.7k positions, 16 above 2.8k: attention_ref_kernel)
    best = R / G, *virtual_rows = R;
    if (s <= 76 * 1024 && (long)((a.n_tok + best - 1) / best) * a.kv.n_kv >= 2 * num_sms) break;
  }
  return best;
}

cudaError_t launch_attention_ref_rows(const AttnArgs& a, int rows, int virtual_rows, cudaStream_t st) {
  const size_t smem = (2 * TILE_F + (size_t)a.max_kv_len * virtual_rows + page_ints(a)) * sizeof(float);
#define QIE_ROWS(NP, R)                            \
  if (a.kv.hd == 64 * NP && virtual_rows == R) {   \
    return a.k_pages ? launch_rows<NP, R, true>(a, rows, smem, st) : launch_rows<NP, R, false>(a, rows, smem, st); \
  }
  QIE_ROWS(1, 32)
  QIE_ROWS(1, 16)
  QIE_ROWS(1, 8)
  QIE_ROWS(2, 16)
  QIE_ROWS(2, 8)
  QIE_ROWS(4, 8)
#undef QIE_ROWS
  return cudaErrorInvalidValue;
}

}  // namespace qie
