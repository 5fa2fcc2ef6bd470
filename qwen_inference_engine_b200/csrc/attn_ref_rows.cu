// attn_ref_rows.cu -- reference-order attention of many rows of one sequence (prompts), bit for bit what attention_ref_kernel
// (ops_ref_order.cu) and the reference's selfattention (layers/src/self_attension.cu:10-149) compute per row and head.
//
// The order is serial per row and head -- a product tree over the head, a sum of exponentials over the positions, an fma chain per output
// -- but rows and heads are independent of each other.  A CTA takes `rows` consecutive rows times the G query heads of one kv head, up
// to R "virtual rows", one per lane (or per SP = hd / 64 lanes): they share every key and value row.
//   scores : lane = (virtual row, key slot); the query sits in 32 registers of bf16 pairs, the key is read as it is and broadcast.  fma.rn.f32.bf16 takes
//            the products, two of the tree's first stride in one rounding where that is exact (Magnitudes), and packed sums the rest: 64 + 16
//            instructions a score.  hd 128 / 256: a lane holds the elements e = c modulo SP, whose strides >= SP are the tree's first levels; the
//            last one or two levels are shuffles.  Scores go to S[position][virtual row] in shared memory.
//   softmax: exponentials and quotients by all threads, eight chains at a time; the serial sum by one lane per virtual row (R chains side by side)
//   values : a tile is widened to fp32 in shared memory once; lane = (one or two virtual rows, 4 columns); o = fma(p, v, o) over ascending positions
// What bounds it: instruction issue (2.3 a cycle, 16 warps an SM at 128 registers) and the latency of the steps; fp32 arithmetic is 36 % of the
// time.  One block per (row, head) spent its time in single-thread chains and shuffles: 500 rows behind 300 cached positions, 14 heads of 64:
// 824 us.  Keys widened to fp32 as well, the query in 64 registers, a product and a sum for every element, a division for every score and weight: 105; now
// 79.  12 heads of 128: 178, now 137; 28 of 128 355 and 257; 16 of 256 386 and 304.
// Positions behind a row's own are never multiplied in (a value there may be infinite).
#include <math_constants.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "ref_math.cuh"

namespace qie {
namespace {

constexpr int NT = 256, NWARP = NT / 32;
constexpr int TILE = 4096;                 // elements of a key or value tile: 64 rows of 64, 32 of 128, 16 of 256
constexpr int KROW = 144;                  // bytes of a key's element class: 64 bf16 and 16 bytes, so that the rows a warp reads together lie on other banks
constexpr int AHEAD = 2;                   // tiles on their way in registers, one set each
static_assert(64 * KROW <= TILE * 4, "two buffers of keys fit where two of values do");
constexpr int MAX_R = 32;

// page ids a CTA keeps in shared memory (a multiple of 4: what follows stays 16-byte aligned)
__host__ __device__ inline int page_ints(const AttnArgs& a) { return a.k_pages ? 0 : ((a.max_kv_len + a.kv.page_size - 1) / a.kv.page_size + 3) & ~3; }
// eight elements; rows off a 16-byte boundary (ANY: a caller's own pages, a slice) are read in words
template <bool ANY>
__device__ __forceinline__ uint4 load8(const bf16* p) {
  if (!ANY || (reinterpret_cast<uintptr_t>(p) & 15) == 0) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// A lane's part of a score's product tree, depth first over the 16-byte pieces of its 64 elements: leaf l is pieces l and l + 4 (stride 32), then strides
// 16 and 8.
template <bool FUSED, int STEP, class Q, class G>
__device__ __forceinline__ void score_tree(float (&t)[4][2], int l, const Q& q, G& get) {
  if constexpr (STEP == 4) {
    uint32_t x[4], y[4];
    get(l, x), get(l + 4, y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float p[2];
      fma16(p[0], p[1], q[4 * l + i], x[i], -0.f, -0.f);
      if constexpr (FUSED) {
        fma16(t[i][0], t[i][1], q[4 * l + 16 + i], y[i], p[0], p[1]);
      } else {
        fma16(t[i][0], t[i][1], q[4 * l + 16 + i], y[i], -0.f, -0.f);
        add2(t[i][0], t[i][1], p[0], p[1]);
      }
    }
  } else {
    float o[4][2];
    score_tree<FUSED, 2 * STEP>(t, l, q, get);
    score_tree<FUSED, 2 * STEP>(o, l + STEP, q, get);
#pragma unroll
    for (int i = 0; i < 4; ++i) add2(t[i][0], t[i][1], o[i][0], o[i][1]);
  }
}

// Softmax: the position that a thread reads as the u-th behind k0, where its positions are `step` apart; its first one again where that is behind
// `end`, since the last one in front of the end is another thread's, which writes it in the same pass.
__host__ __device__ constexpr int own_position(int k0, int u, int step, int end) { return k0 + u * step < end ? k0 + u * step : k0; }
constexpr bool reads_own_positions(int turn, int step, int end) {
  for (int first = 0; first < step; ++first)
    for (int k0 = first; k0 < end; k0 += turn * step)
      for (int u = 0; u < turn; ++u)
        if (own_position(k0, u, step, end) % step != first || own_position(k0, u, step, end) >= end) return false;
  return true;
}
static_assert(reads_own_positions(8, NT / 8, 333) && reads_own_positions(8, NT / 16, 131) && reads_own_positions(8, NT / 32, 70) && reads_own_positions(2, NT / 8, 1) &&
                  reads_own_positions(2, NT / 8, 45), "a position belongs to one thread");

template <int NP, int R, bool ANY>
__global__ void __launch_bounds__(NT, 2) attention_ref_rows_kernel(AttnArgs a, int rows) {
  pdl_wait();
  pdl_trigger();
  const bool PL = ANY && a.k_pages;  // page lists
  constexpr int HD = 64 * NP, TK = TILE / HD;
  constexpr int SP = NP, KS = 32 / (R * SP);  // lanes of a score, keys of a warp side by side
  constexpr int RP = R * HD >= 1024 ? 2 : 1;       // values: rows of a lane, of 4 columns each
  constexpr int VT = R * HD / (4 * RP), LT = VT == NT ? NT : NT - VT, PIECES = TILE / 8 / LT;  // threads that compute and that fetch there, pieces of a thread
  static_assert(KS >= 1 && VT <= NT && LT * PIECES * 8 == TILE, "lanes of a warp, threads of a block");
  extern __shared__ __align__(16) float sm[];
  float* tile = sm;
  int* pages = reinterpret_cast<int*>(sm + 2 * TILE);  // page ids (page lists: read where they are used)
  float* S = sm + 2 * TILE + page_ints(a);             // [position][R]
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
  const size_t page_stride = a.kv.page_stride();
  const bf16* const base[2] = {PL ? nullptr : a.kv.chunk(0, a.layer, 0, kvh), PL ? nullptr : a.kv.chunk(0, a.layer, 1, kvh)};
  auto row_of = [&](int k, auto is_v) -> const bf16* {
    constexpr bool V = decltype(is_v)::value;
    const int pg = shift >= 0 ? k >> shift : k / psz, off = k - pg * psz;
    if (PL) return (V ? a.v_pages : a.k_pages)[pg] + (size_t)off * pl_row + pl_off;
    return base[V] + (size_t)pages[pg] * page_stride + off * HD;
  };
  const int n_tiles = (max_len + TK - 1) / TK;
  const std::false_type keys{};
  const std::true_type values{};
  // A thread's pieces of a tile, eight elements each, are asked for AHEAD tiles early: a tile's arithmetic is shorter than the way from memory.  (Each set of
  // registers has code of its own: to move one is to wait for it.)
  // ---- scores: lane = (element class, virtual row, key slot)
  const int c = lane % SP;
  {
    const int r = lane / SP % R, ks = lane / (SP * R);
    uint4 pre[AHEAD][2];
    auto fetch = [&](uint4 (&pre)[2], int tl) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int e = (tid + u * NT) * 8;
        pre[u] = load8<ANY>(row_of(min(tl * TK + e / HD, max_len - 1), keys) + e % HD);
      }
    };
#pragma unroll
    for (int t = 0; t < AHEAD; ++t)
      if (t < n_tiles) fetch(pre[t], t);
    // keys go by element class as they are; whether a magnitude is beyond the range of the fused products
    auto next_keys = [&](int tl) {
      auto put = [&](uint4 (&pre)[2]) {
        unsigned char* dst = reinterpret_cast<unsigned char*>(tile) + (tl & 1) * 64 * KROW;
        Magnitudes mag;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int e = (tid + u * NT) * 8;
          const uint32_t w[4] = {pre[u].x, pre[u].y, pre[u].z, pre[u].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) mag.see(w[i]);
          unsigned char* d = dst + e / HD * SP * KROW + e % HD / SP * 2;
          if constexpr (SP == 1) *reinterpret_cast<uint4*>(d) = pre[u];
          if constexpr (SP == 2) {
            *reinterpret_cast<uint2*>(d) = make_uint2(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410));
            *reinterpret_cast<uint2*>(d + KROW) = make_uint2(__byte_perm(w[0], w[1], 0x7632), __byte_perm(w[2], w[3], 0x7632));
          }
          if constexpr (SP == 4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<uint32_t*>(d + i * KROW) = __byte_perm(w[i / 2], w[2 + i / 2], i & 1 ? 0x7632 : 0x5410);
          }
        }
        if (tl + AHEAD < n_tiles) fetch(pre, tl + AHEAD);
        return mag.beyond();
      };
      return tl & 1 ? put(pre[1]) : put(pre[0]);
    };
    uint32_t q[32];  // two neighbours of the lane's 64 elements each
    bool beyond = false;
    if (r < n * G) {
      const bf16* src = a.q + (size_t)(row0 + r / G) * a.n_q * HD + (size_t)(kvh * G + r % G) * HD;
      const uint32_t half = c & 1 ? 0x7632u : 0x5410u;
      Magnitudes mag;
#pragma unroll
      for (int ch = 0; ch < HD / 8; ++ch) {
        const uint4 x = load8<true>(src + ch * 8);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) mag.see(w[i]);
        if constexpr (SP == 1) q[4 * ch] = w[0], q[4 * ch + 1] = w[1], q[4 * ch + 2] = w[2], q[4 * ch + 3] = w[3];
        if constexpr (SP == 2) q[2 * ch] = __byte_perm(w[0], w[1], half), q[2 * ch + 1] = __byte_perm(w[2], w[3], half);
        if constexpr (SP == 4) q[ch] = c & 2 ? __byte_perm(w[1], w[3], half) : __byte_perm(w[0], w[2], half);
      }
      beyond = mag.beyond();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) q[i] = 0u;
    }
    const Quot den = quot_of(__fsqrt_rn((float)HD));
    const bool first = next_keys(0);
    const bool always = __syncthreads_or(beyond || first);  // products and sums apart: in all tiles for the queries (and for the first keys, which share the barrier)
    bool apart = always;                                    // in this tile
    const int len = s_len[r];
    float mx = -1e9f;
    for (int tl = 0; tl < n_tiles; ++tl) {
      const bool next = tl + 1 < n_tiles && next_keys(tl + 1);
      const unsigned char* kt = reinterpret_cast<const unsigned char*>(tile) + (tl & 1) * 64 * KROW + c * KROW;
      const int end = min(TK, max_len - tl * TK);  // (a warp's lanes go round together: its first key decides)
      float* s_out = S + tl * TK * R + r;
      const int seen = len - tl * TK;
      auto scores = [&](auto fused) {
#pragma unroll 1
        for (int k0 = warp * KS; k0 < end; k0 += NWARP * KS) {
          const int kk = k0 + ks;
          const unsigned char* kr = kt + kk * SP * KROW;
          float s[4][2];
          auto get = [&](int l, uint32_t (&w)[4]) {
            const uint4 x = *reinterpret_cast<const uint4*>(kr + (l << 4));
            w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
          };
          score_tree<decltype(fused)::value, 1>(s, 0, q, get);
#pragma unroll
          for (int m = 2; m >= 1; m >>= 1)  // strides 4 and 2
#pragma unroll
            for (int i = 0; i < m; ++i) add2(s[i][0], s[i][1], s[i + m][0], s[i + m][1]);
          float dot = __fadd_rn(s[0][0], s[0][1]);
#pragma unroll
          for (int m = SP / 2; m >= 1; m >>= 1) dot = __fadd_rn(dot, __shfl_xor_sync(0xffffffffu, dot, m));  // the head's last strides
          const float sc = SP == 2 ? quot1(dot, den) : __fmul_rn(dot, SP == 1 ? 0.125f : 0.0625f);  // by the square root of 64, 128, 256
          if (kk < seen) mx = fmaxf(mx, sc);
          if (c == 0 && kk < end) s_out[kk * R] = sc;
        }
      };
      if (apart) scores(std::false_type{});
      else scores(std::true_type{});
      apart = __syncthreads_or(next) || always;
    }
#pragma unroll
    for (int s = SP * R; s < 32; s <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
    if (lane < SP * R && c == 0) s_max[warp][lane / SP] = mx;
    __syncthreads();
  }
  const bool fetches = LT == NT || tid >= VT;
  // (the first values are on their way during the softmax)
  const int vtid = LT == NT ? tid : tid - VT;
  uint4 pre[AHEAD][PIECES];
  auto fetch = [&](uint4 (&pre)[PIECES], int tl) {
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
      const int e = (vtid + u * LT) * 8;
      pre[u] = load8<ANY>(row_of(min(tl * TK + e / HD, max_len - 1), values) + e % HD);
    }
  };
#pragma unroll
  for (int t = 0; t < AHEAD; ++t)
    if (fetches && t < n_tiles) fetch(pre[t], t);
  // ---- softmax
  {
    const int r = tid % R, len = s_len[r];
    float m = s_max[0][r];
#pragma unroll
    for (int w = 1; w < NWARP; ++w) m = fmaxf(m, s_max[w][r]);
    constexpr int KT = NT / R;  // a thread's positions are KT apart; it takes eight at a time, whose chains run side by side
    // Up to 4 KT positions: two at a time, the sums' loads in their own turn, plain divisions; the long forms are more instructions than there is work (cycles
    // of the three steps at 17 positions 600 1250 730, so 330 770 330; 17 rows of 14 heads of 64 by the operator 6.5 us, so 6.0; one row at 200 with
    // the short forms 11.4, with the long ones 9.9).
    auto exponentials = [&](auto turn) {
      constexpr int U = decltype(turn)::value;
      for (int k0 = tid / R; k0 < max_len; k0 += U * KT) {
        float e[U];
#pragma unroll
        for (int u = 0; u < U; ++u) e[u] = S[own_position(k0, u, KT, max_len) * R + r];
#pragma unroll
        for (int u = 0; u < U; ++u) e[u] = expf(__fsub_rn(e[u], m));
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k0 + u * KT < max_len) S[(k0 + u * KT) * R + r] = k0 + u * KT < len ? e[u] : 0.f;
      }
    };
    const bool few = max_len <= 4 * KT;
    if (few) exponentials(std::integral_constant<int, 2>{});
    else exponentials(std::integral_constant<int, 8>{});
    __syncthreads();
    if (tid < R) {  // one chain per virtual row; zeros behind a row's positions leave its sum as it is
      float sum = 0.f, e[16];
      int k = 0;
      if (few) {
        for (; k + 16 <= max_len; k += 16) {
#pragma unroll
          for (int i = 0; i < 16; ++i) e[i] = S[(k + i) * R + tid];
#pragma unroll
          for (int i = 0; i < 16; ++i) sum = __fadd_rn(sum, e[i]);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) e[i] = S[i * R + tid];
        for (; k + 16 <= max_len; k += 16) {
          float next[16];
          const float* p = S + min(k + 16, max_len - 16) * R + tid;
#pragma unroll
          for (int i = 0; i < 16; ++i) next[i] = p[i * R], sum = __fadd_rn(sum, e[i]);
#pragma unroll
          for (int i = 0; i < 16; ++i) e[i] = next[i];
        }
      }
      for (; k < max_len; ++k) sum = __fadd_rn(sum, S[k * R + tid]);
      s_sum[tid] = sum;
    }
    __syncthreads();
    if (few) {
      const float sum = s_sum[r];
#pragma unroll 2
      for (int k = tid / R; k < len; k += KT) S[k * R + r] = __fdiv_rn(S[k * R + r], sum);
    } else {
      constexpr int U = 8;
      const Quot sum = quot_of(s_sum[r]);
      for (int k0 = tid / R; k0 < len; k0 += U * KT) {
        float e[U];
#pragma unroll
        for (int u = 0; u < U; ++u) e[u] = S[own_position(k0, u, KT, len) * R + r];
        quot32(e, sum);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k0 + u * KT < len) S[(k0 + u * KT) * R + r] = e[u];
      }
    }
  }
  // ---- values: RP rows x 4 columns a lane; the threads that are left fetch the next tile
  const int vr = tid % (R / RP) * RP, d0 = tid / (R / RP) * 4;
  const int len[2] = {s_len[vr], s_len[vr + RP - 1]};  // (vr < R for the threads that only fetch, too)
  float o[RP][4];
#pragma unroll
  for (int i = 0; i < RP; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  auto next_values = [&](int tl) {  // widened once for all rows
    auto put = [&](uint4 (&pre)[PIECES]) {
      float* dst = tile + (tl & 1) * TILE + vtid * 8;
#pragma unroll
      for (int u = 0; u < PIECES; ++u) {
        const uint4 w = pre[u];
        *reinterpret_cast<float4*>(dst + u * LT * 8) = make_float4(lo2f(w.x), hi2f(w.x), lo2f(w.y), hi2f(w.y));
        *reinterpret_cast<float4*>(dst + u * LT * 8 + 4) = make_float4(lo2f(w.z), hi2f(w.z), lo2f(w.w), hi2f(w.w));
      }
      if (tl + AHEAD < n_tiles) fetch(pre, tl + AHEAD);
    };
    if (tl & 1) put(pre[1]);
    else put(pre[0]);
  };
  if (fetches) next_values(0);
  __syncthreads();
  for (int tl = 0; tl < n_tiles; ++tl) {
    if (fetches && tl + 1 < n_tiles) next_values(tl + 1);
    if (VT == NT || tid < VT) {
      const float* vt = tile + (tl & 1) * TILE + d0;
      const float* pt = S + (size_t)tl * TK * R + vr;
      constexpr int U = 4;  // positions whose operands are read ahead of the arithmetic on U others
      float4 x[2][U];
      float p[2][U][RP];
      auto read = [&](int b, int kk) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          x[b][u] = *reinterpret_cast<const float4*>(vt + (kk + u) * HD);
          if constexpr (RP == 2) {
            const float2 w = *reinterpret_cast<const float2*>(pt + (kk + u) * R);
            p[b][u][0] = w.x, p[b][u][1] = w.y;
          } else {
            p[b][u][0] = pt[(kk + u) * R];
          }
        }
      };
      auto add = [&](int i, float w, const float4& v) {
        o[i][0] = __fmaf_rn(w, v.x, o[i][0]), o[i][1] = __fmaf_rn(w, v.y, o[i][1]);
        o[i][2] = __fmaf_rn(w, v.z, o[i][2]), o[i][3] = __fmaf_rn(w, v.w, o[i][3]);
      };
      auto use = [&](int b) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int i = 0; i < RP; ++i) add(i, p[b][u][i], x[b][u]);
      };
      const int all = min(TK, min_len - tl * TK) / (2 * U) * (2 * U);  // (all rows see these)
      int kk = 0;
      if (all > 0) {
        read(0, 0);
        for (; kk < all; kk += 2 * U) {
          read(1, kk + U);
          use(0);
          read(0, min(kk + 2 * U, all - U));  // (never behind the scores)
          use(1);
        }
      }
      const int end = min(TK, max(len[0], len[RP - 1]) - tl * TK);  // (negative for lanes without a row)
      for (; kk < end; kk += U) {  // (loads U at a time here as well; one position after the other took as long as the rest of the values at 17)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int at = min(kk + u, end - 1);
          x[0][u] = *reinterpret_cast<const float4*>(vt + at * HD);
#pragma unroll
          for (int i = 0; i < RP; ++i) p[0][u][i] = pt[at * R + i];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int i = 0; i < RP; ++i)
            if (tl * TK + kk + u < len[i]) add(i, p[0][u][i], x[0][u]);
      }
    }
    __syncthreads();
  }
  if (VT < NT && tid >= VT) return;
#pragma unroll
  for (int i = 0; i < RP; ++i) {
    if (vr + i >= n * G) continue;
    bf16* dst = a.out + (size_t)(row0 + (vr + i) / G) * a.n_q * HD + (size_t)(kvh * G + (vr + i) % G) * HD + d0;
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
      if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0) *reinterpret_cast<uint32_t*>(dst + c) = pack2(f2bf(o[i][c]), f2bf(o[i][c + 1]));
      else dst[c] = f2bf(o[i][c]), dst[c + 1] = f2bf(o[i][c + 1]);
    }
  }
}

template <int NP, int R, bool ANY>
cudaError_t launch_rows(const AttnArgs& a, int rows, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(attention_ref_rows_kernel<NP, R, ANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  if (e != cudaSuccess) return e;
  return launch_k(attention_ref_rows_kernel<NP, R, ANY>, dim3((a.n_tok + rows - 1) / rows, a.kv.n_kv), dim3(NT), smem, st, a, rows);
}

}  // namespace

// The most virtual rows whose scores leave room for two CTAs on an SM and whose tiles still make two CTAs for every SM, else fewer: a
// tile shares its key and value rows among its virtual rows, but a short launch needs CTAs, and more than 76 KB of scores cost
// the second CTA.  Measured (us, 32 / 16 / 8 virtual rows; one block per row and head): 500 rows behind 300 positions, 14 heads on 2, 64
// wide 84 / 79 / 104; 820.  64 rows behind 800: 62 / 41 / 30; 291.  One row at 801: 56 / 38 / 29; 120.  512 rows: 63 / 46 / 59.  12 heads on
// 2, 128 wide, 500 rows behind 300: - / 137 / 166; 981.
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
  const size_t smem = (2 * TILE + (size_t)a.max_kv_len * virtual_rows + page_ints(a)) * sizeof(float);
  const bool any = a.k_pages || (reinterpret_cast<uintptr_t>(a.kv.pool) & 15) != 0;  // (a pool's rows are multiples of 128 bytes apart)
#define QIE_ROWS(NP, R)                            \
  if (a.kv.hd == 64 * NP && virtual_rows == R) {   \
    return any ? launch_rows<NP, R, true>(a, rows, smem, st) : launch_rows<NP, R, false>(a, rows, smem, st); \
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
