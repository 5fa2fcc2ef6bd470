// attn_ref_decode.cu -- reference-order attention of rows on their own (decode steps, few rows of a prompt), bit for bit what
// attention_ref_kernel (ops_ref_order.cu) and the reference's selfattention (layers/src/self_attension.cu:10-149) compute per row and head.
//
// CTA = one row and up to eight query heads of one kv head, whose key and value rows are read once for all of them.
//   scores : a lane has two rows of 64 keys (one of 128) in registers as bf16 pairs, the queries are broadcast from shared memory in the order that the
//            tree takes them, so that few partial sums are open.  fma.rn.f32.bf16 takes the products, two of the tree's first stride in one rounding where
//            that is exact (Magnitudes), packed sums the rest.  Each warp asks for groups of its own and computes them, no barrier between.
//   softmax: a warp per head; the serial sum is walked by every lane from broadcast quads
//   values : lane = two columns of one or two heads, o = fma(p, v, o) over ascending positions; a ring of value rows is kept full by bulk copies
// What bounds it, cycles of a CTA at 2000 positions, 7 heads of 64 (35.8 us for 64 rows; 50 in the persistent kernel, 71 by attn_ref_rows.cu's tiles of one
// row): scores 19k (products and sums alone 13k: 1.3 cycles of a scheduler a product), largest and exponentials 3k, serial sum 9.4k (4.2 an addition), quotients
// 1.5k, values 24k (9.4 a position: a scheduler takes a 4-byte load a lane every 4 cycles and a broadcast quad every 8, so 8 for two heads).
// Rows of four instead of two columns a lane, widened values in shared memory, four heads of one column: 10 to 12 a position.
#include <cuda.h>
#include <math_constants.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "head_math.cuh"
#include "kernels.h"
#include "launch.h"
#include "ref_math.cuh"
#include "tc_ptx.cuh"

namespace qie {
namespace {

constexpr int NW = 8, NT = NW * 32 + 32;  // warps that compute, and one that copies values
constexpr int SLOT = 8192;                // bytes of a warp's keys: 64 rows of 64, 32 of 128
constexpr int VTILE = 16384;              // bytes of a stage of values: 128 rows of 64, 64 of 128
constexpr int MAX_STAGES = 5;
constexpr int OFF_DEAD = 8 * (2 * MAX_STAGES + NW), HEADER = 256;  // barriers, a wait ran out
static_assert(OFF_DEAD + 4 <= HEADER, "header");

__host__ __device__ inline int score_pitch(int max_kv_len) { return (max_kv_len + 127) & ~127; }
struct Layout {
  int q, pages, score, k, v, total;  // byte offsets
};
__host__ __device__ inline Layout layout_of(int hd, int hp, int max_kv_len, int page_size, int stages, bool post) {
  Layout l;
  l.q = HEADER;  // the queries; behind them the row's own key and value (post)
  l.pages = l.q + (hp + (post ? 2 : 0)) * hd * 2;
  l.score = l.pages + ((((max_kv_len + page_size - 1) / page_size) * 4 + 15) & ~15);
  l.k = (l.score + hp * score_pitch(max_kv_len) * 4 + 1023) & ~1023;  // (the copies' swizzle counts rows from there)
  l.v = l.k + NW * SLOT;
  l.total = l.v + stages * VTILE;
  return l;
}

__device__ __forceinline__ void bar_compute() { asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory"); }
__device__ __forceinline__ bool bar_or(bool x) {
  uint32_t y;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred p, 1, %2, p;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(y) : "r"((uint32_t)x), "n"(NW * 32) : "memory");
  return y != 0;
}
__host__ __device__ constexpr int brev(int u, int bits) {
  int r = 0;
  for (int i = 0; i < bits; ++i) r |= ((u >> i) & 1) << (bits - 1 - i);
  return r;
}
__host__ __device__ constexpr int ones_at_end(int u) {
  int n = 0;
  while (u & 1) ++n, u >>= 1;
  return n;
}

// The scores of RW rows of a lane against one head: leaves are the pairs m and m + half of a row, m in bit-reversed order, so that a partial sum meets its
// partner as early as there is one.
template <int NP, int RW, bool FUSED>
__device__ __forceinline__ void dots(float (&out)[RW], const uint32_t (&k)[RW][32 * NP], uint4 (&w)[4], const uint4* __restrict__ qc, const uint4* __restrict__ qn) {
  constexpr int BITS = NP == 1 ? 4 : 5, LEAVES = 16 * NP, QUADS = 8 * NP;
  float st[RW][BITS][2], x[RW][2];
#pragma unroll
  for (int u = 0; u < QUADS; ++u) {
    const uint4 q = w[u & 3];
    w[u & 3] = u + 4 < QUADS ? qc[u + 4] : qn[u + 4 - QUADS];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int leaf = 2 * u + s, m = brev(leaf, BITS), t = ones_at_end(leaf);
      const uint32_t qa = s ? q.z : q.x, qb = s ? q.w : q.y;
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        float a[2], p[2];
        fma16(p[0], p[1], qa, k[r][m], -0.f, -0.f);
        if constexpr (FUSED) {
          fma16(a[0], a[1], qb, k[r][m + LEAVES], p[0], p[1]);
        } else {
          fma16(a[0], a[1], qb, k[r][m + LEAVES], -0.f, -0.f);
          add2(a[0], a[1], p[0], p[1]);
        }
#pragma unroll
        for (int b = 0; b < BITS; ++b)
          if (b < t) add2(a[0], a[1], st[r][b][0], st[r][b][1]);
        if (t < BITS) st[r][t][0] = a[0], st[r][t][1] = a[1];
        x[r][0] = a[0], x[r][1] = a[1];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RW; ++r) out[r] = __fadd_rn(x[r][0], x[r][1]);
}

// o[h] = fma(p[h][k], v[k], o[h]) for ascending positions: two columns of NH heads.  v: the lane's columns of the first position, rows of PITCH bytes.
// Weights and values of U positions are read ahead of the arithmetic on U others.
template <int NH, int PITCH>
struct Weigh {
  static constexpr int U = 8;
  uint32_t v[2][U];
  float4 p[2][NH][U / 4];
  __device__ __forceinline__ void load(int b, const unsigned char* v0, const float* p0, const float* p1) {
#pragma unroll
    for (int j = 0; j < U; ++j) v[b][j] = *reinterpret_cast<const uint32_t*>(v0 + j * PITCH);
#pragma unroll
    for (int j = 0; j < U / 4; ++j) {
      p[b][0][j] = *reinterpret_cast<const float4*>(p0 + 4 * j);
      if (NH == 2) p[b][NH - 1][j] = *reinterpret_cast<const float4*>(p1 + 4 * j);
    }
  }
  __device__ __forceinline__ void use(int b, float2 (&o)[2]) const {
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const float2 x = make_float2(lo2f(v[b][j]), hi2f(v[b][j]));
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        const float4 q = p[b][h][j / 4];
        const float w = j % 4 == 0 ? q.x : j % 4 == 1 ? q.y : j % 4 == 2 ? q.z : q.w;
        o[h] = __ffma2_rn(make_float2(w, w), x, o[h]);
      }
    }
  }
  template <int ROWS>
  __device__ __forceinline__ void all(const unsigned char* v0, const float* p0, const float* p1, float2 (&o)[2]) {
    load(0, v0, p0, p1);
#pragma unroll
    for (int c = 0; c < ROWS / U; ++c) {
      if (c + 1 < ROWS / U) load((c + 1) & 1, v0 + (c + 1) * U * PITCH, p0 + (c + 1) * U, p1 + (c + 1) * U);
      use(c & 1, o);
    }
  }
  __device__ __forceinline__ void some(const unsigned char* v0, const float* p0, const float* p1, int n, float2 (&o)[2]) {
    int k = 0;
#pragma unroll 1
    for (; k + 2 * U <= n; k += 2 * U) {
      load(0, v0 + k * PITCH, p0 + k, p1 + k);
      load(1, v0 + (k + U) * PITCH, p0 + k + U, p1 + k + U);
      use(0, o);
      use(1, o);
    }
#pragma unroll 1
    for (; k < n; ++k) {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(v0 + k * PITCH);
      const float2 x = make_float2(lo2f(w), hi2f(w));
      o[0] = __ffma2_rn(make_float2(p0[k], p0[k]), x, o[0]);
      if (NH == 2) o[1] = __ffma2_rn(make_float2(p1[k], p1[k]), x, o[1]);
    }
  }
};

// POST: the queries, the key and the value of the row come from the projections: bias, head norm and rotary position as in qkv_post_kernel (head_ops.cu), queries back in place,
// key and value into the pool by the first part of a kv head.  The last position's key and value are read from shared memory, all others from the pool.
template <int NP, bool POST>
__global__ void __launch_bounds__(NT, 1) attention_ref_decode_kernel(const AttnRefCall a, const int hp, const int stages, const int box, const __grid_constant__ CUtensorMap kvm,
                                                                     const QkvPostArgs post) {
  constexpr int HD = 64 * NP, RW = 2 / NP, GK = 32 * RW, ROW = HD * 2, WORDS = 32 * NP, TV = VTILE / ROW;
  extern __shared__ __align__(1024) unsigned char smem[];
  volatile int* const dead = reinterpret_cast<volatile int*>(smem + OFF_DEAD);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = a.n_q / a.kv.n_kv, parts = (G + hp - 1) / hp;
  const int kvh = blockIdx.x / parts, part = blockIdx.x - kvh * parts, b = blockIdx.y;
  const int h0 = kvh * G + part * hp, hs = min(hp, G - part * hp);
  const Layout lay = layout_of(HD, hp, a.max_kv_len, a.kv.page_size, stages, POST);
  const uint32_t bars = smem_u32(smem);  // full and empty of the values' stages, full of the warps' keys
  auto vfull = [&](int s) { return bars + 8 * s; };
  auto vempty = [&](int s) { return bars + 8 * (MAX_STAGES + s); };
  const uint32_t kfull = bars + 8 * (2 * MAX_STAGES + warp);
  int* const pages = reinterpret_cast<int*>(smem + lay.pages);
  float* const score = reinterpret_cast<float*>(smem + lay.score);
  const int SP = score_pitch(a.max_kv_len);
  // values: a warp's unit is one head (up to eight units) or two, and 64 of its columns
  const int pair = hs * NP > (NP == 1 ? 4 : 8) ? 2 : 1, units = (hs + pair - 1) / pair * NP;
  if (tid == 0) {
    *dead = 0;
    for (int s = 0; s < stages; ++s) mbar_init_tc(vfull(s), 1), mbar_init_tc(vempty(s), units);
    for (int w = 0; w < NW; ++w) mbar_init_tc(bars + 8 * (2 * MAX_STAGES + w), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Where the kernel in front of this one writes nothing but the queries and the row's own position (a.early), all else is read before it ends.
  if (!a.early) pdl_wait();
  const int len = a.pos[b] + 1, ready = a.early && !POST ? len - 1 : len;  // positions that are there already, or are not read
  const int kept = POST ? len - 1 : len;                                    // positions whose values come from the pool
  unsigned char* const own = smem + lay.q + hp * HD * 2;                    // (POST) the row's key, then its value
  bf16* const out = a.out + (size_t)b * a.n_q * HD + (size_t)h0 * HD;
  if (len <= 0) {  // no position: zeros, and no page to read
    if (a.early) pdl_wait();
    for (int i = tid; i < hs * HD; i += NT) out[i] = f2bf(0.f);
    return;
  }
  const int ng = (len + GK - 1) / GK;  // groups of keys: warp g modulo NW has group g
  const int psz = a.kv.page_size, shift = (psz & (psz - 1)) == 0 ? __ffs(psz) - 1 : -1;
  {
    const int* bt = a.block_table + (size_t)a.slot[b] * a.max_pages;
    for (int i = tid; i <= (len - 1) / psz; i += NT) pages[i] = bt[i];
  }
  __syncthreads();

  if (warp == NW) {
    // ---- copies of values: whole pages of rows, one request each
    const size_t page_stride = a.kv.page_stride();
    const bf16* const vbase = a.kv.chunk(0, a.layer, 1, kvh);
    int s = 0;
    uint32_t ph = 1;  // (the first pass over the ring waits for nothing)
    bool waits = a.early;
    for (int k0 = 0; k0 < kept; k0 += TV) {
      const int n = min(TV, kept - k0);
      if (waits && (k0 + n > ready || ph == 0)) pdl_wait(), waits = false;  // (a wait's limit counts this kernel's time: stages come free behind the wait only)
      if (!mbar_wait_tc(vempty(s), ph, dead)) break;
      const uint32_t full = vfull(s), dst = smem_u32(smem + lay.v + s * VTILE);
      if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(n * ROW) : "memory");
      __syncwarp();
      const int first = k0 / psz, last = (k0 + n - 1) / psz;
      for (int pg = first + lane; pg <= last; pg += 32) {
        const int from = max(k0, pg * psz), to = min(k0 + n, (pg + 1) * psz);
        const bf16* src = vbase + (size_t)pages[pg] * page_stride + (size_t)(from - pg * psz) * HD;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(dst + (from - k0) * ROW), "l"(src), "r"((to - from) * ROW), "r"(full) : "memory");
      }
      if (++s == stages) s = 0, ph ^= 1;
    }
    __syncwarp();
  } else {
    // ---- scores
    const unsigned char* const slot = smem + lay.k + warp * SLOT;
    const uint32_t slot_u = smem_u32(slot);
    // A group of keys: boxes of `box` rows of a page, their 64 columns behind one another.  Each warp asks for its own: the warp that copies the values takes
    // 160 cycles for a request and could not keep up (41 us instead of 36).
    auto copy = [&](int g) {
      const int n = min(GK, len - g * GK), boxes = (n + box - 1) / box;
      if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(kfull), "r"(boxes * box * ROW) : "memory");
      __syncwarp();
      if (lane < boxes * NP) {
        const int i = lane / NP, half = lane % NP, k = g * GK + i * box, pg = shift >= 0 ? k >> shift : k / psz;
        const int row = (((pages[pg] * a.kv.n_layers + a.layer) * 2) * a.kv.n_kv + kvh) * psz + (k - pg * psz);
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     ::"r"(slot_u + half * GK * 128 + i * box * 128), "l"(&kvm), "r"(kfull), "r"(half * 64), "r"(row) : "memory");
      }
    };
    const bool asked = warp < ng && (warp + 1) * GK <= ready;
    if (asked || (POST && warp < ng)) copy(warp);
    // queries in the tree's order: quad u is pairs m0, m0 + half, m1, m1 + half of leaves 2 u and 2 u + 1
    constexpr int BITS = NP == 1 ? 4 : 5;
    Magnitudes mag;
    if constexpr (POST) {
      using Hd = Head<NP>;
      const int at = tid / Hd::LH, l = tid % Hd::LH, kind = at < hs ? 0 : at == hs ? 1 : 2;  // a head of the CTA: queries, the key, the value
      const int ps = len - 1;
      const bf16 *bias = kind == 0 ? post.q_bias : kind == 1 ? post.k_bias : post.v_bias, *w = kind == 0 ? post.q_norm_w : post.k_norm_w;
      const float *co = post.cos_t + (size_t)ps * Hd::HALF, *si = post.sin_t + (size_t)ps * Hd::HALF;
      if (at <= hs) {  // (on their way while the projections run)
        const int first = post.rope_half ? 8 * l : 4 * l, second = post.rope_half ? 8 * l + 4 : Hd::HALF / 2 + 4 * l;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(co + first)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(co + second)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(si + first)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(si + second)));
      }
      pdl_wait();
      if (warp * 32 / Hd::LH <= hs + 1) {  // (whole warps: the sum of squares is an exchange)
        const bf16* src = kind == 0 ? post.q_in + (size_t)b * post.q_in_stride + (size_t)(h0 + at) * HD : (kind == 1 ? post.k : post.v) + (size_t)b * post.kv_stride + (size_t)kvh * HD;
        const size_t head = kind == 0 ? h0 + at : kvh;
        Hd x;
        x.template load<true>(src, l);
        if (bias) x.template add_bias<true>(bias + head * HD, l);
        const float sum = x.squares();
        if (kind != 2) {
          if (w) x.template norm<true>(sum, w, l, post.eps);
          if (post.rope_half) x.template rope_half<true>(co, si, l);
          else x.template rope<true>(co, si, l);
        }
        if (kind == 0) {
          x.template store<true>(post.q + (size_t)b * a.n_q * HD + head * HD, l);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t pair = pack2f(x.x[2 * j], x.x[2 * j + 1]);
            mag.see(pair);
            reinterpret_cast<uint32_t*>(smem + lay.q)[at * WORDS + 2 * (int)(__brev(4 * l + j % 4) >> (32 - BITS)) + j / 4] = pair;
          }
        } else if (at <= hs + 1) {
          x.template store<true>(reinterpret_cast<bf16*>(own) + (kind - 1) * HD, l);
          if (part == 0) x.template store<true>(a.kv.chunk(pages[ps / psz], a.layer, kind - 1, kvh) + (size_t)(ps % psz) * HD, l);
        }
      }
    } else {
      if (a.early) pdl_wait();
      if (!asked && warp < ng) copy(warp);
      for (int i = tid; i < hs * WORDS; i += NW * 32) {
        const int h = i / WORDS, e = i % WORDS, leaf = e >> 1;
        const uint32_t w = *reinterpret_cast<const uint32_t*>(a.q + (size_t)b * a.n_q * HD + (size_t)(h0 + h) * HD + 2 * (brev(leaf, BITS) + (e & 1) * 16 * NP));
        mag.see(w);
        reinterpret_cast<uint32_t*>(smem + lay.q)[i] = w;
      }
    }
    const bool q_beyond = bar_or(mag.beyond());
    const Quot den = quot_of(__fsqrt_rn((float)HD));
    const uint4* const q4 = reinterpret_cast<const uint4*>(smem + lay.q);
    constexpr int QUADS = 8 * NP;
    uint32_t kph = 0;
    for (int g = warp; g < ng; g += NW, kph ^= 1) {
      if (!mbar_wait_tc(kfull, kph, dead)) break;
      uint32_t k[RW][WORDS];
      // Keys of at least 2^-63 and below 2^65, whose exponents' upper bits differ, against queries between 2^-62 and 2^62: no product leaves what is
      // exact (Magnitudes).  A test by two instructions a word, 400 cycles a group less than the lowest and the highest one of Magnitudes.
      uint32_t differ = 0xffffffffu;
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        uint32_t row = 0xffffffffu;
        const bool is_own = POST && g * GK + 32 * r + lane == len - 1;
#pragma unroll
        for (int c = 0; c < 8 * NP; ++c) {
          const uint4 t = *reinterpret_cast<const uint4*>(is_own ? own + 16 * c : slot + c / 8 * GK * 128 + (lane + 32 * r) * 128 + ((c % 8 ^ (lane & 7)) << 4));
          const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) k[r][4 * c + i] = w[i], row &= w[i] ^ (w[i] << 1);
        }
        differ &= g * GK + 32 * r + lane < len ? row : 0xffffffffu;
      }
      const bool apart = __any_sync(0xffffffffu, (differ & 0x40004000u) != 0x40004000u) || q_beyond;
      if (g + NW < ng) copy(g + NW);  // (the vote has brought the warp together behind the last of the slot's reads)
      uint4 w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) w[u] = q4[u];
      auto heads = [&](auto fused) {
#pragma unroll 1
        for (int h = 0; h < hs; ++h) {
          float d[RW];
          dots<NP, RW, decltype(fused)::value>(d, k, w, q4 + QUADS * h, q4 + QUADS * (h + 1 < hs ? h + 1 : h));
#pragma unroll
          for (int r = 0; r < RW; ++r) {
            const int at = g * GK + 32 * r + lane;
            const float sc = NP == 1 ? __fmul_rn(d[r], 0.125f) : quot1(d[r], den);  // by the square root of 64 or 128
            if (at < len) score[h * SP + at] = sc;
          }
        }
      };
      if (apart) heads(std::false_type{});
      else heads(std::true_type{});
    }
    bar_compute();
    // ---- softmax: a warp per head
    if (warp < hs) {
      float* const s = score + warp * SP;
      const int n4 = len & ~127;
      float m = -1e9f;
#pragma unroll 4
      for (int k = 4 * lane; k < n4; k += 128) {
        const float4 t = *reinterpret_cast<const float4*>(s + k);
        m = fmaxf(m, fmaxf(fmaxf(t.x, t.y), fmaxf(t.z, t.w)));
      }
      for (int k = n4 + lane; k < len; k += 32) m = fmaxf(m, s[k]);
      m = warp_max(m);
      bool slow = false;  // an exponential below 2^-99
      auto exponential = [&](float x) {
        const float y = __fsub_rn(x, m);
        slow = slow || y < -68.f;
        return expf(y);
      };
#pragma unroll 2
      for (int k = 4 * lane; k < n4; k += 128) {
        const float4 t = *reinterpret_cast<const float4*>(s + k);
        *reinterpret_cast<float4*>(s + k) = make_float4(exponential(t.x), exponential(t.y), exponential(t.z), exponential(t.w));
      }
      for (int k = n4 + lane; k < len; k += 32) s[k] = exponential(s[k]);
      slow = __any_sync(0xffffffffu, slow);  // (and every lane's stores are there)
      float sum = 0.f;
      {
        const int n16 = len & ~15;
        float4 e[2][4];
        auto read = [&](int b, int k) {
#pragma unroll
          for (int u = 0; u < 4; ++u) e[b][u] = *reinterpret_cast<const float4*>(s + k + 4 * u);
        };
        auto add = [&](int b) {
#pragma unroll
          for (int u = 0; u < 4; ++u) sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, e[b][u].x), e[b][u].y), e[b][u].z), e[b][u].w);
        };
        read(0, 0);
        int k = 0;
#pragma unroll 1
        for (; k + 32 <= n16; k += 32) {
          read(1, k + 16);
          add(0);
          read(0, min(k + 32, SP - 16));
          add(1);
        }
        if (k < n16) add(0), k += 16;
        for (; k < len; ++k) sum = __fadd_rn(sum, s[k]);
      }
      const Quot d = quot_of(sum);
      __syncwarp();
      if (!slow && d.ok) {
#pragma unroll 2
        for (int k = 4 * lane; k < n4; k += 128) {
          float4 t = *reinterpret_cast<const float4*>(s + k);
          *reinterpret_cast<float4*>(s + k) = make_float4(quot32_fast(t.x, d), quot32_fast(t.y, d), quot32_fast(t.z, d), quot32_fast(t.w, d));
        }
        for (int k = n4 + lane; k < len; k += 32) s[k] = quot32_fast(s[k], d);
      } else {
#pragma unroll 1
        for (int k = lane; k < len; k += 32) s[k] = quot1(s[k], d);
      }
    }
    bar_compute();
    pdl_trigger();
    // ---- values
    if (warp < units) {
      const int hu = warp / NP * pair, col = warp % NP * 64 + 2 * lane, nh = min(pair, hs - hu);
      const float* const p0 = score + hu * SP;
      const float* const p1 = nh == 2 ? p0 + SP : p0;  // (a last head without a second: the same chain twice, in the code of the others)
      float2 o[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      auto go = [&](auto heads) {
        int s = 0;
        uint32_t ph = 0;
        Weigh<decltype(heads)::value, ROW> w;
#pragma unroll 1
        for (int k0 = 0; k0 < kept; k0 += TV) {
          if (!mbar_wait_tc(vfull(s), ph, dead)) break;
          const unsigned char* v = smem + lay.v + s * VTILE + col * 2;
          if (k0 + TV <= kept) w.template all<TV>(v, p0 + k0, p1 + k0, o);
          else w.some(v, p0 + k0, p1 + k0, kept - k0, o);
          __syncwarp();
          if (lane == 0) mbar_arrive_tc(vempty(s));
          if (++s == stages) s = 0, ph ^= 1;
        }
        if constexpr (POST) w.some(own + HD * 2 + col * 2, p0 + kept, p1 + kept, 1, o);
      };
      if (pair == 2) go(std::integral_constant<int, 2>{});
      else go(std::integral_constant<int, 1>{});
      const bool bad = *dead;
      for (int h = 0; h < nh; ++h) {
        const float2 x = bad ? make_float2(CUDART_NAN_F, CUDART_NAN_F) : o[h];
        *reinterpret_cast<uint32_t*>(out + (size_t)(hu + h) * HD + col) = pack2(f2bf(x.x), f2bf(x.y));
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    drain_tc(dead);
    report_tc(dead, a.status);
  }
}

}  // namespace

static int heads_of(const AttnArgs& a, int num_sms, int* stages, bool post) {
  const int G = a.n_q / a.kv.n_kv, hd = a.kv.hd;
  auto at16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if ((hd != 64 && hd != 128) || a.k_pages || a.kv.page_size % 8 || !at16(a.kv.pool) || !at16(a.q) || !at16(a.out)) return 0;
  if ((unsigned long long)a.kv.n_pages * a.kv.n_layers * 2 * a.kv.n_kv * a.kv.page_size >= 1ull << 31) return 0;  // rows of the tensor map
  const int tasks = a.n_tok * a.kv.n_kv;
  int parts = (G + 7) / 8;
  while (parts < G && (long)tasks * (parts + 1) <= num_sms) ++parts;
  for (int hp = (G + parts - 1) / parts; hp >= 1; --hp)
    for (int st = MAX_STAGES; st >= 2; --st)
      if (layout_of(hd, hp, a.max_kv_len, a.kv.page_size, st, post).total <= 226 * 1024) {
        *stages = st;
        return hp;
      }
  return 0;
}

static cudaError_t launch_decode(const AttnRefCall& a, int heads, int stages, const QkvPostArgs* post, cudaStream_t st) {
  const int G = a.n_q / a.kv.n_kv, parts = (G + heads - 1) / heads;
  const size_t smem = layout_of(a.kv.hd, heads, a.max_kv_len, a.kv.page_size, stages, post != nullptr).total;
  int box = 8;  // rows of a copy: as many as a page and a group hold
  while (a.kv.page_size % (2 * box) == 0 && 2 * box * a.kv.hd * 2 <= SLOT) box *= 2;
  TensorMap2D kvm;
  cudaError_t e = make_tensor_map_kv(&kvm, a.kv.pool, (unsigned long long)a.kv.n_pages * a.kv.n_layers * 2ull * a.kv.n_kv * a.kv.page_size, a.kv.hd, box);
  if (e != cudaSuccess) return e;
  auto go = [&](auto kernel, PerDeviceOnce& set) {
    if (set.need()) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
      if (e != cudaSuccess) return e;
      set.done();
    }
    return launch_k(kernel, dim3(parts * a.kv.n_kv, a.n_tok), dim3(NT), smem, st, a, heads, stages, box, *reinterpret_cast<const CUtensorMap*>(&kvm), post ? *post : QkvPostArgs{});
  };
  static PerDeviceOnce set[3];
  if (post) return go(attention_ref_decode_kernel<1, true>, set[2]);
  return a.kv.hd == 64 ? go(attention_ref_decode_kernel<1, false>, set[0]) : go(attention_ref_decode_kernel<2, false>, set[1]);
}

// A CTA takes 5 to 6 us before its positions count, so several waves of short contexts are quicker by one block per row and head or per row (a kv head's heads side by side).  us a step of
// four layers, 1024 wide, by those kernels and by this one: a head a kv head, nine waves and more up to 128 positions (16 heads of 64 on 16, 150 rows at 20 397 617, 256 at 20 560 961,
// at 60 773 1022, at 100 995 1070; 8 on 8, 256 at 20 429 601, at 100 676 657); parts of a kv head's heads, three waves up to 128 positions (16 on 1, 200 at 20 276 312, at
// 100 295 324), from four waves on up to 512 of 64, 1024 of 128 (256 at 20 292 351, at 200 339 384, at 400 386 425; 16 of 128 on 1 314 370, 401 437, 498 535).  All else is quicker
// here or nearly so (256 rows at 20 against the kernels before: 14 heads of 64 on 2 340 350, 12 of 128 on 2 353 364; 200 of 4 on 4 323 362).
bool attention_ref_decode_step(const AttnArgs& a, int num_sms, int heads) {
  const int G = a.n_q / a.kv.n_kv;
  const long ctas = (long)a.n_tok * a.kv.n_kv * ((G + heads - 1) / heads), waves = (ctas + num_sms - 1) / num_sms;
  if (G == 1) return waves < 9 || a.max_kv_len > 128;
  if (G > 8) return waves < 3 || a.max_kv_len > (waves == 3 ? 128 : 8 * a.kv.hd);
  return true;
}

// Heads of a CTA, 0 where this kernel does not take the call.
int attention_ref_decode_heads(const AttnArgs& a, int num_sms, int* stages) { return heads_of(a, num_sms, stages, false); }

cudaError_t launch_attention_ref_decode(const AttnRefCall& a, int heads, int stages, cudaStream_t st) { return launch_decode(a, heads, stages, nullptr, st); }

// What launch_qkv_post and this kernel do, in one launch: the store and the way back of the queries and a start of a kernel less, and the keys of a step are
// asked for while the projections run.  us a step of 24 layers, 14 heads of 64 on 2, two launches and one: 64 rows at 2048 positions 1712 1693, 16 at 500 994 971, 5 at 100 892
// 860.  Heads of 128 keep two: 28 layers, 12 heads on 2, 32 rows at 500 1759 1777, 8 at 100 1457 1488, 16 at 1000 1870 1906 (64 at 300 1834 1821).  Nor where a row or a
// table is off a 16-byte boundary.
static int post_heads(const AttnRefCall& a, const QkvPostArgs& p, int num_sms, int* stages) {
  uintptr_t at = 0;
  for (const void* q : {(const void*)p.q, (const void*)p.q_in, (const void*)p.k, (const void*)p.v, (const void*)p.q_norm_w, (const void*)p.k_norm_w, (const void*)p.cos_t,
                        (const void*)p.sin_t, (const void*)p.q_bias, (const void*)p.k_bias, (const void*)p.v_bias})
    at |= reinterpret_cast<uintptr_t>(q);
  if (a.kv.hd != 64 || !a.decode || !a.early || a.n_tok < 1 || at % 16 || p.q_in_stride % 8 || p.kv_stride % 8) return 0;
  const int heads = heads_of(a, num_sms, stages, true);
  return heads && attention_ref_decode_step(a, num_sms, heads) ? heads : 0;
}

bool attention_ref_post_takes(const AttnRefCall& a, const QkvPostArgs& p, int num_sms) {
  int stages = 0;
  return post_heads(a, p, num_sms, &stages) > 0;
}

cudaError_t launch_attention_ref_post(const AttnRefCall& a, const QkvPostArgs& p, int num_sms, cudaStream_t st) {
  int stages = 0;
  const int heads = post_heads(a, p, num_sms, &stages);
  return heads ? launch_decode(a, heads, stages, &p, st) : cudaErrorInvalidValue;
}

}  // namespace qie
