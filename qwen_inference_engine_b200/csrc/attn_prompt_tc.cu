// attn_prompt_tc.cu -- causal prompt attention over the paged KV pool on tcgen05 / TMEM, head sizes 64 and 128, pages of 16 positions
// (fast numerics; the contract of attn_prefill_fast.cu: rows are consecutive positions of one sequence, keys and values are in the pool).
//
// A CTA owns 128 query rows of one head and walks the causal range in tiles of 64 keys; two CTAs share an SM.
//   S = Q K^T  : tcgen05.mma, 128 x 64 fp32 in one of two TMEM buffers, issued two tiles ahead of its softmax, behind the product that
//                read the weights there
//   softmax    : warps 0-3, one thread per row (= TMEM lane): 64 scores in registers, no exchange between threads.  The weights go back over
//                the scores' columns as bf16, where the second product takes its A operand from
//   O += P V   : accumulates in TMEM; where a maximum grew, the row's warp scales O behind its exponentials, when the product of the
//                tile before is in.  (A reference that lags the maximum by up to 2^8 saves 3 % and costs 4 % of precision: the largest weight
//                is then no power of two and gets rounded.)
//   warp 4     : the products.  warp 5: copies, TMA boxes of a page x 64 columns with the 128-byte swizzle into two stages of K and of V.
//                (One warp for both was the bottleneck: a request costs it 50 cycles, 400 - 600 a tile.)
// Query tiles whose first 64 rows see at most `two_term` positions keep the weights as bf16 hi + lo pairs (two products): every row has them for
// which attn_prefill_fast.cu, with its tiles of 64 rows, does, and up to 64 rows more.
// Short launches split a query tile's keys over a cluster (pick_parts), summed through distributed shared memory.
// What bounds it: the chain of a tile, 1500 - 1600 cycles alone on an SM: exponentials 620 (512 are the unit's floor), maximum 190, scaling O
// 140 - 220 and waiting for its product 140, waiting for S 250, TMEM reads and writes 140.  14 heads of 64, 3000 rows: 105 us with mma.sync,
// 45 here; 12 heads of 128, 4096 rows: 140 us (128-key tiles, O in registers, one CTA an SM), 72 here = 720 TFLOP/s.
// Every wait has a limit; when one runs out the CTA stores values that are not numbers and reports it.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "cluster.cuh"
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "pack.cuh"
#include "tc_ptx.cuh"

namespace qie {
namespace {

constexpr int TQ = 128, TK = 64;
constexpr int QBLK = TQ * 128, KBLK = TK * 128;  // [rows][64 columns] bf16 in 8-row swizzle atoms
constexpr int NSOFT = 128, NTHR = NSOFT + 64;      // + a warp for the products, one for the copies
constexpr int MAXP = 1024;                       // page ids in shared memory
constexpr uint32_t TMEM_COLS = 256;              // two tiles of scores, O

template <int HD>
struct PromptSmem {
  static constexpr int TILE = HD / 64 * KBLK;    // K and V: two stages each
  static constexpr int Q = 0, K = HD / 64 * QBLK, V = K + 2 * TILE, BAR = V + 2 * TILE, PAGES = BAR + 128, END = PAGES + MAXP * 4 + 1024;
  // A CTA allocates TMEM_COLS of an SM's 512 columns and a third one would wait for them while it keeps its cluster's other CTAs from
  // ending: shared memory is reserved so that a third does not fit (head size 64 needs 53 of the 76 KB).  Registers alone do not promise it.
  static constexpr int TOTAL = END > 76 * 1024 ? END : 76 * 1024;
  static_assert(512 / TMEM_COLS == 2 && 3 * (TOTAL + 1024) > 228 * 1024, "no more CTAs on an SM than its TMEM columns allow");
  static_assert(2 * (TOTAL + 1024 + 2 * TQ * 4 + 64) <= 228 * 1024, "two of them");
  static constexpr int PITCH = (HD + 4) * 4;     // a part's O rows
  static_assert(TQ * PITCH <= BAR, "O rows fit over the operands");
};
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
      "%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// two scores at once: x * s + n, and a + b
__device__ __forceinline__ void fma2(float& x, float& y, unsigned long long s, unsigned long long n) {
  asm("{\n\t.reg .b64 v;\n\tmov.b64 v, {%0, %1};\n\tfma.rn.f32x2 v, v, %2, %3;\n\tmov.b64 {%0, %1}, v;\n\t}" : "+f"(x), "+f"(y) : "l"(s), "l"(n));
}
__device__ __forceinline__ void add2(float& a, float& b, float x, float y) {
  asm("{\n\t.reg .b64 u, v;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tadd.rn.f32x2 u, u, v;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "+f"(a), "+f"(b) : "f"(x), "f"(y));
}
__device__ __forceinline__ unsigned long long twice(float x) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
  return v;
}
template <int HD>
__global__ void __launch_bounds__(NTHR, 2) attn_prompt_tc_kernel(FastAttnArgs a, int two_term, int parts_max, int alone, const __grid_constant__ CUtensorMap kvm) {
  using SM = PromptSmem<HD>;
  constexpr int NB = HD / 64;  // column blocks
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int dead_s;
  __shared__ float s_max[TQ], s_sum[TQ];  // at the end: the part's reference maximum and sum of a row
  volatile int* dead = &dead_s;
  pdl_wait();
  pdl_trigger();
  const uint32_t s0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* sg = smem_raw + (s0 - smem_u32(smem_raw));
  // barriers in pairs, by the tile's parity
  const uint32_t bar_s = s0 + SM::BAR, bar_p = bar_s + 16, bar_o = bar_s + 32, bar_k = bar_s + 48, bar_v = bar_s + 64, slot = bar_s + 80;
  int* s_pages = reinterpret_cast<int*>(sg + SM::PAGES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // parts of a query tile are the CTAs of a cluster; then heads, longest query tiles first
  const int part = blockIdx.x % parts_max, h = blockIdx.x / parts_max, qt = gridDim.y - 1 - blockIdx.y, G = a.n_q / a.kv.n_kv, kvh = h / G;
  const int t0 = qt * TQ, n_rows = min(TQ, a.n_tok - t0), Dq = a.n_q * HD;
  const int* bt = a.block_table + (size_t)a.slot[t0] * a.max_pages;
  const int pos_first = a.pos[t0], kv_len = pos_first + n_rows, all_tiles = (kv_len + TK - 1) / TK, n_pages = (kv_len + 15) / 16;
  // The host knows the block table's width and not the sequence's length: where sharing out the tiles that there are saves fewer than the sum over
  // the cluster costs, its first CTA does them all and the others are done.
  const bool split = parts_max > 1 && all_tiles - (all_tiles + parts_max - 1) / parts_max > alone;
  if (!split && part > 0) return;
  const int parts = split ? parts_max : 1;
  const int per = (all_tiles + parts - 1) / parts, first = min(all_tiles, part * per), n_tiles = min(all_tiles, first + per) - first;
  const bool two = pos_first + min(n_rows, 64) <= two_term;
  if (tid == 0) {
    dead_s = 0;
    for (int i = 0; i < 2; ++i)
      mbar_init_tc(bar_s + 8 * i, 1), mbar_init_tc(bar_p + 8 * i, NSOFT), mbar_init_tc(bar_o + 8 * i, 1), mbar_init_tc(bar_k + 8 * i, 1), mbar_init_tc(bar_v + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == NSOFT / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = tid; i < min(MAXP, n_pages); i += NTHR) s_pages[i] = bt[i];
  if (n_tiles > 0)
    for (int i = tid; i < TQ * NB * 8; i += NTHR) {  // Q rows, those behind the chunk repeat the last (never stored)
      const int r = i / (NB * 8), ch = i - r * (NB * 8);
      cp_async16(s0 + SM::Q + (ch >> 3) * QBLK + r * 128 + (((ch & 7) ^ (r & 7)) << 4), a.q + (size_t)(t0 + min(r, n_rows - 1)) * Dq + (size_t)h * HD + ch * 8);
    }
  cp_async_commit();
  cp_async_wait<0>();
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(slot));
  const uint32_t t_o = tmem + 128;  // scores: columns 0 .. 63 and 64 .. 127, the weights over them

  if (warp == NSOFT / 32 + 1) {
    // ---- copies
    auto copy = [&](int t, int is_v) {  // 4 page chunks x NB column blocks; chunks behind the last page repeat it (their keys are masked)
      const int pg = lane / NB & 3, nb = lane % NB, pi = min((first + t) * 4 + pg, n_pages - 1), page = pi < MAXP ? s_pages[pi] : bt[pi];
      const int row = (((page * a.kv.n_layers + a.layer) * 2 + is_v) * a.kv.n_kv + kvh) * 16;
      const uint32_t bar = (is_v ? bar_v : bar_k) + 8u * (uint32_t)(t & 1), dst = s0 + (is_v ? SM::V : SM::K) + (t & 1) * SM::TILE + nb * KBLK + pg * 16 * 128;
      if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)SM::TILE) : "memory");
      __syncwarp();
      if (lane < 4 * NB)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     ::"r"(dst), "l"(&kvm), "r"(bar), "r"(nb * 64), "r"(row)
                     : "memory");
      __syncwarp();
    };
    for (int t = 0; t < min(2, n_tiles); ++t) copy(t, 0), copy(t, 1);
    for (int t = 0; t + 2 < n_tiles; ++t) {
      const uint32_t b = 8u * (uint32_t)(t & 1), ph = (uint32_t)((t >> 1) & 1);
      mbar_wait_tc(bar_s + b, ph, dead);  // S(t) has read K(t)
      copy(t + 2, 0);
      mbar_wait_tc(bar_o + b, ph, dead);  // P V(t) has read V(t)
      copy(t + 2, 1);
    }
  } else if (warp == NSOFT / 32) {
    // ---- products
    const uint32_t id_s = idesc_tc(TQ, TK, false), id_o = idesc_tc(TQ, HD, true);
    const uint64_t dq = desc_k_tc(s0 + SM::Q), dk = desc_k_tc(s0 + SM::K), dv = desc_mn_tc(s0 + SM::V, KBLK);  // (steps are sums: in units of 16 bytes)
    auto issue_s = [&](int t) {
      const uint64_t k = dk + (uint64_t)((t & 1) * (SM::TILE >> 4));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_tc()) {
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          umma_tc(tmem + (uint32_t)((t & 1) * TK), dq + (uint64_t)(((kk >> 2) * QBLK + (kk & 3) * 32) >> 4), k + (uint64_t)(((kk >> 2) * KBLK + (kk & 3) * 32) >> 4), id_s,
                  kk != 0);
        umma_commit_tc(bar_s + 8u * (uint32_t)(t & 1));
      }
      __syncwarp();
    };
    auto issue_pv = [&](int t) {
      const uint32_t p = tmem + (uint32_t)((t & 1) * TK);
      const uint64_t v = dv + (uint64_t)((t & 1) * (SM::TILE >> 4));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_tc()) {
        for (int lo = 0; lo < (two ? 2 : 1); ++lo)  // 32 columns of hi, 32 of lo
#pragma unroll
          for (int kk = 0; kk < TK / 16; ++kk) umma_ts_tc(t_o, p + (uint32_t)(lo * 32 + kk * 8), v + (uint64_t)(kk * 128), id_o, t > 0 || kk > 0 || lo > 0);
        umma_commit_tc(bar_o + 8u * (uint32_t)(t & 1));
      }
      __syncwarp();
    };
    for (int t = 0; t < min(2, n_tiles); ++t) {
      mbar_wait_tc(bar_k + 8 * t, 0, dead);
      issue_s(t);
    }
    for (int t = 0; t < n_tiles; ++t) {
      const uint32_t b = 8u * (uint32_t)(t & 1), ph = (uint32_t)((t >> 1) & 1);
      mbar_wait_tc(bar_v + b, ph, dead);
      mbar_wait_tc(bar_p + b, ph, dead);
      issue_pv(t);
      if (t + 2 < n_tiles) {
        mbar_wait_tc(bar_k + b, ph ^ 1, dead);
        mbar_wait_tc(bar_o + b, ph, dead);  // S(t + 2) goes over the weights that P V(t) reads, and only products on one accumulator are
        issue_s(t + 2);                     // ordered by their issue.  (The weights of t + 1 are a softmax away: nothing is lost.)
      }
    }
  } else {
    // ---- softmax: this thread's row
    const int row = tid, my_pos = pos_first + min(row, n_rows - 1);
    const uint32_t la = (uint32_t)(warp * 32) << 16;
    const float sl2 = a.scale_log2;
    float m_ref = -INFINITY, l_run = 0.f;
    auto tiles = [&](auto pairs) {  // pairs: weights as hi + lo
      for (int t = 0; t < n_tiles; ++t) {
        const uint32_t b = 8u * (uint32_t)(t & 1), ph = (uint32_t)((t >> 1) & 1), ts = tmem + la + (uint32_t)((t & 1) * TK);
        const int last = my_pos - (first + t) * TK;  // the last key of the tile that the row sees
        mbar_wait_tc(bar_s + b, ph, dead);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[64];
        ld32(ts, r);
        ld32(ts + 32, r + 32);
        wait_ld();
        if (last < TK - 1) {
#pragma unroll
          for (int j = 0; j < TK; ++j)
            if (j > last) r[j] = 0xff800000u;  // -inf
        }
        float mx[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mx[i] = max3(__uint_as_float(r[i]), __uint_as_float(r[i + 4]), __uint_as_float(r[i + 8]));
#pragma unroll
        for (int j = 12; j + 8 <= TK; j += 8)
#pragma unroll
          for (int i = 0; i < 4; ++i) mx[i] = max3(mx[i], __uint_as_float(r[j + i]), __uint_as_float(r[j + 4 + i]));
#pragma unroll
        for (int i = 0; i < 4; ++i) mx[i] = fmaxf(mx[i], __uint_as_float(r[60 + i]));
        const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2);
        const bool grow = __any_sync(0xffffffffu, m_new > m_ref);
        const float f = m_new > -INFINITY ? ex2_tc(m_ref - m_new) : 1.f;
        m_ref = m_new;
        const unsigned long long s2 = twice(sl2), n2 = twice(m_new > -INFINITY ? -m_new : 0.f);
        float rs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < TK; c += 32) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float e0 = __uint_as_float(r[c + 2 * e]), e1 = __uint_as_float(r[c + 2 * e + 1]);
            fma2(e0, e1, s2, n2);
            e0 = ex2_tc(e0), e1 = ex2_tc(e1);
            add2(rs[2 * (e & 1)], rs[2 * (e & 1) + 1], e0, e1);
            hi[e] = pack2f(e0, e1);
            if constexpr (pairs.value) lo[e] = pack2f(e0 - lo2f(hi[e]), e1 - hi2f(hi[e]));
          }
          tmem_st16_tc(ts + c / 2, hi);
          if constexpr (pairs.value) tmem_st16_tc(ts + 32 + c / 2, lo);
        }
        l_run = l_run * f + ((rs[0] + rs[1]) + (rs[2] + rs[3]));
        if (grow && t > 0) {  // scale O by the new reference; behind the exponentials the product of the tile before is in
          mbar_wait_tc(bar_o + (b ^ 8u), (uint32_t)(((t - 1) >> 1) & 1), dead);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int c = 0; c < HD; c += 64) {
            uint32_t o[64];
            ld32(t_o + la + c, o);
            ld32(t_o + la + c + 32, o + 32);
            wait_ld();
#pragma unroll
            for (int j = 0; j < 64; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
            st32(t_o + la + c, o);
            st32(t_o + la + c + 32, o + 32);
          }
        }
        if (first + t == all_tiles - 1 && kv_len % TK) {  // value rows behind the sequence: whatever the pool holds there must not meet a zero weight
          mbar_wait_tc(bar_v + b, ph, dead);
          if (row < TK && (first + t) * TK + row >= kv_len)
#pragma unroll
            for (int i = 0; i < NB * 8; ++i)
              asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(s0 + SM::V + (t & 1) * SM::TILE + (i >> 3) * KBLK + row * 128 + (i & 7) * 16), "r"(0u) : "memory");
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        wait_st();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive_tc(bar_p + b);
      }
    };
    if (two) tiles(std::true_type{});
    else tiles(std::false_type{});
    if (n_tiles > 0) mbar_wait_tc(bar_o + 8u * (uint32_t)((n_tiles - 1) & 1), (uint32_t)(((n_tiles - 1) >> 1) & 1), dead);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t r[32];
    if (parts == 1) {
      const float inv = *dead ? __int_as_float(0x7fc00000) : 1.f / l_run;
      bf16* dst = a.out + (size_t)(t0 + row) * Dq + (size_t)h * HD;
#pragma unroll
      for (int c = 0; c < HD; c += 32) {
        ld32(t_o + la + c, r);
        wait_ld();
        if (row < n_rows) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = pack2f(__uint_as_float(r[j + 2 * i]) * inv, __uint_as_float(r[j + 2 * i + 1]) * inv);
            *reinterpret_cast<uint4*>(dst + c + j) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    } else {
      s_max[row] = m_ref, s_sum[row] = *dead ? __int_as_float(0x7fc00000) : l_run;
      if (n_tiles > 0) {  // this part's O: fp32 rows over the operands, which no product reads any more
        const uint32_t dst = s0 + (uint32_t)row * SM::PITCH;
#pragma unroll
        for (int c = 0; c < HD; c += 32) {
          ld32(t_o + la + c, r);
          wait_ld();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (uint32_t)(c + j) * 4u), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3]) : "memory");
        }
      }
    }
  }
  if (parts > 1) {
    // ---- every part sums its share of the rows over the cluster
    cluster_sync_all();
    const int rows = TQ / parts, n_parts = (all_tiles + per - 1) / per;  // parts without tiles have nothing to add
    for (int i = tid; i < rows * (HD / 4); i += NTHR) {
      const int row = part * rows + i / (HD / 4), c = i % (HD / 4) * 4;
      if (row >= n_rows) break;
      float m[8], l[8], top = -INFINITY;
      float4 o[8];
#pragma unroll
      for (int p = 0; p < 8; ++p)
        if (p < n_parts) {
          uint32_t am, as, ao;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(am) : "r"(smem_u32(&s_max[row])), "r"(p));
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(as) : "r"(smem_u32(&s_sum[row])), "r"(p));
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ao) : "r"(s0 + (uint32_t)row * SM::PITCH + (uint32_t)c * 4u), "r"(p));
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(m[p]) : "r"(am) : "memory");
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l[p]) : "r"(as) : "memory");
          asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(o[p].x), "=f"(o[p].y), "=f"(o[p].z), "=f"(o[p].w) : "r"(ao) : "memory");
          top = fmaxf(top, m[p]);
        }
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      float total = 0.f;
#pragma unroll
      for (int p = 0; p < 8; ++p)
        if (p < n_parts) {
          // A row sees nothing of a part behind its position.  A sum that is no number (a wait ran out, or no score of the part is one) counts
          // whatever the maximum beside it.
          const float f = l[p] != l[p] ? l[p] : m[p] > -INFINITY ? ex2_tc(m[p] - top) : 0.f;
          if (f != 0.f) {
            sum.x += o[p].x * f, sum.y += o[p].y * f, sum.z += o[p].z * f, sum.w += o[p].w * f;
            total += l[p] * f;
          }
        }
      const float inv = 1.f / total;
      *reinterpret_cast<uint2*>(a.out + (size_t)(t0 + row) * Dq + (size_t)h * HD + c) = make_uint2(pack2f(sum.x * inv, sum.y * inv), pack2f(sum.z * inv, sum.w * inv));
    }
    cluster_sync_all();  // nobody leaves while others read its rows
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == NSOFT / 32) {
    drain_tc(dead);
    if (lane == 0) report_tc(dead, a.status);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// Parts of a query tile's keys, one CTA of a cluster each: the longest tile sets the time of a short launch, but the sum over the cluster
// costs.  The estimate is tiles of the longest row / parts x time of a tile (more where CTAs share an SM) + the sum; all CTAs run
// at once and most have an SM to themselves.  Measured (us; 1, 2, 4, 8 parts): 128 rows behind 1500, 12 heads of 128: 29 24 19 14; 16 rows behind 800, 14 heads of 64: 15 12
// 10 10; 1000 rows behind 1000, 12 heads of 128: 35 30 40 49; 2000 rows, 12 heads of 128: 36 41 53 85; 64 rows of 64: 5.3 8.5 7.8 7.1.
template <int HD>
int pick_parts(const FastAttnArgs& a, int* alone) {
  const float tile = HD == 64 ? 0.78f : 0.85f, shared = HD == 64 ? 1.25f : 1.45f;
  const float sum[4] = {0.f, HD == 64 ? 3.9f : 6.3f, HD == 64 ? 2.5f : 4.2f, HD == 64 ? 1.8f : 3.2f};
  const int tiles = (a.max_kv_len + TK - 1) / TK;
  const long ctas = (long)a.n_q * ((a.n_tok + TQ - 1) / TQ);
  int best = 0;
  float cost = 0.f;
  for (int i = 0; i < 4; ++i) {
    const int p = 1 << i;
    // (240 and 200 CTAs of 148 SMs' 296 places: clusters do not find every gap.  700 rows, 12 heads of 128: 15, with 288 CTAs 22)
    if (p > 1 && ctas * p * 148 > (HD == 64 ? 240L : 200L) * a.num_sms) break;
    const float c = (float)((tiles + p - 1) / p) * tile * (ctas * p > a.num_sms ? shared : 1.f) + sum[i];
    if (i == 0 || c < cost) cost = c, best = i;
  }
  *alone = (int)(sum[best] / tile);
  return 1 << best;
}

template <int HD>
cudaError_t launch_hd(const FastAttnArgs& a, int two_term, const TensorMap2D& kvm, cudaStream_t st) {
  int alone = 0;
  const int parts = pick_parts<HD>(a, &alone);
  static PerDeviceOnce set;
  if (set.need()) {
    cudaError_t e = cudaFuncSetAttribute(attn_prompt_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, PromptSmem<HD>::TOTAL);
    if (e != cudaSuccess) return e;
    set.done();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(a.n_q * parts, (a.n_tok + TQ - 1) / TQ);
  cfg.blockDim = dim3(NTHR);
  cfg.dynamicSmemBytes = PromptSmem<HD>::TOTAL;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int na = 0;
  if (parts > 1) {
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = parts;
    at[na].val.clusterDim.y = at[na].val.clusterDim.z = 1;
    ++na;
  }
  if (g_use_pdl) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, attn_prompt_tc_kernel<HD>, a, two_term, parts, alone, *reinterpret_cast<const CUtensorMap*>(&kvm));
}

// a pair of CTAs: the wait is the first one's, the report the other one's
__global__ void __cluster_dims__(2) wait_selftest_kernel(int* status) {
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int dead_s;
  const bool one = threadIdx.x == 0;
  if (one) dead_s = 0, mbar_init_tc(smem_u32(&bar), 1);
  cluster_sync_all();
  if (blockIdx.x == 0 && one) {
    mbar_wait_tc(smem_u32(&bar), 0, &dead_s);
    tell_other_tc(&dead_s);
  }
  cluster_sync_all();
  if (blockIdx.x == 1 && one) report_tc(&dead_s, status);
}

}  // namespace

cudaError_t launch_wait_selftest(int* status, cudaStream_t st) {
  wait_selftest_kernel<<<2, 32, 0, st>>>(status);
  return cudaGetLastError();
}

bool attention_prompt_tc_takes(const FastAttnArgs& a) {
  return (a.kv.hd == 64 || a.kv.hd == 128) && a.kv.page_size == 16 && a.n_q % a.kv.n_kv == 0 &&
         ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.kv.pool)) & 15) == 0 &&
         (unsigned long long)a.kv.n_pages * a.kv.n_layers * 2ull * a.kv.n_kv * 16 < (1ull << 31);
}

cudaError_t launch_attention_prompt_tc(const FastAttnArgs& a, int two_term, cudaStream_t st) {
  if (a.n_tok == 0) return cudaSuccess;
  if (!attention_prompt_tc_takes(a)) return cudaErrorInvalidValue;
  TensorMap2D kvm;
  cudaError_t e = make_tensor_map_kv(&kvm, a.kv.pool, (unsigned long long)a.kv.n_pages * a.kv.n_layers * 2ull * a.kv.n_kv * 16, a.kv.hd, 16);
  if (e != cudaSuccess) return e;
  return a.kv.hd == 64 ? launch_hd<64>(a, two_term, kvm, st) : launch_hd<128>(a, two_term, kvm, st);
}

}  // namespace qie
