// gemm_tcgen05.cu -- C[M,Nout] = A[M,K] * W[Nout,K]^T on the 5th-gen tensor cores
// (tcgen05.mma, accumulator in TMEM, operands staged by TMA): batched decode
// (M = sequences) and prefill (M = prompt tokens).  Without a split over K the results are the bits of the
// reference's wmma kernel (layers/src/matrix_mul.cu:165-288; launch_gemm_ref_rows); fast numerics
// may split K (a fixed-order sum of the splits) and match it within the bf16 tolerance.
//
// Swap-AB: the weight tile is the UMMA "A" operand (M = 128 weight rows = 128 TMEM lanes),
// the activations are the "B" operand (N = BN tokens, 16..128; up to 256 in the persistent kernel), both K-major, 128-byte
// swizzle, BLOCK_K = 64 bf16.  D[w_row, token] lives in TMEM: lane = weight row, column =
// token.  Decode is HBM-bound on the weights: each CTA streams its [128 x Kslice] weight
// slab exactly once through a TMA/mbarrier ring.
//   warp 0 : TMA producer (one elected lane); weight tiles are requested BEFORE the PDL
//            wait on the previous kernel, activation tiles after it
//   warp 1 : TMEM alloc/dealloc + MMA issuer (one elected lane, tcgen05.mma / commit)
//   warps 2-5 : epilogue, TMEM -> registers (tcgen05.ld 32x32b) -> ...
// Split-K without a workspace: the S K-slices of one output tile are the S CTAs of a
// thread-block CLUSTER (grid.y = cluster dim).  Each CTA parks its fp32 partial tile in its
// own shared memory, the cluster synchronises, and CTA r sums rows [r*128/S, (r+1)*128/S)
// of all S partials through distributed shared memory (ld.shared::cluster) in rank order
// -- deterministic -- and applies the epilogue.  No partials in HBM/L2, no second launch.
// Epilogues keep the reference's rounding points:
//   EPI_STORE     C = bf16(acc)
//   EPI_RESIDUAL  x = bf16(float(x) + float(bf16(acc)))
//   EPI_SILU_MUL  h = bf16(bf16(up) * bf16(silu(bf16(gate))));  the CTA's 128-lane tile is
//                 64 gate rows (lanes 0-63) + the same 64 up rows (lanes 64-127)
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "cluster.cuh"
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "tc_ptx.cuh"

namespace qie {

static constexpr int BM = 128;  // weight rows per CTA (UMMA M)
static constexpr int BK = 64;   // k elements per stage (128 B rows, SWIZZLE_128B)
template <int BN, bool HALF, int KB, int TM>
struct TcCfg {  // HALF: a ring that leaves room for a second CTA (16 tokens); KB: k-blocks of a stage; TM: weight rows of a tile
  static constexpr int STAGES = TM == 64 ? 220 / (KB * (8 + BN / 8)) : (HALF ? 6 : BN <= 16 ? 12 : BN <= 32 ? 11 : BN <= 64 ? 9 : 7) / KB;  // what 227 KiB hold
};

// ------------------------------------------------------------------ PTX wrappers (tc_ptx.cuh has the rest)
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
template <int CTAS = 1>  // 2: the barrier may be the other CTA's of a pair
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  if constexpr (CTAS == 2) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
    return;
  }
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(c1), "r"(c2)
      : "memory");
}
// gate and up as one matrix (make_tensor_map_gate_up)
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c1, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(c1), "r"(0), "r"(c3)
      : "memory");
}
template <int CTAS = 1>
__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t cols) {
  if constexpr (CTAS == 2) {  // a warp of either CTA
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    return;
  }
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int CTAS = 1>
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  if constexpr (CTAS == 2) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
    return;
  }
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  tmem_ld16_tc(taddr, r);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void mark_bad(uint32_t (&r)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) r[j] = 0x7fc00000u;
}

__device__ __forceinline__ float silu_ref_f(float x) {
  float sg = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x)));
  return __fmul_rn(x, sg);
}

// tolerance-mode SiLU for the epilogue of prompts (more than 128 rows): ex2.approx + rcp.approx (relative error ~1e-6, far inside the bf16 rounding
// that follows) instead of expf + an IEEE division (~35 instructions per element on the epilogue warps that pace the
// K = 1536 gate/up tiles)
__device__ __forceinline__ float silu_fast_f(float x) {
  return __fdividef(x, 1.0f + __expf(-x));
}

struct TcSeg {
  int rows;   // weight rows of this segment
  int tile0;  // first tile index
  int ld;     // row stride of its output
  bf16* out;  // its first output column
};

struct TcArgs {
  int M, K;
  int nseg, n_tiles, splits, kb_per_split, kb_total;
  int epi, dual, w_static;
  int ref_silu;    // persistent kernel: SiLU as the reference computes it (expf, IEEE division); the others always do
  int bn, stages;  // persistent kernel: tokens of a tile (a multiple of 16), stages of its ring
  int tokens_first;  // ... neighbouring CTAs have a weight tile's token tiles, else a token tile's weight tiles
  int* status;     // host word that a wait which ran out sets, or null
  int vec;         // persistent kernel: rows of the output take 16-byte stores
  int staged;  // splits == 1 and 8-element aligned outputs: epilogue through a bf16 tile in shared memory, 16-byte global accesses
  TcSeg seg[3];
};

// DUAL: gate/up tiles (EPI_SILU_MUL), instantiations of their own: with their epilogue in the others' code each product took 0.1 to 0.2 us more (us, 128 rows of
// 896 x 4864 5.06 4.91, of 1536 x 8960 7.17 6.87, prompts of 300 rows of 1.5B widths, four layers, 457 446).  The epilogue of the others stays in one branch, and the compiler is told
// that one CTA an SM is enough: without the two, tiles of 64 tokens took 0.1 us more (us in graphs of twenty alike, without, with: 1000 rows of 896 x 896 5.10 4.97, 128 of 896 x 4864 5.01
// 4.88, 512 of 1536 x 1536 6.75 6.61; a decode step of 16 sequences at 500 positions 978 971).
template <int BN, bool HALF, int KB, int TM, bool AHEAD, bool DUAL>
__global__ void __launch_bounds__(DUAL ? 256 : 192, 1) gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w0,
                                                            const __grid_constant__ CUtensorMap map_w1,
                                                            const __grid_constant__ CUtensorMap map_w2,
                                                            const __grid_constant__ CUtensorMap map_x, TcArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int dead_s;
  volatile int* const dead = &dead_s;
  if (threadIdx.x == 0) dead_s = 0;  // (a barrier follows before any wait)
  constexpr int A_BLK = TM * BK * 2, A_BYTES = KB * A_BLK;  // 16 KiB a k-block (8 of 64 rows)
  constexpr int B_BLK = BN * BK * 2, B_BYTES = KB * B_BLK;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
  constexpr int TC_STAGES = TcCfg<BN, HALF, KB, TM>::STAGES;
  static_assert(TC_STAGES * STAGE_BYTES >= BN * (BM + 32) * 4, "reduction tile must fit in the pipeline ring");
  // 1024-byte alignment for SWIZZLE_128B (same offset in every CTA of a cluster: the dynamic
  // shared window starts at the same address in all CTAs of a kernel)
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = smem0 + TC_STAGES * STAGE_BYTES;  // full[S], empty[S], tmem_full, slot
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (TC_STAGES + s); };
  const uint32_t tmem_full_bar = bars + 8u * (2 * TC_STAGES);
  const uint32_t slot = tmem_full_bar + 8u;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x, split = blockIdx.y, ttile = blockIdx.z;
  int si = 0;
  while (si + 1 < g.nseg && tile >= g.seg[si + 1].tile0) ++si;
  // dual (gate/up): one tile = 64 gate rows + the same 64 up rows; segment 0 = gate map, 1 = up map
  const CUtensorMap* map_w = DUAL ? &map_w0 : (si == 0 ? &map_w0 : (si == 1 ? &map_w1 : &map_w2));
  const int row0 = DUAL ? tile * (BM / 2) : (tile - g.seg[si].tile0) * TM;
  const int seg_rows = g.seg[si].rows, ld = g.seg[si].ld;
  bf16* const out = g.seg[si].out;
  const int kb0 = split * g.kb_per_split;
  const int kb1 = min(g.kb_total, kb0 + g.kb_per_split);
  const int nkb = max(0, kb1 - kb0), nst = (nkb + KB - 1) / KB;  // k-blocks, stages of them
  const int tok_base = ttile * BN;

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map_w) : "memory");
    if (DUAL && KB == 1) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w1) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    for (int s = 0; s < TC_STAGES; ++s) {
      mbar_init_tc(full_bar(s), 1);
      mbar_init_tc(empty_bar(s), 1);
    }
    mbar_init_tc(tmem_full_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(slot));

  auto load_w = [&](int i, int s) {
    const uint32_t sa = smem0 + s * STAGE_BYTES;
    if constexpr (KB > 1) {  // one request for the k-blocks of a stage (behind the matrix: zeros, which no product reads)
      if constexpr (DUAL) tma_load_4d(sa, &map_w0, full_bar(s), row0, kb0 + i * KB);
      else tma_load_3d(sa, map_w, full_bar(s), row0, kb0 + i * KB);
      return;
    }
    if (DUAL) {  // two 64-row boxes: gate rows -> lanes 0-63, up rows -> lanes 64-127
      tma_load_2d(sa, &map_w0, full_bar(s), (kb0 + i) * BK, row0);
      tma_load_2d(sa + A_BYTES / 2, &map_w1, full_bar(s), (kb0 + i) * BK, row0);
    } else {
      tma_load_2d(sa, map_w, full_bar(s), (kb0 + i) * BK, row0);
    }
  };

  auto load_x = [&](int i, int s) {
    const uint32_t sb = smem0 + s * STAGE_BYTES + A_BYTES;
    if constexpr (KB > 1) tma_load_3d(sb, &map_x, full_bar(s), tok_base, kb0 + i * KB);
    else tma_load_2d(sb, &map_x, full_bar(s), (kb0 + i) * BK, tok_base);
  };

  // The loops of both roles carry stage, parity and descriptors from step to step.  With a division by the stage count, a clock read per wait and descriptors built per product a step took 0.27 us
  // whatever the tile's width (76 steps at K = 4864: 22.8 us on an idle chip), then 0.18 us (15.7 us).  The products of a step
  // themselves take 0.025 us at 16 tokens, 0.27 us at 256.  With two k-blocks a stage (KB) a k-block takes 0.13 us: us before and after, in graphs, in the
  // reference's order: 64 rows of 896 x 896 4.6 4.1, 4864 x 896 15.7 12.3, 8960 x 1536 27.3 20.7, 18944 x 3584 56.2 42.8; 512 rows 4864 x 896 16.6 13.7.  Tiles of 64 weight rows and four
  // k-blocks a stage, the wait for the next stage between the products: 4.1 4.0, 12.6 8.4, 21.2 13.6, 51.9 35; 14.0 11.5 (launch_gemm_tcgen05).
  if (warp == 0) {
    if (elect_tc()) {
      // Weights never depend on the previous kernel: start streaming them BEFORE waiting for
      // it (programmatic dependent launch), as soon as its CTAs leave room for the ring.
      const int pre = g.w_static ? min(nst, TC_STAGES) : 0;
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(full_bar(i), STAGE_BYTES);
        load_w(i, i);
      }
      pdl_wait();  // activations are produced by the previous kernel
      for (int i = 0; i < pre; ++i) load_x(i, i);
      int s = pre == TC_STAGES ? 0 : pre;
      uint32_t ph = pre == TC_STAGES ? 0 : 1;  // the first pass over the ring waits for nothing
      for (int i = pre; i < nst; ++i) {
        if (!mbar_wait_tc(empty_bar(s), ph, dead)) break;
        mbar_expect_tx(full_bar(s), STAGE_BYTES);
        load_w(i, s);
        load_x(i, s);
        if (++s == TC_STAGES) s = 0, ph ^= 1;
      }
      pdl_trigger();  // (one thread's counts for the block)
    }
    __syncwarp();
  } else if (warp == 1) {
    pdl_wait();  // (a wait's limit counts this kernel's time, not its predecessor's)
    const uint32_t idesc = idesc_tc(TM, BN, false);
    const uint64_t ad0 = desc_k_tc(smem0), bd0 = desc_k_tc(smem0 + A_BYTES);
    int s = 0;
    uint32_t ph = 0;
    auto products = [&](int i, int b, int st) {  // of a k-block of stage i, which lies in slot st
      if (b == 0 || i * KB + b < nkb)
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {  // 16 bf16 = 32 bytes along K inside the 128-byte swizzle atom
          const uint64_t step = (uint64_t)(st * (STAGE_BYTES >> 4));
          umma_tc(tmem_base, ad0 + step + b * (A_BLK >> 4) + 2 * k, bd0 + step + b * (B_BLK >> 4) + 2 * k, idesc, (i | b | k) != 0);
        }
    };
    if constexpr (AHEAD) {
      // Many stages: whether the next one is there is asked in front of a stage's last products.  The tensor core has about four products ahead (160 cycles at 16 tokens
      // and 128 rows, 39 each; 94 of 64 rows, 23 each), less than a wait behind a commit takes.
      if (elect_tc()) {
        bool there = false;
        for (int i = 0; i < nst; ++i) {
          if (!there) mbar_wait_tc(full_bar(s), ph, dead);
          tc_fence_after();
          const int st = s;
          if (++s == TC_STAGES) s = 0, ph ^= 1;
#pragma unroll
          for (int b = 0; b < KB; ++b) {
            if (b == KB - 1) there = mbar_ready_tc(full_bar(s), ph);
            products(i, b, st);
          }
          umma_commit_tc(empty_bar(st));  // frees the smem stage once the MMAs have read it
        }
        umma_commit_tc(tmem_full_bar);  // accumulator complete
      }
    } else {
      for (int i = 0; i < nst; ++i) {
        mbar_wait_tc(full_bar(s), ph, dead);
        tc_fence_after();
        if (elect_tc()) {
#pragma unroll
          for (int b = 0; b < KB; ++b) products(i, b, s);
          umma_commit_tc(empty_bar(s));
        }
        __syncwarp();
        if (++s == TC_STAGES) s = 0, ph ^= 1;
      }
      if (elect_tc()) umma_commit_tc(tmem_full_bar);
    }
    __syncwarp();
  }

  // ================= epilogue =================
  if (g.staged) {
    // No split-K (prefill / large batches): lane = weight row, column = token, but the output is
    // [token][weight row] -- per-lane 2-byte global accesses would serialise (and the residual's
    // read-modify-write would expose one DRAM round trip per token).  The tile is transposed
    // through shared memory as bf16 [token][128 rows] (the pipeline ring is idle by now), then
    // written -- or read-modified-written -- with independent 16-byte accesses, a 256-byte
    // contiguous run per token.  Rounding points are the reference's (R3 / R8 / R9).
    constexpr uint32_t PITCH = TM * 2;
    const uint32_t stg = smem0;
    auto drain = [&]() {  // four warps
      const int qd = warp & 3;
      pdl_wait();  // `out` may still be read (residual) by the previous kernel
      if (nkb > 0) {
        mbar_wait_tc(tmem_full_bar, 0, dead);
        tc_fence_after();
      }
      const bool bad = *dead;
      // (64 rows lie in the lower half of each quarter's lanes)
      const int lane_row = TM == 64 ? qd * 16 + lane : qd * 32 + lane;
      const bool has_row = TM == 128 || lane < 16;
#pragma unroll
      for (int c0 = 0; c0 < BN; c0 += 16) {
        uint32_t r[16];
        if (nkb > 0) {
          tmem_ld16(tmem_base + ((uint32_t)(qd * 32) << 16) + c0, r);
          if (bad) mark_bad(r);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = 0u;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const unsigned short hb = __bfloat16_as_ushort(f2bf(__uint_as_float(r[j])));
          if (has_row) asm volatile("st.shared.u16 [%0], %1;" ::"r"(stg + (uint32_t)(c0 + j) * PITCH + (uint32_t)lane_row * 2u), "h"(hb) : "memory");
        }
      }
      tc_fence_before();
    };
    if constexpr (DUAL) {
      if (warp >= 2 && warp < 6) drain();
      __syncthreads();
      // gate rows sit in lanes 0-63, the matching up rows in lanes 64-127.  All eight warps: 64 tokens are 4096 SiLUs of some 40 instructions
      pdl_wait();
      const int total = min(BN, g.M - tok_base) * (BM / 8);
      for (int c = threadIdx.x; c < total; c += blockDim.x) {
        const int tok = c >> 4, part = c & 15;
        const int w_row = row0 + part * 4;
        if (w_row >= seg_rows) continue;
        const uint32_t at = stg + (uint32_t)tok * PITCH + (uint32_t)part * 8u;
        uint32_t gs[2], us[2], o2[2];
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(gs[0]), "=r"(gs[1]) : "r"(at) : "memory");
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(us[0]), "=r"(us[1]) : "r"(at + BM) : "memory");
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float a0 = __fmul_rn(lo2f(us[e]), bf2f(f2bf(silu_ref_f(lo2f(gs[e])))));
          const float a1 = __fmul_rn(hi2f(us[e]), bf2f(f2bf(silu_ref_f(hi2f(gs[e])))));
          o2[e] = pack2(f2bf(a0), f2bf(a1));
        }
        *reinterpret_cast<uint2*>(out + (size_t)(tok_base + tok) * ld + w_row) = make_uint2(o2[0], o2[1]);
      }
    } else if (warp >= 2) {
      drain();
      asm volatile("bar.sync 2, 128;" ::: "memory");  // the four warps that drain
      const int t = threadIdx.x - 64;
      auto lds128 = [](uint32_t addr) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
        return v;
      };
      const int total = min(BN, g.M - tok_base) * (TM / 8);
      for (int c = t; c < total; c += 4 * 128) {
        uint4 y[4], x[4];
        bf16* dst[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int cc = c + u * 128;
          const int tok = cc >> (TM == 128 ? 4 : 3), part = cc & (TM / 8 - 1);
          const int w_row = row0 + part * 8;
          ok[u] = cc < total && w_row < seg_rows;
          dst[u] = out + (size_t)(tok_base + tok) * ld + w_row;
          if (ok[u]) {
            y[u] = lds128(stg + (uint32_t)tok * PITCH + (uint32_t)part * 16u);
            if (g.epi == EPI_RESIDUAL) x[u] = *reinterpret_cast<const uint4*>(dst[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (!ok[u]) continue;
          if (g.epi == EPI_RESIDUAL) {
            const uint32_t xs[4] = {x[u].x, x[u].y, x[u].z, x[u].w}, ys[4] = {y[u].x, y[u].y, y[u].z, y[u].w};
            uint32_t o4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o4[e] = pack2(f2bf(__fadd_rn(lo2f(xs[e]), lo2f(ys[e]))), f2bf(__fadd_rn(hi2f(xs[e]), hi2f(ys[e]))));
            *reinterpret_cast<uint4*>(dst[u]) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
          } else {
            *reinterpret_cast<uint4*>(dst[u]) = y[u];
          }
        }
      }
    }
    __syncthreads();
    if (warp == 1) {
      drain_tc(dead);
    if (lane == 0) report_tc(dead, g.status);
      tc_fence_after();
      tmem_dealloc(tmem_base, TMEM_COLS);
    }
    return;
  }
  // red[token][lane] fp32 (conflict-free: a warp writes 32 consecutive floats per token);
  // it reuses the pipeline ring, which is idle once tmem_full has fired.  CTA r of the cluster reduces rows
  // [r * rows_per, (r + 1) * rows_per); a token's pitch is a tile's row plus rows_per values (at most 32), so that the 16-byte reads of
  // eight neighbouring threads (the rows of a token, then the next token) fall on different banks.
  const uint32_t red = smem0;
  const bool epi_warp = warp >= 2;
  const int qd = warp & 3;  // TMEM lane quarter of this epilogue warp
  const bool via_smem = TM == BM && (g.splits > 1 || DUAL);  // (the tile below has 128 lanes of rows: 64-row tiles are never split, launch_bn)
  const int tile_rows = DUAL ? BM / 2 : TM;  // output rows produced by this tile
  const int rows_per = ((tile_rows + g.splits - 1) / g.splits + 3) & ~3;
  const uint32_t pitch = (uint32_t)(BM + min(rows_per, 32)) * 4u;
  if (epi_warp) {
    pdl_wait();  // `out` may still be read (residual) by the previous kernel
    if (nkb > 0) {
      mbar_wait_tc(tmem_full_bar, 0, dead);
      tc_fence_after();
    }
    const bool bad = *dead;
    // TMEM lane = row inside the tile (of 64 rows: the lower half of each quarter's lanes)
    const int lane_row = TM == 64 ? qd * 16 + lane : qd * 32 + lane;
    const bool has_row = TM == 128 || lane < 16;
#pragma unroll
    for (int c0 = 0; c0 < BN; c0 += 16) {
      uint32_t r[16];
      if (nkb > 0) {
        tmem_ld16(tmem_base + ((uint32_t)(qd * 32) << 16) + c0, r);
        if (bad) mark_bad(r);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = 0u;
      }
      if (via_smem) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(red + (uint32_t)(c0 + j) * pitch + (uint32_t)lane_row * 4u), "r"(r[j]) : "memory");
      } else {
        // no split, single accumulator: epilogue straight from registers
        const int w_row = row0 + lane_row;
        if (has_row && w_row < seg_rows) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int tok = tok_base + c0 + j;
            if (tok < g.M) {
              bf16* dst = out + (size_t)tok * ld + w_row;
              const float v = __uint_as_float(r[j]);
              if (g.epi == EPI_RESIDUAL)
                *dst = f2bf(__fadd_rn(bf2f(*dst), bf2f(f2bf(v))));
              else
                *dst = f2bf(v);
            }
          }
        }
      }
    }
    tc_fence_before();
  }
  if (via_smem) {
    // all partial tiles of the cluster are parked in shared memory
    if (g.splits > 1) cluster_sync_all();
    else __syncthreads();
    if (epi_warp) {
      const int t = threadIdx.x - 64;  // 0..127
      const int S = g.splits;
      const int rbeg = split * rows_per;
      const int groups = max(0, min(rows_per, tile_rows - rbeg)) / 4;  // (tile_rows and rows_per are multiples of 4)
      const int n_tok = min(BN, g.M - tok_base);
      // A thread reduces four rows of a token, one 16-byte read per split; every read of an item is requested before the first sum.
      // With one 4-byte read per value and split the reduction of 64 tokens over 8 CTAs took 5.1 us, now 3.2.
      constexpr int MAXS = 8;  // portable cluster size
      uint32_t rb[MAXS];
#pragma unroll
      for (int sp = 0; sp < MAXS; ++sp) {
        rb[sp] = red;
        if (S > 1 && sp < S) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb[sp]) : "r"(red), "r"(sp));
      }
      auto ld4 = [&](int sp, uint32_t off, float (&v)[4]) {
        if (S > 1)
          asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(rb[sp] + off) : "memory");
        else
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(red + off) : "memory");
      };
      const bool vec = ld % 4 == 0 && seg_rows % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
      for (int o = t; o < groups * n_tok; o += 128) {
        const int tok = o / groups, rr = rbeg + (o - tok * groups) * 4, w_row = row0 + rr;
        if (w_row >= seg_rows) continue;
        const uint32_t off = (uint32_t)tok * pitch + (uint32_t)rr * 4u;
        float v[MAXS][4], v2[MAXS][4];
#pragma unroll
        for (int sp = 0; sp < MAXS; ++sp)
          if (sp < S) {
            ld4(sp, off, v[sp]);
            if (DUAL) ld4(sp, off + (uint32_t)(BM / 2) * 4u, v2[sp]);  // the up half of the tile
          }
        bf16* dst = out + (size_t)(tok_base + tok) * ld + w_row;
        float old[4] = {0.f, 0.f, 0.f, 0.f};
        if (g.epi == EPI_RESIDUAL) {
          if (vec) {
            const uint2 x = *reinterpret_cast<const uint2*>(dst);
            old[0] = lo2f(x.x), old[1] = hi2f(x.x), old[2] = lo2f(x.y), old[3] = hi2f(x.y);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (w_row + e < seg_rows) old[e] = bf2f(dst[e]);
          }
        }
        bf16 y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float acc = 0.f, acc2 = 0.f;
#pragma unroll
          for (int sp = 0; sp < MAXS; ++sp)
            if (sp < S) {  // rank order
              acc += v[sp][e];
              if (DUAL) acc2 += v2[sp][e];
            }
          if (g.epi == EPI_STORE) {
            y[e] = f2bf(acc);
          } else if (g.epi == EPI_RESIDUAL) {
            y[e] = f2bf(__fadd_rn(old[e], bf2f(f2bf(acc))));
          } else {
            const float gt = bf2f(f2bf(acc)), up = bf2f(f2bf(acc2));
            y[e] = f2bf(__fmul_rn(up, bf2f(f2bf(silu_ref_f(gt)))));
          }
        }
        if (vec) {
          *reinterpret_cast<uint2*>(dst) = make_uint2(pack2(y[0], y[1]), pack2(y[2], y[3]));
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (w_row + e < seg_rows) dst[e] = y[e];
        }
      }
    }
    // nobody may exit (and release its shared memory) while a peer still reads it
    if (g.splits > 1) cluster_sync_all();
  }
  __syncthreads();
  if (warp == 1) {
    drain_tc(dead);
    if (lane == 0) report_tc(dead, g.status);
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ persistent variant
// Same tiles, same math, for launches without split-K: ONE CTA per SM walks the output tiles (weight tile fastest, so neighbouring
// CTAs share a token tile in L2), the accumulator is double buffered in TMEM (2 x 256 columns), and the epilogue of tile j (TMEM ->
// bf16 staging tile in shared memory -> global memory, 64 tokens at a time) runs on warps 2-9 while warps 0/1 already
// stream and multiply tile j+1.  ncu on the one-tile-per-CTA kernel showed the tensor pipe 32-47 % active at K = 1536: per tile
// ~2.5 us of prologue and ~8 us of epilogue sat next to a ~7-9 us mainloop.
// A tile has g.bn tokens, any multiple of 16 (pick_tile): with 256 always, 4096 tokens x 1536 outputs were 192 tiles on 148 SMs, two
// waves filled to 65 %.  The ring takes the stages that fit: 4 of 48 KiB at 256 tokens, 10 of 18 KiB at 16.
static constexpr int PBN = 256;                   // TMEM columns of an accumulator
static constexpr int P_STEP = 64;                 // tokens of a staging tile (two of them)
static constexpr int P_RING = 4 * (BM * BK * 2 + PBN * BK * 2);     // 192 KiB
static constexpr int P_MAX_STAGES = 10;
static constexpr int P_EPI = 256;                 // epilogue threads (8 warps)
static constexpr int P_THREADS = 64 + P_EPI;      // + TMA warp + MMA warp
static constexpr int P_STAGING = 2 * P_STEP * BM * 2;               // bf16 [2][64 tokens][128 rows] = 32 KiB

// CTAS 2: a pair of CTAs, a cluster, has two neighbouring weight tiles and one token tile; either brings its own weights and half of the tokens, and the
// first one's MMA warp multiplies both tiles at once (cta_group::2).
template <int CTAS>
__global__ void __launch_bounds__(P_THREADS) gemm_tcgen05_persist_kernel(const __grid_constant__ CUtensorMap map_w0,
                                                                   const __grid_constant__ CUtensorMap map_w1,
                                                                   const __grid_constant__ CUtensorMap map_w2,
                                                                   const __grid_constant__ CUtensorMap map_x, TcArgs g,
                                                                   int token_tiles) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int dead_s;
  volatile int* const dead = &dead_s;
  if (threadIdx.x == 0) dead_s = 0;  // (a barrier follows before any wait)
  constexpr int A_BYTES = BM * BK * 2;
  constexpr uint32_t TMEM_COLS = 512;  // two accumulators
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int bn = g.bn, stages = g.stages, own = bn / CTAS, stage_bytes = A_BYTES + own * BK * 2;
  const uint32_t stg = smem0 + P_RING;
  const uint32_t bars = stg + P_STAGING;  // full[S], empty[S], tmem_full[2], tmem_empty[2], slot
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (P_MAX_STAGES + s); };
  auto tfull_bar = [&](int b) { return bars + 8u * (2 * P_MAX_STAGES + b); };
  auto tempty_bar = [&](int b) { return bars + 8u * (2 * P_MAX_STAGES + 2 + b); };
  const uint32_t slot = bars + 8u * (2 * P_MAX_STAGES + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pairs = (g.n_tiles + CTAS - 1) / CTAS, total = pairs * token_tiles;
  const int nkb = g.kb_total;
  const int inner = g.tokens_first ? token_tiles : pairs;  // tiles that neighbours walk
  const int rank = CTAS == 1 ? 0 : blockIdx.x % CTAS, at0 = blockIdx.x / CTAS, step_t = gridDim.x / CTAS;
  auto leader = [&](uint32_t bar) {  // the barrier of the pair's first CTA
    uint32_t r = bar;
    if (CTAS > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(bar), "r"(0));
    return r;
  };

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w0) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w1) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w2) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    for (int s = 0; s < stages; ++s) {
      mbar_init_tc(full_bar(s), 1);
      mbar_init_tc(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init_tc(tfull_bar(b), 1);
      mbar_init_tc(tempty_bar(b), CTAS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc<CTAS>(slot, TMEM_COLS);
  tc_fence_before();
  if (CTAS > 1) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(slot));

  // tile -> (weight tile, token tile, segment) ; dual: one tile = 64 gate rows + the same 64 up rows
  auto tile_geom = [&](int t, int& tile, int& ttile, int& si, int& row0) {
    const int slow = t / inner, fast = t - slow * inner;
    tile = (g.tokens_first ? slow : fast) * CTAS + rank;
    ttile = g.tokens_first ? fast : slow;
    si = 0;
    while (si + 1 < g.nseg && tile >= g.seg[si + 1].tile0) ++si;
    row0 = g.dual ? tile * (BM / 2) : (tile - g.seg[si].tile0) * BM;
  };

  if (warp == 0) {
    if (elect_tc()) {
      int s = 0;
      uint32_t ph = 1;
      bool go = true;
      auto load_w = [&](int kb, int si, int row0) {
        const uint32_t sa = smem0 + s * stage_bytes;
        if (g.dual) {
          tma_load_2d<CTAS>(sa, &map_w0, leader(full_bar(s)), kb * BK, row0);
          tma_load_2d<CTAS>(sa + A_BYTES / 2, &map_w1, leader(full_bar(s)), kb * BK, row0);
        } else {
          tma_load_2d<CTAS>(sa, si == 0 ? &map_w0 : (si == 1 ? &map_w1 : &map_w2), leader(full_bar(s)), kb * BK, row0);
        }
      };
      int tile, ttile, si, row0;
      // the first stages' weights in front of the wait for the previous kernel, which wrote the activations
      int pre = 0;
      if (g.w_static && at0 < total) {
        tile_geom(at0, tile, ttile, si, row0);
        for (pre = min(nkb, stages); s < pre; ++s) {
          if (rank == 0) mbar_expect_tx(full_bar(s), CTAS * stage_bytes);
          load_w(s, si, row0);
        }
        s = 0;
      }
      pdl_wait();
      for (int t = at0; t < total && go; t += step_t) {
        tile_geom(t, tile, ttile, si, row0);
        for (int kb = 0; kb < nkb; ++kb) {
          if (pre > 0) {  // (the first stages: nothing to wait for)
            --pre;
          } else {
            if (!(go = mbar_wait_tc(empty_bar(s), ph, dead))) break;
            if (rank == 0) mbar_expect_tx(full_bar(s), CTAS * stage_bytes);
            load_w(kb, si, row0);
          }
          tma_load_2d<CTAS>(smem0 + s * stage_bytes + A_BYTES, &map_x, leader(full_bar(s)), kb * BK, ttile * bn + rank * own);
          if (++s == stages) s = 0, ph ^= 1;
        }
      }
      pdl_trigger();
    }
    __syncwarp();
  } else if (warp == 1) {
    pdl_wait();  // as above
    const uint32_t idesc = idesc_tc(BM * CTAS, bn, false);
    const uint64_t ad0 = desc_k_tc(smem0), bd0 = desc_k_tc(smem0 + A_BYTES);
    int s = 0, j = 0;
    uint32_t ph = 0;
    for (int t = rank == 0 ? at0 : total; t < total; t += step_t, ++j) {
      const int buf = j & 1;
      mbar_wait_tc(tempty_bar(buf), (((uint32_t)j >> 1) & 1) ^ 1, dead);  // epilogue has drained this accumulator
      tc_fence_after();
      const uint32_t acc = tmem_base + (uint32_t)buf * PBN;
      for (int kb = 0; kb < nkb; ++kb) {
        mbar_wait_tc(full_bar(s), ph, dead);
        tc_fence_after();
        const uint64_t step = (uint64_t)(s * (stage_bytes >> 4));
        if (elect_tc()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma_tc<CTAS>(acc, ad0 + step + 2 * k, bd0 + step + 2 * k, idesc, (kb | k) != 0);
          umma_commit_tc<CTAS>(empty_bar(s));
        }
        __syncwarp();
        if (++s == stages) s = 0, ph ^= 1;
      }
      if (elect_tc()) {
        if (CTAS > 1) tell_other_tc(dead);
        umma_commit_tc<CTAS>(tfull_bar(buf));
      }
      __syncwarp();
    }
  } else {
    // ---- epilogue warps 2-9: two warps per TMEM lane quarter, each draining half of the columns (with four warps the
    // epilogue of a K = 1536 tile -- drain, SiLU * up, 64 KiB of stores -- took longer than the tile's mainloop).  64 tokens at a time
    // go through one of two staging tiles, so one barrier a step is enough: who drains into a tile has passed the barrier behind its
    // last readers.  Plain results leave by bulk copies, a token's 256 bytes each; residuals are requested before the drain.
    // With two barriers per 128 tokens, 16-byte stores by all threads and residuals requested behind the barrier (us, weights in L2; cuBLAS
    // 78): 4096 tokens, 1536 x 8960 82 -> 78; 2000: 42.7 -> 41.0; 1000: 24.6 -> 23.6; 18944 x 3584 with residual, 400: 75 -> 70.
    constexpr uint32_t PITCH = BM * 2;
    const int qd = warp & 3;
    const int lane_row = qd * 32 + lane;
    const int tq = threadIdx.x - 64;
    auto lds128 = [](uint32_t addr) {
      uint4 v;
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
      return v;
    };
    const bool bulk = g.vec && !g.dual && g.epi == EPI_STORE;
    const int copier = lane < P_STEP / 8 ? (warp - 2) * (P_STEP / 8) + lane : P_STEP;  // the token whose copy this thread issues
    pdl_wait();  // `out` may still be read (residual) by the previous kernel
    int j = 0, it = 0;
    for (int t = at0; t < total; t += step_t, ++j) {
      int tile, ttile, si, row0;
      tile_geom(t, tile, ttile, si, row0);
      const int seg_rows = g.seg[si].rows, ld = g.seg[si].ld;
      bf16* const out = g.seg[si].out;
      const int tok_base = ttile * bn;
      const int buf = j & 1;
      const uint32_t acc = tmem_base + (uint32_t)buf * PBN + ((uint32_t)(qd * 32) << 16);
      const int n_tok_all = min(bn, g.M - tok_base);
      bool bad = false;
#pragma unroll 1
      for (int h0 = 0; h0 < bn; h0 += P_STEP, ++it) {
        const int width = min(P_STEP, bn - h0), n_tok = max(0, min(P_STEP, n_tok_all - h0));
        const uint32_t st0 = stg + (uint32_t)(it & 1) * (P_STEP * PITCH);
        constexpr int U = P_STEP * (BM / 8) / P_EPI;  // 16-byte pieces of a thread
        uint4 x[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = tq + u * P_EPI, w_row = row0 + (c & 15) * 8;
          ok[u] = (c >> 4) < n_tok && w_row < seg_rows;
          if (!g.dual && g.epi == EPI_RESIDUAL && ok[u])
            x[u] = *reinterpret_cast<const uint4*>(out + (size_t)(tok_base + h0 + (c >> 4)) * ld + w_row);
        }
        if (h0 == 0) {
          mbar_wait_tc(tfull_bar(buf), ((uint32_t)j >> 1) & 1, dead);
          tc_fence_after();
          bad = *dead;
        }
#pragma unroll
        for (int c0 = ((warp - 2) >> 2) * 16; c0 < P_STEP; c0 += 32) {  // every other 16 columns: the quarter's second warp has the rest
          if (c0 >= width) break;
          uint32_t r[16];
          tmem_ld16(acc + h0 + c0, r);
          if (bad) mark_bad(r);
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const unsigned short hb = __bfloat16_as_ushort(f2bf(__uint_as_float(r[q])));
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(st0 + (uint32_t)(c0 + q) * PITCH + (uint32_t)lane_row * 2u), "h"(hb) : "memory");
          }
        }
        tc_fence_before();
        if (bulk) {
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the other staging tile has been read: the next step may write it
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (h0 + P_STEP >= bn && tq == 0) mbar_arrive_tc<CTAS>(leader(tempty_bar(buf)));  // the MMA warp may overwrite this accumulator (tile j+2)
        if (bulk) {
          if (copier < n_tok && row0 < seg_rows) {  // (a pair's second tile may lie behind the last one)
            bf16* dst = out + (size_t)(tok_base + h0 + copier) * ld + row0;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(st0 + (uint32_t)copier * PITCH),
                         "r"(2 * min(BM, seg_rows - row0))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        } else if (!g.vec) {  // an odd number of columns (plain results only): 2 bytes a thread, neighbours side by side
          for (int c = tq; c < n_tok * BM; c += P_EPI) {
            const int tok = c / BM, r = c % BM;
            unsigned short y;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(y) : "r"(st0 + (uint32_t)tok * PITCH + (uint32_t)r * 2u) : "memory");
            if (row0 + r < seg_rows) out[(size_t)(tok_base + h0 + tok) * ld + row0 + r] = __ushort_as_bfloat16(y);
          }
        } else if (!g.dual) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (!ok[u]) continue;
            const int c = tq + u * P_EPI;
            const uint4 y = lds128(st0 + (uint32_t)(c >> 4) * PITCH + (uint32_t)(c & 15) * 16u);
            const uint32_t xs[4] = {x[u].x, x[u].y, x[u].z, x[u].w}, ys[4] = {y.x, y.y, y.z, y.w};
            uint32_t o4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o4[e] = pack2(f2bf(__fadd_rn(lo2f(xs[e]), lo2f(ys[e]))), f2bf(__fadd_rn(hi2f(xs[e]), hi2f(ys[e]))));
            *reinterpret_cast<uint4*>(out + (size_t)(tok_base + h0 + (c >> 4)) * ld + row0 + (c & 15) * 8) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
          }
        } else {
          const int totalc = n_tok * (BM / 16);
          for (int c = tq; c < totalc; c += P_EPI) {
            const int tok = c >> 3, part = c & 7;
            const int w_row = row0 + part * 8;
            if (w_row >= seg_rows) continue;
            const uint4 gt = lds128(st0 + (uint32_t)tok * PITCH + (uint32_t)part * 16u);
            const uint4 up = lds128(st0 + (uint32_t)tok * PITCH + (uint32_t)(BM / 2) * 2u + (uint32_t)part * 16u);
            const uint32_t gs[4] = {gt.x, gt.y, gt.z, gt.w}, us[4] = {up.x, up.y, up.z, up.w};
            uint32_t o4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float s0 = g.ref_silu ? silu_ref_f(lo2f(gs[e])) : silu_fast_f(lo2f(gs[e]));
              const float s1 = g.ref_silu ? silu_ref_f(hi2f(gs[e])) : silu_fast_f(hi2f(gs[e]));
              const float a0 = __fmul_rn(lo2f(us[e]), bf2f(f2bf(s0)));
              const float a1 = __fmul_rn(hi2f(us[e]), bf2f(f2bf(s1)));
              o4[e] = pack2(f2bf(a0), f2bf(a1));
            }
            *reinterpret_cast<uint4*>(out + (size_t)(tok_base + h0 + tok) * ld + w_row) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
          }
        }
      }
    }
    if (bulk) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // written, before the CTA gives its shared memory back
  }
  if (CTAS > 1) cluster_sync_all();  // (the other one's operands and barriers are read and written to the end)
  else __syncthreads();
  if (warp == 1) {
    drain_tc(dead);
    if (lane == 0) report_tc(dead, g.status);
    tc_fence_after();
    tmem_dealloc<CTAS>(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// 2-D bf16 row-major [rows, K] tensor, box = [box_rows, 64], 128-byte swizzle, OOB -> 0
cudaError_t make_tensor_map_2d(TensorMap2D* out, const bf16* base, int rows, int K, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Weight matrix [rows, K] viewed as a 3-D tensor {64 k-elements, rows, K/64 k-blocks} so that
// ONE TMA request moves a box of 8 rows x kc k-elements (8 x kc x 2 bytes) into shared
// memory as [k-block][row][64] with the 128-byte swizzle (decode_mega.cu weight ring).
cudaError_t make_tensor_map_w3d(TensorMap2D* out, const bf16* base, int rows, int K, int kc, int ld, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return cudaErrorNotSupported;
  if ((K % 64) || (kc % 64) || kc / 64 > 256) return cudaErrorInvalidValue;
  if (ld <= 0) ld = K;  // a column slice of a wider matrix (tensor parallel o_proj / down_proj) has ld > K
  cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(K / 64)};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, 128};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)(kc / 64)};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Two matrices of rows x K as one tensor {64 of a k-block, rows, which one, k-blocks}: a box is 64 rows of both, [k-block][which][row][64] in shared memory, so that
// one request brings a gate/up tile's k-blocks.  Not supported where the second one does not lie behind the first, or 2^40 bytes away.
static cudaError_t make_tensor_map_gate_up(TensorMap2D* out, const bf16* gate, const bf16* up, int rows, int K, int kb) {
  EncodeTiledFn enc = get_encode();
  const uintptr_t lo = reinterpret_cast<uintptr_t>(gate), hi = reinterpret_cast<uintptr_t>(up);
  if (!enc || K % 64 || (lo | hi) % 16 || hi <= lo || hi - lo >= 1ull << 40) return cudaErrorNotSupported;
  cuuint64_t dims[4] = {64, (cuuint64_t)rows, 2, (cuuint64_t)(K / 64)};
  cuuint64_t strides[3] = {(cuuint64_t)K * 2, (cuuint64_t)(hi - lo), 128};
  cuuint32_t box[4] = {64, 64, 2, (cuuint32_t)kb};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)gate, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorNotSupported;
}

// KV pool [page][layer][k|v][head][slot][64] bf16 viewed as rows of 128 bytes (one head of one cached position).
// One TMA request moves box_rows consecutive slots of a (page, layer, K|V, head) chunk into shared memory; the
// 128-byte swizzle puts 16-byte chunk c of row r at chunk c ^ (r & 7), so that threads reading one row each
// (attention scores) and a warp reading one row together (PV) are both free of bank conflicts.
cudaError_t make_tensor_map_kv(TensorMap2D* out, const bf16* pool, unsigned long long rows, int hd, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return cudaErrorNotSupported;
  if ((hd != 64 && hd != 128) || box_rows < 1 || box_rows > 256 || rows == 0 || rows >= (1ull << 31)) return cudaErrorInvalidValue;
  cuuint64_t dims[2] = {(cuuint64_t)hd, (cuuint64_t)rows};  // head_dim 128: two 64-column boxes per row (the swizzle spans 128 bytes)
  cuuint64_t strides[1] = {(cuuint64_t)hd * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)pool, dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t make_tensor_map_pages(TensorMap2D* out, const bf16* base, int row_elems, int page_size, int n_pages, size_t page_elems, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return cudaErrorNotSupported;
  if (row_elems % 8 || page_elems % 8 || box_rows < 1 || box_rows > 256 || (reinterpret_cast<uintptr_t>(base) & 15)) return cudaErrorInvalidValue;
  cuuint64_t dims[3] = {(cuuint64_t)row_elems, (cuuint64_t)page_size, (cuuint64_t)n_pages};
  cuuint64_t strides[2] = {(cuuint64_t)row_elems * 2, (cuuint64_t)page_elems * 2};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int BN, bool HALF, int KB, int TM, bool AHEAD, bool DUAL = false>
static cudaError_t launch_bn(const TcArgs& g, const CUtensorMap* const (&w)[3], const TensorMap2D& x, int token_tiles, cudaStream_t st) {
  constexpr int STAGE_BYTES = KB * (TM * BK * 2 + BN * BK * 2);
  constexpr size_t smem = (size_t)TcCfg<BN, HALF, KB, TM>::STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(TM == BM || !DUAL, "gate/up tiles have 128 rows");
  if (TM != BM && g.splits > 1) return cudaErrorInvalidValue;
  static PerDeviceOnce set;
  if (set.need()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, HALF, KB, TM, AHEAD, DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, HALF, KB, TM, AHEAD, DUAL>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    set.done();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(g.n_tiles, g.splits, token_tiles);
  cfg.blockDim = dim3(DUAL && g.staged ? 256 : 192);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int na = 0;
  if (g.splits > 1) {
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = 1;
    at[na].val.clusterDim.y = g.splits;
    at[na].val.clusterDim.z = 1;
    ++na;
  }
  if (g_use_pdl) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<BN, HALF, KB, TM, AHEAD, DUAL>, *w[0], *w[1], *w[2], *reinterpret_cast<const CUtensorMap*>(&x), g);
}

template <int KB>
static cudaError_t launch_tile(int bn, bool half, bool ahead, const TcArgs& g, const CUtensorMap* const (&w)[3], const TensorMap2D& x, int token_tiles, cudaStream_t st) {
  constexpr int TM = KB == 4 ? 64 : BM;
  auto go = [&](auto n) {
    constexpr int BN = decltype(n)::value;
    if constexpr (KB < 4)
      if (g.dual) return launch_bn<BN, false, KB, TM, false, true>(g, w, x, token_tiles, st);
    if constexpr (KB > 1 || BN == 128)
      if (ahead) return launch_bn<BN, false, KB, TM, true>(g, w, x, token_tiles, st);
    return launch_bn<BN, false, KB, TM, false>(g, w, x, token_tiles, st);
  };
  if constexpr (KB != 4)
    if (half) return g.dual ? launch_bn<16, true, KB, TM, false, true>(g, w, x, token_tiles, st) : launch_bn<16, true, KB, TM, false>(g, w, x, token_tiles, st);
  switch (bn) {
    case 16: return go(std::integral_constant<int, 16>{});
    case 32: return go(std::integral_constant<int, 32>{});
    case 64: return go(std::integral_constant<int, 64>{});
    default:
      if constexpr (KB == 1) return go(std::integral_constant<int, 128>{});
  }
  return cudaErrorInvalidValue;
}

struct TcTile {
  int bn, splits;
  bool persist, half;
};
// Tokens of a tile and splits over K.  Measured on B200 in graphs of the same launch, weights in L2 (us), with stages of one k-block, 0.19 us each at any
// width up to 128.  Stages of two, which came later (up to 64 tokens, launch_gemm_tcgen05), take 0.13 a k-block: the choices between 64 and 128 tokens
// and between splits are still those of the older figure.
//  * One wave of CTAs: the smallest of 16 ... 128 tokens whose tiles all fit on the SMs, since narrower tiles fill and drain faster: 896 x 896,
//    1000 tokens: 64 7.1, 128 7.8, 256 9.5 (a split over 5 CTAs: 50.8).
//  * More tiles than that: the persistent kernel.  256 tokens, unless a width with fuller waves takes less than 0.9 of waves x width
//    (1536 outputs at 4096 rows: 107 -> 86 with 176; a few per cent less on paper were none: 8960 outputs 82.7 with 256, 85.5 with
//    224).  Below 160 tokens the loop, not the tensor core, sets a tile's time, so of those the narrowest wins, whose ring holds most
//    k-blocks: 151936 x 896 for one row 79 -> 47.  (Odd output widths too, with 2-byte stores: one 256-token tile per CTA took 45 us for 1 x 896 x
//    20001.)  Up to 16 rows and two tiles an SM: one tile per CTA, two CTAs an SM beside each other (1 x 896 x 20001, weights from memory: persistent 11.3, 9.0).
//  * Few tiles and a long K: a cluster of 2, 4 or 8 CTAs splits K (never in the reference's order).  Its reduction costs about
//    1.1 us + (0.1, 0.055, 0.045) us x tokens that are there, a k-block 0.19 us: 4864 x 896 at 64 tokens 16.0 without, 6.9 with 8 x 32 tokens.  All
//    clusters have to run at once (`most` clusters of a size fit on 148 SMs; they do not pack every SM: 28 clusters of 5 took two rounds, 49 us
//    against 27 with 4).
static TcTile pick_tile(int M, int tiles, int nkb, int num_sms, bool may_split) {
  auto ctas = [&](int bn) { return (long)tiles * ((M + bn - 1) / bn); };
  TcTile best{16, 1, false, false};
  while (best.bn < 256 && ctas(best.bn) > num_sms) best.bn *= 2;
  if (best.bn < 256) {
    if (!may_split) return best;
    float cost = 0.19f * nkb;
    static const int most[3] = {64, 28, 14};
    static const float per_token[3] = {0.1f, 0.055f, 0.045f};
    for (int i = 0; i < 3; ++i)
      for (int bn = 16; bn <= 128; bn *= 2) {
        const int s = 2 << i;
        if (nkb < 2 * s || ctas(bn) * 148 > (long)most[i] * num_sms || (bn > 16 && bn / 2 >= M)) continue;
        const float c = 0.19f * ((nkb + s - 1) / s) + 1.1f + per_token[i] * std::min(bn, M);
        if (c < cost) cost = c, best.bn = bn, best.splits = s;
      }
    return best;
  }
  if (M <= 16 && tiles <= 2 * num_sms) {
    best.bn = 16, best.half = true;
    return best;
  }
  best.persist = true;
  auto waves = [&](int bn) { return (ctas(bn) + num_sms - 1) / num_sms * std::max(bn, 160); };
  long cost = waves(256) * 9 / 10;
  for (int bn = 16; bn < 256; bn += 16)
    if (waves(bn) < cost) cost = waves(bn), best.bn = bn;
  return best;
}

// Tokens of a pair's tile, 0 where single CTAs of `bn` tokens stay.  Costs of a wave are in units of about 1 ns a k-block: a single CTA's operands take it 1.0 a row of 128
// bytes that it brings from L2 (256 tokens: 48 KB, 0.4 us), a pair's CTA 1.22 a row or the products 1.36 a token, whichever is more; a pair's start and end cost
// 1.2 us more, and few waves have to gain by more.  Below PAIR_KB k-blocks a tile the epilogue sets the pace.  us in graphs, single CTAs and pairs: 4096 rows 1536 x 8960 78 72 (256
// tokens), 8960 x 1536 83 78 (192), 3584 x 3584 79 70 (224), 2048 rows of 1536 x 8960 40 38, 1500 of 3584 x 3584 33.4 31.0 (160); stay: 2048 of 3584 x 3584 36.6 37.6
// (224), 1000 rows 21.1 23.2 (224), 700 of 3584 x 4608 19.8 20.3 (192), 4096 of 1536 x 1536 18.4 18.4 (192), of 896 x 4864 33.3 32.2 to 36.8.
static constexpr int PAIR_KB = 20;
static int pick_pair(int M, int tiles, int nkb, int num_sms, int pairs, int bn) {
  if (pairs <= 0 || nkb < PAIR_KB) return 0;
  auto waves = [&](int t, int b, int at) { return ((long)t * ((M + b - 1) / b) + at - 1) / at; };
  const float single = (float)waves(tiles, bn, num_sms) * (float)(BM + bn);
  int best = 0;
  float cost = single;
  for (int b = 256; b >= 128; b -= 32) {
    const long n = waves((tiles + 1) / 2, b, pairs);
    const float c = (float)n * std::max(1.22f * (float)(BM + b / 2), 1.36f * (float)b) + 1200.f / (float)nkb;
    if (c < (best ? 0.97f * cost : cost) && c < single * (n > 2 ? 0.97f : n == 2 ? 0.93f : 0.9f)) cost = c, best = b;
  }
  return best;
}

static constexpr size_t P_SMEM = (size_t)P_RING + P_STAGING + 1024 /*align*/ + 256 /*barriers*/;
template <int CTAS>
static cudaError_t persist_attributes() {
  static PerDeviceOnce set;
  if (!set.need()) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_persist_kernel<CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P_SMEM);
  if (e == cudaSuccess) set.done();
  return e;
}

// at: CTAs, or pairs of them, that run at once
template <int CTAS>
static cudaError_t launch_persist(TcArgs g, int bn, int at, const CUtensorMap* const (&w)[3], const bf16* xp, int M, int K, cudaStream_t st) {
  TensorMap2D x;
  cudaError_t e = make_tensor_map_2d(&x, xp, M, K, bn / CTAS);
  if (e != cudaSuccess || (e = persist_attributes<CTAS>()) != cudaSuccess) return e;
  const int token_tiles = (M + bn - 1) / bn;
  g.bn = bn;
  long w_rows = 0;  // K elements each, like the tokens
  for (int i = 0; i < g.nseg; ++i) w_rows += (g.dual ? 2 : 1) * g.seg[i].rows;
  // A wave's CTAs share a token tile and bring all weights, which the next wave finds in L2 unless they are too many: then the CTAs share weight tiles and bring all
  // tokens, if those are few.  (64 MB: half of the L2.)  us of 3584 x 18944 (136 MB): 400 rows 57.7 48.9, 4096 single CTAs 477 363, pairs 423 333; 896 x 151936, 1000 rows 280 241; 18944 x 3584, 1000
  // rows 161 135, but 2048 (78 MB of tokens) 228 255.
  g.tokens_first = 2 * w_rows * K > 64l << 20 && 2 * M < w_rows;
  g.stages = std::min(P_MAX_STAGES, P_RING / (BM * BK * 2 + bn / CTAS * BK * 2));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(CTAS * std::min<long>(at, (long)((g.n_tiles + CTAS - 1) / CTAS) * token_tiles)));
  cfg.blockDim = dim3(P_THREADS);
  cfg.dynamicSmemBytes = P_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at_[2];
  int na = 0;
  if (CTAS > 1) {
    at_[na].id = cudaLaunchAttributeClusterDimension;
    at_[na].val.clusterDim.x = CTAS;
    at_[na].val.clusterDim.y = at_[na].val.clusterDim.z = 1;
    ++na;
  }
  if (g_use_pdl) {
    at_[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at_[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = at_;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, gemm_tcgen05_persist_kernel<CTAS>, *w[0], *w[1], *w[2], *reinterpret_cast<const CUtensorMap*>(&x), g, token_tiles);
}

// pairs of CTAs of the persistent kernel that run at once on this device, 0 if there is no telling
static int pairs_at_once() {
  static std::atomic<int> known[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n) return n > 0 ? n : 0;
  if (persist_attributes<2>() != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(P_THREADS);
  cfg.dynamicSmemBytes = P_SMEM;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_tcgen05_persist_kernel<2>, &cfg) != cudaSuccess) n = 0, (void)cudaGetLastError();
  known[dev].store(n > 0 ? n : -1, std::memory_order_relaxed);
  return n > 0 ? n : 0;
}

cudaError_t launch_gemm_tcgen05(const TcGemm& t, int num_sms, cudaStream_t st, int* launches) {
  if (t.M < 1 || t.K < BK || (t.K % 8) || t.nseg < 1 || t.nseg > 3) return cudaErrorInvalidValue;
  TcArgs g{};
  g.M = t.M;
  g.K = t.K;
  g.nseg = t.nseg;
  g.epi = t.epi;
  g.dual = t.epi == EPI_SILU_MUL;
  g.w_static = t.w_static;
  // The short SiLU is for prompts, whose epilogue paces the tile at K = 1536.  Up to 128 rows no tile waits
  // for it, and fast numerics keep the reference's.
  g.ref_silu = t.exact || t.M <= 128;
  g.status = t.status;
  int tiles = 0;
  auto segments = [&](int tm) {  // tiles of tm weight rows
    int cols = 0;
    tiles = 0;
    for (int i = 0; i < t.nseg; ++i) {
      g.seg[i] = t.outs[i] ? TcSeg{t.rows[i], tiles, t.lds[i], t.outs[i]} : TcSeg{t.rows[i], tiles, t.ld_out, t.out + cols};
      tiles += (t.rows[i] + tm - 1) / tm;
      cols += t.rows[i];
    }
  };
  if (g.dual) {
    // segments = (gate, up) with equal row counts; the weight maps must have 64-row boxes
    if (t.nseg != 2 || t.rows[0] != t.rows[1]) return cudaErrorInvalidValue;
    g.seg[0] = TcSeg{t.rows[0], 0, t.ld_out, t.out};
    g.nseg = 1;
    tiles = (t.rows[0] + BM / 2 - 1) / (BM / 2);
  } else {
    segments(BM);
  }
  g.kb_total = (t.K + BK - 1) / BK;
  bool vec = true;  // 16-byte stores reach every row of the outputs
  for (int i = 0; i < g.nseg; ++i)
    vec = vec && g.seg[i].rows % 8 == 0 && g.seg[i].ld % 8 == 0 && (reinterpret_cast<uintptr_t>(g.seg[i].out) & 15) == 0;
  TcTile tl = pick_tile(t.M, tiles, g.kb_total, num_sms, !t.exact);
  // Tiles of 64 weight rows where they all fit on the SMs and a CTA brings fewer rows: with few tiles and a long K a CTA takes its operands at 138 GB/s from L2, whatever
  // the tile (a k-block of 128 rows and 16 tokens 0.13 us, 32 0.15, 64 0.174).  Four k-blocks a stage (two of 64 rows 0.10 us, four 0.07): from eight on, so that at most one of
  // three stages is short (of 64 tokens, whose ring holds three, from twenty on: 64 rows of 896 x 4864 4.9 5.1), and not where there would be fewer CTAs (1000 rows of 2048
  // x 300, 96 and 80: 8.6 8.8).  us of 128 and of 64 rows, reference order: 64 rows 4864 x 896 12.6 8.4, 8960 x 1536 21.2 13.6, 896 x 1152 4.5 4.0; 512 rows 4864 x 896
  // 14.0 11.5; 200 rows 8960 x 1536 22.9 17.5.  Their maps are made here, so the weights' place has to be known.
  int tm = BM;
  bool wp = true;
  for (int i = 0; i < t.nseg; ++i) wp = wp && t.wp[i];
  if (!tl.persist && !tl.half && tl.splits == 1 && !g.dual && wp && t.K % BK == 0 && g.kb_total >= 8) {
    long tiles64 = 0;
    for (int i = 0; i < t.nseg; ++i) tiles64 += (t.rows[i] + 63) / 64;
    int bn = 16;
    while (bn < 128 && tiles64 * ((t.M + bn - 1) / bn) > num_sms) bn *= 2;
    const auto ctas = [&](long n, int b) { return n * ((t.M + b - 1) / b); };
    if (bn <= (g.kb_total >= 20 ? 64 : 32) && 64 + bn < BM + tl.bn && ctas(tiles64, bn) >= ctas(tiles, tl.bn)) tm = 64, tl.bn = bn, segments(64);
  }
  g.n_tiles = tiles;
  const int token_tiles = (t.M + tl.bn - 1) / tl.bn;
  g.kb_per_split = (g.kb_total + tl.splits - 1) / tl.splits;
  g.splits = (g.kb_total + g.kb_per_split - 1) / g.kb_per_split;
  g.staged = g.splits == 1 && vec;
  g.vec = vec;
  // the weights' maps, in boxes of one, two or four k-blocks: those that the caller keeps, else made here
  const CUtensorMap* w[3];
  TensorMap2D made[3], x;
  const int kb = tm == BM ? 2 : 4;  // k-blocks of a stage of more than one
  auto maps = [&](bool two) {
    for (int i = 0; i < t.nseg; ++i) {
      const TensorMap2D* m = tm == 64 ? nullptr : two ? t.w2[i] : t.w[i];
      if (!m) {
        if (!t.wp[i]) return false;
        const cudaError_t e = two ? make_tensor_map_w3d(&made[i], t.wp[i], t.rows[i], t.K, kb * BK, 0, tm) : make_tensor_map_2d(&made[i], t.wp[i], t.rows[i], t.K, g.dual ? BM / 2 : BM);
        if (e != cudaSuccess) return false;
        m = &made[i];
      }
      w[i] = reinterpret_cast<const CUtensorMap*>(m);
    }
    for (int i = t.nseg; i < 3; ++i) w[i] = w[0];
    return true;
  };
  auto gate_up = [&]() {  // one map of both
    if (!t.wp[0] || !t.wp[1] || make_tensor_map_gate_up(&made[0], t.wp[0], t.wp[1], t.rows[0], t.K, 2) != cudaSuccess) return false;
    for (int i = 0; i < 3; ++i) w[i] = reinterpret_cast<const CUtensorMap*>(&made[0]);
    return true;
  };
  if (launches) *launches = 1;
  // The MMA warp asks ahead for the next stage from 16 stages on, eight of 128 tokens (us without and with: 64 rows 4864 x 896 8.7 8.2, 8960 x 1536 14.3 13.6; 1000 rows
  // 15.5 14.5, 35.3 30.8; 1500 of 896 x 896 7.1 6.8; 4 stages of four k-blocks, 896 x 896, 3.7 4.0).  Not for gate/up (nothing) and clusters (few stages, or weights
  // from memory: 300 rows of 8960 x 1536 in two 26.2 26.8).
  auto ahead = [&](int stage) { return g.splits == 1 && !g.dual && (g.kb_total + stage - 1) / stage >= (tl.bn == 128 ? 8 : 16); };
  // Two k-blocks a stage where tensor maps can express them (whole k-blocks, and the weights' place is known): half the requests, waits and commits.  Up
  // to 64 tokens: of 128 the ring holds three such stages, too few on the way (8960 x 1536 at 1000 rows 34.8 with stages of one, 37.1).  Gate/up tiles
  // take both matrices by one request (make_tensor_map_gate_up), one for three of stages of one: a request takes its warp 140 to 270 cycles (896 x 2 x 4864 behind a norm, 64 rows
  // 7.7 -> 6.7 us; 24 layers in fast numerics, 16 rows, 963 -> 939 us a step.  Not for wider and persistent tiles, whose k-blocks take as long: 200 rows 310 312).  Not for 3 or 5 k-blocks: the half of the last stage that is not there is a box of zeros to bring, a quarter of
  // the operands (us with stages of one and of two, 1000 rows: 192 x 130 3.7 4.0, 320 x 130 4.3 4.6, 448 x 130 4.7 4.7, 576 x 130 4.5 4.2).
  const bool whole = g.splits > 1 || g.kb_total % 2 == 0 || g.kb_total > 5;
  if (!tl.persist && tl.bn <= 64 && t.K % BK == 0 && g.kb_per_split >= 2 && whole && (g.dual ? gate_up() : maps(true)) &&
      make_tensor_map_w3d(&x, t.x, t.M, t.K, kb * BK, 0, tl.bn) == cudaSuccess)
    return tm == 64 ? launch_tile<4>(tl.bn, false, ahead(4), g, w, x, token_tiles, st) : launch_tile<2>(tl.bn, tl.half, ahead(2), g, w, x, token_tiles, st);
  if (tm != BM || !maps(false)) {
    if (launches) *launches = 0;
    return cudaErrorNotSupported;
  }
  if (tl.persist) {
    // (widths of the residual stream and of the feed-forward are inner dimensions too, so multiples of 8)
    if (!vec && t.epi != EPI_STORE) return cudaErrorInvalidValue;
    const int pairs = g.kb_total < PAIR_KB ? 0 : pairs_at_once(), pair_bn = pick_pair(t.M, tiles, g.kb_total, num_sms, pairs, tl.bn);
    return pair_bn ? launch_persist<2>(g, pair_bn, pairs, w, t.x, t.M, t.K, st) : launch_persist<1>(g, tl.bn, num_sms, w, t.x, t.M, t.K, st);
  }
  const cudaError_t e = make_tensor_map_2d(&x, t.x, t.M, t.K, tl.bn);
  if (e != cudaSuccess) return e;
  return launch_tile<1>(tl.bn, tl.half, ahead(1), g, w, x, token_tiles, st);
}

// Reference-order products of any number of rows.  The chain of tcgen05.mma over ascending k of 16 into one accumulator gives the bits of
// the reference's chain of m16n8k16 products: 1.5e9 outputs of 84 combinations of shape and distribution (values of 2^+-60, cancelling
// sums, subnormals, overflow, infinities, NaN) showed no difference, and tests/test_gpu_gemm_exact.py repeats a part of them.  So
// the reference order takes the tcgen05 kernels without the split over K, at every row count: 896 x 4864 at 1000 rows 290 us ->
// 12.6 (the mma.sync kernel runs 64 rows a launch and reads the weights again for each), at 16 rows 10.5 -> 4.7; 4864 x 896 at 400 rows
// 737 -> 16.5; 896 x 151936 at 1 row 79 -> 47.  The mma.sync kernel keeps what TMA or the tile cannot express: K below one k-block (two for up to 8 rows), fp32 outputs (the partial sums
// of tensor parallelism), column slices of a wider matrix.  Operands off a 16-byte boundary are refused: both kernels read 16 bytes at a time.
cudaError_t launch_gemm_ref_rows(const GemmArgs& a, int num_sms, cudaStream_t st, int w_static, int* launches, int* status) {
  if (launches) *launches = 0;
  // (up to 8 rows of less than two k-blocks: the mma.sync kernel starts up quicker, 8 x 64 x 512 in 1.95 us, 2.05 here; from 128 on no longer)
  bool tc = a.M >= 1 && a.K >= (a.M <= 8 ? 2 * BK : BK) && a.K % 8 == 0 && a.lda == a.K && a.epi != EPI_STORE_F32 && a.nseg <= 3 &&
            (reinterpret_cast<uintptr_t>(a.A) & 15) == 0;
  for (int i = 0; i < a.nseg; ++i) tc = tc && (a.seg[i].ldw == 0 || a.seg[i].ldw == a.K);
  if (tc) {
    const bool dual = a.epi == EPI_SILU_MUL;
    TcGemm t{};
    t.x = a.A;
    t.nseg = dual ? 2 : a.nseg;
    t.M = a.M;
    t.K = a.K;
    t.epi = a.epi;
    t.exact = 1;
    t.status = status;
    t.w_static = w_static;
    t.out = a.seg[0].out;
    t.ld_out = a.seg[0].ld_out;
    for (int i = 0; i < t.nseg; ++i) {
      const GemmSeg& sg = a.seg[dual ? 0 : i];
      t.wp[i] = dual && i ? sg.W2 : sg.W;
      t.rows[i] = sg.rows;
      t.outs[i] = sg.out;
      t.lds[i] = sg.ld_out;
    }
    const cudaError_t e = launch_gemm_tcgen05(t, num_sms, st, launches);
    if (e != cudaErrorNotSupported) return e;  // (no tensor map expresses these weights)
  }
  for (int r0 = 0; r0 < a.M; r0 += 64) {
    GemmArgs c = a;
    c.A = a.A + (size_t)r0 * a.lda;
    c.M = std::min(64, a.M - r0);
    for (int i = 0; i < a.nseg; ++i)  // EPI_STORE_F32: `out` is a float*, twice the bf16 stride
      c.seg[i].out = a.seg[i].out + (size_t)r0 * a.seg[i].ld_out * (a.epi == EPI_STORE_F32 ? 2 : 1);
    cudaError_t e = launch_gemm_ref_order(c, num_sms, st);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  return cudaSuccess;
}

}  // namespace qie
