// tc_ptx.cuh -- tcgen05, TMEM and mbarrier instructions with waits that have a limit, for kernels whose CTA finishes without waiting
// once a wait ran out.
#pragma once
#include "common.cuh"

namespace qie {

__device__ __forceinline__ void mbar_init_tc(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
template <int CTAS = 1>  // 2: the barrier may be the other CTA's of a pair
__device__ __forceinline__ void mbar_arrive_tc(uint32_t bar) {
  if constexpr (CTAS == 2) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
  else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Waits for the phase of this parity.  After about two seconds it sets *dead, and from then on no wait of the CTA waits: its kernel stores values
// that are not numbers, lets copies in flight land (drain_tc), reports (report_tc) and returns.  The clock is read only where a wait is long.
constexpr long long WAIT_CYCLES_TC = 4000000000ll;
__device__ __forceinline__ bool mbar_wait_tc(uint32_t bar, uint32_t parity, volatile int* dead) {
  long long t0 = 0;
  for (int i = 0;; ++i) {
    uint32_t done = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 31) == 31) {
      if (*dead) return false;
      if (i == 31) t0 = clock64();
      else if (clock64() - t0 > WAIT_CYCLES_TC) break;
    }
  }
  *dead = 1;
  return false;
}
__device__ __forceinline__ bool mbar_ready_tc(uint32_t bar, uint32_t parity) {  // without waiting
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ void drain_tc(const volatile int* dead) {
  if (*dead)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
}
// For pairs of CTAs that work on one tile: a wait that ran out in this one counts for the other one too, whose results hang on this one's operands.  One thread, ahead of the
// arrival that lets the other one go on; the word is read back, so it is there before that arrival.
__device__ __forceinline__ void tell_other_tc(volatile int* dead) {
  if (!*dead) return;
  uint32_t rank, there;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(const_cast<int*>(dead))), "r"(rank ^ 1u));
  asm volatile("st.volatile.shared::cluster.u32 [%0], 1;" ::"r"(there) : "memory");
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  asm volatile("{\n\t.reg .b32 seen;\n\tld.volatile.shared::cluster.u32 seen, [%0];\n\t}" ::"r"(there) : "memory");
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
}
// one thread, behind the CTA's last wait: status is a word that the host reads (mapped memory), or null
__device__ __forceinline__ void report_tc(const volatile int* dead, int* status) {
  if (*dead && status) {
    *reinterpret_cast<volatile int*>(status) = 1;
    __threadfence_system();
  }
}
// one lane of the converged warp; under a branch on it the compiler emits tcgen05 and TMA instructions once (under a branch on the
// lane number each of them goes through code for any set of active lanes)
__device__ __forceinline__ bool elect_tc() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
template <int CTAS = 1>  // 2: the operands lie in both CTAs of a pair at the same places, as do the accumulators
__device__ __forceinline__ void umma_tc(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  if constexpr (CTAS == 2) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
    return;
  }
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
template <int CTAS = 1>  // 2: arrives at the barrier of that place in both CTAs
__device__ __forceinline__ void umma_commit_tc(uint32_t bar) {
  if constexpr (CTAS == 2) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((unsigned short)3) : "memory");
    return;
  }
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16_tc(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16_tc(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st8_tc(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
               "r"(r[6]), "r"(r[7]), "r"(taddr)
               : "memory");
}
// A from TMEM: row = lane, a 32-bit column holds two consecutive k
__device__ __forceinline__ void umma_ts_tc(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
// K-major operand, SWIZZLE_128B, 8-row atoms 1024 bytes apart
__device__ __forceinline__ uint64_t desc_k_tc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// MN-major operand (rows are k: [k][column]), SWIZZLE_128B: blocks of 64 columns `blk` bytes apart, groups of 8 k 1024
__device__ __forceinline__ uint64_t desc_mn_tc(uint32_t smem_addr, uint32_t blk) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)(blk >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// D = F32, A = B = BF16, N >> 3 at [17,23), M >> 4 at [24,29), bit 16: B is MN-major
__device__ __forceinline__ uint32_t idesc_tc(int m, int n, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ float ex2_tc(float x) {  // 2^x; 2^(-inf) = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

}  // namespace qie
