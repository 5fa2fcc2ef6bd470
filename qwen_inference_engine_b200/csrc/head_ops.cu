// head_ops.cu -- what stands between the q/k/v projections and attention: head norms (layers/src/qk_norm.cu:43-80), rotary positions
// (layers/src/RoPE.cu:6-22) and the store into the KV pool (layers/src/include_cuda.cu:165-279), as one kernel for the engine
// and as single operators.  Compiled with -fmad=false, every result by the reference's sequence of IEEE operations (ref_math.cuh).
//
// A head of 64 NP values belongs to LH = 4 NP lanes, a warp has 32 / LH heads; they may be of different tokens and kinds.  Lane l holds the 16-byte
// pieces l and l + LH: the tree's first stride (half a head) is in the lane, the strides down to 8 are exchanges between the LH lanes, 4, 2, 1
// are in the lane again; interleaved and half-rotation partners are in the lane as well.  Square root, reciprocal and page lookup are done once
// for all heads of a warp.  One head after the other on 32 lanes with 4-byte accesses took about 250 instructions a head of 128, here 75.
// What bounds it now: latency of the loads and DRAM; behind a projection 4096 tokens of 16 heads of 128 took 23.5 us
// and take 11.2, 512 tokens of 18 heads of 64 6.5 and 3.1; head norms and positions alone, 1000 x 12 heads of 128, 3.4 and 3.0, now 2.3 and 2.0 (positions of few heads: 32 lanes a head, see the rule).
#include <initializer_list>

#include "common.cuh"
#include "head_math.cuh"
#include "kernels.h"
#include "launch.h"
#include "ref_math.cuh"

namespace qie {
namespace {

// Where the kernel in front writes nothing but the projections (a.early), the row's position, its place in the pool and the tables' lines are fetched before it ends: three reads, one
// behind the other, of 2.9 us behind the projections of 64 rows (24 layers, 64 rows at 2048 positions, 1807 -> 1785 us a step).
template <int NP, bool V>
__global__ void __launch_bounds__(128) qkv_post_kernel(QkvPostArgs a) {
  using H = Head<NP>;
  constexpr int HD = 64 * NP;
  if (!a.early) pdl_wait();
  const int heads = a.n_q + 2 * a.kv.n_kv, all = a.n_tok * heads;  // q heads, k heads, v heads
  const int at = (blockIdx.x * 128 + threadIdx.x) / H::LH, l = threadIdx.x % H::LH;
  const int g = min(at, all - 1), tok = g / heads, h = g - tok * heads;
  const int kind = h < a.n_q ? 0 : h < a.n_q + a.kv.n_kv ? 1 : 2, kh = h - a.n_q - (kind == 2 ? a.kv.n_kv : 0);  // kh: head within k / v
  const bf16* src = kind == 0 ? a.q_in + (size_t)tok * a.q_in_stride + (size_t)h * HD : (kind == 1 ? a.k : a.v) + (size_t)tok * a.kv_stride + (size_t)kh * HD;
  const int ps = a.pos[tok];
  const float *co = a.cos_t + (size_t)ps * H::HALF, *si = a.sin_t + (size_t)ps * H::HALF;
  if (a.early && kind != 2) {
    const int first = a.rope_half ? 8 * l : 4 * l, second = a.rope_half ? 8 * l + 4 : H::HALF / 2 + 4 * l;
    for (const float* p : {co + first, co + second, si + first, si + second}) asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(p)));
  }
  bf16* dst = a.q + (size_t)tok * a.n_q * HD + (size_t)h * HD;
  if (kind != 0) {
    const int page = a.block_table[(size_t)a.slot[tok] * a.max_pages + ps / a.kv.page_size];
    dst = a.kv.chunk(page, a.layer, kind - 1, kh) + (size_t)(ps % a.kv.page_size) * HD;
  }
  if (a.early) pdl_wait();
  pdl_trigger();
  H x;
  x.template load<V>(src, l);
  const bf16* bias = kind == 0 ? a.q_bias : kind == 1 ? a.k_bias : a.v_bias;
  if (bias) x.template add_bias<V>(bias + (size_t)(kind == 0 ? h : kh) * HD, l);
  const float sum = x.squares();
  const bf16* w = kind == 0 ? a.q_norm_w : a.k_norm_w;
  if (kind != 2) {
    if (w) x.template norm<V>(sum, w, l, a.eps);
    if (a.rope_half)
      x.template rope_half<V>(co, si, l);
    else
      x.template rope<V>(co, si, l);
  }
  if (at < all) x.template store<V>(dst, l);  // (v: bf16 -> fp32 -> bf16 is the identity)
}

template <int NP, bool V>
__global__ void __launch_bounds__(128) qknorm_ref_kernel(bf16* x, const bf16* __restrict__ w, int n_tok, int row_dim, int n_heads) {
  pdl_wait();
  pdl_trigger();
  using H = Head<NP>;
  const int all = n_tok * n_heads, at = (blockIdx.x * 128 + threadIdx.x) / H::LH, l = threadIdx.x % H::LH;
  const int g = min(at, all - 1), tok = g / n_heads;
  bf16* p = x + (size_t)tok * row_dim + (size_t)(g - tok * n_heads) * 64 * NP;
  H v;
  v.template load<V>(p, l);
  v.template norm<V>(v.squares(), w, l, 1e-04f);
  if (at < all) v.template store<V>(p, l);
}

template <int NP, bool V>
__global__ void __launch_bounds__(128) rope_ref_kernel(const float* __restrict__ cos_t, const float* __restrict__ sin_t, bf16* x, int n_tok, const int* __restrict__ pos,
                                                       int pos0, int row_dim, int n_heads) {
  pdl_wait();
  pdl_trigger();
  using H = Head<NP>;
  const int all = n_tok * n_heads, at = (blockIdx.x * 128 + threadIdx.x) / H::LH, l = threadIdx.x % H::LH;
  if (at >= all) return;
  const int tok = at / n_heads, ps = pos ? pos[tok] : pos0 + tok;
  bf16* p = x + (size_t)tok * row_dim + (size_t)(at - tok * n_heads) * 64 * NP;
  H v;
  v.template load<V>(p, l);
  v.template rope<V>(cos_t + (size_t)ps * H::HALF, sin_t + (size_t)ps * H::HALF, l);
  v.template store<V>(p, l);
}

// The same with a head on 32 lanes, 4 bytes an access: where there are so few heads that a lane's 16 elements are a chain and leave SMs idle.
template <int NP>
__global__ void __launch_bounds__(128) rope_ref_pairs_kernel(const float* __restrict__ cos_t, const float* __restrict__ sin_t, bf16* x, int n_tok, const int* __restrict__ pos,
                                                             int pos0, int row_dim, int n_heads) {
  pdl_wait();
  pdl_trigger();
  const int at = (blockIdx.x * 128 + threadIdx.x) / 32, l = threadIdx.x % 32;
  if (at >= n_tok * n_heads) return;
  const int tok = at / n_heads, ps = pos ? pos[tok] : pos0 + tok;
  bf16* p = x + (size_t)tok * row_dim + (size_t)(at - tok * n_heads) * 64 * NP;
  float v[NP][2];
  head_load<NP>(v, p, l);
  head_rope<NP>(v, cos_t + (size_t)ps * 32 * NP, sin_t + (size_t)ps * 32 * NP, l);
  head_store<NP>(v, p, l);
}

bool on16(std::initializer_list<const void*> ps) {
  for (const void* p : ps)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

}  // namespace

// (head sizes are multiples of 64, so heads of an aligned row are aligned; strides off 8 elements and other addresses take 4-byte accesses)
#define QIE_HEADS(hd, vec, CALL)                                                                                  \
  if (hd == 64) { constexpr int NP = 1; if (vec) { constexpr bool V = true; CALL; } else { constexpr bool V = false; CALL; } }         \
  else if (hd == 128) { constexpr int NP = 2; if (vec) { constexpr bool V = true; CALL; } else { constexpr bool V = false; CALL; } }   \
  else if (hd == 256) { constexpr int NP = 4; if (vec) { constexpr bool V = true; CALL; } else { constexpr bool V = false; CALL; } }   \
  else return cudaErrorInvalidValue

static unsigned blocks_of(long heads, int hd) { return (unsigned)((heads * (hd / 16) + 127) / 128); }

cudaError_t launch_qkv_post(const QkvPostArgs& a, cudaStream_t st) {
  const long heads = (long)a.n_tok * (a.n_q + 2 * a.kv.n_kv);
  if (heads == 0) return cudaSuccess;
  const bool vec = on16({a.q, a.q_in, a.k, a.v, a.q_norm_w, a.k_norm_w, a.cos_t, a.sin_t, a.q_bias, a.k_bias, a.v_bias, a.kv.pool}) && a.q_in_stride % 8 == 0 &&
                   a.kv_stride % 8 == 0;
  QIE_HEADS(a.kv.hd, vec, return launched(launch_spread<qkv_post_kernel<NP, V>>(dim3(blocks_of(heads, a.kv.hd)), dim3(128), 0, st, a)));
}

cudaError_t launch_qknorm_ref(bf16* x, const bf16* w, int hd, int n_tok, int row_dim, int n_heads, cudaStream_t st) {
  const long heads = (long)n_tok * n_heads;
  if (heads == 0) return cudaSuccess;
  QIE_HEADS(hd, (on16({x, w}) && row_dim % 8 == 0),
            (void)launch_k(qknorm_ref_kernel<NP, V>, dim3(blocks_of(heads, hd)), dim3(128), 0, st, x, w, n_tok, row_dim, n_heads));
  return cudaGetLastError();
}

cudaError_t launch_rope_ref(const float* cos_t, const float* sin_t, bf16* x, int n_tok, const int* pos, int pos0, int hd, int row_dim, int n_heads, cudaStream_t st) {
  const long heads = (long)n_tok * n_heads;
  if (heads == 0) return cudaSuccess;
  // 16 elements a lane from 2048 heads of 64 on, as many elements of wider ones; off a 16-byte boundary from 6144 (256 wide from 40000 heads, since 32 lanes
  // read whole sectors and 16 do not).  us with 32 lanes and with 16 elements, alone: 17 heads of 64 1.2 1.3, 2800 1.6 1.8, 4000 1.7 1.8, 7168 2.5 1.8;
  // behind a norm and head norms 32 lanes are 1 us slower from about 3500 heads on (1792 of 128, the three operators 7.7 and 6.7) and the same below; off
  // a boundary 1 head 1.2 1.4, 4000 1.8 2.0, 7168 2.6 2.2; 14000 of 256 there 4.5 5.5, 42000 11.7 10.9.
  const bool vec = on16({x, cos_t, sin_t}) && row_dim % 8 == 0;
  if (heads * hd > 64L * (vec ? 2048 : hd < 256 ? 6144 : 160000)) {
    QIE_HEADS(hd, vec, (void)launch_k(rope_ref_kernel<NP, V>, dim3(blocks_of(heads, hd)), dim3(128), 0, st, cos_t, sin_t, x, n_tok, pos, pos0, row_dim, n_heads));
    return cudaGetLastError();
  }
  const auto pairs = hd == 64 ? rope_ref_pairs_kernel<1> : hd == 128 ? rope_ref_pairs_kernel<2> : hd == 256 ? rope_ref_pairs_kernel<4> : nullptr;
  if (!pairs) return cudaErrorInvalidValue;
  (void)launch_k(pairs, dim3((unsigned)((heads + 3) / 4)), dim3(128), 0, st, cos_t, sin_t, x, n_tok, pos, pos0, row_dim, n_heads);
  return cudaGetLastError();
}

}  // namespace qie
