// launch.h -- kernel launch helper with programmatic dependent launch (PDL).
// Every kernel of the decode step starts with pdl_wait() (griddepcontrol.wait: all
// prerequisite grids complete, their writes visible) before it touches global memory, and
// calls pdl_trigger() (griddepcontrol.launch_dependents) behind it so the NEXT kernel's
// CTAs can be scheduled, set up their barriers/TMEM/tensor-map prefetch and -- for the
// GEMMs -- start streaming weights while this kernel is still running, where shared memory holds CTAs of both (a GEMM's ring of 192 to 224 KB
// lets it in beside a kernel of a few KB, or when CTAs of this one have left).  Never ahead of its own wait: then a third kernel comes in while the first one runs,
// and every start and end of a step's graph takes longer (GEMMs and decode attention that did, us a step of 24 layers of 0.5B widths and now: 64 rows at 2048 positions 1784 -> 1713,
// 48 at 300 1188 -> 1067, 16 at 500 1120 -> 996, 5 at 100 963 -> 895; 28 layers of 1.5B widths, 32 at 500 1856 -> 1760; fast numerics 1426 -> 1345, 931 -> 913).  A GEMM lets the next
// one in when its last load is on its way (behind its wait: 16 rows 1021, 1.5B 1782), decode attention when the softmax is done (in front of it 1754 and 1092 with GEMMs as they
// were, behind the softmax 1753 and 1067, at its end 1800 and 1128).  Launched without
// the attribute both instructions are no-ops, so the same kernels work eagerly.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <utility>

namespace qie {

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

extern bool g_use_pdl;  // engine.cu; set per process from QIE_PDL (default on)

// Function attributes (opt-in dynamic shared memory, cluster size) are per DEVICE: a process that creates engines on
// several devices must set them on each.  One flag per device ordinal instead of a process-wide `static bool`.
// Two threads that meet here both set the attributes.
struct PerDeviceOnce {
  std::atomic<unsigned long long> mask[4] = {};
  bool need() const {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 256) return true;
    return ((mask[d >> 6].load(std::memory_order_acquire) >> (d & 63)) & 1ull) == 0ull;
  }
  void done() {
    int d = 0;
    if (cudaGetDevice(&d) == cudaSuccess && d >= 0 && d < 256) mask[d >> 6].fetch_or(1ull << (d & 63), std::memory_order_release);
  }
};

template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                            Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_use_pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// What a launcher returns: the launch's own error, or one that an earlier call left; either way none is left for the next.
inline cudaError_t launched(cudaError_t e) {
  const cudaError_t last = cudaGetLastError();
  return e != cudaSuccess ? e : last;
}

// an attribute of a device, asked for once (0: the runtime does not say)
template <cudaDeviceAttr A>
inline int device_attribute(int dev) {
  static std::atomic<int> known[64] = {};
  int v = dev >= 0 && dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
  if (v == 0 && cudaDeviceGetAttribute(&v, A, dev) == cudaSuccess && dev >= 0 && dev < 64) known[dev].store(v, std::memory_order_relaxed);
  return v;
}

// The same for kernels of a few CTAs an SM that follow a GEMM.  A GEMM's CTAs fill the shared memory of their SMs; its dependents are scheduled when all
// of them have started, and so all at once onto the SMs that the GEMM left idle (36 of 148 with 112 tiles), where up to 16 CTAs then share an SM
// beside others without one.  Dynamic shared memory that they do not need leaves room for ceil(grid / SMs) of them on an SM.
// 512 rows of the norm behind a GEMM of 512 x 896 x 896: both 17.4 us without, 10.9 with the norm launched behind the GEMM's end, 10.6 so.
// Grids of at most one CTA an SM and of more than an SM's threads take at once are launched as they are.  Kernels have at most 700 bytes of static shared memory.
template <auto kernel, typename... Args>
inline cudaError_t launch_spread(dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  static PerDeviceOnce set;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int sms = device_attribute<cudaDevAttrMultiProcessorCount>(dev), all = device_attribute<cudaDevAttrMaxSharedMemoryPerMultiprocessor>(dev),
            most = device_attribute<cudaDevAttrMaxSharedMemoryPerBlockOptin>(dev);
  if (sms <= 0 || all <= 0 || most <= 0) return cudaErrorUnknown;
  const size_t ctas = (size_t)grid.x * grid.y * grid.z, per = (ctas + sms - 1) / sms;
  if (per > 1 && per * block.x <= 2048) {
    const size_t pad = (all / (per + 1) + 128) / 128 * 128 - 1024;  // (a CTA takes 1 KB more; per + 1 of them are more than there is)
    if (pad > smem) {
      if (set.need()) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - 1024);
        if (e != cudaSuccess) return e;
        set.done();
      }
      smem = pad;
    }
  }
  return launch_k(kernel, grid, block, smem, st, std::forward<Args>(args)...);
}

}  // namespace qie
