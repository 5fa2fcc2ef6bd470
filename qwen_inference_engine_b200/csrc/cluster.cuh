// cluster.cuh -- the barrier of a thread-block cluster.
#pragma once

namespace qie {

// Every thread of every CTA of the cluster.  The .aligned forms want a warp's threads together, and the loops in front of them end per
// thread: __syncwarp brings them there whatever the compiler makes of the loop.
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace qie
