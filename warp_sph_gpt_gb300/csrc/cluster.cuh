// cluster.cuh -- start of a thread-block cluster.
//
// The CTAs of a cluster are scheduled together, but one may run before another
// has started, and the shared memory of a CTA may be accessed by its peers only
// once it has.  A kernel whose CTAs write into a peer's shared memory calls
// cluster_started() first thing and cluster_wait_started() before the first such
// access, each by all threads of all its CTAs: the barrier passes while the
// kernel does its own work.
#pragma once

namespace sd {

__device__ __forceinline__ void cluster_started() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_started() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

}  // namespace sd
