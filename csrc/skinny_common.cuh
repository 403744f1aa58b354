// Cluster and programmatic-launch helpers of the decoding kernels.
#pragma once
#include "common.cuh"

namespace kf {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctaid() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Programmatic dependent launch.  wait: all work the previous kernel of the stream did (and everything before it) is
// complete and visible; returns at once in a kernel that was launched without the attribute.  launch: the next kernel
// of the stream may start its set-up; only ever called AFTER wait, so that whatever starts early still finds every
// kernel but its immediate predecessor complete.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace kf
