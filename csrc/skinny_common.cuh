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

// (x, y) rotated by the angle of (c, s), spelled out because which of two products is fused with their sum decides one bf16 value in
// 10^5, and the compiler chooses differently from kernel to kernel.  This is the choice of the rotary kernel.
__device__ __forceinline__ void rotate_pair(float x, float y, float c, float s, float& rx, float& ry) {
  rx = __fmaf_rn(x, c, -__fmul_rn(y, s));
  ry = __fmaf_rn(y, c, __fmul_rn(x, s));
}

// The same in the epilogue of a generation step.  Heads of 64 keep the bits of the rotary kernel, which rotated them before that
// epilogue did; heads of 128 keep those that the epilogue has always had, with the other product fused in the second half.
__device__ __forceinline__ void rotate_pair_step(int hd, float x, float y, float c, float s, float& rx, float& ry) {
  float other;
  rotate_pair(x, y, c, s, rx, other);
  ry = hd == 64 ? other : __fmaf_rn(x, s, __fmul_rn(y, c));
}

__device__ __forceinline__ float norm_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace kf
