// Building blocks of the CTA-pair (tcgen05 cta_group::2) kernels: cluster rank / barrier, TMA loads whose bytes are
// counted on the leader CTA's barrier, the pair MMA, commits that reach both CTAs, remote barrier arrival and the
// pair forms of the tensor-memory allocator.  TMA loads carry no cluster multicast.
#pragma once
#include "common.cuh"

namespace kf {
namespace pairops {

constexpr uint32_t PEER_BIT_MASK = 0xFEFFFFFFu;  // clears the CTA-rank bit of a shared::cluster address

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA load whose completion bytes are counted on the LEADER CTA's barrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* m, uint32_t leader_bar, int c0,
                                                 int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(m), "r"(leader_bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void mma_pair_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_pair_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at the same shared-memory offset in both CTAs of the pair once all MMAs retired.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)0x3)
      : "memory");
}
// Arrival on a barrier of either CTA of the pair by an epilogue warp that hands an accumulator back: its values are in registers
// (tcgen05.wait::ld and the fence before), and no thread reads memory of this one after it.  It releases at CTA scope; at cluster scope
// it waited for every store the warp has in flight first, 3000 clocks per tile of the grouped weight gradient.
__device__ __forceinline__ void arrive_on_cta(uint32_t bar, uint32_t cta) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar),
      "r"(cta)
      : "memory");
}
// Arrival by a thread whose warp has written shared memory that the other CTA's matrix instructions are issued to read
// (fence.proxy.async before): releases at cluster scope, for the issuing thread's wait that acquires there (mbar_wait_cluster).
__device__ __forceinline__ void arrive_release_on_cta(uint32_t bar, uint32_t cta) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar),
      "r"(cta)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(ncols) : "memory");
}

// Bounded wait on a barrier of this CTA whose arrivals come from the other CTA of the pair (cluster-scope acquire).
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, int* status, int code) {
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((++spins & 0x3ff) == 0) {
      if (*reinterpret_cast<volatile int*>(status) != 0) return false;
      if (clock64() - t0 > KF_WAIT_CYCLES) {
        atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}

// Tile width of a pair launch for an (M, N) product and what it costs: rounds of tiles over the pairs, times the columns of a
// tile (multiples of 32 from 128 to 256, 256 rows), times a
// penalty for narrow tiles, whose operand bytes per MMA cycle exceed those of a 256-wide tile (64 per SM and clock): 10 % for
// the 96 of a 128-wide one, which is what a single-CTA 128 x 256 tile needs and loses against a pair.  A narrower tile has to
// save 4 %: less is within what the model leaves out.
inline int pair_tile_width(int M, int N, int pairs, float* cost_out) {
  const int m_blocks = (M + 255) / 256;
  int best = 256;
  float best_cost = 3.4e38f;
  for (int tn = 256; tn >= 128; tn -= 32) {
    const long long tiles = (long long)m_blocks * ((N + tn - 1) / tn);
    const long long rounds = (tiles + pairs - 1) / pairs;
    const float bytes_per_clk = (128.f + 0.5f * tn) * 64.f / tn;
    const float cost = float(rounds) * tn * (1.f + 0.1f * (bytes_per_clk - 64.f) / 32.f);
    if (cost < best_cost * (best == 256 ? 0.96f : 1.f)) {
      best = tn;
      best_cost = cost;
    }
  }
  if (cost_out) *cost_out = best_cost;
  return best;
}

}  // namespace pairops
}  // namespace kf
