// Weight gradient of the ragged grouped GEMM with CTA pairs (tcgen05 cta_group::2):
//
//   Out[e] (M x N) = A[rows of expert e, :M]^T * B[rows of expert e, :N]        for every expert e
//
// Same contract as the single-CTA kernel in grouped_wgrad_tcgen05.cu; a pair of CTAs owns a 256 x 256 tile of one
// expert's output.  CTA r loads, for every 64-row block of the expert's token range, columns [m0 + 128 r, + 128) of A
// and [n0 + 128 r, + 128) of B (both MN-major: the reduction index is the slow one in memory), 32 KB per CTA and
// k-block instead of the 48 KB of the 128 x 256 single-CTA tile.
//
// The ragged tail: the last 64-row block of an expert usually runs into the next expert's rows, and every CTA has to
// zero those rows of ITS OWN shared-memory stage before the MMAs read it.  Two hand-over protocols therefore:
//   full 64-row blocks   as in gemm_tcgen05_2cta.cu: both CTAs' TMA bytes are counted on the leader's full[s]
//   the tail block       (at most one per tile) each CTA's loads complete on its own tail[s]; warp 6 of each CTA waits
//                        for it, zeroes the foreign rows of its own stage up to the next multiple of 16 (only those
//                        k-steps are issued), fences them towards the async proxy and arrives (release) on the leader's
//                        ready[s]; the issuing thread waits for both arrivals (cluster-scope acquire) before the MMAs.
//                        The ring runs ahead of the MMAs, so the rows are usually clear before their turn; zeroing all
//                        64 rows inside the issuing warp held up every tile by about as long as a k-block (64 experts of
//                        2048 x 1408 over 10 662 rows: 484 -> 397 us for three gradients; 8 of 2048 x 7168: 464 -> 414).
//   empty[s]             both CTAs: released by the leader's tcgen05.commit, multicast to the pair
//   tfull[a] / tempty[a] as in gemm_tcgen05_2cta.cu (8 epilogue-warp arrivals on the leader)
// full[s] completes a phase per full block in stage s, tail[s] and ready[s] one per tail block; every side waits for all
// phases of its barriers in order and keeps one parity bit per stage for each.
// (Relaying every block through the peer's warp was measured 2.4x slower than the single-CTA kernel.)
// All waits are bounded; TMA loads carry no cluster multicast.
//
// Epilogue.  An expert's reduction is short (167 rows = 3 k-blocks of 0.4 us for 64 experts over 10 662 rows), so the tile's
// way out, not its products, sets the pace.  With one row per thread every 16-byte store of a warp touched 32 different
// lines: 5.5 us per tile.  Each epilogue warp therefore stages 32 rows x 64 columns in shared memory (two 4 KB buffers,
// 128-byte swizzle: no bank conflicts) and one lane stores them with TMA: whole lines, asynchronously, clipped at the
// expert's last row and column by the 3-D tensor map.  Three gradients of 64 experts of 2048 x 1408 over 10 662 rows: 685 -> 480 us
// with this; of 8 experts of 2048 x 7168 over 4096 rows: 530 -> 441 us.
//
// What held such short tiles up after that was synchronisation: arrivals that waited for the warp's stores (see arrive_on_cta), row
// offsets read from global memory by every role of every tile (400 clocks each), and the cleared rows' addresses.  The three
// gradients, 64 experts: 417 -> 304 us (3.7 TB/s of gradients written); 8 experts: 374 -> 304 us (1190 TFLOP/s), sixth stage included.
// (The arrival after the cleared rows, which does publish memory, releases at cluster scope: layers of 8 and of 64 experts 1301 -> 1303
// and 1143 -> 1151 us, within their spread.)
//
// Replaces the per-expert weight-gradient products that autograd derives for the padded `torch._grouped_mm`
// call of the reference (kempnerforge/model/moe.py:20-145).
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tile_math.h"
#include "pair_common.cuh"

namespace kf {
namespace gwg2 {

using namespace kf::pairops;

constexpr int CTA_M = 128, TILE_M = 256, TILE_N = 256, HALF_N = 128, BK = 64, STAGES = 6, UMMA_K = 16;
constexpr int BLOCK_BYTES = 64 * BK * 2;  // one {64 columns, BK rows} box
constexpr int A_BYTES = (CTA_M / 64) * BLOCK_BYTES, B_BYTES = (HALF_N / 64) * BLOCK_BYTES;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int THREADS = 224, TMEM_COLS = 512;
constexpr int OUT_BYTES = 32 * 64 * 2;  // one staged box: 32 rows x 64 columns of one epilogue warp
constexpr int MAX_TABLE = 256;           // up to so many experts the row offsets are kept in shared memory
constexpr size_t SMEM = size_t(STAGES) * STAGE_BYTES + 4 * 2 * OUT_BYTES + 1024 + 256 + (MAX_TABLE + 1) * 4;

using Tile = tilemath::WgradTile;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
kf_grouped_wgrad_tcgen05_2cta(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                              const __grid_constant__ CUtensorMap map_o, const int* __restrict__ row_offsets, int E, int M, int N,
                              int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t out_smem = smem_base + STAGES * STAGE_BYTES;  // [epilogue warp][2] boxes
  const uint32_t bar_base = out_smem + 4 * 2 * OUT_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto ready_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
  auto tail_bar = [&](int s) { return bar_base + 8u * (3 * STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (4 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (4 * STAGES + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (4 * STAGES + 4);
  const uint32_t tmem_slot = bar_base + 8u * (4 * STAGES + 5);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int m_blocks = (M + TILE_M - 1) / TILE_M, n_blocks = (N + TILE_N - 1) / TILE_N;
  const int num_tiles = E * m_blocks * n_blocks;

  // Every role of every tile looks its expert's rows up; from global memory that held each of them up by 400 clocks.
  int* table = reinterpret_cast<int*>(smem_raw + (bar_base + 256 - smem_u32(smem_raw)));
  const int* offsets = E <= MAX_TABLE ? table : row_offsets;
  if (E <= MAX_TABLE)
    for (int i = threadIdx.x; i <= E; i += THREADS) table[i] = row_offsets[i];
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
      mbar_init(ready_bar(s), 2);  // the tail warps of both CTAs
      mbar_init(tail_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 8);
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    tma_prefetch_desc(&map_o);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) {
      int it = 0;
      uint32_t full_parity = 0, tail_parity = 0, last_tail = 0;  // bit s: next phases of stage s, kind of its last use
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const Tile tl = tilemath::wgrad_decode(t, m_blocks, n_blocks, TILE_M, TILE_N, offsets);
        const int k_blocks = (tl.rows + BK - 1) / BK;
        const int m0 = tl.m0 + int(rank) * CTA_M, n0 = tl.n0 + int(rank) * HALF_N;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t a_dst = smem_base + s * STAGE_BYTES, b_dst = a_dst + A_BYTES;
          const int row = tl.row0 + kb * BK;
          if (tl.rows - kb * BK < BK) {
            // tail block: every CTA's bytes complete on its own tail barrier (its warp 6 zeroes the foreign rows)
            mbar_expect_tx(tail_bar(s), STAGE_BYTES);
#pragma unroll
            for (int c = 0; c < CTA_M / 64; ++c) tma_load_2d(a_dst + c * BLOCK_BYTES, &map_a, tail_bar(s), m0 + 64 * c, row);
#pragma unroll
            for (int c = 0; c < HALF_N / 64; ++c) tma_load_2d(b_dst + c * BLOCK_BYTES, &map_b, tail_bar(s), n0 + 64 * c, row);
            tail_parity ^= 1u << s;
            last_tail |= 1u << s;
          } else {
            full_parity ^= 1u << s;
            last_tail &= ~(1u << s);
            const uint32_t lead_full = full_bar(s) & PEER_BIT_MASK;
            if (leader) mbar_expect_tx(full_bar(s), 2 * STAGE_BYTES);
#pragma unroll
            for (int c = 0; c < CTA_M / 64; ++c) tma_load_2d_pair(a_dst + c * BLOCK_BYTES, &map_a, lead_full, m0 + 64 * c, row);
#pragma unroll
            for (int c = 0; c < HALF_N / 64; ++c) tma_load_2d_pair(b_dst + c * BLOCK_BYTES, &map_b, lead_full, n0 + 64 * c, row);
          }
        }
      }
      // Copies into this CTA's shared memory are complete once the stages they filled were consumed (empty flipped)
      // or, on the error path, once the barrier that counts them flipped.
      for (int s = 0; s < min(it, STAGES); ++s) {
        if ((last_tail >> s) & 1) mbar_wait(tail_bar(s), ((tail_parity >> s) & 1) ^ 1, status, KF_ERR_WAIT_DRAIN);
        else if (leader) mbar_wait(full_bar(s), ((full_parity >> s) & 1) ^ 1, status, KF_ERR_WAIT_DRAIN);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(TILE_M, TILE_N, true, true);
      int it = 0, tile_iter = 0;
      uint32_t full_parity = 0, ready_parity = 0;  // bit s: parity of the next full / tail use of stage s
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
        const Tile tl = tilemath::wgrad_decode(t, m_blocks, n_blocks, TILE_M, TILE_N, offsets);
        const int k_blocks = (tl.rows + BK - 1) / BK;
        const int acc = tile_iter & 1;
        if (!mbar_wait(tempty_bar(acc), ((tile_iter >> 1) & 1) ^ 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TILE_N;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const int valid = tl.rows - kb * BK;
          if (valid >= BK) {
            if (!mbar_wait(full_bar(s), (full_parity >> s) & 1, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
            full_parity ^= 1u << s;
          } else {
            if (!mbar_wait_cluster(ready_bar(s), (ready_parity >> s) & 1, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
            ready_parity ^= 1u << s;
          }
          tc_fence_after();
          const uint32_t a_src = smem_base + s * STAGE_BYTES, b_src = a_src + A_BYTES;
          const int steps = valid < BK ? (valid + UMMA_K - 1) / UMMA_K : BK / UMMA_K;
          for (int k = 0; k < steps; ++k)
            mma_pair_f16(d_tmem, umma_desc_sw128(a_src + k * (UMMA_K * 128), BLOCK_BYTES, 1024),
                         umma_desc_sw128(b_src + k * (UMMA_K * 128), BLOCK_BYTES, 1024), idesc, (kb | k) != 0);
          commit_pair(empty_bar(s));
        }
        if (ok) commit_pair(tfull_bar(acc));
      }
      // every MMA must have retired before either CTA gives up its shared or tensor memory
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain_bar)
                   : "memory");
      mbar_wait(drain_bar, 0, status, KF_ERR_WAIT_DRAIN);
    }
    __syncwarp();
  } else if (warp == 6) {
    // ------------------------------------------------------------ tail rows of this CTA's stages (both CTAs)
    int it = 0;
    uint32_t tail_parity = 0;  // bit s: parity of the next tail use of stage s
    for (int t = pair; t < num_tiles; t += num_pairs) {
      const Tile tl = tilemath::wgrad_decode(t, m_blocks, n_blocks, TILE_M, TILE_N, offsets);
      const int k_blocks = (tl.rows + BK - 1) / BK;
      const int valid = tl.rows - (k_blocks - 1) * BK;
      if (k_blocks > 0 && valid < BK) {
        const int s = (it + k_blocks - 1) % STAGES;
        if (!__all_sync(0xffffffffu, mbar_wait(tail_bar(s), (tail_parity >> s) & 1, status, KF_ERR_WAIT_FULL))) break;
        tail_parity ^= 1u << s;
        static_assert(STAGE_BYTES == 4 * BLOCK_BYTES, "a lane owns one 16-byte chunk of the rows of one of four blocks");
        const int end = (valid + UMMA_K - 1) / UMMA_K * UMMA_K;  // rows the MMAs will read
        const uint32_t chunk = smem_base + s * STAGE_BYTES + (lane >> 3) * BLOCK_BYTES + (lane & 7) * 16;
        for (int r = valid; r < end; ++r)
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(chunk + r * 128), "r"(0u) : "memory");
        fence_async_smem();
        __syncwarp();
        if (lane == 0) arrive_release_on_cta(ready_bar(s), 0);  // this CTA's half of the stage is in place
      }
      it += k_blocks;
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5 of both CTAs)
    const int quarter = warp & 3;
    int tile_iter = 0, boxes = 0;
    bool ok = true;
    for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
      const Tile tl = tilemath::wgrad_decode(t, m_blocks, n_blocks, TILE_M, TILE_N, offsets);
      const int acc = tile_iter & 1;
      if (!mbar_wait(tfull_bar(acc), (tile_iter >> 1) & 1, status, KF_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int row0 = tl.m0 + int(rank) * CTA_M + quarter * 32;  // first of this warp's 32 rows
      const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * TILE_N;
      const int n_boxes = row0 < M ? min(TILE_N / 64, (N - tl.n0 + 63) / 64) : 0;
#pragma unroll 1
      for (int c = 0; c < n_boxes; ++c, ++boxes) {
        uint32_t lo[32], hi[32];
        if (tl.rows > 0) {
          tmem_ld_32x32(t_row + c * 64, lo);
          tmem_ld_32x32(t_row + c * 64 + 32, hi);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) lo[i] = hi[i] = 0u;
        }
        const uint32_t box = out_smem + uint32_t((quarter * 2 + (boxes & 1)) * OUT_BYTES);
        if (lane == 0) tma_store_wait_read<1>();  // the store that last used this buffer has read it
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t* v = q < 4 ? lo + q * 8 : hi + (q - 4) * 8;
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) w[i] = pack_bf16(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(box + uint32_t(lane * 128 + ((q ^ (lane & 7)) << 4))),
                       "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(&map_o, box, tl.n0 + c * 64, row0, tl.e);
          tma_store_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_on_cta(tempty_bar(acc), 0);
    }
    if (lane == 0) tma_store_wait<0>();
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's shared and tensor memory stay alive until the leader's MMAs have retired
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// Contract of kf_grouped_wgrad_bf16 (grouped_wgrad_tcgen05.cu), which dispatches here.
int launch_grouped_wgrad_2cta(const void* A, const void* B, void* Out, const void* offsets, int rows, int E, int M, int N,
                              long long lda, long long ldb, int num_sms, cudaStream_t stream, int* status) {
  CUtensorMap ma, mb;
  int rc = make_map_2d_bf16(&ma, A, rows, M, lda, 64, BK);
  if (rc) return 100 + rc;
  rc = make_map_2d_bf16(&mb, B, rows, N, ldb, 64, BK);
  if (rc) return 200 + rc;
  CUtensorMap mo;
  rc = make_map_3d_bf16(&mo, Out, E, M, N, 64, 32, N);
  if (rc) return 300 + rc;
  const long long tiles = (long long)E * ((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N);
  int pairs = num_sms / 2;
  if (tiles < pairs) pairs = (int)tiles;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kf_grouped_wgrad_tcgen05_2cta, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_set = true;
  }
  kf_grouped_wgrad_tcgen05_2cta<<<pairs * 2, THREADS, SMEM, stream>>>(
      ma, mb, mo, reinterpret_cast<const int*>(offsets), E, M, N, status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace gwg2
}  // namespace kf
