// Ragged grouped GEMM (mixture-of-experts feed-forward) with CTA pairs (tcgen05 cta_group::2):
//
//   C[rows of expert e, :N] (+)= A[rows of expert e, :K] * op(B_e)          for every expert e
//
// Same contract as the single-CTA kernel in grouped_gemm_tcgen05.cu (expert-sorted rows, int32 `offsets` on the
// device, nothing padded, no host read), with the tiling of the dense CTA-pair GEMM: two CTAs on neighbouring SMs own
// a 256 x 256 output tile, CTA r loads 128 of the tile's rows of A and 128 of its rows / columns of B, the leader
// issues 256 x 256 x 16 MMAs that read both CTAs' shared memory.  Per CTA and k-block 32 KB are loaded instead of the
// 48 KB of the 128 x 256 single-CTA tile, which leaves six pipeline stages and takes the shared-memory read port off
// the critical path.  A row tile never crosses an expert boundary: tiles are counted per expert (256 rows each, the
// last one partial) and the epilogue stores only the rows that belong to the expert.
//
// SWIGLU: two weight operands (gate: map_b, up: map_b2) of N = F hidden units each; a tile covers 128 hidden units,
// the leader CTA loads their gate weights and the peer the matching up weights, so every CTA's accumulator holds
// [gate 128 | up 128] for its 128 rows; the epilogue writes h = silu(gate) * up and optionally the pre-activations.
//
// EPI == 2: SwiGLU backward in the epilogue of the down projection's input-gradient product (see the launcher).
//
// EPI == 3: C = A_1 B_e + A_2 B2_e with A = [A_1 | A_2] side by side (the input gradient of the gate and up projections as
// one product over K = 2 F): no second pass over C, and the sum is rounded once.
//
// NE > 1: every expert's weight has a tensor map of its own (up to NE of them, kernel parameters), so the weights of
// separate Linear modules are read where they are; NE == 1: one packed (E, .., ..) tensor.  For 8 experts of 2048 x 7168
// the copies this saves move 1.4 GB per forward pass.
//
// Synchronisation as in gemm_tcgen05_2cta.cu (all waits bounded); TMA loads carry no cluster multicast.
// Replaces the padded torch._grouped_mm calls of the reference (kempnerforge/model/moe.py:20-145).
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tile_math.h"
#include "pair_common.cuh"

namespace kf {
namespace grp2 {

using namespace kf::pairops;

constexpr int CTA_M = 128, TILE_M = 256, TILE_N = 256, HALF_N = 128, BK = 64, STAGES = 6, UMMA_K = 16;
constexpr int A_BYTES = CTA_M * BK * 2, B_BYTES = HALF_N * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int THREADS = 192, TMEM_COLS = 512;
constexpr int MAX_EXPERTS = 256;
constexpr int BOX_BYTES = 2048;  // rows of an epilogue warp on their way to or from global memory; two per warp
constexpr size_t SMEM = size_t(STAGES) * STAGE_BYTES + 8 * BOX_BYTES + 1024 + 256 + (MAX_EXPERTS + 1) * 4;

using Tile = tilemath::GroupedTile;

template <int NE>
struct Maps {
  CUtensorMap m[NE];
};
constexpr int MAX_SEPARATE = 32;  // experts with a tensor map of their own (two operands: 8 KB of kernel parameters)

template <bool B_MN, int EPI, int NE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
kf_grouped_gemm_tcgen05_2cta(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ Maps<NE> maps_b,
                             const __grid_constant__ Maps<(EPI & 1) ? NE : 1> maps_b2, __nv_bfloat16* __restrict__ C,
                             __nv_bfloat16* __restrict__ GU, const int* __restrict__ offsets, int E, int N, int K,
                             long long ldc, long long ldgu, int accumulate, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t box_smem = smem_base + STAGES * STAGE_BYTES;
  const uint32_t bar_base = box_smem + 8 * BOX_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 5);
  uint8_t* bar_gen = smem_raw + (bar_base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(bar_gen + 8 * (2 * STAGES + 5));
  int* tile_start = reinterpret_cast<int*>(bar_gen + 256);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  constexpr bool SWIGLU = EPI == 1;
  constexpr int TN = SWIGLU ? HALF_N : TILE_N;  // output columns (hidden units) per tile
  const int n_blocks = (N + TN - 1) / TN;
  const int k_blocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 8);
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    if (NE == 1) {
      tma_prefetch_desc(&maps_b.m[0]);
      if (EPI & 1) tma_prefetch_desc(&maps_b2.m[0]);
    }
    tilemath::grouped_tile_starts(offsets, E, TILE_M, tile_start);  // both CTAs of a pair compute the same table
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
  const int num_tiles = tile_start[E] * n_blocks;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) {
      int it = 0;
      bool ok = true;
      // the leader fetches the gate weights (or the first 128 columns), the peer the up weights (or the last 128)
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const Tile tl = tilemath::grouped_decode(t, n_blocks, tile_start, offsets, E, TILE_M);
        const int m0 = tl.row0 + int(rank) * CTA_M;
        const int n0 = SWIGLU ? tl.nb * TN : tl.nb * TN + int(rank) * HALF_N;
        const int me = NE > 1 ? tl.e : 0;              // tensor map and first row of the expert's weight inside it
        const int e_n = NE > 1 ? 0 : tl.e * N, e_k = NE > 1 ? 0 : tl.e * (EPI == 3 ? K / 2 : K);
        const CUtensorMap* my_b = (SWIGLU && !leader) ? &maps_b2.m[me] : &maps_b.m[me];
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(empty_bar(s), ph ^ 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t a_dst = smem_base + s * STAGE_BYTES;
          const uint32_t b_dst = a_dst + A_BYTES;
          const uint32_t lead_full = full_bar(s) & PEER_BIT_MASK;
          if (leader) mbar_expect_tx(full_bar(s), 2 * STAGE_BYTES);
          const int k0 = kb * BK;
          tma_load_2d_pair(a_dst, &map_a, lead_full, k0, m0);
          int kw = k0;                                 // reduction index inside the weight
          if (EPI == 3 && k0 >= K / 2) {
            my_b = &maps_b2.m[me];
            kw = k0 - K / 2;
          }
          if (!B_MN) {
            tma_load_2d_pair(b_dst, my_b, lead_full, kw, e_n + n0);
          } else {
#pragma unroll
            for (int c = 0; c < HALF_N / 64; ++c)
              tma_load_2d_pair(b_dst + c * (64 * BK * 2), my_b, lead_full, n0 + 64 * c, e_k + kw);
          }
        }
      }
      // Copies into this CTA's shared memory are complete once the stages they filled were consumed (empty
      // flipped) or, on the error path, once the leader's full barrier flipped.
      if (leader)
        for (int j = max(0, it - STAGES); j < it; ++j)
          mbar_wait(full_bar(j % STAGES), (j / STAGES) & 1, status, KF_ERR_WAIT_DRAIN);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(TILE_M, TILE_N, false, B_MN);
      int it = 0, tile_iter = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
        const int acc = tile_iter & 1;
        const uint32_t acc_ph = (tile_iter >> 1) & 1;
        if (!mbar_wait(tempty_bar(acc), acc_ph ^ 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TILE_N;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(full_bar(s), ph, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_src = smem_base + s * STAGE_BYTES;
          const uint32_t b_src = a_src + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t bd = B_MN ? umma_desc_sw128(b_src + k * (UMMA_K * 128), 64 * BK * 2, 1024)
                                     : umma_desc_sw128(b_src + k * (UMMA_K * 2), 16, 1024);
            mma_pair_f16(d_tmem, umma_desc_sw128(a_src + k * (UMMA_K * 2), 16, 1024), bd, idesc, (kb | k) != 0);
          }
          commit_pair(empty_bar(s));
        }
        if (ok) commit_pair(tfull_bar(acc));
      }
      // every MMA must have retired before either CTA gives up its shared or tensor memory
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain_bar)
                   : "memory");
      mbar_wait(drain_bar, 0, status, KF_ERR_WAIT_DRAIN);
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5 of both CTAs)
    const int quarter = warp & 3;
    int tile_iter = 0;
    bool ok = true;
    for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
      const Tile tl = tilemath::grouped_decode(t, n_blocks, tile_start, offsets, E, TILE_M);
      const int acc = tile_iter & 1;
      const int r0 = int(rank) * CTA_M + quarter * 32;  // first row of this warp inside the 256-row tile
      const int rows = max(0, min(32, tl.valid - r0));  // how many of its 32 rows belong to the expert
      const int col0 = tl.nb * TN, width = min(TN, N - col0);
      const uint32_t box = box_smem + uint32_t(quarter * 2) * BOX_BYTES, box2 = box + BOX_BYTES;
      __nv_bfloat16* c0 = C + size_t(tl.row0 + r0) * ldc + col0;
      __nv_bfloat16* gu0 = GU ? GU + size_t(tl.row0 + r0) * ldgu + col0 : nullptr;
      Rows32 g_next, u_next;
      if constexpr (EPI == 2) {  // the first pre-activations travel while the tile's products are still running
        g_next = load_rows32(gu0, ldgu, lane, rows, width);
        u_next = load_rows32(gu0 + N, ldgu, lane, rows, width);
      }
      if (!mbar_wait(tfull_bar(acc), (tile_iter >> 1) & 1, status, KF_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * TILE_N;
#pragma unroll 1
      for (int c = 0; c * 32 < width; ++c) {
        const int cols = min(32, width - c * 32);
        if constexpr (EPI == 2) {
          // SwiGLU backward: the accumulator is dh[rows, F] (never written); GU = the saved pre-activations [rows, 2F]
          // (gate | up), C = d[gate | up] [rows, 2F] (may be the same buffer: a warp reads a chunk before it writes it, and
          // no other warp touches its rows)
          uint32_t v[32];
          tmem_ld_32x32(t_row + c * 32, v);
          const Rows32 g_now = g_next, u_now = u_next;  // chunk c + 1 is fetched while chunk c is worked on
          if ((c + 1) * 32 < width) {
            g_next = load_rows32(gu0 + (c + 1) * 32, ldgu, lane, rows, width - (c + 1) * 32);
            u_next = load_rows32(gu0 + N + (c + 1) * 32, ldgu, lane, rows, width - (c + 1) * 32);
          }
          Rows32 g = to_own_row(box, lane, g_now), u = to_own_row(box2, lane, u_now);
          tmem_ld_wait();
          swiglu_bwd_row(v, g, u);
          store_rows32(box, lane, g, c0 + c * 32, ldc, rows, cols);
          store_rows32(box2, lane, u, c0 + N + c * 32, ldc, rows, cols);
        } else if constexpr (SWIGLU) {
          uint32_t g[32], u[32];
          tmem_ld_32x32(t_row + c * 32, g);
          tmem_ld_32x32(t_row + TN + c * 32, u);
          tmem_ld_wait();
          if (gu0) {
            store_rows32(box, lane, pack_row32(g), gu0 + c * 32, ldgu, rows, cols);
            store_rows32(box2, lane, pack_row32(u), gu0 + N + c * 32, ldgu, rows, cols);
          }
          swiglu_chunk(g, u);
          store_rows32(box, lane, pack_row32(g), c0 + c * 32, ldc, rows, cols);
        } else {
          uint32_t v[32];
          tmem_ld_32x32(t_row + c * 32, v);
          tmem_ld_wait();
          if (accumulate) {
            if (lane < rows) store_chunk<__nv_bfloat16>(c0 + size_t(lane) * ldc + c * 32, v, cols, true, nullptr);
          } else {
            store_rows32(box, lane, pack_row32(v), c0 + c * 32, ldc, rows, cols);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_on_cta(tempty_bar(acc), 0);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's shared and tensor memory stay alive until the leader's MMAs have retired
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <bool B_MN, int EPI, int NE>
static int launch(const CUtensorMap& ma, const Maps<NE>& mb, const Maps<(EPI & 1) ? NE : 1>& mb2, void* C, void* GU,
                  const void* offsets, int E, int N, int K, long long ldc, long long ldgu, int accumulate, int pairs,
                  cudaStream_t st, int* status) {
  auto kern = kf_grouped_gemm_tcgen05_2cta<B_MN, EPI, NE>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_set = true;
  }
  kern<<<pairs * 2, THREADS, SMEM, st>>>(ma, mb, mb2, reinterpret_cast<__nv_bfloat16*>(C), reinterpret_cast<__nv_bfloat16*>(GU),
                                         reinterpret_cast<const int*>(offsets), E, N, K, ldc, ldgu, accumulate, status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

// Weight operand: the packed tensor (NE == 1, *w) or one pointer per expert.  Each expert's matrix is [N][K] (K
// contiguous, boxes of 128 rows) or, b_mn, [K][N] (N contiguous, 64 x 64 boxes).
template <int NE>
static int make_weight_maps(Maps<NE>& m, const void* const* w, int E, int N, int K, int b_mn) {
  for (int e = 0; e < (NE > 1 ? E : 1); ++e) {
    const uint64_t n = NE > 1 ? 1 : E;
    const int rc = b_mn ? make_map_2d_bf16(&m.m[e], w[e], n * K, N, N, 64, BK) : make_map_2d_bf16(&m.m[e], w[e], n * N, K, K, BK, HALF_N);
    if (rc) return rc;
  }
  return 0;
}

static int pair_count(int rows, int E, int n_blocks, int num_sms) {
  const int upper = ((rows + TILE_M - 1) / TILE_M + E) * n_blocks;  // at most one partial tile per expert
  return upper < num_sms / 2 ? upper : num_sms / 2;
}

template <int EPI, int NE>
static int run(const void* A, const void* const* W, const void* const* W2, void* C, void* GU, const void* offsets, int rows,
               int E, int N, int K, int KW, long long lda, long long ldc, long long ldgu, int b_mn, int accumulate, int num_sms,
               cudaStream_t st, int* status) {
  CUtensorMap ma;
  Maps<NE> mb;
  Maps<(EPI & 1) ? NE : 1> mb2;
  int rc = make_map_2d_bf16(&ma, A, rows, K, lda, BK, CTA_M);
  if (rc) return 100 + rc;
  rc = make_weight_maps<NE>(mb, W, E, N, KW, b_mn);
  if (!rc && (EPI & 1)) rc = make_weight_maps<(EPI & 1) ? NE : 1>(mb2, W2, E, N, KW, b_mn);
  if (rc) return 200 + rc;
  if (!(EPI & 1)) mb2.m[0] = mb.m[0];
  const int tn = EPI == 1 ? HALF_N : TILE_N;
  const int pairs = pair_count(rows, E, (N + tn - 1) / tn, num_sms);
  return b_mn ? launch<true, EPI, NE>(ma, mb, mb2, C, GU, offsets, E, N, K, ldc, ldgu, accumulate, pairs, st, status)
              : launch<false, EPI, NE>(ma, mb, mb2, C, GU, offsets, E, N, K, ldc, ldgu, accumulate, pairs, st, status);
}

// Contracts of kf_grouped_gemm_acc_bf16 / kf_grouped_swiglu_bf16 (grouped_gemm_tcgen05.cu), which dispatch here.
int launch_grouped_gemm_2cta(const void* A, const void* B, void* C, const void* offsets, int rows, int E, int N, int K,
                             long long lda, long long ldc, int b_mn, int accumulate, int num_sms, cudaStream_t st, int* status) {
  return run<0, 1>(A, &B, nullptr, C, nullptr, offsets, rows, E, N, K, K, lda, ldc, 0, b_mn, accumulate, num_sms, st, status);
}

int launch_grouped_swiglu_2cta(const void* A, const void* Wg, const void* Wu, void* H, void* GU, const void* offsets, int rows,
                               int E, int F, int K, long long lda, long long ldh, long long ldgu, int b_mn, int num_sms,
                               cudaStream_t st, int* status) {
  return run<1, 1>(A, &Wg, &Wu, H, GU, offsets, rows, E, F, K, K, lda, ldh, ldgu, b_mn, 0, num_sms, st, status);
}

// d[gate | up] (rows x 2F, may alias GU) from dy (rows x K) and the down weights: W [E][F][K] (b_mn == 0: K
// contiguous) or [E][K][F] (b_mn == 1); the accumulator dh = dy W_e^T (resp. dy W_e) is consumed by the epilogue.
int launch_grouped_swiglu_bwd_2cta(const void* DY, const void* W, const void* GU, void* DGU, const void* offsets, int rows,
                                   int E, int F, int K, long long lda, long long ldgu, int b_mn, int num_sms, cudaStream_t st,
                                   int* status) {
  return run<2, 1>(DY, &W, nullptr, DGU, const_cast<void*>(GU), offsets, rows, E, F, K, K, lda, ldgu, ldgu, b_mn, 0, num_sms, st,
                   status);
}

}  // namespace grp2
}  // namespace kf

extern "C" void* kf_status_device_ptr();

extern "C" {

// The grouped products of an expert feed-forward with either packed weights (separate == 0: w[0] is the (E, .., ..) tensor)
// or one matrix per expert (separate != 0: w[e], E <= 32; host arrays of device pointers).  CTA-pair tiles; rows >= 1.
//   kind 0: C = A W_e;  1: C = silu(A W_e) * (A W2_e), GU (optional) the pre-activations;  2: C = SwiGLU'(GU) * (A W_e);
//   kind 3: C = A[:, :K/2] W_e + A[:, K/2:] W2_e  (K / 2 a multiple of 64).
// W_e: [N][K] (b_mn == 0) or [K][N] (b_mn == 1, K % 64 == 0); kind 3: K / 2 in its place.  Pitches multiples of 8.
int kf_grouped_experts_bf16(int kind, const void* A, const void* const* w, const void* const* w2, int separate, void* C,
                            void* GU, const void* offsets, int rows, int E, int N, int K, long long lda, long long ldc,
                            long long ldgu, int b_mn, int num_sms, void* stream) {
  using namespace kf::grp2;
  const int KW = kind == 3 ? K / 2 : K;
  if (E < 1 || E > (separate ? MAX_SEPARATE : MAX_EXPERTS) || (lda & 7) || (ldc & 7) || (GU && (ldgu & 7)) || (K & 7) ||
      (N & 7) || ((b_mn || kind == 3) && (KW % BK)) || num_sms < 2 || kind < 0 || kind > 3)
    return 5;
  if (rows <= 0) return 0;
  int* status = reinterpret_cast<int*>(kf_status_device_ptr());
  cudaStream_t st = (cudaStream_t)stream;
#define KF_EXPERTS(EPI_)                                                                                                      \
  return separate ? run<EPI_, MAX_SEPARATE>(A, w, w2, C, GU, offsets, rows, E, N, K, KW, lda, ldc, ldgu, b_mn, 0, num_sms, st, status) \
                  : run<EPI_, 1>(A, w, w2, C, GU, offsets, rows, E, N, K, KW, lda, ldc, ldgu, b_mn, 0, num_sms, st, status)
  switch (kind) {
    case 0: KF_EXPERTS(0);
    case 1: KF_EXPERTS(1);
    case 2: KF_EXPERTS(2);
    default: KF_EXPERTS(3);
  }
#undef KF_EXPERTS
}

}  // extern "C"
