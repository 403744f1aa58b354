// Ragged grouped GEMM (mixture-of-experts feed-forward) with CTA pairs (tcgen05 cta_group::2):
//
//   C[rows of expert e, :N] (+)= A[rows of expert e, :K] * op(B_e)          for every expert e
//
// Same contract as the single-CTA kernel in grouped_gemm_tcgen05.cu: expert-sorted rows, int32 `offsets` on the device, nothing padded,
// no host read.
//
// Tiles.  The weights are the M side of the MMA (256 rows of B_e per pair, 128 per CTA) and the tokens its N side, as in
// gemm_tokens_tcgen05_2cta.cu: an expert's rows are cut into equal tiles of a multiple of 32, up to 256, and never cross its end.  An
// MMA's time follows its N side (see warp_index in common.cuh; a k-block of a pair takes about 1.45 ns per token and 70 ns), so a tile costs what
// its tokens do.  With the tokens as the M side every tile was 256 rows: 167 rows per expert (64 experts, top 6 of 1777 tokens) paid for
// 256, and 520 for 768.  The widest tile allowed is chosen on the device, once per CTA, so that rounds of tiles over the pairs times the
// average tile are least: 8 experts of about 512 rows and 2048 output columns are 160 tiles of 256, three rounds of the 74 pairs, or
// 192 tiles of 192 in the same three.
// All token tiles of a block of 256 weight rows are neighbours in the tile order, so the weights cross the L2 cache once.
// What bounds them now: 64 experts stream their weights (gate and up 738 MB: 113 us at the copy rate), 8 experts run the tensor cores at
// the clock that the power cap leaves (518 clocks per k-block of 512).  Measured, us, tokens as M side / as N side, in the order
// gate | up, down, SwiGLU gradient, input gradient: 64 experts of 2048 x 1408 over 10 662 rows 166, 90, 141, 156 / 160, 90, 118, 149;
// whole layers, forward and backward: 64 experts over 598 tokens 860 / 769, over 1457 1200 / 1071; 8 experts of 2048 x 7168 over 2048
// tokens, where some experts have more than 512 rows, 1270 / 1216, over 1484 1429 / 1362.
//
// kind 1, SwiGLU: gate (maps_b) and up weights (maps_b2), 128 hidden units per tile: a CTA's accumulator lanes hold 64 gate and the 64
// matching up units; h = silu(gate) * up and optionally the pre-activations are written.
// kind 2: SwiGLU backward in the epilogue of the down projection's input-gradient product (see the launcher).
// kind 3: C = A_1 B_e + A_2 B2_e with A = [A_1 | A_2] side by side (the input gradient of the gate and up projections as
// one product over K = 2 F): no second pass over C, and the sum is rounded once.
//
// NE > 1: every expert's weight has a tensor map of its own (up to NE of them, kernel parameters), so the weights of
// separate Linear modules are read where they are; NE == 1: one packed (E, .., ..) tensor.  For 8 experts of 2048 x 7168
// the copies this saves move 1.4 GB per forward pass.
//
// Synchronisation as in gemm_tcgen05_2cta.cu (all waits bounded); TMA loads carry no cluster multicast.
// Replaces the padded torch._grouped_mm calls of the reference (kempnerforge/model/moe.py:20-145).
#include "pair_common.cuh"
#include "tile_math.h"
#include "tokens_epilogue.cuh"

namespace kf {
namespace grp2 {

using namespace kf::pairops;
using kf2::tokens::Output;
using kf2::tokens::WARP_BYTES;
using tilemath::TokenTiles;

constexpr int CTA_M = 128, TILE_M = 256, MAX_N = 256, BK = 64, STAGES = 6, UMMA_K = 16;
constexpr int A_BYTES = CTA_M * BK * 2, B_BYTES = MAX_N / 2 * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int THREADS = 192, TMEM_COLS = 512;
constexpr int MAX_EXPERTS = 256;
constexpr int BAR_BYTES = 192;
constexpr size_t SMEM = size_t(STAGES) * STAGE_BYTES + 4 * WARP_BYTES + 1024 + BAR_BYTES + (MAX_EXPERTS + 1) * 4;

template <int NE>
struct Maps {
  CUtensorMap m[NE];
};
constexpr int MAX_SEPARATE = 32;  // experts with a tensor map of their own (two operands: 8 KB of kernel parameters)

// map_a.m[i]: boxes of 16 (i + 1) token rows, what a CTA of the pair loads of a tile of 32 (i + 1).
template <bool B_MN, int KIND, int NE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
kf_grouped_gemm_tcgen05_2cta(const __grid_constant__ Maps<8> map_a, const __grid_constant__ Maps<NE> maps_b,
                             const __grid_constant__ Maps<(KIND & 1) ? NE : 1> maps_b2, const __grid_constant__ Output out,
                             const int* __restrict__ row_offsets, int E, int N, int K, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t box_smem = smem_base + STAGES * STAGE_BYTES;
  const uint32_t bar_base = box_smem + 4 * WARP_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 5);
  uint8_t* bar_gen = smem_raw + (bar_base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(bar_gen + 8 * (2 * STAGES + 5));
  volatile int* widest_ptr = reinterpret_cast<volatile int*>(bar_gen + 8 * (2 * STAGES + 6));
  static_assert(8 * (2 * STAGES + 7) <= BAR_BYTES, "barriers, tensor-memory address, widest tile and number of tiles");
  int* offsets = reinterpret_cast<int*>(bar_gen + BAR_BYTES);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  constexpr bool SWIGLU = KIND == 1;
  constexpr int TILE_F = SWIGLU ? TILE_M / 2 : TILE_M, CTA_F = TILE_F / 2;  // features (hidden units) per tile and per CTA
  const int f_blocks = (N + TILE_F - 1) / TILE_F;
  const int k_blocks = (K + BK - 1) / BK;

  for (int i = threadIdx.x; i <= E; i += THREADS) offsets[i] = row_offsets[i];
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
    if (NE == 1) {
      tma_prefetch_desc(&maps_b.m[0]);
      if (KIND & 1) tma_prefetch_desc(&maps_b2.m[0]);
    }
  }
  __syncthreads();  // the offsets are in place
  if (warp == 0) {  // widest token tile: the same choice in every CTA
    int best = MAX_N, total = 0;
    float best_cost = 3.4e38f;
    for (int widest = MAX_N; widest >= tilemath::NARROWEST_TOKENS; widest -= 32) {
      int tiles = 0, clocks = 0;
      for (int e = lane; e < E; e += 32) {
        const int rows = offsets[e + 1] - offsets[e], n = tilemath::ceil_div(rows, widest);
        tiles += n;
        clocks += n * tilemath::token_tile_cost(tilemath::token_tile_width(rows, n));
      }
      tiles = __reduce_add_sync(0xffffffffu, tiles);
      clocks = __reduce_add_sync(0xffffffffu, clocks);
      const float cost = tilemath::token_rounds_cost(tiles, clocks, f_blocks, num_pairs);
      if (cost < best_cost) {
        best_cost = cost;
        best = widest;
        total = tiles * f_blocks;
      }
    }
    if (lane == 0) {
      widest_ptr[0] = best;
      widest_ptr[1] = total;
    }
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
  const int widest = widest_ptr[0], num_tiles = widest_ptr[1];

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) {
      int it = 0;
      bool ok = true;
      TokenTiles walk(offsets, f_blocks, widest);
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const auto tl = walk.at(t);
        const int half = tl.width >> 1;
        const int n0 = tl.row0 + int(rank) * half, f0 = tl.fb * TILE_F + int(rank) * CTA_F;
        const CUtensorMap* my_a = &map_a.m[(tl.width >> 5) - 1];
        const int me = NE > 1 ? tl.e : 0;              // tensor map and first row of the expert's weight inside it
        const int e_n = NE > 1 ? 0 : tl.e * N, e_k = NE > 1 ? 0 : tl.e * (KIND == 3 ? K / 2 : K);
        const CUtensorMap* my_b = &maps_b.m[me];
        const uint32_t bytes = 2u * (A_BYTES + half * BK * 2);
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t w_dst = smem_base + s * STAGE_BYTES;
          const uint32_t lead_full = full_bar(s) & PEER_BIT_MASK;
          if (leader) mbar_expect_tx(full_bar(s), bytes);
          const int k0 = kb * BK;
          tma_load_2d_pair(w_dst + A_BYTES, my_a, lead_full, k0, n0);
          int kw = k0;                                 // reduction index inside the weight
          if (KIND == 3 && k0 >= K / 2) {
            my_b = &maps_b2.m[me];
            kw = k0 - K / 2;
          }
          if constexpr (B_MN) {  // two boxes of 64 features; SwiGLU: 64 gate units, the 64 matching up units
            tma_load_2d_pair(w_dst, my_b, lead_full, f0, e_k + kw);
            if constexpr (SWIGLU) tma_load_2d_pair(w_dst + A_BYTES / 2, &maps_b2.m[me], lead_full, f0, e_k + kw);
            else tma_load_2d_pair(w_dst + A_BYTES / 2, my_b, lead_full, f0 + 64, e_k + kw);
          } else if constexpr (SWIGLU) {
            tma_load_2d_pair(w_dst, my_b, lead_full, kw, e_n + f0);
            tma_load_2d_pair(w_dst + A_BYTES / 2, &maps_b2.m[me], lead_full, kw, e_n + f0);
          } else {
            tma_load_2d_pair(w_dst, my_b, lead_full, kw, e_n + f0);
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
      int it = 0, tile_iter = 0;
      bool ok = true;
      TokenTiles walk(offsets, f_blocks, widest);
      for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
        const uint32_t idesc = umma_idesc_bf16(TILE_M, walk.at(t).width, B_MN, false);
        const int acc = tile_iter & 1;
        if (!mbar_wait(tempty_bar(acc), ((tile_iter >> 1) & 1) ^ 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * MAX_N;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(full_bar(s), (it / STAGES) & 1, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t w_src = smem_base + s * STAGE_BYTES, a_src = w_src + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t wd = B_MN ? umma_desc_sw128(w_src + k * (UMMA_K * 128), 64 * BK * 2, 1024)
                                     : umma_desc_sw128(w_src + k * (UMMA_K * 2), 16, 1024);
            mma_pair_f16(d_tmem, wd, umma_desc_sw128(a_src + k * (UMMA_K * 2), 16, 1024), idesc, (kb | k) != 0);
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
    TokenTiles walk(offsets, f_blocks, widest);
    for (int t = pair; t < num_tiles; t += num_pairs, ++tile_iter) {
      const auto tl = walk.at(t);
      const int acc = tile_iter & 1;
      const bool ok = kf2::tokens::tile_epilogue<KIND == 1 ? 1 : KIND == 2 ? 3 : 0>(
          out, box_smem, quarter, lane, tl.fb * TILE_F + int(rank) * CTA_F, tl.row0, tl.valid,
          tmem_base + (uint32_t(quarter * 32) << 16) + acc * MAX_N,
          [&] { return mbar_wait(tfull_bar(acc), (tile_iter >> 1) & 1, status, KF_ERR_WAIT_TMEM_FULL); });
      if (!ok) break;
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

template <bool B_MN, int KIND, int NE>
static int launch(const Maps<8>& ma, const Maps<NE>& mb, const Maps<(KIND & 1) ? NE : 1>& mb2, const Output& out,
                  const void* offsets, int E, int N, int K, int pairs, cudaStream_t st, int* status) {
  auto kern = kf_grouped_gemm_tcgen05_2cta<B_MN, KIND, NE>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_set = true;
  }
  kern<<<pairs * 2, THREADS, SMEM, st>>>(ma, mb, mb2, out, reinterpret_cast<const int*>(offsets), E, N, K, status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

// Weight operand: the packed tensor (NE == 1, *w) or one pointer per expert.  Each expert's matrix is [N][K] (K
// contiguous, boxes of `box` rows) or, b_mn, [K][N] (N contiguous, 64 x 64 boxes).
template <int NE>
static int make_weight_maps(Maps<NE>& m, const void* const* w, int E, int N, int K, int b_mn, int box) {
  for (int e = 0; e < (NE > 1 ? E : 1); ++e) {
    const uint64_t n = NE > 1 ? 1 : E;
    const int rc = b_mn ? make_map_2d_bf16(&m.m[e], w[e], n * K, N, N, 64, BK) : make_map_2d_bf16(&m.m[e], w[e], n * N, K, K, BK, box);
    if (rc) return rc;
  }
  return 0;
}

template <int KIND, int NE>
static int run(const void* A, const void* const* W, const void* const* W2, void* C, void* GU, const void* offsets, int rows,
               int E, int N, int K, int KW, long long lda, long long ldc, long long ldgu, int b_mn, int accumulate, int num_sms,
               cudaStream_t st, int* status) {
  if (ldc > 0x7fffffffll || ldgu > 0x7fffffffll) return 6;
  Maps<8> ma;
  Maps<NE> mb;
  Maps<(KIND & 1) ? NE : 1> mb2;
  int rc = 0;
  for (int i = 0; i < 8 && !rc; ++i) rc = make_map_2d_bf16(&ma.m[i], A, rows, K, lda, BK, 16 * (i + 1));
  if (rc) return 100 + rc;
  rc = make_weight_maps<NE>(mb, W, E, N, KW, b_mn, KIND == 1 ? CTA_M / 2 : CTA_M);
  if (!rc && (KIND & 1)) rc = make_weight_maps<(KIND & 1) ? NE : 1>(mb2, W2, E, N, KW, b_mn, KIND == 1 ? CTA_M / 2 : CTA_M);
  if (rc) return 200 + rc;
  if (!(KIND & 1)) mb2.m[0] = mb.m[0];
  Output out{};
  out.out = reinterpret_cast<__nv_bfloat16*>(C);
  out.aux = reinterpret_cast<const __nv_bfloat16*>(KIND == 1 || KIND == 2 ? GU : accumulate ? C : nullptr);
  out.F = N;
  out.ldo = (int)ldc;
  out.lda = (int)(KIND == 1 || KIND == 2 ? ldgu : ldc);
  const int tile_f = KIND == 1 ? TILE_M / 2 : TILE_M;
  // at most so many tiles: the narrowest, one partial tile per expert
  const long long upper = ((long long)(rows / tilemath::NARROWEST_TOKENS) + E) * ((N + tile_f - 1) / tile_f);
  const int pairs = upper < num_sms / 2 ? (int)upper : num_sms / 2;
  return b_mn ? launch<true, KIND, NE>(ma, mb, mb2, out, offsets, E, N, K, pairs, st, status)
              : launch<false, KIND, NE>(ma, mb, mb2, out, offsets, E, N, K, pairs, st, status);
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
