// bf16 GEMM with CTA pairs whose tile is cut to the number of tokens:  out[T, F] = x[T, K] * W^T.
//
// What bounds a product over a ragged number of rows is the rounds of tiles: the pair kernel of gemm_tcgen05_2cta.cu has the
// rows of x as the M side of the MMA, which is 256 whatever T is, so 1554 rows are seven row tiles of which the last holds
// 18.  Here the roles are exchanged: 256 rows of W (output features) are the M side, and the tokens are its N side, whose width is
// a multiple of 32 up to 256, chosen per launch: 1554 tokens are 7 tiles of 224 or 9 of 192.  Which of the two kernels runs,
// and at which width, is decided by rounds x (512 + width), see tokens_width.  The sums over K have the same order, and so the
// same bits, either way.
// What bounds a narrow tile is the shared-memory port, through which its MMAs read the 256 rows of W whatever the width: a k-block
// takes 210 ns at 96 tokens, 245 at 128, 285 at 160, 330 at 192, 390 at 224 and 430 at 256, where the products are the longer part (a
// ring of eight stages instead of six, which the width leaves room for, gives 1 %).  Against 256 x 256 tiles, both with lane 0 issuing
// the products, a block of a 7B model over 1554 tokens, us: o 56 -> 50, gate and up 280 -> 268, down 163 -> 151, q | k | v
// 74 -> 73; over 300 tokens o 35 -> 26, down 95 -> 74.  With an elected thread the block over 1554 tokens takes another tenth less.
//
// The epilogue, which turns the accumulators back into rows of tokens, is in tokens_epilogue.cuh.
//
// EPI 0: (+ residual); 1: SwiGLU over W = [gate ; up]; 2: rotary embedding of the first columns of q | k | v; 3: SwiGLU gradient.
// W_MN: W is stored [K][F] (a weight read for an input gradient), else [F][K]; up to three matrices stacked along F, or along K.
// Warps, rings, barriers and bounded waits are those of gemm_tcgen05_2cta.cu.
#include "pair_common.cuh"
#include "tile_math.h"
#include "tokens_epilogue.cuh"

namespace kf2 {
namespace tokens {

using namespace kf;
using namespace kf::pairops;

constexpr int CTA_M = 128, TILE_M = 256, MAX_N = 256;
constexpr int BK = 64, UMMA_K = 16, MAX_STAGES = 9;
constexpr int A_BYTES = CTA_M * BK * 2, RING_BYTES = 192 * 1024;  // the ring holds as many stages as the width leaves room for
constexpr int THREADS = 192, TMEM_COLS = 512;
constexpr int GROUP = 8;             // token tiles that share one sweep over the feature tiles
constexpr size_t SMEM_BYTES = size_t(RING_BYTES) + 4 * WARP_BYTES + 1024 + 256;

struct Weights {
  CUtensorMap map[3];
  int start[3];  // first stacked row (W_MN: first k) of each matrix; INT_MAX when absent
};

struct Args : Output {
  int K;
};

struct Tile {
  int fb, tok0, tokens;  // block of features, first token and how many
};

template <bool W_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
kf_gemm_tokens_2cta(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ Weights ws, const __grid_constant__ Args a,
                    int tile_n, int stages, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t box_smem = smem_base + RING_BYTES;
  const int half_n = tile_n >> 1, stage_bytes = A_BYTES + half_n * BK * 2;  // tokens each CTA of the pair contributes
  const uint32_t bar_base = box_smem + 4 * WARP_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
  auto tfull_bar = [&](int i) { return bar_base + 8u * (2 * MAX_STAGES + i); };
  auto tempty_bar = [&](int i) { return bar_base + 8u * (2 * MAX_STAGES + 2 + i); };
  const uint32_t drain_bar = bar_base + 8u * (2 * MAX_STAGES + 4);
  const uint32_t tmem_slot = bar_base + 8u * (2 * MAX_STAGES + 5);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  constexpr int TILE_F = EPI == 1 ? TILE_M / 2 : TILE_M, CTA_F = TILE_F / 2;  // features (hidden units) per tile and per CTA
  const int f_blocks = (a.F + TILE_F - 1) / TILE_F, k_blocks = (a.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tfull_bar(i), 1);
      mbar_init(tempty_bar(i), 8);
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&ws.map[0]);
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
  const int t_blocks = (a.T + tile_n - 1) / tile_n, num_tiles = f_blocks * t_blocks;
  auto tile_at = [&](int t) {
    Tile x;
    int tb;
    tilemath::raster(t, t_blocks, f_blocks, GROUP, tb, x.fb);
    x.tok0 = tb * tile_n;
    x.tokens = min(tile_n, a.T - x.tok0);
    return x;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) {
      int s = 0, fills = 0;  // stage, and how many were filled altogether
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const Tile tl = tile_at(t);
        const int n0 = tl.tok0 + int(rank) * half_n, f0 = tl.fb * TILE_F + int(rank) * CTA_F;
        const int sg = W_MN || EPI == 1 ? 0 : int(f0 >= ws.start[1]) + int(f0 >= ws.start[2]);
        const int r0 = f0 - (W_MN ? 0 : ws.start[sg]);
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(empty_bar(s), phase ^ 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t a_dst = smem_base + s * stage_bytes, b_dst = a_dst + A_BYTES;
          const uint32_t lead_full = full_bar(s) & PEER_BIT_MASK;
          if (leader) mbar_expect_tx(full_bar(s), 2 * stage_bytes);
          const int k0 = kb * BK;
          tma_load_2d_pair(b_dst, &map_x, lead_full, k0, n0);
          if constexpr (W_MN) {
            const int ks = int(k0 >= ws.start[1]) + int(k0 >= ws.start[2]);
#pragma unroll
            for (int c = 0; c < CTA_M / 64; ++c)
              tma_load_2d_pair(a_dst + c * (64 * BK * 2), &ws.map[ks], lead_full, f0 + 64 * c, k0 - ws.start[ks]);
          } else if constexpr (EPI == 1) {
            tma_load_2d_pair(a_dst, &ws.map[0], lead_full, k0, f0);  // 64 gate rows, the 64 matching up rows
            tma_load_2d_pair(a_dst + A_BYTES / 2, &ws.map[1], lead_full, k0, f0);
          } else {
            tma_load_2d_pair(a_dst, &ws.map[sg], lead_full, k0, r0);
          }
          ++fills;
          if (++s == stages) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      // see gemm_tcgen05_2cta.cu: copies into this CTA are complete once their stages were consumed or the leader's barrier flipped
      if (leader)
        for (int j = max(0, fills - stages); j < fills; ++j)
          mbar_wait(full_bar(j % stages), (j / stages) & 1, status, KF_ERR_WAIT_DRAIN);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      int s = 0, tile_iter = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t idesc = umma_idesc_bf16(TILE_M, tile_n, W_MN, false);
      for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
        const int acc = tile_iter & 1;
        if (!mbar_wait(tempty_bar(acc), ((tile_iter >> 1) & 1) ^ 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * MAX_N;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(full_bar(s), phase, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_src = smem_base + s * stage_bytes, b_src = a_src + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t ad = W_MN ? umma_desc_sw128(a_src + k * (UMMA_K * 128), 64 * BK * 2, 1024)
                                     : umma_desc_sw128(a_src + k * (UMMA_K * 2), 16, 1024);
            mma_pair_f16(d_tmem, ad, umma_desc_sw128(b_src + k * (UMMA_K * 2), 16, 1024), idesc, (kb | k) != 0);
          }
          commit_pair(empty_bar(s));
          if (++s == stages) {
            s = 0;
            phase ^= 1;
          }
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
    for (int t = pair; t < num_tiles; t += num_pairs, ++tile_iter) {
      const Tile tl = tile_at(t);
      const int acc = tile_iter & 1;
      const bool ok = tile_epilogue<EPI>(
          a, box_smem, quarter, lane, tl.fb * TILE_F + int(rank) * CTA_F, tl.tok0, tl.tokens,
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
  cluster_sync_all();  // the peer's shared memory / tensor memory stay valid until both CTAs are done
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// rows[i]: rows of matrix i of the stack ([F][K], or W_MN [K][F]).
template <bool W_MN, int EPI>
static int launch(const void* x, int ldx, const void* const* w, const int* rows, int n_seg, int ldw, const Args& a, int tile_n,
                  int num_sms, int* status, cudaStream_t stream) {
  CUtensorMap mx;
  Weights ws;
  int rc = make_map_2d_bf16(&mx, x, a.T, a.K, ldx, BK, tile_n / 2);
  if (rc) return 100 + rc;
  int at = 0;
  for (int i = 0; i < n_seg; ++i) {
    if (at % (W_MN ? BK : EPI == 1 ? 8 : CTA_M)) return 6;
    rc = W_MN ? make_map_2d_bf16(&ws.map[i], w[i], rows[i], a.F, ldw, 64, BK)
              : make_map_2d_bf16(&ws.map[i], w[i], rows[i], a.K, ldw, BK, EPI == 1 ? CTA_M / 2 : CTA_M);
    if (rc) return 200 + rc;
    ws.start[i] = at;
    at += rows[i];
  }
  for (int i = n_seg; i < 3; ++i) {
    ws.map[i] = ws.map[0];
    ws.start[i] = 0x7fffffff;
  }
  auto kern = kf_gemm_tokens_2cta<W_MN, EPI>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_set = true;
  }
  constexpr int TILE_F = EPI == 1 ? TILE_M / 2 : TILE_M;
  const int tiles = ((a.F + TILE_F - 1) / TILE_F) * ((a.T + tile_n - 1) / tile_n);
  const int pairs = tiles < num_sms / 2 ? tiles : num_sms / 2, stages = min(MAX_STAGES, RING_BYTES / (A_BYTES + tile_n / 2 * BK * 2));
  kern<<<pairs * 2, THREADS, SMEM_BYTES, stream>>>(mx, ws, a, tile_n, stages, status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace tokens

// Width (tokens) of the launch for T tokens and m_rows rows of W (gate and up counted both), its rounds of tiles and its cost:
// rounds x (512 + width).  A narrow tile saves products, not the fetch of its 256 rows of W: over 64 k-blocks a round takes 23.5 us
// at 256 tokens, 23.1 at 224 and 21.7 at 160 (14336 units over 777 tokens), and widths below 128 gain nothing more.
int tokens_width(int T, int m_rows, int num_sms, float* cost, int* rounds) {
  const int pairs = num_sms / 2, m_blocks = (m_rows + tokens::TILE_M - 1) / tokens::TILE_M;
  int best = 256;
  float best_cost = 3.4e38f;
  for (int n = 256; n >= 128; n -= 32) {
    const long long r = ((long long)m_blocks * ((T + n - 1) / n) + pairs - 1) / pairs;
    if (float(r) * float(512 + n) < best_cost) {
      best = n;
      best_cost = float(r) * float(512 + n);
      if (rounds) *rounds = int(r);
    }
  }
  if (cost) *cost = best_cost;
  return best;
}

// The launches; `tile_n` from tokens_width.
int launch_tokens_plain(const void* x, const void* const* w, const int* rows, int n_seg, int w_mn, void* out, const void* residual, int T,
                        int F, int K, int ldx, int ldw, int ldo, int ldr, int tile_n, int num_sms, cudaStream_t stream, int* status) {
  tokens::Args a{{(__nv_bfloat16*)out, (const __nv_bfloat16*)residual, T, F, ldo, ldr, nullptr, nullptr, 1, 0, 128}, K};
  return w_mn ? tokens::launch<true, 0>(x, ldx, w, rows, n_seg, ldw, a, tile_n, num_sms, status, stream)
              : tokens::launch<false, 0>(x, ldx, w, rows, n_seg, ldw, a, tile_n, num_sms, status, stream);
}
int launch_tokens_swiglu(const void* x, const void* wg, const void* wu, void* h, const void* gu, int T, int F, int K, int ldx, int ldw,
                         int ldh, int ldgu, int tile_n, int num_sms, cudaStream_t stream, int* status) {
  const void* w[3] = {wg, wu, nullptr};
  const int rows[3] = {F, F, 0};
  tokens::Args a{{(__nv_bfloat16*)h, (const __nv_bfloat16*)gu, T, F, ldh, ldgu, nullptr, nullptr, 1, 0, 128}, K};
  return tokens::launch<false, 1>(x, ldx, w, rows, 2, ldw, a, tile_n, num_sms, status, stream);
}
int launch_tokens_rope(const void* x, const void* const* w, const int* rows, int n_seg, void* out, int T, int F, int K, int ldx, int ldw,
                       int ldo, const float* cosT, const float* sinT, int S, int rope_cols, int hd, int tile_n, int num_sms,
                       cudaStream_t stream, int* status) {
  tokens::Args a{{(__nv_bfloat16*)out, nullptr, T, F, ldo, 0, cosT, sinT, S, rope_cols, hd}, K};
  return tokens::launch<false, 2>(x, ldx, w, rows, n_seg, ldw, a, tile_n, num_sms, status, stream);
}
int launch_tokens_swiglu_bwd(const void* dy, const void* w, const void* gu, void* dgu, int T, int F, int K, int ldy, int ldw, int ldgu,
                             int tile_n, int num_sms, cudaStream_t stream, int* status) {
  const void* ws[3] = {w, nullptr, nullptr};
  const int rows[3] = {K, 0, 0};
  tokens::Args a{{(__nv_bfloat16*)dgu, (const __nv_bfloat16*)gu, T, F, ldgu, ldgu, nullptr, nullptr, 1, 0, 128}, K};
  return tokens::launch<true, 3>(dy, ldy, ws, rows, 1, ldw, a, tile_n, num_sms, status, stream);
}

}  // namespace kf2
