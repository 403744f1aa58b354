// bf16 GEMM with CTA pairs whose tile is cut to the number of tokens:  out[T, F] = x[T, K] * W^T.
//
// What bounds a product over a ragged number of rows is the rounds of tiles: the pair kernel of gemm_tcgen05_2cta.cu has the
// rows of x as the M side of the MMA, which is 256 whatever T is, so 1554 rows are seven row tiles of which the last holds
// 18.  Here the roles are exchanged: 256 rows of W (output features) are the M side, and the tokens are its N side, whose width is
// a multiple of 32 up to 256, chosen per launch: 1554 tokens are 7 tiles of 224 or 9 of 192.  Which of the two kernels runs,
// and at which width, is decided by rounds x (512 + width), see tokens_width.  The sums over K have the same order, and so the
// same bits, either way.
// What bounds a narrow tile is not the products but the fetch of its 256 rows of W (a ring of eight stages instead of six, which
// the width leaves room for, gives 1 %).  A block of a 7B model over 1554 tokens, us: o 56 -> 50, gate and up 280 -> 268, down
// 163 -> 151, q | k | v 74 -> 73; over 300 tokens o 35 -> 26, down 95 -> 74.
//
// The accumulator holds a feature per lane and a token per column.  The epilogue turns 32 x 32 blocks through shared memory
// (fp32, XOR-swizzled 16-byte chunks: no bank conflicts), after which a lane holds 32 features of one token, as in the other
// kernel.  Where two features are combined (gate and up of a hidden unit, the two halves of a rotary pair) the blocks of the two
// warps that hold them are read by both, half the features each (boxes of 16 rows that bring both into one warp were tried: nine
// copies per k-block instead of three are slower than the products).
//
// EPI 0: (+ residual); 1: SwiGLU over W = [gate ; up]; 2: rotary embedding of the first columns of q | k | v; 3: SwiGLU gradient.
// W_MN: W is stored [K][F] (a weight read for an input gradient), else [F][K]; up to three matrices stacked along F, or along K.
// Warps, rings, barriers and bounded waits are those of gemm_tcgen05_2cta.cu.
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tile_math.h"
#include "pair_common.cuh"

namespace kf2 {
namespace tokens {

using namespace kf;
using namespace kf::pairops;

constexpr int CTA_M = 128, TILE_M = 256, MAX_N = 256;
constexpr int BK = 64, UMMA_K = 16, MAX_STAGES = 9;
constexpr int A_BYTES = CTA_M * BK * 2, RING_BYTES = 192 * 1024;  // the ring holds as many stages as the width leaves room for
constexpr int THREADS = 192, TMEM_COLS = 512;
constexpr int GROUP = 8;             // token tiles that share one sweep over the feature tiles
constexpr int TURN_BYTES = 4096;     // a warp's 32 x 32 fp32 block on its way from features to tokens
constexpr int BOX_BYTES = 2048;      // a warp's 32 x 32 bf16 block on its way to or from global memory
constexpr size_t SMEM_BYTES = size_t(RING_BYTES) + 4 * (TURN_BYTES + 2 * BOX_BYTES) + 1024 + 256;

struct Weights {
  CUtensorMap map[3];
  int start[3];  // first stacked row (W_MN: first k) of each matrix; INT_MAX when absent
};

struct Args {
  __nv_bfloat16* out;        // [T][ldo]
  const __nv_bfloat16* aux;  // residual [T][lda] (0), pre-activations to write (1, or null) or to read (3) [T][lda] = gate | up
  int T, F, K, ldo, lda;     // F: output features (1 and 3: hidden units)
  const float *cosT, *sinT;  // [S][hd / 2]
  int S, rope_cols, hd;
};

struct Tile {
  int fb, tok0, tokens;  // block of features, first token and how many
};

// 16 columns of 32 rows: 32 contiguous bytes per row, two lanes each.
__device__ __forceinline__ void store_rows16(uint32_t box, int lane, const uint4& lo, const uint4& hi, __nv_bfloat16* dst, size_t ld,
                                             int rows) {
  auto at = [&](int row, int q) { return box + uint32_t(row * 32 + ((q ^ ((row >> 2) & 1)) << 4)); };
  __syncwarp();
  sts128(at(lane, 0), lo);
  sts128(at(lane, 1), hi);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = i * 16 + (lane >> 1), ch = lane & 1;
    if (row < rows) *reinterpret_cast<uint4*>(dst + row * ld + ch * 8) = lds128(at(row, ch));
  }
}
__device__ __forceinline__ void meet(int bar) { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool meet_all(int bar, bool ok) {
  int all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, 64, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
               : "=r"(all)
               : "r"(int(ok)), "r"(bar)
               : "memory");
  return all != 0;
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

template <bool W_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
kf_gemm_tokens_2cta(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ Weights ws, const __grid_constant__ Args a,
                    int tile_n, int stages, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t box_smem = smem_base + RING_BYTES;
  const int half_n = tile_n >> 1, stage_bytes = A_BYTES + half_n * BK * 2;  // tokens each CTA of the pair contributes
  const uint32_t bar_base = box_smem + 4 * (TURN_BYTES + 2 * BOX_BYTES);
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
    const uint32_t turn = box_smem + uint32_t(quarter) * (TURN_BYTES + 2 * BOX_BYTES), box = turn + TURN_BYTES, box2 = box + BOX_BYTES;
    // 1, 2: two warps meet, one with the first halves (gate, or the dimensions below hd / 2) and one with the second; each takes
    // 16 features of either.  Halves of 64 rows are two warps apart, those of a head of 64 one.
    constexpr bool MEET = EPI == 1 || EPI == 2;
    const int apart = EPI == 2 && a.hd == 64 ? 1 : 2, first = quarter & ~apart, share = quarter & apart ? 1 : 0;
    const int meet_bar = 1 + (apart == 1 ? quarter >> 1 : quarter & 1);
    const uint32_t turn1 = box_smem + uint32_t(first) * (TURN_BYTES + 2 * BOX_BYTES),
                   turn2 = turn1 + uint32_t(apart) * (TURN_BYTES + 2 * BOX_BYTES);
    int tile_iter = 0;
    for (int t = pair; t < num_tiles; t += num_pairs, ++tile_iter) {
      const Tile tl = tile_at(t);
      const int acc = tile_iter & 1;
      const int tok0 = tl.tok0, tokens = tl.tokens;
      const int f0 = tl.fb * TILE_F + int(rank) * CTA_F;  // this CTA's first feature
      const int lo = first * 32 + share * 16;  // 1, 2: first of its 16 hidden units or dimensions
      // this warp's first feature and how many of its 32 (1: 16 hidden units, 2: 16 pairs) exist
      const int fw = f0 + (MEET ? lo : quarter * 32);
      const int cols = max(0, min(MEET ? 16 : 32, a.F - fw));
      const __nv_bfloat16* aux = EPI != 2 && a.aux ? a.aux + size_t(tok0) * a.lda + fw : nullptr;
      Rows32 g_next, u_next;
      if (EPI == 3 || (EPI == 0 && aux)) {  // travels while the tile's products are still running
        g_next = load_rows32(aux, a.lda, lane, tokens, cols);
        if (EPI == 3) u_next = load_rows32(aux + a.F, a.lda, lane, tokens, cols);
      }
      bool ok = mbar_wait(tfull_bar(acc), (tile_iter >> 1) & 1, status, KF_ERR_WAIT_TMEM_FULL);
      if (MEET) ok = meet_all(meet_bar, ok);  // both warps go on, or neither
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * MAX_N;
#pragma unroll 1
      for (int c = 0; c * 32 < tokens; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(t_row + c * 32, v);
        const int left = tokens - c * 32;  // tokens from this block on
        const Rows32 g_now = g_next, u_now = u_next;
        if ((EPI == 3 || (EPI == 0 && aux)) && left > 32) {
          g_next = load_rows32(aux + size_t(c + 1) * 32 * a.lda, a.lda, lane, left - 32, cols);
          if (EPI == 3) u_next = load_rows32(aux + a.F + size_t(c + 1) * 32 * a.lda, a.lda, lane, left - 32, cols);
        }
        tmem_ld_wait();
        // the previous block has been read
        if (MEET) meet(meet_bar);
        else __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(turn + uint32_t(i * 128 + (((lane >> 2) ^ (i & 7)) << 4) + (lane & 3) * 4)), "r"(v[i])
                       : "memory");
        if (MEET) meet(meet_bar);
        else __syncwarp();
        float f[32];  // features of token tok0 + c * 32 + lane
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int ch = MEET ? 4 * share + (q & 3) : q;
          const uint4 u = lds128((!MEET ? turn : q < 4 ? turn1 : turn2) + uint32_t(lane * 128 + ((ch ^ (lane & 7)) << 4)));
          f[4 * q] = __uint_as_float(u.x);
          f[4 * q + 1] = __uint_as_float(u.y);
          f[4 * q + 2] = __uint_as_float(u.z);
          f[4 * q + 3] = __uint_as_float(u.w);
        }
        __nv_bfloat16* out = a.out + size_t(tok0 + c * 32) * a.ldo + fw;
        if constexpr (EPI == 0) {
          if (aux) {
            const Rows32 r = to_own_row(box2, lane, g_now);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t w[4] = {r.q[q].x, r.q[q].y, r.q[q].z, r.q[q].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 p = unpack_bf16(w[e]);
                f[q * 8 + 2 * e] += p.x;
                f[q * 8 + 2 * e + 1] += p.y;
              }
            }
          }
          Rows32 o;
#pragma unroll
          for (int q = 0; q < 4; ++q) o.q[q] = pack8(f + q * 8);
          store_rows32(box, lane, o, out, a.ldo, left, cols);
        } else if constexpr (EPI == 1) {
          if (a.aux && cols > 0) {
            __nv_bfloat16* gu = const_cast<__nv_bfloat16*>(aux) + size_t(c) * 32 * a.lda;
            store_rows16(box, lane, pack8(f), pack8(f + 8), gu, a.lda, left);
            store_rows16(box2, lane, pack8(f + 16), pack8(f + 24), gu + a.F, a.lda, left);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) {  // the activation sees bf16 pre-activations, as in swiglu_chunk
            const float g = __bfloat162float(__float2bfloat16(f[i])), u = __bfloat162float(__float2bfloat16(f[16 + i]));
            f[i] = g / (1.f + __expf(-g)) * u;
          }
          if (cols > 0) store_rows16(box, lane, pack8(f), pack8(f + 8), out, a.ldo, left);
        } else if constexpr (EPI == 2) {
          const int half = a.hd >> 1;
          if (fw < a.rope_cols) {
            const int pos = min(tok0 + c * 32 + lane, a.T - 1) % a.S, m = lo & (half - 1);
            const float *cr = a.cosT + size_t(pos) * half + m, *sr = a.sinT + size_t(pos) * half + m;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 cs = *reinterpret_cast<const float4*>(cr + q * 4), sn = *reinterpret_cast<const float4*>(sr + q * 4);
              const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float x = f[q * 4 + i], y = f[16 + q * 4 + i];
                f[q * 4 + i] = x * cv[i] - y * sv[i];
                f[16 + q * 4 + i] = y * cv[i] + x * sv[i];
              }
            }
          }
          if (cols > 0) {
            store_rows16(box, lane, pack8(f), pack8(f + 8), out, a.ldo, left);
            store_rows16(box2, lane, pack8(f + 16), pack8(f + 24), out + half, a.ldo, left);
          }
        } else {
          uint32_t dh[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) dh[i] = __float_as_uint(f[i]);
          Rows32 g = to_own_row(box, lane, g_now), u = to_own_row(box2, lane, u_now);
          swiglu_bwd_row(dh, g, u);
          store_rows32(box, lane, g, out, a.ldo, left, cols);
          store_rows32(box2, lane, u, out + a.F, a.ldo, left, cols);
        }
      }
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
  tokens::Args a{(__nv_bfloat16*)out, (const __nv_bfloat16*)residual, T, F, K, ldo, ldr, nullptr, nullptr, 1, 0, 128};
  return w_mn ? tokens::launch<true, 0>(x, ldx, w, rows, n_seg, ldw, a, tile_n, num_sms, status, stream)
              : tokens::launch<false, 0>(x, ldx, w, rows, n_seg, ldw, a, tile_n, num_sms, status, stream);
}
int launch_tokens_swiglu(const void* x, const void* wg, const void* wu, void* h, const void* gu, int T, int F, int K, int ldx, int ldw,
                         int ldh, int ldgu, int tile_n, int num_sms, cudaStream_t stream, int* status) {
  const void* w[3] = {wg, wu, nullptr};
  const int rows[3] = {F, F, 0};
  tokens::Args a{(__nv_bfloat16*)h, (const __nv_bfloat16*)gu, T, F, K, ldh, ldgu, nullptr, nullptr, 1, 0, 128};
  return tokens::launch<false, 1>(x, ldx, w, rows, 2, ldw, a, tile_n, num_sms, status, stream);
}
int launch_tokens_rope(const void* x, const void* const* w, const int* rows, int n_seg, void* out, int T, int F, int K, int ldx, int ldw,
                       int ldo, const float* cosT, const float* sinT, int S, int rope_cols, int hd, int tile_n, int num_sms,
                       cudaStream_t stream, int* status) {
  tokens::Args a{(__nv_bfloat16*)out, nullptr, T, F, K, ldo, 0, cosT, sinT, S, rope_cols, hd};
  return tokens::launch<false, 2>(x, ldx, w, rows, n_seg, ldw, a, tile_n, num_sms, status, stream);
}
int launch_tokens_swiglu_bwd(const void* dy, const void* w, const void* gu, void* dgu, int T, int F, int K, int ldy, int ldw, int ldgu,
                             int tile_n, int num_sms, cudaStream_t stream, int* status) {
  const void* ws[3] = {w, nullptr, nullptr};
  const int rows[3] = {K, 0, 0};
  tokens::Args a{(__nv_bfloat16*)dgu, (const __nv_bfloat16*)gu, T, F, K, ldgu, ldgu, nullptr, nullptr, 1, 0, 128};
  return tokens::launch<true, 3>(dy, ldy, ws, rows, 1, ldw, a, tile_n, num_sms, status, stream);
}

}  // namespace kf2
