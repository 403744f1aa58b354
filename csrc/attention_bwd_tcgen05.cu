// Flash attention backward on the 5th-generation tensor cores (head dim 64 or 128; the sizes below are those of 128).
//
// One CTA owns a tile of 128 keys of one (batch, KV head) and walks over every query head of the group and
// every 64-row query tile that can see those keys.  All five GEMMs of the backward pass run on tcgen05 with
// the *transposed* score tile, so that each softmax thread owns one key row and the products that feed the
// dK / dV accumulators can be taken straight from tensor memory / shared memory without a transpose:
//
//   S^T  = K  Q_i^T                      (128 keys x 64 queries, smem x smem -> TMEM)
//   dP^T = V  dO_i^T                     (128 x 64)
//   P^T  = exp2(S^T * c - lse_i),  dS^T = P^T * (dP^T - D_i)                (softmax warps; two elements per instruction,
//                                       the factor `scale` of dS is applied to the finished dK and dQ instead:
//                                       1250 -> 1085 us at 2 x 4096 tokens, 32 heads)
//   dV  += P^T  dO_i                     (A from TMEM, 128 x 128 accumulator, lives in TMEM for the whole CTA)
//   dK  += dS^T Q_i                      (A from TMEM, 128 x 128 accumulator)
//   dQ_i^T = K^T dS                      (128 head-dim rows x 64 queries; added to an fp32 dQ by a bulk reduction)
//
//   warp 0     : TMA producer (K, V once; Q_i / dO_i ring of three stages)
//   warp 1     : MMA issuer
//   warps 2-5  : softmax of queries 0..31 of the tile (one thread per key row) and the final dK / dV store
//   warps 10-13: softmax of queries 32..63 (the same key rows): two warps per scheduler hide each other's
//                exp2 / conversion latencies, and 32 scores + 32 dP per thread leave registers for instruction-level
//                parallelism (with 64 + 64 per thread the P / dS arithmetic was latency bound: 2400 of the 4100
//                cycles of an iteration)
//   warps 6-9  : dQ reduction (TMEM -> shared-memory tile -> one cp.reduce.async.bulk.tensor add per tile;
//                or, as a fallback mode, red.global.add.f32 per element)
//
// What bounds an iteration is the shared-memory port (128 bytes per clock).  The MMAs read their operands through it (176 KB: a
// 128 x 64 tile of 16 k takes the 48 clocks of its 6 KB, not the 32 of its products), the copies of Q_i and dO_i write 32 KB, dS^T
// 16 KB, and the fp32 dQ tile crosses it twice: 2300 clocks of the 2500 that one takes.  Hence dS^T comes from tensor memory for dK,
// where it lies behind P^T of the same 32 queries in the columns of S^T that only their own warp has read; no warp has to wait for
// another before it writes there.  The two halves of the queries synchronise apart (128 threads), so a scheduler's two warps drift
// into different phases.  With the statistics fetched untouched (see fetch_stat), backward with its pre- and post-pass, us:
// 2 x 4096 tokens, 32 query and 8 key heads of 128: 831 -> 779; 3000, 40 heads: 386 -> 363; 4 x 2048, 12 heads of 64: 230 -> 197.
//
// Head dim 64 adds nothing up in memory: each key tile writes its dQ tiles to a part of its own, and the post-pass adds the parts in
// the order of the key tiles, so equal inputs give equal bits (the library's backward, which such models had before, repeats itself
// at their usual lengths).  It has half the products per score and the same softmax, so it is bound by the softmax warps.  Backward
// with its pre- and post-pass, 12 causal heads, us, parts / one accumulator that all tiles add to: 100 positions 16.4 / 17.3, 3 x 333
// 26 / 27, 1024 43 / 43, 2048 74 / 70, 2 x 1600 87 / 78.  (The library's backward for 100, 3 x 333 and 2048: 16, 19 and 40, before
// the copies around it.)
//
// D_i = rowsum(dO_i * O_i) comes from a small pre-pass; a post-pass converts the fp32 dQ to bf16.
// Replaces the backward of F.scaled_dot_product_attention (kempnerforge/model/attention.py:227-231) for the
// causal / document-masked training path, without expanding grouped KV heads.
#include "attention_common.cuh"
#include "doc_blocks.cuh"

namespace kf {
namespace attnb {

constexpr int BLK_K = 128;  // keys per CTA
constexpr int BLK_Q = 64;   // queries per iteration
constexpr int THREADS = 448;
constexpr int TMEM_COLS = 512;
// S^T buffers 0 / 1 (fp32, 64 columns each).  In place of the 32 columns of either half of the queries its warps leave bf16 pairs:
// columns 0 - 15 P^T and 16 - 31 dS^T of the first half, 32 - 47 P^T and 48 - 63 dS^T of the second.
constexpr int ST_COL = 0;
constexpr int DPT_COL = 128;  // dP^T (fp32, 64 cols)
constexpr int DQT_COL = 192;  // dQ^T (fp32, 64 cols)
constexpr int DV_COL = 256;   // dV accumulator (fp32, HD cols)
constexpr int DK_COL = 384;   // dK accumulator (fp32, HD cols)
constexpr int KV_BLOCK_BYTES = BLK_K * 128;     // 16 KB: [128 rows x 128 B], HD / 64 of them per K / V tile
constexpr int Q_BLOCK_BYTES = BLK_Q * 128;      // 8 KB: [64 rows x 128 B], HD / 64 of them per Q_i / dO_i tile
constexpr int DS_BYTES = BLK_K * BLK_Q * 2;     // 16 KB: [128 key rows x 128 B]
constexpr int STAGES = 3;  // Q_i / dO_i ring: a tile is loaded one whole iteration before its scores are issued
constexpr int AUX_BYTES = 2048;  // barriers, row statistics, doc ids

template <int HD>
struct Cfg {
  static constexpr int BLOCKS = HD / 64;
  static constexpr int KV_TILE_BYTES = BLOCKS * KV_BLOCK_BYTES;
  static constexpr int Q_TILE_BYTES = BLOCKS * Q_BLOCK_BYTES;
  static constexpr size_t SMEM =
      2 * size_t(KV_TILE_BYTES) + STAGES * 2 * size_t(Q_TILE_BYTES) + 2 * DS_BYTES + 1024 /*align*/ + AUX_BYTES;
  static constexpr int DQ_STAGE_BYTES = BLK_Q * HD * 4;  // one dQ tile [64 queries][HD] fp32 for the bulk reduction
  static constexpr size_t SMEM_DQ_TMA = SMEM + DQ_STAGE_BYTES;
};

using attn::fadd2;
using attn::fast_exp2;
using attn::ffma2;
using attn::fmul2;
using attn::pack2;
using attn::tmem_ld_32x32_at;
using attn::unpack2;

__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void red_add_f32(float* addr, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory");
}

// fp32 tile in shared memory (row-major, the tensor map's box) added to global memory by the TMA unit
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, uint32_t smem_src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map),
               "r"(x), "r"(y), "r"(z), "r"(smem_src)
               : "memory");
}
// contiguous bytes, both ends on 16 bytes
__device__ __forceinline__ void bulk_store(float* dst, uint32_t smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

template <int HD, bool CAUSAL, bool HAS_DOC>
__global__ void __launch_bounds__(THREADS, 1)
kf_attn_bwd_tcgen05(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                    const __grid_constant__ CUtensorMap map_dq, int dq_tma, const float* __restrict__ LSE, const float* __restrict__ Dsum, const int* __restrict__ doc_ids,
                    float* __restrict__ dQacc, __nv_bfloat16* __restrict__ dK, __nv_bfloat16* __restrict__ dV, int Sq,
                    int Sk, int H, int group, long long lddk, long long lddv, float scale, int* status,
                    const float* __restrict__ cosT, const float* __restrict__ sinT, const int2* __restrict__ doc_range) {
  constexpr int KV_TILE_BYTES = Cfg<HD>::KV_TILE_BYTES, Q_TILE_BYTES = Cfg<HD>::Q_TILE_BYTES, BLOCKS = Cfg<HD>::BLOCKS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t k_smem = smem_base;
  const uint32_t v_smem = k_smem + KV_TILE_BYTES;
  const uint32_t q_smem = v_smem + KV_TILE_BYTES;                 // STAGES tiles
  const uint32_t do_smem = q_smem + STAGES * Q_TILE_BYTES;        // STAGES tiles
  const uint32_t ds_smem = do_smem + STAGES * Q_TILE_BYTES;
  const uint32_t bar_base = ds_smem + 2 * DS_BYTES;  // dS^T is double buffered
  uint8_t* ds_gen = smem_gen + 2 * KV_TILE_BYTES + STAGES * 2 * Q_TILE_BYTES;
  uint8_t* bar_gen = ds_gen + 2 * DS_BYTES;
  // barriers (8 B each)
  const uint32_t kv_full = bar_base;
  auto qdo_full = [&](int st) { return bar_base + 8u * (1 + st); };     // 3
  auto stage_free = [&](int st) { return bar_base + 8u * (4 + st); };   // 3
  auto ds_free = [&](int buf) { return bar_base + 8u * (7 + buf); };    // 2
  // one per dS^T buffer: a warp may arrive for tile t + 1 before another has for t (but not for t + 2, whose scores wait for both)
  auto ds_ready = [&](int buf) { return bar_base + 8u * (buf ? 17 : 10); };
  const uint32_t sdp_full = bar_base + 8u * 9, mma_done = bar_base + 8u * 11,
                 dq_free = bar_base + 8u * 12, drain_bar = bar_base + 8u * 13, sdp_taken = bar_base + 8u * 14,
                 final_bar = bar_base + 8u * 15, tmem_slot = bar_base + 8u * 16;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(bar_gen + 128);
  float* stat_smem = reinterpret_cast<float*>(bar_gen + 256);       // [2][half][lse2 | D][32]
  int* docq_smem = reinterpret_cast<int*>(bar_gen + 256 + 1024);    // [2][half][32]
  uint32_t* act = reinterpret_cast<uint32_t*>(bar_gen + 256 + 1024 + 512);  // active query tiles (one bit each)
  const uint32_t dq_stage = bar_base + AUX_BYTES;                   // only allocated when dq_tma

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  // grid: x = (batch, KV head), y = key tile.  Blocks are handed out x-fastest, so with a causal mask all the
  // heaviest key tiles (the earliest: every query sees them) start first and the lightest ones fill the tail.
  const int n_kv_tiles = gridDim.y;
  const int kt = CAUSAL ? blockIdx.y : (n_kv_tiles - 1 - blockIdx.y);
  const int Hkv_ = H / group;
  const int hk = blockIdx.x % Hkv_, b = blockIdx.x / Hkv_;
  const int k0 = kt * BLK_K;
  const int n_q_tiles = (Sq + BLK_Q - 1) / BLK_Q;
  const int i_start = CAUSAL ? min(n_q_tiles, k0 / BLK_Q) : 0;
  // packed documents: query tiles whose id range misses the key tile's are left out by every role alike
  const bool skip = HAS_DOC && doc_range != nullptr && docblk::fits(n_q_tiles);
  if (HAS_DOC && skip) {
    static_assert(BLK_Q == docblk::ROWS, "one id range per query tile");
    const int n64 = docblk::n_blocks(Sk);
    const int2* rg = doc_range + size_t(b) * n64;
    const tilemath::IdRange own = docblk::ids(docblk::merged(rg, n64, k0 / docblk::ROWS, BLK_K / docblk::ROWS));
    docblk::build_mask(act, n_q_tiles, [&](int j) { return tilemath::query_tile_walked(j, i_start, docblk::ids(rg[j]), own); });
  }
  const float scale_log2 = scale * 1.4426950408889634f;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int st = 0; st < STAGES; ++st) {
      mbar_init(qdo_full(st), 1);
      mbar_init(stage_free(st), 1);
    }
    mbar_init(sdp_full, 1);
    mbar_init(ds_ready(0), 8);
    mbar_init(ds_ready(1), 8);
    mbar_init(mma_done, 1);
    mbar_init(dq_free, 4);
    mbar_init(sdp_taken, 8);
    mbar_init(final_bar, 1);
    mbar_init(ds_free(0), 1);
    mbar_init(ds_free(1), 1);
    mbar_init(drain_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  const int n_i = skip ? docblk::count(act, n_q_tiles) : n_q_tiles - i_start;
  const int n_iter = n_i * group;
  // iteration -> (query head, first query): every role walks the active query tiles of each head in order
  struct Walk {
    int i, head;
  };
  auto walk_begin = [&]() { return Walk{skip ? docblk::next(act, 0, n_q_tiles) : i_start, hk * group}; };
  auto walk_next = [&](Walk w) {
    w.i = skip ? docblk::next(act, w.i + 1, n_q_tiles) : w.i + 1;
    if (w.i >= n_q_tiles) {
      w.i = skip ? docblk::next(act, 0, n_q_tiles) : i_start;
      ++w.head;
    }
    return w;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      bool ok = true;
      int issued = 0;
      mbar_expect_tx(kv_full, 2 * KV_TILE_BYTES);
#pragma unroll
      for (int c = 0; c < BLOCKS; ++c) {
        tma_load_3d(k_smem + c * KV_BLOCK_BYTES, &map_k, kv_full, hk * HD + 64 * c, k0, b);
        tma_load_3d(v_smem + c * KV_BLOCK_BYTES, &map_v, kv_full, hk * HD + 64 * c, k0, b);
      }
      Walk wk = walk_begin();
      for (int it = 0; it < n_iter; ++it, wk = walk_next(wk)) {
        const int st = it % STAGES;
        const int use = it / STAGES;
        if (use > 0 && !mbar_wait(stage_free(st), (use - 1) & 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
        const int hq = wk.head;
        const int q0 = wk.i * BLK_Q;
        mbar_expect_tx(qdo_full(st), 2 * Q_TILE_BYTES);
#pragma unroll
        for (int c = 0; c < BLOCKS; ++c) {
          tma_load_3d(q_smem + st * Q_TILE_BYTES + c * Q_BLOCK_BYTES, &map_q, qdo_full(st), hq * HD + 64 * c,
                      q0, b);
          tma_load_3d(do_smem + st * Q_TILE_BYTES + c * Q_BLOCK_BYTES, &map_do, qdo_full(st), hq * HD + 64 * c,
                      q0, b);
        }
        ++issued;
      }
      if (!ok) {
        mbar_wait(kv_full, 0, status, KF_ERR_WAIT_DRAIN);
        for (int it = max(0, issued - STAGES); it < issued; ++it)
          mbar_wait(qdo_full(it % STAGES), (it / STAGES) & 1, status, KF_ERR_WAIT_DRAIN);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_st = umma_idesc_bf16(128, BLK_Q, false, false);  // S^T, dP^T
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, HD, false, true);     // dV, dK (B = rows of Q_i / dO_i)
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, BLK_Q, true, true);    // dQ^T = K^T dS
      bool ok = mbar_wait(kv_full, 0, status, KF_ERR_WAIT_FULL);
      // S^T(t) = K Q^T into score buffer t & 1 and dP^T(t) = V dO^T: all operands with the head dim contiguous
      auto issue_scores = [&](int t) -> bool {
        const int st = t % STAGES, buf = t & 1;
        const uint32_t qs = q_smem + st * Q_TILE_BYTES, dos = do_smem + st * Q_TILE_BYTES;
        if (!mbar_wait(qdo_full(st), (t / STAGES) & 1, status, KF_ERR_WAIT_FULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t a_off = (kk / 4) * KV_BLOCK_BYTES + (kk % 4) * 32;
          const uint32_t b_off = (kk / 4) * Q_BLOCK_BYTES + (kk % 4) * 32;
          tc_mma_f16(tmem_base + ST_COL + buf * BLK_Q, umma_desc_sw128(k_smem + a_off, 16, 1024),
                     umma_desc_sw128(qs + b_off, 16, 1024), idesc_st, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t a_off = (kk / 4) * KV_BLOCK_BYTES + (kk % 4) * 32;
          const uint32_t b_off = (kk / 4) * Q_BLOCK_BYTES + (kk % 4) * 32;
          tc_mma_f16(tmem_base + DPT_COL, umma_desc_sw128(v_smem + a_off, 16, 1024),
                     umma_desc_sw128(dos + b_off, 16, 1024), idesc_st, kk != 0);
        }
        tc_commit(sdp_full);
        return true;
      };
      if (ok && n_iter > 0) ok = issue_scores(0);
      for (int it = 0; it < n_iter && ok; ++it) {
        const int st = it % STAGES, buf = it & 1;
        const uint32_t qs = q_smem + st * Q_TILE_BYTES, dos = do_smem + st * Q_TILE_BYTES;
        const uint32_t dss = ds_smem + buf * DS_BYTES;
        // The next tile's scores run while the softmax warps work on this one.  S^T(it+1) goes to the other
        // score buffer (its old P^T was read by an MMA issued earlier by this thread); dP^T has one buffer,
        // free once the softmax warps have copied dP^T(it) into registers.
        if (it + 1 < n_iter) {
          if (!mbar_wait(sdp_taken, it & 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
          if (!issue_scores(it + 1)) { ok = false; break; }
        }
        if (!mbar_wait(ds_ready(buf), (it >> 1) & 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        if (it > 0 && !mbar_wait(dq_free, (it - 1) & 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        // dV += P^T dO_i : A = P^T from TMEM (8 columns per 16 queries, the second half of the queries 32 columns on),
        // B = dO_i rows (head dim contiguous)
#pragma unroll
        for (int kk = 0; kk < BLK_Q / 16; ++kk)
          tc_mma_f16_ts(tmem_base + DV_COL, tmem_base + ST_COL + buf * BLK_Q + (kk >> 1) * (BLK_Q / 2) + (kk & 1) * 8,
                        umma_desc_sw128(dos + kk * 2048, Q_BLOCK_BYTES, 1024), idesc_acc, (it | kk) != 0);
        // dK += dS^T Q_i : A = dS^T from TMEM (behind P^T of the same queries), B = Q_i rows
#pragma unroll
        for (int kk = 0; kk < BLK_Q / 16; ++kk)
          tc_mma_f16_ts(tmem_base + DK_COL, tmem_base + ST_COL + buf * BLK_Q + (kk >> 1) * (BLK_Q / 2) + 16 + (kk & 1) * 8,
                        umma_desc_sw128(qs + kk * 2048, Q_BLOCK_BYTES, 1024), idesc_acc, (it | kk) != 0);
        // dQ_i^T = K^T dS : A = K rows read with the head dim as M, B = dS^T rows read with the query dim as N.  With 64
        // head dims the upper half of M is whatever follows K in shared memory (V): those 64 lanes are never read.
#pragma unroll
        for (int kk = 0; kk < BLK_K / 16; ++kk)
          tc_mma_f16(tmem_base + DQT_COL, umma_desc_sw128(k_smem + kk * 2048, KV_BLOCK_BYTES, 1024),
                     umma_desc_sw128(dss + kk * 2048, DS_BYTES, 1024), idesc_dq, kk != 0);
        tc_commit(stage_free(st));
        tc_commit(ds_free(buf));
        tc_commit(mma_done);
      }
      if (ok) tc_commit(final_bar);  // every MMA of this CTA has retired: dK / dV are final
      if (!ok) {
        tc_commit(drain_bar);
        mbar_wait(drain_bar, 0, status, KF_ERR_WAIT_DRAIN);
      }
    }
  } else if (warp < 6 || warp >= 10) {
    // ------------------------------------------------------------ softmax warps: one thread per (key row, half of the queries)
    constexpr int HQ = BLK_Q / 2;             // queries per thread
    const int half = warp >= 10 ? 1 : 0;
    const int quarter = warp & 3;
    const int r_local = quarter * 32 + lane;  // key row of this thread
    const int kpos = k0 + r_local;
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16);
    const int t128 = quarter * 32 + lane;     // 0 .. 31 of a half fetch -lse (log2 units), 32 .. 63 -D, 64 .. 95 document ids
    int doc_k = 0;
    if (HAS_DOC) doc_k = kpos < Sk ? doc_ids[size_t(b) * Sk + kpos] : -2;
    bool ok = true;
    // the statistics of this half's queries of iteration `t`, fetched one iteration ahead so that the global-memory latency
    // hides under the arithmetic of the current tile: as they lie in memory, because the first instruction that touches a loaded
    // value waits for it (the factor applied here held every tile up by 800 cycles)
    auto fetch_stat = [&](int t, const Walk& w) -> float {
      if (t128 >= (HAS_DOC ? 96 : 64) || t >= n_iter) return 0.f;
      const int qq = w.i * BLK_Q + half * HQ + lane;
      const size_t idx = (size_t(b) * H + w.head) * Sq + qq;
      if (t128 < 32) return qq < Sq ? LSE[idx] : INFINITY;  // P = 0 for padding rows
      if (t128 < 64) return qq < Sq ? Dsum[idx] : 0.f;
      return __int_as_float(qq < Sq ? doc_ids[size_t(b) * Sq + qq] : -1);
    };
    Walk ahead = walk_begin();
    float stat_next = fetch_stat(0, ahead);
    const uint64_t scale2 = pack2(scale_log2, scale_log2);
    for (int it = 0; it < n_iter; ++it) {
      const int q0 = ahead.i * BLK_Q;
      ahead = walk_next(ahead);
      float* stat = stat_smem + ((it & 1) * 2 + half) * (2 * HQ);
      int* dq_doc = docq_smem + ((it & 1) * 2 + half) * HQ;
      if (t128 < 64) stat[t128] = stat_next * (t128 < 32 ? -1.4426950408889634f : -1.f);
      else if (HAS_DOC && t128 < 96) dq_doc[lane] = __float_as_int(stat_next);
      group_sync(half == 0 ? 1 : 3, 128);  // the halves run apart: a scheduler holds one warp of each
      stat_next = fetch_stat(it + 1, ahead);
      if (ok && !mbar_wait(sdp_full, it & 1, status, KF_ERR_WAIT_TMEM_FULL)) ok = false;
      tc_fence_after();
      const uint32_t t_s = t_lane + ST_COL + (it & 1) * BLK_Q;
      uint32_t sv[HQ], dp[HQ];
      tmem_ld_32x32_at(t_s + half * HQ, sv);
      tmem_ld_32x32_at(t_lane + DPT_COL + half * HQ, dp);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sdp_taken);  // dP^T is in registers: the next tile's dP^T may be computed
      const bool tile_masked = HAS_DOC || (CAUSAL && q0 < k0 + BLK_K - 1) || (k0 + BLK_K > Sk) || (q0 + BLK_Q > Sq);
      uint32_t pk[HQ / 2], dsk[HQ / 2];
#pragma unroll
      for (int i4 = 0; i4 < HQ / 4; ++i4) {
        // four queries per step: their -lse / -D come as two 16-byte broadcast reads of two pairs each
        const ulonglong2 l4 = *reinterpret_cast<const ulonglong2*>(stat + 4 * i4);
        const ulonglong2 d4 = *reinterpret_cast<const ulonglong2*>(stat + HQ + 4 * i4);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = 4 * i4 + 2 * u;       // index inside this thread's half
          float p0, p1, s0, s1;
          unpack2(ffma2(pack2(__uint_as_float(sv[c]), __uint_as_float(sv[c + 1])), scale2, u == 0 ? l4.x : l4.y), p0, p1);
          p0 = fast_exp2(p0);
          p1 = fast_exp2(p1);
          if (tile_masked) {
            const int qpos = q0 + half * HQ + c;
            bool v0 = kpos < Sk && qpos < Sq, v1 = kpos < Sk && qpos + 1 < Sq;
            if (CAUSAL) {
              v0 = v0 && kpos <= qpos;
              v1 = v1 && kpos <= qpos + 1;
            }
            if (HAS_DOC) {
              v0 = v0 && dq_doc[c] == doc_k;
              v1 = v1 && dq_doc[c + 1] == doc_k;
            }
            p0 = v0 ? p0 : 0.f;
            p1 = v1 ? p1 : 0.f;
          }
          unpack2(fmul2(pack2(p0, p1), fadd2(pack2(__uint_as_float(dp[c]), __uint_as_float(dp[c + 1])), u == 0 ? d4.x : d4.y)),
                  s0, s1);
          pk[2 * i4 + u] = pack_bf16(p0, p1);
          dsk[2 * i4 + u] = pack_bf16(s0, s1);
        }
      }
      // P^T over the start of this half of S^T (bf16 pairs: 16 columns for 32 queries), which this warp alone has read
      // and dS^T behind it
      tmem_st_32x16(t_s + half * HQ, pk);
      tmem_st_32x16(t_s + half * HQ + HQ / 2, dsk);
      // dS^T into shared memory, 128B-swizzled rows (16-byte chunk c of row r lives at chunk c ^ (r % 8));
      // the dQ MMAs, its only readers, must have finished with it (two buffers: those of iteration it-2 were this one's last)
      if (it > 1 && ok && !mbar_wait(ds_free(it & 1), ((it >> 1) - 1) & 1, status, KF_ERR_WAIT_TMEM_FULL)) ok = false;
      {
        uint8_t* row_ptr = ds_gen + (it & 1) * DS_BYTES + r_local * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) {   // this thread's 32 queries = four 16-byte chunks of the row
          uint4 w = make_uint4(dsk[4 * c], dsk[4 * c + 1], dsk[4 * c + 2], dsk[4 * c + 3]);
          *reinterpret_cast<uint4*>(row_ptr + (((half * 4 + c) ^ (r_local & 7)) << 4)) = w;
        }
      }
      fence_async_smem();  // generic-proxy stores -> visible to the tensor core's async-proxy reads
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready(it & 1));
    }
    // ---- epilogue: dK / dV accumulators -> bf16 rows of the key tile (first softmax group: one thread per key row)
    if (half != 0) ok = false;
    if (ok && n_iter > 0 && !mbar_wait(final_bar, 0, status, KF_ERR_WAIT_TMEM_FULL)) ok = false;
    if (ok && cosT != nullptr && n_iter > 0) {
      // dK leaves through the inverse rotary embedding (the forward rotated K after the projection): columns
      // (i, i + 64) of a head are a pair, the angle is that of the key's position
      tc_fence_after();
      __nv_bfloat16* dst = dK + (size_t(b) * Sk + kpos) * lddk + size_t(hk) * HD;
      const float* cr = cosT + size_t(min(kpos, Sk - 1)) * (HD / 2);
      const float* sr = sinT + size_t(min(kpos, Sk - 1)) * (HD / 2);
#pragma unroll 1
      for (int c = 0; c < HD / 64; ++c) {
        uint32_t lo[32], hi[32];
        tmem_ld_32x32_at(t_lane + DK_COL + c * 32, lo);
        tmem_ld_32x32_at(t_lane + DK_COL + HD / 2 + c * 32, hi);
        tmem_ld_wait();
        if (kpos < Sk) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float a[8], bb[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float cv = cr[c * 32 + 8 * i + e], sv2 = sr[c * 32 + 8 * i + e];
              const float x = __uint_as_float(lo[8 * i + e]) * scale, y = __uint_as_float(hi[8 * i + e]) * scale;
              a[e] = x * cv + y * sv2;
              bb[e] = y * cv - x * sv2;
            }
            uint4 w0, w1;
            w0.x = pack_bf16(a[0], a[1]); w0.y = pack_bf16(a[2], a[3]); w0.z = pack_bf16(a[4], a[5]); w0.w = pack_bf16(a[6], a[7]);
            w1.x = pack_bf16(bb[0], bb[1]); w1.y = pack_bf16(bb[2], bb[3]); w1.z = pack_bf16(bb[4], bb[5]); w1.w = pack_bf16(bb[6], bb[7]);
            *reinterpret_cast<uint4*>(dst + c * 32 + 8 * i) = w0;
            *reinterpret_cast<uint4*>(dst + HD / 2 + c * 32 + 8 * i) = w1;
          }
        }
      }
    }
    if (ok) {
      tc_fence_after();
#pragma unroll 1
      for (int which = 0; which < ((cosT != nullptr && n_iter > 0) ? 1 : 2); ++which) {
        __nv_bfloat16* dst = which == 0 ? dV + (size_t(b) * Sk + kpos) * lddv + size_t(hk) * HD
                                        : dK + (size_t(b) * Sk + kpos) * lddk + size_t(hk) * HD;
        const uint32_t col0 = which == 0 ? DV_COL : DK_COL;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          if (n_iter > 0) {
            tmem_ld_32x32_at(t_lane + col0 + c * 32, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
          const float f = which == 0 ? 1.f : scale;
          if (kpos < Sk) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 w;
              w.x = pack_bf16(__uint_as_float(o[8 * i + 0]) * f, __uint_as_float(o[8 * i + 1]) * f);
              w.y = pack_bf16(__uint_as_float(o[8 * i + 2]) * f, __uint_as_float(o[8 * i + 3]) * f);
              w.z = pack_bf16(__uint_as_float(o[8 * i + 4]) * f, __uint_as_float(o[8 * i + 5]) * f);
              w.w = pack_bf16(__uint_as_float(o[8 * i + 6]) * f, __uint_as_float(o[8 * i + 7]) * f);
              *reinterpret_cast<uint4*>(dst + c * 32 + 8 * i) = w;
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ dQ reduction warps (6..9)
    const int quarter = warp & 3;
    const int d = quarter * 32 + lane;  // head-dim index = TMEM lane of dQ^T
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16);
    const bool elected = threadIdx.x == 192;  // issues, commits and waits for the bulk reductions
    bool ok = true;
    Walk wk = walk_begin();
    for (int it = 0; it < n_iter; ++it, wk = walk_next(wk)) {
      const int hq = wk.head;
      const int q0 = wk.i * BLK_Q;
      if (ok && !mbar_wait(mma_done, it & 1, status, KF_ERR_WAIT_TMEM_FULL)) ok = false;
      tc_fence_after();
      uint32_t v[BLK_Q];
      tmem_ld_32x32_at(t_lane + DQT_COL, v);
      tmem_ld_32x32_at(t_lane + DQT_COL + 32, v + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_free);  // the values are in registers: the next dQ^T may be computed
      if (HD == 64 || dq_tma) {
        // transpose through shared memory into a [query][head dim] tile.  Head dim 128: the tile that the tensor map describes, added
        // by one bulk reduction, which leaves out the rows past the end of the sequence.  64: 16 KB in this key tile's own part,
        // which has rows for padding queries
        if (elected) bulk_wait_read_all();  // the previous copy has read the staging tile
        group_sync(2, 128);
#pragma unroll
        for (int c = 0; c < BLK_Q; ++c)
          if (HD == 128 || d < HD)
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(dq_stage + uint32_t(c * HD + d) * 4u), "r"(v[c]) : "memory");
        fence_async_smem();
        group_sync(2, 128);
        if (elected && ok) {
          if constexpr (HD == 64)
            bulk_store(dQacc + (((size_t(kt) * (gridDim.x / Hkv_) + b) * H + hq) * n_q_tiles + wk.i) * (BLK_Q * HD), dq_stage,
                       BLK_Q * HD * 4);
          else
            tma_reduce_add_3d(&map_dq, dq_stage, hq * HD, q0, b);
          bulk_commit();
        }
      } else if (ok) {
        float* base = dQacc + ((size_t(b) * Sq + q0) * H + hq) * HD + d;
#pragma unroll
        for (int c = 0; c < BLK_Q; ++c)
          if (q0 + c < Sq) red_add_f32(base + size_t(c) * H * HD, __uint_as_float(v[c]));
      }
    }
    if ((HD == 64 || dq_tma) && elected) bulk_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// D[b, h, s] = sum_d O[b, s, h, d] * dO[b, s, h, d]: HD / 8 lanes x 16 bytes per (b, s, h) row, 8 (16) rows per warp with all
// eight loads of a lane in flight.  Memory-bound; one row per warp with one 8-byte load per lane and operand ran at a quarter
// of the copy rate (80 us at 8192 x 32 heads, 134 MB), this form took 35 us with
// 64-bit divisions for its rows and takes 28 with 32-bit ones (3000 x 40 heads 19.4 -> 14.2; 20 and 9 at the copy rate).
template <int HD>
__global__ void __launch_bounds__(256) kf_attn_bwd_dot(const __nv_bfloat16* __restrict__ O, const __nv_bfloat16* __restrict__ dO,
                                                          float* __restrict__ D, int B, int S, int H, long long ldo,
                                                          long long lddo) {
  const int rows = B * S * H;  // 2^31 rows would be 275 GB of O
  constexpr int LANES = HD / 8, PER = 32 / LANES;  // lanes per row, rows per warp and load
  const int r0 = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * (4 * PER);
  const int lane = threadIdx.x & 31, sub = lane / LANES, c = (lane % LANES) * 8;
  if (r0 >= rows) return;
  uint4 a[4], g[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int row = r0 + u * PER + sub < rows ? r0 + u * PER + sub : rows - 1, bs = row / H, h = row - bs * H;
    a[u] = *reinterpret_cast<const uint4*>(O + bs * ldo + h * HD + c);
    g[u] = *reinterpret_cast<const uint4*>(dO + bs * lddo + h * HD + c);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, gw[4] = {g[u].x, g[u].y, g[u].z, g[u].w};
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16(aw[i]), y = unpack_bf16(gw[i]);
      acc += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int row = r0 + u * PER + sub;
    if (lane % LANES == 0 && row < rows) {
      const int bs = row / H, b = bs / S;
      D[(b * H + (row - bs * H)) * S + (bs - b * S)] = acc;
    }
  }
}

// scale * fp32 (rows x cols contiguous) -> bf16 rows with pitch ld
__global__ void kf_f32_to_bf16_rows(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long rows,
                                    int cols, long long ld, float scale) {
  const long long n4 = rows * (cols / 4);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / (cols / 4);
    const int c = (i % (cols / 4)) * 4;
    const float4 v = *reinterpret_cast<const float4*>(src + r * cols + c);
    uint2 w;
    w.x = pack_bf16(v.x * scale, v.y * scale);
    w.y = pack_bf16(v.z * scale, v.w * scale);
    *reinterpret_cast<uint2*>(dst + r * ld + c) = w;
  }
}

// scale * fp32 dQ [rows][H * 128] -> bf16 rows with pitch ld, through the inverse rotary embedding of position (row % S)
__global__ void kf_dq_finish_rope(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long rows, int H,
                                  long long ld, const float* __restrict__ cosT, const float* __restrict__ sinT, int S,
                                  float scale) {
  constexpr int HD = 128, HALF = HD / 2;
  const long long n4 = rows * H * (HALF / 4);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const int j = (i % (HALF / 4)) * 4;
    const long long rh = i / (HALF / 4);
    const int h = rh % H;
    const long long r = rh / H;
    const int pos = r % S;
    float4 a = *reinterpret_cast<const float4*>(src + (r * H + h) * HD + j);
    float4 b = *reinterpret_cast<const float4*>(src + (r * H + h) * HD + HALF + j);
    a.x *= scale; a.y *= scale; a.z *= scale; a.w *= scale;
    b.x *= scale; b.y *= scale; b.z *= scale; b.w *= scale;
    const float4 c = *reinterpret_cast<const float4*>(cosT + size_t(pos) * HALF + j);
    const float4 s = *reinterpret_cast<const float4*>(sinT + size_t(pos) * HALF + j);
    uint2 lo, hi;
    lo.x = pack_bf16(a.x * c.x + b.x * s.x, a.y * c.y + b.y * s.y);
    lo.y = pack_bf16(a.z * c.z + b.z * s.z, a.w * c.w + b.w * s.w);
    hi.x = pack_bf16(b.x * c.x - a.x * s.x, b.y * c.y - a.y * s.y);
    hi.y = pack_bf16(b.z * c.z - a.z * s.z, b.w * c.w - a.w * s.w);
    *reinterpret_cast<uint2*>(dst + r * ld + h * HD + j) = lo;
    *reinterpret_cast<uint2*>(dst + r * ld + h * HD + HALF + j) = hi;
  }
}

// Head dim 64: scale * the sum of the parts [key tile][b][head][query tile][64 queries][64] -> bf16 rows with pitch ld, in the order of
// the key tiles; with cosT through the inverse rotary embedding.  causal: a query's keys end with its own tile.
__global__ void kf_dq_add_parts(const float* __restrict__ parts, __nv_bfloat16* __restrict__ dst, int B, int S, int H, int key_tiles,
                                int causal, long long ld, const float* __restrict__ cosT, const float* __restrict__ sinT, float scale) {
  constexpr int HD = 64, HALF = HD / 2;
  const int n_q_tiles = (S + BLK_Q - 1) / BLK_Q;
  const size_t part = size_t(B) * H * n_q_tiles * (BLK_Q * HD);
  const long long n4 = (long long)B * S * H * (HALF / 4);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const int j = (i % (HALF / 4)) * 4;
    const long long rh = i / (HALF / 4), r = rh / H;
    const int h = rh % H, pos = r % S, b = r / S;
    const float* src = parts + ((size_t(b) * H + h) * n_q_tiles * BLK_Q + pos) * HD + j;
    const int n = causal ? min(key_tiles, pos / BLK_K + 1) : key_tiles;
    float4 a = *reinterpret_cast<const float4*>(src), c = *reinterpret_cast<const float4*>(src + HALF);
#pragma unroll 4
    for (int t = 1; t < n; ++t) {
      const float4 u = *reinterpret_cast<const float4*>(src + t * part), v = *reinterpret_cast<const float4*>(src + t * part + HALF);
      a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
      c.x += v.x; c.y += v.y; c.z += v.z; c.w += v.w;
    }
    const float lo[4] = {a.x * scale, a.y * scale, a.z * scale, a.w * scale}, hi[4] = {c.x * scale, c.y * scale, c.z * scale, c.w * scale};
    float x[4], y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float cs = cosT ? cosT[size_t(pos) * HALF + j + e] : 1.f, sn = cosT ? sinT[size_t(pos) * HALF + j + e] : 0.f;
      x[e] = cosT ? lo[e] * cs + hi[e] * sn : lo[e];
      y[e] = cosT ? hi[e] * cs - lo[e] * sn : hi[e];
    }
    __nv_bfloat16* out = dst + r * ld + h * HD + j;
    *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
    *reinterpret_cast<uint2*>(out + HALF) = make_uint2(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]));
  }
}

}  // namespace attnb
}  // namespace kf

extern "C" void* kf_status_device_ptr();

namespace kf {
namespace attnb {
static int g_dq_mode = 1;  // 0: red.global per element, 1: bulk tensor reduction from shared memory (1.75x faster)

// fp32 [planes][rows][cols] without gaps -> tensor map with an unswizzled (box_cols x box_rows x 1) box
inline int make_map_3d_f32_plain(CUtensorMap* map, const void* base, uint64_t planes, uint64_t rows, uint64_t cols,
                                 uint32_t box_cols, uint32_t box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -1;
  cuuint64_t dims[3] = {cols, rows, planes};
  cuuint64_t strides[2] = {cols * 4, rows * cols * 4};
  cuuint32_t box[3] = {box_cols, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}
}  // namespace attnb
}  // namespace kf

namespace kf {
namespace attnb {
template <int HD>
static int run(const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse,
                          void* dsum, void* dq_acc, void* dq, void* dk, void* dv, const void* doc, int B, int Sq, int Sk,
                          int H, int Hkv, long long ldq, long long ldk, long long ldv, long long ldo,
                          long long lddo, long long lddq, long long lddk, long long lddv, float scale, int causal,
                          const void* cosT, const void* sinT, const void* doc_range, cudaStream_t st) {
  using C = Cfg<HD>;
  constexpr int hd = HD;
  CUtensorMap mq, mk, mv, mdo;
  int rc = make_map_3d_bf16(&mq, q, B, Sq, uint64_t(H) * hd, 64, BLK_Q, ldq);
  if (rc) return 100 + rc;
  rc = make_map_3d_bf16(&mk, k, B, Sk, uint64_t(Hkv) * hd, 64, BLK_K, ldk);
  if (rc) return 200 + rc;
  rc = make_map_3d_bf16(&mv, v, B, Sk, uint64_t(Hkv) * hd, 64, BLK_K, ldv);
  if (rc) return 250 + rc;
  rc = make_map_3d_bf16(&mdo, d_o, B, Sq, uint64_t(H) * hd, 64, BLK_Q, lddo);
  if (rc) return 270 + rc;
  const int dq_tma = HD == 128 ? g_dq_mode : 1;
  CUtensorMap mdq = mq;
  if (HD == 128) rc = make_map_3d_f32_plain(&mdq, dq_acc, B, Sq, uint64_t(H) * hd, HD, BLK_Q);
  if (rc) return 280 + rc;
  const size_t smem_bytes = dq_tma ? C::SMEM_DQ_TMA : C::SMEM;
  const int key_tiles = (Sk + BLK_K - 1) / BLK_K, q_tiles = (Sq + BLK_Q - 1) / BLK_Q;
  // pre-pass: D = rowsum(dO * O); zero the fp32 dQ accumulator (the parts of head dim 64 where documents leave tiles out)
  {
    const long long rows = (long long)B * Sq * H;
    const int threads = 256;
    constexpr int ROWS_PER_WARP = 4 * 32 / (HD / 8);
    const long long blocks = ((rows + ROWS_PER_WARP - 1) / ROWS_PER_WARP * 32 + threads - 1) / threads;
    kf_attn_bwd_dot<HD><<<(unsigned)blocks, threads, 0, st>>>(reinterpret_cast<const __nv_bfloat16*>(o),
                                                             reinterpret_cast<const __nv_bfloat16*>(d_o),
                                                             reinterpret_cast<float*>(dsum), B, Sq, H, ldo, lddo);
    cudaError_t e = cudaSuccess;
    if (HD == 128) e = cudaMemsetAsync(dq_acc, 0, size_t(B) * Sq * H * hd * sizeof(float), st);
    else if (doc) e = cudaMemsetAsync(dq_acc, 0, size_t(key_tiles) * B * H * q_tiles * BLK_Q * hd * sizeof(float), st);
    if (e != cudaSuccess) return 400 + (int)e;
  }
  int* status = reinterpret_cast<int*>(kf_status_device_ptr());
  dim3 grid(Hkv * B, key_tiles);
#define KF_BWD_LAUNCH(C_, D_)                                                                                      \
  {                                                                                                                \
    auto kern = kf_attn_bwd_tcgen05<HD, C_, D_>;                                                                       \
    static bool attr_set = false;                                                                                  \
    if (!attr_set) {                                                                                               \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_DQ_TMA);   \
      if (e != cudaSuccess) return 300 + (int)e;                                                                   \
      attr_set = true;                                                                                             \
    }                                                                                                              \
    kern<<<grid, THREADS, smem_bytes, st>>>(mq, mk, mv, mdo, mdq, dq_tma, reinterpret_cast<const float*>(lse),     \
                                      reinterpret_cast<const float*>(dsum), reinterpret_cast<const int*>(doc),     \
                                      reinterpret_cast<float*>(dq_acc), reinterpret_cast<__nv_bfloat16*>(dk),      \
                                      reinterpret_cast<__nv_bfloat16*>(dv), Sq, Sk, H, H / Hkv, lddk, lddv, scale, \
                                      status, reinterpret_cast<const float*>(cosT),                                \
                                      reinterpret_cast<const float*>(sinT),                                        \
                                      reinterpret_cast<const int2*>(doc_range));                                   \
  }
  if (doc) {
    if (causal) KF_BWD_LAUNCH(true, true) else KF_BWD_LAUNCH(false, true)
  } else {
    if (causal) KF_BWD_LAUNCH(true, false) else KF_BWD_LAUNCH(false, false)
  }
#undef KF_BWD_LAUNCH
  {
    const long long rows = (long long)B * Sq;
    const int cols = H * hd;
    if (HD == 64)
      kf_dq_add_parts<<<1184, 256, 0, st>>>(reinterpret_cast<const float*>(dq_acc), reinterpret_cast<__nv_bfloat16*>(dq), B, Sq, H,
                                            key_tiles, causal, lddq, reinterpret_cast<const float*>(cosT),
                                            reinterpret_cast<const float*>(sinT), scale);
    else if (cosT)
      kf_dq_finish_rope<<<1184, 256, 0, st>>>(reinterpret_cast<const float*>(dq_acc), reinterpret_cast<__nv_bfloat16*>(dq),
                                              rows, H, lddq, reinterpret_cast<const float*>(cosT),
                                              reinterpret_cast<const float*>(sinT), Sq, scale);
    else
      kf_f32_to_bf16_rows<<<1184, 256, 0, st>>>(reinterpret_cast<const float*>(dq_acc),
                                                reinterpret_cast<__nv_bfloat16*>(dq), rows, cols, lddq, scale);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace attnb
}  // namespace kf

extern "C" {

// How the backward kernel adds its dQ tiles to the fp32 accumulator (head dim 128): 0 = red.global per element,
// 1 = one bulk tensor reduction per tile (default).  Returns the previous mode.
int kf_attn_bwd_dq_mode(int mode) {
  const int prev = kf::attnb::g_dq_mode;
  if (mode == 0 || mode == 1) kf::attnb::g_dq_mode = mode;
  return prev;
}

// Backward attention (head dim 64 or 128).  q / k / v / o / do: rows (b * S + s) with pitches ld*, heads side by
// side; lse: fp32 [B][H][Sq] from the forward; dsum: fp32 scratch [B][H][Sq]; dq_acc: fp32 scratch, [B][Sq][H][128] (zeroed
// here) or, for head dim 64, [ceil(Sk / 128)][B][H][ceil(Sq / 64) * 64][64]; dq / dk / dv: bf16 outputs with pitches lddq / lddk /
// lddv (they may be slices of one fused gradient buffer).  doc: optional int32 [B][S].  Requires Sq == Sk when causal or doc.
// kf_attn_bwd_rope_bf16: the same, and dq / dk additionally pass through the inverse rotary embedding (cosT / sinT:
// fp32 [Sq][hd / 2], position = index inside the sequence), i.e. they are gradients with respect to the un-rotated
// projections when q / k were rotated after the projection.  Null tables = no rotation.  doc_range (optional): the id
// ranges kf_doc_blocks wrote for `doc`; query tiles without a visible pair are skipped with it.
int kf_attn_bwd_rope_bf16(const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse,
                          void* dsum, void* dq_acc, void* dq, void* dk, void* dv, const void* doc, int B, int Sq, int Sk,
                          int H, int Hkv, int hd, long long ldq, long long ldk, long long ldv, long long ldo,
                          long long lddo, long long lddq, long long lddk, long long lddv, float scale, int causal,
                          const void* cosT, const void* sinT, const void* doc_range, void* stream) {
  using namespace kf::attnb;
  if ((hd != 64 && hd != 128) || Hkv <= 0 || H % Hkv != 0) return 3;
  if ((causal || doc) && Sq != Sk) return 4;
  if ((ldq | ldk | ldv | ldo | lddo | lddq | lddk | lddv) & 7) return 5;
  auto fn = hd == 64 ? run<64> : run<128>;
  return fn(q, k, v, o, d_o, lse, dsum, dq_acc, dq, dk, dv, doc, B, Sq, Sk, H, Hkv, ldq, ldk, ldv, ldo, lddo, lddq, lddk, lddv, scale,
            causal, cosT, sinT, doc_range, (cudaStream_t)stream);
}

int kf_attn_bwd_bf16(const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse,
                     void* dsum, void* dq_acc, void* dq, void* dk, void* dv, const void* doc, int B, int Sq, int Sk,
                     int H, int Hkv, int hd, long long ldq, long long ldk, long long ldv, long long ldo,
                     long long lddo, long long lddq, long long lddk, long long lddv, float scale, int causal,
                     void* stream) {
  return kf_attn_bwd_rope_bf16(q, k, v, o, d_o, lse, dsum, dq_acc, dq, dk, dv, doc, B, Sq, Sk, H, Hkv, hd, ldq, ldk, ldv,
                               ldo, lddo, lddq, lddk, lddv, scale, causal, nullptr, nullptr, nullptr, stream);
}

}  // extern "C"
