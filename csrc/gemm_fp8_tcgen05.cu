// FP8 GEMM on the 5th-generation tensor cores (tcgen05.mma kind::f8f6f4) plus the casts that feed it.
//
//   C[M,N] (+)= alpha * A8[M,K] * B8[N,K]^T      alpha = 1 / (scale_a * scale_b), read from device memory
//
// A8 / B8 are e4m3 or e5m2 bytes with the reduction dim contiguous ("K-major"); tensorwise scales are
// computed on the device (abs-max -> scale) and never visit the host.  Structure and synchronisation of the bf16
// pair kernel (gemm_tcgen05_2cta.cu): a CTA pair owns a 256 x tile_n tile, each CTA loads 128 rows of A and half of
// B's rows (128 K-bytes per stage, 6 stages, 128B swizzle), the leader issues tcgen05.mma cta_group::2, both
// epilogues read their own tensor memory (two accumulators) and store through shared memory.
//
// What bounds it: the operand stream.  8-bit products take half the tensor cycles of 16-bit ones per byte pair, so a
// 128 x 256 tile of a single CTA asks for 96 bytes per SM and clock; the pair needs 64.  tile_n follows the rounds of
// tiles over the pairs (2000 x 14 336: 448 tiles of 256 columns are 6.05 rounds, 512 of 224 are 6.9).
// Single-CTA 128 x 256 tiles -> pairs: 2000 x 14 336 from 4096 103 -> 88 us, 14 336 x 4096 from 2000 163 -> 115, 8192 x 6144 from
// 4096 154 -> 135 (3.05 PFLOP/s), 1 x 4096 from 4096 20.5 -> 20.5; the same bits.
// The transposed operands that dgrad / wgrad need are written by the cast kernel itself (one read of the
// bf16 source produces the row-major and the transposed fp8 copy), so every GEMM runs K-major.
//
// Covers the reference's float8 training path (torchao tensorwise scaling through
// kempnerforge/distributed/parallel.py:125-174): e4m3 for activations and weights, e5m2 for gradients.
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "pair_common.cuh"
#include "tile_math.h"
#include <cuda_fp8.h>

namespace kf {
namespace f8 {

using namespace kf::pairops;

constexpr int CTA_M = 128;    // rows of A per CTA
constexpr int TILE_M = 256;   // rows per CTA pair
constexpr int MAX_N = 256;    // columns of the widest tile
constexpr int BK = 128;       // fp8 elements = bytes per row of a stage
constexpr int UMMA_K = 32;    // K per tcgen05.mma for 8-bit inputs
constexpr int STAGES = 6;
constexpr int A_BYTES = CTA_M * BK;            // 16 KB
constexpr int B_BYTES = (MAX_N / 2) * BK;      // 16 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int TMEM_COLS = 512;
constexpr int GROUP_M = 8;
constexpr int BOX_BYTES = 2048;  // one staged 32 x 32 box per epilogue warp

// What the epilogue makes of the product.  SWIGLU: B is [gate ; up] with N rows each; the leader's half of a tile is gate rows and the
// peer's the matching up rows, C[M, N] = silu(gate) * up, and G[M, 2N] (optional) receives the pre-activations.  SWIGLU_BWD: the product
// is the gradient of the hidden activation (never stored), G[M, 2N] holds the saved pre-activations and C[M, 2N] receives their
// gradients.  Both round where the separate passes store bf16, in the same order of operations, and leave the largest magnitude that
// each warp stored in amax[block * 8 + warp], for the cast to fp8 that follows.
//
// In place of the product, a pass over 2N + N columns and a maximum, us (gate | up and the gradient, the latter's product from 4096):
// 2000 x 14 336 from 4096 201 -> 180 and 132 -> 113, 256 rows 45 -> 40 and 33 -> 29, 2448 x 8192 from 2048 91 -> 75 and 72 -> 61,
// 4096 x 3584 from 1024 52 -> 43 and 49 -> 46.  Where K is short the epilogue is what is waited for (five boxes of shared-memory traffic
// per chunk next to the operands'): eight warps (four: 3584 units from 1024 45 and 50) that each take every other chunk, and rows of G
// loaded 32 bytes per lane straight to their owners (through the boxes 52).
enum Kind { PLAIN = 0, SWIGLU = 1, SWIGLU_BWD = 2 };
template <int KIND> constexpr int EPI_WARPS = KIND == PLAIN ? 4 : 8;  // one or two for each quarter of the tensor memory
template <int KIND> constexpr int THREADS = 64 + 32 * EPI_WARPS<KIND>;
template <int KIND> constexpr size_t SMEM = size_t(STAGES) * STAGE_BYTES + EPI_WARPS<KIND> * BOX_BYTES + 1024 + 256;

// Instruction descriptor for kind::f8f6f4: fp32 accumulate, A/B format 0 = e4m3, 1 = e5m2, both K-major.
__host__ __device__ constexpr uint32_t idesc_f8(int m, int n, int a_fmt, int b_fmt) {
  return (1u << 4) | (uint32_t(a_fmt) << 7) | (uint32_t(b_fmt) << 10) | (uint32_t(n >> 3) << 17) |
         (uint32_t(m >> 4) << 24);
}

// of the eight bf16 values of a 16-byte word
__device__ __forceinline__ float absmax8(const uint4 v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  float m = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16(w[j]);
    m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
  return m;
}
// of the first `valid` (a multiple of eight) values of a row
__device__ __forceinline__ float absmax_row(const Rows32& r, int valid, float m) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (q * 8 < valid) m = fmaxf(m, absmax8(r.q[q]));
  return m;
}
// the lane's own row of a box of 32 x 32 (rows, cols: how many exist, cols a multiple of 16; the rest is zero); src and ld on 32 bytes
__device__ __forceinline__ Rows32 load_own_row(const __nv_bfloat16* src, size_t ld, int lane, int rows, int cols) {
  Rows32 r;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint4 &a = r.q[2 * h], &b = r.q[2 * h + 1];
    a = b = make_uint4(0, 0, 0, 0);
    if (lane < rows && h * 16 < cols)
      asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                   : "l"(src + lane * ld + h * 16));
  }
  return r;
}
// bf16 row of silu(gate) * up, operation for operation what kf_swiglu_fwd computes
__device__ __forceinline__ Rows32 swiglu_row(const Rows32& gate, const Rows32& up) {
  Rows32 h;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t gw[4] = {gate.q[q].x, gate.q[q].y, gate.q[q].z, gate.q[q].w}, uw[4] = {up.q[q].x, up.q[q].y, up.q[q].z, up.q[q].w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 g = unpack_bf16(gw[e]), u = unpack_bf16(uw[e]);
      o[e] = pack_bf16(g.x / (1.f + __expf(-g.x)) * u.x, g.y / (1.f + __expf(-g.y)) * u.y);
    }
    h.q[q] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  return h;
}
// gate and up are replaced by their gradients, operation for operation what kf_swiglu_bwd computes
__device__ __forceinline__ void swiglu_grad_row(const Rows32& dh, Rows32& gate, Rows32& up) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t dw[4] = {dh.q[q].x, dh.q[q].y, dh.q[q].z, dh.q[q].w};
    uint32_t gw[4] = {gate.q[q].x, gate.q[q].y, gate.q[q].z, gate.q[q].w}, uw[4] = {up.q[q].x, up.q[q].y, up.q[q].z, up.q[q].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = unpack_bf16(gw[e]), b = unpack_bf16(uw[e]), d = unpack_bf16(dw[e]);
      const float s0 = 1.f / (1.f + __expf(-a.x)), s1 = 1.f / (1.f + __expf(-a.y));
      const float silu0 = a.x * s0, silu1 = a.y * s1;
      uw[e] = pack_bf16(d.x * silu0, d.y * silu1);
      gw[e] = pack_bf16(d.x * b.x * s0 * (1.f + a.x * (1.f - s0)), d.y * b.y * s1 * (1.f + a.y * (1.f - s1)));
    }
    gate.q[q] = make_uint4(gw[0], gw[1], gw[2], gw[3]);
    up.q[q] = make_uint4(uw[0], uw[1], uw[2], uw[3]);
  }
}

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS<KIND>, 1)
kf_gemm_fp8_tcgen05_2cta(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         __nv_bfloat16* __restrict__ C, int M, int N, int K, int ldc, int accumulate, int a_fmt, int b_fmt,
                         int tile_n, const float* __restrict__ scale_a, const float* __restrict__ scale_b,
                         __nv_bfloat16* __restrict__ G, int ldg, float* __restrict__ amax, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t box_smem = smem_base + STAGES * STAGE_BYTES;
  const uint32_t bar_base = box_smem + EPI_WARPS<KIND> * BOX_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 5);
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int half_n = tile_n >> 1;
  const int m_blocks = (M + TILE_M - 1) / TILE_M;
  const int cols = KIND == SWIGLU ? half_n : tile_n;  // columns of 0 .. N that a tile covers
  const int n_blocks = (N + cols - 1) / cols;
  const int num_tiles = m_blocks * n_blocks;
  const int k_blocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 2 * EPI_WARPS<KIND>);  // the epilogue warps of both CTAs
    }
    mbar_init(drain_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
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
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        int tm, tn;
        tilemath::raster(t, m_blocks, n_blocks, GROUP_M, tm, tn);
        const int m0 = tm * TILE_M + int(rank) * CTA_M, n0 = tn * cols + int(rank) * (KIND == SWIGLU ? N : half_n);
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(empty_bar(s), ph ^ 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
          const uint32_t a_dst = smem_base + s * STAGE_BYTES;
          const uint32_t lead_full = full_bar(s) & PEER_BIT_MASK;
          if (leader) mbar_expect_tx(full_bar(s), 2 * (A_BYTES + half_n * BK));
          tma_load_2d_pair(a_dst, &map_a, lead_full, kb * BK, m0);
          tma_load_2d_pair(a_dst + A_BYTES, &map_b, lead_full, kb * BK, n0);
        }
      }
      // copies into this CTA's shared memory are complete once their stages were consumed or, on the error path, once
      // the leader's full barrier flipped
      if (leader)
        for (int j = max(0, it - STAGES); j < it; ++j)
          mbar_wait(full_bar(j % STAGES), (j / STAGES) & 1, status, KF_ERR_WAIT_DRAIN);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      const uint32_t idesc = idesc_f8(TILE_M, tile_n, a_fmt, b_fmt);
      int it = 0, tile_iter = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
        const int acc = tile_iter & 1;
        const uint32_t acc_ph = (tile_iter >> 1) & 1;
        if (!mbar_wait(tempty_bar(acc), acc_ph ^ 1, status, KF_ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * MAX_N;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(full_bar(s), ph, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_src = smem_base + s * STAGE_BYTES;
          const uint32_t b_src = a_src + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            // 32 one-byte elements per step = 32 B along the swizzled 128 B row
            mma_pair_f8(d_tmem, umma_desc_sw128(a_src + k * UMMA_K, 16, 1024),
                        umma_desc_sw128(b_src + k * UMMA_K, 16, 1024), idesc, (kb | k) != 0);
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
    // ------------------------------------------------------------ epilogue (warps 2.. of both CTAs)
    const int quarter = warp & 3, first = (warp - 2) >> 2;
    constexpr int STEP = EPI_WARPS<KIND> / 4;
    const uint32_t box = box_smem + uint32_t(warp - 2) * BOX_BYTES;
    const float alpha = 1.0f / (scale_a[0] * scale_b[0]);
    float largest = 0.f;
    int tile_iter = 0;
    bool ok = true;
    for (int t = pair; t < num_tiles && ok; t += num_pairs, ++tile_iter) {
      int tm, tn;
      tilemath::raster(t, m_blocks, n_blocks, GROUP_M, tm, tn);
      const int acc = tile_iter & 1;
      const uint32_t acc_ph = (tile_iter >> 1) & 1;
      if (!mbar_wait(tfull_bar(acc), acc_ph, status, KF_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int row0 = tm * TILE_M + int(rank) * CTA_M + quarter * 32;  // this warp's rows, and how many exist
      const int rows = max(0, min(32, M - row0));
      const int col0 = tn * cols, width = min(cols, N - col0);
      const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * MAX_N;
      __nv_bfloat16* c0 = C + size_t(row0) * ldc + col0;
      __nv_bfloat16* g0 = KIND == PLAIN || G == nullptr ? nullptr : G + size_t(row0) * ldg + col0;
      Rows32 g_next, u_next;  // saved pre-activations of the chunk that follows: under way while this one is worked on
      if (KIND == SWIGLU_BWD) {
        g_next = load_own_row(g0 + first * 32, ldg, lane, rows, width - first * 32);
        u_next = load_own_row(g0 + N + first * 32, ldg, lane, rows, width - first * 32);
      }
#pragma unroll 1
      for (int c = first; c * 32 < width; c += STEP) {
        uint32_t v[32], w[32];
        tmem_ld_32x32(t_row + c * 32, v);
        if (KIND == SWIGLU) tmem_ld_32x32(t_row + half_n + c * 32, w);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
        const int valid = min(32, width - c * 32);
        if (KIND == SWIGLU) {
#pragma unroll
          for (int i = 0; i < 32; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
          const Rows32 gate = pack_row32(v), up = pack_row32(w), h = swiglu_row(gate, up);
          largest = absmax_row(h, valid, largest);
          if (g0 != nullptr) {
            store_rows32(box, lane, gate, g0 + c * 32, ldg, rows, valid);
            store_rows32(box, lane, up, g0 + N + c * 32, ldg, rows, valid);
          }
          store_rows32(box, lane, h, c0 + c * 32, ldc, rows, valid);
        } else if (KIND == SWIGLU_BWD) {
          Rows32 gate = g_next, up = u_next;
          if (const int n = (c + STEP) * 32; n < width) {
            g_next = load_own_row(g0 + n, ldg, lane, rows, width - n);
            u_next = load_own_row(g0 + N + n, ldg, lane, rows, width - n);
          }
          swiglu_grad_row(pack_row32(v), gate, up);
          largest = absmax_row(up, valid, absmax_row(gate, valid, largest));
          store_rows32(box, lane, gate, c0 + c * 32, ldc, rows, valid);
          store_rows32(box, lane, up, c0 + N + c * 32, ldc, rows, valid);
        } else if (!accumulate)
          store_rows32(box, lane, pack_row32(v), c0 + c * 32, ldc, rows, valid);
        else if (lane < rows)
          store_chunk<__nv_bfloat16>(c0 + size_t(lane) * ldc + c * 32, v, valid, true, nullptr);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_on_cta(tempty_bar(acc), 0);
    }
    if (KIND != PLAIN) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, o));
      if (lane == 0) amax[blockIdx.x * EPI_WARPS<KIND> + warp - 2] = largest;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// rows x cols one-byte matrix, row pitch ld bytes -> tensor map with (128 x box_rows) boxes, 128B swizzle
static int make_map_2d_u8(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                          uint32_t box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

// ------------------------------------------------------------------ abs-max -> scale, cast (+ transpose)
constexpr float E4M3_MAX = 448.f;
constexpr float E5M2_MAX = 57344.f;

constexpr int AMAX_BLOCKS = 1024;  // partial maxima (and the size of their buffer)

// partial[block] = max |x| over the block's share; four independent 16-byte loads in flight per thread
__global__ void __launch_bounds__(256) kf_absmax_bf16(const __nv_bfloat16* __restrict__ x, long long n, float* __restrict__ partial) {
  __shared__ float red[8];
  float m = 0.f;
  const long long n8 = n / 8, stride = (long long)gridDim.x * blockDim.x;
  const uint4* x8 = reinterpret_cast<const uint4*>(x);
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n8; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = x8[i + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) m = fmaxf(m, absmax8(v[u]));
  }
  for (; i < n8; i += stride) m = fmaxf(m, absmax8(x8[i]));
  if (blockIdx.x == 0)
    for (long long j = n8 * 8 + threadIdx.x; j < n; j += blockDim.x) m = fmaxf(m, fabsf(__bfloat162float(x[j])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w]);
    partial[blockIdx.x] = m;
  }
}

// fp8_max / max(largest of n partial maxima, tiny), in every thread of a block of 256
__device__ __forceinline__ float scale_of(const float* __restrict__ partial, int n, float fp8_max, float* red) {
  float m = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) m = fmaxf(m, partial[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) m = fmaxf(m, red[w]);
  return fp8_max / fmaxf(m, 1e-12f);
}
__global__ void __launch_bounds__(256) kf_scale_from_amax(const float* __restrict__ partial, int n, float* __restrict__ scale, float fp8_max) {
  __shared__ float red[8];
  const float s = scale_of(partial, n, fp8_max, red);
  if (threadIdx.x == 0) scale[0] = s;
}

template <bool E5M2>
__device__ __forceinline__ uint8_t to_fp8(float v) {
  return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, E5M2 ? __NV_E5M2 : __NV_E4M3);
}

// One 128 x 128 tile per block: reads bf16 x[rows][cols] (pitch ldx), writes the scaled fp8 copy row-major (out, pitch
// ld_out bytes, may be null) and transposed (out_t[cols][rows], pitch ld_t bytes, may be null).
// Memory-bound: 2 bytes in, 1 (or 2) bytes out per element.  16-byte loads, 8-byte row-major stores, 16-byte transposed
// stores, whole 128-byte lines on every side; the tile is transposed through shared memory as 4-byte words (word w of row
// r at w ^ 4 * (r / 16 % 8): the 32 lanes of a transposed read hit 32 different banks) and byte permutes.  The casts of an fp8
// 7B feed-forward over 2000 tokens took 145 us with 4-byte loads and byte-wise transposes, 88 us so (their maxima 60 -> 40).
//
// partial (optional): n partial maxima of |x|; every block makes the scale from them while its tile is under way, and the first one
// stores it for the products.  A kernel of one block in between was a launch and a drain: feed-forwards with their backward, of 240 rows
// x 4096 450 -> 422 us, of 2448 x 2048 449 -> 439, of 1008 x 4096 614 -> 610; over 2000 x 4096 no change (1067: the power limit).
template <bool E5M2>
__global__ void __launch_bounds__(256)
kf_cast_fp8(const __nv_bfloat16* __restrict__ x, int rows, int cols, long long ldx, const float* __restrict__ partial, int n,
            float* __restrict__ scale, uint8_t* __restrict__ out, long long ld_out, uint8_t* __restrict__ out_t, long long ld_t) {
  __shared__ uint32_t tile[128][32];
  __shared__ float red[8];
  const int r0 = blockIdx.y * 128, c0 = blockIdx.x * 128;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // 16 threads x 8 columns, 16 rows per step
  const int c = c0 + tx * 8;
  const bool wide_in = c + 7 < cols && (ldx & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const bool wide_out = c + 7 < cols && (ld_out & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
  uint4 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + ty + 16 * i;
    v[i] = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      const __nv_bfloat16* p = x + size_t(r) * ldx + c;
      if (wide_in) {
        v[i] = *reinterpret_cast<const uint4*>(p);
      } else {
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (c + e < cols) w[e >> 1] |= uint32_t(*reinterpret_cast<const unsigned short*>(p + e)) << (16 * (e & 1));
        v[i] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
  float s;
  if (partial != nullptr) {
    s = scale_of(partial, n, E5M2 ? E5M2_MAX : E4M3_MAX, red);
    if ((blockIdx.x | blockIdx.y | threadIdx.x) == 0) scale[0] = s;
  } else {
    s = scale[0];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rl = ty + 16 * i, r = r0 + rl;
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
    uint32_t q[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16(w[j]);
      q[j >> 1] |= (uint32_t(to_fp8<E5M2>(f.x * s)) | (uint32_t(to_fp8<E5M2>(f.y * s)) << 8)) << (16 * (j & 1));
    }
    if (out && r < rows) {
      uint8_t* o = out + size_t(r) * ld_out + c;
      if (wide_out) {
        *reinterpret_cast<uint2*>(o) = make_uint2(q[0], q[1]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (c + e < cols) o[e] = uint8_t(q[e >> 2] >> (8 * (e & 3)));
      }
    }
    if (out_t) *reinterpret_cast<uint2*>(&tile[rl][(tx * 2) ^ (((rl >> 4) & 7) << 2)]) = make_uint2(q[0], q[1]);
  }
  if (!out_t) return;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int rg = lane & 7, cg = (threadIdx.x >> 5) * 4 + (lane >> 3);  // 16 source rows x 4 source columns per thread
  uint32_t t[4][4];                                                     // [column][word of four rows]
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t a[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) a[j] = tile[rg * 16 + i * 4 + j][cg ^ (rg << 2)];
    // 4 x 4 byte transpose
    const uint32_t p0 = __byte_perm(a[0], a[1], 0x5140), p1 = __byte_perm(a[0], a[1], 0x7362);
    const uint32_t p2 = __byte_perm(a[2], a[3], 0x5140), p3 = __byte_perm(a[2], a[3], 0x7362);
    t[0][i] = __byte_perm(p0, p2, 0x5410);
    t[1][i] = __byte_perm(p0, p2, 0x7632);
    t[2][i] = __byte_perm(p1, p3, 0x5410);
    t[3][i] = __byte_perm(p1, p3, 0x7632);
  }
  const int r = r0 + rg * 16;
  const bool wide_t = r + 15 < rows && (ld_t & 15) == 0 && (reinterpret_cast<uintptr_t>(out_t) & 15) == 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int oc = c0 + cg * 4 + j;
    if (oc >= cols) continue;
    uint8_t* o = out_t + size_t(oc) * ld_t + r;
    if (wide_t) {
      *reinterpret_cast<uint4*>(o) = make_uint4(t[j][0], t[j][1], t[j][2], t[j][3]);
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e)
        if (r + e < rows) o[e] = uint8_t(t[j][e >> 2] >> (8 * (e & 3)));
    }
  }
}

// One product; rows of B: N, or 2N for SWIGLU.  With a SwiGLU: N a multiple of 16, G and its rows on 32 bytes.
template <int KIND>
static int launch(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, int ldc, int a_fmt, int b_fmt,
                  const void* scale_a, const void* scale_b, int accumulate, void* G, int ldg, void* amax, int* count, int num_sms,
                  void* stream, int* status) {
  if ((lda & 15) || (ldb & 15) || (ldc & 7) || (ldg & 7) || M <= 0 || N <= 0 || K <= 0) return 5;
  if (num_sms < 2 || (KIND != PLAIN && ((N & 15) || (ldg & 15) || (reinterpret_cast<uintptr_t>(G) & 31)))) return 5;
  const int b_rows = KIND == SWIGLU ? 2 * N : N;
  int pairs = num_sms / 2;
  const int tile_n = pair_tile_width(M, b_rows, pairs, nullptr);
  const int cols = KIND == SWIGLU ? tile_n / 2 : tile_n;
  CUtensorMap ma, mb;
  int rc = make_map_2d_u8(&ma, A, M, K, lda, CTA_M);
  if (rc) return 100 + rc;
  rc = make_map_2d_u8(&mb, B, b_rows, K, ldb, tile_n / 2);
  if (rc) return 200 + rc;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kf_gemm_fp8_tcgen05_2cta<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM<KIND>);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_set = true;
  }
  const int tiles = ((M + TILE_M - 1) / TILE_M) * ((N + cols - 1) / cols);
  if (tiles < pairs) pairs = tiles;
  if (count != nullptr) *count = pairs * 2 * EPI_WARPS<KIND>;
  kf_gemm_fp8_tcgen05_2cta<KIND><<<pairs * 2, THREADS<KIND>, SMEM<KIND>, (cudaStream_t)stream>>>(
      ma, mb, reinterpret_cast<__nv_bfloat16*>(C), M, N, K, ldc, accumulate, a_fmt, b_fmt, tile_n,
      reinterpret_cast<const float*>(scale_a), reinterpret_cast<const float*>(scale_b), reinterpret_cast<__nv_bfloat16*>(G), ldg,
      reinterpret_cast<float*>(amax), status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace f8
}  // namespace kf

extern "C" void* kf_status_device_ptr();

extern "C" {

// C[M,N] (+)= A8[M,K] * B8[N,K]^T / (scale_a * scale_b).  Pitches lda / ldb in bytes (multiples of 16),
// ldc in elements (multiple of 8).  a_fmt / b_fmt: 0 = e4m3, 1 = e5m2.  scale_* are device pointers.
int kf_gemm_fp8(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, int ldc,
                int a_fmt, int b_fmt, const void* scale_a, const void* scale_b, int accumulate, int num_sms,
                void* stream) {
  using namespace kf::f8;
  return launch<PLAIN>(A, B, C, M, N, K, lda, ldb, ldc, a_fmt, b_fmt, scale_a, scale_b, accumulate, nullptr, 0, nullptr, nullptr, num_sms,
                       stream, reinterpret_cast<int*>(kf_status_device_ptr()));
}

// H[M,F] = silu(gate) * up of [gate | up] = A8 * B8^T / (scale_a * scale_b), e4m3 operands, B8 = [gate ; up] (2F rows); partial[0 .. *count)
// = partial maxima of |H|, eight per SM at most.  GU[M,2F] (optional) receives the pre-activations.
int kf_gemm_fp8_swiglu(const void* A, const void* B, void* H, void* GU, int M, int F, int K, long long lda, long long ldb, int ldh, int ldgu,
                       const void* scale_a, const void* scale_b, void* partial, int* count, int num_sms, void* stream) {
  using namespace kf::f8;
  return launch<SWIGLU>(A, B, H, M, F, K, lda, ldb, ldh, 0, 0, scale_a, scale_b, 0, GU, ldgu, partial, count, num_sms, stream,
                        reinterpret_cast<int*>(kf_status_device_ptr()));
}

// DGU[M,2F] = SwiGLU'(GU) * (A8 * B8^T / (scale_a * scale_b)), A8 e5m2 (the incoming gradient), B8 e4m3 with F rows; partial and count
// as above, of |DGU|.
int kf_gemm_fp8_swiglu_bwd(const void* A, const void* B, const void* GU, void* DGU, int M, int F, int K, long long lda, long long ldb, int ldgu,
                           const void* scale_a, const void* scale_b, void* partial, int* count, int num_sms, void* stream) {
  using namespace kf::f8;
  return launch<SWIGLU_BWD>(A, B, DGU, M, F, K, lda, ldb, ldgu, 1, 0, scale_a, scale_b, 0, const_cast<void*>(GU), ldgu, partial, count,
                            num_sms, stream, reinterpret_cast<int*>(kf_status_device_ptr()));
}

// partial[0 .. *count) = partial maxima of |x| of n bf16 values; partial holds AMAX_BLOCKS (1024) floats.
int kf_fp8_absmax_bf16(const void* x, long long n, void* partial, int* count, void* stream) {
  using namespace kf::f8;
  long long blocks = (n / 8 + 1023) / 1024;  // four loads per thread before a block is added
  if (blocks < 1) blocks = 1;
  if (blocks > AMAX_BLOCKS) blocks = AMAX_BLOCKS;
  *count = (int)blocks;
  kf_absmax_bf16<<<(int)blocks, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const __nv_bfloat16*>(x), n,
                                                                reinterpret_cast<float*>(partial));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

// scale[0] = fp8_max / absmax(x) for n bf16 values; amax_scratch holds AMAX_BLOCKS (1024) floats.  For callers that want the scale
// itself (tests, benchmarks): the fp8 layers leave it to the cast, which makes it of the partial maxima.
int kf_fp8_scale_bf16(const void* x, long long n, int e5m2, void* amax_scratch, void* scale, void* stream) {
  using namespace kf::f8;
  int count = 0;
  if (const int rc = kf_fp8_absmax_bf16(x, n, amax_scratch, &count, stream)) return rc;
  kf_scale_from_amax<<<1, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const float*>(amax_scratch), count,
                                                          reinterpret_cast<float*>(scale), e5m2 ? E5M2_MAX : E4M3_MAX);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

// fp8(x * scale) row-major into out (optional) and transposed into out_t (optional).  With n > 0 the scale is fp8_max / the largest of
// partial[0 .. n), and is stored in scale[0]; else it is read there.
int kf_fp8_cast_bf16(const void* x, int rows, int cols, long long ldx, const void* partial, int n, void* scale, int e5m2, void* out,
                     long long ld_out, void* out_t, long long ld_t, void* stream) {
  using namespace kf::f8;
  auto pp = n > 0 ? reinterpret_cast<const float*>(partial) : nullptr;
  dim3 grid((cols + 127) / 128, (rows + 127) / 128);
  auto xp = reinterpret_cast<const __nv_bfloat16*>(x);
  auto sp = reinterpret_cast<float*>(scale);
  if (e5m2)
    kf_cast_fp8<true><<<grid, 256, 0, (cudaStream_t)stream>>>(xp, rows, cols, ldx, pp, n, sp, (uint8_t*)out, ld_out,
                                                              (uint8_t*)out_t, ld_t);
  else
    kf_cast_fp8<false><<<grid, 256, 0, (cudaStream_t)stream>>>(xp, rows, cols, ldx, pp, n, sp, (uint8_t*)out, ld_out,
                                                               (uint8_t*)out_t, ld_t);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // extern "C"
