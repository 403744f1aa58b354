// bf16 GEMM for few rows (decoding, short prompts):  out[M, N] = x[M, K] * W[N, K]^T  for M up to 256.
//
// What bounds it: every byte of W is read once and used for M rows only, so the kernel is a weight stream; the tensor
// cores are idle most of the time whatever the tile.  The tile kernels of gemm_tcgen05.cu give such a call
// ceil(N / 256) blocks (16 of 148 SMs for a 4096-wide projection), each with one 4-stage ring in flight.  Here
//   * the operands are swapped: 128 rows of W are the M side of the MMA, the tokens (padded to NT = 16 .. 256) its N
//     side, so nothing is computed for 128-row padding of x and the accumulator is NT columns of tensor memory;
//   * K is split over a thread-block cluster of up to 8 CTAs; the partial tiles meet in distributed shared memory and
//     are added in a fixed order (deterministic, fp32, no workspace, one launch);
//   * W may be up to three matrices stacked along N (q | k | v, gate | up): each has its own tensor map, so separate
//     Linear weights are read where they are instead of being concatenated first;
//   * the launch is programmatic: barriers, tensor memory and the first ring of W tiles are set up while the previous
//     kernel of the stream drains; x is read only after griddepcontrol.wait.  (Every kernel of this library that
//     triggers its dependents does so after its own wait, so when a block of this grid starts, all work before the
//     immediately preceding kernel is complete and visible; the caller asks for such a launch only where that kernel
//     itself writes no weights, see block_infer.cu.)
//
// With NORM the operand is RMSNorm(x) and x comes in as it is: the four epilogue warps, idle until the accumulator is done,
// compute each row's scale and write the normalised 64-column blocks into the ring, in the arithmetic and order of
// kf_rmsnorm_fwd (the same bits).  A norm kernel of its own is a link of 2 - 3 us in the chain of a generation step (wait,
// load, two block barriers, drain); up to NORM_ROWS rows every CTA repeats that work from L2 for less (a 7B block on one token
// 95.7 -> 92.0 us).
//
// Epilogues: 0 = (+ residual); 1 = SwiGLU over W = [gate ; up] (64 gate and the matching 64 up rows share a tile);
// 2 = rotary embedding of the q and k heads (64 or 128 wide) with k and v stored straight into the KV cache.
//
//   warp 0: TMA producer; warp 1: MMA issuer, owns TMEM; warps 2-5: accumulator -> shared memory; all: reduction + store
//
// Covers the Linear call sites of the reference during generation (kempnerforge/model/generate.py:66-131).
#include "skinny_args.cuh"

namespace kf {
namespace skinny {

constexpr int WROWS = 128;
constexpr int BK = 64;
constexpr int THREADS = 192;
constexpr int W_BYTES = WROWS * BK * 2;  // 16 KB
static_assert(NORM_ROWS <= 4, "a warp writes one ring stage: 8 lanes per row");

template <int NT>
struct Cfg {
  static constexpr int X_BYTES = NT * BK * 2;
  static constexpr int STAGE = W_BYTES + X_BYTES;
  // two CTAs per SM up to 64 tokens (about 100 KB of ring each), one above
  static constexpr int STAGES = NT <= 16 ? 6 : NT <= 32 ? 5 : NT <= 64 ? 4 : NT <= 128 ? 6 : 4;
  static constexpr int RED_BYTES = NT * WROWS * 4;  // reduction buffer, aliases the ring
  static constexpr int BODY = STAGES * STAGE > RED_BYTES ? STAGES * STAGE : RED_BYTES;
  static constexpr size_t SMEM = size_t(BODY) + 1024 + 256;
};

__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <int NT, int EPI, bool NORM>
__global__ void __launch_bounds__(THREADS)
kf_gemm_skinny(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
               const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_w2,
               const __grid_constant__ Args a, int* status) {
  using C = Cfg<NT>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + C::BODY;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (C::STAGES + s); };
  const uint32_t acc_bar = bar_base + 8u * (2 * C::STAGES);
  const uint32_t tmem_slot = bar_base + 8u * (2 * C::STAGES + 1);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  float* norm_red = reinterpret_cast<float*>(smem_raw + (bar_base + 128 - smem_u32(smem_raw)));  // [NORM_ROWS][8]
  static_assert(8 * (2 * C::STAGES + 1) + 4 <= 128 && NORM_ROWS * 8 * 4 <= 128, "barriers, then the partial sums");
  float* red = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));
  constexpr int TMEM_COLS = NT < 32 ? 32 : NT;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int splits = int(cluster_nctaid()), rank = int(cluster_ctarank());
  const int tile = int(blockIdx.x) / splits;
  const int k_blocks = (a.K + BK - 1) / BK;
  const int kb0 = k_blocks * rank / splits, kb1 = k_blocks * (rank + 1) / splits;
  const int n_kb = kb1 - kb0;
  int seg = 0;
  if (EPI != 1) {
    if (a.n_seg > 1 && tile >= a.tile0[1]) seg = 1;
    if (a.n_seg > 2 && tile >= a.tile0[2]) seg = 2;
  }
  const int row0 = (tile - (EPI == 1 ? 0 : a.tile0[seg])) * (EPI == 1 ? 64 : WROWS);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), NORM ? 2 : 1);  // NORM: and the warp that wrote the x block
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_bar, 1);
    mbar_fence_init();
    if (!NORM) tma_prefetch_desc(&map_x);
    tma_prefetch_desc(seg == 0 ? &map_w0 : seg == 1 ? &map_w1 : &map_w2);
    if (EPI == 1) tma_prefetch_desc(&map_w1);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  bool ok = true;
  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      auto load_w = [&](int i) {
        const int s = i % C::STAGES, k0 = (kb0 + i) * BK;
        const uint32_t dst = smem_base + s * C::STAGE;
        mbar_expect_tx(full_bar(s), NORM ? W_BYTES : C::STAGE);
        if (EPI == 1) {
          tma_load_2d(dst, &map_w0, full_bar(s), k0, row0);
          tma_load_2d(dst + W_BYTES / 2, &map_w1, full_bar(s), k0, row0);
        } else {
          tma_load_2d(dst, seg == 0 ? &map_w0 : seg == 1 ? &map_w1 : &map_w2, full_bar(s), k0, row0);
        }
      };
      auto load_x = [&](int i) {
        const int s = i % C::STAGES;
        tma_load_2d(smem_base + s * C::STAGE + W_BYTES, &map_x, full_bar(s), (kb0 + i) * BK, 0);
      };
      const int pre = min(n_kb, C::STAGES);
      if (a.pdl == PDL_WAIT_FIRST) grid_dep_wait();
      for (int i = 0; i < pre; ++i) load_w(i);
      if (!NORM) {
        grid_dep_wait();
        for (int i = 0; i < pre; ++i) load_x(i);
      }
      int i = pre;
      for (; i < n_kb; ++i) {
        const int s = i % C::STAGES;
        if (!mbar_wait(empty_bar(s), ((i / C::STAGES) - 1) & 1, status, KF_ERR_WAIT_EMPTY)) { ok = false; break; }
        load_w(i);
        if (!NORM) load_x(i);
      }
      // on the error path nobody consumes the stages: wait for the copies still landing in this CTA's shared memory
      if (!ok)
        for (int j = max(0, i - C::STAGES); j < i; ++j)
          mbar_wait(full_bar(j % C::STAGES), (j / C::STAGES) & 1, status, KF_ERR_WAIT_DRAIN);
    }
    __syncwarp();
    grid_dep_wait();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(WROWS, NT, false, false);
      for (int i = 0; i < n_kb; ++i) {
        const int s = i % C::STAGES;
        if (!mbar_wait(full_bar(s), (i / C::STAGES) & 1, status, KF_ERR_WAIT_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t w_src = smem_base + s * C::STAGE, x_src = w_src + W_BYTES;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          tc_mma_f16(tmem_base, umma_desc_sw128(w_src + k * 32, 16, 1024), umma_desc_sw128(x_src + k * 32, 16, 1024),
                     idesc, (i | k) != 0);
        tc_commit(empty_bar(s));
      }
      tc_commit(acc_bar);  // every MMA has retired: the accumulator is final, the ring is free
      if (!ok) mbar_wait(acc_bar, 0, status, KF_ERR_WAIT_DRAIN);
    }
    __syncwarp();
    grid_dep_wait();
  } else {
    // ------------------------------------------------------------ accumulator -> reduction buffer [token][W row]
    const int quarter = warp & 3;
    grid_dep_wait();
    if constexpr (NORM) {
      const int t = threadIdx.x - 64, nvec = a.K >> 3;  // threads t and t + 128 of the norm kernel's 256
      for (int r = 0; r < a.M; ++r) {
        const __nv_bfloat16* xr = a.x + size_t(r) * a.ldx;
        float ss[2] = {0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; ++h)
          for (int v = t + 128 * h; v < nvec; v += 256) add_squares(*reinterpret_cast<const uint4*>(xr + v * 8), ss[h]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ss[h] = norm_warp_sum(ss[h]);
          if (lane == 0) norm_red[r * 8 + (t >> 5) + 4 * h] = ss[h];
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const int r = lane >> 3, ch = lane & 7;  // this lane's row and 16-byte chunk of a block
      float rstd = 0.f;
      for (int i = 0; i < a.M; ++i) {
        const float ri = norm_rstd(norm_red + i * 8, lane, a.K, a.eps);
        if (i == r) rstd = ri;
      }
      const __nv_bfloat16* xr = a.x + size_t(r < a.M ? r : 0) * a.ldx;
      for (int i = t >> 5; i < n_kb; i += 4) {
        const int s = i % C::STAGES, col = (kb0 + i) * BK + ch * 8;
        uint4 u = make_uint4(0, 0, 0, 0);
        if (r < a.M && col < a.K)
          u = norm_vec(*reinterpret_cast<const uint4*>(xr + col), *reinterpret_cast<const uint4*>(a.gain + col), rstd);
        if (i >= C::STAGES && !mbar_wait(empty_bar(s), ((i / C::STAGES) - 1) & 1, status, KF_ERR_WAIT_EMPTY)) break;
        if (r < a.M) {  // rows past M feed accumulator columns that nobody reads
          const uint32_t dst = smem_base + s * C::STAGE + W_BYTES + uint32_t(r * 128 + ((ch ^ (r & 7)) << 4));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w) : "memory");
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full_bar(s));
      }
    }
    ok = mbar_wait(acc_bar, 0, status, KF_ERR_WAIT_TMEM_FULL);
    tc_fence_after();
    const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16);
    float* dst = red + quarter * 32 + lane;
#pragma unroll 1
    for (int c = 0; c < (NT + 31) / 32; ++c) {
      if (c * 32 >= a.M) break;
      if constexpr (NT == 16) {
        uint32_t v[16];
        tmem_ld_32x16(t_row, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i < a.M) dst[i * WROWS] = __uint_as_float(v[i]);
      } else {
        uint32_t v[32];
        tmem_ld_32x32(t_row + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (c * 32 + i < a.M) dst[(c * 32 + i) * WROWS] = __uint_as_float(v[i]);
      }
    }
  }
  tc_fence_before();
  cluster_sync_all();  // partial tiles of every split are in shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  grid_dep_launch();

  // ------------------------------------------------------------ sum over the splits (fixed order), epilogue, store
  const uint32_t red_addr = smem_base;
  auto sum8 = [&](int t, int n, float (&f)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = 0.f;
    const uint32_t off = red_addr + uint32_t(t * WROWS + n) * 4u;
#pragma unroll 1
    for (int r = 0; r < splits; ++r) {
      const uint32_t src = mapa_shared(off, r);
      const float4 u = ld_cluster_f4(src), v = ld_cluster_f4(src + 16);
      f[0] += u.x; f[1] += u.y; f[2] += u.z; f[3] += u.w;
      f[4] += v.x; f[5] += v.y; f[6] += v.z; f[7] += v.w;
    }
  };
  auto store8 = [&](__nv_bfloat16* p, const float (&f)[8]) {
    uint4 u;
    u.x = pack_bf16(f[0], f[1]);
    u.y = pack_bf16(f[2], f[3]);
    u.z = pack_bf16(f[4], f[5]);
    u.w = pack_bf16(f[6], f[7]);
    *reinterpret_cast<uint4*>(p) = u;
  };
  const int first = rank * THREADS + threadIdx.x, step = splits * THREADS;
  if constexpr (EPI == 0) {
    const int valid = min(WROWS, a.rows[seg] - row0);
    for (int i = first; i < a.M * (WROWS / 8); i += step) {
      const int t = i / (WROWS / 8), n = (i % (WROWS / 8)) * 8;
      if (n >= valid) continue;
      float f[8];
      sum8(t, n, f);
      const int col = a.col[seg] + row0 + n;
      if (a.residual) {
        if (a.round_first)
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __bfloat162float(__float2bfloat16(f[e]));
        const uint4 o = *reinterpret_cast<const uint4*>(a.residual + size_t(t) * a.ldr + col);
        const float2 p = unpack_bf16(o.x), q = unpack_bf16(o.y), r = unpack_bf16(o.z), s = unpack_bf16(o.w);
        f[0] += p.x; f[1] += p.y; f[2] += q.x; f[3] += q.y;
        f[4] += r.x; f[5] += r.y; f[6] += s.x; f[7] += s.y;
      }
      store8(a.out + size_t(t) * a.ldo + col, f);
    }
  } else if constexpr (EPI == 1) {
    const int valid = min(64, a.rows[0] - row0);
    for (int i = first; i < a.M * 8; i += step) {
      const int t = i >> 3, n = (i & 7) * 8;
      if (n >= valid) continue;
      float g[8], u[8];
      sum8(t, n, g);
      sum8(t, 64 + n, u);
#pragma unroll
      for (int e = 0; e < 8; ++e) {  // the activation sees bf16 pre-activations, like the large-M epilogue
        const float gf = __bfloat162float(__float2bfloat16(g[e])), uf = __bfloat162float(__float2bfloat16(u[e]));
        g[e] = gf / (1.f + __expf(-gf)) * uf;
      }
      store8(a.out + size_t(t) * a.ldo + row0 + n, g);
    }
  } else {
    // one head of 128 columns or two of 64 per tile: pairs (n, n + half).  Tokens t = (batch, new position).
    const int half = a.hd >> 1, vec = half >> 3;  // 8-wide pieces of a half head; 8 pairs of pieces per token and tile
    for (int i = first; i < a.M * 8; i += step) {
      const int t = i >> 3, head = (i & 7) / vec, m = (i & 7) % vec * 8, n = head * a.hd + m;
      const int b = t / a.S, pos = t - b * a.S;
      if (row0 + n >= a.rows[seg]) continue;
      float lo[8], hi[8];
      sum8(t, n, lo);
      sum8(t, n + half, hi);
      if (seg < 2) {
        const float* cs = a.cosT + size_t(pos) * half + m;
        const float* sn = a.sinT + size_t(pos) * half + m;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          // the projection is rounded to bf16 before the rotation, like the separate kernels do
          const float x = __bfloat162float(__float2bfloat16(lo[e])), y = __bfloat162float(__float2bfloat16(hi[e]));
          rotate_pair_step(a.hd, x, y, cs[e], sn[e], lo[e], hi[e]);
        }
      }
      __nv_bfloat16* p = seg == 0 ? a.out + size_t(t) * a.ldo + row0 + n
                                  : (seg == 1 ? a.kc : a.vc) + size_t(b) * a.cache_batch + size_t(pos) * a.kv_cols + row0 + n;
      store8(p, lo);
      store8(p + half, hi);
    }
  }
  cluster_sync_all();  // the buffers stay valid until every CTA of the cluster has read them
}

// Number of CTAs a K range is split over: enough of them to fill the SMs, at least MIN_KB ring steps each.  Weights of less
// than 8 MB (512 blocks of 128 x 64) are not split, so that the projections of small models sum over K in the order of the tile
// kernels and keep their bits: in a model of a few layers every rounding travels on, and one that falls differently moves the
// logits by as much as all of them together are off.  That costs time (one row, L2 flushed, unsplit / split: 768 x 768 7.0 / 5.6
// us, 2304 x 768 7.3 / 6.1, 768 x 2048 12.7 / 6.6, 1024 x 3072 17.6 / 7.9), which gemm_small.cu gets back for up to 16 rows.
static bool small_weight(int tiles, int k_blocks) { return tiles * k_blocks < 512; }

static int pick_splits(int tiles, int k_blocks, int num_sms, int per_sm) {
  constexpr int MIN_KB = 4;
  if (small_weight(tiles, k_blocks)) return 1;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= num_sms * per_sm && k_blocks >= 2 * s * MIN_KB) s *= 2;
  return s;
}

template <int NT, int EPI, bool NORM = false>
static int launch(const CUtensorMap& mx, const CUtensorMap (&mw)[3], const Args& a, int tiles, int num_sms, int* status,
                  cudaStream_t stream) {
  using C = Cfg<NT>;
  auto kern = kf_gemm_skinny<NT, EPI, NORM>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 16 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_set[dev] = true;
  }
  const int splits = pick_splits(tiles, (a.K + BK - 1) / BK, num_sms, NT <= 64 ? 2 : 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * splits));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, mx, mw[0], mw[1], mw[2], a, status);
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

template <int EPI>
static int dispatch(const void* x, int ldx, const void* const* w, const int* ldw, Args& a, int tiles, int num_sms,
                    int* status, cudaStream_t stream) {
  const int nt = a.M <= 16 ? 16 : a.M <= 32 ? 32 : a.M <= 64 ? 64 : a.M <= 128 ? 128 : 256;
  CUtensorMap mx, mw[3];
  int rc = 0;
  a.x = (const __nv_bfloat16*)x;
  a.ldx = ldx;
  if (a.gain && a.M > NORM_ROWS) return 5;
  // the bulk copies of the small kernel and the vector loads of the norm need what the encoding of a tensor map checks by itself
  auto off16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  if (off16(x) || off16(a.gain)) return 101;
  for (int i = 0; i < a.n_seg; ++i)
    if (off16(w[i])) return 201;
  if (small_fits(a, EPI, small_weight(tiles, (a.K + BK - 1) / BK), num_sms)) return run_small(EPI, w, ldw, a, status, stream);
  if (!a.gain) rc = make_map_2d_bf16(&mx, x, a.M, a.K, ldx, BK, nt);
  if (rc) return 100 + rc;
  for (int i = 0; i < a.n_seg; ++i) {
    rc = make_map_2d_bf16(&mw[i], w[i], a.rows[i], a.K, ldw[i], BK, EPI == 1 ? 64 : WROWS);
    if (rc) return 200 + rc;
  }
  for (int i = a.n_seg; i < 3; ++i) mw[i] = mw[0];  // never read
  if constexpr (EPI != 0) {
    if (a.gain) return launch<16, EPI, true>(mw[0], mw, a, tiles, num_sms, status, stream);
  }
  switch (nt) {
    case 16: return launch<16, EPI>(mx, mw, a, tiles, num_sms, status, stream);
    case 32: return launch<32, EPI>(mx, mw, a, tiles, num_sms, status, stream);
    case 64: return launch<64, EPI>(mx, mw, a, tiles, num_sms, status, stream);
    case 128: return launch<128, EPI>(mx, mw, a, tiles, num_sms, status, stream);
    default: return launch<256, EPI>(mx, mw, a, tiles, num_sms, status, stream);
  }
}

}  // namespace skinny
}  // namespace kf

extern "C" void* kf_status_device_ptr();

extern "C" {

// out[M, sum rows] = x W^T (+ residual), W = up to three [rows_i][K] matrices stacked along the output; 1 <= M <= 256.
// round_first: the product is rounded to bf16 before the residual is added (the arithmetic of a projection and an addition in
// two kernels, which keeps a whole model's logits with those of the op-by-op path); otherwise the sum is rounded once.
// All pitches in elements, multiples of 8; rows_i and K multiples of 8; bases 16-byte aligned.
int kf_gemm_skinny_bf16(const void* x, const void* w0, const void* w1, const void* w2, void* out, const void* residual,
                        int M, int K, int n0, int n1, int n2, int ldx, int ldw0, int ldw1, int ldw2, int ldo, int ldr,
                        int round_first, int pdl, int num_sms, void* stream) {
  using namespace kf::skinny;
  if (M < 1 || M > 256 || K < 8 || n0 < 8 || ((K | n0 | n1 | n2 | ldx | ldw0 | ldw1 | ldw2 | ldo | (residual ? ldr : 0)) & 7))
    return 5;
  const void* w[3] = {w0, w1, w2};
  const int ldw[3] = {ldw0, ldw1, ldw2}, n[3] = {n0, n1, n2};
  Args a{};
  a.out = (__nv_bfloat16*)out;
  a.residual = (const __nv_bfloat16*)residual;
  a.M = M; a.K = K; a.ldo = ldo; a.ldr = ldr; a.pdl = pdl;
  a.round_first = round_first;
  int tiles = 0, col = 0;
  for (a.n_seg = 0; a.n_seg < 3 && w[a.n_seg] && n[a.n_seg] > 0; ++a.n_seg) {
    a.tile0[a.n_seg] = tiles;
    a.rows[a.n_seg] = n[a.n_seg];
    a.col[a.n_seg] = col;
    tiles += (n[a.n_seg] + WROWS - 1) / WROWS;
    col += n[a.n_seg];
  }
  return dispatch<0>(x, ldx, w, ldw, a, tiles, num_sms, (int*)kf_status_device_ptr(), (cudaStream_t)stream);
}

// Rows up to which kf_gemm_skinny_norm_* take the norm of their input along.
int kf_skinny_norm_rows() { return kf::skinny::NORM_ROWS; }

// h[M, F] = silu(n Wg^T) * (n Wu^T); 1 <= M <= 256.  gain null: n = x; else n = RMSNorm(x) with it, M <= kf_skinny_norm_rows().
int kf_gemm_skinny_norm_swiglu_bf16(const void* x, const void* gain, float eps, const void* wg, const void* wu, void* h, int M,
                                    int F, int K, int ldx, int ldwg, int ldwu, int ldh, int pdl, int num_sms, void* stream) {
  using namespace kf::skinny;
  if (M < 1 || M > 256 || K < 8 || F < 8 || ((K | F | ldx | ldwg | ldwu | ldh) & 7)) return 5;
  const void* w[3] = {wg, wu, nullptr};
  const int ldw[3] = {ldwg, ldwu, 0};
  Args a{};
  a.out = (__nv_bfloat16*)h;
  a.M = M; a.K = K; a.ldo = ldh; a.pdl = pdl;
  a.gain = (const __nv_bfloat16*)gain;
  a.eps = eps;
  a.n_seg = 2;
  a.rows[0] = a.rows[1] = F;
  return dispatch<1>(x, ldx, w, ldw, a, (F + 63) / 64, num_sms, (int*)kf_status_device_ptr(), (cudaStream_t)stream);
}

int kf_gemm_skinny_swiglu_bf16(const void* x, const void* wg, const void* wu, void* h, int M, int F, int K, int ldx,
                               int ldwg, int ldwu, int ldh, int pdl, int num_sms, void* stream) {
  return kf_gemm_skinny_norm_swiglu_bf16(x, nullptr, 0.f, wg, wu, h, M, F, K, ldx, ldwg, ldwu, ldh, pdl, num_sms, stream);
}

// Fused q | k | v projection of M = B * S new tokens with the rotary embedding: q (rotated) -> q_out [M][ldq], k (rotated)
// and v -> cache rows kc / vc ([B][..][kv_cols], `cache_batch` elements between batch entries, pointing at the first new
// position).  cosT / sinT: fp32 [S][hd / 2] of the new positions.  hd 64 or 128; q_cols and kv_cols multiples of it.
// gain null: of x itself; else of RMSNorm(x) with it, M <= kf_skinny_norm_rows().
int kf_gemm_skinny_norm_qkv_bf16(const void* x, const void* gain, float eps, const void* wq, const void* wk, const void* wv,
                                 void* q_out, void* kc, void* vc, int M, int S, int K, int q_cols, int kv_cols, int hd, int ldx,
                                 int ldwq, int ldwk, int ldwv, int ldq, long long cache_batch, const void* cosT,
                                 const void* sinT, int pdl, int num_sms, void* stream) {
  using namespace kf::skinny;
  if ((hd != 64 && hd != 128) || M < 1 || M > 256 || S < 1 || M % S || K < 8 || ((K | ldx | ldwq | ldwk | ldwv | ldq) & 7) ||
      (cache_batch & 7) || q_cols % hd || kv_cols % hd || q_cols < hd || kv_cols < hd)
    return 5;
  const void* w[3] = {wq, wk, wv};
  const int ldw[3] = {ldwq, ldwk, ldwv}, n[3] = {q_cols, kv_cols, kv_cols};
  Args a{};
  a.out = (__nv_bfloat16*)q_out;
  a.M = M; a.K = K; a.ldo = ldq; a.pdl = pdl;
  a.kc = (__nv_bfloat16*)kc;
  a.vc = (__nv_bfloat16*)vc;
  a.cache_batch = cache_batch;
  a.cosT = (const float*)cosT;
  a.sinT = (const float*)sinT;
  a.S = S; a.kv_cols = kv_cols; a.hd = hd;
  a.gain = (const __nv_bfloat16*)gain;
  a.eps = eps;
  int tiles = 0;
  for (a.n_seg = 0; a.n_seg < 3; ++a.n_seg) {
    a.tile0[a.n_seg] = tiles;
    a.rows[a.n_seg] = n[a.n_seg];
    tiles += (n[a.n_seg] + WROWS - 1) / WROWS;
  }
  return dispatch<2>(x, ldx, w, ldw, a, tiles, num_sms, (int*)kf_status_device_ptr(), (cudaStream_t)stream);
}

}  // extern "C"
