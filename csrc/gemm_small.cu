// bf16 GEMM for up to 16 rows against a small weight (less than 8 MB):  out[M, N] = x[M, K] * W[N, K]^T.
//
// What bounds it: latency.  Such a weight is read in a few microseconds by all SMs together, and its sums over K stay in one
// piece (pick_splits in gemm_skinny_tcgen05.cu says why), so a generation step of a small model is a chain of K / 16 dependent
// MMAs after another.  One tcgen05.mma that adds to the accumulator of the one before it takes 70 ns at 16 columns, whatever
// the rows; mma.sync m16n8k16 takes a quarter of that and gives the same fp32 bits (compared with the tile kernels over K from
// 16 to 4800).  Hence
//   * a CTA owns 16 rows of W: the m16n8k16 tile of one warp, up to two of them for up to 16 tokens;
//   * the CTA's whole strip of W (16 rows; beside x it has room for K up to 4800 with 8 rows of x, 3616 with 16) is requested with
//     one bulk copy per row before the previous kernel of the stream has finished (a programmatic launch: only behind a kernel
//     that writes no weights and no gain, see block_infer.cu), so that only x, the chain and the store remain behind it;
//   * the accumulator of a thread holds rows g and g + 8 of the tile, which are made gate and up of one hidden unit, or the two
//     halves of a rotary pair: no exchange before the epilogue;
//   * optionally the norm of x is taken along, in the arithmetic and order of kf_rmsnorm_fwd (the same bits).
// One row, repeated launches, us, this kernel / the weight-streaming kernel unsplit: 768 x 768 3.4 / 7.1, 768 x 2048 5.2 / 12.7,
// 768 x 3072 6.6 / 17.3.  A block of the 125M model on one token (five kernels): 45 -> 18 us on the device.
//
// Epilogues as in gemm_skinny_tcgen05.cu: 0 = (+ residual), 1 = SwiGLU, 2 = rotary embedding with k and v into the cache.
#include "skinny_args.cuh"

namespace kf {
namespace skinny {

constexpr int SMALL_THREADS = 128;
constexpr int SMALL_ROWS = 16;   // rows of W per CTA

__device__ __forceinline__ void bulk_row(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Rows of W and x lie 16 bytes further apart than they are long: no bank conflicts for ldmatrix.
__host__ __device__ constexpr size_t small_smem(int K, int nt, bool norm) {
  return size_t(SMALL_ROWS + 8 * nt) * (2 * K + 16) + (norm ? 2 * size_t(K) : 0) + 16 + NORM_ROWS * 8 * 4;
}

struct SmallWeights {
  const __nv_bfloat16* w[3];
  int ldw[3];
};

template <int EPI, bool NORM, int NT>
__global__ void __launch_bounds__(SMALL_THREADS)
kf_gemm_small(const __grid_constant__ SmallWeights sw, const __grid_constant__ Args a, int* status) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int K = a.K, pitch = 2 * K + 16;
  const uint32_t w_smem = smem_u32(smem_raw), x_smem = w_smem + SMALL_ROWS * pitch, g_smem = x_smem + 8 * NT * pitch;
  uint8_t* x_gen = smem_raw + SMALL_ROWS * pitch;
  const uint8_t* g_gen = x_gen + 8 * NT * pitch;
  const uint32_t w_bar = g_smem + (NORM ? 2 * K : 0), x_bar = w_bar + 8;
  float* red = reinterpret_cast<float*>(smem_raw + (x_bar + 8 - w_smem));  // [NORM_ROWS][8]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // the tile's first and second eight rows of their matrices
  const int tile = blockIdx.x;
  int seg = 0;
  if (EPI != 1) {
    if (a.n_seg > 1 && tile >= a.tile0[1]) seg = 1;
    if (a.n_seg > 2 && tile >= a.tile0[2]) seg = 2;
  }
  const int j = tile - (EPI == 1 ? 0 : a.tile0[seg]);
  int r_lo, r_hi, m0 = 0;
  if (EPI == 0) {
    r_lo = j * SMALL_ROWS;
    r_hi = r_lo + 8;
  } else if (EPI == 1) {
    r_lo = r_hi = j * 8;
  } else {
    const int half = a.hd >> 1, per_head = half >> 3;
    m0 = j % per_head * 8;
    r_lo = j / per_head * a.hd + m0;
    r_hi = r_lo + half;
  }
  const int seg_hi = EPI == 1 ? 1 : seg;
  const bool has_hi = r_hi < a.rows[seg_hi];

  if (tid == 0) {
    mbar_init(w_bar, 1);
    mbar_init(x_bar, 1);
    mbar_fence_init();
    if (a.pdl == PDL_WAIT_FIRST) grid_dep_wait();
    mbar_expect_tx(w_bar, uint32_t(has_hi ? 16 : 8) * 2 * K + (NORM ? 2 * K : 0));
    for (int r = 0; r < 8; ++r)
      bulk_row(w_smem + r * pitch, sw.w[seg] + size_t(r_lo + r) * sw.ldw[seg], 2 * K, w_bar);
    if (has_hi)
      for (int r = 0; r < 8; ++r)
        bulk_row(w_smem + (8 + r) * pitch, sw.w[seg_hi] + size_t(r_hi + r) * sw.ldw[seg_hi], 2 * K, w_bar);
    if (NORM) bulk_row(g_smem, a.gain, 2 * K, w_bar);
  }
  const int g = lane >> 2, t2 = (lane & 3) * 2;  // this thread's rows g and g + 8, tokens nt * 8 + t2 and t2 + 1
  __syncthreads();
  grid_dep_wait();
  grid_dep_launch();
  if (tid == 0) {
    mbar_expect_tx(x_bar, uint32_t(a.M) * 2 * K);
    for (int r = 0; r < a.M; ++r) bulk_row(x_smem + r * pitch, a.x + size_t(r) * a.ldx, 2 * K, x_bar);
  }
  float cs[NT][2], sn[NT][2];
  if (EPI == 2 && warp == 0 && seg < 2) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int tok = nt * 8 + t2 + e;
        const size_t at = tok < a.M ? size_t(tok % a.S) * (a.hd >> 1) + m0 + g : 0;
        cs[nt][e] = a.cosT[at];
        sn[nt][e] = a.sinT[at];
      }
  }
  float res[NT][4];
  if (EPI == 0 && warp == 0 && a.residual) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int tok = nt * 8 + t2 + (e & 1);
        const bool in = tok < a.M && (e < 2 || has_hi);
        const int col = a.col[seg] + (e < 2 ? r_lo : r_hi) + g;
        res[nt][e] = in ? __bfloat162float(a.residual[size_t(tok) * a.ldr + col]) : 0.f;
      }
  }
  bool ok = mbar_wait(x_bar, 0, status, KF_ERR_WAIT_FULL);
  if constexpr (NORM) {
    const int nvec = K >> 3;
    for (int r = 0; r < a.M; ++r) {  // threads t and t + 128 of the norm kernel's 256
      float ss[2] = {0.f, 0.f};
#pragma unroll
      for (int h = 0; h < 2; ++h)
        for (int v = tid + 128 * h; v < nvec; v += 256) add_squares(*reinterpret_cast<const uint4*>(x_gen + r * pitch + v * 16), ss[h]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ss[h] = norm_warp_sum(ss[h]);
        if (lane == 0) red[r * 8 + warp + 4 * h] = ss[h];
      }
    }
    ok = mbar_wait(w_bar, 0, status, KF_ERR_WAIT_FULL) && ok;  // the gain
    __syncthreads();
    for (int r = 0; r < a.M; ++r) {
      const float rstd = norm_rstd(red + r * 8, lane, K, a.eps);
      for (int v = tid; v < nvec; v += SMALL_THREADS) {
        uint4* p = reinterpret_cast<uint4*>(x_gen + r * pitch + v * 16);
        *p = norm_vec(*p, *reinterpret_cast<const uint4*>(g_gen + v * 16), rstd);
      }
    }
    __syncthreads();
  }
  // No thread leaves while copies are still landing: every thread has waited for x, the first warp also waits for W.
  if (warp != 0) return;
  ok = mbar_wait(w_bar, 0, status, KF_ERR_WAIT_FULL) && ok;
  if (!ok) {
    mbar_wait(x_bar, 0, status, KF_ERR_WAIT_DRAIN);
    mbar_wait(w_bar, 0, status, KF_ERR_WAIT_DRAIN);
    return;
  }

  float d[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) d[nt][0] = d[nt][1] = d[nt][2] = d[nt][3] = 0.f;
  const int mi = lane >> 3, lr = lane & 7;
  const uint32_t a_addr = w_smem + uint32_t((lr + (mi & 1) * 8) * pitch + (mi >> 1) * 16);
  const uint32_t b_addr = x_smem + uint32_t(lr * pitch + mi * 16);
#pragma unroll 4
  for (int k = 0; k < K; k += 32) {
    uint32_t a0[4], a1[4];
    ldsm4(a_addr + k * 2, a0);
    ldsm4(a_addr + k * 2 + 32, a1);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      uint32_t b[4];
      ldsm4(b_addr + nt * 8 * pitch + k * 2, b);
      mma16816(d[nt], a0, b[0], b[1]);
      mma16816(d[nt], a1, b[2], b[3]);
    }
  }

#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int tok = nt * 8 + t2 + e;
      if (tok >= a.M) continue;
      float lo = d[nt][e], hi = d[nt][2 + e];
      if (EPI == 0) {
        if (a.residual) {
          if (a.round_first) {
            lo = __bfloat162float(__float2bfloat16(lo));
            hi = __bfloat162float(__float2bfloat16(hi));
          }
          lo += res[nt][e];
          hi += res[nt][2 + e];
        }
        __nv_bfloat16* p = a.out + size_t(tok) * a.ldo + a.col[seg] + g;
        p[r_lo] = __float2bfloat16(lo);
        if (has_hi) p[r_hi] = __float2bfloat16(hi);
      } else {
        lo = __bfloat162float(__float2bfloat16(lo));
        hi = __bfloat162float(__float2bfloat16(hi));
        if (EPI == 1) {
          a.out[size_t(tok) * a.ldo + r_lo + g] = __float2bfloat16(lo / (1.f + __expf(-lo)) * hi);
        } else {
          if (seg < 2) rotate_pair_step(a.hd, lo, hi, cs[nt][e], sn[nt][e], lo, hi);
          const int b = tok / a.S, pos = tok - b * a.S;
          __nv_bfloat16* p = seg == 0 ? a.out + size_t(tok) * a.ldo
                                      : (seg == 1 ? a.kc : a.vc) + size_t(b) * a.cache_batch + size_t(pos) * a.kv_cols;
          p[r_lo + g] = __float2bfloat16(lo);
          p[r_hi + g] = __float2bfloat16(hi);
        }
      }
    }
}

template <int EPI, bool NORM, int NT>
static int launch_small(const SmallWeights& sw, const Args& a, int tiles, int* status, cudaStream_t stream) {
  auto kern = kf_gemm_small<EPI, NORM, NT>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return 300 + (int)e;
    if (dev < 16) attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles);
  cfg.blockDim = dim3(SMALL_THREADS);
  cfg.dynamicSmemBytes = small_smem(a.K, NT, NORM);
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = a.pdl ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, sw, a, status);
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

// Up to 16 rows, sums that stay in one piece, and all CTAs resident at once: their strips in shared memory (1 KB per CTA is the
// system's), their threads within the 2048 of an SM.
bool small_fits(const Args& a, int epi, bool one_piece, int num_sms) {
  if (a.M > 16 || a.K % 32 || !one_piece) return false;
  const size_t smem = small_smem(a.K, (a.M + 7) / 8, a.gain != nullptr);
  int tiles = 0;
  for (int i = 0; i < a.n_seg; ++i) tiles += (a.rows[i] + SMALL_ROWS - 1) / SMALL_ROWS;
  return smem <= 232448 && tiles <= num_sms * min(int(233472 / (smem + 1024)), 2048 / SMALL_THREADS);
}

int run_small(int epi, const void* const* w, const int* ldw, Args& a, int* status, cudaStream_t stream) {
  SmallWeights sw{};
  for (int i = 0; i < a.n_seg; ++i) {
    sw.w[i] = (const __nv_bfloat16*)w[i];
    sw.ldw[i] = ldw[i];
  }
  int tiles = 0;
  for (int i = 0; i < (epi == 1 ? 1 : a.n_seg); ++i) {
    a.tile0[i] = tiles;
    tiles += epi == 1 ? a.rows[0] / 8 : (a.rows[i] + SMALL_ROWS - 1) / SMALL_ROWS;
  }
  const bool two = a.M > 8;
#define KF_SMALL(E, N_) return two ? launch_small<E, N_, 2>(sw, a, tiles, status, stream) : launch_small<E, N_, 1>(sw, a, tiles, status, stream)
  if (epi == 0) KF_SMALL(0, false);
  if (epi == 1 && a.gain) return launch_small<1, true, 1>(sw, a, tiles, status, stream);
  if (epi == 1) KF_SMALL(1, false);
  if (a.gain) return launch_small<2, true, 1>(sw, a, tiles, status, stream);
  KF_SMALL(2, false);
#undef KF_SMALL
}

}  // namespace skinny
}  // namespace kf
