// Epilogue of the CTA-pair kernels whose tiles have weight rows (features) as the M side and tokens as the N side
// (gemm_tokens_tcgen05_2cta.cu, grouped_gemm_tcgen05_2cta.cu).
//
// The accumulator holds a feature per lane and a token per column.  The epilogue turns 32 x 32 blocks through shared memory
// (fp32, XOR-swizzled 16-byte chunks: no bank conflicts), after which a lane holds 32 features of one token, as in the
// kernels with tokens as rows.  Where two features are combined (gate and up of a hidden unit, the two halves of a rotary pair) the
// blocks of the two warps that hold them are read by both, half the features each (boxes of 16 rows that bring both into one warp
// were tried: nine copies per k-block instead of three are slower than the products).
#pragma once
#include "common.cuh"
#include "gemm_epilogue.cuh"

namespace kf2 {
namespace tokens {

using namespace kf;

constexpr int TURN_BYTES = 4096;     // a warp's 32 x 32 fp32 block on its way from features to tokens
constexpr int BOX_BYTES = 2048;      // a warp's 32 x 32 bf16 block on its way to or from global memory
constexpr int WARP_BYTES = TURN_BYTES + 2 * BOX_BYTES;

// EPI 0: (+ residual); 1: SwiGLU over W = [gate ; up]; 2: rotary embedding of the first columns of q | k | v; 3: SwiGLU gradient.
struct Output {
  __nv_bfloat16* out;        // [T][ldo]
  const __nv_bfloat16* aux;  // residual [T][lda] (0), pre-activations to write (1, or null) or to read (3) [T][lda] = gate | up
  int T, F, ldo, lda;        // F: output features (1 and 3: hidden units)
  const float *cosT, *sinT;  // [S][hd / 2]
  int S, rope_cols, hd;
};

// 16 columns of 32 rows: 32 contiguous bytes per row, two lanes each; cols: how many of the 16 exist (a multiple of 8).
__device__ __forceinline__ void store_rows16(uint32_t box, int lane, const uint4& lo, const uint4& hi, __nv_bfloat16* dst, size_t ld,
                                             int rows, int cols) {
  auto at = [&](int row, int q) { return box + uint32_t(row * 32 + ((q ^ ((row >> 2) & 1)) << 4)); };
  __syncwarp();
  sts128(at(lane, 0), lo);
  sts128(at(lane, 1), hi);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = i * 16 + (lane >> 1), ch = lane & 1;
    if (row < rows && ch * 8 < cols) *reinterpret_cast<uint4*>(dst + row * ld + ch * 8) = lds128(at(row, ch));
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

// One tile: features [f0, f0 + 128) of the CTA (1: 64 hidden units), token rows [tok0, tok0 + tokens).  t_row: the warp's 32 lanes of the
// accumulator; wait(): until it is complete, false if that failed.  Called by the four epilogue warps alike.
template <int EPI, typename Wait>
__device__ __forceinline__ bool tile_epilogue(const Output& a, uint32_t box_smem, int quarter, int lane, int f0, int tok0, int tokens,
                                              uint32_t t_row, Wait wait) {
  const uint32_t turn = box_smem + uint32_t(quarter) * WARP_BYTES, box = turn + TURN_BYTES, box2 = box + BOX_BYTES;
  // 1, 2: two warps meet, one with the first halves (gate, or the dimensions below hd / 2) and one with the second; each takes
  // 16 features of either.  Halves of 64 rows are two warps apart, those of a head of 64 one.
  constexpr bool MEET = EPI == 1 || EPI == 2;
  const int apart = EPI == 2 && a.hd == 64 ? 1 : 2, first = quarter & ~apart, share = quarter & apart ? 1 : 0;
  const int meet_bar = 1 + (apart == 1 ? quarter >> 1 : quarter & 1);
  const uint32_t turn1 = box_smem + uint32_t(first) * WARP_BYTES, turn2 = turn1 + uint32_t(apart) * WARP_BYTES;
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
  bool ok = wait();
  if (MEET) ok = meet_all(meet_bar, ok);  // both warps go on, or neither
  if (!ok) return false;
  tc_fence_after();
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
      if (a.aux) {
        __nv_bfloat16* gu = const_cast<__nv_bfloat16*>(aux) + size_t(c) * 32 * a.lda;
        store_rows16(box, lane, pack8(f), pack8(f + 8), gu, a.lda, left, cols);
        store_rows16(box2, lane, pack8(f + 16), pack8(f + 24), gu + a.F, a.lda, left, cols);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {  // the activation sees bf16 pre-activations, as in swiglu_chunk
        const float g = __bfloat162float(__float2bfloat16(f[i])), u = __bfloat162float(__float2bfloat16(f[16 + i]));
        f[i] = g / (1.f + __expf(-g)) * u;
      }
      store_rows16(box, lane, pack8(f), pack8(f + 8), out, a.ldo, left, cols);
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
      {
        store_rows16(box, lane, pack8(f), pack8(f + 8), out, a.ldo, left, cols);
        store_rows16(box2, lane, pack8(f + 16), pack8(f + 24), out + half, a.ldo, left, cols);
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
  return true;
}

}  // namespace tokens
}  // namespace kf2
