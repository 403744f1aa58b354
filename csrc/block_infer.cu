// One transformer block on one new token per sequence, launched from one native call.
//
// At decoding sizes the kernels take 2 - 40 us each and a Python-level launch (attribute lookups, argument conversion,
// output allocation) 5 - 15 us, so the block is launch-bound from Python.  This entry issues the whole chain
//   RMSNorm -> q|k|v projection (rotary embedding, k and v into the cache) -> attention over the cache
//   -> o projection (+ x) -> RMSNorm -> gate|up projection (SwiGLU) -> down projection (+ residual)
// as programmatic launches: each kernel sets up (and streams its first weight tiles) while its predecessor drains.  Up to
// kf_skinny_norm_rows() sequences the projections take their norms along: five kernels in the chain instead of seven.
//
// Inside the chain a kernel may fetch weights ahead of its wait, because the kernel before it writes none.  The kernel before the
// chain is the caller's, which may have written any operand of the first one (a weight copied in, rotary tables built for this step),
// so the first kernel waits before it reads anything.  A 7B block on one token: 93.7 us so, 96.4 with an ordinary launch.
#include "skinny_args.cuh"

extern "C" {
int kf_rmsnorm_fwd_pdl_bf16(const void* x, const void* w, void* y, void* rstd, int rows, int D, float eps, int pdl,
                            void* stream);
int kf_gemm_skinny_bf16(const void* x, const void* w0, const void* w1, const void* w2, void* out, const void* residual,
                        int M, int K, int n0, int n1, int n2, int ldx, int ldw0, int ldw1, int ldw2, int ldo, int ldr,
                        int round_first, int pdl, int num_sms, void* stream);
int kf_skinny_norm_rows();
int kf_gemm_skinny_norm_swiglu_bf16(const void* x, const void* gain, float eps, const void* wg, const void* wu, void* h, int M,
                                    int F, int K, int ldx, int ldwg, int ldwu, int ldh, int pdl, int num_sms, void* stream);
int kf_gemm_skinny_norm_qkv_bf16(const void* x, const void* gain, float eps, const void* wq, const void* wk, const void* wv,
                                 void* q_out, void* kc, void* vc, int M, int S, int K, int q_cols, int kv_cols, int hd, int ldx,
                                 int ldwq, int ldwk, int ldwv, int ldq, long long cache_batch, const void* cosT,
                                 const void* sinT, int pdl, int num_sms, void* stream);
int kf_attn_decode_bf16(const void* q, const void* k, const void* v, void* o, int B, int Sk, int H, int Hkv, int hd,
                        long long ldq, long long ldo, long long kv_row, long long k_batch, long long v_batch, float scale,
                        int n_old, int pdl, int num_sms, void* stream);
int kf_attn_fwd_pdl_bf16(const void* q, const void* k, const void* v, void* o, void* lse, const void* doc, int B, int Sq, int Sk,
                         int H, int Hkv, int hd, long long ldq, long long ldk, long long ldv, long long ldo, float scale,
                         int causal, int pdl, void* stream);

// Attention half of a block for one new token in each of B sequences: h1 = x + Attention(RMSNorm(x)); with wd != null
// also the SwiGLU half: y = h1 + MLP(RMSNorm(h1)).  All matrices [out][in] contiguous; x, h1, y [B][D] contiguous.
// a: x, wn1, wq, wk, wv, wo, wn2, wg, wu, wd, kc, vc, scratch, rstd, h1, y, cosT, sinT (device pointers), then
//    B, D, H, Hkv, hd, F, pos, cache_batch, num_sms;  r: eps1, eps2, scale
//   scratch: bf16, B * (D + H * hd) elements (+ B * F with wd), kept between calls for separate parts; rstd: fp32 [B]
//   kc / vc: cache [B][positions][Hkv][hd], cache_batch elements between batch entries; `pos` = index of the new token
//   cosT / sinT: fp32 [1][hd / 2], the row of the new position
//   a[27]: parts to run (1 = up to the cache, 2 = attention, 4 = the rest); a[28]: attention kernel (0 = split over the cache,
//   1 = the 128-row tile kernel, B == 1); a[29]: attention output [B][H * hd] (written by part 2, read by part 4); a[30]: fp32
//   [H] scratch of the tile kernel
// first: the block's first kernel follows a kernel of the caller's.
static int block_decode(const long long* a, const double* r, bool first, void* stream) {
  void* p[18];
  for (int i = 0; i < 18; ++i) p[i] = reinterpret_cast<void*>(a[i]);
  const void *x = p[0], *wn1 = p[1], *wq = p[2], *wk = p[3], *wv = p[4], *wo = p[5], *wn2 = p[6], *wg = p[7], *wu = p[8],
             *wd = p[9], *cosT = p[16], *sinT = p[17];
  void *kc = p[10], *vc = p[11], *scratch = p[12], *rstd = p[13], *h1 = p[14], *y = p[15];
  const int B = (int)a[18], D = (int)a[19], H = (int)a[20], Hkv = (int)a[21], hd = (int)a[22], F = (int)a[23], pos = (int)a[24];
  const long long cache_batch = a[25];
  const int num_sms = (int)a[26], parts = (int)a[27], tile_attention = (int)a[28];
  const float eps1 = (float)r[0], eps2 = (float)r[1], scale = (float)r[2];
  typedef __nv_bfloat16 bf;
  if (B < 1 || B > 256 || D < 8 || (D & 7)) return 5;
  const int qc = H * hd, kvc = Hkv * hd;
  bf* n = (bf*)scratch;                 // [B][D]
  bf* q = n + (size_t)B * D;            // [B][qc]
  bf* hid = q + (size_t)B * qc;         // [B][F]
  const bool norm_along = B <= kf_skinny_norm_rows();
  void* att = reinterpret_cast<void*>(a[29]);
  int rc;
  if (parts & 1) {
    const long long row = (long long)pos * kvc;
    if (!norm_along) {
      rc = kf_rmsnorm_fwd_pdl_bf16(x, wn1, n, rstd, B, D, eps1, 1, stream);
      if (rc) return 1000 + rc;
    }
    rc = kf_gemm_skinny_norm_qkv_bf16(norm_along ? x : n, norm_along ? wn1 : nullptr, eps1, wq, wk, wv, q, (bf*)kc + row, (bf*)vc + row,
                                      B, 1, D, qc, kvc, hd, D, D, D, D, qc, cache_batch, cosT, sinT,
                                      first && norm_along ? kf::skinny::PDL_WAIT_FIRST : kf::skinny::PDL_EARLY_WEIGHTS, num_sms, stream);
    if (rc) return 2000 + rc;
  }
  if (parts & 2) {
    rc = tile_attention ? kf_attn_fwd_pdl_bf16(q, kc, vc, att, reinterpret_cast<void*>(a[30]), nullptr, 1, 1, pos + 1, H, Hkv, hd,
                                               qc, kvc, kvc, qc, scale, 0, 1, stream)
                        : kf_attn_decode_bf16(q, kc, vc, att, B, pos + 1, H, Hkv, hd, qc, qc, kvc, cache_batch, cache_batch,
                                              scale, pos, 1, num_sms, stream);
    if (rc) return 3000 + rc;
  }
  if (!(parts & 4)) return 0;
  // after a foreign attention kernel the programmatic launch would rest on that kernel's own triggers
  rc = kf_gemm_skinny_bf16(att, wo, nullptr, nullptr, h1, x, B, qc, D, 0, 0, qc, qc, 0, 0, D, D, 1, (parts & 2) != 0, num_sms,
                           stream);
  if (rc) return 4000 + rc;
  if (!wd) return 0;
  if (!norm_along) {
    rc = kf_rmsnorm_fwd_pdl_bf16(h1, wn2, n, rstd, B, D, eps2, 1, stream);
    if (rc) return 5000 + rc;
  }
  rc = kf_gemm_skinny_norm_swiglu_bf16(norm_along ? h1 : n, norm_along ? wn2 : nullptr, eps2, wg, wu, hid, B, F, D, D, D, D, F, 1,
                                       num_sms, stream);
  if (rc) return 6000 + rc;
  rc = kf_gemm_skinny_bf16(hid, wd, nullptr, nullptr, y, h1, B, F, D, 0, 0, F, F, 0, 0, D, D, 1, 1, num_sms, stream);
  return rc ? 7000 + rc : 0;
}

int kf_block_decode_bf16(const long long* a, const double* r, void* stream) { return block_decode(a, r, true, stream); }

// n blocks in a row: a holds 31 values per block, r three.  The blocks may share their intermediates (scratch, rstd, h1, attention):
// a kernel of the chain writes only after all kernels before it are complete.
int kf_blocks_decode_bf16(const long long* a, const double* r, int n, void* stream) {
  for (int i = 0; i < n; ++i) {
    const int rc = block_decode(a + 31 * i, r + 3 * i, i == 0, stream);
    if (rc) return rc;
  }
  return 0;
}

}  // extern "C"
