// Forward and backward of one dense transformer block, each issued from one native call.
//
// A block's forward is seven to eight kernels, its backward fifteen to twenty; issued one by one from Python each costs 10 - 20 us
// of host time (output allocation, argument conversion, tensor checks), so a small model's training step waits for the host:
// 284 us of kernels took 1000 us at 3 x 333 tokens of the 125M shape.  These entries issue the kernels that the op-by-op path
// of ops/fused_block.py issues for the same shapes, in its order, on buffers that the caller lays out; they decide nothing else.
// That step: 856 -> 459 us, 260 of them on the device.
#include "common.cuh"

extern "C" {
int kf_rmsnorm_fwd_bf16(const void*, const void*, void*, void*, int, int, float, void*);
int kf_rmsnorm_bwd_bf16(const void*, const void*, const void*, const void*, void*, void*, void*, void*, int, int, const void*, void*);
int kf_gemm_rope_bf16(const void*, const void*, const void*, const void*, void*, int, int, int, int, int, int, int, int, const void*,
                      const void*, int, int, int, int, void*);
int kf_gemm_bf16(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, int, int, void*);
int kf_gemm_swiglu_bf16(const void*, const void*, const void*, void*, void*, int, int, int, int, int, int, int, int, void*);
int kf_gemm_swiglu_bwd_bf16(const void*, const void*, const void*, void*, int, int, int, int, int, int, int, void*);
int kf_gemm_dgrad_stacked_bf16(const void*, const void*, const void*, const void*, void*, int, int, int, int, int, int, int, int, int,
                               void*);
int kf_gemm_split_k_bf16(const void*, const void*, void*, void*, int, int, int, int, int, int, int, int, void*);
int kf_attn_fwd_bf16(const void*, const void*, const void*, void*, void*, const void*, int, int, int, int, int, int, long long,
                     long long, long long, long long, float, int, void*);
int kf_attn_fwd2_bf16(const void*, const void*, const void*, void*, void*, const void*, const void*, int, int, int, int, int, int,
                      long long, long long, long long, long long, float, int, void*);
int kf_attn_bwd_rope_bf16(const void*, const void*, const void*, const void*, const void*, const void*, void*, void*, void*, void*,
                          void*, const void*, int, int, int, int, int, int, long long, long long, long long, long long, long long,
                          long long, long long, long long, float, int, const void*, const void*, const void*, void*);
}

namespace kf {
namespace blocktrain {

typedef __nv_bfloat16 bf;

// What both directions are given, in the order of the caller's array.
struct Block {
  const void *x, *wn1, *wq, *wk, *wv, *wo, *wn2, *wg, *wu, *wd, *cosT, *sinT;
  void *n1, *rstd1, *qkv, *attn, *lse, *h1, *n2, *rstd2, *gu, *hmid;
  int B, S, D, H, Hkv, hd, F, num_sms;
  int T, qc, kvc, nq;  // tokens, columns of q, of k and of q | k | v
};
constexpr int N_PTRS = 22, N_BLOCK = 30;

static Block read(const long long* a) {
  Block b;
  const void** in[12] = {&b.x, &b.wn1, &b.wq, &b.wk, &b.wv, &b.wo, &b.wn2, &b.wg, &b.wu, &b.wd, &b.cosT, &b.sinT};
  void** out[10] = {&b.n1, &b.rstd1, &b.qkv, &b.attn, &b.lse, &b.h1, &b.n2, &b.rstd2, &b.gu, &b.hmid};
  for (int i = 0; i < 12; ++i) *in[i] = reinterpret_cast<const void*>(a[i]);
  for (int i = 0; i < 10; ++i) *out[i] = reinterpret_cast<void*>(a[12 + i]);
  int* dims[8] = {&b.B, &b.S, &b.D, &b.H, &b.Hkv, &b.hd, &b.F, &b.num_sms};
  for (int i = 0; i < 8; ++i) *dims[i] = (int)a[N_PTRS + i];
  b.T = b.B * b.S;
  b.qc = b.H * b.hd;
  b.kvc = b.Hkv * b.hd;
  b.nq = b.qc + 2 * b.kvc;
  return b;
}

// What the kernels of the chain assume beyond their own checks; the caller takes the op-by-op path otherwise.
static bool covered(const Block& b) {
  return b.B >= 1 && b.S >= 1 && (long long)b.B * b.S > 256 && (long long)b.B * b.S <= 0x7fffffff / 2 && (b.hd == 64 || b.hd == 128) &&
         b.Hkv > 0 && b.H % b.Hkv == 0 && b.D % 64 == 0 && b.nq % 256 == 0 && b.qc % 128 == 0 && b.kvc % 128 == 0 && b.F % 256 == 0 &&
         b.num_sms >= 2;
}

}  // namespace blocktrain
}  // namespace kf

#define KF_STEP(base, call)                 \
  do {                                      \
    const int rc_ = (call);                 \
    if (rc_) return (base) * 1000 + rc_;    \
  } while (0)

extern "C" {

// y = block(x) for x [B * S][D], causal attention, every matrix [out][in] contiguous bf16.  a: x, wn1, wq, wk, wv, wo, wn2, wg, wu, wd,
// cosT, sinT (fp32 [S][hd / 2]), then what the backward needs: n1 [T][D], rstd1, qkv [T][qc + 2 kvc], attn [T][qc], lse [B][H][S],
// h1 [T][D], n2 [T][D], rstd2, gu [T][2F] (0: not kept), hmid [T][F]; then B, S, D, H, Hkv, hd, F, num_sms; then y (0: the output is
// not wanted, as in a recomputation).  r: eps, attention scale.  More than 256 rows, D % 64, F % 256, q | k | v % 256, q and k % 128.
int kf_block_train_fwd_bf16(const long long* a, const double* r, void* st) {
  using namespace kf::blocktrain;
  const Block b = read(a);
  void* y = reinterpret_cast<void*>(a[N_BLOCK]);
  if (!covered(b)) return 5;
  const float eps = (float)r[0], scale = (float)r[1];
  const bf* q = (const bf*)b.qkv;
  KF_STEP(1, kf_rmsnorm_fwd_bf16(b.x, b.wn1, b.n1, b.rstd1, b.T, b.D, eps, st));
  KF_STEP(2, kf_gemm_rope_bf16(b.n1, b.wq, b.wk, b.wv, b.qkv, b.T, b.qc, b.kvc, b.kvc, b.D, b.D, b.D, b.nq, b.cosT, b.sinT, b.S,
                               b.qc + b.kvc, b.hd, b.num_sms, st));
  if (b.S > 128)
    KF_STEP(3, kf_attn_fwd2_bf16(q, q + b.qc, q + b.qc + b.kvc, b.attn, b.lse, nullptr, nullptr, b.B, b.S, b.S, b.H, b.Hkv, b.hd, b.nq,
                                 b.nq, b.nq, b.qc, scale, 1, st));
  else
    KF_STEP(3, kf_attn_fwd_bf16(q, q + b.qc, q + b.qc + b.kvc, b.attn, b.lse, nullptr, b.B, b.S, b.S, b.H, b.Hkv, b.hd, b.nq, b.nq, b.nq,
                                b.qc, scale, 1, st));
  KF_STEP(4, kf_gemm_bf16(b.attn, b.wo, b.h1, b.x, b.T, b.D, b.qc, b.qc, b.qc, b.D, b.D, 0, 0, 0, 0, 0, b.num_sms, st));
  KF_STEP(5, kf_rmsnorm_fwd_bf16(b.h1, b.wn2, b.n2, b.rstd2, b.T, b.D, eps, st));
  KF_STEP(6, kf_gemm_swiglu_bf16(b.n2, b.wg, b.wu, b.hmid, b.gu, b.T, b.F, b.D, b.D, b.D, b.F, 2 * b.F, b.num_sms, st));
  if (y) KF_STEP(7, kf_gemm_bf16(b.hmid, b.wd, y, b.h1, b.T, b.D, b.F, b.F, b.F, b.D, b.D, 0, 0, 0, 0, 0, b.num_sms, st));
  return 0;
}

// Gradients of the above.  a: as there, then dy [T][D], dx [T][D], dWqkv [qc + 2 kvc][D], dWo [D][qc], dWgu [2F][D], dWd [D][F],
// dwn1 [D], dwn2 [D]; dh1 [T][D], dattn [T][qc], dqkv [T][qc + 2 kvc], dq_acc fp32 (as kf_attn_bwd_rope_bf16 wants it),
// dsum fp32 [B][H][S], partial (kf_rmsnorm_bwd_blocks(T) * D fp32); accumulate into dWqkv, dWo, dWgu, dWd (0 or 1 each); stacked: q | k | v and gate | up each lie
// back to back; ws and pieces of a split gate | up input gradient (stacked only; 0 and 1: not split).  gu is overwritten.
int kf_block_train_bwd_bf16(const long long* a, const double* r, void* st) {
  using namespace kf::blocktrain;
  const Block b = read(a);
  void* p[14];
  for (int i = 0; i < 14; ++i) p[i] = reinterpret_cast<void*>(a[N_BLOCK + i]);
  void *dy = p[0], *dx = p[1], *dwqkv = p[2], *dwo = p[3], *dwgu = p[4], *dwd = p[5], *dwn1 = p[6], *dwn2 = p[7], *dh1 = p[8],
       *dattn = p[9], *dqkv = p[10], *dq_acc = p[11], *dsum = p[12], *partial = p[13];
  const long long* f = a + N_BLOCK + 14;
  const int acc_qkv = (int)f[0], acc_o = (int)f[1], acc_gu = (int)f[2], acc_d = (int)f[3], stack_qkv = (int)f[4], stack_gu = (int)f[5],
            pieces = (int)f[7];
  void* ws = reinterpret_cast<void*>(f[6]);
  if (!covered(b) || !b.gu) return 5;
  const float scale = (float)r[1];
  // dW [rows][cols] (+)= dout [T][rows]^T in [T][cols]
  auto wgrad = [&](const void* dout, const void* in, void* dw, int rows, int cols, int acc) {
    return kf_gemm_bf16(dout, in, dw, nullptr, rows, cols, b.T, rows, cols, cols, 0, 1, 1, 0, acc, 0, b.num_sms, st);
  };
  // din [T][cols] = dout [T][rows] W [rows][cols]
  auto dgrad = [&](const void* dout, const void* w, void* din, int rows, int cols) {
    return kf_gemm_bf16(dout, w, din, nullptr, b.T, cols, rows, rows, cols, cols, 0, 0, 1, 0, 0, 0, b.num_sms, st);
  };
  KF_STEP(1, wgrad(dy, b.hmid, dwd, b.D, b.F, acc_d));
  KF_STEP(2, kf_gemm_swiglu_bwd_bf16(dy, b.wd, b.gu, b.gu, b.T, b.F, b.D, b.D, b.F, 2 * b.F, b.num_sms, st));
  if (pieces > 1)
    KF_STEP(3, kf_gemm_split_k_bf16(b.gu, b.wg, dh1, ws, b.T, b.D, 2 * b.F, 2 * b.F, b.D, b.D, pieces, b.num_sms, st));
  else if (stack_gu)
    KF_STEP(3, dgrad(b.gu, b.wg, dh1, 2 * b.F, b.D));
  else
    KF_STEP(3, kf_gemm_dgrad_stacked_bf16(b.gu, b.wg, b.wu, nullptr, dh1, b.T, b.D, b.F, b.F, 0, 2 * b.F, b.D, b.D, b.num_sms, st));
  KF_STEP(4, wgrad(b.gu, b.n2, dwgu, 2 * b.F, b.D, acc_gu));
  KF_STEP(5, kf_rmsnorm_bwd_bf16(dh1, b.h1, b.wn2, b.rstd2, dh1, partial, dwn2, nullptr, b.T, b.D, dy, st));
  KF_STEP(6, dgrad(dh1, b.wo, dattn, b.D, b.qc));
  KF_STEP(7, wgrad(dh1, b.attn, dwo, b.D, b.qc, acc_o));
  const bf* q = (const bf*)b.qkv;
  bf* dq = (bf*)dqkv;
  KF_STEP(8, kf_attn_bwd_rope_bf16(q, q + b.qc, q + b.qc + b.kvc, b.attn, dattn, b.lse, dsum, dq_acc, dq, dq + b.qc, dq + b.qc + b.kvc,
                                   nullptr, b.B, b.S, b.S, b.H, b.Hkv, b.hd, b.nq, b.nq, b.nq, b.qc, b.qc, b.nq, b.nq, b.nq, scale, 1,
                                   b.cosT, b.sinT, nullptr, st));
  if (stack_qkv)
    KF_STEP(9, dgrad(dqkv, b.wq, dx, b.nq, b.D));
  else
    KF_STEP(9, kf_gemm_dgrad_stacked_bf16(dqkv, b.wq, b.wk, b.wv, dx, b.T, b.D, b.qc, b.kvc, b.kvc, b.nq, b.D, b.D, b.num_sms, st));
  KF_STEP(10, wgrad(dqkv, b.n1, dwqkv, b.nq, b.D, acc_qkv));
  KF_STEP(11, kf_rmsnorm_bwd_bf16(dx, b.x, b.wn1, b.rstd1, dx, partial, dwn1, nullptr, b.T, b.D, dh1, st));
  return 0;
}

}  // extern "C"
