// What the few-row GEMMs (gemm_skinny_tcgen05.cu, gemm_small.cu) are given, and the norm that both can take along.
#pragma once
#include "common.cuh"
#include "skinny_common.cuh"

namespace kf {
namespace skinny {

// Args::pdl.  0: an ordinary launch.  PDL_EARLY_WEIGHTS: a programmatic launch behind a kernel that writes no weights and no gain; they
// are fetched while it runs.  PDL_WAIT_FIRST: a programmatic launch behind any kernel; nothing is read before the wait, only barriers and
// tensor memory are set up.
constexpr int PDL_EARLY_WEIGHTS = 1, PDL_WAIT_FIRST = 2;

constexpr int NORM_ROWS = 4;  // rows up to which a projection takes the norm of its input along

struct Args {
  __nv_bfloat16* out;            // [M][ldo]
  const __nv_bfloat16* residual; // [M][ldr] or null (epilogue 0)
  int M, K, ldo, ldr;
  int round_first;               // residual: round the product to bf16 before adding, as separate kernels do
  int n_seg;
  int tile0[4];   // first tile of each segment (epilogue 1: of the hidden dimension)
  int rows[3];    // rows of each segment
  int col[3];     // output column of each segment's first row
  // epilogue 2
  __nv_bfloat16 *kc, *vc;        // cache rows [batch][position][kv_dim], already offset to the first new position
  long long cache_batch;         // elements between batch entries
  const float *cosT, *sinT;      // [S][hd / 2], row 0 = first new position
  int S, kv_cols, hd;
  const __nv_bfloat16 *x, *gain; // [M][ldx]; [K] with the norm, else null
  int ldx;
  float eps;
  int pdl;                       // how the launch follows the previous kernel, see above
};

// The arithmetic of kf_rmsnorm_fwd, whose block of 256 threads adds the squares of every 256th vector of 8 per thread, then
// 32 threads by shuffles, then the eight warps.
__device__ __forceinline__ void add_squares(const uint4 u, float& ss) {
  const float2 p = unpack_bf16(u.x), q = unpack_bf16(u.y), w = unpack_bf16(u.z), z = unpack_bf16(u.w);
  const float e[8] = {p.x, p.y, q.x, q.y, w.x, w.y, z.x, z.y};
#pragma unroll
  for (int i = 0; i < 8; ++i) ss += e[i] * e[i];
}
__device__ __forceinline__ float norm_rstd(const float* warp_sums, int lane, int D, float eps) {
  return rsqrtf(norm_warp_sum(lane < 8 ? warp_sums[lane] : 0.f) / D + eps);
}
__device__ __forceinline__ uint4 norm_vec(const uint4 x, const uint4 gain, float rstd) {
  const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, gw[4] = {gain.x, gain.y, gain.z, gain.w};
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 xv = unpack_bf16(xw[e]), gv = unpack_bf16(gw[e]);
    o[e] = pack_bf16(xv.x * rstd * gv.x, xv.y * rstd * gv.y);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// gemm_small.cu: whether it takes the product (rows, K, M and gain set; one_piece: its sums over K are not to be split), and the
// launch.
bool small_fits(const Args& a, int epi, bool one_piece, int num_sms);
int run_small(int epi, const void* const* w, const int* ldw, Args& a, int* status, cudaStream_t stream);

}  // namespace skinny
}  // namespace kf
