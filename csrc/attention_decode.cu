// Attention of one new token per sequence against a KV cache (generation step).
//
// What bounds it: each cached key and value is read once and used for the `group` query heads that share it, so the
// kernel is a stream over the cache; the arithmetic is a few per cent of the tensor cores' rate even on the warp-level
// MMA.  A 128-row query tile (the prefill kernels) would compute 127 rows of padding and give one block per (batch,
// query head), i.e. 32 blocks that each walk the whole cache and read every key `group` times.  Here
//   * one cluster per (batch, KV head): all query heads of the group are the 16 rows of an m16n8k16 MMA, so K and V
//     are read once; the keys are split over the cluster's CTAs (up to 8) and over the four warps of each CTA;
//   * K and V tiles of 64 keys move through a three-stage cp.async ring, two stages of which are in flight while the third is
//     read (head dim 128, two CTAs per SM: 128 KB in flight per SM), 16-byte chunks XOR-swizzled so that ldmatrix is free of
//     bank conflicts;
//   * the partial (max, sum, output) triples are merged in shared memory and then across the cluster through
//     distributed shared memory, in a fixed order: one launch, no workspace, bit-reproducible.
// Generation uses the form for head dim 128; with 64 the block keeps the bits of the separate ops (ops/cuda.py, block_decode).
// The cache may be a view of a larger one (any batch stride; rows 16-byte aligned), so growing caches need no copy.
//
// Replaces F.scaled_dot_product_attention for the cached step of the reference (kempnerforge/model/attention.py:213-231).
#include "common.cuh"
#include "skinny_common.cuh"

namespace kf {
namespace decode {

constexpr int THREADS = 128;
constexpr int TILE = 64;     // keys per ring stage, 16 per warp
constexpr int STAGES = 3;
constexpr int ROWS = 16;     // query heads per cluster (MMA rows)

template <int HD>
struct Cfg {
  static constexpr int TILE_BYTES = TILE * HD * 2;
  static constexpr int RING = STAGES * 2 * TILE_BYTES;
  static constexpr int PART = 4 * ROWS * HD * 4;                 // per-warp partial outputs, alias the ring
  static constexpr int BODY = RING > PART ? RING : PART;
  static constexpr int MERGED = ROWS * HD * 4;                   // the CTA's merged partial
  static constexpr int STATS = (4 + 1) * ROWS * 2 * 4;           // (max, sum) per warp and merged
  static constexpr size_t SMEM = size_t(BODY) + MERGED + STATS;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;  // 0 source bytes: the chunk is filled with zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ float ld_cluster_f1(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// exp2(m - top) with the empty partial (m = -inf) weighing nothing
__device__ __forceinline__ float weight(float m, float top) { return m == -INFINITY ? 0.f : fast_exp2(m - top); }

template <int HD>
__global__ void __launch_bounds__(THREADS)
kf_attn_decode(const __nv_bfloat16* __restrict__ Q, const __nv_bfloat16* __restrict__ K, const __nv_bfloat16* __restrict__ V,
               __nv_bfloat16* __restrict__ O, int Sk, int H, int group, long long ldq, long long ldo, long long kv_row,
               long long k_batch, long long v_batch, float scale_log2, int n_old) {
  using C = Cfg<HD>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t ring = smem_u32(smem_raw);
  float* part = reinterpret_cast<float*>(smem_raw);
  float* merged = reinterpret_cast<float*>(smem_raw + C::BODY);
  float* stats = reinterpret_cast<float*>(smem_raw + C::BODY + C::MERGED);  // [5][ROWS][2]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = int(cluster_nctaid()), rank = int(cluster_ctarank());
  const int blocks_per_kv = (group + ROWS - 1) / ROWS;
  const int hk = int(blockIdx.y) / blocks_per_kv, hb = int(blockIdx.y) % blocks_per_kv;
  const int b = int(blockIdx.z);
  const int n_heads = min(ROWS, group - hb * ROWS);     // query heads of this cluster
  const int h0 = hk * group + hb * ROWS;

  const int n_tiles = (Sk + TILE - 1) / TILE;
  const int t0 = int((long long)n_tiles * rank / splits), t1 = int((long long)n_tiles * (rank + 1) / splits);
  const __nv_bfloat16* kb = K + (long long)b * k_batch + (long long)hk * HD;
  const __nv_bfloat16* vb = V + (long long)b * v_batch + (long long)hk * HD;

  constexpr int CHUNKS = HD / 8;                        // 16-byte chunks per row
  auto issue = [&](int t) {
    const uint32_t ks = ring + uint32_t((t - t0) % STAGES) * 2u * C::TILE_BYTES, vs = ks + C::TILE_BYTES;
#pragma unroll
    for (int i = 0; i < TILE * CHUNKS / THREADS; ++i) {
      const int idx = threadIdx.x + i * THREADS, r = idx / CHUNKS, c = idx % CHUNKS;
      const int pos = t * TILE + r;
      const bool in = pos < Sk;
      const long long off = (long long)(in ? pos : 0) * kv_row + c * 8;
      const uint32_t dst = uint32_t(r * HD * 2 + ((c ^ (r & 7)) << 4));
      cp_async16(ks + dst, kb + off, in);
      cp_async16(vs + dst, vb + off, in);
    }
  };
  // Tiles that hold only positions older than the previous kernel's writes may be fetched before it has finished.
  int t = t0;
  for (; t < min(t1, t0 + STAGES - 1) && (t + 1) * TILE <= n_old; ++t) {
    issue(t);
    cp_commit();
  }
  grid_dep_wait();
  for (; t < t0 + STAGES - 1; ++t) {
    if (t < t1) issue(t);
    cp_commit();
  }
  grid_dep_launch();

  // query rows as MMA A fragments (rows past the group are zero)
  uint32_t qa[HD / 16][4];
  {
    const int g = lane >> 2, c = (lane & 3) * 2;
    const __nv_bfloat16* q0 = Q + (long long)b * ldq + (long long)(h0 + g) * HD;
#pragma unroll
    for (int kk = 0; kk < HD / 16; ++kk) {
      qa[kk][0] = g < n_heads ? *reinterpret_cast<const uint32_t*>(q0 + kk * 16 + c) : 0u;
      qa[kk][1] = g + 8 < n_heads ? *reinterpret_cast<const uint32_t*>(q0 + 8 * HD + kk * 16 + c) : 0u;
      qa[kk][2] = g < n_heads ? *reinterpret_cast<const uint32_t*>(q0 + kk * 16 + 8 + c) : 0u;
      qa[kk][3] = g + 8 < n_heads ? *reinterpret_cast<const uint32_t*>(q0 + 8 * HD + kk * 16 + 8 + c) : 0u;
    }
  }
  float o[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

  for (t = t0; t < t1; ++t) {
    cp_wait<STAGES - 2>();
    __syncthreads();  // tile t has landed for every thread, and the stage refilled below has been consumed
    if (t + STAGES - 1 < t1) issue(t + STAGES - 1);
    cp_commit();
    const int key0 = t * TILE + warp * 16;
    if (key0 >= Sk) continue;
    const uint32_t ks = ring + uint32_t((t - t0) % STAGES) * 2u * C::TILE_BYTES, vs = ks + C::TILE_BYTES;
    const int mi = lane >> 3, lr = lane & 7;
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    {
      const int r = warp * 16 + lr + (mi >> 1) * 8;
      const uint32_t row = ks + uint32_t(r * HD * 2);
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
        uint32_t f[4];
        ldsm4(row + uint32_t(((kk * 2 + (mi & 1)) ^ lr) << 4), f);
        mma16816(s[0], qa[kk], f[0], f[1]);
        mma16816(s[1], qa[kk], f[2], f[3]);
      }
    }
    const int kc = key0 + (lane & 3) * 2;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = kc + n * 8 + (e & 1) < Sk ? s[n][e] * scale_log2 : -INFINITY;
    uint32_t pa[4];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      float mx = fmaxf(fmaxf(s[0][2 * hf], s[0][2 * hf + 1]), fmaxf(s[1][2 * hf], s[1][2 * hf + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float mn = fmaxf(m[hf], mx);
      const float base = mn == -INFINITY ? 0.f : mn;
      const float alpha = weight(m[hf], base);
      m[hf] = mn;
      float p[2][2], sum = 0.f;
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          p[n][e] = fast_exp2(s[n][2 * hf + e] - base);
          sum += p[n][e];
        }
      l[hf] = l[hf] * alpha + sum;  // this thread's four keys; the quad is summed at the end
      pa[hf] = pack_bf16(p[0][0], p[0][1]);
      pa[2 + hf] = pack_bf16(p[1][0], p[1][1]);
#pragma unroll
      for (int i = 0; i < HD / 8; ++i) {
        o[i][2 * hf] *= alpha;
        o[i][2 * hf + 1] *= alpha;
      }
    }
    {
      const int r = warp * 16 + lr + (mi & 1) * 8;
      const uint32_t row = vs + uint32_t(r * HD * 2);
#pragma unroll
      for (int d = 0; d < HD / 16; ++d) {
        uint32_t f[4];
        ldsm4_t(row + uint32_t(((d * 2 + (mi >> 1)) ^ lr) << 4), f);
        mma16816(o[2 * d], pa, f[0], f[1]);
        mma16816(o[2 * d + 1], pa, f[2], f[3]);
      }
    }
  }
  cp_wait<0>();
  __syncthreads();  // the ring is idle: it becomes the partial buffer

  // ---- merge: warps of this CTA
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    l[hf] += __shfl_xor_sync(0xffffffffu, l[hf], 1);
    l[hf] += __shfl_xor_sync(0xffffffffu, l[hf], 2);
    const int r = (lane >> 2) + hf * 8;
    if ((lane & 3) == 0) {
      stats[(warp * ROWS + r) * 2] = m[hf];
      stats[(warp * ROWS + r) * 2 + 1] = l[hf];
    }
    if (r < n_heads) {
      float* dst = part + (warp * ROWS + r) * HD + (lane & 3) * 2;
#pragma unroll
      for (int i = 0; i < HD / 8; ++i)
        *reinterpret_cast<float2*>(dst + i * 8) = make_float2(o[i][2 * hf], o[i][2 * hf + 1]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_heads * (HD / 4); i += THREADS) {
    const int r = i / (HD / 4), d = (i % (HD / 4)) * 4;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) top = fmaxf(top, stats[(w * ROWS + r) * 2]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = weight(stats[(w * ROWS + r) * 2], top);
      const float4 v = *reinterpret_cast<const float4*>(part + (w * ROWS + r) * HD + d);
      acc.x += f * v.x; acc.y += f * v.y; acc.z += f * v.z; acc.w += f * v.w;
      sum += f * stats[(w * ROWS + r) * 2 + 1];
    }
    *reinterpret_cast<float4*>(merged + r * HD + d) = acc;
    if (d == 0) {
      stats[(4 * ROWS + r) * 2] = top;
      stats[(4 * ROWS + r) * 2 + 1] = sum;
    }
  }
  cluster_sync_all();
  // ---- merge: CTAs of the cluster, each one its share of the output
  const uint32_t merged_a = ring + C::BODY, stats_a = ring + C::BODY + C::MERGED + 4 * ROWS * 2 * 4;
  for (int i = rank * THREADS + threadIdx.x; i < n_heads * (HD / 4); i += splits * THREADS) {
    const int r = i / (HD / 4), d = (i % (HD / 4)) * 4;
    float top = -INFINITY;
    for (int c = 0; c < splits; ++c) top = fmaxf(top, ld_cluster_f1(mapa_shared(stats_a + r * 8, c)));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float sum = 0.f;
    for (int c = 0; c < splits; ++c) {
      const float f = weight(ld_cluster_f1(mapa_shared(stats_a + r * 8, c)), top);
      const float4 v = ld_cluster_f4(mapa_shared(merged_a + uint32_t(r * HD + d) * 4u, c));
      acc.x += f * v.x; acc.y += f * v.y; acc.z += f * v.z; acc.w += f * v.w;
      sum += f * ld_cluster_f1(mapa_shared(stats_a + r * 8 + 4, c));
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    uint2 w;
    w.x = pack_bf16(acc.x * inv, acc.y * inv);
    w.y = pack_bf16(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(O + (long long)b * ldo + (long long)(h0 + r) * HD + d) = w;
  }
  cluster_sync_all();
}

template <int HD>
static int launch(const void* q, const void* k, const void* v, void* o, int B, int Sk, int H, int Hkv, long long ldq,
                  long long ldo, long long kv_row, long long k_batch, long long v_batch, float scale, int n_old, int pdl,
                  int num_sms, cudaStream_t stream) {
  using C = Cfg<HD>;
  auto kern = kf_attn_decode<HD>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return 300 + (int)e;
    if (dev < 16) attr_set[dev] = true;
  }
  const int group = H / Hkv;
  const int ny = Hkv * ((group + ROWS - 1) / ROWS);
  // two CTAs per SM, at least one 64-key tile per CTA
  int splits = 1;
  while (splits < 8 && (long long)B * ny * splits * 2 <= 2LL * num_sms && Sk > splits * TILE) splits *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)splits, (unsigned)ny, (unsigned)B);
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
  cfg.numAttrs = pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v,
                                     (__nv_bfloat16*)o, Sk, H, group, ldq, ldo, kv_row, k_batch, v_batch,
                                     scale * 1.4426950408889634f, n_old);
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace decode
}  // namespace kf

extern "C" {

// o[B][H * hd] = softmax(q k^T * scale) v over Sk cached positions.  q rows of pitch ldq with the heads side by side;
// k / v: position p of batch entry b, KV head j at base + b * batch + p * kv_row + j * hd (elements).  hd 64 or 128; all
// strides multiples of 8, bases 16-byte aligned.  n_old: with pdl, the leading positions that the previous kernel of the
// stream does not write (0 otherwise).
int kf_attn_decode_bf16(const void* q, const void* k, const void* v, void* o, int B, int Sk, int H, int Hkv, int hd,
                        long long ldq, long long ldo, long long kv_row, long long k_batch, long long v_batch, float scale,
                        int n_old, int pdl, int num_sms, void* stream) {
  using namespace kf::decode;
  if ((hd != 64 && hd != 128) || Hkv <= 0 || H % Hkv != 0 || B < 1 || B > 65535 || Sk < 1) return 3;
  if ((ldq | ldo | kv_row | k_batch | v_batch) & 7) return 5;
  if (hd == 128)
    return launch<128>(q, k, v, o, B, Sk, H, Hkv, ldq, ldo, kv_row, k_batch, v_batch, scale, pdl ? n_old : 0, pdl, num_sms,
                       (cudaStream_t)stream);
  return launch<64>(q, k, v, o, B, Sk, H, Hkv, ldq, ldo, kv_row, k_batch, v_batch, scale, pdl ? n_old : 0, pdl, num_sms,
                    (cudaStream_t)stream);
}

}  // extern "C"
