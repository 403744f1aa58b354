// Epilogue helpers shared by the 1-CTA and 2-CTA tcgen05 GEMM kernels: conversion of one 32-column
// accumulator chunk (held by one thread for one output row) to bf16 / fp32 global stores, with
// optional accumulation into the destination and an optional residual operand; the SwiGLU forward / backward
// arithmetic of the fused epilogues.
#pragma once
#include "common.cuh"

namespace kf {

template <typename OutT>
__device__ __forceinline__ void store_chunk(OutT* dst, const uint32_t (&acc)[32], int valid_cols,
                                            bool accumulate, const OutT* residual);

template <>
__device__ __forceinline__ void store_chunk<__nv_bfloat16>(__nv_bfloat16* dst, const uint32_t (&acc)[32],
                                                           int valid_cols, bool accumulate,
                                                           const __nv_bfloat16* residual) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    if (v * 8 >= valid_cols) break;
    uint4* p = reinterpret_cast<uint4*>(dst + v * 8);
    float f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(acc[v * 8 + i]);
    if (accumulate) {
      uint4 old = *p;
      float2 a = unpack_bf16(old.x), b = unpack_bf16(old.y), c = unpack_bf16(old.z), d = unpack_bf16(old.w);
      f[0] += a.x; f[1] += a.y; f[2] += b.x; f[3] += b.y;
      f[4] += c.x; f[5] += c.y; f[6] += d.x; f[7] += d.y;
    }
    if (residual) {
      uint4 old = *reinterpret_cast<const uint4*>(residual + v * 8);
      float2 a = unpack_bf16(old.x), b = unpack_bf16(old.y), c = unpack_bf16(old.z), d = unpack_bf16(old.w);
      f[0] += a.x; f[1] += a.y; f[2] += b.x; f[3] += b.y;
      f[4] += c.x; f[5] += c.y; f[6] += d.x; f[7] += d.y;
    }
    uint4 out;
    out.x = pack_bf16(f[0], f[1]);
    out.y = pack_bf16(f[2], f[3]);
    out.z = pack_bf16(f[4], f[5]);
    out.w = pack_bf16(f[6], f[7]);
    *p = out;
  }
}

template <>
__device__ __forceinline__ void store_chunk<float>(float* dst, const uint32_t (&acc)[32], int valid_cols,
                                                   bool accumulate, const float* residual) {
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    if (v * 4 >= valid_cols) break;
    float4* p = reinterpret_cast<float4*>(dst + v * 4);
    float4 o = make_float4(__uint_as_float(acc[v * 4]), __uint_as_float(acc[v * 4 + 1]),
                           __uint_as_float(acc[v * 4 + 2]), __uint_as_float(acc[v * 4 + 3]));
    if (accumulate) {
      float4 old = *p;
      o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
    }
    if (residual) {
      float4 r = *reinterpret_cast<const float4*>(residual + v * 4);
      o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w;
    }
    *p = o;
  }
}

// SwiGLU forward on one 32-column chunk: g <- silu(g) * u.  The activation sees the bf16-rounded pre-activations,
// like the two-kernel path (GEMM writes bf16 gate | up, the element-wise kernel reads them back).
__device__ __forceinline__ void swiglu_chunk(uint32_t (&g)[32], const uint32_t (&u)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float gf = __bfloat162float(__float2bfloat16(__uint_as_float(g[i])));
    const float uf = __bfloat162float(__float2bfloat16(__uint_as_float(u[i])));
    g[i] = __float_as_uint(gf / (1.f + __expf(-gf)) * uf);
  }
}

// ---- 32 rows x 32 columns of a warp between registers (one row per lane) and global memory, through shared memory.
// A lane that reads or writes its own row touches 32 different lines per 16-byte instruction and half a sector of each;
// four lanes per row move 64 contiguous bytes, eight rows per instruction.  `box`: 2 KB of shared memory of this warp,
// 16-byte chunk q of row r at slot q ^ (r / 2 % 4) of its 64 bytes (no bank conflicts either way).  Grouped products: SwiGLU
// gradients of 8 experts of 2048 x 7168 over 4096 rows 156 -> 142 us, of 64 of 2048 x 1408 over 10 662 rows 133 -> 122.
__device__ __forceinline__ uint32_t box_row_chunk(uint32_t box, int row, int q) {
  return box + uint32_t(row * 64 + ((q ^ ((row >> 1) & 3)) << 4));
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
struct Rows32 {
  uint4 q[4];  // as moved: chunk lane % 4 of rows lane / 4 + 8 i; or, after an exchange, the four chunks of row `lane`
};
// `src`: first row and column of the box; rows / cols: how many of the 32 exist (the rest reads as zero).
__device__ __forceinline__ Rows32 load_rows32(const __nv_bfloat16* src, size_t ld, int lane, int rows, int cols) {
  Rows32 r;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = i * 8 + (lane >> 2), ch = lane & 3;
    r.q[i] = row < rows && ch * 8 < cols ? *reinterpret_cast<const uint4*>(src + row * ld + ch * 8) : make_uint4(0, 0, 0, 0);
  }
  return r;
}
// moved layout -> the lane's own row
__device__ __forceinline__ Rows32 to_own_row(uint32_t box, int lane, const Rows32& m) {
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) sts128(box_row_chunk(box, i * 8 + (lane >> 2), lane & 3), m.q[i]);
  __syncwarp();
  Rows32 r;
#pragma unroll
  for (int q = 0; q < 4; ++q) r.q[q] = lds128(box_row_chunk(box, lane, q));
  return r;
}
__device__ __forceinline__ void store_rows32(uint32_t box, int lane, const Rows32& own, __nv_bfloat16* dst, size_t ld, int rows,
                                             int cols) {
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) sts128(box_row_chunk(box, lane, q), own.q[q]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = i * 8 + (lane >> 2), ch = lane & 3;
    if (row < rows && ch * 8 < cols) *reinterpret_cast<uint4*>(dst + row * ld + ch * 8) = lds128(box_row_chunk(box, row, ch));
  }
}
__device__ __forceinline__ Rows32 pack_row32(const uint32_t (&v)[32]) {
  Rows32 r;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t* f = v + q * 8;
    r.q[q] = make_uint4(pack_bf16(__uint_as_float(f[0]), __uint_as_float(f[1])), pack_bf16(__uint_as_float(f[2]), __uint_as_float(f[3])),
                        pack_bf16(__uint_as_float(f[4]), __uint_as_float(f[5])), pack_bf16(__uint_as_float(f[6]), __uint_as_float(f[7])));
  }
  return r;
}

// SwiGLU backward on one 32-column chunk of one row: `dh` holds the gradient of the hidden activation (fp32 accumulator
// values), gate / up the saved bf16 pre-activations; they are replaced by the gradients.  The incoming gradient is rounded to
// bf16 first, like the two-kernel path.
__device__ __forceinline__ void swiglu_bwd_row(const uint32_t (&dh)[32], Rows32& gate, Rows32& up) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t gw[4] = {gate.q[q].x, gate.q[q].y, gate.q[q].z, gate.q[q].w}, uw[4] = {up.q[q].x, up.q[q].y, up.q[q].z, up.q[q].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 g2 = unpack_bf16(gw[e]), u2 = unpack_bf16(uw[e]);
      const float d0 = __bfloat162float(__float2bfloat16(__uint_as_float(dh[q * 8 + 2 * e])));
      const float d1 = __bfloat162float(__float2bfloat16(__uint_as_float(dh[q * 8 + 2 * e + 1])));
      const float s0 = 1.f / (1.f + __expf(-g2.x)), s1 = 1.f / (1.f + __expf(-g2.y));
      uw[e] = pack_bf16(d0 * g2.x * s0, d1 * g2.y * s1);
      gw[e] = pack_bf16(d0 * u2.x * s0 * (1.f + g2.x * (1.f - s0)), d1 * u2.y * s1 * (1.f + g2.y * (1.f - s1)));
    }
    gate.q[q] = make_uint4(gw[0], gw[1], gw[2], gw[3]);
    up.q[q] = make_uint4(uw[0], uw[1], uw[2], uw[3]);
  }
}

}  // namespace kf
