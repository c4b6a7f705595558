// Warp-level pieces of the query-major simplicial kernels (simplicial_small_fwd.cu, simplicial_small_bwd.cu).
//
// For one query i the logits over all key pairs are a matrix product, S_i[j,k] = (K1 o q_i) K2^T, and so is everything
// after it: W_i = P_i V2, out_i = sum_j v1_j o W_i[j,:].  A molecule of at most 32 atoms gives a 32 x 32 matrix per
// query, which one warp holds in registers, so a warp takes a query from the logits to the output without a barrier.
#pragma once

#include "common.cuh"
#include "simplicial_sm100.cuh"
#include "sparse_attn_mma.cuh"

namespace mf {

constexpr int kRowBytes = kD * 2;            // one 64-channel bf16 row in shared memory
constexpr int kSmallRows = 32;               // keys / queries of a small molecule
constexpr int kSmallTile = kSmallRows * kRowBytes;

// 16-byte chunk `chunk` of row `row`; chunks are XOR-swizzled with the row so that ldmatrix is free of bank conflicts
__device__ __forceinline__ uint32_t row_chunk(uint32_t tile, int row, int chunk) {
  return tile + row * kRowBytes + ((chunk ^ (row & 7)) << 4);
}

// Where a lane reads its fragments: the swizzle is an XOR of the address with a multiple of 32 (or 64) bytes, so one base per
// access pattern serves every tile and every step (tiles start on 128-byte boundaries and have 128-byte rows).
struct FragBase {
  uint32_t a, b, t;
  __device__ __forceinline__ explicit FragBase(uint32_t tile0, int lane)
      : a(row_chunk(tile0, lane & 15, lane >> 4)),
        b(row_chunk(tile0, lane & 7, lane >> 3)),
        t(row_chunk(tile0, (lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1)) {}
};
// A operand (16 rows of the tile x 16 channels): rows 16*mt, channels 16*ks; `tile` = offset of the tile behind tile0
__device__ __forceinline__ void load_a(uint32_t (&r)[4], const FragBase& f, int tile, int mt, int ks) {
  ldmatrix_x4(r, (f.a ^ (ks << 5)) + tile + mt * 16 * kRowBytes);
}
// B operand (rows of the tile as columns): rows 8*nt, channels 32*kp .. +31 (two k-steps)
__device__ __forceinline__ void load_b(uint32_t (&r)[4], const FragBase& f, int tile, int nt, int kp) {
  ldmatrix_x4(r, (f.b ^ (kp << 6)) + tile + nt * 8 * kRowBytes);
}
// Transposed view, channels 16*dt (rows of the fragment) x tile rows 16*js (columns): the A operand of a product over
// the tile's rows; r[0], r[2] (channels +0..7) and r[1], r[3] (+8..15) are also its 8-wide B operands
__device__ __forceinline__ void load_t(uint32_t (&r)[4], const FragBase& f, int tile, int dt, int js) {
  ldmatrix_x4_trans(r, (f.t ^ (dt << 5)) + tile + js * 16 * kRowBytes);
}
// B operands of a product over the tile's rows 16*ks: channels 16*dp (r[0], r[1]) and 16*dp + 8 (r[2], r[3])
__device__ __forceinline__ void load_t2(uint32_t (&r)[4], const FragBase& f, int tile, int dp, int ks) {
  ldmatrix_x4_trans(r, (f.a ^ (dp << 5)) + tile + ks * 16 * kRowBytes);
}
// One row, channel pairs as an A / B operand holds them: r[c] = channels 8 c + 2 (lane % 4) + {0, 1}
__device__ __forceinline__ void load_row_pairs(uint32_t (&r)[8], uint32_t tile, int row, int lane) {
  uint32_t a[4], b[4];
  const uint32_t at = row_chunk(tile, row, lane >> 3);
  ldmatrix_x4(a, at);
  ldmatrix_x4(b, at ^ 64u);
#pragma unroll
  for (int c = 0; c < 4; ++c) r[c] = a[c], r[4 + c] = b[c];
}
// One row, r[c] = channel 8 c + lane / 4 in both halves
__device__ __forceinline__ void load_row_dup(uint32_t (&r)[8], uint32_t tile, int row, int lane) {
  uint32_t a[4], b[4];
  const uint32_t at = row_chunk(tile, row, lane >> 3);
  ldmatrix_x4_trans(a, at);
  ldmatrix_x4_trans(b, at ^ 64u);
#pragma unroll
  for (int c = 0; c < 4; ++c) r[c] = a[c], r[4 + c] = b[c];
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// 8 x 8 tile of 16-bit values, transposed across the warp
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// d (16x8, fp32) += a (16x16) * b (16x8); not volatile, so that independent products may be interleaved with other work
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = a * b
__device__ __forceinline__ void mma16_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// two fp32 operations per instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{ .reg .b64 ra, rb, rc, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mov.b64 rc, {%6, %7}; "
      "fma.rn.f32x2 rd, ra, rb, rc; mov.b64 {%0, %1}, rd; }"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{ .reg .b64 ra, rb, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; add.rn.f32x2 rd, ra, rb; mov.b64 {%0, %1}, rd; }"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{ .reg .b64 ra, rb, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mul.rn.f32x2 rd, ra, rb; mov.b64 {%0, %1}, rd; }"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// Sums of the eight values over the four lanes of a quad; every lane keeps two of them: v[0], v[1] = values e0, e0 + 1
// with e0 = 4 (lane & 1) + 2 ((lane >> 1) & 1).
__device__ __forceinline__ void quad_sum8(float (&v)[8], int lane) {
  const bool odd = lane & 1, upper = (lane >> 1) & 1;
  float t[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float keep = odd ? v[4 + e] : v[e], give = odd ? v[e] : v[4 + e];
    t[e] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float keep = upper ? t[2 + e] : t[e], give = upper ? t[e] : t[2 + e];
    v[e] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
  }
}

}  // namespace mf
