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

// The softmax is shifted by a value that need not be the maximum: as long as the shifted sum stays within 2^-60 .. 2^60,
// nothing overflows and nothing that matters underflows.  The forward kernels take shift 0 and do the queries whose sum leaves
// that range again, with their exact maxima.
constexpr float kSumLow = 8.6736174e-19f, kSumHigh = 1.1529215e18f;

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
__device__ __forceinline__ void quad_reduce(float& v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
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

// c (16 x 8 tiles, rows j, columns k) = (X o x_i) Y^T for two key-major tiles X, Y and the row x_i
template <int MT, int NT>
__device__ __forceinline__ void pair_product(float (&c)[MT][NT][4], const FragBase& fb, int x, int y, const uint32_t (&row)[8]) {
#pragma unroll
  for (int kp = 0; kp < 2; ++kp) {
    uint32_t b[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) load_b(b[nt], fb, y, nt, kp);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int ks = 2 * kp + k;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        uint32_t a[4];
        load_a(a, fb, x, mt, ks);
        a[0] = mul_bf16x2(a[0], row[2 * ks]);
        a[1] = mul_bf16x2(a[1], row[2 * ks]);
        a[2] = mul_bf16x2(a[2], row[2 * ks + 1]);
        a[3] = mul_bf16x2(a[3], row[2 * ks + 1]);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          if (ks == 0) mma16_first(c[mt][nt], a, b[nt][2 * k], b[nt][2 * k + 1]);
          else mma16(c[mt][nt], a, b[nt][2 * k], b[nt][2 * k + 1]);
        }
      }
    }
  }
}

// ---- low-rank residuals (simplicial_small_res_fwd.cu, simplicial_small_bwd.cu) ------------------------------------------
// For one query i, angle logits L_i R_i^T and message sums are products over the rank as well.  The fp32 factors of a query,
// (n x rank) each, are staged in shared memory as two bf16 tiles, x = hi + lo, and a product is hi hi + hi lo + lo hi: the
// dropped lo lo term is 2^-16 of it.  Rows of RK x 16 ranks, zero beyond the rank and beyond the last key.
template <int RK>
struct RankTile {
  static constexpr int kRow = RK * 32;                // bytes
  static constexpr int kTile = kSmallRows * kRow;     // one of hi / lo
  uint32_t base;                                      // hi at base, lo behind it

  // chunks of 16 bytes, swizzled so that eight consecutive rows fall into different banks
  __device__ __forceinline__ uint32_t at(int row, int chunk) const {
    return base + row * kRow + ((chunk ^ (RK == 1 ? (row >> 2) & 1 : (row >> 1) & 3)) << 4);
  }
  // A operand over ranks (rows 16*mt x ranks 16*rk), B operand over ranks (rows 16*np, +8: two row tiles at once)
  __device__ __forceinline__ void load_a(uint32_t (&r)[4], int lo, int mt, int rk, int lane) const {
    ldmatrix_x4(r, at(mt * 16 + (lane & 15), 2 * rk + (lane >> 4)) + lo * kTile);
  }
  __device__ __forceinline__ void load_b2(uint32_t (&r)[4], int lo, int np, int rk, int lane) const {
    ldmatrix_x4(r, at(np * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * rk + ((lane >> 3) & 1)) + lo * kTile);
  }
  // Transposed: ranks 16*rk as rows x tile rows 16*js as columns (A operand over the tile's rows); r[0], r[2] / r[1], r[3]
  // are the B operands (tile rows 16*js, ranks 16*rk / 16*rk + 8)
  __device__ __forceinline__ void load_t(uint32_t (&r)[4], int lo, int rk, int js, int lane) const {
    ldmatrix_x4_trans(r, at(js * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * rk + ((lane >> 3) & 1)) + lo * kTile);
  }
};

__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack2_bf16(x, y);
  lo = pack2_bf16(x - bf16_lo(hi), y - bf16_hi(hi));
}

__device__ __forceinline__ void store_shared64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

// Stages rows [0, n) of F factors of one query (row-major, `rank` floats each) by one warp, column r of the first
// one times scale0[r] when given; rows of hidden keys become zeros.  All loads are issued before the first value is used: a query's factors come from DRAM.
template <int F, int RK>
__device__ __forceinline__ void stage_factors(const RankTile<RK> (&t)[F], const float* const (&src)[F], int n, int rank, uint32_t kmask,
                                              const float* scale0, int lane) {
  bool fast = (rank & 3) == 0;
#pragma unroll
  for (int f = 0; f < F; ++f) fast = fast && (reinterpret_cast<uintptr_t>(src[f]) & 15) == 0;
  if (fast) {
    const int q = rank >> 2, total = n * q;
    float4 x[F][4 * RK];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int s = 0; s < 4 * RK; ++s) {
        const int idx = lane + 32 * s;
        x[f][s] = idx < total ? __ldg(reinterpret_cast<const float4*>(src[f]) + idx) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
    for (int s = 0; s < 4 * RK; ++s) {
      const int idx = lane + 32 * s;
      if (idx < total) {
        const int row = idx / q, c = idx - row * q;
        const bool ok = (kmask >> row) & 1u;
#pragma unroll
        for (int f = 0; f < F; ++f) {
          float4 v = ok ? x[f][s] : make_float4(0.f, 0.f, 0.f, 0.f);
          if (f == 0 && scale0) v.x *= scale0[4 * c], v.y *= scale0[4 * c + 1], v.z *= scale0[4 * c + 2], v.w *= scale0[4 * c + 3];
          uint32_t h0, l0, h1, l1;
          split_bf16(v.x, v.y, h0, l0);
          split_bf16(v.z, v.w, h1, l1);
          const uint32_t a = t[f].at(row, c >> 1) + (c & 1) * 8;
          store_shared64(a, h0, h1);
          store_shared64(a + RankTile<RK>::kTile, l0, l1);
        }
      }
    }
  } else {
    for (int idx = lane; idx < n * rank; idx += 32) {
      const int row = idx / rank, r = idx - row * rank;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        uint32_t h, l;
        split_bf16(((kmask >> row) & 1u) ? src[f][idx] * (f == 0 && scale0 ? scale0[r] : 1.f) : 0.f, 0.f, h, l);
        const uint32_t a = t[f].at(row, r >> 3) + (r & 7) * 2;
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)h) : "memory");
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(a + RankTile<RK>::kTile), "h"((uint16_t)l) : "memory");
      }
    }
  }
}
// Brings `bytes` from `p` on into L2 (one line per lane and step): the factors of the query that comes next
__device__ __forceinline__ void prefetch_l2(const float* p, int bytes, int lane) {
  for (int o = lane * 128; o < bytes; o += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p) + o));
}

// c[mt][nt] += L_i R_i^T over the rank
template <int MT, int NT, int RK>
__device__ __forceinline__ void add_rank_product(float (&c)[MT][NT][4], const RankTile<RK>& left, const RankTile<RK>& right, int lane) {
#pragma unroll
  for (int rk = 0; rk < RK; ++rk)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      uint32_t ah[4], al[4];
      left.load_a(ah, 0, mt, rk, lane);
      left.load_a(al, 1, mt, rk, lane);
#pragma unroll
      for (int np = 0; np < (NT + 1) / 2; ++np) {
        uint32_t bh[4], bl[4];
        right.load_b2(bh, 0, np, rk, lane);
        right.load_b2(bl, 1, np, rk, lane);
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (2 * np + t < NT) {
            float(&d)[4] = c[mt][2 * np + t < NT ? 2 * np + t : 0];
            mma16(d, ah, bh[2 * t], bh[2 * t + 1]);
            mma16(d, ah, bl[2 * t], bl[2 * t + 1]);
            mma16(d, al, bh[2 * t], bh[2 * t + 1]);
          }
      }
    }
}

// t (ranks 16*rk x j, as W^T) = F^T P^T for a factor F (keys x rank) and P (or dS) as pk[mt][nt][hh] holds it
template <int MT, int NK, int RK>
__device__ __forceinline__ void rank_sums(float (&t)[2 * MT][4], const RankTile<RK>& f, const uint32_t (&pk)[MT][NK][2], int rk, int lane) {
#pragma unroll
  for (int ks = 0; ks < NK / 2; ++ks) {
    uint32_t h[4], l[4];
    f.load_t(h, 0, rk, ks, lane);
    f.load_t(l, 1, rk, ks, lane);
#pragma unroll
    for (int jt = 0; jt < 2 * MT; ++jt) {
      const uint32_t b0 = pk[jt >> 1][2 * ks][jt & 1], b1 = pk[jt >> 1][2 * ks + 1][jt & 1];
      if (ks == 0) mma16_first(t[jt], h, b0, b1);
      else mma16(t[jt], h, b0, b1);
      mma16(t[jt], l, b0, b1);
    }
  }
}

}  // namespace mf
