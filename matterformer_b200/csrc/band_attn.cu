// Local-window attention, bf16, head_dim 64, windows of 32, 64 and 128: query i sees keys i - w/2 .. i + w/2 - 1
// (same operator as sparse_attn_mma.cu, which serves the other shapes).
//
// A band is short, so a tile's whole neighbourhood fits shared memory: a CTA owns kRows rows and loads them with the w/2 rows
// before and after, once.  A warp owns 16 rows; the w + 16 partner rows that they can see are w/16 + 1 chunks of 16 with a
// fixed pattern: the first and the last chunk are triangles, everything between is visible, so no bitmaps, no walk and no
// masks except at the ends of a structure.  Forward: no running maximum (the softmax shift is 0 unless a row's sum leaves
// 2^-60 .. 2^60; then the warp looks for its maxima and starts over).  Backward: one launch; the warp's 16 rows first as
// queries (dq), then as keys (dk, dv), from the same shared rows; delta = dO . out is formed on load.  Every output row has
// one owner: no atomics, bit-identical reruns.
//
// W = 0: structures of at most 32 tokens under a window that reaches every pair (a trunk's molecules).  The halo is the tile itself,
// a warp sees two chunks, and nothing but the structure's end is masked.  1 024 molecules of 9 - 29 tokens x 8
// heads: forward 37 -> 25 us, backward 104 -> 53 us (two launches of the 32-row walk before).
//
// What bounds it: issue slots and the L1 / shared-memory path (operand fragments, at 16 rows per warp), while a CTA's loads overlap only
// with the other CTAs of the SM.  The 128-row tiles arrive by bulk tensor copies: as 16-byte copies of the threads they took a
// quarter of the forward kernel's instructions and a share of the L1 path; 64-row tiles, which serve calls of a few microseconds,
// keep those (a map is encoded on the host for each call).  Interior chunks take no masks and two elements an instruction.  32 cells of
// 4096 tokens x 8 heads, window 64: forward 144 -> 117 us, backward 381 -> 317 us (HBM floors 82 and 164 us); window 32 125 -> 102 and
// 342 -> 248, window 128 207 -> 167 and 779 -> 681.  The 32-row walk with its three passes: 219 and 311 + 322 us at window 64.
#include "common.cuh"
#include "simplicial_warp.cuh"
#include "sm100_primitives.cuh"
#include "tensor_map.cuh"

namespace mf {
namespace {

struct BandParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  const __nv_bfloat16* grad_out;
  const int32_t* num_atoms;
  __nv_bfloat16* out;  // backward: read
  float* lse;
  __nv_bfloat16* dq;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int H, N;
  float scale;
  RowLayout in, act;  // rows of q, k, v and their gradients; rows of out and grad_out
  BoundedWaits waits; // of the tiles that arrive by bulk copies (kind 0)
};

__device__ int32_t g_band_status = 0;  // MF_ERR_DEVICE_TIMEOUT after an expired wait

// The wide tiles bring their rows by bulk tensor copies, which zero what lies outside [0, N): forward k, v, q, backward q, k, v, dO.
struct BandMaps {
  CUtensorMap m[4];
};
struct NoMaps {};
template <int kRows>
using MapsOf = std::conditional_t<kRows == 128, BandMaps, NoMaps>;

// Waits for the copies on `bar` and clears the rows of `tiles` tiles that lie in [n, N) (they may hold NaN).  False: the wait expired,
// for every thread alike; the CTA then writes zeros (clear_rows) and ends.
template <int kThreads, int kTiles>
__device__ __forceinline__ bool tiles_arrived(uint64_t* bar, uint8_t* smem, const int (&at)[kTiles], const int (&first)[kTiles],
                                              const int (&rows)[kTiles], int n, const BoundedWaits& waits) {
  bool ok = mbar_wait_for(bar, 0, waits.limit);
  if (!ok) ok = mbar_wait(bar, 0);  // the copies write to this CTA: none is in flight when it gives up
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) atomicExch(&g_band_status, MF_ERR_DEVICE_TIMEOUT);
    return false;
  }
  bool edge = false;
#pragma unroll
  for (int t = 0; t < kTiles; ++t) {
    if (first[t] + rows[t] <= n) continue;
    edge = true;
    for (int idx = threadIdx.x + 8 * max(n - first[t], 0); idx < 8 * rows[t]; idx += kThreads)
      *reinterpret_cast<uint4*>(smem + at[t] + 16 * idx) = make_uint4(0u, 0u, 0u, 0u);
  }
  if (edge) __syncthreads();  // (the same for all threads)
  return true;
}

// rows [first, first + rows) of one head that lie below N
template <int kThreads>
__device__ __forceinline__ void clear_rows(__nv_bfloat16* dst, long long stride, int first, int rows, int N) {
  for (int idx = threadIdx.x; idx < 8 * min(rows, N - first); idx += kThreads)
    *reinterpret_cast<uint4*>(dst + (first + (idx >> 3)) * stride + (idx & 7) * 8) = make_uint4(0u, 0u, 0u, 0u);
}

// rows [first, first + rows) of one head into a swizzled tile; rows outside [0, n) become zeros
template <int kThreads>
__device__ __forceinline__ void load_band(uint32_t tile, const __nv_bfloat16* src, long long stride, int first, int rows, int n) {
  for (int idx = threadIdx.x; idx < rows * 8; idx += kThreads) {
    const int r = idx >> 3, c = idx & 7, row = first + r;
    const bool ok = row >= 0 && row < n;
    cp_async16(row_chunk(tile, r, c), src + (ok ? row : 0) * stride + c * 8, ok);
  }
}

// c (16 x 16) = A (16 x 64, fragments) . 16 rows of the tile from byte offset `at`
__device__ __forceinline__ void chunk_product(float (&c)[2][4], const uint32_t (&a)[4][4], const FragBase& fb, int at) {
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int kp = 0; kp < 2; ++kp) {
      uint32_t b[4];
      load_b(b, fb, at, nt, kp);
      if (kp == 0) mma16_first(c[nt], a[0], b[0], b[1]);
      else mma16(c[nt], a[2], b[0], b[1]);
      mma16(c[nt], a[2 * kp + 1], b[2], b[3]);
    }
}
// acc (16 x 64) += P (16 x 16, packed as an A operand) . rows of the chunk
__device__ __forceinline__ void chunk_accumulate(float (&acc)[8][4], const uint32_t (&p)[4], const FragBase& fb, int at) {
#pragma unroll
  for (int dp = 0; dp < 4; ++dp) {
    uint32_t b[4];
    load_t2(b, fb, at, dp, 0);
    mma16(acc[2 * dp], p, b[0], b[1]);
    mma16(acc[2 * dp + 1], p, b[2], b[3]);
  }
}
__device__ __forceinline__ void pack_chunk(uint32_t (&p)[4], const float (&s)[2][4]) {
  p[0] = pack2_bf16(s[0][0], s[0][1]);
  p[1] = pack2_bf16(s[0][2], s[0][3]);
  p[2] = pack2_bf16(s[1][0], s[1][1]);
  p[3] = pack2_bf16(s[1][2], s[1][3]);
}
// 16 x 64 accumulator to bf16 rows; rows at or beyond N are skipped.  The four lanes of a row exchange their words first (a
// 4 x 4 transposition), so that a lane stores 16 bytes: stored as they are, every instruction touches eight rows in pieces
// of 16 bytes, and these pieces, not the arithmetic, filled the load/store pipe.
__device__ __forceinline__ void store_rows(__nv_bfloat16* dst, long long stride, const float (&acc)[8][4], int row, int N, float lo,
                                           float hi) {
  const int quad = threadIdx.x & 3;
  const bool q0 = quad & 1, q1 = quad >> 1;
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const float mul = hh ? hi : lo;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t w[4];  // tiles 4 half + t; after the exchange: tile 4 half + quad, columns 2 t, 2 t + 1
#pragma unroll
      for (int t = 0; t < 4; ++t) w[t] = pack2_bf16(acc[4 * half + t][2 * hh] * mul, acc[4 * half + t][2 * hh + 1] * mul);
#pragma unroll
      for (int t = 0; t < 2; ++t) {  // across quad bit 0: tiles 2 t and 2 t + 1
        const uint32_t other = __shfl_xor_sync(0xffffffffu, q0 ? w[2 * t] : w[2 * t + 1], 1);
        if (q0) w[2 * t] = other; else w[2 * t + 1] = other;
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) {  // across quad bit 1: tiles t and t + 2
        const uint32_t other = __shfl_xor_sync(0xffffffffu, q1 ? w[t] : w[t + 2], 2);
        if (q1) w[t] = other; else w[t + 2] = other;
      }
      if (row + 8 * hh < N)
        *reinterpret_cast<uint4*>(dst + (row + 8 * hh) * stride + 32 * half + 8 * quad) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

template <int W, int kRows>
__global__ void __launch_bounds__(kRows * 2, W == 0 ? 12 : W == 128 ? (kRows == 128 ? 2 : 4) : (kRows == 128 ? 3 : 6)) band_fwd_kernel(const __grid_constant__ BandParams p, const __grid_constant__ MapsOf<kRows> maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  wait_for_previous();
  constexpr bool kDense = W == 0;
  constexpr int kHalf = W / 2, kHalo = kRows + W, kThreads = kRows * 2, kChunks = kDense ? kRows / 16 : W / 16 + 1;
  constexpr int kTv = kHalo * kRowBytes, kTq = 2 * kTv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2;
  const int t0 = blockIdx.x * kRows, bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H, N = p.N;
  const int n = min(p.num_atoms[b], N);
  const uint32_t tile = (uint32_t)__cvta_generic_to_shared(smem);
  const long long in0 = p.in.at(b, h, 0), act0 = p.act.at(b, h, 0);
  if (t0 < n) {
    if constexpr (kRows == 128) {
      uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kTq + kRows * kRowBytes);
      if (threadIdx.x == 0) {
        mbar_init(bar, 1 + (p.waits.withheld == 0));
        mbar_fence_init();
        mbar_arrive_expect_tx(bar, (2 * kHalo + kRows) * kRowBytes);
        tma_load_strided_rows(tile, &maps.m[0], t0 - kHalf, h, b, bar);
        tma_load_strided_rows(tile + kTq, &maps.m[2], t0, h, b, bar);
        tma_load_strided_rows(tile + kTv, &maps.m[1], t0 - kHalf, h, b, bar);
      }
      __syncthreads();
      if (!tiles_arrived<kThreads, 3>(bar, smem, {0, kTv, kTq}, {t0 - kHalf, t0 - kHalf, t0}, {kHalo, kHalo, kRows}, n, p.waits)) {
        clear_rows<kThreads>(p.out + act0, p.act.token, t0, kRows, N);
        for (int i = threadIdx.x; i < min(kRows, N - t0); i += kThreads) p.lse[(size_t)bh * N + t0 + i] = 0.f;
        return;
      }
    } else {
      load_band<kThreads>(tile, p.k + in0, p.in.token, t0 - kHalf, kHalo, n);
      load_band<kThreads>(tile + kTq, p.q + in0, p.in.token, t0, kRows, n);
      load_band<kThreads>(tile + kTv, p.v + in0, p.in.token, t0 - kHalf, kHalo, n);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
    }
  }
  const int i0 = t0 + warp * 16, row = i0 + row8;  // the lane's rows: row and row + 8
  if (i0 >= N) return;
  // everything a warp reads lies at fixed offsets from its rows (dense: from the structure's first)
  const FragBase fb(tile + (kDense ? 0 : warp * 16 * kRowBytes), lane);
  const int mine = kDense ? warp * 16 * kRowBytes : 0;
  float o[8][4], l[2] = {0.f, 0.f}, shift[2] = {0.f, 0.f};
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[t][e] = 0.f;
  if (i0 < n) {
    uint32_t q[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) load_a(q[ks], fb, kTq + mine, 0, ks);
    const float sc2 = p.scale * kLog2e;
    // sets the hidden pairs of chunk c: the two triangles, and keys outside the structure
    auto hide = [&](float(&s)[2][4], int c, float value) {
      const int key0 = kDense ? 16 * c : i0 - kHalf + 16 * c;
      const bool ends = key0 < 0 || key0 + 16 > n;
      if (!ends && (kDense || (c != 0 && c != kChunks - 1))) return;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = row8 + 8 * (e >> 1), rel = nt * 8 + 2 * quad + (e & 1);
          bool seen = key0 + rel >= 0 && key0 + rel < n;
          if (!kDense && c == 0) seen = seen && rel >= r;
          if (!kDense && c == kChunks - 1) seen = seen && rel < r;
          if (!seen) s[nt][e] = value;
        }
    };
    for (bool exact = false;; exact = true) {
      if (exact) {
        float m[2] = {-INFINITY, -INFINITY};
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c) {
          float s[2][4];
          chunk_product(s, q, fb, c * 16 * kRowBytes);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[nt][e] *= sc2;
          hide(s, c, -INFINITY);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e >> 1] = fmaxf(m[e >> 1], s[nt][e]);
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          m[hh] = fmaxf(m[hh], __shfl_xor_sync(0xffffffffu, m[hh], 1));
          m[hh] = fmaxf(m[hh], __shfl_xor_sync(0xffffffffu, m[hh], 2));
          shift[hh] = m[hh] > -INFINITY ? m[hh] : 0.f;
        }
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[t][e] = 0.f;
      }
      float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      const float2 factor = make_float2(sc2, sc2);
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        float s[2][4];
        chunk_product(s, q, fb, c * 16 * kRowBytes);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const float2 x = fma2(make_float2(s[nt][2 * hh], s[nt][2 * hh + 1]), factor, make_float2(-shift[hh], -shift[hh]));
            s[nt][2 * hh] = fast_exp2(x.x), s[nt][2 * hh + 1] = fast_exp2(x.y);
          }
        hide(s, c, 0.f);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) l2[hh] = add2(l2[hh], make_float2(s[nt][2 * hh], s[nt][2 * hh + 1]));
        uint32_t pk[4];
        pack_chunk(pk, s);
        chunk_accumulate(o, pk, fb, kTv + c * 16 * kRowBytes);
      }
      bool fine = true;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        l[hh] = l2[hh].x + l2[hh].y;
        quad_reduce(l[hh]);
        if (row + 8 * hh < n) fine = fine && l[hh] >= kSumLow && l[hh] <= kSumHigh;
      }
      if (exact || __all_sync(0xffffffffu, fine)) break;
    }
  }
  float inv[2];
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const bool have = row + 8 * hh < n && l[hh] != 0.f;
    inv[hh] = have ? 1.f / l[hh] : 0.f;
    if (quad == 0 && row + 8 * hh < N) p.lse[(size_t)bh * N + row + 8 * hh] = have ? (shift[hh] + log2f(l[hh])) * kLn2 : 0.f;
  }
  store_rows(p.out + act0, p.act.token, o, row, N, inv[0], inv[1]);
}

template <int W, int kRows>
__global__ void __launch_bounds__(kRows * 2, W == 0 ? 6 : kRows == 128 ? (W == 128 ? 1 : 2) : (W == 128 ? 2 : 3)) band_bwd_kernel(const __grid_constant__ BandParams p, const __grid_constant__ MapsOf<kRows> maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  wait_for_previous();
  constexpr bool kDense = W == 0;
  constexpr int kHalf = W / 2, kHalo = kRows + W, kThreads = kRows * 2, kChunks = kDense ? kRows / 16 : W / 16 + 1;
  constexpr int kTk = kHalo * kRowBytes, kTv = 2 * kTk, kTg = 3 * kTk;  // q, k, v, grad_out
  float* lse = reinterpret_cast<float*>(smem + 4 * kTk);  // of the halo rows, in the log2 domain
  float* delta = lse + kHalo;
  [[maybe_unused]] uint64_t* bar = reinterpret_cast<uint64_t*>(delta + kHalo);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2;
  const int t0 = blockIdx.x * kRows, first = t0 - kHalf, bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H, N = p.N;
  const int n = min(p.num_atoms[b], N);
  const uint32_t tile = (uint32_t)__cvta_generic_to_shared(smem);
  const long long in0 = p.in.at(b, h, 0), act0 = p.act.at(b, h, 0);
  if (t0 < n) {
    if constexpr (kRows == 128) {
      if (threadIdx.x == 0) {
        mbar_init(bar, 1 + (p.waits.withheld == 0));
        mbar_fence_init();
        mbar_arrive_expect_tx(bar, 4 * kHalo * kRowBytes);
#pragma unroll
        for (int t = 0; t < 4; ++t) tma_load_strided_rows(tile + t * kTk, &maps.m[t], first, h, b, bar);
      }
    } else {
      load_band<kThreads>(tile + kTg, p.grad_out + act0, p.act.token, first, kHalo, n);
      load_band<kThreads>(tile, p.q + in0, p.in.token, first, kHalo, n);
      load_band<kThreads>(tile + kTk, p.k + in0, p.in.token, first, kHalo, n);
      load_band<kThreads>(tile + kTv, p.v + in0, p.in.token, first, kHalo, n);
      cp_async_commit();
    }
    // delta of the halo rows, eight lanes per row, all loads first (of dO their own ones, or the tile once it is there)
    constexpr int kSteps = kHalo * 8 / kThreads;
    static_assert(kHalo * 8 % kThreads == 0, "whole steps");
    uint4 x[kSteps], g[kSteps];
    float ls[kSteps];
    const int r0 = threadIdx.x >> 3, c = threadIdx.x & 7;
#pragma unroll
    for (int t = 0; t < kSteps; ++t) {
      const int row = first + r0 + t * (kThreads / 8);
      x[t] = g[t] = make_uint4(0u, 0u, 0u, 0u);
      ls[t] = INFINITY;  // no weight for rows outside the structure
      if (row >= 0 && row < n) {
        x[t] = *reinterpret_cast<const uint4*>(p.out + act0 + row * p.act.token + c * 8);
        if constexpr (kRows != 128) g[t] = *reinterpret_cast<const uint4*>(p.grad_out + act0 + row * p.act.token + c * 8);
        if (c == 0) ls[t] = p.lse[(size_t)bh * N + row] * kLog2e;
      }
    }
    if constexpr (kRows == 128) {
      __syncthreads();  // the barrier exists
      if (!tiles_arrived<kThreads, 4>(bar, smem, {0, kTk, kTv, kTg}, {first, first, first, first}, {kHalo, kHalo, kHalo, kHalo}, n, p.waits)) {
        clear_rows<kThreads>(p.dq + in0, p.in.token, t0, kRows, N);
        clear_rows<kThreads>(p.dk + in0, p.in.token, t0, kRows, N);
        clear_rows<kThreads>(p.dv + in0, p.in.token, t0, kRows, N);
        return;
      }
#pragma unroll
      for (int t = 0; t < kSteps; ++t) g[t] = *reinterpret_cast<const uint4*>(smem + row_chunk(kTg, r0 + t * (kThreads / 8), c));
    }
#pragma unroll
    for (int t = 0; t < kSteps; ++t) {
      float d = fmaf(bf16_lo(x[t].x), bf16_lo(g[t].x), bf16_hi(x[t].x) * bf16_hi(g[t].x));
      d = fmaf(bf16_lo(x[t].y), bf16_lo(g[t].y), fmaf(bf16_hi(x[t].y), bf16_hi(g[t].y), d));
      d = fmaf(bf16_lo(x[t].z), bf16_lo(g[t].z), fmaf(bf16_hi(x[t].z), bf16_hi(g[t].z), d));
      d = fmaf(bf16_lo(x[t].w), bf16_lo(g[t].w), fmaf(bf16_hi(x[t].w), bf16_hi(g[t].w), d));
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      if (c == 0) {
        delta[r0 + t * (kThreads / 8)] = d;
        lse[r0 + t * (kThreads / 8)] = ls[t];
      }
    }
    if constexpr (kRows != 128) cp_async_wait<0>();
    __syncthreads();
  }
  const int i0 = t0 + warp * 16, row = i0 + row8;
  if (i0 >= N) return;
  // everything a warp reads lies at fixed offsets from its rows (dense: from the structure's first)
  const FragBase fb(tile + (kDense ? 0 : warp * 16 * kRowBytes), lane);
  const int mine = kDense ? warp * 16 * kRowBytes : 0;
  const int own = kHalf * kRowBytes + mine;  // the warp's rows inside the halo
  const float2 factor = make_float2(p.scale * kLog2e, p.scale * kLog2e);
  uint32_t a[4][4], g[4][4];
  float acc0[8][4], acc1[8][4];
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc0[t][e] = 0.f;
  if (i0 < n) {  // ---- the rows as queries.  (Keys outside the structure have zero rows: whatever weight they get meets zeros.)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) load_a(a[ks], fb, own, 0, ks), load_a(g[ks], fb, kTg + own, 0, ks);
    const int r0 = warp * 16 + kHalf + row8;
    const float la = lse[r0], lb = lse[r0 + 8], da = delta[r0], db = delta[r0 + 8];
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const int at = c * 16 * kRowBytes;
      float s[2][4], dp[2][4];
      chunk_product(s, a, fb, kTk + at);
      chunk_product(dp, g, fb, kTv + at);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float lr = hh ? lb : la, dr = hh ? db : da;
          const float2 x = fma2(make_float2(s[nt][2 * hh], s[nt][2 * hh + 1]), factor, make_float2(-lr, -lr));
          // a logit of 0 against zero rows may give a huge weight where the row's log-sum-exp is very negative: bounded, so
          // that it stays finite and 0 . weight = 0
          float2 pr = make_float2(fast_exp2(fminf(x.x, 100.f)), fast_exp2(fminf(x.y, 100.f)));
          const int r = row8 + 8 * hh, rel = nt * 8 + 2 * quad;
          if (!kDense && c == 0) pr.x = rel < r ? 0.f : pr.x, pr.y = rel + 1 < r ? 0.f : pr.y;
          if (!kDense && c == kChunks - 1) pr.x = rel >= r ? 0.f : pr.x, pr.y = rel + 1 >= r ? 0.f : pr.y;
          pr = mul2(pr, add2(make_float2(dp[nt][2 * hh], dp[nt][2 * hh + 1]), make_float2(-dr, -dr)));
          s[nt][2 * hh] = pr.x, s[nt][2 * hh + 1] = pr.y;  // (the scale comes with the sums)
        }
      uint32_t pk[4];
      pack_chunk(pk, s);
      chunk_accumulate(acc0, pk, fb, kTk + at);
    }
  }
  store_rows(p.dq + in0, p.in.token, acc0, row, N, row < n ? p.scale : 0.f, row + 8 < n ? p.scale : 0.f);
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc0[t][e] = acc1[t][e] = 0.f;
  if (i0 < n) {  // ---- the rows as keys: key j is seen by queries j - w/2 + 1 .. j + w/2
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) load_a(a[ks], fb, kTk + own, 0, ks), load_a(g[ks], fb, kTv + own, 0, ks);
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const int at = c * 16 * kRowBytes;
      float s[2][4], dp[2][4];
      chunk_product(s, a, fb, at);
      chunk_product(dp, g, fb, kTg + at);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int q0 = ((kDense ? 0 : warp) + c) * 16 + nt * 8 + 2 * quad;
        const float2 l = *reinterpret_cast<const float2*>(&lse[q0]), d = *reinterpret_cast<const float2*>(&delta[q0]);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float2 x = fma2(make_float2(s[nt][2 * hh], s[nt][2 * hh + 1]), factor, make_float2(-l.x, -l.y));
          float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          const int r = row8 + 8 * hh, rel = nt * 8 + 2 * quad;
          if (!kDense && c == 0) pr.x = rel <= r ? 0.f : pr.x, pr.y = rel + 1 <= r ? 0.f : pr.y;
          if (!kDense && c == kChunks - 1) pr.x = rel > r ? 0.f : pr.x, pr.y = rel + 1 > r ? 0.f : pr.y;
          s[nt][2 * hh] = pr.x, s[nt][2 * hh + 1] = pr.y;
          pr = mul2(pr, add2(make_float2(dp[nt][2 * hh], dp[nt][2 * hh + 1]), make_float2(-d.x, -d.y)));
          dp[nt][2 * hh] = pr.x, dp[nt][2 * hh + 1] = pr.y;
        }
      }
      uint32_t pk[4];
      pack_chunk(pk, s);
      chunk_accumulate(acc1, pk, fb, kTg + at);  // dv += P^T dO
      pack_chunk(pk, dp);
      chunk_accumulate(acc0, pk, fb, at);        // dk += dS^T Q
    }
  }
  const bool lo = row < n, hi = row + 8 < n;
#pragma unroll
  for (int t = 0; t < 8; ++t)  // (selected, not multiplied: a row beyond the structure may have met an infinite weight)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (!(e < 2 ? lo : hi)) acc0[t][e] = acc1[t][e] = 0.f;
  store_rows(p.dk + in0, p.in.token, acc0, row, N, p.scale, p.scale);
  store_rows(p.dv + in0, p.in.token, acc1, row, N, 1.f, 1.f);
}

// *done: whether the launch was made; tiles of 128 rows need maps of their tensors.
template <int W, int kRows>
int launch_band(const BandParams& p, int B, bool backward, cudaStream_t s, bool* done = nullptr) {
  constexpr int halo = (kRows + W) * kRowBytes;
  const int bytes = 16 + (backward ? 4 * halo + (kRows + W) * 8 : 2 * halo + kRows * kRowBytes);
  MapsOf<kRows> maps{};
  if constexpr (kRows == 128) {
    const __nv_bfloat16* src[4] = {backward ? p.q : p.k, backward ? p.k : p.v, backward ? p.v : p.q, backward ? p.grad_out : nullptr};
    *done = true;
    for (int t = 0; t < (backward ? 4 : 3); ++t) {
      const RowLayout& l = t == 3 ? p.act : p.in;
      *done = *done && make_strided_rows_tensor_map(&maps.m[t], src[t], p.N, {p.H, B}, l.token, {l.head, l.batch},
                                                    !backward && t == 2 ? kRows : kRows + W);
    }
    if (!*done) return MF_OK;
  }
  auto kernel = backward ? band_bwd_kernel<W, kRows> : band_fwd_kernel<W, kRows>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(band_attn_kernel)");
  launch_dependent(kernel, dim3((p.N + kRows - 1) / kRows, B * p.H), dim3(kRows * 2), bytes, s, p, maps);
  MF_CHECK_LAUNCH("band_attn_kernel");
  return MF_OK;
}
template <int W>
int launch_either(const BandParams& p, int B, bool wide, bool backward, cudaStream_t s) {
  bool done = false;
  const int rc = wide ? launch_band<W, 128>(p, B, backward, s, &done) : MF_OK;
  return rc != MF_OK || done ? rc : launch_band<W, 64>(p, B, backward, s);
}

}  // namespace

// Windows whose chunks are whole, structures long enough that a tile is not mostly halo, or short enough that the window
// reaches every pair of a 32-row tile; those between stay on the 32-row walk.  Forward + backward of 64 structures x 8 heads,
// walk | band: 96 tokens 42 | 33 us (window 32), 44 | 44 (64), 49 | 66 (128).  Under a window of 128 a tile is mostly halo up
// to 192 tokens: 87 | 100 us at 160, 107 | 106 at 192, 145 | 126 at 256; there the band serves calls whose tiles are all
// resident at once, two to an SM (4 structures of 160: 23 | 17), where the walk's three launches cost more than the halo.
constexpr int kDenseTokens = 32;  // under windows of 64 and 128
bool band_attn_applies(const MfSparseAttnArgs& a) {
  if (a.dtype != MF_DTYPE_BF16 || a.head_dim != 64) return false;
  if (a.tokens <= kDenseTokens) return a.window == 64 || a.window == 128;
  if (a.tokens < 96) return false;
  if (a.window == 128) return a.tokens >= 192 || (long long)a.batch * a.heads * ((a.tokens + 63) / 64) <= 2 * 148;
  return a.window == 32 || a.window == 64;
}

// 128-row tiles re-read half as much halo; 64-row ones spread a call over twice as many CTAs, which pays while the wide ones
// would not cover the chip.  Forward + backward at window 64, 64 | 128 rows: 8 structures of 128 tokens (64 wide tiles) 14.7 |
// 16.3 us, 128 tiles 17.3 | 16.4, 256 tiles 29.1 | 22.5, 576 tiles 50.4 | 42.2; windows 32 and 128 turn at the same place.
bool band_attn_wide(const MfSparseAttnArgs& a) {
  return a.tokens > kDenseTokens && (long long)a.batch * a.heads * ((a.tokens + 127) / 128) >= 128;
}

int band_attn(const MfSparseAttnArgs& a, const RowLayout* layouts, bool backward, cudaStream_t stream, BoundedWaits waits) {
  BandParams p{};
  p.waits = waits;
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.k = static_cast<const __nv_bfloat16*>(a.k);
  p.v = static_cast<const __nv_bfloat16*>(a.v);
  p.grad_out = static_cast<const __nv_bfloat16*>(a.grad_out);
  p.num_atoms = a.num_atoms;
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.lse = a.lse;
  p.dq = static_cast<__nv_bfloat16*>(a.dq);
  p.dk = static_cast<__nv_bfloat16*>(a.dk);
  p.dv = static_cast<__nv_bfloat16*>(a.dv);
  p.H = a.heads, p.N = a.tokens, p.scale = a.scale;
  p.in = layouts ? layouts[0] : contiguous_rows(a.heads, a.tokens);
  p.act = layouts ? layouts[1] : contiguous_rows(a.heads, a.tokens);
  if (a.tokens <= kDenseTokens) return launch_band<0, kDenseTokens>(p, a.batch, backward, stream);
  const bool wide = band_attn_wide(a);
  switch (a.window) {
    case 32: return launch_either<32>(p, a.batch, wide, backward, stream);
    case 64: return launch_either<64>(p, a.batch, wide, backward, stream);
    default: return launch_either<128>(p, a.batch, wide, backward, stream);
  }
}

int band_attn_status(int32_t* host_status, cudaStream_t stream, bool clear) {
  cudaError_t e = cudaMemcpyFromSymbolAsync(host_status, g_band_status, sizeof(int32_t), 0, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  constexpr int32_t kNone = MF_OK;
  if (e == cudaSuccess && clear) e = cudaMemcpyToSymbolAsync(g_band_status, &kNone, sizeof(int32_t), 0, cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess && clear) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_error(e, "band attention status read-back");
  return MF_OK;
}

}  // namespace mf
