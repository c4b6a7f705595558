// 2-simplicial attention, forward, for molecules of at most 32 tokens in bf16 (see simplicial_warp.cuh).
//
// A CTA holds one (batch, head) in shared memory; a warp owns 16 queries, whose q fragments and all k2 fragments stay in
// registers, and walks over the first keys j: S = (Q o k1_j) K2^T (16 x 32 logits, 16 registers), P = exp2(S), repacked in
// place as the A operand of W = P V2, out += v1_j o W.  Row sums stay per lane until the end, and no running maximum is
// needed (see kSumLow), so a step has no cross-lane operation and no barrier.  Small batches give a row tile to several
// warps, which take every second or fourth j and are added up in a fixed order.
//
// What bounds it: instruction issue of the softmax next to the mma.sync pipe (43 % busy at 1024 molecules of 9-29 atoms x 8
// heads).  Measured there: 140 us, against 358 us for tcgen05 tiles that put four heads on the 128 rows of a tile (every
// row then meets the keys of all four heads, and a step passes through tensor memory with four barrier waits); one query per
// step with the keys on both sides of the product (so that sums need shuffles in every step) took 195 us.
#include "common.cuh"
#include "simplicial.cuh"
#include "simplicial_warp.cuh"

namespace mf {
namespace {

struct SmallFwdParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k1;
  const __nv_bfloat16* v1;
  const __nv_bfloat16* k2;
  const __nv_bfloat16* v2;
  const uint8_t* query_valid;
  const uint8_t* key_valid;
  const uint8_t* pair_valid;
  const float* u;  // factorized bias gate_i * ((u_ij + v_ik) + w_jk)
  const float* v_bias;
  const float* w;
  const float* gate;
  float* out;
  float* lse;
  __nv_bfloat16* out_cast;
  int H, N;
  const int32_t* order;  // heavy molecules first, or NULL
  float q_scale;
  RowLayout in, act;
};

template <bool kBias>
struct SmallFwdShared {
  __align__(128) uint8_t tile[5][kSmallTile];   // q, k2, k1, v1, v2
  float u[kBias ? kSmallRows : 1][33];          // bias u_ij
  float v[kBias ? kSmallRows : 1][33];          // bias v_ik
  float gate[kBias ? kSmallRows : 1];
  float w[kBias ? kSmallRows : 1][kSmallRows];  // bias w_jk
  uint32_t visible[kSmallRows];                 // bit k of word j: the pair (j, k) counts
};

// What a warp keeps over the walk: its 16 queries and all second keys, as operands of the logit product.
template <int NT, bool kBias>
struct SmallFwdRows {
  uint32_t q[4][4];
  uint32_t k2[NT][2][4];
  float v[kBias ? NT : 1][4];  // bias v_ik in the layout of the logits
  float gate[2];
};

// Logits of the warp's 16 queries against the pairs (j, k); hidden pairs are -inf.
template <int NT, bool kHoles, bool kBias>
__device__ __forceinline__ void small_logits(float (&s)[NT][4], const SmallFwdShared<kBias>& sm, const SmallFwdRows<NT, kBias>& r,
                                             uint32_t k1, int mt, int j, int n) {
  const int lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2;
  uint32_t kf[8];
  load_row_pairs(kf, k1, j, lane);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    uint32_t a[4] = {mul_bf16x2(r.q[ks][0], kf[2 * ks]), mul_bf16x2(r.q[ks][1], kf[2 * ks]),
                     mul_bf16x2(r.q[ks][2], kf[2 * ks + 1]), mul_bf16x2(r.q[ks][3], kf[2 * ks + 1])};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const uint32_t b0 = r.k2[nt][ks >> 1][2 * (ks & 1)], b1 = r.k2[nt][ks >> 1][2 * (ks & 1) + 1];
      if (ks == 0) mma16_first(s[nt], a, b0, b1);
      else mma16(s[nt], a, b0, b1);
    }
  }
  if constexpr (kBias) {
    const float ua = sm.u[mt * 16 + row8][j], ub = sm.u[mt * 16 + 8 + row8][j];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const float2 w = *reinterpret_cast<const float2*>(&sm.w[j][nt * 8 + 2 * quad]);
      const float2 x = add2(add2(make_float2(ua, ua), make_float2(r.v[nt][0], r.v[nt][1])), w);
      const float2 y = add2(add2(make_float2(ub, ub), make_float2(r.v[nt][2], r.v[nt][3])), w);
      s[nt][0] = fmaf(r.gate[0], x.x, s[nt][0]);
      s[nt][1] = fmaf(r.gate[0], x.y, s[nt][1]);
      s[nt][2] = fmaf(r.gate[1], y.x, s[nt][2]);
      s[nt][3] = fmaf(r.gate[1], y.y, s[nt][3]);
    }
  }
  if constexpr (kHoles) {
    const uint32_t word = sm.visible[j] >> (2 * quad);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (!((word >> (nt * 8)) & 1u)) s[nt][0] = -INFINITY, s[nt][2] = -INFINITY;
      if (!((word >> (nt * 8 + 1)) & 1u)) s[nt][1] = -INFINITY, s[nt][3] = -INFINITY;
    }
  } else {  // only the last 8-key column tile is partly hidden
    if ((NT - 1) * 8 + 2 * quad >= n) s[NT - 1][0] = -INFINITY, s[NT - 1][2] = -INFINITY;
    if ((NT - 1) * 8 + 2 * quad + 1 >= n) s[NT - 1][1] = -INFINITY, s[NT - 1][3] = -INFINITY;
  }
}

// The 16 queries of row tile `mt` against the first keys js, js + JS, ...; JS warps share a row tile and are added up.
template <int NT, bool kHoles, bool kBias, int kWarps>
__device__ __forceinline__ void small_fwd_rows(const SmallFwdParams& p, SmallFwdShared<kBias>& sm, int b, int h, int n,
                                               uint32_t qmask) {
  constexpr int KS = (NT + 1) / 2;  // 16-key steps of the second product
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2;
  const int N = p.N, bh = b * p.H + h, nq = 32 - __clz(qmask);
  const int row_tiles = (nq + 15) >> 4, JS = kWarps / row_tiles;
  const int mt = warp % row_tiles, js = warp / row_tiles;
  const uint32_t qt = (uint32_t)__cvta_generic_to_shared(sm.tile[0]), k1 = qt + 2 * kSmallTile, v1 = qt + 3 * kSmallTile;
  const FragBase fb(qt, lane);
  SmallFwdRows<NT, kBias> r;
  const uint32_t scale2 = pack2_bf16(p.q_scale, p.q_scale);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    load_a(r.q[ks], fb, 0, mt, ks);
#pragma unroll
    for (int e = 0; e < 4; ++e) r.q[ks][e] = mul_bf16x2(r.q[ks][e], scale2);
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int kp = 0; kp < 2; ++kp) load_b(r.k2[nt][kp], fb, kSmallTile, nt, kp);
  const int ia = mt * 16 + row8, ib = ia + 8;
  if constexpr (kBias) {
    r.gate[0] = sm.gate[ia], r.gate[1] = sm.gate[ib];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) r.v[nt][e] = sm.v[e < 2 ? ia : ib][nt * 8 + 2 * quad + (e & 1)];
  }
  // q and k2 live in registers from here on; their place takes the v1 rows in fp32
  float(&v1f)[kSmallRows][kD] = *reinterpret_cast<float(*)[kSmallRows][kD]>(sm.tile[0]);
  __syncthreads();
  for (int idx = threadIdx.x; idx < n * 8; idx += 32 * kWarps) {
    const int j = idx >> 3, c = idx & 7;
    uint4 x;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(row_chunk(v1, j, c)));
    *reinterpret_cast<float4*>(&v1f[j][8 * c]) = make_float4(bf16_lo(x.x), bf16_hi(x.x), bf16_lo(x.y), bf16_hi(x.y));
    *reinterpret_cast<float4*>(&v1f[j][8 * c + 4]) = make_float4(bf16_lo(x.z), bf16_hi(x.z), bf16_lo(x.w), bf16_hi(x.w));
  }
  __syncthreads();

  float2 o[8][2], l[2];  // [8-channel tile][row ia / ib]
  float shift[2] = {0.f, 0.f};
  const float2 zero2 = make_float2(0.f, 0.f);
  bool exact = false;
  while (true) {
#pragma unroll
    for (int t = 0; t < 8; ++t) o[t][0] = o[t][1] = zero2;
    l[0] = l[1] = zero2;
    if (js < JS) {
      for (int j = js; j < n; j += JS) {
        if (sm.visible[j] == 0u) continue;
        float s[NT][4];
        small_logits<NT, kHoles, kBias>(s, sm, r, k1, mt, j, n);
        uint32_t pk[2 * KS][2];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float2 c = make_float2(-shift[hh], -shift[hh]), le = make_float2(kLog2e, kLog2e);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            float2 x = fma2(make_float2(s[nt][2 * hh], s[nt][2 * hh + 1]), le, c);
            x.x = fast_exp2(x.x);
            x.y = fast_exp2(x.y);
            l[hh] = add2(l[hh], x);
            pk[nt][hh] = pack2_bf16(x.x, x.y);
          }
          if (NT & 1) pk[2 * KS - 1][hh] = 0u;
        }
        // W = P V2 (16 queries x 64 channels), out += v1_j o W
#pragma unroll
        for (int dp = 0; dp < 4; ++dp) {
          float w0[4], w1[4];
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            uint32_t bv[4];
            load_t2(bv, fb, 4 * kSmallTile, dp, ks);
            const uint32_t a[4] = {pk[2 * ks][0], pk[2 * ks][1], pk[2 * ks + 1][0], pk[2 * ks + 1][1]};
            if (ks == 0) mma16_first(w0, a, bv[0], bv[1]), mma16_first(w1, a, bv[2], bv[3]);
            else mma16(w0, a, bv[0], bv[1]), mma16(w1, a, bv[2], bv[3]);
          }
          const float2 va = *reinterpret_cast<const float2*>(&v1f[j][16 * dp + 2 * quad]);
          const float2 vb = *reinterpret_cast<const float2*>(&v1f[j][16 * dp + 8 + 2 * quad]);
          o[2 * dp][0] = fma2(make_float2(w0[0], w0[1]), va, o[2 * dp][0]);
          o[2 * dp][1] = fma2(make_float2(w0[2], w0[3]), va, o[2 * dp][1]);
          o[2 * dp + 1][0] = fma2(make_float2(w1[0], w1[1]), vb, o[2 * dp + 1][0]);
          o[2 * dp + 1][1] = fma2(make_float2(w1[2], w1[3]), vb, o[2 * dp + 1][1]);
        }
      }
    }
    float ls[2];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      ls[hh] = l[hh].x + l[hh].y;
      ls[hh] += __shfl_xor_sync(0xffffffffu, ls[hh], 1);
      ls[hh] += __shfl_xor_sync(0xffffffffu, ls[hh], 2);
    }
    l[0].x = ls[0], l[1].x = ls[1];
    bool fine = true;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
      if ((qmask >> (hh ? ib : ia)) & 1u) fine &= ls[hh] >= kSumLow && ls[hh] <= kSumHigh;
    // every warp of the CTA takes part in the decision: the warps of one row tile are added up with one shift
    if (exact || __syncthreads_and(fine || js >= JS)) break;
    exact = true;
    float m[2] = {-INFINITY, -INFINITY};
    for (int j = 0; j < n; ++j) {
      if (sm.visible[j] == 0u) continue;
      float s[NT][4];
      small_logits<NT, kHoles, kBias>(s, sm, r, k1, mt, j, n);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        m[0] = fmaxf(m[0], fmaxf(s[nt][0], s[nt][1]));
        m[1] = fmaxf(m[1], fmaxf(s[nt][2], s[nt][3]));
      }
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      m[hh] = fmaxf(m[hh], __shfl_xor_sync(0xffffffffu, m[hh], 1));
      m[hh] = fmaxf(m[hh], __shfl_xor_sync(0xffffffffu, m[hh], 2));
      shift[hh] = m[hh] > -INFINITY ? m[hh] * kLog2e : 0.f;
    }
  }
  if (JS > 1) {  // the other warps of the row tile, in a fixed order, through the place of the tiles
    constexpr int kStride = 34;  // o (32) and l (2) of a lane
    float(*part)[kStride][32] = reinterpret_cast<float(*)[kStride][32]>(sm.tile[0]);
    static_assert((kWarps - 1) * kStride * 32 * 4 <= 5 * kSmallTile, "partial rows of all but one warp fit the tiles");
    __syncthreads();
    if (js > 0 && js < JS) {
      float(&mine)[kStride][32] = part[(js - 1) * row_tiles + mt];
#pragma unroll
      for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) mine[4 * t + 2 * hh][lane] = o[t][hh].x, mine[4 * t + 2 * hh + 1][lane] = o[t][hh].y;
      mine[32][lane] = l[0].x, mine[33][lane] = l[1].x;
    }
    __syncthreads();
    if (js == 0)
      for (int q = 1; q < JS; ++q) {
        const float(&other)[kStride][32] = part[(q - 1) * row_tiles + mt];
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
            o[t][hh] = add2(o[t][hh], make_float2(other[4 * t + 2 * hh][lane], other[4 * t + 2 * hh + 1][lane]));
        l[0].x += other[32][lane], l[1].x += other[33][lane];
      }
  }
  if (js == 0) {
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int i = hh ? ib : ia;
      if (i >= nq) continue;
      const float sum = l[hh].x;
      const bool have = ((qmask >> i) & 1u) && sum != 0.f;
      const float inv = have ? 1.f / sum : 0.f;
      float* out = p.out + ((size_t)bh * N + i) * kD + 2 * quad;
      __nv_bfloat16* oc = p.out_cast ? p.out_cast + p.act.at(b, h, i) + 2 * quad : nullptr;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float2 x = have ? make_float2(o[t][hh].x * inv, o[t][hh].y * inv) : zero2;
        *reinterpret_cast<float2*>(out + 8 * t) = x;
        if (oc) *reinterpret_cast<uint32_t*>(oc + 8 * t) = pack2_bf16(x.x, x.y);
      }
      if (quad == 0) p.lse[(size_t)bh * N + i] = have ? (shift[hh] + log2f(sum)) * kLn2 : 0.f;
    }
  }
}

template <bool kBias, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, kBias ? 12 / kWarps : (kWarps == 4 ? 4 : 14 / kWarps)) simplicial_small_fwd_kernel(const __grid_constant__ SmallFwdParams p) {
  __shared__ SmallFwdShared<kBias> sm;
  wait_for_previous();
  const int tid = threadIdx.x, lane = tid & 31;
  const int N = p.N, h = blockIdx.x % p.H, b = p.order ? p.order[blockIdx.x / p.H] : blockIdx.x / p.H, bh = b * p.H + h;
  const uint32_t kmask = __ballot_sync(0xffffffffu, lane < N && p.key_valid[(size_t)b * N + min(lane, N - 1)] > 0);
  const uint32_t qmask = __ballot_sync(0xffffffffu, lane < N && p.query_valid[(size_t)b * N + min(lane, N - 1)] > 0);
  const int n = 32 - __clz(kmask), nq = 32 - __clz(qmask);
  // queries beyond the last valid one, and all of them when no key is visible
  for (int idx = tid + 16 * (n > 0 ? nq : 0); idx < 16 * N; idx += 32 * kWarps) {
    const int i = idx >> 4, c = 4 * (idx & 15);
    *reinterpret_cast<float4*>(p.out + ((size_t)bh * N + i) * kD + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.out_cast) *reinterpret_cast<uint2*>(p.out_cast + p.act.at(b, h, i) + c) = make_uint2(0u, 0u);
    if (c == 0) p.lse[(size_t)bh * N + i] = 0.f;
  }
  if (n == 0 || nq == 0) return;
  {
    const __nv_bfloat16* src[5] = {p.q, p.k2, p.k1, p.v1, p.v2};
    const uint32_t t0 = (uint32_t)__cvta_generic_to_shared(sm.tile[0]);
    // a hole in a mask takes the full-size variant, which reads all rows of k2 and v2
    const bool all = p.pair_valid || (kmask & (kmask + 1)) != 0u;
    const int rows[5] = {(nq + 15) & ~15, all ? kSmallRows : (n + 7) & ~7, n, n, all ? kSmallRows : (n + 15) & ~15};
#pragma unroll
    for (int t = 0; t < 5; ++t)
      for (int idx = tid; idx < 8 * rows[t]; idx += 32 * kWarps) {
        const int r = idx >> 3, c = idx & 7;
        const bool ok = ((t == 0 ? qmask : kmask) >> r) & 1u;
        cp_async16(row_chunk(t0 + t * kSmallTile, r, c), src[t] + p.in.at(b, h, ok ? r : 0) + c * 8, ok);
      }
    // the bias along with the tiles: its loads wait for nothing but the masks (loaded when they were needed, they were the
    // largest stall of a CTA that lives for a few steps: 256 molecules of 9-29 atoms 68 -> 57 us, 512 of 10-32 134 -> 101)
    if constexpr (kBias) {
      for (int idx = tid; idx < kSmallRows * kSmallRows; idx += 32 * kWarps) {
        const int x = idx >> 5, y = idx & 31;
        const bool row = x < nq && y < n, pair = x < n && y < n;
        const size_t at = (size_t)bh * N * N + (row || pair ? x * N + y : 0);
        cp_async4(&sm.u[x][y], p.u + at, row);
        cp_async4(&sm.v[x][y], p.v_bias + at, row);
        cp_async4(&sm.w[x][y], p.w + at, pair);
      }
      for (int x = tid; x < kSmallRows; x += 32 * kWarps) cp_async4(&sm.gate[x], p.gate + (size_t)bh * N + min(x, N - 1), x < nq);
    }
    cp_async_commit();
  }
  bool hole = (kmask & (kmask + 1)) != 0u;
  for (int j = tid >> 5; j < kSmallRows; j += kWarps) {
    uint32_t word = (j < N && ((kmask >> j) & 1u)) ? kmask : 0u;
    if (p.pair_valid && word != 0u) {
      const uint32_t pv = __ballot_sync(0xffffffffu, lane < N && p.pair_valid[((size_t)b * N + j) * N + min(lane, N - 1)] > 0);
      hole |= (pv & kmask) != kmask;
      word &= pv;
    }
    if (lane == 0) sm.visible[j] = word;
  }
  cp_async_wait<0>();
  hole = __syncthreads_or(hole) != 0;
  if (hole) small_fwd_rows<4, true, kBias, kWarps>(p, sm, b, h, 32 - __clz(kmask), qmask);
  else if (n <= 8) small_fwd_rows<1, false, kBias, kWarps>(p, sm, b, h, n, qmask);
  else if (n <= 16) small_fwd_rows<2, false, kBias, kWarps>(p, sm, b, h, n, qmask);
  else if (n <= 24) small_fwd_rows<3, false, kBias, kWarps>(p, sm, b, h, n, qmask);
  else small_fwd_rows<4, false, kBias, kWarps>(p, sm, b, h, n, qmask);
}

// Molecules by their number of keys, the largest first (the order decides when a molecule runs, not what it computes).
__global__ void __launch_bounds__(1024) simplicial_small_order_kernel(const uint8_t* __restrict__ key_valid, int B, int N, int32_t* keys,
                                                                     int32_t* order) {
  __shared__ int start[kSmallRows + 1];
  wait_for_previous();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid <= kSmallRows) start[tid] = 0;
  __syncthreads();
  constexpr int kAtOnce = 16;  // molecules of a warp whose masks are on their way together
  for (int b0 = kAtOnce * warp; b0 < B; b0 += 32 * kAtOnce) {
    uint8_t v[kAtOnce];
#pragma unroll
    for (int t = 0; t < kAtOnce; ++t) v[t] = __ldg(key_valid + (size_t)min(b0 + t, B - 1) * N + min(lane, N - 1));
    int mine = 0;
#pragma unroll
    for (int t = 0; t < kAtOnce; ++t) {
      const uint32_t m = __ballot_sync(0xffffffffu, lane < N && v[t] > 0);
      if (lane == t) mine = 32 - __clz(m);
    }
    if (lane < kAtOnce && b0 + lane < B) {
      keys[b0 + lane] = mine;
      atomicAdd(&start[kSmallRows - mine], 1);
    }
  }
  __syncthreads();
  if (warp == 0) {  // exclusive sums; the last class holds the empty molecules
    const int mine = start[lane];
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += x;
    }
    start[lane] = sum - mine;
    if (lane == 31) start[kSmallRows] = sum;
  }
  __syncthreads();
  for (int b = tid; b < B; b += 1024) order[atomicAdd(&start[kSmallRows - keys[b]], 1)] = b;
}

}  // namespace

// Where a batch is several waves of CTAs, the last ones to start should be small: molecules of 9-29 atoms x 8 heads, in the order
// given | heavy first: backward with the bias 128 molecules 131 | 108 us, 256 244 | 199, without 256 159 | 130, 1024 546 | 489; with the
// residuals 64 243 | 210; forward 1024 141 | 128, 256 with the bias 61 | 58, 64 with the residuals 70 | 55.  The list takes a launch
// (it is lost where all molecules are of one size: 1024 of 29 atoms forward 213 | 219, backward 800 | 807, 256 with the bias backward
// 310 | 316, which a caller who knows avoids by giving no workspace): it is made where it pays several times over.
size_t simplicial_small_order_bytes(int batch, int heads, bool backward, bool residual) {
  const long long bh = (long long)batch * heads;
  return bh >= (residual ? 512 : backward ? 1024 : 4096) ? align_up(2 * (size_t)batch * sizeof(int32_t), 256) : 0;
}
int simplicial_small_order(const uint8_t* key_valid, int batch, int tokens, void* workspace, size_t workspace_bytes, size_t need,
                           const int32_t** order, cudaStream_t stream) {
  *order = nullptr;
  if (need == 0 || !workspace || workspace_bytes < need) return MF_OK;  // (a caller may leave it out)
  int32_t* keys = static_cast<int32_t*>(workspace);
  launch_dependent(simplicial_small_order_kernel, dim3(1), dim3(1024), 0, stream, key_valid, batch, tokens, keys, keys + batch);
  MF_CHECK_LAUNCH("simplicial_small_order_kernel");
  *order = keys + batch;
  return MF_OK;
}

int simplicial_small_fwd(const MfSimplicialFwdArgs& a, const TileLayouts* layouts, cudaStream_t stream) {
  SmallFwdParams p{};
  const int rc = simplicial_small_order(a.pair_key_valid, a.batch, a.tokens, a.workspace, a.workspace_bytes,
                                        simplicial_small_order_bytes(a.batch, a.heads, false, false), &p.order, stream);
  if (rc != MF_OK) return rc;
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.k1 = static_cast<const __nv_bfloat16*>(a.k1);
  p.v1 = static_cast<const __nv_bfloat16*>(a.v1);
  p.k2 = static_cast<const __nv_bfloat16*>(a.k2);
  p.v2 = static_cast<const __nv_bfloat16*>(a.v2);
  p.query_valid = a.query_valid;
  p.key_valid = a.pair_key_valid;
  p.pair_valid = a.pair_valid;
  p.u = a.u;
  p.v_bias = a.v_bias;
  p.w = a.w;
  p.gate = a.gate;
  p.out = a.out;
  p.lse = a.lse;
  p.out_cast = static_cast<__nv_bfloat16*>(a.out_cast);
  p.H = a.heads;
  p.N = a.tokens;
  p.q_scale = layouts ? layouts->q_scale : 1.f;
  p.in = layouts ? layouts->in : contiguous_rows(a.heads, a.tokens);
  p.act = layouts ? layouts->act : contiguous_rows(a.heads, a.tokens);
  const int bh = a.batch * a.heads;
  // Two warps per (batch, head), one for each row tile, once that fills the chip several times over; fewer molecules are split
  // over four.  9-29 atoms x 8 heads, 2 | 4 warps: 64 molecules 20.2 | 15.8 us, 256 45.7 | 42.7, 512 76.4 | 77.6, 1024 140 |
  // 148; with the bias 23.9 | 23.3, 57.2 | 56.9, 119 | 123, 222 | 239.
  const int warps = bh >= 4096 ? 2 : 4;
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, true, stream);
#define MF_LAUNCH(BIAS, W) launch_dependent(simplicial_small_fwd_kernel<BIAS, W>, dim3(bh), dim3(32 * W), 0, stream, p)
  if (a.u) {
    if (warps == 2) MF_LAUNCH(true, 2);
    else MF_LAUNCH(true, 4);
  } else {
    if (warps == 2) MF_LAUNCH(false, 2);
    else MF_LAUNCH(false, 4);
  }
#undef MF_LAUNCH
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, false, stream);
  MF_CHECK_LAUNCH("simplicial_small_fwd_kernel");
  return MF_OK;
}

}  // namespace mf
