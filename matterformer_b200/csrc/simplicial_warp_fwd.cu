// 2-simplicial attention, forward, 33 to 192 tokens in bf16, with or without the factorized bias (see simplicial_warp.cuh).
//
// Query by query, as matrix products over key blocks of 32 x 32: S = (K1 o q_i) K2^T, P = exp2(S), W^T += V2^T P^T over the
// second keys of a block row, out_i += sum_j v1_j o W_j.  All of K1, K2, V1, V2 of one (batch, head) sits in shared memory; a
// warp keeps the block row's K1 o q_i and W^T in registers and needs no barrier and no exchange with other warps.  The
// softmax shift is 0 unless the query's sum leaves 2^-60 .. 2^60, in which case it is done again with its exact maximum.
// Blocks in which every pair counts take no masks.
//
// Bound by the mma.sync pipe, busy 52 % of the time, and the instructions and dependencies around it.  64 molecules of 20-181 atoms,
// 8 heads: 851 us, in the order given 893 (1 058 row-packed on tcgen05); 16 molecules of 20-131 atoms 113 (283).  With the bias (26 %
// busy, the loads of v and w) it serves short calls, see uses_tri_forward(), and callers that give no workspace: 1 821 us for that
// batch against 848 of simplicial_tri.cu, which needs one.
#include <type_traits>

#include "common.cuh"
#include "simplicial.cuh"
#include "simplicial_warp.cuh"

namespace mf {
namespace {

struct WarpFwdParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k1;
  const __nv_bfloat16* v1;
  const __nv_bfloat16* k2;
  const __nv_bfloat16* v2;
  const uint8_t* query_valid;
  const uint8_t* key_valid;
  const uint8_t* pair_valid;
  const float* u;
  const float* v_bias;
  const float* w;
  const float* gate;
  float* out;
  float* lse;
  __nv_bfloat16* out_cast;
  const int32_t* order;  // heavy molecules first, or NULL
  int H, N, chunk;  // chunk: queries per CTA
  int even;         // rows of v_bias and w start on 8-byte boundaries
};

constexpr int kFwdWarps = 12;                  // 168 registers each fill the register file
constexpr int kFwdThreads = 32 * kFwdWarps;
constexpr int kBlocks = kMaxKeys / 32;

struct WarpFwdHeader {
  uint32_t visible[kMaxKeys][kBlocks];  // bit k of word (j, kb): the pair (j, 32 kb + k) counts
  uint8_t full[kBlocks][kBlocks];       // every pair of the block counts
  uint32_t kmask[kBlocks], qmask[kBlocks];
};

// The block row jb (16 MT rows) of query i.
template <bool kBias>
struct QueryState {
  float o[8];
  float2 l;
  float m;  // exact pass: running maximum
};

template <bool kBias, bool kMaxPass, int MT>
__device__ __forceinline__ void block_row(const WarpFwdParams& p, const WarpFwdHeader& hd, const FragBase& fb, int tile_bytes,
                                          const uint32_t (&qf)[8], int bh, int i, int jb, int n, float shift, QueryState<kBias>& st) {
  const int lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2;
  const int tk2 = tile_bytes, tv1 = 2 * tile_bytes, tv2 = 3 * tile_bytes;
  const int nb = (n + 31) >> 5;
  uint32_t a[MT][4][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      load_a(a[mt][ks], fb, jb * 32 * kRowBytes, mt, ks);
      a[mt][ks][0] = mul_bf16x2(a[mt][ks][0], qf[2 * ks]);
      a[mt][ks][1] = mul_bf16x2(a[mt][ks][1], qf[2 * ks]);
      a[mt][ks][2] = mul_bf16x2(a[mt][ks][2], qf[2 * ks + 1]);
      a[mt][ks][3] = mul_bf16x2(a[mt][ks][3], qf[2 * ks + 1]);
    }
  float ur[MT][2], g = 0.f;
  const size_t row = ((size_t)bh * p.N + i) * p.N;
  if constexpr (kBias) {
    g = p.gate[(size_t)bh * p.N + i];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int j = 32 * jb + 16 * mt + 8 * hh + row8;
        ur[mt][hh] = j < n ? p.u[row + j] : 0.f;
      }
  }
  float w[4][2 * MT][4];  // W^T: channels 16 dt x j tiles
#pragma unroll
  for (int dt = 0; dt < 4; ++dt)
#pragma unroll
    for (int jt = 0; jt < 2 * MT; ++jt)
#pragma unroll
      for (int e = 0; e < 4; ++e) w[dt][jt][e] = 0.f;
  auto block = [&](int kb, auto tiles) {  // 32 x 32, or 16 wide where the molecule ends in the first half
    constexpr int NT = decltype(tiles)::value;
    const bool full = hd.full[jb][kb];
    const int at2 = kb * 32 * kRowBytes;
    float s[MT][NT][4];
#pragma unroll
    for (int kp = 0; kp < 2; ++kp)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        uint32_t b[4];
        load_b(b, fb, tk2 + at2, nt, kp);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          if (kp == 0) mma16_first(s[mt][nt], a[mt][0], b[0], b[1]);
          else mma16(s[mt][nt], a[mt][2], b[0], b[1]);
          mma16(s[mt][nt], a[mt][2 * kp + 1], b[2], b[3]);
        }
      }
    if constexpr (kBias) {
      const int k0 = 32 * kb + 2 * quad, j0 = 32 * jb + row8;
      const float* vr = p.v_bias + row + k0;
      const float* wr = p.w + ((size_t)bh * p.N + j0) * p.N + k0;
      if (full && p.even) {  // whole pairs of keys on 8-byte boundaries
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const float2 v = *reinterpret_cast<const float2*>(vr + 8 * nt);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const float2 x = add2(add2(make_float2(ur[mt][hh], ur[mt][hh]), v),
                                    *reinterpret_cast<const float2*>(wr + (16 * mt + 8 * hh) * p.N + 8 * nt));
              const float2 y = fma2(make_float2(g, g), x, make_float2(s[mt][nt][2 * hh], s[mt][nt][2 * hh + 1]));
              s[mt][nt][2 * hh] = y.x, s[mt][nt][2 * hh + 1] = y.y;
            }
        }
      } else {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const bool ka = k0 + 8 * nt < n, kc = k0 + 8 * nt + 1 < n;
          const float va = ka ? vr[8 * nt] : 0.f, vb = kc ? vr[8 * nt + 1] : 0.f;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const bool jin = j0 + 16 * mt + 8 * hh < n;
              const float* x = wr + (16 * mt + 8 * hh) * p.N + 8 * nt;
              const float wa = (jin && ka) ? x[0] : 0.f, wb = (jin && kc) ? x[1] : 0.f;
              s[mt][nt][2 * hh] = fmaf(g, (ur[mt][hh] + va) + wa, s[mt][nt][2 * hh]);
              s[mt][nt][2 * hh + 1] = fmaf(g, (ur[mt][hh] + vb) + wb, s[mt][nt][2 * hh + 1]);
            }
        }
      }
    }
    if (!full) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const uint32_t vis = hd.visible[32 * jb + 16 * mt + 8 * hh + row8][kb] >> (2 * quad);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            if (!((vis >> (8 * nt)) & 1u)) s[mt][nt][2 * hh] = -INFINITY;
            if (!((vis >> (8 * nt + 1)) & 1u)) s[mt][nt][2 * hh + 1] = -INFINITY;
          }
        }
    }
    if constexpr (kMaxPass) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) st.m = fmaxf(st.m, s[mt][nt][e]);
      return;
    }
    uint32_t pk[MT][NT][2];
    const float2 le = make_float2(kLog2e, kLog2e), c = make_float2(-shift, -shift);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float2 x = fma2(make_float2(s[mt][nt][2 * hh], s[mt][nt][2 * hh + 1]), le, c);
          x.x = fast_exp2(x.x);
          x.y = fast_exp2(x.y);
          st.l = add2(st.l, x);
          pk[mt][nt][hh] = pack2_bf16(x.x, x.y);
        }
#pragma unroll
    for (int dt = 0; dt < 4; ++dt)
#pragma unroll
      for (int ks = 0; ks < NT / 2; ++ks) {
        uint32_t v[4];
        load_t(v, fb, tv2 + at2, dt, ks);
#pragma unroll
        for (int jt = 0; jt < 2 * MT; ++jt) mma16(w[dt][jt], v, pk[jt >> 1][2 * ks][jt & 1], pk[jt >> 1][2 * ks + 1][jt & 1]);
      }
  };
  const int last = n - 32 * (nb - 1);
#pragma unroll 1
  for (int kb = 0; kb < nb - (last <= 16); ++kb) block(kb, std::integral_constant<int, 4>{});
  if (last <= 16) block(nb - 1, std::integral_constant<int, 2>{});
  if constexpr (!kMaxPass) {
#pragma unroll
    for (int dt = 0; dt < 4; ++dt) {
      float2 lo = make_float2(0.f, 0.f), hi = lo;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        uint32_t v[4];
        load_t(v, fb, tv1 + jb * 32 * kRowBytes, dt, mt);
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          const float(&c)[4] = w[dt][2 * mt + jj];
          lo = fma2(make_float2(c[0], c[1]), make_float2(bf16_lo(v[2 * jj]), bf16_hi(v[2 * jj])), lo);
          hi = fma2(make_float2(c[2], c[3]), make_float2(bf16_lo(v[2 * jj + 1]), bf16_hi(v[2 * jj + 1])), hi);
        }
      }
      st.o[2 * dt] += lo.x + lo.y;
      st.o[2 * dt + 1] += hi.x + hi.y;
    }
  }
}

template <bool kBias>
__global__ void __launch_bounds__(kFwdThreads, 1) simplicial_warp_fwd_kernel(const __grid_constant__ WarpFwdParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = lane & 3, row8 = lane >> 2;
  const int N = p.N, b = p.order ? p.order[blockIdx.y / p.H] : blockIdx.y / p.H, bh = b * p.H + blockIdx.y % p.H;
  WarpFwdHeader& hd = *reinterpret_cast<WarpFwdHeader*>(smem);
  constexpr int kHeader = (sizeof(WarpFwdHeader) + 127) / 128 * 128;
  const uint32_t tile0 = (uint32_t)__cvta_generic_to_shared(smem) + kHeader;
  if (warp < kBlocks) {
    const int t = 32 * warp + lane;
    const uint32_t k = __ballot_sync(0xffffffffu, t < N && p.key_valid[(size_t)b * N + min(t, N - 1)] > 0);
    const uint32_t q = __ballot_sync(0xffffffffu, t < N && p.query_valid[(size_t)b * N + min(t, N - 1)] > 0);
    if (lane == 0) hd.kmask[warp] = k, hd.qmask[warp] = q;
  }
  __syncthreads();
  int n = 0, nq = 0;
#pragma unroll
  for (int t = 0; t < kBlocks; ++t) {
    if (hd.kmask[t]) n = 32 * t + 32 - __clz(hd.kmask[t]);
    if (hd.qmask[t]) nq = 32 * t + 32 - __clz(hd.qmask[t]);
  }
  const int i0 = blockIdx.x * p.chunk, i1 = min(i0 + p.chunk, N);
  if (n == 0) nq = 0;
  for (int idx = tid + 16 * max(nq - i0, 0); idx < 16 * (i1 - i0); idx += kFwdThreads) {  // queries beyond the last valid one
    const size_t at = ((size_t)bh * N + i0 + (idx >> 4)) * kD + 4 * (idx & 15);
    *reinterpret_cast<float4*>(p.out + at) = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.out_cast) *reinterpret_cast<uint2*>(p.out_cast + at) = make_uint2(0u, 0u);
    if ((idx & 15) == 0) p.lse[(size_t)bh * N + i0 + (idx >> 4)] = 0.f;
  }
  if (i0 >= nq) return;
  const int rows = (n + 31) & ~31, tile_bytes = rows * kRowBytes, nb = rows >> 5;
  {
    const __nv_bfloat16* src[4] = {p.k1, p.k2, p.v1, p.v2};
    const size_t base = (size_t)bh * N * kD;
#pragma unroll
    for (int t = 0; t < 4; ++t)
      for (int idx = tid; idx < 8 * rows; idx += kFwdThreads) {
        const int r = idx >> 3, c = idx & 7;
        const bool ok = (hd.kmask[r >> 5] >> (r & 31)) & 1u;
        cp_async16(row_chunk(tile0 + t * tile_bytes, r, c), src[t] + base + (size_t)(ok ? r : 0) * kD + c * 8, ok);
      }
    cp_async_commit();
  }
  for (int item = warp; item < rows * nb; item += kFwdWarps) {
    const int j = item / nb, kb = item - j * nb;
    uint32_t word = (hd.kmask[j >> 5] >> (j & 31)) & 1u ? hd.kmask[kb] : 0u;
    if (p.pair_valid && word) {
      const int k = 32 * kb + lane;
      word &= __ballot_sync(0xffffffffu, k < N && p.pair_valid[((size_t)b * N + j) * N + min(k, N - 1)] > 0);
    }
    if (lane == 0) hd.visible[j][kb] = word;
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int item = warp; item < nb * nb; item += kFwdWarps) {
    const int jb = item / nb, kb = item - jb * nb;
    const bool all = __all_sync(0xffffffffu, hd.visible[32 * jb + lane][kb] == 0xffffffffu);
    if (lane == 0) hd.full[jb][kb] = all;
  }
  __syncthreads();

  const FragBase fb(tile0, lane);
  const int half = n - 32 * (nb - 1) <= 16;  // the last block row holds keys in its first 16 rows only
  for (int i = i0 + warp; i < min(i1, nq); i += kFwdWarps) {
    const bool valid = (hd.qmask[i >> 5] >> (i & 31)) & 1u;
    QueryState<kBias> st;
    float shift = 0.f, l = 0.f;
    if (valid) {
      uint32_t qf[8];
      const __nv_bfloat16* q = p.q + ((size_t)bh * N + i) * kD + 2 * quad;
#pragma unroll
      for (int c = 0; c < 8; ++c) qf[c] = *reinterpret_cast<const uint32_t*>(q + 8 * c);
      for (bool exact = false;; exact = true) {
        if (exact) {
          st.m = -INFINITY;
#pragma unroll 1
          for (int jb = 0; jb < nb; ++jb) block_row<kBias, true, 2>(p, hd, fb, tile_bytes, qf, bh, i, jb, n, 0.f, st);
          const float m = warp_max(st.m);
          shift = m > -INFINITY ? m * kLog2e : 0.f;
        }
        st.l = make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < 8; ++e) st.o[e] = 0.f;
#pragma unroll 1
        for (int jb = 0; jb < nb - half; ++jb) block_row<kBias, false, 2>(p, hd, fb, tile_bytes, qf, bh, i, jb, n, shift, st);
        if (half) block_row<kBias, false, 1>(p, hd, fb, tile_bytes, qf, bh, i, nb - 1, n, shift, st);
        l = warp_sum(st.l.x + st.l.y);
        if (exact || (l >= kSumLow && l <= kSumHigh)) break;
      }
      quad_sum8(st.o, lane);
    }
    const bool have = valid && l != 0.f;
    const float inv = have ? 1.f / l : 0.f;
    const int d0 = (4 * (quad & 1) + 2 * (quad >> 1)) * 8 + row8;  // the lane's two channels: d0 and d0 + 8
    const float x0 = have ? st.o[0] * inv : 0.f, x1 = have ? st.o[1] * inv : 0.f;
    const size_t at = ((size_t)bh * N + i) * kD + d0;
    p.out[at] = x0;
    p.out[at + 8] = x1;
    if (p.out_cast) p.out_cast[at] = __float2bfloat16_rn(x0), p.out_cast[at + 8] = __float2bfloat16_rn(x1);
    if (lane == 0) p.lse[(size_t)bh * N + i] = have ? (shift + log2f(l)) * kLn2 : 0.f;
  }
}

// Molecules by the index of their last key, the largest first (the order decides when a molecule runs, not what it computes).
constexpr int kMostOrdered = 1024;
__global__ void __launch_bounds__(1024) simplicial_warp_order_kernel(const uint8_t* __restrict__ key_valid, int B, int N, int32_t* order) {
  __shared__ int last[kMostOrdered], start[kMaxKeys + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, words = (N + 31) >> 5;
  if (tid < B) last[tid] = 0;
  if (tid <= kMaxKeys) start[tid] = 0;
  __syncthreads();
  constexpr int kAtOnce = 8;  // mask words of a warp that are on their way together
  for (int i0 = kAtOnce * warp; i0 < B * words; i0 += 32 * kAtOnce) {
    uint8_t v[kAtOnce];
#pragma unroll
    for (int t = 0; t < kAtOnce; ++t) {
      const int i = min(i0 + t, B * words - 1), b = i / words, k = 32 * (i - b * words) + lane;
      v[t] = k < N ? __ldg(key_valid + (size_t)b * N + k) : 0;
    }
#pragma unroll
    for (int t = 0; t < kAtOnce; ++t) {
      const uint32_t m = __ballot_sync(0xffffffffu, v[t] > 0);
      const int i = min(i0 + t, B * words - 1), b = i / words;
      if (lane == 0 && m) atomicMax(&last[b], 32 * (i - b * words) + 32 - __clz(m));
    }
  }
  __syncthreads();
  const int mine = tid < B ? kMaxKeys - last[tid] : 0;
  if (tid < B) atomicAdd(&start[mine], 1);
  __syncthreads();
  if (warp == 0) {  // exclusive sums
    int before = 0;
    for (int c = 0; c <= kMaxKeys; c += 32) {
      const int n = c + lane <= kMaxKeys ? start[c + lane] : 0;
      int sum = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += x;
      }
      if (c + lane <= kMaxKeys) start[c + lane] = before + sum - n;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
  }
  __syncthreads();
  if (tid < B) order[atomicAdd(&start[mine], 1)] = tid;
}

// Queries per CTA: see simplicial_warp_fwd
int queries_per_cta(int bh, int tokens) {
  int chunk = tokens >= 128 ? 24 : tokens > 64 ? 48 : 96;
  while (chunk > 12 && (long long)bh * ((tokens + chunk - 1) / chunk) < 296) chunk >>= 1;
  return chunk;
}

}  // namespace

// Workspace of the list above, which a caller may leave out.  A CTA runs with the square of its molecule's size, so in the order
// given a launch ends with a few large ones: 8 heads, 20-181 atoms, 64 molecules 893 | 851 us heavy first, 24-192 8 molecules 181 |
// 140, 20-100 32 134 | 107, 20-160 4 76 | 64, 20-64 64 103 | 85, 10-48 64 60 | 48.  The list takes a launch of 3 us (and nothing is
// gained where all molecules are of one size: 64 of 64 tokens 153 | 157 us, 8 of 192 396 | 398), so it is made from a wave and a half of
// CTAs and about 50 us on.
size_t simplicial_warp_order_bytes(const MfSimplicialFwdArgs& a) {
  const int batch = a.batch, tokens = a.tokens;
  const long long bh = (long long)batch * a.heads;
  const int chunk = queries_per_cta((int)bh, tokens);
  const bool pays = !a.u && batch > 3 && batch <= kMostOrdered && bh * ((tokens + chunk - 1) / chunk) >= 222 &&
                    bh * tokens * tokens * tokens >= 30000000ll;
  return pays ? align_up((size_t)batch * sizeof(int32_t), 256) : 0;
}

int simplicial_warp_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream) {
  WarpFwdParams p{};
  const size_t need = simplicial_warp_order_bytes(a);
  if (need > 0 && a.workspace && a.workspace_bytes >= need) {
    int32_t* order = static_cast<int32_t*>(a.workspace);
    simplicial_warp_order_kernel<<<1, 1024, 0, stream>>>(a.pair_key_valid, a.batch, a.tokens, order);
    MF_CHECK_LAUNCH("simplicial_warp_order_kernel");
    p.order = order;
  }
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.k1 = static_cast<const __nv_bfloat16*>(a.k1);
  p.v1 = static_cast<const __nv_bfloat16*>(a.v1);
  p.k2 = static_cast<const __nv_bfloat16*>(a.k2);
  p.v2 = static_cast<const __nv_bfloat16*>(a.v2);
  p.query_valid = a.query_valid, p.key_valid = a.pair_key_valid, p.pair_valid = a.pair_valid;
  p.u = a.u, p.v_bias = a.v_bias, p.w = a.w, p.gate = a.gate;
  p.out = a.out, p.lse = a.lse, p.out_cast = static_cast<__nv_bfloat16*>(a.out_cast);
  p.H = a.heads, p.N = a.tokens;
  p.even = a.tokens % 2 == 0 && ((reinterpret_cast<uintptr_t>(a.v_bias) | reinterpret_cast<uintptr_t>(a.w)) & 7) == 0;
  // Queries per CTA: two per warp keep the last wave short on large molecules (a CTA of 24 queries against 36 blocks runs 50
  // times as long as its loads take); smaller molecules need more to pay for their loads, small batches fewer to fill the chip.
  // 64 molecules x 8 heads, 24 | 48 | 96 queries: up to 64 tokens 107 | 102 | 95 us, 96 215 | 207 | 222, 127 392 | 378 | 408,
  // 128 401 | 384 | 410, 192 1 004 | 977 | 1 035; with the bias 176 | 173 | 166, 387 | 382 | 401, 833 | 831 | 891, 773 | 775 |
  // 839, 2 076 | 2 131 | 2 296.  Halved below two CTAs per SM: 2 molecules of up to 192 tokens, 12 | 24 | 48: 62 | 101 | 183 us.
  const int bh = a.batch * a.heads;
  const int chunk = queries_per_cta(bh, a.tokens);
  p.chunk = chunk;
  constexpr int header = (int)((sizeof(WarpFwdHeader) + 127) / 128 * 128);
  const int rows = (a.tokens + 31) & ~31, bytes = header + 4 * rows * kRowBytes;
  auto kernel = a.u ? simplicial_warp_fwd_kernel<true> : simplicial_warp_fwd_kernel<false>;
  // (the limit is one for all sizes: another host thread must not lower it between here and the launch)
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, header + 4 * kMaxKeys * kRowBytes);
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(simplicial_warp_fwd_kernel)");
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, true, stream);
  kernel<<<dim3((a.tokens + chunk - 1) / chunk, bh), kFwdThreads, bytes, stream>>>(p);
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, false, stream);
  MF_CHECK_LAUNCH("simplicial_warp_fwd_kernel");
  return MF_OK;
}

}  // namespace mf
