// 2-simplicial attention in fp32 on CUDA cores for molecules of at most 64 tokens, head sizes 32 and 64, without geometry
// operands (those and all other shapes: simplicial_generic.cu).
//
// A lane owns one key k of the second set, a warp walks over queries i, and for one query over the first keys j:
//   s_jk = sum_d (q_i k1_j)_d k2_kd      A_i[k] += dS_jk k1_j      B_i[k] += P_jk v1_j
// From the sums over j come, without another pass over the pairs,
//   out_i = sum_k v2_k o B_i[k]    dq_i = sum_k k2_k o A_i[k]    dk2_k += q_i o A_i[k]    dv2_k += dO_i o B_i[k]
// and dk1, dv1 from the same kernel with the two key sets exchanged.  Rows of the walked set are broadcast from shared
// memory, the owned row and the sums stay in registers.  The backward pass is one launch of four kinds of CTAs (K side with
// dS, V side with P, for either key set); the warps of a CTA share a (batch, head) and are added up in a fixed order.
//
// What bounds it: at the sizes fp32 is used at (8 molecules of up to 29 atoms x 8 heads) latency, the two kernels take 16 and 58 of the
// call's 89 us on 256 CTAs, less than one wave, each warp with up to four queries of eight dependent steps; fp32 issue beyond.
#include "common.cuh"
#include "simplicial.cuh"

namespace mf {
namespace {

constexpr int kWarps = 8, kThreads = 32 * kWarps, kMaxTok = 64;

struct F32Params {
  const float* grad_out;
  const float* q;
  const float* k1;
  const float* v1;
  const float* k2;
  const float* v2;
  const uint8_t* query_valid;
  const uint8_t* key_valid;
  const uint8_t* pair_valid;
  float* out;  // backward: read
  float* lse;
  float* dq;
  float* dk1;
  float* dv1;
  float* dk2;
  float* dv2;
  int H, N;
};

// rows [0, rows) of a (N, D) matrix into shared memory with `stride` floats per row; rows with `mask` clear become zeros
template <int D>
__device__ __forceinline__ void load_rows(float* dst, int stride, const float* src, int rows, uint64_t mask) {
  for (int idx = threadIdx.x; idx < rows * (D / 4); idx += kThreads) {
    const int r = idx / (D / 4), c = idx % (D / 4);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((mask >> r) & 1ull) v = *reinterpret_cast<const float4*>(src + (size_t)r * D + 4 * c);
    *reinterpret_cast<float4*>(dst + r * stride + 4 * c) = v;
  }
}

__device__ __forceinline__ uint64_t valid_mask(const uint8_t* v, int N) {
  const int lane = threadIdx.x & 31;
  const uint32_t lo = __ballot_sync(0xffffffffu, lane < N && v[min(lane, N - 1)] > 0);
  const uint32_t hi = __ballot_sync(0xffffffffu, lane + 32 < N && v[min(lane + 32, N - 1)] > 0);
  return ((uint64_t)hi << 32) | lo;
}

// Four logits of the lane's key: x[t] = sum_d w[t][d] own[d], w = four rows in shared memory that all lanes read
template <int D>
__device__ __forceinline__ void dot4(float (&x)[4], const float* w, const float4 (&own)[D / 4]) {
  float2 a[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) a[t] = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < D / 4; ++c)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float4 y = *reinterpret_cast<const float4*>(w + t * D + 4 * c);
      a[t] = fma2(make_float2(y.x, y.y), make_float2(own[c].x, own[c].y), a[t]);
      a[t] = fma2(make_float2(y.z, y.w), make_float2(own[c].z, own[c].w), a[t]);
    }
#pragma unroll
  for (int t = 0; t < 4; ++t) x[t] = a[t].x + a[t].y;
}
// the same with the owned row read from shared memory (each lane its own row)
template <int D>
__device__ __forceinline__ void dot4_row(float (&x)[4], const float* w, const float* own) {
  float2 a[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) a[t] = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < D / 4; ++c) {
    const float4 o = *reinterpret_cast<const float4*>(own + 4 * c);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float4 y = *reinterpret_cast<const float4*>(w + t * D + 4 * c);
      a[t] = fma2(make_float2(y.x, y.y), make_float2(o.x, o.y), a[t]);
      a[t] = fma2(make_float2(y.z, y.w), make_float2(o.z, o.w), a[t]);
    }
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) x[t] = a[t].x + a[t].y;
}
// sum[d] += c * row[d]
template <int D>
__device__ __forceinline__ void axpy(float4 (&sum)[D / 4], float c, const float* row) {
  const float2 cc = make_float2(c, c);
#pragma unroll
  for (int t = 0; t < D / 4; ++t) {
    const float4 y = *reinterpret_cast<const float4*>(row + 4 * t);
    const float2 lo = fma2(cc, make_float2(y.x, y.y), make_float2(sum[t].x, sum[t].y));
    const float2 hi = fma2(cc, make_float2(y.z, y.w), make_float2(sum[t].z, sum[t].w));
    sum[t] = make_float4(lo.x, lo.y, hi.x, hi.y);
  }
}
// Sums over the lanes of D values per lane; lane l gets elements l and (D == 64) l + 32 of the sum, in res.
template <int D>
__device__ __forceinline__ void lane_sums(float (&v)[D], float (&res)[D / 32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < D / 32; ++h) {
    float* x = v + 32 * h;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int e = 0; e < o; ++e) {
        const float keep = up ? x[o + e] : x[e], give = up ? x[e] : x[o + e];
        x[e] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    res[h] = x[0];
  }
}

template <int D>
__device__ __forceinline__ void products(float (&v)[D], const float4 (&a)[D / 4], const float* row) {
#pragma unroll
  for (int c = 0; c < D / 4; ++c) {
    const float4 y = *reinterpret_cast<const float4*>(row + 4 * c);
    v[4 * c] = a[c].x * y.x, v[4 * c + 1] = a[c].y * y.y, v[4 * c + 2] = a[c].z * y.z, v[4 * c + 3] = a[c].w * y.w;
  }
}

// bit j: the pair of walked key j and owned key k counts (the sets exchanged: pair (k, j))
__device__ __forceinline__ uint64_t visible_bits(const F32Params& p, int b, int k, uint64_t kmask, bool exchanged) {
  if (!((kmask >> k) & 1ull)) return 0ull;
  if (!p.pair_valid) return kmask;
  const uint8_t* pv = p.pair_valid + (size_t)b * p.N * p.N;
  uint64_t bits = 0;
  for (int j = 0; j < p.N; ++j)
    if (pv[exchanged ? (size_t)k * p.N + j : (size_t)j * p.N + k] > 0) bits |= 1ull << j;
  return bits & kmask;
}

template <int D>
struct FwdShared {
  float k1[kMaxTok + 4][D], v1[kMaxTok][D];        // walked set (rows beyond the last key: zeros)
  float k2[kMaxTok][D + 4], v2[kMaxTok][D + 4];    // owned set, padded: lanes read different rows
  float w[kWarps][4][D];                           // q_i o k1_j of four first keys
  float s[kWarps][kMaxTok][32];                    // logits of a query, one column per lane
};

template <int D>
__global__ void __launch_bounds__(kThreads, D == 32 ? 2 : 1) simplicial_f32_fwd_kernel(const __grid_constant__ F32Params p) {
  extern __shared__ __align__(16) uint8_t smem[];
  FwdShared<D>& sm = *reinterpret_cast<FwdShared<D>*>(smem);
  const int N = p.N, bh = blockIdx.x, b = bh / p.H, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t kmask = valid_mask(p.key_valid + (size_t)b * N, N), qmask = valid_mask(p.query_valid + (size_t)b * N, N);
  const int n = 64 - __clzll(kmask);
  const size_t base = (size_t)bh * N * D;
  load_rows<D>(&sm.k1[0][0], D, p.k1 + base, min(n + 4, N), kmask);
  for (int idx = threadIdx.x; idx < 4 * D; idx += kThreads) sm.k1[N][idx] = 0.f;
  load_rows<D>(&sm.v1[0][0], D, p.v1 + base, n, kmask);
  load_rows<D>(&sm.k2[0][0], D + 4, p.k2 + base, n, kmask);
  load_rows<D>(&sm.v2[0][0], D + 4, p.v2 + base, n, kmask);
  __syncthreads();
  float* w = sm.w[warp][0];
  for (int i = blockIdx.y * kWarps + warp; i < N; i += gridDim.y * kWarps) {
    const bool have = ((qmask >> i) & 1ull) && n > 0;
    float m_all = -INFINITY, l_all = 0.f, o_all[D / 32];
#pragma unroll
    for (int h = 0; h < D / 32; ++h) o_all[h] = 0.f;
    if (have) {
      float qv[D / 32];
#pragma unroll
      for (int h = 0; h < D / 32; ++h) qv[h] = p.q[base + (size_t)i * D + lane + 32 * h];
      for (int half = 0; half < n; half += 32) {
        const int k = half + lane;
        const uint64_t vis = visible_bits(p, b, min(k, N - 1), k < n ? kmask : 0ull, false);
        float4 own[D / 4], acc[D / 4];
#pragma unroll
        for (int c = 0; c < D / 4; ++c) {
          own[c] = *reinterpret_cast<const float4*>(&sm.k2[min(k, kMaxTok - 1)][4 * c]);
          acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float m = -INFINITY;
        for (int j = 0; j < n; j += 4) {
          __syncwarp();
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int h = 0; h < D / 32; ++h) w[t * D + lane + 32 * h] = qv[h] * sm.k1[j + t][lane + 32 * h];
          __syncwarp();
          float s[4];
          dot4<D>(s, w, own);
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (j + t < n) {
              s[t] = ((vis >> (j + t)) & 1ull) ? s[t] : -INFINITY;
              m = fmaxf(m, s[t]);
              sm.s[warp][j + t][lane] = s[t];
            }
        }
        m = warp_max(m);
        if (m == -INFINITY) continue;
        float l = 0.f;
        for (int j = 0; j < n; ++j) {
          const float pr = expf(sm.s[warp][j][lane] - m);
          l += pr;
          axpy<D>(acc, pr, sm.v1[j]);
        }
        l = warp_sum(l);
        float v[D], o[D / 32];
        products<D>(v, acc, sm.v2[min(k, n - 1)]);
        lane_sums<D>(v, o);
        const float m_new = fmaxf(m_all, m), a = expf(m_all - m_new), c = expf(m - m_new);
        l_all = l_all * a + l * c;
#pragma unroll
        for (int h = 0; h < D / 32; ++h) o_all[h] = o_all[h] * a + o[h] * c;
        m_all = m_new;
      }
    }
    const bool any = have && l_all > 0.f;
#pragma unroll
    for (int h = 0; h < D / 32; ++h) p.out[base + (size_t)i * D + lane + 32 * h] = any ? o_all[h] / l_all : 0.f;
    if (lane == 0) p.lse[(size_t)bh * N + i] = any ? m_all + logf(l_all) : 0.f;
  }
}

template <int D>
struct BwdShared {
  float wk[kMaxTok + 4][D], wv[kMaxTok + 4][D];  // walked set
  union {
    struct {
      float ok[kMaxTok][D + 4], ov[kMaxTok][D + 4];  // owned set
    };
    float part[kWarps][32][D + 4];                   // the warps' gradients of the 32 owned keys
  };
  float w[kWarps][2][4][D];  // q_i o walked K, dO_i o walked V of four walked keys
  float row[kWarps][D];      // q_i
  float dq[kMaxTok][D];
};

// One kind of CTA.  Only the one that produces dq needs A_i by itself; the others add q_i o k_j (or dO_i o v_j), which the
// logits were formed from, straight to their gradient.
template <int D, bool key_side, bool exchanged>
__device__ __forceinline__ void f32_bwd_side(const F32Params& p, BwdShared<D>& sm) {
  constexpr bool direct = !key_side || exchanged;
  const int N = p.N, bh = blockIdx.x, b = bh / p.H, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t kmask = valid_mask(p.key_valid + (size_t)b * N, N), qmask = valid_mask(p.query_valid + (size_t)b * N, N);
  const int n = qmask ? 64 - __clzll(kmask) : 0, nq = n ? 64 - __clzll(qmask) : 0;
  const size_t base = (size_t)bh * N * D;
  const float *wk = exchanged ? p.k2 : p.k1, *wv = exchanged ? p.v2 : p.v1, *ok = exchanged ? p.k1 : p.k2, *ov = exchanged ? p.v1 : p.v2;
  float* grad = key_side ? (exchanged ? p.dk1 : p.dk2) : (exchanged ? p.dv1 : p.dv2);
  load_rows<D>(&sm.wk[0][0], D, wk + base, min(n + 4, N), kmask);
  load_rows<D>(&sm.wv[0][0], D, wv + base, min(n + 4, N), kmask);
  for (int idx = threadIdx.x; idx < 4 * D; idx += kThreads) sm.wk[N][idx] = 0.f, sm.wv[N][idx] = 0.f;
  if (!direct)
    for (int idx = threadIdx.x; idx < N * D; idx += kThreads) sm.dq[0][idx] = 0.f;
  float *w1 = sm.w[warp][0][0], *w2 = sm.w[warp][1][0];
#pragma unroll 1
  for (int half = 0; half < N; half += 32) {
    const int k = half + lane;
    float4 g2[D / 4];
#pragma unroll
    for (int c = 0; c < D / 4; ++c) g2[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();  // the gradients of the previous half have left
    if (half < n) {
      load_rows<D>(&sm.ok[0][0], D + 4, ok + base, n, kmask);
      load_rows<D>(&sm.ov[0][0], D + 4, ov + base, n, kmask);
    }
    __syncthreads();
    const uint64_t vis = k < n ? visible_bits(p, b, k, kmask, exchanged) : 0ull;
    const float *own_k = sm.ok[min(k, max(n, 1) - 1)], *own_v = sm.ov[min(k, max(n, 1) - 1)];
#pragma unroll 1
    for (int i = warp; i < nq && half < n; i += kWarps) {
      if (!((qmask >> i) & 1ull)) continue;
      float qv[D / 32], gv[D / 32], delta = 0.f;
#pragma unroll
      for (int h = 0; h < D / 32; ++h) {
        const size_t at = base + (size_t)i * D + lane + 32 * h;
        qv[h] = p.q[at], gv[h] = p.grad_out[at];
        if (key_side) delta = fmaf(gv[h], p.out[at], delta);
        if (!direct) sm.row[warp][lane + 32 * h] = qv[h];
      }
      if (key_side) delta = warp_sum(delta);
      const float lse = p.lse[(size_t)bh * N + i];
      float4 a[D / 4];
#pragma unroll
      for (int c = 0; c < D / 4; ++c) a[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
      for (int j = 0; j < n; j += 4) {
        __syncwarp();
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int h = 0; h < D / 32; ++h) {
            w1[t * D + lane + 32 * h] = qv[h] * sm.wk[j + t][lane + 32 * h];
            w2[t * D + lane + 32 * h] = gv[h] * sm.wv[j + t][lane + 32 * h];
          }
        __syncwarp();
        float s[4], dp[4];
        dot4_row<D>(s, w1, own_k);
        if (key_side) dot4_row<D>(dp, w2, own_v);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          float c = ((vis >> (j + t)) & 1ull) && j + t < n ? expf(s[t] - lse) : 0.f;
          if (key_side) c *= dp[t] - delta;
          if (t) __syncwarp();  // (keeps the row loads of all four keys from being hoisted into registers at once)
          axpy<D>(direct ? g2 : a, c, !direct ? sm.wk[j + t] : (key_side ? w1 : w2) + t * D);
        }
      }
      if constexpr (!direct) {
#pragma unroll
        for (int c = 0; c < D / 4; ++c) {
          const float4 y = *reinterpret_cast<const float4*>(&sm.row[warp][4 * c]);
          const float2 lo = fma2(make_float2(a[c].x, a[c].y), make_float2(y.x, y.y), make_float2(g2[c].x, g2[c].y));
          const float2 hi = fma2(make_float2(a[c].z, a[c].w), make_float2(y.z, y.w), make_float2(g2[c].z, g2[c].w));
          g2[c] = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
        float v[D], o[D / 32];
        products<D>(v, a, own_k);
        lane_sums<D>(v, o);
#pragma unroll
        for (int h = 0; h < D / 32; ++h) sm.dq[i][lane + 32 * h] += o[h];
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < D / 4; ++c) *reinterpret_cast<float4*>(&sm.part[warp][lane][4 * c]) = g2[c];
    __syncthreads();
    for (int idx = threadIdx.x; idx < 32 * D; idx += kThreads) {
      const int r = idx / D, d = idx % D;
      if (half + r >= N) continue;
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < kWarps; ++q) sum += sm.part[q][r][d];
      grad[base + (size_t)(half + r) * D + d] = sum;
    }
  }
  if (!direct) {
    __syncthreads();
    for (int idx = threadIdx.x; idx < N * D; idx += kThreads) p.dq[base + idx] = sm.dq[0][idx];
  }
}

template <int D>
__global__ void __launch_bounds__(kThreads, D == 32 ? 2 : 1) simplicial_f32_bwd_kernel(const __grid_constant__ F32Params p) {
  extern __shared__ __align__(16) uint8_t smem[];
  BwdShared<D>& sm = *reinterpret_cast<BwdShared<D>*>(smem);
  switch (blockIdx.y) {
    case 0: f32_bwd_side<D, true, false>(p, sm); break;
    case 1: f32_bwd_side<D, true, true>(p, sm); break;
    case 2: f32_bwd_side<D, false, false>(p, sm); break;
    default: f32_bwd_side<D, false, true>(p, sm); break;
  }
}

template <int D, bool kBackward>
int launch_f32(const F32Params& p, int bh, cudaStream_t stream) {
  const int bytes = kBackward ? (int)sizeof(BwdShared<D>) : (int)sizeof(FwdShared<D>);
  auto kernel = kBackward ? simplicial_f32_bwd_kernel<D> : simplicial_f32_fwd_kernel<D>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(simplicial_f32_kernel)");
  // forward: enough CTAs to fill the chip, each taking every gridDim.y-th group of eight queries
  const int groups = (p.N + kWarps - 1) / kWarps, wanted = (296 + bh - 1) / bh;
  const dim3 grid(bh, kBackward ? 4 : (wanted < groups ? wanted : groups));
  kernel<<<grid, kThreads, bytes, stream>>>(p);
  MF_CHECK_LAUNCH("simplicial_f32_kernel");
  return MF_OK;
}

template <typename Args>
F32Params common_params(const Args& a) {
  F32Params p{};
  p.q = static_cast<const float*>(a.q);
  p.k1 = static_cast<const float*>(a.k1);
  p.v1 = static_cast<const float*>(a.v1);
  p.k2 = static_cast<const float*>(a.k2);
  p.v2 = static_cast<const float*>(a.v2);
  p.query_valid = a.query_valid, p.key_valid = a.pair_key_valid, p.pair_valid = a.pair_valid;
  p.H = a.heads, p.N = a.tokens;
  return p;
}

}  // namespace

int simplicial_f32_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream) {
  F32Params p = common_params(a);
  p.out = a.out, p.lse = a.lse;
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, true, stream);
  const int rc = a.head_dim == 32 ? launch_f32<32, false>(p, a.batch * a.heads, stream) : launch_f32<64, false>(p, a.batch * a.heads, stream);
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, false, stream);
  return rc;
}

int simplicial_f32_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream) {
  F32Params p = common_params(a);
  p.grad_out = static_cast<const float*>(a.grad_out);
  p.out = const_cast<float*>(a.out), p.lse = const_cast<float*>(a.lse);
  p.dq = static_cast<float*>(a.dq), p.dk1 = static_cast<float*>(a.dk1), p.dv1 = static_cast<float*>(a.dv1);
  p.dk2 = static_cast<float*>(a.dk2), p.dv2 = static_cast<float*>(a.dv2);
  profile_mark(MF_PROFILE_SIMPLICIAL_BWD, true, stream);
  const int rc = a.head_dim == 32 ? launch_f32<32, true>(p, a.batch * a.heads, stream) : launch_f32<64, true>(p, a.batch * a.heads, stream);
  profile_mark(MF_PROFILE_SIMPLICIAL_BWD, false, stream);
  return rc;
}

}  // namespace mf
