// 2-simplicial attention, forward, for molecules of at most 32 tokens in bf16 with the low-rank residuals
// (angle: logits += agate_i ra^-1/2 L_i R_i^T, message: out_i += sum_r c_ir basis_r; with or without the factorized bias).
//
// The residual factors belong to one query, L_i and R_i are (keys x rank): for a fixed query both residuals are matrix
// products like the attention itself, so this kernel walks query by query (the kernel without residuals walks over first
// keys, where the factors would be different for every row).  A warp takes a query: 32 x 32 logits in registers, factors
// staged in its own shared memory as hi + lo bf16 (see RankTile), exact maximum, P as the B operand of W^T = V2^T P^T and
// of T^T = MR^T P^T, c_ir = sum_j ML_jr T_jr.  The bias and the basis of the head come to shared memory with the tiles: loaded where
// a query needs them they were most of its instructions (64 molecules of 9-29 atoms with the bias at rank 16 60 -> 50 us, 32 of 10-32 at
// rank 32 75 -> 58).  One variant of the walk for all sizes: narrower ones for small molecules took that back (see simplicial_small_bwd.cu).
#include "common.cuh"
#include "simplicial.cuh"
#include "simplicial_warp.cuh"

namespace mf {
namespace {

struct ResFwdParams {
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
  const float* al;
  const float* ar;
  const float* agate;
  const float* ml;
  const float* mr;
  const float* basis;
  int ra, rm;
  float* out;
  float* lse;
  __nv_bfloat16* out_cast;
  int H, N;
  const int32_t* order;  // heavy molecules first, or NULL
};

constexpr int kResWarps = 4;

template <int RK>
struct ResFwdShared {
  __align__(128) uint8_t tile[5][kSmallTile];                            // q, k1, v1, k2, v2
  __align__(128) uint8_t factor[kResWarps][4][2 * RankTile<RK>::kTile];  // L, R, ML, MR of the warp's query
  uint32_t visible[kSmallRows];
  // bias: w_jk as the fragments of the logits hold it, u_ij, v_ik and the gate
  float4 w[8][32];
  float u[kSmallRows][kSmallRows], v[kSmallRows][kSmallRows], gate[kSmallRows];
  float basis[16 * RK][kD];  // of the head, zeros beyond the rank
};

// The queries of a warp.
template <int RK>
__device__ __forceinline__ void res_fwd_queries(const ResFwdParams& p, ResFwdShared<RK>& sm, int bh, int n, uint32_t kmask,
                                                uint32_t qmask) {
  constexpr int MT = 2, NT = 4, KS = NT / 2;  // 16-row and 8-column tiles of the logits, 16-key steps over the second keys
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2, N = p.N;
  const uint32_t qt = (uint32_t)__cvta_generic_to_shared(sm.tile[0]);
  const FragBase fb(qt, lane);
  constexpr int kTk1 = kSmallTile, kTv1 = 2 * kSmallTile, kTk2 = 3 * kSmallTile, kTv2 = 4 * kSmallTile;
  const uint32_t f0 = (uint32_t)__cvta_generic_to_shared(sm.factor[warp][0]);
  const RankTile<RK> left{f0}, right{f0 + 2 * RankTile<RK>::kTile}, mleft{f0 + 4 * RankTile<RK>::kTile}, mright{f0 + 6 * RankTile<RK>::kTile};
  uint32_t vis[MT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) vis[mt][hh] = sm.visible[mt * 16 + hh * 8 + row8] >> (2 * quad);

  for (int i = warp; i < N; i += kResWarps) {
    const size_t qi = (size_t)bh * N + i;
    bool have = ((qmask >> i) & 1u) && n > 0;
    float l = 0.f, m = -INFINITY, o[8];
    float coef[2 * RK];  // message coefficients of ranks 8 e + row8
    if (have) {
      __syncwarp();
      const size_t qa = qi * N * p.ra, qm = qi * N * p.rm;
      if (p.al && p.ml && p.ra == p.rm) {
        stage_factors<4, RK>({left, right, mleft, mright}, {p.al + qa, p.ar + qa, p.ml + qm, p.mr + qm}, n, p.ra, kmask, nullptr, lane);
      } else {
        if (p.al) stage_factors<2, RK>({left, right}, {p.al + qa, p.ar + qa}, n, p.ra, kmask, nullptr, lane);
        if (p.ml) stage_factors<2, RK>({mleft, mright}, {p.ml + qm, p.mr + qm}, n, p.rm, kmask, nullptr, lane);
      }
      if (i + kResWarps < N) {
        const size_t next = (size_t)kResWarps * N;
        if (p.al) prefetch_l2(p.al + qa + next * p.ra, n * p.ra * 4, lane), prefetch_l2(p.ar + qa + next * p.ra, n * p.ra * 4, lane);
        if (p.ml) prefetch_l2(p.ml + qm + next * p.rm, n * p.rm * 4, lane), prefetch_l2(p.mr + qm + next * p.rm, n * p.rm * 4, lane);
      }
      __syncwarp();
      float s[MT][NT][4];
      {
        uint32_t qf[8];
        load_row_pairs(qf, qt, i, lane);
        pair_product<MT, NT>(s, fb, kTk1, kTk2, qf);
      }
      if (p.u) {
        const float g = sm.gate[i];
        float ur[MT][2];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) ur[mt][0] = sm.u[i][mt * 16 + row8], ur[mt][1] = sm.u[i][mt * 16 + 8 + row8];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const float2 v = *reinterpret_cast<const float2*>(&sm.v[i][nt * 8 + 2 * quad]);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const float4 w = sm.w[mt * 4 + nt][lane];
            s[mt][nt][0] = fmaf(g, (ur[mt][0] + v.x) + w.x, s[mt][nt][0]);
            s[mt][nt][1] = fmaf(g, (ur[mt][0] + v.y) + w.y, s[mt][nt][1]);
            s[mt][nt][2] = fmaf(g, (ur[mt][1] + v.x) + w.z, s[mt][nt][2]);
            s[mt][nt][3] = fmaf(g, (ur[mt][1] + v.y) + w.w, s[mt][nt][3]);
          }
        }
      }
      if (p.al) {
        float ad[MT][NT][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) ad[mt][nt][e] = 0.f;
        add_rank_product<MT, NT, RK>(ad, left, right, lane);
        const float g = p.agate[qi] * rsqrtf((float)p.ra);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[mt][nt][e] = fmaf(g, ad[mt][nt][e], s[mt][nt][e]);
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (!((vis[mt][e >> 1] >> (nt * 8 + (e & 1))) & 1u)) s[mt][nt][e] = -INFINITY;
            m = fmaxf(m, s[mt][nt][e]);
          }
      m = warp_max(m);
      have = m > -INFINITY;
      const float m2 = have ? m * kLog2e : 0.f;
      uint32_t pk[MT][NT][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const float a = fast_exp2(fmaf(s[mt][nt][2 * hh], kLog2e, -m2)), c = fast_exp2(fmaf(s[mt][nt][2 * hh + 1], kLog2e, -m2));
            l += a + c;
            pk[mt][nt][hh] = pack2_bf16(a, c);
          }
      l = warp_sum(l);
#pragma unroll
      for (int dt = 0; dt < 4; ++dt) {
        float w[2 * MT][4];
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          uint32_t a[4];
          load_t(a, fb, kTv2, dt, ks);
#pragma unroll
          for (int jt = 0; jt < 2 * MT; ++jt) {
            const uint32_t b0 = pk[jt >> 1][2 * ks][jt & 1], b1 = pk[jt >> 1][2 * ks + 1][jt & 1];
            if (ks == 0) mma16_first(w[jt], a, b0, b1);
            else mma16(w[jt], a, b0, b1);
          }
        }
        float lo = 0.f, hi = 0.f;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          uint32_t v[4];
          load_t(v, fb, kTv1, dt, mt);
#pragma unroll
          for (int jj = 0; jj < 2; ++jj) {
            const float* c = w[2 * mt + jj];
            lo = fmaf(c[0], bf16_lo(v[2 * jj]), fmaf(c[1], bf16_hi(v[2 * jj]), lo));
            hi = fmaf(c[2], bf16_lo(v[2 * jj + 1]), fmaf(c[3], bf16_hi(v[2 * jj + 1]), hi));
          }
        }
        o[2 * dt] = lo, o[2 * dt + 1] = hi;
      }
      quad_sum8(o, lane);
      if (p.ml) {
        // T^T (ranks x j) = MR^T P^T, c_r = sum_j ML_jr T_jr
#pragma unroll
        for (int rk = 0; rk < RK; ++rk) {
          float t[2 * MT][4], lo = 0.f, hi = 0.f;
          rank_sums<MT, NT, RK>(t, mright, pk, rk, lane);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            uint32_t mh[4], mo[4];
            mleft.load_t(mh, 0, rk, mt, lane);
            mleft.load_t(mo, 1, rk, mt, lane);
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              const float* c = t[2 * mt + jj];
              const uint32_t a0 = mh[2 * jj], a1 = mo[2 * jj], b0 = mh[2 * jj + 1], b1 = mo[2 * jj + 1];
              lo = fmaf(c[0], bf16_lo(a0) + bf16_lo(a1), fmaf(c[1], bf16_hi(a0) + bf16_hi(a1), lo));
              hi = fmaf(c[2], bf16_lo(b0) + bf16_lo(b1), fmaf(c[3], bf16_hi(b0) + bf16_hi(b1), hi));
            }
          }
#pragma unroll
          for (int x = 1; x < 4; x <<= 1) {
            lo += __shfl_xor_sync(0xffffffffu, lo, x);
            hi += __shfl_xor_sync(0xffffffffu, hi, x);
          }
          coef[2 * rk] = lo, coef[2 * rk + 1] = hi;
        }
      }
    }
    const int d0 = (4 * (quad & 1) + 2 * (quad >> 1)) * 8 + row8;  // the lane's two channels: d0 and d0 + 8
    float x0 = have ? o[0] : 0.f, x1 = have ? o[1] : 0.f;
    if (p.ml && have) {
      const float scale = rsqrtf((float)p.rm);
#pragma unroll
      for (int e = 0; e < 2 * RK; ++e)
#pragma unroll
        for (int r8 = 0; r8 < 8; ++r8) {
          const float c = __shfl_sync(0xffffffffu, coef[e], 4 * r8) * scale;
          x0 = fmaf(c, sm.basis[8 * e + r8][d0], x0);
          x1 = fmaf(c, sm.basis[8 * e + r8][d0 + 8], x1);
        }
    }
    const float inv = have ? 1.f / l : 0.f;
    x0 *= inv, x1 *= inv;
    float* out = p.out + qi * kD + d0;
    out[0] = x0, out[8] = x1;
    if (p.out_cast) {
      __nv_bfloat16* oc = p.out_cast + qi * kD + d0;
      oc[0] = __float2bfloat16_rn(x0), oc[8] = __float2bfloat16_rn(x1);
    }
    if (lane == 0) p.lse[qi] = have ? m + logf(l) : 0.f;
  }
}

template <int RK>
__global__ void __launch_bounds__(32 * kResWarps, 2) simplicial_small_res_fwd_kernel(const __grid_constant__ ResFwdParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  ResFwdShared<RK>& sm = *reinterpret_cast<ResFwdShared<RK>*>(smem);
  wait_for_previous();
  constexpr int kThreads = 32 * kResWarps;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int N = p.N, h = blockIdx.x % p.H, b = p.order ? p.order[blockIdx.x / p.H] : blockIdx.x / p.H, bh = b * p.H + h;
  const uint32_t kmask = __ballot_sync(0xffffffffu, lane < N && p.key_valid[(size_t)b * N + min(lane, N - 1)] > 0);
  const uint32_t qmask = __ballot_sync(0xffffffffu, lane < N && p.query_valid[(size_t)b * N + min(lane, N - 1)] > 0);
  const int n = 32 - __clz(kmask);
  const RowLayout rows{(long long)p.H * N * kD, (long long)N * kD, kD};
  {
    const __nv_bfloat16* src[5] = {p.q, p.k1, p.v1, p.k2, p.v2};
    const uint32_t t0 = (uint32_t)__cvta_generic_to_shared(sm.tile[0]);
#pragma unroll
    for (int t = 0; t < 5; ++t)
      for (int idx = tid; idx < 8 * kSmallRows; idx += kThreads) {
        const int r = idx >> 3, c = idx & 7;
        const bool ok = ((t == 0 ? qmask : kmask) >> r) & 1u;
        cp_async16(row_chunk(t0 + t * kSmallTile, r, c), src[t] + rows.at(b, h, ok ? r : 0) + c * 8, ok);
      }
    if (p.ml)
      for (int idx = tid; idx < 16 * RK * kD; idx += kThreads) {
        const int r = idx / kD;
        cp_async4(&sm.basis[r][idx % kD], p.basis + ((size_t)h * p.rm + min(r, p.rm - 1)) * kD + idx % kD, r < p.rm);
      }
    if (p.u && n > 0) {
      for (int idx = tid; idx < N * kSmallRows; idx += kThreads) {
        const int x = idx >> 5, y = idx & 31;
        const size_t at = ((size_t)bh * N + x) * N + min(y, n - 1);
        cp_async4(&sm.u[x][y], p.u + at, y < n);
        cp_async4(&sm.v[x][y], p.v_bias + at, y < n);
      }
      for (int x = tid; x < N; x += kThreads) cp_async4(&sm.gate[x], p.gate + (size_t)bh * N + x, true);
      for (int idx = tid; idx < 4 * 8 * 32; idx += kThreads) {
        const int f = idx >> 7, ln = (idx >> 2) & 31, e = idx & 3;
        const int j = (f >> 2) * 16 + 8 * (e >> 1) + (ln >> 2), k = (f & 3) * 8 + 2 * (ln & 3) + (e & 1);
        const bool ok = j < n && k < n;
        cp_async4(reinterpret_cast<float*>(&sm.w[f][ln]) + e, p.w + (size_t)bh * N * N + (ok ? j * N + k : 0), ok);
      }
    }
    cp_async_commit();
  }
  for (int idx = tid; idx < (int)sizeof(sm.factor) / 16; idx += kThreads) reinterpret_cast<float4*>(sm.factor)[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = warp; j < kSmallRows; j += kResWarps) {
    uint32_t word = (j < N && ((kmask >> j) & 1u)) ? kmask : 0u;
    if (p.pair_valid && word != 0u)
      word &= __ballot_sync(0xffffffffu, lane < N && p.pair_valid[((size_t)b * N + j) * N + min(lane, N - 1)] > 0);
    if (lane == 0) sm.visible[j] = word;
  }
  cp_async_wait<0>();
  __syncthreads();
  res_fwd_queries<RK>(p, sm, bh, n, kmask, qmask);
}

}  // namespace

int simplicial_small_res_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream) {
  ResFwdParams p{};
  const int rc = simplicial_small_order(a.pair_key_valid, a.batch, a.tokens, a.workspace, a.workspace_bytes,
                                        simplicial_small_order_bytes(a.batch, a.heads, false, true), &p.order, stream);
  if (rc != MF_OK) return rc;
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.k1 = static_cast<const __nv_bfloat16*>(a.k1);
  p.v1 = static_cast<const __nv_bfloat16*>(a.v1);
  p.k2 = static_cast<const __nv_bfloat16*>(a.k2);
  p.v2 = static_cast<const __nv_bfloat16*>(a.v2);
  p.query_valid = a.query_valid, p.key_valid = a.pair_key_valid, p.pair_valid = a.pair_valid;
  p.u = a.u, p.v_bias = a.v_bias, p.w = a.w, p.gate = a.gate;
  p.al = a.angle_left, p.ar = a.angle_right, p.agate = a.angle_gate;
  p.ml = a.message_left, p.mr = a.message_right, p.basis = a.message_basis;
  p.ra = a.angle_left ? a.angle_rank : 1, p.rm = a.message_left ? a.message_rank : 1;
  p.out = a.out, p.lse = a.lse, p.out_cast = static_cast<__nv_bfloat16*>(a.out_cast);
  p.H = a.heads, p.N = a.tokens;
  auto launch = [&](auto kernel, int bytes) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) launch_dependent(kernel, dim3(a.batch * a.heads), dim3(32 * kResWarps), bytes, stream, p);
    return e;
  };
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, true, stream);
  const cudaError_t e = max(p.ra, p.rm) <= 16 ? launch(simplicial_small_res_fwd_kernel<1>, (int)sizeof(ResFwdShared<1>))
                                              : launch(simplicial_small_res_fwd_kernel<2>, (int)sizeof(ResFwdShared<2>));
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(simplicial_small_res_fwd_kernel)");
  profile_mark(MF_PROFILE_SIMPLICIAL_FWD, false, stream);
  MF_CHECK_LAUNCH("simplicial_small_res_fwd_kernel");
  return MF_OK;
}

}  // namespace mf
