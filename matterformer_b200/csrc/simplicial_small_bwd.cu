// 2-simplicial attention, backward, for molecules of at most 32 tokens in bf16 (see simplicial_warp.cuh).
//
// For one query i every gradient is a product of 32 x 32 matrices that a warp holds in registers: S_i = (K1 o q_i) K2^T and
// P_i as in the forward pass, dP_i = (V1 o dO_i) V2^T, dS_i = P_i o (dP_i - delta_i), and with U_i = dS_i K2, W_i = P_i V2
//
//   dq_i = sum_j k1_j o U_i[j]     dk1_j += q_i o U_i[j]      dk2 += dS_i^T (K1 o q_i)
//                                  dv1_j += dO_i o W_i[j]     dv2 += P_i^T (V1 o dO_i)
//
// Four accumulators of 32 x 64 do not fit one warp, so the queries are walked twice: the V side (P: dv1, dv2), then the K side
// (dS: dq, dk1, dk2 and the bias gradients), which forms S_i and P_i again; 64 + 64 accumulator registers each, no barrier
// and no shared-memory exchange during a walk.  The warps of a CTA share one (batch, head), split its queries and are added
// up in a fixed order.  The products over the keys k take P and dS as the logit product left them (U^T = K2^T dS^T has dS
// as its B operand), those over j an 8x8 transposition in registers.  delta_i = dO_i . out_i is formed on load.
// Every output has one writer: no atomics, no workspace, nothing to zero beforehand.
//
// What bounds it: latency at two warps per scheduler (255 registers; the mma.sync pipe is 38 % busy, shared memory 46 %).
// Measured at 1024 molecules of 9-29 atoms x 8 heads: 547 us, against 980 + 39 us for the tcgen05 tile kernel and its delta
// pass; with the two sides on two warps of a pair 613 us (the V side waits for the K side, and two code paths share the
// instruction cache).
#include "common.cuh"
#include "simplicial.cuh"
#include "simplicial_warp.cuh"

namespace mf {
namespace {

struct SmallBwdParams {
  const __nv_bfloat16* grad_out;
  const __nv_bfloat16* q;
  const __nv_bfloat16* k1;
  const __nv_bfloat16* v1;
  const __nv_bfloat16* k2;
  const __nv_bfloat16* v2;
  const float* out;
  const float* lse;
  const uint8_t* query_valid;
  const uint8_t* key_valid;
  const uint8_t* pair_valid;
  const float* u;
  const float* v_bias;
  const float* w;
  const float* gate;
  float* du;
  float* dv_bias;
  float* dw;
  float* dgate;
  // low-rank residuals and their gradients (RK > 0)
  const float* al;
  const float* ar;
  const float* agate;
  const float* ml;
  const float* mr;
  const float* basis;
  float* dal;
  float* dar;
  float* dagate;
  float* dml;
  float* dmr;
  float* mcoef;  // rm^-1/2 sum_jk P ml mr, from which the caller forms the gradient of basis
  int ra, rm;
  __nv_bfloat16* dq;
  __nv_bfloat16* dk1;
  __nv_bfloat16* dv1;
  __nv_bfloat16* dk2;
  __nv_bfloat16* dv2;
  int H, N;
  const int32_t* order;  // heavy molecules first, or NULL
  float q_scale;
  RowLayout in, act;
};

constexpr int kAccStride = kD + 4;  // fp32 rows of the gradient stage

template <bool kBias, int RK = 0, int kWarps = 1>
struct SmallBwdShared {
  __align__(128) uint8_t tile[6][kSmallTile];  // q (a row becomes dq once its warp is done with it), k1, v1, k2, v2, grad_out
  union {
    float acc[2][kSmallRows][kAccStride];      // sums of the side just walked: first-key and second-key gradient
    float4 dw[4][8][32];                       // K side walk: the warps' dw_jk as the fragments of the logits hold it
  };
  float lse2[kSmallRows], delta[kSmallRows];
  uint32_t visible[kSmallRows];                // bit k of word j: the pair (j, k) counts
  float4 w[kBias ? 8 : 1][32];                 // bias w_jk as the fragments of the logits hold it
  float u[kBias ? kSmallRows : 1][kSmallRows], v[kBias ? kSmallRows : 1][kSmallRows], gate[kBias ? kSmallRows : 1];
  // RK > 0: rm^-1/2 dO_i . basis_r, and the residual factors of the query that each warp works on
  float dc[RK ? kSmallRows : 1][RK ? 16 * RK : 1];
  __align__(128) uint8_t factor[RK ? kWarps : 1][4][RK ? 2 * RankTile<RK ? RK : 1>::kTile : 16];
};

constexpr int kTq = 0, kTk1 = kSmallTile, kTv1 = 2 * kSmallTile, kTk2 = 3 * kSmallTile, kTv2 = 4 * kSmallTile, kTgo = 5 * kSmallTile;

// One walk; warp w takes the queries w, w + kWarps, ....  Leaves the two sums in sm.acc and all warps at a barrier.
template <int MT, int NT, bool kHoles, bool kBias, int RK, int kWarps, bool kKeySide, typename Shared>
__device__ __forceinline__ void small_bwd_side(const SmallBwdParams& p, Shared& sm, int bh, int n, uint32_t kmask,
                                               uint32_t qmask) {
  constexpr int KS = (NT + 1) / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, row8 = lane >> 2;
  const uint32_t qt = (uint32_t)__cvta_generic_to_shared(sm.tile[0]);
  const FragBase fb(qt, lane);
  constexpr int x1 = kKeySide ? kTk1 : kTv1, x2 = kKeySide ? kTk2 : kTv2, xr = kKeySide ? kTq : kTgo;
  uint32_t vis[MT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
      vis[mt][hh] = kHoles ? sm.visible[mt * 16 + hh * 8 + row8] >> (2 * quad) : (mt * 16 + hh * 8 + row8 < n ? ~0u : 0u);

  float a1[4][2 * MT][4], a2[KS][8][4];  // first-key gradient [channels][j], second-key gradient [k][channels]
#pragma unroll
  for (int dt = 0; dt < 4; ++dt)
#pragma unroll
    for (int jt = 0; jt < 2 * MT; ++jt)
#pragma unroll
      for (int e = 0; e < 4; ++e) a1[dt][jt][e] = 0.f;
#pragma unroll
  for (int kt = 0; kt < KS; ++kt)
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) a2[kt][t][e] = 0.f;
  const bool bias = kBias && (RK == 0 || p.u != nullptr);
  using Factor = RankTile<RK ? RK : 1>;
  const uint32_t f0 = (uint32_t)__cvta_generic_to_shared(sm.factor[RK ? warp : 0][0]);
  const Factor left{f0}, right{f0 + 2 * Factor::kTile}, mleft{f0 + 4 * Factor::kTile}, mright{f0 + 6 * Factor::kTile};
  const float a_scale = RK ? rsqrtf((float)p.ra) : 0.f, m_scale = RK ? rsqrtf((float)p.rm) : 0.f;
  if (bias && kKeySide) {
#pragma unroll
    for (int f = 0; f < 8; ++f) sm.dw[warp][f][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  const int nq = 32 - __clz(qmask);
  for (int i = warp; i < nq; i += kWarps) {
    if (!((qmask >> i) & 1u)) continue;
    float s[MT][NT][4];
    {
      uint32_t qf[8];
      load_row_pairs(qf, qt, i, lane);
      pair_product<MT, NT>(s, fb, kTk1, kTk2, qf);
    }
    float ga = 0.f;  // gate and scale of the angle residual
    if constexpr (RK > 0) {
      const size_t qi = (size_t)bh * p.N + i;
      __syncwarp();
      const size_t qa = qi * p.N * p.ra, qm = qi * p.N * p.rm;
      if (p.al) stage_factors<2>({left, right}, {p.al + qa, p.ar + qa}, n, p.ra, kmask, nullptr, lane);
      if (p.ml)  // K side: only ML_r (dO_i . basis_r) enters dP
        stage_factors<2>({mleft, mright}, {p.ml + qm, p.mr + qm}, n, p.rm, kmask, kKeySide ? sm.dc[i] : nullptr, lane);
      if (i + kWarps < nq) {
        const size_t next = (size_t)kWarps * p.N;
        if (p.al) prefetch_l2(p.al + qa + next * p.ra, n * p.ra * 4, lane), prefetch_l2(p.ar + qa + next * p.ra, n * p.ra * 4, lane);
        if (p.ml) prefetch_l2(p.ml + qm + next * p.rm, n * p.rm * 4, lane), prefetch_l2(p.mr + qm + next * p.rm, n * p.rm * 4, lane);
      }
      __syncwarp();
      if (p.al) {
        ga = p.agate[qi] * a_scale;
        float ad[MT][NT][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) ad[mt][nt][e] = 0.f;
        add_rank_product<MT, NT>(ad, left, right, lane);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[mt][nt][e] = fmaf(ga, ad[mt][nt][e], s[mt][nt][e]);
      }
    }
    float ul = 0.f, vl = 0.f, g = 0.f;  // bias: u_i,lane, v_i,lane
    if (bias) {
      ul = sm.u[i][lane], vl = sm.v[i][lane], g = sm.gate[i];
      float ur[MT][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) ur[mt][hh] = __shfl_sync(0xffffffffu, ul, mt * 16 + hh * 8 + row8);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const float va = __shfl_sync(0xffffffffu, vl, nt * 8 + 2 * quad), vb = __shfl_sync(0xffffffffu, vl, nt * 8 + 2 * quad + 1);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const float4 w = sm.w[mt * 4 + nt][lane];
          s[mt][nt][0] = fmaf(g, (ur[mt][0] + va) + w.x, s[mt][nt][0]);
          s[mt][nt][1] = fmaf(g, (ur[mt][0] + vb) + w.y, s[mt][nt][1]);
          s[mt][nt][2] = fmaf(g, (ur[mt][1] + va) + w.z, s[mt][nt][2]);
          s[mt][nt][3] = fmaf(g, (ur[mt][1] + vb) + w.w, s[mt][nt][3]);
        }
      }
    }
    const float lse2 = sm.lse2[i];
    const float2 le = make_float2(kLog2e, kLog2e);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const float c = vis[mt][hh] ? -lse2 : -INFINITY;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float2 x = fma2(make_float2(s[mt][nt][2 * hh], s[mt][nt][2 * hh + 1]), le, make_float2(c, c));
          x.x = fast_exp2(x.x);
          x.y = fast_exp2(x.y);
          if (kHoles) {
            if (!((vis[mt][hh] >> (nt * 8)) & 1u)) x.x = 0.f;
            if (!((vis[mt][hh] >> (nt * 8 + 1)) & 1u)) x.y = 0.f;
          } else if (nt == NT - 1 || MT == 1) {  // MT == 1 serves 1 to 16 keys
            if (nt * 8 + 2 * quad >= n) x.x = 0.f;
            if (nt * 8 + 2 * quad + 1 >= n) x.y = 0.f;
          }
          s[mt][nt][2 * hh] = x.x, s[mt][nt][2 * hh + 1] = x.y;
        }
      }
    if constexpr (kKeySide) {
      float dp[MT][NT][4];
      {
        uint32_t gf[8];
        load_row_pairs(gf, qt + kTgo, i, lane);
        pair_product<MT, NT>(dp, fb, kTv1, kTv2, gf);
        if constexpr (RK > 0) {
          if (p.ml) add_rank_product<MT, NT>(dp, mleft, mright, lane);
        }
      }
      const float nd = -sm.delta[i];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const float2 d = add2(make_float2(dp[mt][nt][2 * hh], dp[mt][nt][2 * hh + 1]), make_float2(nd, nd));
            const float2 x = mul2(make_float2(s[mt][nt][2 * hh], s[mt][nt][2 * hh + 1]), d);
            s[mt][nt][2 * hh] = x.x, s[mt][nt][2 * hh + 1] = x.y;
          }
      if (bias) {
        float rs[MT][2], cs[8], wsum = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) cs[e] = 0.f;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          rs[mt][0] = rs[mt][1] = 0.f;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const float(&x)[4] = s[mt][nt];
            rs[mt][0] += x[0] + x[1];
            rs[mt][1] += x[2] + x[3];
            cs[2 * nt] += x[0] + x[2];
            cs[2 * nt + 1] += x[1] + x[3];
            const float4 w = sm.w[mt * 4 + nt][lane];
            wsum = fmaf(x[0], w.x, fmaf(x[1], w.y, fmaf(x[2], w.z, fmaf(x[3], w.w, wsum))));
            float4& dw = sm.dw[warp][mt * 4 + nt][lane];
            float4 t = dw;
            t.x = fmaf(g, x[0], t.x), t.y = fmaf(g, x[1], t.y), t.z = fmaf(g, x[2], t.z), t.w = fmaf(g, x[3], t.w);
            dw = t;
          }
        }
        // row sums over the quad, column sums over the eight row groups; lane l ends up with row l and with column l
        float r4[4] = {rs[0][0], rs[0][1], MT > 1 ? rs[MT - 1][0] : 0.f, MT > 1 ? rs[MT - 1][1] : 0.f};
        const bool q0 = quad & 1, q1 = quad >> 1;
        float ra = (q0 ? r4[2] : r4[0]) + __shfl_xor_sync(0xffffffffu, q0 ? r4[0] : r4[2], 1);
        float rb = (q0 ? r4[3] : r4[1]) + __shfl_xor_sync(0xffffffffu, q0 ? r4[1] : r4[3], 1);
        float rsum = (q1 ? rb : ra) + __shfl_xor_sync(0xffffffffu, q1 ? ra : rb, 2);  // row 16 q0 + 8 q1 + row8
        const bool c0 = row8 & 1, c1 = (row8 >> 1) & 1, c2 = row8 >> 2;
        float t4[4], t2[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) t4[e] = (c0 ? cs[4 + e] : cs[e]) + __shfl_xor_sync(0xffffffffu, c0 ? cs[e] : cs[4 + e], 4);
#pragma unroll
        for (int e = 0; e < 2; ++e) t2[e] = (c1 ? t4[2 + e] : t4[e]) + __shfl_xor_sync(0xffffffffu, c1 ? t4[e] : t4[2 + e], 8);
        float csum = (c2 ? t2[1] : t2[0]) + __shfl_xor_sync(0xffffffffu, c2 ? t2[0] : t2[1], 16);
        const int rrow = 16 * (int)q0 + 8 * (int)q1 + row8;                             // row of rsum
        const int ccol = 8 * (2 * (int)c0 + (int)c1) + 2 * quad + (int)c2;              // column of csum
        const size_t at = ((size_t)bh * p.N + i) * p.N;
        if (p.du && rrow < p.N) p.du[at + rrow] = g * rsum;
        if (p.dv_bias && ccol < p.N) p.dv_bias[at + ccol] = g * csum;
        if (p.dgate) {
          // sum dS (u + v + w), the common offset of u and v taken out first
          const float off = __shfl_sync(0xffffffffu, ul, 0);
          const float uo = __shfl_sync(0xffffffffu, ul, rrow) - off, vo = __shfl_sync(0xffffffffu, vl, ccol) + off;
          const float tot = warp_sum((rrow < n ? uo * rsum : 0.f) + (ccol < n ? vo * csum : 0.f) + wsum);
          if (lane == 0) p.dgate[(size_t)bh * p.N + i] = tot;
        }
      }
    }
    // P or dS in bf16: pk[mt][nt][hh] = two keys k of one row j; at = its transpose, the A operand over j
    uint32_t pk[MT][2 * KS][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2 * KS; ++nt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) pk[mt][nt][hh] = nt < NT ? pack2_bf16(s[mt][nt < NT ? nt : 0][2 * hh], s[mt][nt < NT ? nt : 0][2 * hh + 1]) : 0u;
    uint32_t at[KS][MT][4];
#pragma unroll
    for (int kt = 0; kt < KS; ++kt)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        at[kt][mt][0] = transpose8x8(pk[mt][2 * kt][0]);
        at[kt][mt][1] = 2 * kt + 1 < NT ? transpose8x8(pk[mt][2 * kt + 1][0]) : 0u;
        at[kt][mt][2] = transpose8x8(pk[mt][2 * kt][1]);
        at[kt][mt][3] = 2 * kt + 1 < NT ? transpose8x8(pk[mt][2 * kt + 1][1]) : 0u;
      }
    if constexpr (RK > 0) {
      // K side: X = dS R_i and dS^T L_i give dL, dR and the gate; V side: T = P MR_i and P^T ML_i give dML, dMR and the
      // coefficients of the basis
      const Factor &fl = kKeySide ? left : mleft, &fr = kKeySide ? right : mright;
      const int rank = kKeySide ? p.ra : p.rm;
      const size_t qi = (size_t)bh * p.N + i;
      float *gl = kKeySide ? p.dal : p.dml, *gr = kKeySide ? p.dar : p.dmr, gate_sum = 0.f;
      if (kKeySide ? p.al != nullptr : p.ml != nullptr) {
#pragma unroll
        for (int rk = 0; rk < RK; ++rk) {
          float t[2 * MT][4], lo = 0.f, hi = 0.f;
          rank_sums<MT>(t, fr, pk, rk, lane);
          float c[KS][2][4];
#pragma unroll
          for (int kt = 0; kt < KS; ++kt)
#pragma unroll
            for (int e = 0; e < 4; ++e) c[kt][0][e] = c[kt][1][e] = 0.f;
          const int ra = 16 * rk + row8, rb = ra + 8;
          const float sa = kKeySide ? ga : sm.dc[i][ra], sb = kKeySide ? ga : sm.dc[i][rb];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            uint32_t h[4], l[4];
            fl.load_t(h, 0, rk, mt, lane);
            fl.load_t(l, 1, rk, mt, lane);
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              const float* x = t[2 * mt + jj];
              lo = fmaf(x[0], bf16_lo(h[2 * jj]) + bf16_lo(l[2 * jj]), fmaf(x[1], bf16_hi(h[2 * jj]) + bf16_hi(l[2 * jj]), lo));
              hi = fmaf(x[2], bf16_lo(h[2 * jj + 1]) + bf16_lo(l[2 * jj + 1]),
                        fmaf(x[3], bf16_hi(h[2 * jj + 1]) + bf16_hi(l[2 * jj + 1]), hi));
              if (gl) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int j = (2 * mt + jj) * 8 + 2 * quad + (e & 1), r = e < 2 ? ra : rb;
                  if (j < p.N && r < rank) gl[(qi * p.N + j) * rank + r] = (e < 2 ? sa : sb) * x[e];
                }
              }
            }
#pragma unroll
            for (int kt = 0; kt < KS; ++kt) {
              mma16(c[kt][0], at[kt][mt], h[0], h[2]);
              mma16(c[kt][0], at[kt][mt], l[0], l[2]);
              mma16(c[kt][1], at[kt][mt], h[1], h[3]);
              mma16(c[kt][1], at[kt][mt], l[1], l[3]);
            }
          }
          if (gr) {
#pragma unroll
            for (int kt = 0; kt < KS; ++kt)
#pragma unroll
              for (int t8 = 0; t8 < 2; ++t8)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int k = kt * 16 + (e >> 1) * 8 + row8, r = 16 * rk + 8 * t8 + 2 * quad + (e & 1);
                  if (k < p.N && r < rank) gr[(qi * p.N + k) * rank + r] = (kKeySide ? ga : sm.dc[i][r]) * c[kt][t8][e];
                }
          }
          if constexpr (kKeySide) {
            gate_sum += lo + hi;
          } else {
            quad_reduce(lo);
            quad_reduce(hi);
            if (p.mcoef && quad == 0) {
              if (ra < rank) p.mcoef[qi * rank + ra] = m_scale * lo;
              if (rb < rank) p.mcoef[qi * rank + rb] = m_scale * hi;
            }
          }
        }
        if (kKeySide && p.dagate) {
          gate_sum = warp_sum(gate_sum);
          if (lane == 0) p.dagate[qi] = a_scale * gate_sum;
        }
      }
    }
    uint32_t xd[8];
    load_row_dup(xd, qt + xr, i, lane);
    float dq[8];
#pragma unroll
    for (int dt = 0; dt < 4; ++dt) {
      float c[2 * MT][4];
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t a[4];
        load_t(a, fb, x2, dt, ks);
#pragma unroll
        for (int jt = 0; jt < 2 * MT; ++jt) {
          const uint32_t b0 = pk[jt >> 1][2 * ks][jt & 1], b1 = pk[jt >> 1][2 * ks + 1][jt & 1];
          if (ks == 0) mma16_first(c[jt], a, b0, b1);
          else mma16(c[jt], a, b0, b1);
        }
      }
      const float xa = bf16_hi(xd[2 * dt]), xb = bf16_hi(xd[2 * dt + 1]);
      float2 lo = make_float2(0.f, 0.f), hi = lo;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        uint32_t kf[4];
        load_t(kf, fb, x1, dt, mt);
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          const int jt = 2 * mt + jj;
          const float2 ca = make_float2(c[jt][0], c[jt][1]), cb = make_float2(c[jt][2], c[jt][3]);
          float(&acc)[4] = a1[dt][jt];
          const float2 na = fma2(ca, make_float2(xa, xa), make_float2(acc[0], acc[1]));
          const float2 nb = fma2(cb, make_float2(xb, xb), make_float2(acc[2], acc[3]));
          acc[0] = na.x, acc[1] = na.y, acc[2] = nb.x, acc[3] = nb.y;
          if constexpr (kKeySide) {
            lo = fma2(ca, make_float2(bf16_lo(kf[2 * jj]), bf16_hi(kf[2 * jj])), lo);
            hi = fma2(cb, make_float2(bf16_lo(kf[2 * jj + 1]), bf16_hi(kf[2 * jj + 1])), hi);
          }
        }
        const uint32_t b0 = mul_bf16x2(kf[0], xd[2 * dt]), b1 = mul_bf16x2(kf[2], xd[2 * dt]);
        const uint32_t b2 = mul_bf16x2(kf[1], xd[2 * dt + 1]), b3 = mul_bf16x2(kf[3], xd[2 * dt + 1]);
#pragma unroll
        for (int kt = 0; kt < KS; ++kt) {
          mma16(a2[kt][2 * dt], at[kt][mt], b0, b1);
          mma16(a2[kt][2 * dt + 1], at[kt][mt], b2, b3);
        }
      }
      if constexpr (kKeySide) dq[2 * dt] = lo.x + lo.y, dq[2 * dt + 1] = hi.x + hi.y;
    }
    if constexpr (kKeySide) {
      quad_sum8(dq, lane);
      const int d0 = (4 * (quad & 1) + 2 * (quad >> 1)) * 8 + row8;
      __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(sm.tile[0]);
      row[row_chunk(0, i, d0 >> 3) / 2 + (d0 & 7)] = __float2bfloat16_rn(dq[0] * p.q_scale);
      row[row_chunk(0, i, (d0 >> 3) + 1) / 2 + (d0 & 7)] = __float2bfloat16_rn(dq[1] * p.q_scale);
    }
  }

  if (bias && kKeySide) {
    __syncthreads();
    if (p.dw) {
      float* dw = p.dw + (size_t)bh * p.N * p.N;
      for (int idx = threadIdx.x; idx < p.N * p.N; idx += 32 * kWarps) {
        const int j = idx / p.N, k = idx - j * p.N;
        float v = 0.f;
        if (j < n && k < n) {
          const int f = (j >> 4) * 4 + (k >> 3), ln = 4 * (j & 7) + ((k & 7) >> 1), e = 2 * ((j >> 3) & 1) + (k & 1);
#pragma unroll
          for (int q = 0; q < kWarps; ++q) v += reinterpret_cast<const float*>(&sm.dw[q][f][ln])[e];
        }
        dw[idx] = v;
      }
    }
  }
#pragma unroll 1
  for (int q = 0; q < kWarps; ++q) {
    __syncthreads();
    if (q != warp) continue;
#pragma unroll
    for (int dt = 0; dt < 4; ++dt)
#pragma unroll
      for (int jt = 0; jt < 2 * MT; ++jt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float& o = sm.acc[0][jt * 8 + 2 * quad + (e & 1)][dt * 16 + (e >> 1) * 8 + row8];
          o = (q ? o : 0.f) + a1[dt][jt][e];
        }
#pragma unroll
    for (int kt = 0; kt < KS; ++kt)
#pragma unroll
      for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          float2& o = *reinterpret_cast<float2*>(&sm.acc[1][kt * 16 + hh * 8 + row8][8 * t + 2 * quad]);
          const float2 old = q ? o : make_float2(0.f, 0.f);
          o = make_float2(old.x + a2[kt][t][2 * hh], old.y + a2[kt][t][2 * hh + 1]);
        }
  }
  __syncthreads();
}

// Both walks and the gradient rows; a lane writes eight channels.
template <int MT, int NT, bool kHoles, bool kBias, int RK, int kWarps, typename Shared>
__device__ __forceinline__ void small_bwd_walks(const SmallBwdParams& p, Shared& sm, int b, int h, int n,
                                                uint32_t kmask, uint32_t qmask) {
  const int bh = b * p.H + h;
  auto store_rows = [&](__nv_bfloat16* g1, __nv_bfloat16* g2) {
    for (int idx = threadIdx.x; idx < 16 * p.N; idx += 32 * kWarps) {
      const int t = idx & 1, r = idx >> 4, c = (idx >> 1) & 7;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < n && ((kmask >> r) & 1u)) {
        const float4 x = *reinterpret_cast<const float4*>(&sm.acc[t][r][8 * c]), y = *reinterpret_cast<const float4*>(&sm.acc[t][r][8 * c + 4]);
        v.x = pack2_bf16(x.x, x.y), v.y = pack2_bf16(x.z, x.w), v.z = pack2_bf16(y.x, y.y), v.w = pack2_bf16(y.z, y.w);
      }
      *reinterpret_cast<uint4*>((t ? g2 : g1) + p.in.at(b, h, r) + 8 * c) = v;
    }
  };
  small_bwd_side<MT, NT, kHoles, kBias, RK, kWarps, false>(p, sm, bh, n, kmask, qmask);
  store_rows(p.dv1, p.dv2);
  __syncthreads();
  small_bwd_side<MT, NT, kHoles, kBias, RK, kWarps, true>(p, sm, bh, n, kmask, qmask);
  store_rows(p.dk1, p.dk2);
}

// kSizes: the variants for molecules beyond 16 keys that the kernel holds, 1 = up to 24, 2 = up to 32.  (Three variants on an SM at a time
// strain its instruction cache; without the bias that costs more than the narrower one saves.  9-29 atoms, both | the wider one alone:
// 64 molecules 60.8 | 57.6 us, 1 024 492 | 480, with the bias 256 187 | 192.)
template <bool kBias, int RK, int kWarps, int kSizes>
__global__ void __launch_bounds__(32 * kWarps, 8 / kWarps) simplicial_small_bwd_kernel(const __grid_constant__ SmallBwdParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  using Shared = SmallBwdShared<kBias, RK, kWarps>;
  Shared& sm = *reinterpret_cast<Shared*>(smem);
  wait_for_previous();
  const bool bias = kBias && (RK == 0 || p.u != nullptr);
  constexpr int kThreads = 32 * kWarps;
  const int tid = threadIdx.x, lane = tid & 31;
  const int N = p.N, h = blockIdx.x % p.H, b = p.order ? p.order[blockIdx.x / p.H] : blockIdx.x / p.H, bh = b * p.H + h;
  const uint32_t kmask = __ballot_sync(0xffffffffu, lane < N && p.key_valid[(size_t)b * N + min(lane, N - 1)] > 0);
  const uint32_t qmask = __ballot_sync(0xffffffffu, lane < N && p.query_valid[(size_t)b * N + min(lane, N - 1)] > 0);
  const int n = qmask ? 32 - __clz(kmask) : 0, nq = n ? 32 - __clz(qmask) : 0;
  if (n > 0) {
    const __nv_bfloat16* src[6] = {p.q, p.k1, p.v1, p.k2, p.v2, p.grad_out};
    const uint32_t t0 = (uint32_t)__cvta_generic_to_shared(sm.tile[0]);
    // a hole in a mask takes the full-size variant, which reads all rows
    const int key_rows = (RK > 0 || p.pair_valid || (kmask & (kmask + 1)) != 0u) ? kSmallRows : (n + 15) & ~15;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const bool query = t == 0 || t == 5;
      const uint32_t mask = query ? qmask : kmask;
      for (int idx = tid; idx < 8 * (query ? nq : key_rows); idx += kThreads) {
        const int r = idx >> 3, c = idx & 7;
        const bool ok = (mask >> r) & 1u;
        cp_async16(row_chunk(t0 + t * kSmallTile, r, c), src[t] + (t == 5 ? p.act : p.in).at(b, h, ok ? r : 0) + c * 8, ok);
      }
    }
    // the bias along with the tiles, so that no query of a walk waits for its rows (256 molecules of 9-29 atoms 193 -> 186 us, 512 of
    // 10-32 408 -> 389)
    if (bias) {
      for (int idx = tid; idx < nq * kSmallRows; idx += kThreads) {
        const int x = idx >> 5, y = idx & 31;
        const size_t at = ((size_t)bh * N + x) * N + min(y, n - 1);
        cp_async4(&sm.u[x][y], p.u + at, y < n);
        cp_async4(&sm.v[x][y], p.v_bias + at, y < n);
      }
      for (int x = tid; x < nq; x += kThreads) cp_async4(&sm.gate[x], p.gate + (size_t)bh * N + x, true);
      for (int idx = tid; idx < 4 * 8 * 32; idx += kThreads) {
        const int f = idx >> 7, ln = (idx >> 2) & 31, e = idx & 3;
        const int j = (f >> 2) * 16 + 8 * (e >> 1) + (ln >> 2), k = (f & 3) * 8 + 2 * (ln & 3) + (e & 1);
        const bool ok = j < n && k < n;
        cp_async4(reinterpret_cast<float*>(&sm.w[f][ln]) + e, p.w + (size_t)bh * N * N + (ok ? j * N + k : 0), ok);
      }
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
  if constexpr (RK > 0) {
    for (int idx = tid; idx < (int)sizeof(sm.factor) / 16; idx += kThreads)
      reinterpret_cast<float4*>(sm.factor)[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // delta_i = dO_i . out_i, eight lanes per query
  for (int idx = tid; idx < ((8 * nq + 31) & ~31); idx += kThreads) {
    const int i = idx >> 3, c = idx & 7;
    float d = 0.f;
    if (i < nq && ((qmask >> i) & 1u)) {
      const float4* o = reinterpret_cast<const float4*>(p.out + ((size_t)bh * N + i) * kD + c * 8);
      const uint4 g = *reinterpret_cast<const uint4*>(p.grad_out + p.act.at(b, h, i) + c * 8);
      const float4 x = o[0], y = o[1];
      d = fmaf(x.x, bf16_lo(g.x), fmaf(x.y, bf16_hi(g.x), fmaf(x.z, bf16_lo(g.y), x.w * bf16_hi(g.y))));
      d = fmaf(y.x, bf16_lo(g.z), fmaf(y.y, bf16_hi(g.z), fmaf(y.z, bf16_lo(g.w), fmaf(y.w, bf16_hi(g.w), d))));
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (c == 0 && i < nq) {
      sm.delta[i] = d;
      sm.lse2[i] = p.lse[(size_t)bh * N + i] * kLog2e;
    }
  }
  cp_async_wait<0>();
  hole = __syncthreads_or(hole) != 0;
  if (n > 0 && p.q_scale != 1.f) {  // a power of two: exact
    const uint32_t scale2 = pack2_bf16(p.q_scale, p.q_scale);
    uint4* q = reinterpret_cast<uint4*>(sm.tile[0]);
    for (int idx = tid; idx < 8 * nq; idx += kThreads) {
      uint4 v = q[idx];
      v.x = mul_bf16x2(v.x, scale2), v.y = mul_bf16x2(v.y, scale2), v.z = mul_bf16x2(v.z, scale2), v.w = mul_bf16x2(v.w, scale2);
      q[idx] = v;
    }
    __syncthreads();
  }
  if constexpr (RK > 0) {
    if (n > 0 && p.ml) {
      const uint32_t go = (uint32_t)__cvta_generic_to_shared(sm.tile[5]);
      const float m_scale = rsqrtf((float)p.rm);
      for (int idx = tid; idx < nq * p.rm; idx += kThreads) {
        const int i = idx / p.rm, r = idx - i * p.rm;
        const float4* bs = reinterpret_cast<const float4*>(p.basis + ((size_t)h * p.rm + r) * kD);
        float d = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 x;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(row_chunk(go, i, c)));
          const float4 y = bs[2 * c], z = bs[2 * c + 1];
          d = fmaf(bf16_lo(x.x), y.x, fmaf(bf16_hi(x.x), y.y, fmaf(bf16_lo(x.y), y.z, fmaf(bf16_hi(x.y), y.w, d))));
          d = fmaf(bf16_lo(x.z), z.x, fmaf(bf16_hi(x.z), z.y, fmaf(bf16_lo(x.w), z.z, fmaf(bf16_hi(x.w), z.w, d))));
        }
        sm.dc[i][r] = m_scale * d;
      }
      __syncthreads();
    }
    // one variant for all sizes: four of them on an SM at a time do not fit its instruction cache (64 molecules of 9-29 atoms at rank 16
    // 174 us with one, 227 with a variant for each size class)
    if (n > 0) small_bwd_walks<2, 4, true, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
  } else if (n > 0) {
    if (hole) small_bwd_walks<2, 4, true, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
    else if (n <= 16) small_bwd_walks<1, 2, false, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
    else if constexpr (kSizes == 1) small_bwd_walks<2, 3, false, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
    else if constexpr (kSizes == 2) small_bwd_walks<2, 4, false, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
    else if (n <= 24) small_bwd_walks<2, 3, false, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
    else small_bwd_walks<2, 4, false, kBias, RK, kWarps>(p, sm, b, h, n, kmask, qmask);
  }
  // the rows of dq, and everything when the molecule has no valid query or key
  __nv_bfloat16* dst[5] = {p.dq, p.dk1, p.dv1, p.dk2, p.dv2};
  for (int idx = tid; idx < (n > 0 ? 1 : 5) * 8 * N; idx += kThreads) {
    const int t = idx / (8 * N), rem = idx - t * 8 * N, r = rem >> 3, c = rem & 7;
    *reinterpret_cast<uint4*>(dst[t] + p.in.at(b, h, r) + 8 * c) =
        t == 0 && r < nq && ((qmask >> r) & 1u) ? *reinterpret_cast<const uint4*>(sm.tile[0] + row_chunk(0, r, c)) : make_uint4(0u, 0u, 0u, 0u);
  }
  if constexpr (RK > 0) {  // residual gradients of queries that no warp took
    float* rows[6] = {p.dal, p.dar, p.dml, p.dmr, p.dagate, p.mcoef};
    const int len[6] = {N * p.ra, N * p.ra, N * p.rm, N * p.rm, 1, p.rm};
    for (int i = tid >> 5; i < N; i += kWarps)
      if (i >= nq || !((qmask >> i) & 1u)) {
#pragma unroll
        for (int t = 0; t < 6; ++t)
          if (rows[t])
            for (int x = lane; x < len[t]; x += 32) rows[t][((size_t)bh * N + i) * len[t] + x] = 0.f;
      }
  }
  if (bias) {
    if (n == 0 && p.dw)
      for (int idx = tid; idx < N * N; idx += kThreads) p.dw[(size_t)bh * N * N + idx] = 0.f;
    // rows of du, dv and dgate that no query wrote
    for (int i = tid >> 5; i < N; i += kWarps)
      if (i >= nq || !((qmask >> i) & 1u)) {
        const size_t at = ((size_t)bh * N + i) * N;
        if (lane < N) {
          if (p.du) p.du[at + lane] = 0.f;
          if (p.dv_bias) p.dv_bias[at + lane] = 0.f;
        }
        if (p.dgate && lane == 0) p.dgate[(size_t)bh * N + i] = 0.f;
      }
  }
}

}  // namespace

int simplicial_small_bwd(const MfSimplicialBwdArgs& a, const TileLayouts* layouts, cudaStream_t stream) {
  SmallBwdParams p{};
  const int rc = simplicial_small_order(a.pair_key_valid, a.batch, a.tokens, a.workspace, a.workspace_bytes,
                                        simplicial_small_order_bytes(a.batch, a.heads, true, a.angle_left || a.message_left), &p.order, stream);
  if (rc != MF_OK) return rc;
  p.grad_out = static_cast<const __nv_bfloat16*>(a.grad_out);
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.k1 = static_cast<const __nv_bfloat16*>(a.k1);
  p.v1 = static_cast<const __nv_bfloat16*>(a.v1);
  p.k2 = static_cast<const __nv_bfloat16*>(a.k2);
  p.v2 = static_cast<const __nv_bfloat16*>(a.v2);
  p.out = a.out;
  p.lse = a.lse;
  p.query_valid = a.query_valid;
  p.key_valid = a.pair_key_valid;
  p.pair_valid = a.pair_valid;
  p.u = a.u, p.v_bias = a.v_bias, p.w = a.w, p.gate = a.gate;
  p.du = a.du, p.dv_bias = a.dv_bias, p.dw = a.dw, p.dgate = a.dgate;
  p.al = a.angle_left, p.ar = a.angle_right, p.agate = a.angle_gate;
  p.ml = a.message_left, p.mr = a.message_right, p.basis = a.message_basis;
  p.dal = a.dangle_left, p.dar = a.dangle_right, p.dagate = a.dangle_gate;
  p.dml = a.dmessage_left, p.dmr = a.dmessage_right, p.mcoef = a.message_coeff;
  p.ra = a.angle_left ? a.angle_rank : 1, p.rm = a.message_left ? a.message_rank : 1;
  p.dq = static_cast<__nv_bfloat16*>(a.dq);
  p.dk1 = static_cast<__nv_bfloat16*>(a.dk1);
  p.dv1 = static_cast<__nv_bfloat16*>(a.dv1);
  p.dk2 = static_cast<__nv_bfloat16*>(a.dk2);
  p.dv2 = static_cast<__nv_bfloat16*>(a.dv2);
  p.H = a.heads;
  p.N = a.tokens;
  p.q_scale = layouts ? layouts->q_scale : 1.f;
  p.in = layouts ? layouts->in : contiguous_rows(a.heads, a.tokens);
  p.act = layouts ? layouts->act : contiguous_rows(a.heads, a.tokens);
  const int bh = a.batch * a.heads;
  // Eight warps of 255 registers fill an SM: four (batch, head)s of two warps each, or two of four.  9-29 atoms x 8 heads, 2 | 4
  // warps: 16 molecules 40.2 | 27.3 us, 64 54.1 | 55.1, 128 95.1 | 91.6, 256 152 | 166, 1024 548 | 623; with the bias the two
  // stay within 3 % of each other from 64 molecules on (128: 131 | 121).  The residuals keep four: their factors are staged per
  // warp, 64 molecules at rank 16 315 | 219 us, 256 1 022 | 785; at rank 32 557 | 507 and 2 109 | 1 951.
  const int warps = bh >= 1024 ? 2 : 4;
  profile_mark(MF_PROFILE_SIMPLICIAL_BWD, true, stream);
  cudaError_t e = cudaSuccess;
#define MF_LAUNCH(BIAS, RK, S, SIZES)                                                                                      \
  do {                                                                                                                 \
    constexpr int bytes = (int)sizeof(SmallBwdShared<BIAS, RK, S>);                                                        \
    auto kernel = simplicial_small_bwd_kernel<BIAS, RK, S, SIZES>;                                                         \
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);                                  \
    if (e == cudaSuccess) launch_dependent(kernel, dim3(bh), dim3(32 * S), bytes, stream, p);                              \
  } while (0)
  if (a.angle_left || a.message_left) {
    if (max(p.ra, p.rm) <= 16) MF_LAUNCH(true, 1, 4, 2);
    else MF_LAUNCH(true, 2, 4, 2);
  } else if (a.u) {
    if (warps == 2) MF_LAUNCH(true, 0, 2, 3);
    else MF_LAUNCH(true, 0, 4, 3);
  } else if (a.tokens <= 24) {
    if (warps == 2) MF_LAUNCH(false, 0, 2, 1);
    else MF_LAUNCH(false, 0, 4, 1);
  } else {
    if (warps == 2) MF_LAUNCH(false, 0, 2, 2);
    else MF_LAUNCH(false, 0, 4, 2);
  }
#undef MF_LAUNCH
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(simplicial_small_bwd_kernel)");
  profile_mark(MF_PROFILE_SIMPLICIAL_BWD, false, stream);
  MF_CHECK_LAUNCH("simplicial_small_bwd_kernel");
  return MF_OK;
}

}  // namespace mf
