// 2-simplicial attention with the factorized bias, backward, 33 to 192 tokens in bf16 (see simplicial_warp.cuh).
//
// First key by first key: for one j the logits over all queries and second keys are a matrix product, and with
//   S_j = (Q o k1_j) K2^T + bias,  dP_j = (dO o v1_j) V2^T,  P = exp(S - lse),  dS = P o (dP - delta)
// five products give all five gradients (query by query it takes six):
//   T_j = dS_j^T Q  -> dk2 += k1_j o T_j, dk1_j = colsum(K2 o T_j)        R_j = P_j^T dO -> dv2 += v1_j o R_j, dv1_j = colsum(V2 o R_j)
//   U_j = dS_j K2   -> dq += k1_j o U_j
// and of the bias gate_i ((u_ij + v_ik) + w_jk): du_ij = gate_i sum_k dS, dv_ik = gate_i sum_j dS, dw_jk = sum_i gate_i dS,
// dgate_i = sum_jk dS ((u_ij + v_ik) + w_jk)  (triton_simplicial_attention.py:660-682).
// A warp owns a block of 16 second keys x 32 queries and walks over the first keys, so that dk2, dv2, dq and the gradient
// of v stay in its registers; the transposed logits (keys as rows) leave dS and P in the registers as the operands of
// T and R.  The eight warps of a CTA go through the first keys in step: what they contribute to row j of dk1, dv1, du and dw
// meets in shared memory and is added up in a fixed order, so results are bit-identical from run to run.
//
// Bound by latency: two warps per scheduler (255 registers) issue an instruction in every third cycle, the tensor pipe is busy
// for a fifth of the time.  64 molecules of 20-181 atoms, 8 heads: 5.91 ms, against 7.81 ms of 128-query tcgen05 tiles, which
// waited for the bias and for the sums over rows and columns of every tile; 32 molecules of 20-64 atoms 0.27 against 0.43 ms.
// Without a bias those tiles have little to wait for, and row-packed ones (simplicial_rows_bwd.cu) are the faster kernel: 1.97
// against 3.8 ms.
#include "common.cuh"
#include "simplicial.cuh"
#include "simplicial_warp.cuh"

namespace mf {
namespace {

constexpr int kBwdWarps = 8;
constexpr int kBwdThreads = 32 * kBwdWarps;
constexpr int kBlocks = kMaxKeys / 32;
constexpr int kUStride = 34;  // floats: pairs of queries stay on 8-byte boundaries

struct WarpBwdParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k1;
  const __nv_bfloat16* v1;
  const __nv_bfloat16* k2;
  const __nv_bfloat16* v2;
  const __nv_bfloat16* grad_out;
  const float* out;
  const float* lse;
  const uint8_t* query_valid;
  const uint8_t* key_valid;
  const uint8_t* pair_valid;
  const float* u;
  const float* v_bias;
  const float* w;
  const float* gate;
  float* dv_bias;
  float* dw;
  float* du;
  float* dgate;
  // fp32 planes: [split] x (BH, N, 64) of dq, dk1, dv1, one of dk2, dv2; [split] x (BH, N, N), first keys by queries, of du;
  // [split] x (BH, N) of dgate
  float* dq_part;
  float* dk1_part;
  float* dv1_part;
  float* dk2_part;
  float* dv2_part;
  float* du_part;
  float* dgate_part;
  __nv_bfloat16* dq;
  __nv_bfloat16* dk1;
  __nv_bfloat16* dv1;
  __nv_bfloat16* dk2;
  __nv_bfloat16* dv2;
  const BatchInfo* info;
  const int32_t* order;
  int H, N, splits;
  size_t row_plane, pair_plane, gate_plane;  // floats
};

struct WarpBwdShared {
  float sums[2][kBwdWarps][2 * kD];  // a step's contributions to dk1_j, dv1_j
  float du[2][kBwdWarps][32];
  float dw[2][kBwdWarps][16];
  float lse2[kMaxKeys], delta[kMaxKeys], gate[kMaxKeys];
  uint32_t visible[kMaxKeys][kBlocks];  // bit k of word (j, kb): the pair (j, 32 kb + k) counts
  uint32_t kmask[kBlocks], qmask[kBlocks];
};
struct WarpBwdBias {
  float u[kBwdWarps][32][kUStride];     // 32 first keys x the warp's queries
  float4 v[kBwdWarps][4][32];           // the warp's block of v_bias in fragment order
};
constexpr int kSharedBytes = (sizeof(WarpBwdShared) + 127) / 128 * 128;
static_assert(kSharedBytes + sizeof(WarpBwdBias) + 6 * kMaxKeys * kRowBytes <= 232448, "227 KB per CTA");

__device__ __forceinline__ void red_add(float* p, float v) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory"); }
__device__ __forceinline__ void red_add2(float* p, float x, float y) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void put(float* p, float v, bool first) {  // the first writer stores, the others add
  if (first) *p = v;
  else red_add(p, v);
}
__device__ __forceinline__ void put2(float* p, float2 v, bool first) {
  if (first) *reinterpret_cast<float2*>(p) = v;
  else red_add2(p, v.x, v.y);
}
__device__ __forceinline__ void cp_async4(uint32_t smem_addr, const void* gptr, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr), "l"(gptr), "r"(valid ? 4 : 0) : "memory");
}
// d = a * b + c, rows 0-7 of c all c0 and rows 8-15 all c1
__device__ __forceinline__ void mma16_rows(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0, float c1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %10, %11, %11};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t v) { return make_float2(bf16_lo(v), bf16_hi(v)); }

// Sums of eight values over the eight row groups of a warp (lanes with the same lane % 4); a lane keeps the value
// 4 bit4 + 2 bit3 + bit2 of its lane number.
__device__ __forceinline__ float row_sum8(float (&v)[8], int lane) {
#pragma unroll
  for (int off = 16, n = 4; off >= 4; off >>= 1, n >>= 1) {
    const bool upper = lane & off;
#pragma unroll
    for (int t = 0; t < n; ++t) {
      const float give = upper ? v[t] : v[t + n], keep = upper ? v[t + n] : v[t];
      v[t] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
  return v[0];
}

__device__ __forceinline__ int next_key(const uint32_t* kmask, int j, int n) {  // first valid key at or behind j, else n
  while (j < n) {
    const uint32_t w = kmask[j >> 5] >> (j & 31);
    if (w) return j + __ffs(w) - 1;
    j = (j | 31) + 1;
  }
  return n;
}

__global__ void __launch_bounds__(kBwdThreads, 1) simplicial_warp_bwd_kernel(const __grid_constant__ WarpBwdParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  WarpBwdShared& sh = *reinterpret_cast<WarpBwdShared*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = lane & 3, row8 = lane >> 2;
  const int N = p.N, per_b = p.H * p.splits;
  const int b = p.order[blockIdx.x / per_b], h = blockIdx.x % per_b / p.splits, split = blockIdx.x % p.splits;
  const int bh = b * p.H + h;
  const int n = p.info[b].n_keys, nq = p.info[b].n_queries;
  // This CTA's blocks: second keys 16 kb0 .. 16 kb1, all queries; the finalize kernels know which splits have any
  const int nkb = (n + 15) >> 4, per = (nkb + p.splits - 1) / p.splits, kb0 = split * per, nk = min(nkb - kb0, per);
  const int nib = (nq + 31) >> 5, tasks = nk * nib;
  if (nk <= 0 || nib == 0) return;
  const size_t base = (size_t)bh * N * kD;
  const size_t nn = (size_t)N * N;

  if (warp < kBlocks) {
    const int t = 32 * warp + lane;
    const uint32_t k = __ballot_sync(0xffffffffu, t < n && p.key_valid[(size_t)b * N + min(t, N - 1)] > 0);
    const uint32_t q = __ballot_sync(0xffffffffu, t < nq && p.query_valid[(size_t)b * N + min(t, N - 1)] > 0);
    if (lane == 0) sh.kmask[warp] = k, sh.qmask[warp] = q;
  }
  __syncthreads();
  const int rows = (max(n, nq) + 31) & ~31, tile = rows * kRowBytes;
  const uint32_t tile0 = (uint32_t)__cvta_generic_to_shared(smem) + kSharedBytes;
  const int tq = 0, tg = tile, tk2 = 2 * tile, tv2 = 3 * tile, tk1 = 4 * tile, tv1 = 5 * tile;
  WarpBwdBias& bias = *reinterpret_cast<WarpBwdBias*>(smem + kSharedBytes + 6 * tile);
  {
    const __nv_bfloat16* src[6] = {p.q, p.grad_out, p.k2, p.v2, p.k1, p.v1};
#pragma unroll
    for (int t = 0; t < 6; ++t)
      for (int idx = tid; idx < 8 * rows; idx += kBwdThreads) {
        const int r = idx >> 3, c = idx & 7;
        const bool ok = ((t < 2 ? sh.qmask : sh.kmask)[r >> 5] >> (r & 31)) & 1u;
        cp_async16(row_chunk(tile0 + t * tile, r, c), src[t] + base + (size_t)(ok ? r : 0) * kD + c * 8, ok);
      }
    cp_async_commit();
  }
  for (int item = warp; item < rows * kBlocks; item += kBwdWarps) {
    const int j = item / kBlocks, kb = item - j * kBlocks;
    uint32_t word = (sh.kmask[j >> 5] >> (j & 31)) & 1u ? sh.kmask[kb] : 0u;
    if (p.pair_valid && word) {
      const int k = 32 * kb + lane;
      word &= __ballot_sync(0xffffffffu, k < N && p.pair_valid[((size_t)b * N + j) * N + min(k, N - 1)] > 0);
    }
    if (lane == 0) sh.visible[j][kb] = word;
  }
  for (int i = warp; i < rows; i += kBwdWarps) {  // a query that does not count has probability 0 everywhere
    const bool ok = (sh.qmask[i >> 5] >> (i & 31)) & 1u;
    float d = 0.f;
    if (ok) {
      const float2 g = unpack_bf16(reinterpret_cast<const uint32_t*>(p.grad_out + base + (size_t)i * kD)[lane]);
      const float2 o = reinterpret_cast<const float2*>(p.out + base + (size_t)i * kD)[lane];
      d = warp_sum(fmaf(g.x, o.x, g.y * o.y));
    }
    if (lane == 0) {
      sh.lse2[i] = ok ? -p.lse[(size_t)bh * N + i] * kLog2e : -INFINITY;
      sh.delta[i] = -d;
      sh.gate[i] = ok ? p.gate[(size_t)bh * N + i] : 0.f;
    }
  }
  cp_async_wait<0>();
  __syncthreads();

  const FragBase fb(tile0, lane);
  float* dk1_out = p.dk1_part + split * p.row_plane + base;
  float* dv1_out = p.dv1_part + split * p.row_plane + base;
  float* du_out = p.du_part + split * p.pair_plane + bh * nn;
  int buf = 0;
  for (int t0 = 0; t0 < tasks; t0 += kBwdWarps) {
    const int active = min(kBwdWarps, tasks - t0);
    const bool on = warp < active;
    const int task = on ? t0 + warp : t0, ib = task / nk, kl = task - ib * nk, kb = kb0 + kl;  // query block by query block
    const int i0 = 32 * ib, k0 = 16 * kb;
    const int ati = i0 * kRowBytes, atk = k0 * kRowBytes;
    float2 dk2[8][2], dv2[8][2], dq[2][8][2];  // [channel 8 c + row8][keys 8 nt + 2 quad]; [16 mt][channels 8 c + 2 quad][row8, + 8]
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) dk2[c][hh] = dv2[c][hh] = dq[0][c][hh] = dq[1][c][hh] = make_float2(0.f, 0.f);
    // Whose parts this warp adds up: those of its queries (du) if it is the first of its query block among the active warps,
    // those of its keys (dw) if it is the first of its key block
    const int du_end = on && (warp == 0 || kl == 0) ? min(active, warp + nk - kl) : 0;
    const int dw_end = on && warp < nk && p.dw ? active : 0;
    if (!on) {  // nothing of this warp's in the sums
      for (int e = lane; e < 2 * kD; e += 32) sh.sums[0][warp][e] = sh.sums[1][warp][e] = 0.f;
    }
    auto collect = [&](int from, int j) {  // the sums of step j, behind its barrier
      const int e = 16 * warp + (lane & 15), half = 4 * (lane >> 4);
      float x = (sh.sums[from][half][e] + sh.sums[from][half + 1][e]) + (sh.sums[from][half + 2][e] + sh.sums[from][half + 3][e]);
      x += __shfl_xor_sync(0xffffffffu, x, 16);
      if (lane < 16) {
        float* dst = (e < kD ? dk1_out : dv1_out - kD) + (size_t)j * kD + e;
        if (t0 == 0) *dst = x;
        else red_add(dst, x);
      }
      if (du_end) {
        float y = 0.f;
        for (int t = warp; t < du_end; ++t) y += sh.du[from][t][lane];
        if (i0 + lane < N) {
          float* dst = du_out + (size_t)j * N + i0 + lane;
          if (kl == 0) *dst = y;
          else red_add(dst, y);
        }
      }
      if (dw_end && lane < 16 && k0 + lane < N) {
        float z = 0.f;
        for (int t = warp; t < dw_end; t += nk) z += sh.dw[from][t][lane];
        float* dst = p.dw + bh * nn + (size_t)j * N + k0 + lane;
        if (ib == 0) *dst = z;
        else red_add(dst, z);
      }
    };
    float2 dvb[4][2], dg[4];
    float dgu = 0.f, wn[2] = {0.f, 0.f};
    int jb = -1;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      dvb[nt][0] = dvb[nt][1] = dg[nt] = make_float2(0.f, 0.f);
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + 8 * nt + 2 * quad + (e & 1), k = k0 + row8 + 8 * (e >> 1);
        const bool in = ((sh.qmask[ib] >> (i & 31)) & 1u) && ((sh.kmask[k >> 5] >> (k & 31)) & 1u);
        v[e] = in ? p.v_bias[bh * nn + (size_t)i * N + k] : 0.f;
      }
      bias.v[warp][nt][lane] = make_float4(v[0], v[1], v[2], v[3]);
    }
    const uint32_t keys_in = sh.kmask[kb >> 1] >> (16 * (kb & 1) + row8);
    const bool kin[2] = {(keys_in & 1u) != 0u, (keys_in & 256u) != 0u};
    const float* w_at = p.w + bh * nn + k0 + row8;
    int j = next_key(sh.kmask, 0, n), jp = -1;
    if (kin[0]) wn[0] = w_at[(size_t)j * N];
    if (kin[1]) wn[1] = w_at[(size_t)j * N + 8];
#pragma unroll 1
    while (j < n) {
      const int jn = next_key(sh.kmask, j + 1, n);
      if (jp >= 0) collect(buf ^ 1, jp);
      if (on) {
        uint32_t row1[8], pk[4][2], dk[4][2];
        {
          float s[4][4], dp[4][4];
          load_row_pairs(row1, tile0 + tk1, j, lane);
          const uint32_t vis = sh.visible[j][kb >> 1] >> (16 * (kb & 1) + row8);
          const float mask0 = vis & 1u ? 0.f : -INFINITY, mask1 = vis & 256u ? 0.f : -INFINITY;  // pairs that do not count
#pragma unroll
          for (int kp = 0; kp < 2; ++kp) {
            uint32_t a0[4], a1[4];
            load_a(a0, fb, tk2 + atk, 0, 2 * kp);
            load_a(a1, fb, tk2 + atk, 0, 2 * kp + 1);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
              uint32_t x[4];
              load_b(x, fb, tq + ati, nt, kp);
#pragma unroll
              for (int e = 0; e < 4; ++e) x[e] = mul_bf16x2(x[e], row1[4 * kp + e]);
              if (kp == 0) mma16_rows(s[nt], a0, x[0], x[1], mask0, mask1);
              else mma16(s[nt], a0, x[0], x[1]);
              mma16(s[nt], a1, x[2], x[3]);
            }
          }
          uint32_t row2[8];
          load_row_pairs(row2, tile0 + tv1, j, lane);
#pragma unroll
          for (int kp = 0; kp < 2; ++kp) {
            uint32_t a[2][4];
#pragma unroll
            for (int k = 0; k < 2; ++k) load_a(a[k], fb, tv2 + atk, 0, 2 * kp + k);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
              uint32_t x[4];
              load_b(x, fb, tg + ati, nt, kp);
#pragma unroll
              for (int e = 0; e < 4; ++e) x[e] = mul_bf16x2(x[e], row2[4 * kp + e]);
              if (kp == 0) mma16_first(dp[nt], a[0], x[0], x[1]);
              else mma16(dp[nt], a[0], x[0], x[1]);
              mma16(dp[nt], a[1], x[2], x[3]);
            }
          }
          float2 wd[2];
          if (j >> 5 != jb) {  // u of the next 32 first keys, read along the rows and turned
            jb = j >> 5;
            __syncwarp();
            const float* u = p.u + bh * nn + (size_t)i0 * N + 32 * jb + lane;
            const bool in = 32 * jb + lane < N;
            const uint32_t q_in = in ? sh.qmask[ib] : 0u, dst = (uint32_t)__cvta_generic_to_shared(&bias.u[warp][lane][0]);
#pragma unroll 8
            for (int r = 0; r < 32; ++r) {
              const bool ok = (q_in >> r) & 1u;
              cp_async4(dst + 4 * r, ok ? u + (size_t)r * N : p.u, ok);
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
          }
          wd[0] = make_float2(wn[0], wn[0]), wd[1] = make_float2(wn[1], wn[1]);
          if (jn < n) {
            if (kin[0]) wn[0] = w_at[(size_t)jn * N];
            if (kin[1]) wn[1] = w_at[(size_t)jn * N + 8];
          }
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const float2 g = *reinterpret_cast<const float2*>(&sh.gate[i0 + 8 * nt + 2 * quad]);
            const float2 u = *reinterpret_cast<const float2*>(&bias.u[warp][j & 31][8 * nt + 2 * quad]);
            const float4 v = bias.v[warp][nt][lane];
            const float2 s0 = fma2(g, add2(add2(u, make_float2(v.x, v.y)), wd[0]), make_float2(s[nt][0], s[nt][1]));
            const float2 s1 = fma2(g, add2(add2(u, make_float2(v.z, v.w)), wd[1]), make_float2(s[nt][2], s[nt][3]));
            s[nt][0] = s0.x, s[nt][1] = s0.y, s[nt][2] = s1.x, s[nt][3] = s1.y;
          }
          float dus[8];
          float2 dw0 = make_float2(0.f, 0.f), dw1 = dw0;
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const float2 l = *reinterpret_cast<const float2*>(&sh.lse2[i0 + 8 * nt + 2 * quad]);
            const float2 d = *reinterpret_cast<const float2*>(&sh.delta[i0 + 8 * nt + 2 * quad]);
            const float2 le = make_float2(kLog2e, kLog2e);
            float2 p0 = fma2(make_float2(s[nt][0], s[nt][1]), le, l), p1 = fma2(make_float2(s[nt][2], s[nt][3]), le, l);
            p0.x = fast_exp2(p0.x), p0.y = fast_exp2(p0.y), p1.x = fast_exp2(p1.x), p1.y = fast_exp2(p1.y);
            const float2 d0 = mul2(p0, add2(make_float2(dp[nt][0], dp[nt][1]), d));
            const float2 d1 = mul2(p1, add2(make_float2(dp[nt][2], dp[nt][3]), d));
            pk[nt][0] = pack2_bf16(p0.x, p0.y), pk[nt][1] = pack2_bf16(p1.x, p1.y);
            dk[nt][0] = pack2_bf16(d0.x, d0.y), dk[nt][1] = pack2_bf16(d1.x, d1.y);
            const float2 g = *reinterpret_cast<const float2*>(&sh.gate[i0 + 8 * nt + 2 * quad]);
            dvb[nt][0] = add2(dvb[nt][0], d0), dvb[nt][1] = add2(dvb[nt][1], d1);
            dg[nt] = fma2(d0, wd[0], fma2(d1, wd[1], dg[nt]));
            dw0 = fma2(g, d0, dw0), dw1 = fma2(g, d1, dw1);
            const float2 t = add2(d0, d1);
            dus[2 * nt] = t.x, dus[2 * nt + 1] = t.y;
          }
          float x0 = dw0.x + dw0.y, x1 = dw1.x + dw1.y;
          quad_reduce(x0);
          quad_reduce(x1);
          if (quad == 0) sh.dw[buf][warp][row8] = x0, sh.dw[buf][warp][row8 + 8] = x1;
          const float du = row_sum8(dus, lane);
          const int e = 4 * ((lane >> 4) & 1) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1), i = 8 * (e >> 1) + 2 * quad + (e & 1);
          sh.du[buf][warp][i] = du;
          dgu = fmaf(bias.u[warp][j & 31][i], du, dgu);
        }
        {  // U_j = dS_j K2
          uint32_t a[2][4];
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            a[mt][0] = transpose8x8(dk[2 * mt][0]);
            a[mt][1] = transpose8x8(dk[2 * mt + 1][0]);
            a[mt][2] = transpose8x8(dk[2 * mt][1]);
            a[mt][3] = transpose8x8(dk[2 * mt + 1][1]);
          }
#pragma unroll
          for (int dp = 0; dp < 4; ++dp) {
            uint32_t x[4];
            load_t2(x, fb, tk2 + atk, dp, 0);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              const int c = 2 * dp + t;
              const float2 r = unpack_bf16(row1[c]);
#pragma unroll
              for (int mt = 0; mt < 2; ++mt) {
                float o[4];
                mma16_first(o, a[mt], x[2 * t], x[2 * t + 1]);
                dq[mt][c][0] = fma2(r, make_float2(o[0], o[1]), dq[mt][c][0]);
                dq[mt][c][1] = fma2(r, make_float2(o[2], o[3]), dq[mt][c][1]);
              }
            }
          }
        }
        // T_j^T = Q^T dS_j and R_j^T = dO^T P_j (channels as rows): acc += row o T, and the sum over the keys of y o T
        auto keys = [&](const uint32_t(&f)[4][2], int x_tile, int y_tile, int row_tile, float2(&acc)[8][2], float* sums) {
          uint32_t row[8];
          load_row_dup(row, tile0 + row_tile, j, lane);
          float v[8];
#pragma unroll
          for (int dt = 0; dt < 4; ++dt) {
            uint32_t x0[4], x1[4], y[4];
            load_t(x0, fb, x_tile + ati, dt, 0);
            load_t(x1, fb, x_tile + ati, dt, 1);
            load_t(y, fb, y_tile + atk, dt, 0);
            float2 sum[2];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              float o[4];
              mma16_first(o, x0, f[0][nt], f[1][nt]);
              mma16(o, x1, f[2][nt], f[3][nt]);
#pragma unroll
              for (int hh = 0; hh < 2; ++hh) {
                const int c = 2 * dt + hh;
                const float r = bf16_hi(row[c]);
                const float2 t = make_float2(o[2 * hh], o[2 * hh + 1]), k = unpack_bf16(y[2 * nt + hh]);
                acc[c][nt] = fma2(make_float2(r, r), t, acc[c][nt]);
                sum[hh] = nt == 0 ? mul2(k, t) : fma2(k, t, sum[hh]);
              }
            }
            v[2 * dt] = sum[0].x + sum[0].y, v[2 * dt + 1] = sum[1].x + sum[1].y;
          }
          quad_sum8(v, lane);
          const int d0 = (4 * (quad & 1) + 2 * (quad >> 1)) * 8 + row8;  // the lane's two channels: d0 and d0 + 8
          sums[d0] = v[0], sums[d0 + 8] = v[1];
        };
        keys(dk, tq, tk2, tk1, dk2, sh.sums[buf][warp]);
        keys(pk, tg, tv2, tv1, dv2, sh.sums[buf][warp] + kD);
      }
      __syncthreads();  // the other buffer's sums were read before the barrier
      buf ^= 1;
      jp = j;
      j = jn;
    }
    collect(buf ^ 1, jp);
    // the blocks' gradients, one warp after the other: the first block of a query block (key block) stores, the others add
    for (int turn = 0; turn < active; ++turn) {
      if (turn == warp) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int k = k0 + 8 * hh + 2 * quad + e;
            if (k < N) {
              float* d2 = p.dk2_part + base + (size_t)k * kD + row8;
              float* e2 = p.dv2_part + base + (size_t)k * kD + row8;
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                put(d2 + 8 * c, e ? dk2[c][hh].y : dk2[c][hh].x, ib == 0);
                put(e2 + 8 * c, e ? dv2[c][hh].y : dv2[c][hh].x, ib == 0);
              }
            }
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            const int i = i0 + 16 * mt + 8 * hh + row8;
            if (i < N) {
              float* d = p.dq_part + split * p.row_plane + base + (size_t)i * kD + 2 * quad;
#pragma unroll
              for (int c = 0; c < 8; ++c) put2(d + 8 * c, dq[mt][c][hh], kl == 0);
            }
          }
        }
        float x[8];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const float4 v = bias.v[warp][nt][lane];
          const float2 t = fma2(make_float2(v.x, v.y), dvb[nt][0], fma2(make_float2(v.z, v.w), dvb[nt][1], dg[nt]));
          x[2 * nt] = t.x, x[2 * nt + 1] = t.y;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = i0 + 8 * nt + 2 * quad + (e & 1), k = k0 + row8 + 8 * (e >> 1);
            const float d = e & 1 ? dvb[nt][e >> 1].y : dvb[nt][e >> 1].x;
            if (p.dv_bias && i < N && k < N) p.dv_bias[bh * nn + (size_t)i * N + k] = sh.gate[i] * d;
          }
        }
        const float y = row_sum8(x, lane) + dgu;
        const int e = 4 * ((lane >> 4) & 1) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1), i = i0 + 8 * (e >> 1) + 2 * quad + (e & 1);
        if (i < N) {
          float* dst = p.dgate_part + split * p.gate_plane + (size_t)bh * N + i;
          if (kl == 0) *dst = y;
          else red_add(dst, y);
        }
      }
      __syncthreads();
    }
  }
}

// How many splits have blocks
__device__ __forceinline__ int live_splits(const BatchInfo& info, int splits) {
  const int nkb = (info.n_keys + 15) >> 4;
  const int per = (nkb + splits - 1) / splits;
  return per ? (nkb + per - 1) / per : 0;
}

// Sums the planes in a fixed order and writes the gradients; rows of tokens that take no part get exact zeros.
__global__ void __launch_bounds__(256) simplicial_warp_bwd_finalize_kernel(const __grid_constant__ WarpBwdParams p, int BH) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // one thread per 4 elements
  if (idx >= (long long)BH * p.N * (kD / 4)) return;
  const int d4 = (int)(idx % (kD / 4)), row = (int)(idx / (kD / 4) % p.N), bh = (int)(idx / ((long long)(kD / 4) * p.N)), b = bh / p.H;
  const BatchInfo info = p.info[b];
  const int splits = live_splits(info, p.splits);
  const size_t off = ((size_t)bh * p.N + row) * kD + 4 * d4;
  const bool q_ok = row < info.n_queries && p.query_valid[(size_t)b * p.N + row] > 0;
  const bool k_ok = row < info.n_keys && p.key_valid[(size_t)b * p.N + row] > 0 && info.n_queries > 0;
  auto write = [&](__nv_bfloat16* dst, const float* src, bool ok, int planes) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ok)
      for (int s = 0; s < planes; ++s) {
        const float4 v = *reinterpret_cast<const float4*>(src + s * p.row_plane + off);
        a.x += v.x, a.y += v.y, a.z += v.z, a.w += v.w;
      }
    *reinterpret_cast<uint2*>(dst + off) = make_uint2(pack2_bf16(a.x, a.y), pack2_bf16(a.z, a.w));
  };
  write(p.dq, p.dq_part, q_ok, splits);
  write(p.dk1, p.dk1_part, k_ok, splits);
  write(p.dv1, p.dv1_part, k_ok, splits);
  write(p.dk2, p.dk2_part, k_ok, 1);
  write(p.dv2, p.dv2_part, k_ok, 1);
  if (d4 == 0 && p.dgate) {
    float g = 0.f;
    if (q_ok)
      for (int s = 0; s < splits; ++s) g += p.dgate_part[s * p.gate_plane + (size_t)bh * p.N + row];
    p.dgate[(size_t)bh * p.N + row] = g;
  }
}

// du_ij = gate_i sum_k dS from the planes, which hold one first key's sums of all queries in a row: 32 x 32 tiles, turned in
// shared memory.
__global__ void __launch_bounds__(256) simplicial_warp_bwd_du_kernel(const __grid_constant__ WarpBwdParams p) {
  __shared__ float tile[32][33];
  const int bh = blockIdx.z, b = bh / p.H, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32, N = p.N;
  const BatchInfo info = p.info[b];
  const int splits = live_splits(info, p.splits);
  const size_t at = (size_t)bh * N * N;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int j = j0 + warp + 8 * t, i = i0 + lane;
    float v = 0.f;
    if (i < info.n_queries && j < info.n_keys && p.query_valid[(size_t)b * N + i] > 0 && p.key_valid[(size_t)b * N + j] > 0)
      for (int s = 0; s < splits; ++s) v += p.du_part[s * p.pair_plane + at + (size_t)j * N + i];
    tile[warp + 8 * t][lane] = v;
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int i = i0 + warp + 8 * t, j = j0 + lane;
    if (i < N && j < N) p.du[at + (size_t)i * N + j] = p.gate[(size_t)bh * N + i] * tile[lane][warp + 8 * t];
  }
}

struct WarpBwdLayout {
  int splits;
  size_t info, order, row_plane, pair_plane, gate_plane, dq, dk1, dv1, dk2, dv2, du, dgate, total;  // planes in floats, the rest in bytes
};
// Splits: CTAs for two waves, but no more than the batch needs - every split has its own planes of dq, dk1, dv1 and du -
// nor than leave every warp of a CTA a block.
WarpBwdLayout warp_bwd_layout(const MfSimplicialBwdArgs& a) {
  WarpBwdLayout l{};
  const size_t bh = (size_t)a.batch * a.heads, n = a.tokens;
  l.splits = 1;
  const int blocks = ((a.tokens + 15) / 16) * ((a.tokens + 31) / 32);
  while (l.splits < 4 && bh * l.splits < 296 && blocks >= kBwdWarps * (l.splits + 1)) ++l.splits;
  size_t off = simplicial_schedule_layout(a.batch, &l.info, &l.order);
  l.row_plane = align_up(bh * n * kD, 64);
  l.pair_plane = align_up(bh * n * n, 64);
  l.gate_plane = align_up(bh * n, 64);
  auto take = [&](size_t floats) {
    const size_t at = off;
    off += floats * sizeof(float);
    return at;
  };
  l.dq = take(l.row_plane * l.splits);
  l.dk1 = take(l.row_plane * l.splits);
  l.dv1 = take(l.row_plane * l.splits);
  l.dk2 = take(l.row_plane);
  l.dv2 = take(l.row_plane);
  l.du = take(l.pair_plane * l.splits);
  l.dgate = take(l.gate_plane * l.splits);
  l.total = off;
  return l;
}

}  // namespace

size_t simplicial_warp_bwd_workspace_bytes(const MfSimplicialBwdArgs& a) { return warp_bwd_layout(a).total; }

int simplicial_warp_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream) {
  const WarpBwdLayout l = warp_bwd_layout(a);
  char* ws = static_cast<char*>(a.workspace);
  WarpBwdParams p{};
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.k1 = static_cast<const __nv_bfloat16*>(a.k1);
  p.v1 = static_cast<const __nv_bfloat16*>(a.v1);
  p.k2 = static_cast<const __nv_bfloat16*>(a.k2);
  p.v2 = static_cast<const __nv_bfloat16*>(a.v2);
  p.grad_out = static_cast<const __nv_bfloat16*>(a.grad_out);
  p.out = a.out, p.lse = a.lse;
  p.query_valid = a.query_valid, p.key_valid = a.pair_key_valid, p.pair_valid = a.pair_valid;
  p.u = a.u, p.v_bias = a.v_bias, p.w = a.w, p.gate = a.gate;
  p.dv_bias = a.dv_bias, p.dw = a.dw, p.du = a.du, p.dgate = a.dgate;
  auto plane = [&](size_t at) { return reinterpret_cast<float*>(ws + at); };
  p.dq_part = plane(l.dq), p.dk1_part = plane(l.dk1), p.dv1_part = plane(l.dv1), p.dk2_part = plane(l.dk2), p.dv2_part = plane(l.dv2);
  p.du_part = plane(l.du), p.dgate_part = plane(l.dgate);
  p.dq = static_cast<__nv_bfloat16*>(a.dq);
  p.dk1 = static_cast<__nv_bfloat16*>(a.dk1);
  p.dv1 = static_cast<__nv_bfloat16*>(a.dv1);
  p.dk2 = static_cast<__nv_bfloat16*>(a.dk2);
  p.dv2 = static_cast<__nv_bfloat16*>(a.dv2);
  BatchInfo* info = reinterpret_cast<BatchInfo*>(ws + l.info);
  int32_t* order = reinterpret_cast<int32_t*>(ws + l.order);
  p.info = info, p.order = order;
  p.H = a.heads, p.N = a.tokens, p.splits = l.splits;
  p.row_plane = l.row_plane, p.pair_plane = l.pair_plane, p.gate_plane = l.gate_plane;
  const int rc = launch_schedule(a.query_valid, a.pair_key_valid, a.batch, a.tokens, info, order, reinterpret_cast<int32_t*>(ws), stream);
  if (rc != MF_OK) return rc;
  const int bh = a.batch * a.heads, rows = (a.tokens + 31) & ~31;
  const int bytes = kSharedBytes + 6 * rows * kRowBytes + (int)sizeof(WarpBwdBias);
  const cudaError_t e = cudaFuncSetAttribute(simplicial_warp_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(simplicial_warp_bwd_kernel)");
  profile_mark(MF_PROFILE_SIMPLICIAL_BWD, true, stream);
  simplicial_warp_bwd_kernel<<<bh * l.splits, kBwdThreads, bytes, stream>>>(p);
  profile_mark(MF_PROFILE_SIMPLICIAL_BWD, false, stream);
  MF_CHECK_LAUNCH("simplicial_warp_bwd_kernel");
  simplicial_warp_bwd_finalize_kernel<<<(unsigned)(((long long)bh * a.tokens * (kD / 4) + 255) / 256), 256, 0, stream>>>(p, bh);
  MF_CHECK_LAUNCH("simplicial_warp_bwd_finalize_kernel");
  if (a.du) {
    const int t = (a.tokens + 31) / 32;
    simplicial_warp_bwd_du_kernel<<<dim3(t, t, bh), 256, 0, stream>>>(p);
    MF_CHECK_LAUNCH("simplicial_warp_bwd_du_kernel");
  }
  return MF_OK;
}

}  // namespace mf
