// 2-simplicial attention with the factorized bias on the Blackwell tensor cores, forward and backward, 33 to 192 tokens in bf16.
//
// The logits S_ijk = sum_d q_id k1_jd k2_kd + gate_i ((u_ij + v_ik) + w_jk) treat queries, first keys and second keys alike, and so
// do their gradients.  A pass gives every row of a 128-row tile a pair (x, y) of two of the three sets and walks over y; the third
// set is the columns:
//     S[r, z] = sum_d (X_x o Y_y)[d] Z[z, d]      dP[r, z] = sum_d (X'_x o Y'_y)[d] Z'[z, d]     (X', Y', Z' from dO, v1, v2)
//     T = dS Z,  R = P Z',  acc_x += Y_y o T,  acc'_x += Y'_y o R
// The forward pass is the pass (query, first key | second key) with W = P V2 alone; the backward pass runs three of them:
//     1  rows (i, j), columns k: dq_i, du_ij (row sums), dgate_i          (triton_simplicial_attention.py:660-682)
//     2  rows (j, k), columns i: dk1_j, dv1_j, dw_jk
//     3  rows (k, i), columns j: dk2_k, dv2_k, dv_ik
// Every result is a sum along rows that one thread owns, so nothing is transposed through shared memory, nothing crosses lanes
// and nothing is atomic; the price is that S, dP and P are formed three times.  A = X o Y is written to tensor memory, P and dS
// take the place of S and dP there, Z and Z' stay in shared memory: an MMA fetches its 64-row B operand from there and nothing
// else.  Of the bias, the operand of (x, z) is a tile in shared memory, that of (y, z) and of (x, y) comes in stages of a step.
//
// Rows are packed as in simplicial_rows.cuh: `groups` consecutive y per step.  Columns go in chunks of at most 64; chunk q
// belongs to softmax group q & 1, so one group's exponentials run under the other group's products.  The softmax warps do
// nothing else; the row warps write A and add up T and R (one kind of warp for both, with one chain of waits, took 1.4 times
// as long).  One thread issues every MMA, two warps stage the bias operands of coming steps.  Waits are bounded.
//
// The softmax takes shift 0; a tile in which a row's sum leaves 2^-60 .. 2^60 is done again with its exact maxima.
//
// Each pass rounds the products of its own pair of operands (q k1, k1 k2 or k2 q) to bf16 before it forms S.  The log-sum-exp comes
// from the first, so P of the other two is normalised up to that rounding, and dk1, dv1, dw, dk2, dv2, dv belong to logits that
// differ in their last bits from those of dq, du and dgate.  The errors against 64 bits are those of one rounding (2-3e-3).
//
// When a wait expires, the rows of the tile leave as zeros (forward; the failure is shared at the barrier that ends a pass), or a
// last launch clears every gradient (backward).
//
// Bound by the chain of hand-overs of a step (half of the time is left with no MMA and no arithmetic at all) and the softmax
// warps' instructions; the tensor pipe is busy for 16 to 20 % of the time.  The backward kernel spills (326 bytes of stores, 432 of
// loads by ptxas): one register split serves its three passes, whose accumulators differ.  Of the CTAs launched, six per pass, half
// to five sixths find no tile and return (up to 96 tokens a molecule has at most four, up to 64 at most two).
// 64 molecules of 20-181 atoms of 192 tokens, 8 heads: forward 0.86 ms, backward 3.65 ms (mma.sync kernels, query by query and first
// key by first key: 1.82 and 6.09 ms); 64 full ones of 64 tokens 0.19 and 0.68 ms (0.24 and 0.96).  A single molecule of 181: 0.14
// and 0.23 ms (0.12, which is why short forward calls stay there, and 1.54).
#include <climits>

#include "common.cuh"
#include "simplicial.cuh"
#include "simplicial_rows.cuh"
#include "simplicial_sm100.cuh"
#include "simplicial_warp.cuh"
#include "sm100_primitives.cuh"

namespace mf {
namespace {

enum { kFwd = 0, kDq = 1, kDk1 = 2, kDk2 = 3 };  // passes

// Warps: 0-7 softmax (two groups of four), 8-15 rows (two groups of four: operands, accumulators), 16 issues, 17 and 18 load
constexpr int kExpWarps = 8, kRowWarps = 8;
constexpr int kIssuerWarp = kExpWarps + kRowWarps, kBiasLoader = kIssuerWarp + 1, kPairLoader = kIssuerWarp + 2;
constexpr int kTriThreads = 32 * (kIssuerWarp + 4);
// Registers by role: the sum over the warps is the launch's
template <bool kForward>
struct Regs {
  static constexpr int kExp = kForward ? 112 : 88, kRow = kForward ? 96 : 128, kAux = kForward ? 64 : 48;
  static_assert(kExpWarps * kExp + kRowWarps * kRow + 4 * kAux <= kTriThreads / 32 * 96, "register hand-over exceeds the CTA's pool");
};
constexpr int kRegLaunch = 96;
constexpr int kWords = kMaxKeys / 32;
constexpr int kStages = 8;                    // steps whose bias operands are in shared memory
constexpr int kYRows = kMaxKeys + kMaxGroups; // rows Y_y, with those of a last step that is not full

// tensor memory columns: A of two steps | T, R | chunk buffers
constexpr int kColT = 128, kColR = 192, kColS = 256;
constexpr int kTmemCols = 512;

// shared memory (1024-byte aligned)
constexpr int kOffZ = 0;                                        // [192][64] bf16, 128-byte swizzle
constexpr int kOffZ2 = kOffZ + kMaxKeys * 128;
constexpr int kOffY = kOffZ2 + kMaxKeys * 128;                  // [200][64] bf16: the valid Y_y in order
constexpr int kOffY2 = kOffY + kYRows * 128;
constexpr int kOffBits = kOffY2 + kYRows * 128;                 // [192][6]: pairs of keys that count
constexpr int kOffCols = kOffBits + kMaxKeys * kWords * 4;      // [3][192]: -lse log2e, -delta, gate of the queries
constexpr int kOffSums = kOffCols + 3 * kMaxKeys * 4;           // [4 steps][2][128] row sums
constexpr int kOffDgate = kOffSums + 4 * 2 * kTileM * 4;         // [2][128]
constexpr int kOffTile = kOffDgate + 2 * kTileM * 4;         // bias: operand of (x, z), then that of (y, z) by stages
static_assert(kOffTile % 128 == 0, "alignment");
constexpr int tri_smem_bytes(int tokens) {
  // tile: (rows | 1) x columns, stages: groups x columns; rows * groups <= 128, so 129 + kStages rows of floats at most
  return kOffTile + 1024 + kStages * kTileM * 4 + (129 + kStages) * ((tokens + 15) & ~15) * 4;
}

// The split of a molecule into tiles of (x, y) rows, as plan_rows() of simplicial_rows.cuh, but a tile costs kTileCost steps
// besides its own (loads, the pipeline's first and last step).  More than five tiles for the sake of fuller rows save nothing: 64
// molecules of 20-181 atoms, steps + 5 per tile at most 8 | 6 | 4 | 3 tiles: 60.5 | 60.5 | 61.3 | 63.8 thousand.
// A call lasts at least as long as its longest tile, and beyond kShortWalk x the cheapest split may have tiles of one first key a step
// (rows of more than 64 x), 100 to 128 steps long, or of two, up to 96.  There the split with the fewest steps is taken of those, of up to
// six tiles, whose cost is within kSlack hundredths of the lowest.  Backward, 8 heads, us, slack 0 | 7 | 10: 1 molecule of 101 atoms 278 |
// 96 | 78, of 128 345 | 190 | 117, of 181 417 | 229 | 231; 4 of 43-128 343 | 190 | 164, of 60-181 454 | 375 | 375; 64 of 128 3 305 | 3 307 |
// 3 515, of 181 10 357 | 11 009 | 11 015; 64 of 20-181 atoms of 192 tokens, forward + backward, 4 436 | 4 511 | 4 525.
// The split depends on the molecule alone, so that its results do not depend on the batch it is in: more tiles for small batches only
// would cost the large ones nothing.
constexpr int kTileCost = 4, kMostTiles = 6, kShortWalk = 100, kSlack = 7;
struct TriPlan {
  int tiles, rows;
};
__device__ inline TriPlan tri_plan(int nx, int ny) {
  TriPlan best{0, 0};
  if (nx <= 0 || ny <= 0) return best;
  const int most = nx > kShortWalk ? kMostTiles : kMostTiles - 1, slack = nx > kShortWalk ? kSlack : 0;
  int cost[kMostTiles], steps[kMostTiles], lowest = INT_MAX;
#pragma unroll
  for (int t = 0; t < kMostTiles; ++t) {  // t + 1 tiles or fewer
    const int rows = (nx + t) / (t + 1), groups = min(kTileM / rows, kMaxGroups);
    cost[t] = INT_MAX, steps[t] = 0;
    if (rows > kTileM || t >= most) continue;
    steps[t] = (ny + groups - 1) / groups;
    cost[t] = (nx + rows - 1) / rows * (steps[t] + kTileCost);
    lowest = min(lowest, cost[t]);
  }
  const int limit = (100 + slack) * lowest / 100;
  int fewest = INT_MAX, chosen = 0;
#pragma unroll
  for (int t = 0; t < kMostTiles; ++t)
    if (cost[t] <= limit && (slack > 0 ? steps[t] < fewest : fewest == INT_MAX)) fewest = steps[t], chosen = t + 1;
  best.rows = (nx + chosen - 1) / chosen;
  best.tiles = (nx + best.rows - 1) / best.rows;
  return best;
}

struct TriParams {
  const __nv_bfloat16* main[3];   // q, k1, k2
  const __nv_bfloat16* other[3];  // grad_out, v1, v2
  const uint8_t* query_valid;
  const uint8_t* key_valid;
  const uint8_t* pair_valid;
  const float* u;
  const float* v_bias;
  const float* w;
  const float* gate;
  float* out;                     // forward
  float* lse;
  __nv_bfloat16* out_cast;
  const float* lse2;              // backward: -lse log2e and -delta, (BH, N), of valid queries
  const float* ndelta;
  __nv_bfloat16* grad_main[3];    // dq, dk1, dk2
  __nv_bfloat16* grad_other[3];   // -, dv1, dv2
  float* du;
  float* dv_bias;
  float* dw;
  float* dgate;
  const BatchInfo* info;
  const int2* items;              // [0].x = count, then {batch | pass << 16 | tile << 20, rows | tiles << 8}
  int32_t* status;
  int H, N;
  BoundedWaits waits;
};

__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async16_part(uint32_t dst, const void* src, int bytes) {  // zeros behind `bytes`
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_f32(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
template <int kId>  // 1: softmax warps, 2: row warps
__device__ __forceinline__ void group_barrier() {
  asm volatile("bar.sync %0, %1;" ::"n"(kId), "n"(256) : "memory");
}

struct TriShared {
  uint64_t bar_a[2], bar_free[2], bar_s[4], bar_p[4], bar_t[2], bar_d[2];
  uint64_t bar_full[kStages], bar_empty[kStages];
  uint64_t bar_drain;
  uint32_t tmem;
  int gave_up;               // forward: a wait of any thread has expired
  uint32_t mask[2][kWords];  // valid queries, valid keys
  uint8_t ylist[kMaxKeys];   // the valid y in order
};

template <int kPass>
__device__ __forceinline__ void tri_tile(const TriParams& p, TriShared& sh, uint8_t* smem, int2 item, int h) {
  constexpr bool kForward = kPass == kFwd;
  constexpr int X = kPass == kDk1 ? 1 : kPass == kDk2 ? 2 : 0;  // 0 queries, 1 first keys, 2 second keys
  constexpr int Y = (X + 1) % 3, Z = (X + 2) % 3;
  constexpr int kBufs = kForward ? 4 : 2, kBufCols = kForward ? 64 : 128;  // chunk buffers
  constexpr int kACols = kForward ? 32 : 64;                               // tensor memory of one step's A
  constexpr bool kHalf = kPass == kFwd || kPass == kDq;  // one result: each group takes half of its channels
  constexpr int kAcc = kHalf ? 32 : 64;
  constexpr int kSumBufs = kHalf ? 2 : 1;                // T of two steps where there is no R

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = item.x & 0xffff, tile = item.x >> 20, rt = item.y & 0xff, tiles = item.y >> 8;  // rt: rows x of a tile
  const int N = p.N, bh = b * p.H + h;
  const size_t base = (size_t)bh * N * kD, nn = (size_t)bh * N * N;
  const BatchInfo info = p.info[b];
  auto extent = [&](int axis) { return axis == 0 ? info.n_queries : info.n_keys; };
  const int nx = extent(X), nz = extent(Z), ny = Y == 0 ? info.reserved1 : info.reserved0;  // ny: valid ones
  // rows that no tile covers
  if (tile == 0) {
    const int z0 = tiles > 0 ? nx : 0;
    for (int idx = tid; idx < (N - z0) * (kD / 8); idx += kTriThreads) {
      const uint4 zero = make_uint4(0, 0, 0, 0);
      if constexpr (kForward) {
        float4* o = reinterpret_cast<float4*>(p.out + base + (size_t)z0 * kD) + 2 * idx;
        o[0] = o[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.out_cast) reinterpret_cast<uint4*>(p.out_cast + base + (size_t)z0 * kD)[idx] = zero;
      } else {
        reinterpret_cast<uint4*>(p.grad_main[X] + base + (size_t)z0 * kD)[idx] = zero;
        if constexpr (X != 0) reinterpret_cast<uint4*>(p.grad_other[X] + base + (size_t)z0 * kD)[idx] = zero;
      }
    }
    if constexpr (kForward)
      for (int idx = z0 + tid; idx < N; idx += kTriThreads) p.lse[(size_t)bh * N + idx] = 0.f;
  }
  if (tiles == 0) return;  // uniform per CTA

  const int G = min(kTileM / rt, kMaxGroups), steps = (ny + G - 1) / G;  // y per step
  const int units = (nz + 15) >> 4, zpad = 16 * units;             // columns by 16
  const int C = (units + 3) >> 2, per = units / C, extra = units % C;  // chunks of a step: per or per + 1 units

  if (tid == 0) {
    auto count = [&](int which, int n) { return (uint32_t)(n + (p.waits.withheld == which)); };  // (see BoundedWaits)
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.bar_a[i], count(0, kRowWarps));
      mbar_init(&sh.bar_free[i], count(1, 1));
      mbar_init(&sh.bar_t[i], count(2, 1));
      mbar_init(&sh.bar_d[i], count(3, kRowWarps));
    }
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(&sh.bar_s[i], count(4, 1));
      mbar_init(&sh.bar_p[i], count(5, 4));
    }
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&sh.bar_full[i], count(6, 64));
      mbar_init(&sh.bar_empty[i], count(7, kExpWarps));
    }
    mbar_init(&sh.bar_drain, 1);
    mbar_fence_init();
    sh.gave_up = 0;
  }
  if (warp == kIssuerWarp) {
    tmem_alloc(&sh.tmem, kTmemCols);
    tmem_relinquish();
  }
  if (warp < kWords) {
    const int t = 32 * warp + lane;
    const uint32_t q = __ballot_sync(0xffffffffu, t < N && p.query_valid[(size_t)b * N + min(t, N - 1)] > 0);
    const uint32_t k = __ballot_sync(0xffffffffu, t < N && p.key_valid[(size_t)b * N + min(t, N - 1)] > 0);
    if (lane == 0) sh.mask[0][warp] = q, sh.mask[1][warp] = k;
  }
  __syncthreads();
  auto valid = [&](int axis, int t) { return ((sh.mask[axis != 0][t >> 5] >> (t & 31)) & 1u) != 0u; };
  float* cols = reinterpret_cast<float*>(smem + kOffCols);  // -lse log2e | -delta | gate of the queries
  {
    // Z and Z': rows that do not count are zeros
    const uint32_t t0 = smem_u32(smem);
    for (int idx = tid; idx < 8 * zpad; idx += kTriThreads) {
      const int r = idx >> 3, c = idx & 7;
      const bool ok = r < nz && valid(Z, r);
      const size_t at = base + (size_t)(ok ? r : 0) * kD + c * 8;
      cp_async16(row_chunk(t0 + kOffZ, r, c), p.main[Z] + at, ok);
      cp_async16(row_chunk(t0 + kOffZ2, r, c), p.other[Z] + at, ok);
    }
    // Y and Y', without the rows that do not count
    auto y_row = [&](int t) {
      const uint32_t* m = sh.mask[Y != 0];
      int pos = __popc(m[t >> 5] & ((1u << (t & 31)) - 1u));
      for (int c = 0; c < (t >> 5); ++c) pos += __popc(m[c]);
      return pos;
    };
    for (int idx = tid; idx < 8 * min(kMaxKeys, N); idx += kTriThreads) {
      const int r = idx >> 3, c = idx & 7;
      if (!valid(Y, r)) continue;
      const int pos = y_row(r);
      const size_t at = base + (size_t)r * kD + c * 8;
      cp_async16(t0 + kOffY + pos * 128 + c * 16, p.main[Y] + at, true);
      cp_async16(t0 + kOffY2 + pos * 128 + c * 16, p.other[Y] + at, true);
      if (c == 0) sh.ylist[pos] = (uint8_t)r;
    }
    for (int idx = 8 * ny + tid; idx < 8 * steps * G; idx += kTriThreads) {
      *reinterpret_cast<uint4*>(smem + kOffY + idx * 16) = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(smem + kOffY2 + idx * 16) = make_uint4(0, 0, 0, 0);
    }
    cp_async_commit();
    if (tid < kMaxKeys) {
      const bool ok = tid < info.n_queries && valid(0, tid);
      if constexpr (!kForward) {
        cols[tid] = ok ? p.lse2[(size_t)bh * N + tid] : -INFINITY;
        cols[kMaxKeys + tid] = ok ? p.ndelta[(size_t)bh * N + tid] : 0.f;
      }
      cols[2 * kMaxKeys + tid] = ok ? p.gate[(size_t)bh * N + tid] : 0.f;
    }
    // pairs of keys: rows j with bits k (rows k with bits j where the columns are the first keys)
    if (p.pair_valid) {
      uint32_t* bits = reinterpret_cast<uint32_t*>(smem + kOffBits);
      for (int item = warp; item < info.n_keys * kWords; item += kTriThreads / 32) {
        const int a = item / kWords, wd = item - a * kWords, t = 32 * wd + lane;
        uint32_t word = valid(1, a) ? sh.mask[1][wd] : 0u;
        if (word) {
          const int tc = min(t, N - 1), j = Z == 1 ? tc : a, k = Z == 1 ? a : tc;
          word &= __ballot_sync(0xffffffffu, t < N && p.pair_valid[((size_t)b * N + j) * N + k] > 0);
        }
        if (lane == 0) bits[item] = word;
      }
    }
  }
  bool holes = false;  // hidden columns before the last valid one
  for (int wd = 0; wd < kWords; ++wd) {
    const int left = nz - 32 * wd;
    const uint32_t all = left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u;
    holes = holes || (sh.mask[Z != 0][wd] & all) != all;
  }
  const int x0 = tile * rt;
  const int pitch = rt | 1;  // float4s
  float* bpair = reinterpret_cast<float*>(smem + kOffTile);               // [stage][row]
  float4* btile = reinterpret_cast<float4*>(bpair + kStages * kTileM);    // [column / 4][row]
  float* bcol = reinterpret_cast<float*>(btile) + pitch * zpad;           // [stage][group][column]
  // operand of (x, z): v_ik, u_ij, w_jk by pass; zeros where either does not count
  float* dst = reinterpret_cast<float*>(btile);
  if (X == 0 && !holes && (N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.v_bias) & 15) == 0) {  // four columns at a time
    for (int row = warp; row < rt; row += kTriThreads / 32) {
      const int x = x0 + row;
      const bool in = x < nx && valid(X, x);
      for (int z4 = lane; z4 < zpad / 4; z4 += 32) {
        const int bytes = in ? 4 * min(max(nz - 4 * z4, 0), 4) : 0;
        cp_async16_part(smem_u32(btile + z4 * pitch + row), bytes ? p.v_bias + nn + (size_t)x * N + 4 * z4 : p.v_bias, bytes);
      }
    }
  } else if constexpr (X == 0) {
    for (int row = warp; row < rt; row += kTriThreads / 32)
      for (int z = lane; z < zpad; z += 32) {
        const int x = x0 + row;
        const bool ok = x < nx && z < nz && valid(X, x) && valid(Z, z);
        cp_async_f32(dst + ((z >> 2) * pitch + row) * 4 + (z & 3), ok ? p.v_bias + nn + (size_t)x * N + z : p.v_bias, ok);
      }
  } else {
    const float* src = X == 1 ? p.u : p.w;
    for (int z = warp; z < zpad; z += kTriThreads / 32)
      for (int row = lane; row < rt; row += 32) {
        const int x = x0 + row;
        const bool ok = x < nx && z < nz && valid(X, x) && valid(Z, z);
        cp_async_f32(dst + ((z >> 2) * pitch + row) * 4 + (z & 3), ok ? src + nn + (size_t)z * N + x : src, ok);
      }
  }
  cp_async_commit();
  cp_async_wait<0>();
  fence_smem_to_async_proxy();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem;
  bool bad = false;
  auto wait_on = [&](uint64_t* bar, uint32_t phase) {
    if (!bad) bad = !mbar_wait_for(bar, phase & 1u, p.waits.limit);
  };
  auto chunk_units = [&](int c) { return per + (c < extra); };
  auto chunk_start = [&](int c) { return c * per + min(c, extra); };  // in units

  // Forward: mode 0 with shift 0; if a row's sum is out of range, mode 1 finds the maxima and mode 2 does the tile again.
  constexpr int kModes = kForward ? 3 : 1;
  auto next_mode = [&](bool again) {
    if (bad) sh.gave_up = 1;
    return __syncthreads_or(again) != 0;
  };

  if (warp >= kIssuerWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<kForward>::kAux));
    for (int mode = 0; mode < kModes; ++mode) {
      const int s_first = mode * steps;
      if (warp == kIssuerWarp) {
        if (elect_one()) {
          // ------------------------------------------------------------------ issuer
          const uint32_t lz = make_desc_lo(smem_u32(smem + kOffZ), 0), lz2 = make_desc_lo(smem_u32(smem + kOffZ2), 0);
          constexpr uint32_t mn = (kMaxKeys * 128 >> 4) << 16;  // LBO of the MN-major view
          constexpr uint32_t idesc_t = make_idesc_bf16(kTileM, kD, false, true);
          const uint32_t idesc_s = make_idesc_bf16(kTileM, 16 * per, false, false);
          constexpr uint32_t idesc_more = 16u >> 3 << 17;  // 16 columns more
          const int total = steps * C;
          // Two streams of chunks, the logits ahead of the sums: step, chunk of the step, its first unit, buffer
          struct Stream {
            int S, c, u, buf;
          };
          Stream lg{s_first, 0, 0, (int)(mode * total % kBufs)}, sm = lg;
          uint32_t ph_p = (mode * total / kBufs) & 1;  // phase of bar_p for the buffer sm.buf (flips when the ring wraps)
          auto advance = [&](Stream& t, int nu) {
            t.u += nu;
            if (++t.buf == kBufs) t.buf = 0;
            if (++t.c == C) t.c = 0, t.u = 0, ++t.S;
          };
          auto next_logits = [&]() {
            if (lg.c == 0) {
              wait_on(&sh.bar_a[lg.S & 1], lg.S >> 1);
              tc_fence_after_sync();
            }
            const int more = lg.c < extra;
            const uint32_t idesc = idesc_s + (more ? idesc_more : 0u);
            const uint32_t a = tmem + (lg.S & 1) * kACols, d = tmem + kColS + lg.buf * kBufCols, z = lg.u * 128;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ts_lo(d, a + 8 * ks, lz + z + 2 * ks, idesc, ks > 0);
            if constexpr (!kForward) {
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) umma_ts_lo(d + 64, a + 32 + 8 * ks, lz2 + z + 2 * ks, idesc, ks > 0);
            }
            umma_commit(&sh.bar_s[lg.buf]);
            if (lg.c == C - 1) umma_commit(&sh.bar_free[lg.S & 1]);
            advance(lg, per + more);
          };
          // A of step s is built once the row warps have read T of step s - 3: with one chunk a step, three chunks ahead is the limit
          const int ahead = C == 1 ? min(kBufs, 3) : kBufs;
          for (int q = 0; q < min(ahead, total); ++q) next_logits();
#pragma unroll 1
          for (int q = 0; q < total; ++q) {
            wait_on(&sh.bar_p[sm.buf], ph_p);
            if (sm.c == 0 && sm.S >= kSumBufs) wait_on(&sh.bar_d[(sm.S - kSumBufs) & 1], (sm.S - kSumBufs) >> 1);  // the buffer's last sums have been read
            tc_fence_after_sync();
            const int nu = per + (sm.c < extra);
            const uint32_t a = tmem + kColS + sm.buf * kBufCols, z = sm.u * 128, t = tmem + kColT + (kSumBufs == 2 ? 64 * (sm.S & 1) : 0);
            const bool more = sm.c > 0;
#pragma unroll
            for (int kg = 0; kg < 4; ++kg)
              if (kg < nu) umma_ts_lo(t, a + (kForward ? 0 : 64) + 8 * kg, ((kForward ? lz2 : lz) | mn) + z + 128 * kg, idesc_t, more || kg > 0);
            if constexpr (kPass == kDk1 || kPass == kDk2) {
#pragma unroll
              for (int kg = 0; kg < 4; ++kg)
                if (kg < nu) umma_ts_lo(tmem + kColR, a + 8 * kg, (lz2 | mn) + z + 128 * kg, idesc_t, more || kg > 0);
            }
            if (sm.c == C - 1) umma_commit(&sh.bar_t[sm.S & 1]);
            if (sm.buf == kBufs - 1) ph_p ^= 1;
            advance(sm, nu);
            if (q + ahead < total) next_logits();
          }
          // Whoever gave up, no product may be in flight when tensor memory is given back
          umma_commit(&sh.bar_drain);
          if (!mbar_wait_for(&sh.bar_drain, mode & 1, p.waits.limit)) bad = true;
        }
        __syncwarp();
      } else if (warp == kBiasLoader) {
        // ------------------------------------------------------------------ bias operand of (y, z): w_jk, v_ik, u_ij by pass
        const float* src = X == 0 ? p.w : X == 1 ? p.v_bias : p.u;
        const bool vec = X != 1 && !holes && (N & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;  // four columns at a time
        src += nn;
        uint32_t in = 0;  // bit t: column lane + 32 t counts
#pragma unroll
        for (int t = 0; t < kWords; ++t) {
          const int z = lane + 32 * t;
          if (z < nz && valid(Z, z)) in |= 1u << t;
        }
        for (int s = 0; s < steps; ++s) {
          const int S = s_first + s, st = S & (kStages - 1);
          if (S >= kStages) wait_on(&sh.bar_empty[st], S / kStages - 1);
          for (int gg = 0; gg < G; ++gg) {
            const int yy = s * G + gg, y = yy < ny ? sh.ylist[yy] : 0;
            float* dst = bcol + (st * G + gg) * zpad;
            if (vec) {
              for (int z = 4 * lane; z < zpad; z += 128)
                cp_async16_part(smem_u32(dst + z), src + (size_t)y * N + min(z, (nz - 1) & ~3), yy < ny ? 4 * min(max(nz - z, 0), 4) : 0);
            } else {
              const float* at = src + (X == 1 ? (size_t)lane * N + y : (size_t)y * N + lane);
              const size_t step = X == 1 ? (size_t)32 * N : 32;
#pragma unroll
              for (int t = 0; t < kWords; ++t, at += step)
                if (lane + 32 * t < zpad) {
                  const bool ok = yy < ny && ((in >> t) & 1u);
                  cp_async_f32(dst + lane + 32 * t, ok ? at : src, ok);
                }
            }
          }
          cp_async_arrive(&sh.bar_full[st]);
        }
      } else if (warp == kPairLoader) {
        // ------------------------------------------------------------------ bias operand of (x, y): u_ij, w_jk, v_ik by pass
        const float* src = X == 0 ? p.u : X == 1 ? p.w : p.v_bias;
        int rg[4], rx[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int row = lane + 32 * t;
          rg[t] = row / rt, rx[t] = x0 + row - rg[t] * rt;
          if (rg[t] >= G || rx[t] >= nx || !valid(X, rx[t])) rg[t] = 1 << 20;  // no pair
        }
        for (int s = 0; s < steps; ++s) {
          const int S = s_first + s, st = S & (kStages - 1);
          if (S >= kStages) wait_on(&sh.bar_empty[st], S / kStages - 1);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const int yy = s * G + rg[t];
            const bool ok = yy < ny;
            const int y = ok ? sh.ylist[yy] : 0;
            cp_async_f32(bpair + st * kTileM + lane + 32 * t, ok ? src + nn + (X == 2 ? (size_t)y * N + rx[t] : (size_t)rx[t] * N + y) : src, ok);
          }
          cp_async_arrive(&sh.bar_full[st]);
        }
      }
      cp_async_wait<0>();  // (nothing is left, unless a consumer gave up)
      if (kForward && !next_mode(false)) break;
    }
  } else {
    const int r = tid & 127, grp = (tid >> 7) & 1;  // tile row, group
    const int g = r / rt, ii = r - g * rt, x = x0 + ii, gs = g < G ? g : 0;
    const bool row_ok = g < G && x < nx && valid(X, min(x, kMaxKeys - 1));
    const bool warp_live = __any_sync(0xffffffffu, row_ok);
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    float* sums = reinterpret_cast<float*>(smem + kOffSums);
    float* row_l = sums + 2 * kTileM;  // forward: a row's sum and shift for the row warps
    float* row_shift = row_l + kTileM;
    auto warp_arrive = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    if (warp < kExpWarps) {
      // ------------------------------------------------------------------ softmax
      if constexpr (kForward) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Regs<kForward>::kExp));
      else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<kForward>::kExp));
      float shift = 0.f, m_run = -INFINITY;
      float2 dgate = make_float2(0.f, 0.f);
      const uint32_t* bits = reinterpret_cast<const uint32_t*>(smem + kOffBits);
      const bool masks = holes || p.pair_valid;  // else only columns beyond the last one are hidden
      float row_lse = 0.f, row_delta = 0.f, row_gate = 0.f;
      if constexpr (X == 0) {
        if (row_ok) {
          if constexpr (!kForward) row_lse = cols[x], row_delta = cols[kMaxKeys + x];
          row_gate = cols[2 * kMaxKeys + x];
        }
      }
      for (int mode = 0; mode < kModes; ++mode) {
        const int s_first = mode * steps;
        float l_run = 0.f;
        float lse = 0.f, delta = 0.f, gate = 0.f, rs = 0.f;
        float2 rsum = make_float2(0.f, 0.f);
        bool ok = false, seen = false;
        const uint32_t* vis = sh.mask[1];
        const float* colp = bcol;
        // One unit of 16 columns: P and dS from S and dP
        auto unit = [&](uint32_t buf, int z, uint32_t (&sv)[16], const uint32_t (&dv)[16]) {
          float2 t[8];
#pragma unroll
          for (int e4 = 0; e4 < 4; ++e4) {
            const float4 xz = btile[((z >> 2) + e4) * pitch + ii], yz = *reinterpret_cast<const float4*>(colp + z + 4 * e4);
            float4 gz = make_float4(gate, gate, gate, gate);
            if constexpr (Z == 0) gz = *reinterpret_cast<const float4*>(cols + 2 * kMaxKeys + z + 4 * e4);
            const float2 xy = make_float2(rs, rs);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const float2 a = half ? make_float2(xz.z, xz.w) : make_float2(xz.x, xz.y);
              const float2 c = half ? make_float2(yz.z, yz.w) : make_float2(yz.x, yz.y);
              // (u_ij + v_ik) + w_jk
              float2& v = t[2 * e4 + half];
              if constexpr (X == 0) v = add2(add2(xy, a), c);
              else if constexpr (X == 1) v = add2(add2(a, c), xy);
              else v = add2(add2(c, xy), a);
              const int e = 4 * e4 + 2 * half;
              const float2 y = fma2(half ? make_float2(gz.z, gz.w) : make_float2(gz.x, gz.y), v,
                                    make_float2(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])));
              sv[e] = __float_as_uint(y.x), sv[e + 1] = __float_as_uint(y.y);
            }
          }
          uint32_t mask = 0xffffu;
          if constexpr (Z == 0) {
            mask = seen ? 0xffffu : 0u;
          } else {
            if (masks) mask = (vis[z >> 5] >> (z & 16)) & 0xffffu;
            else if (z + 16 > nz) mask = (1u << (nz - z)) - 1u;
          }
          if (!__all_sync(0xffffffffu, mask == 0xffffu)) {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (!((mask >> e) & 1u)) sv[e] = 0xff800000u;  // -infinity
          }
          if constexpr (kForward) {
            if (mode == 1) {
              if (ok) {
#pragma unroll
                for (int e = 0; e < 16; ++e) m_run = fmaxf(m_run, __uint_as_float(sv[e]));
              }
              return;
            }
          }
          uint32_t pk[8], dk[8];
#pragma unroll
          for (int e4 = 0; e4 < 4; ++e4) {
            float4 cl = make_float4(lse, lse, lse, lse), cd = make_float4(delta, delta, delta, delta), cg = cd;
            if constexpr (Z == 0) {
              cl = *reinterpret_cast<const float4*>(cols + z + 4 * e4);
              cd = *reinterpret_cast<const float4*>(cols + kMaxKeys + z + 4 * e4);
              cg = *reinterpret_cast<const float4*>(cols + 2 * kMaxKeys + z + 4 * e4);
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int e = 4 * e4 + 2 * half;
              float2 pr = fma2(make_float2(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), make_float2(kLog2e, kLog2e),
                               half ? make_float2(cl.z, cl.w) : make_float2(cl.x, cl.y));
              pr.x = fast_exp2(pr.x), pr.y = fast_exp2(pr.y);
              if constexpr (kForward) {
                rsum = add2(rsum, pr);
              } else {
                const float2 ds = mul2(pr, add2(make_float2(__uint_as_float(dv[e]), __uint_as_float(dv[e + 1])),
                                                half ? make_float2(cd.z, cd.w) : make_float2(cd.x, cd.y)));
                dk[e >> 1] = pack2_bf16(ds.x, ds.y);
                if constexpr (Z == 0) rsum = fma2(half ? make_float2(cg.z, cg.w) : make_float2(cg.x, cg.y), ds, rsum);
                else rsum = add2(rsum, ds);
                if constexpr (X == 0) dgate = fma2(ds, t[e >> 1], dgate);
              }
              if constexpr (kPass != kDq) pk[e >> 1] = pack2_bf16(pr.x, pr.y);
            }
          }
          if constexpr (kPass != kDq) tmem_st8(buf, pk);
          if constexpr (!kForward) tmem_st8(buf + 64, dk);
        };
#pragma unroll 1
        for (int s = 0; s < steps; ++s) {
          const int S = s_first + s, st = S & (kStages - 1);
          const int yy = s * G + gs;
          ok = row_ok && yy < ny;
          if constexpr (kForward) lse = -shift;
          else lse = row_lse;
          delta = row_delta, gate = row_gate;
          seen = ok;
          if (Y == 0 || p.pair_valid) {
            const int y = yy < ny ? (int)sh.ylist[yy] : 0;
            if constexpr (Y == 0) lse = cols[y], delta = cols[kMaxKeys + y], gate = cols[2 * kMaxKeys + y];
            if (p.pair_valid) {
              vis = bits + (Y == 1 ? y : X == 2 ? min(x, kMaxKeys - 1) : 0) * kWords;  // bits over the columns
              // columns = queries: whether the row's pair of keys counts
              if constexpr (Z == 0) seen = ok && ((bits[x * kWords + (y >> 5)] >> (y & 31)) & 1u);
            }
          }
          if (!ok) lse = -INFINITY;
          colp = bcol + (st * G + gs) * zpad;
          wait_on(&sh.bar_full[st], S / kStages);
          rs = bpair[st * kTileM + r];
          // an infinite w_jk hides the pair from every query whose lse is not NaN; in the columns of padded queries (gate 0) it would be NaN
          if constexpr (Z == 0) seen = seen && fabsf(rs) < INFINITY;
          rsum = make_float2(0.f, 0.f);
#pragma unroll 1
          for (int c = (S * C ^ grp) & 1; c < C; c += 2) {
            const int Q = S * C + c;
            wait_on(&sh.bar_s[Q % kBufs], Q / kBufs);
            if (warp_live) {
              tc_fence_after_sync();
              uint32_t buf = trow + kColS + (Q % kBufs) * kBufCols, dst = buf;
              int z = 16 * chunk_start(c);
              const int z1 = z + 16 * chunk_units(c);
#pragma unroll 1
              for (; z < z1; z += 16, buf += 16, dst += 8) {  // (one copy of the code: the loop has to stay in the instruction caches)
                uint32_t sv[16], dv[16];
                tmem_ld16(buf, sv);
                if constexpr (!kForward) tmem_ld16(buf + 64, dv);
                tmem_ld_wait();
                unit(dst, z, sv, dv);
              }
              if constexpr (!kForward)
                if (c + 2 >= C) sums[((S & 3) * 2 + grp) * kTileM + r] = rsum.x + rsum.y;  // the group's last chunk of the step
              tmem_st_wait();
            }
            tc_fence_before_sync();
            warp_arrive(&sh.bar_p[Q % kBufs]);
          }
          if constexpr (kForward) l_run += rsum.x + rsum.y;
          warp_arrive(&sh.bar_empty[st]);
        }
        if constexpr (kForward) {
          // the rows' sums (mode 1: maxima) over the two groups and the groups of first keys
          bool again = false;
          sums[grp * kTileM + r] = mode == 1 ? m_run : l_run;
          group_barrier<1>();
          if (g < G) {
            float t = mode == 1 ? -INFINITY : 0.f;
            for (int gg = 0; gg < G; ++gg) {
              const float a = sums[gg * rt + ii], c = sums[kTileM + gg * rt + ii];
              t = mode == 1 ? fmaxf(t, fmaxf(a, c)) : t + (a + c);
            }
            if (mode == 1) {
              shift = t > -INFINITY ? t * kLog2e : 0.f;
              again = true;
            } else {
              if (mode == 0) again = row_ok && !bad && !(t >= kSumLow && t <= kSumHigh);
              if (grp == 0) row_l[r] = t, row_shift[r] = shift;
            }
          }
          if (!next_mode(again)) break;
        }
      }
      if constexpr (kPass == kDq) {
        // (the row warps read the last steps' sums; these lie beyond them)
        float* xs = reinterpret_cast<float*>(smem + kOffDgate);
        xs[grp * kTileM + r] = dgate.x + dgate.y;
        group_barrier<1>();
        if (grp == 0 && g == 0 && x < nx && p.dgate) {
          float t = 0.f;
          for (int gg = 0; gg < G; ++gg) t += xs[gg * rt + r] + xs[kTileM + gg * rt + r];
          p.dgate[(size_t)bh * N + x] = row_ok ? t : 0.f;
        }
      }
    } else {
      // ------------------------------------------------------------------ rows: operands and accumulators
      if constexpr (!kForward) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Regs<kForward>::kRow));
      // this thread's part of X_x (half of it forward, else X for group 0 and X' for group 1) as bf16x2
      constexpr int kXw = kForward ? 16 : 32;
      uint32_t xr[kXw];
      {
        const __nv_bfloat16* src = (kForward || grp == 0 ? p.main[X] : p.other[X]) + base + (size_t)(row_ok ? x : 0) * kD + (kForward ? 32 * grp : 0);
#pragma unroll
        for (int c = 0; c < kXw / 4; ++c) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (row_ok) v = __ldg(reinterpret_cast<const uint4*>(src) + c);
          xr[4 * c] = v.x, xr[4 * c + 1] = v.y, xr[4 * c + 2] = v.z, xr[4 * c + 3] = v.w;
        }
      }
      float acc[kAcc];
      for (int mode = 0; mode < kModes; ++mode) {
        const int s_first = mode * steps;
#pragma unroll
        for (int d = 0; d < kAcc; ++d) acc[d] = 0.f;
        // step s: A of step s + 2, T and R of step s
#pragma unroll 1
        for (int s = -2; s < steps; ++s) {
          if (s + 2 < steps) {
            const int S = s_first + s + 2;
            if (S >= 2) wait_on(&sh.bar_free[S & 1], (S >> 1) - 1);
            if (warp_live) {
              tc_fence_after_sync();
              const uint4* y = reinterpret_cast<const uint4*>(smem + (kForward || grp == 0 ? kOffY : kOffY2) + ((s + 2) * G + gs) * 128 + (kForward ? 64 * grp : 0));
#pragma unroll
              for (int half = 0; half < kXw / 16; ++half) {
                uint32_t a[16];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                  const uint4 v = y[4 * half + c];
                  a[4 * c] = mul_bf16x2(xr[16 * half + 4 * c], v.x);
                  a[4 * c + 1] = mul_bf16x2(xr[16 * half + 4 * c + 1], v.y);
                  a[4 * c + 2] = mul_bf16x2(xr[16 * half + 4 * c + 2], v.z);
                  a[4 * c + 3] = mul_bf16x2(xr[16 * half + 4 * c + 3], v.w);
                }
                tmem_st16(trow + (S & 1) * kACols + (kForward ? 16 : 32) * grp + 16 * half, a);
              }
              tmem_st_wait();
            }
            tc_fence_before_sync();
            warp_arrive(&sh.bar_a[S & 1]);
          }
          if (s < 0) continue;
          const int S = s_first + s;
          wait_on(&sh.bar_t[S & 1], S >> 1);
          tc_fence_after_sync();
          const bool ok = row_ok && s * G + gs < ny;
          // gradient of the bias operand of (x, y): the sums of the softmax groups that had a chunk of the step
          float pair_sum = 0.f;
          if constexpr (!kForward) {
            const float* sum = sums + (S & 3) * 2 * kTileM + r;
            if (grp == 0) pair_sum = C == 1 ? sum[(S & 1) * kTileM] : sum[0] + sum[kTileM];
          }
          auto read_done = [&]() {
            tc_fence_before_sync();
            warp_arrive(&sh.bar_d[S & 1]);
          };
          if (warp_live && mode != 1) {
            const uint4* y = reinterpret_cast<const uint4*>(smem + (kForward || (!kHalf && grp) ? kOffY2 : kOffY) + (s * G + gs) * 128 + (kHalf ? 64 * grp : 0));
            const uint32_t src = trow + (kHalf ? kColT + 64 * (S & 1) + 32 * grp : grp ? kColR : kColT);
#pragma unroll
            for (int q = 0; q < kAcc / 32; ++q) {
              uint32_t t[32];
              tmem_ld32(src + 32 * q, t);
              tmem_ld_wait();
              if (q == kAcc / 32 - 1) read_done();
              if (ok) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                  const uint4 v = y[4 * q + c];
                  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    float* a = acc + 32 * q + 8 * c + 2 * e;
                    const uint32_t* te = t + 8 * c + 2 * e;
                    const float2 o = fma2(make_float2(bf16_lo(w[e]), bf16_hi(w[e])), make_float2(__uint_as_float(te[0]), __uint_as_float(te[1])), make_float2(a[0], a[1]));
                    a[0] = o.x, a[1] = o.y;
                  }
                }
              }
            }
          } else {
            read_done();
          }
          if constexpr (!kForward) {
            float* dst = X == 0 ? p.du : X == 1 ? p.dw : p.dv_bias;
            if (grp == 0 && ok && dst) {
              const int y = sh.ylist[s * G + gs];
              if constexpr (X == 0) dst[nn + (size_t)x * N + y] = cols[2 * kMaxKeys + x] * pair_sum;
              else if constexpr (X == 1) dst[nn + (size_t)x * N + y] = pair_sum;
              else dst[nn + (size_t)y * N + x] = cols[2 * kMaxKeys + y] * pair_sum;
            }
          }
        }
        if (kForward && !next_mode(false)) break;
      }
      // ---- rows of one x are added up over the groups in a fixed order and leave
      if (G > 1) {
        group_barrier<2>();  // every product has completed and every staged row has been read
        float* stage = reinterpret_cast<float*>(smem) + grp * kTileM * kAcc;
        constexpr int kQ = kAcc / 4;
#pragma unroll
        for (int c = 0; c < kQ; ++c)
          reinterpret_cast<float4*>(stage + r * kAcc)[c ^ (r & 7)] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
        group_barrier<2>();
        if (g == 0) {
          for (int gg = 1; gg < G; ++gg) {
            const int r2 = gg * rt + r;
#pragma unroll
            for (int c = 0; c < kQ; ++c) {
              const float4 v = reinterpret_cast<const float4*>(stage + r2 * kAcc)[c ^ (r2 & 7)];
              acc[4 * c] += v.x, acc[4 * c + 1] += v.y, acc[4 * c + 2] += v.z, acc[4 * c + 3] += v.w;
            }
          }
        }
      }
      if (g == 0 && x < nx) {
        const float l = kForward ? row_l[r] : 1.f;
        if constexpr (kForward) bad = bad || sh.gave_up;  // (written before the barrier of next_mode)
        const bool have = row_ok && !bad && l != 0.f;
        const float scale = have ? 1.f / l : 0.f;
        if (kForward || !have) {
#pragma unroll
          for (int d = 0; d < kAcc; ++d) acc[d] = have ? acc[d] * scale : 0.f;
        }
        const size_t at = base + (size_t)x * kD + (kHalf ? 32 * grp : 0);
        if constexpr (kForward) {
          float4* o = reinterpret_cast<float4*>(p.out + at);
#pragma unroll
          for (int c = 0; c < kAcc / 4; ++c) o[c] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
          if (grp == 0) p.lse[(size_t)bh * N + x] = have ? (row_shift[r] + log2f(l)) * kLn2 : 0.f;
        }
        __nv_bfloat16* dst = kForward ? p.out_cast : kHalf || grp == 0 ? p.grad_main[X] : p.grad_other[X];
        if (dst) {
          uint4* o = reinterpret_cast<uint4*>(dst + at);
#pragma unroll
          for (int c = 0; c < kAcc / 8; ++c)
            o[c] = make_uint4(pack2_bf16(acc[8 * c], acc[8 * c + 1]), pack2_bf16(acc[8 * c + 2], acc[8 * c + 3]),
                              pack2_bf16(acc[8 * c + 4], acc[8 * c + 5]), pack2_bf16(acc[8 * c + 6], acc[8 * c + 7]));
        }
      }
    }
  }

  tc_fence_before_sync();
  bad = __syncthreads_or(bad) != 0;
  if (bad && tid == 0) atomicExch(p.status, MF_ERR_DEVICE_TIMEOUT);  // (backward: the gradients are cleared by the last launch)
  if (warp == kIssuerWarp) tmem_dealloc(tmem, kTmemCols);
}

__global__ void __maxnreg__(kRegLaunch) simplicial_tri_fwd_kernel(const __grid_constant__ TriParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (an address made from an integer would be a generic one)
  __shared__ TriShared sh;
  wait_for_previous();
  const int at = blockIdx.x / p.H;
  if (at >= p.items[0].x) return;
  tri_tile<kFwd>(p, sh, smem, p.items[1 + at], blockIdx.x % p.H);
}

__global__ void __maxnreg__(kRegLaunch) simplicial_tri_bwd_kernel(const __grid_constant__ TriParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (an address made from an integer would be a generic one)
  __shared__ TriShared sh;
  wait_for_previous();
  const int at = blockIdx.x / p.H, h = blockIdx.x % p.H;
  if (at >= p.items[0].x) return;
  const int2 item = p.items[1 + at];
  const int pass = (item.x >> 16) & 15;
  if (pass == kDq) tri_tile<kDq>(p, sh, smem, item, h);
  else if (pass == kDk1) tri_tile<kDk1>(p, sh, smem, item, h);
  else tri_tile<kDk2>(p, sh, smem, item, h);
}

// Extents of the molecules and the list of tiles, heavy molecules first (by buckets of their mean extent; the order decides when
// a tile runs, not what it computes).  One block: the list is short next to the work it describes.
constexpr int kScheduleThreads = 1024;
__global__ void __launch_bounds__(kScheduleThreads) simplicial_tri_schedule_kernel(const uint8_t* __restrict__ query_valid,
                                                                                  const uint8_t* __restrict__ key_valid, int B, int N,
                                                                                  int backward, BatchInfo* info, int2* items,
                                                                                  int32_t* status) {
  wait_for_previous();
  __shared__ int start[kMaxKeys + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 64) status[tid] = 0;
  for (int t = tid; t <= kMaxKeys; t += kScheduleThreads) start[t] = 0;
  __syncthreads();
  auto plan = [&](const BatchInfo& m, int pass) {
    const bool any = m.reserved0 > 0 && m.reserved1 > 0;
    return tri_plan(pass == kDq || pass == kFwd ? m.n_queries : m.n_keys, any ? pass == kDk2 ? m.reserved1 : m.reserved0 : 0);
  };
  const int first = backward ? kDq : kFwd, last = backward ? kDk2 : kFwd;
  auto bucket = [&](const BatchInfo& m) { return kMaxKeys - (m.n_keys + m.n_queries) / 2; };
  for (int b = warp; b < B; b += kScheduleThreads / 32) {
    int nk = 0, nq = 0, ck = 0, cq = 0;
    for (int t = lane; t < N; t += 32) {
      if (key_valid[(size_t)b * N + t]) nk = t + 1, ++ck;
      if (query_valid[(size_t)b * N + t]) nq = t + 1, ++cq;
    }
    nk = __reduce_max_sync(0xffffffffu, nk), nq = __reduce_max_sync(0xffffffffu, nq);
    ck = __reduce_add_sync(0xffffffffu, ck), cq = __reduce_add_sync(0xffffffffu, cq);
    const BatchInfo m{nk, nq, ck, cq};
    const int tiles = __reduce_add_sync(0xffffffffu, first + lane <= last ? max(plan(m, first + lane).tiles, 1) : 0);
    if (lane == 0) {
      info[b] = m;
      atomicAdd(&start[bucket(m)], tiles);
    }
  }
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
    if (lane == 0) items[0] = make_int2(before, 0);
  }
  __syncthreads();  // (and each warp reads the extents that it wrote)
  for (int b = warp; b < B; b += kScheduleThreads / 32) {  // a lane per pass; at least one tile each: it clears the rows that nothing covers
    const BatchInfo m = info[b];
    const bool mine = first + lane <= last;
    const TriPlan pl = mine ? plan(m, first + lane) : TriPlan{0, 0};
    const int tiles = mine ? max(pl.tiles, 1) : 0, t0 = __shfl_sync(0xffffffffu, tiles, 0), t1 = __shfl_sync(0xffffffffu, tiles, 1);
    const int all = __reduce_add_sync(0xffffffffu, tiles);
    int at = lane == 0 ? 1 + atomicAdd(&start[bucket(m)], all) : 0;
    at = __shfl_sync(0xffffffffu, at, 0) + (lane > 0 ? t0 : 0) + (lane > 1 ? t1 : 0);
    for (int t = 0; t < tiles; ++t) items[at + t] = make_int2(b | (first + lane) << 16 | t << 20, pl.rows | pl.tiles << 8);
  }
}

// -lse log2e and -delta = -dO . out of the valid queries
__global__ void __launch_bounds__(256) simplicial_tri_rows_kernel(const __nv_bfloat16* __restrict__ grad_out, const float* __restrict__ out,
                                                                 const float* __restrict__ lse, const uint8_t* __restrict__ query_valid,
                                                                 int H, int N, int rows, float* __restrict__ lse2,
                                                                 float* __restrict__ ndelta) {
  wait_for_previous();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  if (query_valid[(size_t)(row / (H * N)) * N + row % N] == 0) return;
  const uint32_t g = reinterpret_cast<const uint32_t*>(grad_out + (size_t)row * kD)[lane];
  const float2 o = reinterpret_cast<const float2*>(out + (size_t)row * kD)[lane];
  const float s = warp_sum(fmaf(bf16_lo(g), o.x, bf16_hi(g) * o.y));
  if (lane == 0) lse2[row] = -lse[row] * kLog2e, ndelta[row] = -s;
}

// When a wait expired anywhere every gradient is written as zeros: a row's sums leave while other roles may still give up, and what
// the other CTAs have written belongs to the same call.  Else it returns at once.
struct TriClear {
  uint32_t* at[9];
  size_t words[9];
};
__global__ void __launch_bounds__(256) simplicial_tri_clear_kernel(const __grid_constant__ TriClear c, const int32_t* __restrict__ status) {
  wait_for_previous();
  if (*status == 0) return;
#pragma unroll 1
  for (int t = 0; t < 9; ++t)
    if (c.at[t])
      for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < c.words[t]; i += (size_t)gridDim.x * 256) c.at[t][i] = 0u;
}

struct TriLayout {
  size_t info, items, lse2, ndelta, total;
  int max_items;
};
TriLayout tri_layout(int batch, int heads, int tokens, bool backward) {
  TriLayout l{};
  size_t off = kStatusBytes;
  l.info = off, off = align_up(off + (size_t)batch * sizeof(BatchInfo), 256);
  l.max_items = batch * kMostTiles * (backward ? 3 : 1);
  l.items = off, off = align_up(off + (1 + (size_t)l.max_items) * sizeof(int2), 256);
  if (backward) {
    const size_t rows = align_up((size_t)batch * heads * tokens * sizeof(float), 256);
    l.lse2 = off, off += rows;
    l.ndelta = off, off += rows;
  }
  l.total = off;
  return l;
}

template <typename Args>
void fill_params(TriParams& p, const Args& a, const TriLayout& l) {
  const void* m[3] = {a.q, a.k1, a.k2};
  for (int t = 0; t < 3; ++t) p.main[t] = static_cast<const __nv_bfloat16*>(m[t]);
  p.other[1] = static_cast<const __nv_bfloat16*>(a.v1), p.other[2] = static_cast<const __nv_bfloat16*>(a.v2);
  p.query_valid = a.query_valid, p.key_valid = a.pair_key_valid, p.pair_valid = a.pair_valid;
  p.u = a.u, p.v_bias = a.v_bias, p.w = a.w, p.gate = a.gate;
  char* ws = static_cast<char*>(a.workspace);
  p.status = reinterpret_cast<int32_t*>(ws);
  p.info = reinterpret_cast<BatchInfo*>(ws + l.info);
  p.items = reinterpret_cast<int2*>(ws + l.items);
  p.H = a.heads, p.N = a.tokens;
}

template <typename Kernel>
int launch_tri(Kernel kernel, const TriParams& p, const TriLayout& l, int batch, bool backward, int which, cudaStream_t stream, const char* name) {
  launch_dependent(simplicial_tri_schedule_kernel, dim3(1), dim3(kScheduleThreads), 0, stream, p.query_valid, p.key_valid, batch, p.N,
                   backward, const_cast<BatchInfo*>(p.info), const_cast<int2*>(p.items), p.status);
  MF_CHECK_LAUNCH("simplicial_tri_schedule_kernel");
  // (the limit is one for all sizes: another host thread must not lower it between here and the launch)
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tri_smem_bytes(kMaxKeys));
  if (e != cudaSuccess) return cuda_error(e, name);
  profile_mark(which, true, stream);
  launch_dependent(kernel, dim3((unsigned)l.max_items * p.H), dim3(kTriThreads), tri_smem_bytes(p.N), stream, p);
  profile_mark(which, false, stream);
  MF_CHECK_LAUNCH(name);
  return MF_OK;
}

}  // namespace

size_t simplicial_tri_fwd_workspace_bytes(const MfSimplicialFwdArgs& a) { return tri_layout(a.batch, a.heads, a.tokens, false).total; }
size_t simplicial_tri_bwd_workspace_bytes(const MfSimplicialBwdArgs& a) { return tri_layout(a.batch, a.heads, a.tokens, true).total; }

int simplicial_tri_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream, BoundedWaits waits) {
  const TriLayout l = tri_layout(a.batch, a.heads, a.tokens, false);
  TriParams p{};
  p.waits = waits;
  fill_params(p, a, l);
  p.other[0] = p.main[0];  // (not read)
  p.out = a.out, p.lse = a.lse, p.out_cast = static_cast<__nv_bfloat16*>(a.out_cast);
  return launch_tri(simplicial_tri_fwd_kernel, p, l, a.batch, false, MF_PROFILE_SIMPLICIAL_FWD, stream,
                    "simplicial_tri_fwd_kernel");
}

int simplicial_tri_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream, BoundedWaits waits) {
  const TriLayout l = tri_layout(a.batch, a.heads, a.tokens, true);
  TriParams p{};
  p.waits = waits;
  fill_params(p, a, l);
  char* ws = static_cast<char*>(a.workspace);
  float* lse2 = reinterpret_cast<float*>(ws + l.lse2);
  float* ndelta = reinterpret_cast<float*>(ws + l.ndelta);
  p.other[0] = static_cast<const __nv_bfloat16*>(a.grad_out);
  p.lse2 = lse2, p.ndelta = ndelta;
  void* gm[3] = {a.dq, a.dk1, a.dk2};
  for (int t = 0; t < 3; ++t) p.grad_main[t] = static_cast<__nv_bfloat16*>(gm[t]);
  p.grad_other[1] = static_cast<__nv_bfloat16*>(a.dv1), p.grad_other[2] = static_cast<__nv_bfloat16*>(a.dv2);
  p.du = a.du, p.dv_bias = a.dv_bias, p.dw = a.dw, p.dgate = a.dgate;
  const int rows = a.batch * a.heads * a.tokens;
  launch_dependent(simplicial_tri_rows_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, p.other[0], a.out, a.lse, a.query_valid, a.heads,
                   a.tokens, rows, lse2, ndelta);
  MF_CHECK_LAUNCH("simplicial_tri_rows_kernel");
  const int rc = launch_tri(simplicial_tri_bwd_kernel, p, l, a.batch, true, MF_PROFILE_SIMPLICIAL_BWD, stream, "simplicial_tri_bwd_kernel");
  if (rc != MF_OK) return rc;
  const size_t n = (size_t)rows;
  void* grads[9] = {a.dq, a.dk1, a.dv1, a.dk2, a.dv2, a.du, a.dv_bias, a.dw, a.dgate};
  TriClear c{};
  for (int t = 0; t < 9; ++t) c.at[t] = static_cast<uint32_t*>(grads[t]), c.words[t] = t < 5 ? n * (kD / 2) : t < 8 ? n * a.tokens : n;
  launch_dependent(simplicial_tri_clear_kernel, dim3(148), dim3(256), 0, stream, c, p.status);
  MF_CHECK_LAUNCH("simplicial_tri_clear_kernel");
  return MF_OK;
}

}  // namespace mf
