// Periodic k nearest neighbours with a cell list.
//
// Same result, bit for bit, as the all-pairs kernel (and the CPU oracle): the k smallest
// (minimum-image d2, index) pairs per atom.  Atoms are binned on a per-structure grid over their
// fractional coordinates and every query visits the bins within s cells of its own, s = 1, 2, ...
// A search of half-width s is complete as soon as k neighbours are known and the k-th distance is
// below s*h, where h = min over the axes of (perpendicular cell width / bins on that axis): any atom
// in an unvisited bin lies at least s bins away along some axis, so each of its 27 images is
// farther than s*h.  Candidates are inserted under the lexicographic order (d2, index), so the
// result does not depend on the order in which bins or atoms inside a bin are visited.
//
// A candidate normally costs one distance evaluation instead of 27: the image chosen by rounding the
// fractional delta is the minimum image whenever it is closer than half the smallest cell width, and
// its d2 is evaluated with the same operation sequence the 27-image search uses for that image; a
// candidate whose rounded image is farther than that needs the full search only while the list of
// the k best still holds an entry that far away.
//
// Structures with a coordinate outside [0,1) (where the reference's 27 offsets of the unwrapped
// coordinates are not the nearest images) are searched exhaustively.
#include "common.cuh"
#include "geometry.cuh"

namespace mf {
namespace {

constexpr int kMaxBinsPerAxis = 16;
constexpr int kMaxBins = kMaxBinsPerAxis * kMaxBinsPerAxis * kMaxBinsPerAxis;

struct KnnWorkspace {
  int32_t* counts;   // (B, kMaxBins + 1) bin sizes, then exclusive starts
  int32_t* cursor;   // (B, kMaxBins) fill cursors
  int32_t* keys;     // (B, N) bin of every atom
  int32_t* flags;    // (B) 1 when a coordinate lies outside [0,1)
  float4* sorted;    // (B, N) x, y, z, original index (as int bits), grouped by bin
  float* cell;       // (B, 3, 3) cells, (B, 3) bins per axis and (B, 2) bounds when the setup kernel worked them out
  int32_t* grid;
  float* bounds;
};

__global__ void knn_zero_kernel(int32_t* counts, int32_t* flags, int B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B * (kMaxBins + 1)) counts[i] = 0;
  if (i < B) flags[i] = 0;
}

__global__ void knn_count_kernel(const float* __restrict__ frac, const int32_t* __restrict__ num_atoms,
                                 const int32_t* __restrict__ grid_dims, int n_max, KnnWorkspace w) {
  const int b = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = min(num_atoms[b], n_max);
  if (i >= n) return;
  const float* p = frac + ((size_t)b * n_max + i) * 3;
  const int gx = grid_dims[3 * b], gy = grid_dims[3 * b + 1], gz = grid_dims[3 * b + 2];
  const float x = p[0], y = p[1], z = p[2];
  if (!(x >= 0.f && x < 1.f && y >= 0.f && y < 1.f && z >= 0.f && z < 1.f)) w.flags[b] = 1;
  const int key = (cell_coord(x, gx) * gy + cell_coord(y, gy)) * gz + cell_coord(z, gz);
  w.keys[(size_t)b * n_max + i] = key;
  atomicAdd(&w.counts[(size_t)b * (kMaxBins + 1) + key], 1);
}

// exclusive scan of the bin sizes of one structure (one block per structure, bins <= 4096)
__global__ void __launch_bounds__(1024) knn_scan_kernel(const int32_t* __restrict__ grid_dims, KnnWorkspace w) {
  __shared__ int32_t part[1024];
  const int b = blockIdx.x;
  const int bins = grid_dims[3 * b] * grid_dims[3 * b + 1] * grid_dims[3 * b + 2];
  int32_t* c = w.counts + (size_t)b * (kMaxBins + 1);
  const int per = (bins + 1023) / 1024;  // consecutive bins per thread
  const int lo = threadIdx.x * per;
  int sum = 0;
  for (int t = 0; t < per; ++t)
    if (lo + t < bins) sum += c[lo + t];
  part[threadIdx.x] = sum;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const int v = threadIdx.x >= off ? part[threadIdx.x - off] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int run = part[threadIdx.x] - sum;  // exclusive prefix of this thread's first bin
  for (int t = 0; t < per; ++t) {
    if (lo + t < bins) {
      const int v = c[lo + t];
      c[lo + t] = run;
      w.cursor[(size_t)b * kMaxBins + lo + t] = run;
      run += v;
    }
  }
  if (threadIdx.x == 1023) c[bins] = part[1023];
}

__global__ void knn_fill_kernel(const float* __restrict__ frac, const int32_t* __restrict__ num_atoms, int n_max,
                                KnnWorkspace w) {
  const int b = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = min(num_atoms[b], n_max);
  if (i >= n) return;
  const float* p = frac + ((size_t)b * n_max + i) * 3;
  const int key = w.keys[(size_t)b * n_max + i];
  const int slot = atomicAdd(&w.cursor[(size_t)b * kMaxBins + key], 1);
  w.sorted[(size_t)b * n_max + slot] = make_float4(p[0], p[1], p[2], __int_as_float(i));
}

// Bins along one axis of a structure and what that axis contributes to the two distance bounds of the search (double
// precision; the bounds are rounded down because they serve as lower bounds on distances to atoms that were not visited).
__device__ __forceinline__ int search_bins(const float* c, int axis, int n, int k, double* width) {
  double vol;
  const double w = axis_width(c, axis, &vol);
  vol = fmax(vol, 1e-12);
  // bin edge ~ 1.25 x the radius of a sphere holding k atoms at the mean density
  const double r_est = 1.25 * cbrt(3.0 * k * vol / (4.0 * 3.14159265358979323846 * fmax((double)n, 1.0)));
  *width = w;
  return (int)fmin(fmax(floor(w / r_est), 1.0), (double)kMaxBinsPerAxis);
}
__device__ __forceinline__ void search_bounds(const double (&w)[3], const int (&g)[3], float* bounds) {
  double h = 1e300, wmin = 1e300;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    h = fmin(h, w[a] / g[a]);
    wmin = fmin(wmin, w[a]);
  }
  bounds[0] = __double2float_rd(h * (1.0 - 1e-6));
  bounds[1] = __double2float_rd(0.5 * wmin * (1.0 - 1e-6));
}

__global__ void knn_grid_kernel(const float* __restrict__ cell, const int32_t* __restrict__ num_atoms, int B, int n_max,
                                int k, int32_t* __restrict__ grid_dims, float* __restrict__ bounds) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  double w[3];
  int g[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    g[a] = search_bins(cell + (size_t)b * 9, a, min(num_atoms[b], n_max), k, &w[a]);
    grid_dims[3 * b + a] = g[a];
  }
  search_bounds(w, g, bounds + 2 * b);
}

// Everything before the search in one launch, one CTA per structure: cell, grid, bounds, bin sizes and starts (counted and
// scanned in shared memory), atoms grouped by bin, empty rows of the padding.  Replaces seven launches (cell and grid, zero,
// count, scan, fill, padding), which take longer than the work they do for structures of a few thousand atoms; beyond
// kSetupAtoms one CTA would be slower than the separate kernels.
constexpr int kSetupAtoms = 16384;
__global__ void __launch_bounds__(1024) knn_setup_kernel(const float* __restrict__ frac, const float* __restrict__ lattice,
                                                         const float* __restrict__ cell, const int32_t* __restrict__ num_atoms,
                                                         int n_max, int k, KnnWorkspace w, int32_t* __restrict__ idx,
                                                         float* __restrict__ dist2) {
  __shared__ int32_t bins[kMaxBins];
  __shared__ int32_t part[32];
  __shared__ float sc[9];
  __shared__ double sw[3];
  __shared__ int sg[3];
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, n = min(num_atoms[b], n_max);
  if (tid < 32) {
    if (lattice) {
      if (tid == 0) cell_from_latent(lattice + (size_t)b * 6, sc);
    } else if (tid < 9) {
      sc[tid] = cell[(size_t)b * 9 + tid];
    }
    __syncwarp();
    if (tid < 3) sg[tid] = search_bins(sc, tid, n, k, &sw[tid]);
    if (tid < 9) w.cell[(size_t)b * 9 + tid] = sc[tid];
    __syncwarp();
    if (tid == 0) search_bounds({sw[0], sw[1], sw[2]}, {sg[0], sg[1], sg[2]}, w.bounds + 2 * b);
    if (tid < 3) w.grid[3 * b + tid] = sg[tid];
  } else {
    for (int t = tid - 32; t < kMaxBins; t += 992) bins[t] = 0;
  }
  __syncthreads();
  const int gx = sg[0], gy = sg[1], gz = sg[2];
  const float* pos = frac + (size_t)b * n_max * 3;
  bool outside = false;
  for (int i = tid; i < n; i += 1024) {
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    outside |= !(x >= 0.f && x < 1.f && y >= 0.f && y < 1.f && z >= 0.f && z < 1.f);
    atomicAdd(&bins[(cell_coord(x, gx) * gy + cell_coord(y, gy)) * gz + cell_coord(z, gz)], 1);
  }
  outside = __syncthreads_or(outside) != 0;
  if (tid == 0) w.flags[b] = outside;
  // exclusive scan, four bins per thread
  int c[4], sum = 0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    c[t] = bins[4 * tid + t];
    sum += c[t];
  }
  int run = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += v;
  }
  if (lane == 31) part[tid >> 5] = run;
  __syncthreads();
  if (tid < 32) {
    int v = part[tid];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    part[tid] = v;
  }
  __syncthreads();
  run += (tid >= 32 ? part[(tid >> 5) - 1] : 0) - sum;
  int32_t* start = w.counts + (size_t)b * (kMaxBins + 1);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    bins[4 * tid + t] = run;
    start[4 * tid + t] = run;
    run += c[t];
  }
  if (tid == 1023) start[kMaxBins] = run;
  __syncthreads();
  for (int i = tid; i < n; i += 1024) {
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    const int slot = atomicAdd(&bins[(cell_coord(x, gx) * gy + cell_coord(y, gy)) * gz + cell_coord(z, gz)], 1);
    w.sorted[(size_t)b * n_max + slot] = make_float4(x, y, z, __int_as_float(i));
  }
  for (long long t = tid + (long long)n * k; t < (long long)n_max * k; t += 1024) {
    idx[(size_t)b * n_max * k + t] = -1;
    if (dist2) dist2[(size_t)b * n_max * k + t] = INFINITY;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Warp-cooperative search.  One warp serves one bin of the grid: the atoms of the 3 x 3 x 3 bins around it are the candidates of
// every query atom in the bin, so they are gathered once into shared memory.  The k best live in a list spread over the lanes
// (lane t holds entry t, sorted by (d2, index)).  Two queries are searched together: distances of 64 candidates, two per lane
// and instruction; those within the first shell's reach are compacted, sorted across the lanes and become the list.  Queries
// whose k-th distance does not prove the first shell complete, structures searched exhaustively and neighbourhoods larger than
// the shared-memory list fall back to scanning bins straight from global memory, 32 candidates at a time: a candidate that
// beats the last entry is broadcast and every lane either keeps its entry, takes the candidate, or takes its left neighbour's
// entry.  Small structures without a first shell (fewer than three bins along an axis, or three along each) are searched as
// one list of all their atoms.  The result does not depend on the order of candidates, so it is the same, bit for bit, as the
// one-thread-per-query search.
// ---------------------------------------------------------------------------------------------------------------
// Candidates per warp in shared memory.  A 27-bin neighbourhood holds 27 bins of at least 1.25^3 3 k / 4 pi atoms, 201 at k = 16; from k of
// about 31 on (403 at 32) it does not fit, and every query of such a search scans global memory.
constexpr int kWarpCand = 384;
constexpr int kPairSurv = 128;  // survivors per query of the paired search

// Shared memory of one warp.  The paired search reads its candidates two at a time per coordinate and keeps the image offset
// of each (ox and oy as the upper halves of their fp32 patterns in one word, oz); the other searches hold float4 candidates.
struct alignas(16) KnnWarpMem {
  union {
    float4 cand[kWarpCand];
    struct {
      float nx[kWarpCand], ny[kWarpCand], nz[kWarpCand];  // negated coordinates
      int id[kWarpCand];
    };
  };
  uint32_t oxy[kWarpCand];
  float oz[kWarpCand];
  float2 surv[2][kPairSurv];  // (d2, index bits) of the candidates within the first shell's reach
};

// Two fp32 operations in one instruction, each rounded as its scalar form is.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

template <int KMAX>
__global__ void __launch_bounds__(128, 5) knn_warp_kernel(const float* __restrict__ cell,
                                                       const int32_t* __restrict__ num_atoms,
                                                       const int32_t* __restrict__ grid_dims,
                                                       const float* __restrict__ bounds, int n_max, int k,
                                                       int include_self, KnnWorkspace w, int32_t* __restrict__ idx,
                                                       float* __restrict__ dist2) {
  __shared__ KnnWarpMem mem_s[4];
  const int b = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gx = grid_dims[3 * b], gy = grid_dims[3 * b + 1], gz = grid_dims[3 * b + 2];
  const int n = min(num_atoms[b], n_max);
  const float4* sorted = w.sorted + (size_t)b * n_max;
  const int32_t* start = w.counts + (size_t)b * (kMaxBins + 1);
  const Cell c = load_cell(cell + (size_t)b * 9);
  // the grid has a fixed number of warps per structure; each takes every (warps per structure)-th bin, and where there are
  // more warps than bins (a few small structures) several of them share the queries of a bin
  const int bins = gx * gy * gz, warps = gridDim.x * 4, parts = max(1, min(32, warps / bins));
  for (int item = blockIdx.x * 4 + warp; item < bins * parts; item += warps) {
  const int bin = item % bins, part = item / bins;
  const int q0 = start[bin] + part, q1 = start[bin + 1];
  if (q0 >= q1) continue;
  const float h = bounds[2 * b];           // min over axes of width / bins, rounded down
  const float half_w = bounds[2 * b + 1];  // half the smallest perpendicular width, rounded down
  const float fast_limit2 = half_w * half_w * (1.f - 1e-4f);
  const bool exhaustive = w.flags[b] != 0;
  const int cz = bin % gz, cy = (bin / gz) % gy, cx = bin / (gy * gz);
  const int need = min(k, include_self ? n : n - 1);  // neighbours that exist
  KnnWarpMem& mem = mem_s[warp];

  // ---- the first shell's candidates, gathered once for all queries of the bin
  const bool covers = exhaustive || (gx <= 3 && gy <= 3 && gz <= 3);
  // From three bins per axis on, every neighbour bin is reached once, and whether that is across the cell boundary decides the
  // image.  Rounding the fractional delta finds another image only where the delta exceeds 0.5, and then both images are
  // beyond the reach: from one third of the cell's width on along that axis.
  bool paired = !covers && gx >= 3 && gy >= 3 && gz >= 3;
  int n_cand = 0;
  if (paired) {
    // The bins of a column along z lie one behind the other: nine columns, of one stretch or (where z wraps) two.  Lane t < 9
    // looks up column t; the loads of three columns are in flight together.
    const int zb = cz == 0 ? gz - 1 : 0, zlo = max(cz - 1, 0), zhi = min(cz + 1, gz - 1);
    const bool zwrap = cz == 0 || cz == gz - 1;
    const float ozb = cz == 0 ? 1.f : -1.f;
    int e0 = 0, c0 = 0, e1 = 0, c1 = 0;
    if (lane < 9) {
      const int x = cx + lane / 3 - 1, y = cy + lane % 3 - 1;
      const int col = ((x < 0 ? gx - 1 : (x >= gx ? 0 : x)) * gy + (y < 0 ? gy - 1 : (y >= gy ? 0 : y))) * gz;
      e0 = start[col + zlo];
      c0 = start[col + zhi + 1] - e0;
      if (zwrap) {
        e1 = start[col + zb];
        c1 = start[col + zb + 1] - e1;
      }
    }
    int off = c0 + c1;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += v;
    }
    n_cand = __shfl_sync(0xffffffffu, off, 8);
    off -= c0 + c1;
    paired = n_cand <= kWarpCand;
    if (paired) {
#pragma unroll 1
      for (int t0 = 0; t0 < 9; t0 += 3) {
        float4 v[3];
        int at[3], size[3], s0[3], s1[3], first[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          at[u] = __shfl_sync(0xffffffffu, off, t0 + u);
          s0[u] = __shfl_sync(0xffffffffu, e0, t0 + u);
          s1[u] = __shfl_sync(0xffffffffu, e1, t0 + u);
          first[u] = __shfl_sync(0xffffffffu, c0, t0 + u);
          size[u] = first[u] + __shfl_sync(0xffffffffu, c1, t0 + u);
          if (lane < size[u]) v[u] = __ldg(sorted + (lane < first[u] ? s0[u] + lane : s1[u] + lane - first[u]));
        }
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          const int x = cx + (t0 + u) / 3 - 1, y = cy + (t0 + u) % 3 - 1;
          const float ox = x < 0 ? 1.f : (x >= gx ? -1.f : 0.f), oy = y < 0 ? 1.f : (y >= gy ? -1.f : 0.f);
          const uint32_t oxy = __float_as_uint(ox) | (__float_as_uint(oy) >> 16);
          for (int e = lane; e < size[u]; e += 32) {
            if (e >= 32) v[u] = __ldg(sorted + (e < first[u] ? s0[u] + e : s1[u] + e - first[u]));
            mem.nx[at[u] + e] = -v[u].x;
            mem.ny[at[u] + e] = -v[u].y;
            mem.nz[at[u] + e] = -v[u].z;
            mem.id[at[u] + e] = __float_as_int(v[u].w);
            mem.oxy[at[u] + e] = oxy;
            mem.oz[at[u] + e] = e < first[u] ? 0.f : ozb;
          }
        }
      }
      for (int e = n_cand + lane; e < (n_cand + 63) / 64 * 64; e += 32) {  // (NaN is within no distance)
        mem.nx[e] = __int_as_float(0x7fffffff);
        mem.ny[e] = mem.nz[e] = 0.f;
        mem.id[e] = -1;
        mem.oxy[e] = 0;
        mem.oz[e] = 0.f;
      }
    }
  }
  const bool listed = !paired && n <= kWarpCand;  // all atoms of a small structure
  if (listed)
    for (int e = lane; e < n; e += 32) mem.cand[e] = __ldg(sorted + e);
  __syncwarp();

  // the list of the k best, entry t on lane t
  // entries are 64-bit keys, the bits of d2 (never negative) above the index: one comparison orders by (d2, index)
  constexpr unsigned long long kNone = ((unsigned long long)0x7f800000u << 32) | 0x7fffffffu;
  unsigned long long key = kNone;
  auto key_of = [](float d2, int i) { return ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)i; };
  auto dist_of = [](unsigned long long k) { return __uint_as_float((unsigned)(k >> 32)); };
  int my_id = -1;
  float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
  // A shell that does not cover every bin only counts if the k-th distance ends up below its reach (else the
  // search is repeated with a wider shell), so candidates at or beyond the reach can be dropped unseen.
  float keep_below = INFINITY;
  // d2 of one candidate per lane (INF where it does not count).  The image chosen by rounding the fractional delta is
  // the minimum image whenever it is closer than half the smallest cell width; a candidate whose rounded image is
  // farther needs the 27-image search only if something that far away could still be kept.
  auto distance = [&](float4 o, bool ok, float far_kept) {
    float d2 = INFINITY;
    if (ok && (include_self || __float_as_int(o.w) != my_id)) {
      if (!exhaustive) {
        const float dx = __fsub_rn(me.x, o.x), dy = __fsub_rn(me.y, o.y), dz = __fsub_rn(me.z, o.z);
        // -rint(delta) for |delta| < 1 (ties at +-0.5 go to 0), by comparison: cheaper than three conversions
        const float ox = dx > 0.5f ? -1.f : (dx < -0.5f ? 1.f : 0.f), oy = dy > 0.5f ? -1.f : (dy < -0.5f ? 1.f : 0.f),
                    oz = dz > 0.5f ? -1.f : (dz < -0.5f ? 1.f : 0.f);
        d2 = image_d2(dx, dy, dz, ox, oy, oz, c);
        if (d2 >= fast_limit2 && far_kept >= fast_limit2) d2 = min_image_d2(me.x, me.y, me.z, o.x, o.y, o.z, c);
      } else {
        d2 = min_image_d2(me.x, me.y, me.z, o.x, o.y, o.z, c);
      }
    }
    return d2;
  };
  // the lanes' candidates that beat the current last entry, inserted one at a time
  auto insert_batch = [&](float d2, int oid) {
    const unsigned long long mine = key_of(d2, oid);
    const unsigned long long last = __shfl_sync(0xffffffffu, key, KMAX - 1);
    uint32_t pass = __ballot_sync(0xffffffffu, d2 < keep_below && mine < last);
    while (pass) {
      const int src = __ffs(pass) - 1;
      pass &= pass - 1;
      const unsigned long long ck = __shfl_sync(0xffffffffu, mine, src);
      const uint32_t bal = __ballot_sync(0xffffffffu, lane < KMAX && ck < key);
      const unsigned long long pk = __shfl_up_sync(0xffffffffu, key, 1);
      if (bal == 0u) continue;  // earlier insertions of this batch pushed it out
      const int pos = __ffs(bal) - 1;
      if (lane == pos) key = ck;
      else if (lane > pos && lane < KMAX) key = pk;
    }
  };
  // 32 candidates, one per lane (valid where `ok`)
  auto consider = [&](float4 o, bool ok) {
    const float worst = dist_of(__shfl_sync(0xffffffffu, key, KMAX - 1));
    insert_batch(distance(o, ok, fminf(worst, keep_below)), __float_as_int(o.w));
  };
  // the lanes' 32 entries sorted ascending across the warp (bitonic network, 15 exchanges)
  auto sort_lanes = [&](unsigned long long& v) {
#pragma unroll 1
    for (int k2 = 2; k2 <= 32; k2 <<= 1) {
#pragma unroll 1
      for (int j = k2 >> 1; j > 0; j >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, j);
        const bool keep_min = ((lane & j) == 0) == ((lane & k2) == 0);
        if ((other < v) == keep_min) v = other;
      }
    }
  };
  // All atoms of the bins within s of the query's bin, straight from global memory.  The bins of a column along z are one
  // stretch of the sorted atoms (two where the run wraps): 32 columns are looked up at a time and walked as one list, the next
  // 32 atoms on their way while the current ones are compared.  Few queries come here, but a warp that does is on its own:
  // bin by bin (125 round trips to memory at s = 2) one of them took longer than the whole search of the others.
  auto scan_shell = [&](int s) {
    const int nx = exhaustive ? gx : min(2 * s + 1, gx);
    const int ny = exhaustive ? gy : min(2 * s + 1, gy);
    const int nz = exhaustive ? gz : min(2 * s + 1, gz);
    const int z0 = nz == gz ? 0 : (cz - s + gz) % gz, over = max(z0 + nz - gz, 0);
    for (int t0 = 0; t0 < nx * ny; t0 += 32) {
      int e0 = 0, c0 = 0, e1 = 0, c1 = 0;
      if (t0 + lane < nx * ny) {
        const int bx = ((cx - s + (t0 + lane) / ny) % gx + gx) % gx, by = ((cy - s + (t0 + lane) % ny) % gy + gy) % gy;
        const int col = (bx * gy + by) * gz;
        e0 = start[col + z0];
        c0 = start[col + z0 + nz - over] - e0;
        e1 = start[col];
        c1 = start[col + over] - e1;
      }
      int end = c0 + c1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
      }
      const int total = __shfl_sync(0xffffffffu, end, 31);
      auto load = [&](int p) {  // the p-th atom of these columns
        int t = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          if (__shfl_sync(0xffffffffu, end, t + o - 1) <= p) t += o;
        t = min(t, 31);  // (beyond the last one: not loaded)
        const int f0 = __shfl_sync(0xffffffffu, e0, t), n0 = __shfl_sync(0xffffffffu, c0, t), f1 = __shfl_sync(0xffffffffu, e1, t);
        const int r = p - (__shfl_sync(0xffffffffu, end, t) - n0 - __shfl_sync(0xffffffffu, c1, t));
        return p < total ? __ldg(sorted + (r < n0 ? f0 + r : f1 + r - n0)) : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      float4 next = load(lane);
      for (int p = lane; p - lane < total; p += 32) {
        const float4 o = next;
        next = load(p + 32);
        consider(o, p < total);
      }
    }
    return nx == gx && ny == gy && nz == gz;  // every bin was visited
  };

  const int s_max = max(max(gx, gy), gz);
  const float reach2 = h * h * (1.f - 2e-5f);
  const uint32_t below = (1u << lane) - 1u;
  // Every step below is written once (no unrolled copies, one place that scans a shell, one that finishes a row): with the same
  // steps inlined in several places half of every warp's cycles went into waiting for an instruction.  32 cells of 4 096 atoms,
  // k = 16, this kernel: one query at a time 247 us; with shells beyond the first scanned as stretches 198; two queries at a
  // time, inlined 237; as it stands 155 (2.5 instructions per clock and SM; at four CTAs per SM instead of five 156).
#pragma unroll 1
  for (int q = q0; q < q1; q += 2 * parts) {
    const int qs[2] = {q, q + parts < q1 ? q + parts : q};
    const float4 p0 = __ldg(sorted + qs[0]), p1 = __ldg(sorted + qs[1]);
    uint32_t word0 = 0, word1 = 0;
    int m0 = 0, m1 = 0;
    if (paired) {
      // two candidates of 64 per lane and instruction; both queries read them once
      const F2 qx[2] = {pack2(p0.x, p0.x), pack2(p1.x, p1.x)}, qy[2] = {pack2(p0.y, p0.y), pack2(p1.y, p1.y)},
               qz[2] = {pack2(p0.z, p0.z), pack2(p1.z, p1.z)};
      const int self[2] = {include_self ? -1 : __float_as_int(p0.w), include_self ? -1 : __float_as_int(p1.w)};
      int m[2] = {0, 0};
      const F2 l00 = pack2(c.l00, c.l00), l10 = pack2(c.l10, c.l10), l11 = pack2(c.l11, c.l11), l20 = pack2(c.l20, c.l20),
               l21 = pack2(c.l21, c.l21), l22 = pack2(c.l22, c.l22);
#pragma unroll 1
      for (int e = 2 * lane; e - 2 * lane < n_cand; e += 64) {
        const F2 nx = *reinterpret_cast<const F2*>(mem.nx + e), ny = *reinterpret_cast<const F2*>(mem.ny + e),
                 nz = *reinterpret_cast<const F2*>(mem.nz + e), oz = *reinterpret_cast<const F2*>(mem.oz + e);
        const int2 id = *reinterpret_cast<const int2*>(mem.id + e);
        const uint2 w2 = *reinterpret_cast<const uint2*>(mem.oxy + e);
        const F2 ox = pack2(__uint_as_float(w2.x & 0xffff0000u), __uint_as_float(w2.y & 0xffff0000u)),
                 oy = pack2(__uint_as_float(w2.x << 16), __uint_as_float(w2.y << 16));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const F2 ax = add2(add2(qx[u], nx), ox), ay = add2(add2(qy[u], ny), oy), az = add2(add2(qz[u], nz), oz);
          const F2 rx = fma2(az, l20, fma2(ay, l10, mul2(ax, l00))), ry = fma2(az, l21, mul2(ay, l11)), rz = mul2(az, l22);
          float d0, d1;
          unpack2(fma2(rz, rz, fma2(ry, ry, mul2(rx, rx))), d0, d1);
          const bool k0 = d0 < reach2 && id.x != self[u], k1 = d1 < reach2 && id.y != self[u];
          const uint32_t b0 = __ballot_sync(0xffffffffu, k0), b1 = __ballot_sync(0xffffffffu, k1);
          const int s0 = m[u] + __popc(b0 & below), mid = m[u] + __popc(b0), s1 = mid + __popc(b1 & below);
          if (k0 && s0 < kPairSurv) mem.surv[u][s0] = make_float2(d0, __int_as_float(id.x));
          if (k1 && s1 < kPairSurv) mem.surv[u][s1] = make_float2(d1, __int_as_float(id.y));
          m[u] = mid + __popc(b1);
        }
      }
      __syncwarp();
      // The first 32 survivors sorted by one 32-bit word each: the upper 27 bits of d2 and the slot.
      m0 = m[0], m1 = m[1];
      word0 = lane < m0 ? (__float_as_uint(mem.surv[0][lane].x) & ~31u) | lane : 0xffffffe0u | lane;
      word1 = lane < m1 ? (__float_as_uint(mem.surv[1][lane].x) & ~31u) | lane : 0xffffffe0u | lane;
#pragma unroll
      for (int k2 = 2; k2 <= 32; k2 <<= 1) {
#pragma unroll
        for (int j = k2 >> 1; j > 0; j >>= 1) {
          const bool keep_min = ((lane & j) == 0) == ((lane & k2) == 0);
          const uint32_t other0 = __shfl_xor_sync(0xffffffffu, word0, j), other1 = __shfl_xor_sync(0xffffffffu, word1, j);
          word0 = keep_min ? min(word0, other0) : max(word0, other0);
          word1 = keep_min ? min(word1, other1) : max(word1, other1);
        }
      }
    }
#pragma unroll 1
    for (int u = 0; u < (qs[1] == q ? 1 : 2); ++u) {
      me = u == 0 ? p0 : p1;
      my_id = __float_as_int(me.w);
      key = kNone;
      const int m = u == 0 ? m0 : m1;
      int s = 0;  // half-width of the shell searched so far
      bool all_bins = false;
      if (listed) {
        // the first 32 atoms sorted in one go, the others inserted while they beat the last entry (which also spares most of
        // the far ones the 27-image search)
        keep_below = INFINITY;
        const float4 o = lane < n ? mem.cand[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float d2 = distance(o, lane < n, INFINITY);
        if (d2 < INFINITY) key = key_of(d2, __float_as_int(o.w));
        sort_lanes(key);
        if (lane >= KMAX) key = kNone;
#pragma unroll 1
        for (int c0 = 32; c0 < n; c0 += 32) {
          const bool ok = c0 + lane < n;
          consider(ok ? mem.cand[c0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f), ok);
        }
        all_bins = true;
      } else if (paired && m <= kPairSurv) {
        keep_below = reach2;
        const float2* list = mem.surv[u];
        const float2 sv = lane < m ? list[(u == 0 ? word0 : word1) & 31] : make_float2(INFINITY, __int_as_float(0x7fffffff));
        key = key_of(sv.x, __float_as_int(sv.y));
        // where the words leave two of them out of order (they agree to 2^-18, or in d2 altogether) the full keys are sorted
        const unsigned long long next = __shfl_down_sync(0xffffffffu, key, 1);
        if (__any_sync(0xffffffffu, lane < 31 && next < key)) sort_lanes(key);
        if (lane >= KMAX) key = kNone;
#pragma unroll 1
        for (int c0 = 32; c0 < m; c0 += 32) {
          const bool ok = c0 + lane < m;
          const float2 o = ok ? list[c0 + lane] : make_float2(INFINITY, __int_as_float(0x7fffffff));
          unsigned long long mine = key_of(o.x, __float_as_int(o.y));
          const unsigned long long last = __shfl_sync(0xffffffffu, key, KMAX - 1);
          if (__popc(__ballot_sync(0xffffffffu, mine < last)) <= 10) {
            insert_batch(o.x, __float_as_int(o.y));
            continue;
          }
          // many of them: sorted too, and the two lists merged
          sort_lanes(mine);
          const unsigned long long r = __shfl_sync(0xffffffffu, mine, (KMAX - 1 - lane) & 31);
          if (lane < KMAX && r < key) key = r;
#pragma unroll 1
          for (int j = KMAX / 2; j > 0; j >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
            if ((other < key) == ((lane & j) == 0)) key = other;
          }
        }
        s = 1;
      }
      // complete when the needed neighbours are known and the farthest of them is inside the searched shell
#pragma unroll 1
      while (!all_bins) {
        if (s > 0) {
          const float reach = (float)s * h;
          const float kth = need >= 1 ? dist_of(__shfl_sync(0xffffffffu, key, need - 1)) : 0.f;
          if (exhaustive || kth < reach * reach * (1.f - 2e-5f) || s >= s_max) break;
        }
        ++s;
        key = kNone;
        {  // the reach of the shell, unless it is the last one (every bin, or the largest half-width)
          const bool last = exhaustive || (2 * s + 1 >= gx && 2 * s + 1 >= gy && 2 * s + 1 >= gz) || s >= s_max;
          const float reach_s = (float)s * h;
          keep_below = last ? INFINITY : reach_s * reach_s * (1.f - 2e-5f);
        }
        all_bins = scan_shell(s);
      }
      if (lane < k) {
        const bool have = dist_of(key) < INFINITY;
        idx[((size_t)b * n_max + my_id) * k + lane] = have ? (int)(unsigned)key : -1;
        if (dist2) dist2[((size_t)b * n_max + my_id) * k + lane] = have ? dist_of(key) : INFINITY;
      }
    }
    __syncwarp();  // the survivors are rewritten for the next pair
  }
  __syncwarp();  // the shared-memory list is refilled for the next bin
  }
}

// rows of padded atoms: no neighbours
__global__ void knn_pad_rows_kernel(const int32_t* __restrict__ num_atoms, int n_max, int k, int32_t* __restrict__ idx,
                                    float* __restrict__ dist2) {
  const int b = blockIdx.y;
  const int n = min(num_atoms[b], n_max);
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // (row - n) * k + t
  const long long total = (long long)(n_max - n) * k;
  if (i >= total) return;
  const size_t off = ((size_t)b * n_max + n) * k + i;
  idx[off] = -1;
  if (dist2) dist2[off] = INFINITY;
}

KnnWorkspace carve(void* ws, int B, int N) {
  char* p = static_cast<char*>(ws);
  KnnWorkspace w;
  w.counts = reinterpret_cast<int32_t*>(p);
  p += align_up((size_t)B * (kMaxBins + 1) * 4, 256);
  w.cursor = reinterpret_cast<int32_t*>(p);
  p += align_up((size_t)B * kMaxBins * 4, 256);
  w.keys = reinterpret_cast<int32_t*>(p);
  p += align_up((size_t)B * N * 4, 256);
  w.flags = reinterpret_cast<int32_t*>(p);
  p += align_up((size_t)B * 4, 256);
  w.sorted = reinterpret_cast<float4*>(p);
  p += align_up((size_t)B * N * sizeof(float4), 256);
  w.cell = reinterpret_cast<float*>(p);
  w.grid = reinterpret_cast<int32_t*>(w.cell + 9 * (size_t)B);
  w.bounds = reinterpret_cast<float*>(w.grid + 3 * (size_t)B);
  return w;
}

}  // namespace
}  // namespace mf

using namespace mf;

extern "C" size_t mf_knn_cells_workspace_bytes(int32_t batch, int32_t n_max) {
  const size_t B = batch, N = n_max;
  return align_up(B * (kMaxBins + 1) * 4, 256) + align_up(B * kMaxBins * 4, 256) + align_up(B * N * 4, 256) +
         align_up(B * 4, 256) + align_up(B * N * sizeof(float4), 256) + align_up(B * 14 * 4, 256);
}

extern "C" int mf_knn_search_grid(const float* cell, const int32_t* num_atoms, int32_t batch, int32_t n_max, int32_t k,
                                  int32_t* grid_dims, float* bounds, void* stream) {
  MF_CHECK_ARG(batch >= 0 && n_max >= 0 && k >= 1, "mf_knn_search_grid: bad size");
  if (batch == 0) return MF_OK;
  MF_CHECK_ARG(cell && num_atoms && grid_dims && bounds, "mf_knn_search_grid: null pointer argument");
  knn_grid_kernel<<<(batch + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(cell, num_atoms, batch, n_max, k,
                                                                                      grid_dims, bounds);
  MF_CHECK_LAUNCH("knn_grid_kernel");
  return MF_OK;
}

namespace mf {
namespace {

int knn_check(const void* frac, const void* cell, const void* num_atoms, int batch, int n_max, int k, const void* idx,
              const void* workspace, size_t workspace_bytes, const char* name) {
  MF_CHECK_ARG(batch >= 0 && n_max >= 0, "%s: negative size", name);
  MF_CHECK_ARG(k >= 1 && k <= 32, "%s: k must be in [1, 32], got %d", name, k);
  if (batch == 0 || n_max == 0) return MF_OK;
  MF_CHECK_ARG(frac && cell && num_atoms && idx, "%s: null pointer argument", name);
  MF_CHECK_ARG(batch <= 65535, "%s: batch above 65535", name);
  const size_t need = mf_knn_cells_workspace_bytes(batch, n_max);
  if (!workspace || workspace_bytes < need) {
    set_error("%s: workspace of %zu bytes needed, %zu given", name, need, workspace_bytes);
    return MF_ERR_WORKSPACE_TOO_SMALL;
  }
  return MF_OK;
}

int knn_search(const float* cell, const int32_t* num_atoms, const int32_t* grid_dims, const float* bounds, int batch, int n_max,
               int k, int include_self, const KnnWorkspace& w, int32_t* idx, float* dist2, cudaStream_t s) {
  // at least 256 warps per structure, more when there are few structures: about 4700 (four per scheduler and SM twice over)
  const int wanted = (1184 + batch - 1) / batch;
  dim3 grid(wanted > 64 ? wanted : 64, batch);
  if (k <= 16)
    knn_warp_kernel<16><<<grid, 128, 0, s>>>(cell, num_atoms, grid_dims, bounds, n_max, k, include_self, w, idx, dist2);
  else
    knn_warp_kernel<32><<<grid, 128, 0, s>>>(cell, num_atoms, grid_dims, bounds, n_max, k, include_self, w, idx, dist2);
  MF_CHECK_LAUNCH("knn_warp_kernel");
  return MF_OK;
}

// Binning and search on a grid that already exists, without the setup kernel: structures of any size.
int knn_binned(const float* frac, const float* cell, const int32_t* num_atoms, const int32_t* grid_dims, const float* bounds,
               int batch, int n_max, int k, int include_self, const KnnWorkspace& w, int32_t* idx, float* dist2,
               cudaStream_t s) {
  const int zero_n = batch * (kMaxBins + 1);
  knn_zero_kernel<<<(zero_n + 255) / 256, 256, 0, s>>>(w.counts, w.flags, batch);
  MF_CHECK_LAUNCH("knn_zero_kernel");
  dim3 per_atom((n_max + 255) / 256, batch);
  knn_count_kernel<<<per_atom, 256, 0, s>>>(frac, num_atoms, grid_dims, n_max, w);
  MF_CHECK_LAUNCH("knn_count_kernel");
  knn_scan_kernel<<<batch, 1024, 0, s>>>(grid_dims, w);
  MF_CHECK_LAUNCH("knn_scan_kernel");
  knn_fill_kernel<<<per_atom, 256, 0, s>>>(frac, num_atoms, n_max, w);
  MF_CHECK_LAUNCH("knn_fill_kernel");
  const int rc = knn_search(cell, num_atoms, grid_dims, bounds, batch, n_max, k, include_self, w, idx, dist2, s);
  if (rc != MF_OK) return rc;
  const long long pad = (long long)n_max * k;
  knn_pad_rows_kernel<<<dim3((unsigned)((pad + 255) / 256), batch), 256, 0, s>>>(num_atoms, n_max, k, idx, dist2);
  MF_CHECK_LAUNCH("knn_pad_rows_kernel");
  return MF_OK;
}

__global__ void knn_cell_kernel(const float* __restrict__ lattice, int B, float* __restrict__ cell) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < B) cell_from_latent(lattice + (size_t)b * 6, cell + (size_t)b * 9);
}

}  // namespace
}  // namespace mf

extern "C" int mf_knn_topk_cells(const float* frac, const float* cell, const int32_t* num_atoms,
                                 const int32_t* grid_dims, const float* bounds, int32_t batch, int32_t n_max,
                                 int32_t k, int32_t include_self, int32_t* idx, float* dist2, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  const int rc = knn_check(frac, cell, num_atoms, batch, n_max, k, idx, workspace, workspace_bytes, "mf_knn_topk_cells");
  if (rc != MF_OK || batch == 0 || n_max == 0) return rc;
  MF_CHECK_ARG(grid_dims && bounds, "mf_knn_topk_cells: null pointer argument");
  return knn_binned(frac, cell, num_atoms, grid_dims, bounds, batch, n_max, k, include_self, carve(workspace, batch, n_max), idx,
                    dist2, static_cast<cudaStream_t>(stream));
}

extern "C" int mf_knn_topk_lattice(const float* frac, const float* lattice, int32_t lattice_is_cell, const int32_t* num_atoms,
                                   int32_t batch, int32_t n_max, int32_t k, int32_t include_self, int32_t* idx, float* dist2,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  int rc = knn_check(frac, lattice, num_atoms, batch, n_max, k, idx, workspace, workspace_bytes, "mf_knn_topk_lattice");
  if (rc != MF_OK || batch == 0 || n_max == 0) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const KnnWorkspace w = carve(workspace, batch, n_max);
  if (n_max <= kSetupAtoms) {
    knn_setup_kernel<<<batch, 1024, 0, s>>>(frac, lattice_is_cell ? nullptr : lattice, lattice, num_atoms, n_max, k, w, idx, dist2);
    MF_CHECK_LAUNCH("knn_setup_kernel");
    return knn_search(w.cell, num_atoms, w.grid, w.bounds, batch, n_max, k, include_self, w, idx, dist2, s);
  }
  if (!lattice_is_cell) {
    knn_cell_kernel<<<(batch + 127) / 128, 128, 0, s>>>(lattice, batch, w.cell);
    MF_CHECK_LAUNCH("knn_cell_kernel");
  }
  const float* cell = lattice_is_cell ? lattice : w.cell;
  if ((rc = mf_knn_search_grid(cell, num_atoms, batch, n_max, k, w.grid, w.bounds, stream)) != MF_OK) return rc;
  return knn_binned(frac, cell, num_atoms, w.grid, w.bounds, batch, n_max, k, include_self, w, idx, dist2, s);
}
