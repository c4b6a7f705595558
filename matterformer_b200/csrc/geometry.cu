// Periodic geometry kernels: minimum-image distances, k nearest neighbours,
// cell sort and the radius block list with its per-block pair bitmaps.
//
// Every distance is evaluated with one fixed sequence of IEEE fp32 operations
// (see min_image_d2) that the CPU oracle repeats operation for operation, so
// the integer outputs (neighbour indices, permutation, block lists, bitmaps)
// can be compared bit for bit.
//
// Distance semantics follow PeriodicGeometryAdapter.forward of the reference
// (src/matterformer/geometry/adapters.py:176-190): fractional delta plus each of
// the 27 lattice offsets in itertools.product(range(-1,2), repeat=3) order,
// squared length under the cell metric, first minimum wins.
#include "common.cuh"
#include "geometry.cuh"

namespace mf {

namespace {

// ---------------------------------------------------------------------------
// kNN: one thread per query atom, candidates streamed through shared memory,
// the k best kept as a sorted register list.  Candidates arrive in ascending
// index order and only a strictly smaller distance displaces an entry, so ties
// resolve to the lower index.
// ---------------------------------------------------------------------------
template <int KMAX>
__global__ void __launch_bounds__(128) knn_kernel(const float* __restrict__ frac, const float* __restrict__ cell,
                                                  const int32_t* __restrict__ num_atoms, int n_max, int k,
                                                  int include_self, int32_t* __restrict__ idx,
                                                  float* __restrict__ dist2) {
  __shared__ float sx[128], sy[128], sz[128];
  const int b = blockIdx.y;
  const int n = min(num_atoms[b], n_max);
  const int i = blockIdx.x * 128 + threadIdx.x;
  const float* pos = frac + (size_t)b * n_max * 3;
  const Cell c = load_cell(cell + (size_t)b * 9);
  const bool active = i < n;
  float xi = 0.f, yi = 0.f, zi = 0.f;
  if (active) {
    xi = pos[3 * i + 0];
    yi = pos[3 * i + 1];
    zi = pos[3 * i + 2];
  }
  float bd[KMAX];
  int bi[KMAX];
#pragma unroll
  for (int t = 0; t < KMAX; ++t) {
    bd[t] = INFINITY;
    bi[t] = -1;
  }
  for (int j0 = 0; j0 < n; j0 += 128) {
    __syncthreads();
    const int jl = j0 + threadIdx.x;
    if (jl < n) {
      sx[threadIdx.x] = pos[3 * jl + 0];
      sy[threadIdx.x] = pos[3 * jl + 1];
      sz[threadIdx.x] = pos[3 * jl + 2];
    }
    __syncthreads();
    if (!active) continue;
    const int cnt = min(128, n - j0);
    for (int t = 0; t < cnt; ++t) {
      const int j = j0 + t;
      if (j == i && !include_self) continue;
      const float d2 = min_image_d2(xi, yi, zi, sx[t], sy[t], sz[t], c);
      if (d2 < bd[KMAX - 1]) {
        float cd = d2;
        int ci = j;
        bool shifting = false;
#pragma unroll
        for (int s = 0; s < KMAX; ++s) {
          const bool sw = shifting || (cd < bd[s]);
          const float td = bd[s];
          const int ti = bi[s];
          bd[s] = sw ? cd : td;
          bi[s] = sw ? ci : ti;
          cd = sw ? td : cd;
          ci = sw ? ti : ci;
          shifting = sw;
        }
      }
    }
  }
  if (i < n_max) {
    int32_t* oi = idx + ((size_t)b * n_max + i) * k;
    float* od = dist2 ? dist2 + ((size_t)b * n_max + i) * k : nullptr;
#pragma unroll
    for (int t = 0; t < KMAX; ++t) {
      if (t < k) {
        oi[t] = active ? bi[t] : -1;
        if (od) od[t] = active ? bd[t] : INFINITY;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// cell sort and block list: two launches
//
// Bound by launches and the host: 8 structures of 300-500 atoms took 443 us as 54 launches (the cell and the grid as chains
// of element-wise operations, keys, ranks, one CTA per pair of tiles, compaction) of 132 us on the device, and take 12.5 us as two,
// the second of which is launched while the first one runs.
// ---------------------------------------------------------------------------
// What the second kernel needs of a structure: its cell and the perpendicular widths.
struct StructureInfo {
  float cell[9];
  float width[3];
};

constexpr int kRankAtoms = 64;   // atoms per CTA
constexpr int kRankTile = 2048;  // keys in shared memory at a time

// Grid cell of every atom and its rank = number of atoms with a smaller (cell, index); padded atoms keep their place.
// The cell comes from `lattice` (latents) or `cell`, the grid from `grid_dims` or from the widths and the cutoff; every CTA
// of a structure works both out again, which costs less than a launch.  16 threads share an atom's comparisons.
__global__ void __launch_bounds__(1024) cell_rank_kernel(const float* __restrict__ frac, const float* __restrict__ lattice,
                                                         const float* __restrict__ cell, const int32_t* __restrict__ num_atoms,
                                                         const int32_t* __restrict__ grid_dims, double cutoff, int n_max,
                                                         StructureInfo* __restrict__ info, int32_t* __restrict__ perm) {
  __shared__ int32_t keys[kRankTile];
  __shared__ float sc[9];
  __shared__ int grid[3];
  const int b = blockIdx.y, tid = threadIdx.x;
  const int i0 = blockIdx.x * kRankAtoms;
  launch_dependents();
  // the first positions are on their way while one warp works out the grid
  float first[2][3];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int x = 0; x < 3; ++x) first[t][x] = tid + 1024 * t < n_max ? frac[((size_t)b * n_max + tid + 1024 * t) * 3 + x] : 0.f;
  const int n = min(num_atoms[b], n_max);
  if (tid < 32) {
    if (lattice) {
      if (tid == 0) cell_from_latent(lattice + (size_t)b * 6, sc);
    } else if (tid < 9) {
      sc[tid] = cell[(size_t)b * 9 + tid];
    }
    __syncwarp();
    if (tid < 3) {
      double vol;
      const double w = axis_width(sc, tid, &vol);
      grid[tid] = grid_dims ? grid_dims[3 * b + tid] : (int)fmin(fmax(floor(w / fmax(cutoff, 1e-12)), 1.0), 64.0);
      if (blockIdx.x == 0) info[b].width[tid] = (float)w;
    }
    if (blockIdx.x == 0 && tid < 9) info[b].cell[tid] = sc[tid];
  }
  __syncthreads();
  const int gx = grid[0], gy = grid[1], gz = grid[2];
  auto key_at = [&](const float* p) { return (cell_coord(p[0], gx) * gy + cell_coord(p[1], gy)) * gz + cell_coord(p[2], gz); };
  auto key_of = [&](int i) { return key_at(frac + ((size_t)b * n_max + i) * 3); };
  const int i = i0 + (tid >> 4), part = tid & 15;
  const int ki = i < n ? key_of(i) : 0;
  int rank = 0;
  for (int j0 = 0; j0 < n && i0 < n; j0 += kRankTile) {
    const int cnt = min(kRankTile, n - j0);
    __syncthreads();
    if (j0 == 0) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (tid + 1024 * t < cnt) keys[tid + 1024 * t] = key_at(first[t]);
    } else {
      for (int t = tid; t < cnt; t += 1024) keys[t] = key_of(j0 + t);
    }
    __syncthreads();
#pragma unroll 4
    for (int t = part; t < cnt; t += 16) rank += keys[t] < ki + (j0 + t < i ? 1 : 0);  // ties: the lower index first
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
  if (part == 0 && i < n_max) perm[(size_t)b * n_max + (i < n ? rank : i)] = i;
}

// The largest float whose rounded square root is at most `cutoff`: sqrt(d2) <= cutoff and d2 <= this are the same bit, as a
// correctly rounded square root is monotonous.
__device__ __forceinline__ float squared_cutoff(float cutoff) {
  float t = __fmul_rn(cutoff, cutoff);  // off by a few floats at most
  while (__fsqrt_rn(t) > cutoff) t = __uint_as_float(__float_as_uint(t) - 1u);
  while (t < INFINITY && __fsqrt_rn(__uint_as_float(__float_as_uint(t) + 1u)) <= cutoff) t = __uint_as_float(__float_as_uint(t) + 1u);
  return t;
}

// Whether one of the 27 images of the pair is within the cutoff: the images that min_image_d2 would minimise over, less
// those that lie farther than `limit` by their distance along one axis alone.
__device__ __forceinline__ bool within_cutoff(float dx, float dy, float dz, const Cell& c, const float* width, float limit, float cutoff2) {
  bool hit = false;
#pragma unroll 1
  for (int ox = -1; ox <= 1; ++ox) {
    const float ax = __fadd_rn(dx, (float)ox);
    if (fabsf(ax) * width[0] > limit) continue;
#pragma unroll 1
    for (int oy = -1; oy <= 1; ++oy) {
      const float ay = __fadd_rn(dy, (float)oy);
      if (fabsf(ay) * width[1] > limit) continue;
#pragma unroll
      for (int oz = -1; oz <= 1; ++oz) {
        const float az = __fadd_rn(dz, (float)oz);
        if (fabsf(az) * width[2] > limit) continue;
        hit |= image_d2(dx, dy, dz, (float)ox, (float)oy, (float)oz, c) <= cutoff2;
      }
    }
  }
  return hit;
}

// The offset of -1, 0 or 1 that brings a fractional difference nearest to zero, added to it.
__device__ __forceinline__ float2 nearest_image(float2 d) {
  return add2(d, make_float2(fabsf(d.x) > 0.5f ? copysignf(1.f, -d.x) : 0.f, fabsf(d.y) > 0.5f ? copysignf(1.f, -d.y) : 0.f));
}

// One CTA per row tile I; a warp takes column tiles, a lane the row I*32 + lane of the bitmap.  The active column tiles are
// collected in shared memory and listed at the end.
//
// Bound by instructions once the first loads are in.  What decides how many images of a pair have to be looked at is a bound on
// its distance along each axis: the cutoff with a margin for the rounding of the distances that it stands for, which grows
// with the coordinates and is taken once for a pair of tiles.  Where it is below half of each width, at most one image per axis
// passes, the nearest, and is evaluated without a test, two columns at a time: the same bits as the minimum over 27.  8 structures
// of 300-500 atoms, cutoff 6 Angstrom: 21 us with the loop over images for every pair, 12.4 us with a bound per pair and a column
// per lane, 6.0 us now; 16 of 512-1 024 atoms 66.6 -> 24.8 us.
constexpr int kListWarps = 16;
constexpr int kListAtoms = 1024;  // columns in shared memory at a time
__global__ void __launch_bounds__(32 * kListWarps) block_list_kernel(const float* __restrict__ frac, const StructureInfo* __restrict__ info,
                                                          const int32_t* __restrict__ num_atoms, const int32_t* __restrict__ perm,
                                                          int n_max, int tiles, float cutoff, uint32_t* __restrict__ block_mask,
                                                          int32_t* __restrict__ block_count, int32_t* __restrict__ block_cols) {
  extern __shared__ uint32_t active[];  // bit J
  __shared__ __align__(16) float px[kListAtoms], py[kListAtoms], pz[kListAtoms];  // minus the coordinates of sorted atoms
  __shared__ float reach[kListAtoms / 32];                                        // largest |x| + |y| + |z| of a column tile
  const int I = blockIdx.x, b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* pos = frac + (size_t)b * n_max * 3;
  const int32_t* pb = perm + (size_t)b * n_max;
  const int words = (tiles + 31) / 32;
  for (int t = threadIdx.x; t < words; t += 32 * kListWarps) active[t] = 0u;
  const float cutoff2 = squared_cutoff(cutoff);
  wait_for_previous();
  const int n = min(num_atoms[b], n_max);
  const Cell c = load_cell(info[b].cell);
  const float width[3] = {info[b].width[0], info[b].width[1], info[b].width[2]};
  float sum = 0.f;
#pragma unroll
  for (int t = 0; t < 9; ++t) sum += fabsf(info[b].cell[t]);
  const float margin = 4e-6f * sum, half_width = 0.4999f * fminf(fminf(width[0], width[1]), width[2]);
  const int si = 32 * I + lane;
  float xi = 0.f, yi = 0.f, zi = 0.f;
  if (si < n) {
    const int ai = pb[si];
    xi = pos[3 * ai], yi = pos[3 * ai + 1], zi = pos[3 * ai + 2];
  }
  const float row_reach = warp_max(fabsf(xi) + fabsf(yi) + fabsf(zi));
  const float2 x2 = make_float2(xi, xi), y2 = make_float2(yi, yi), z2 = make_float2(zi, zi);
  const float2 l00 = make_float2(c.l00, c.l00), l10 = make_float2(c.l10, c.l10), l11 = make_float2(c.l11, c.l11),
               l20 = make_float2(c.l20, c.l20), l21 = make_float2(c.l21, c.l21), l22 = make_float2(c.l22, c.l22);
  uint32_t* mask = block_mask + ((size_t)b * tiles + I) * tiles * 32 + lane;
  for (int J0 = 0; J0 < tiles; J0 += kListAtoms / 32) {
    __syncthreads();
    for (int t = warp; t < min(kListAtoms / 32, tiles - J0); t += kListWarps) {
      const int sj = 32 * (J0 + t) + lane;
      float x = 0.f, y = 0.f, z = 0.f;
      if (sj < n) {
        const int aj = pb[sj];
        x = pos[3 * aj], y = pos[3 * aj + 1], z = pos[3 * aj + 2];
      }
      px[32 * t + lane] = -x, py[32 * t + lane] = -y, pz[32 * t + lane] = -z;
      const float far = warp_max(fabsf(x) + fabsf(y) + fabsf(z));
      if (lane == 0) reach[t] = far;
    }
    __syncthreads();
    for (int t = warp; t < min(kListAtoms / 32, tiles - J0); t += kListWarps) {
      const int left = n - 32 * (J0 + t);
      const float limit = fmaf(margin, 1.0001f * (row_reach + reach[t]) + 3.f, cutoff * 1.0001f);
      uint32_t word = 0u;
      if (left <= 0 || 32 * I >= n) {
        // nothing but padding
      } else if (limit < half_width) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 ax = nearest_image(add2(x2, *reinterpret_cast<const float2*>(&px[32 * t + j])));
          const float2 ay = nearest_image(add2(y2, *reinterpret_cast<const float2*>(&py[32 * t + j])));
          const float2 az = nearest_image(add2(z2, *reinterpret_cast<const float2*>(&pz[32 * t + j])));
          const float2 rx = fma2(az, l20, fma2(ay, l10, mul2(ax, l00))), ry = fma2(az, l21, mul2(ay, l11)), rz = mul2(az, l22);
          const float2 d2 = fma2(rz, rz, fma2(ry, ry, mul2(rx, rx)));
          if (d2.x <= cutoff2) word |= 1u << j;
          if (d2.y <= cutoff2) word |= 2u << j;
        }
      } else {
        for (int j = 0; j < min(left, 32); ++j)
          if (within_cutoff(__fadd_rn(xi, px[32 * t + j]), __fadd_rn(yi, py[32 * t + j]), __fadd_rn(zi, pz[32 * t + j]), c, width, limit, cutoff2))
            word |= 1u << j;
      }
      if (si >= n) word = 0u;
      if (left < 32) word &= left > 0 ? (1u << left) - 1u : 0u;
      mask[(size_t)(J0 + t) * 32] = word;
      if (__any_sync(0xffffffffu, word != 0u) && lane == 0) atomicOr(&active[(J0 + t) >> 5], 1u << ((J0 + t) & 31));
    }
  }
  __syncthreads();
  if (warp == 0) {
    int32_t* cols = block_cols + ((size_t)b * tiles + I) * tiles;
    int count = 0;
    for (int w = 0; w < words; ++w) {
      const uint32_t bits = active[w];
      if ((bits >> lane) & 1u) cols[count + __popc(bits & ((1u << lane) - 1u))] = 32 * w + lane;
      count += __popc(bits);
    }
    for (int t = count + lane; t < tiles; t += 32) cols[t] = -1;
    if (lane == 0) block_count[(size_t)b * tiles + I] = count;
  }
}

int radius_blocks(const float* frac, const float* lattice, const float* cell, const int32_t* num_atoms,
                  const int32_t* grid_dims, int32_t batch, int32_t n_max, double cutoff, int32_t* perm, int32_t* block_count,
                  int32_t* block_cols, uint32_t* block_mask, void* workspace, size_t workspace_bytes, const char* name,
                  cudaStream_t s) {
  MF_CHECK_ARG(batch >= 0 && n_max >= 0, "%s: negative size", name);
  MF_CHECK_ARG(cutoff >= 0.0, "%s: cutoff must be non-negative", name);
  if (batch == 0 || n_max == 0) return MF_OK;
  MF_CHECK_ARG(frac && (lattice || cell) && num_atoms && perm && block_count && block_cols && block_mask,
               "%s: null pointer argument", name);
  const size_t need = mf_radius_blocks_workspace_bytes(batch, n_max);
  if (!workspace || workspace_bytes < need) {
    set_error("%s: workspace of %zu bytes needed, %zu given", name, need, workspace_bytes);
    return MF_ERR_WORKSPACE_TOO_SMALL;
  }
  MF_CHECK_ARG(batch <= 65535, "%s: batch above 65535", name);
  const int tiles = (n_max + 31) / 32;
  const size_t words = (size_t)(tiles + 31) / 32 * 4;
  MF_CHECK_ARG(words <= 48 * 1024, "%s: %d tokens are too many", name, (int)n_max);  // 12 million
  StructureInfo* info = static_cast<StructureInfo*>(workspace);
  cell_rank_kernel<<<dim3((n_max + kRankAtoms - 1) / kRankAtoms, batch), 1024, 0, s>>>(frac, lattice, cell, num_atoms, grid_dims,
                                                                                       cutoff, n_max, info, perm);
  MF_CHECK_LAUNCH("cell_rank_kernel");
  if (words > 32 * 1024) {  // with the staged atoms more than a launch takes by default
    const cudaError_t e = cudaFuncSetAttribute(block_list_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024);
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(block_list_kernel)");
  }
  const cudaError_t e = launch_dependent(block_list_kernel, dim3(tiles, batch), dim3(32 * kListWarps), words, s, frac, info, num_atoms, perm,
                                         n_max, tiles, (float)cutoff, block_mask, block_count, block_cols);
  if (e != cudaSuccess) return cuda_error(e, "block_list_kernel");
  return MF_OK;
}

}  // namespace
}  // namespace mf

using namespace mf;

extern "C" int mf_knn_topk(const float* frac, const float* cell, const int32_t* num_atoms, int32_t batch,
                           int32_t n_max, int32_t k, int32_t include_self, int32_t* idx, float* dist2,
                           void* stream) {
  MF_CHECK_ARG(batch >= 0 && n_max >= 0, "mf_knn_topk: negative size");
  MF_CHECK_ARG(k >= 1 && k <= 32, "mf_knn_topk: k must be in [1, 32], got %d", (int)k);
  if (batch == 0 || n_max == 0) return MF_OK;
  MF_CHECK_ARG(frac && cell && num_atoms && idx, "mf_knn_topk: null pointer argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  dim3 grid((n_max + 127) / 128, batch);
  if (k <= 16)
    knn_kernel<16><<<grid, 128, 0, s>>>(frac, cell, num_atoms, n_max, k, include_self, idx, dist2);
  else
    knn_kernel<32><<<grid, 128, 0, s>>>(frac, cell, num_atoms, n_max, k, include_self, idx, dist2);
  MF_CHECK_LAUNCH("knn_kernel");
  return MF_OK;
}

extern "C" size_t mf_radius_blocks_workspace_bytes(int32_t batch, int32_t) {
  return align_up((size_t)batch * sizeof(StructureInfo), 256);
}

extern "C" int mf_cell_sort_blocklist(const float* frac, const float* cell, const int32_t* num_atoms,
                                      const int32_t* grid_dims, int32_t batch, int32_t n_max, float cutoff,
                                      int32_t* perm, int32_t* block_count, int32_t* block_cols,
                                      uint32_t* block_mask, void* workspace, size_t workspace_bytes, void* stream) {
  MF_CHECK_ARG(grid_dims || batch <= 0 || n_max <= 0, "mf_cell_sort_blocklist: null pointer argument");
  return radius_blocks(frac, nullptr, cell, num_atoms, grid_dims, batch, n_max, cutoff, perm, block_count, block_cols,
                       block_mask, workspace, workspace_bytes, "mf_cell_sort_blocklist", static_cast<cudaStream_t>(stream));
}

extern "C" int mf_radius_blocks(const float* frac, const float* lattice, int32_t lattice_is_cell, const int32_t* num_atoms,
                                int32_t batch, int32_t n_max, double cutoff, int32_t* perm, int32_t* block_count,
                                int32_t* block_cols, uint32_t* block_mask, void* workspace, size_t workspace_bytes,
                                void* stream) {
  return radius_blocks(frac, lattice_is_cell ? nullptr : lattice, lattice_is_cell ? lattice : nullptr, num_atoms, nullptr, batch,
                       n_max, cutoff, perm, block_count, block_cols, block_mask, workspace, workspace_bytes, "mf_radius_blocks",
                       static_cast<cudaStream_t>(stream));
}
