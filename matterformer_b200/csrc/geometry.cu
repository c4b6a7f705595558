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
// of element-wise operations, keys, ranks, one CTA per pair of tiles, compaction) of 132 us on the device, and take 27 us
// as two.
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
  const int b = blockIdx.y, tid = threadIdx.x, n = min(num_atoms[b], n_max);
  const int i0 = blockIdx.x * kRankAtoms;
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
  auto key_of = [&](int i) {
    const float* p = frac + ((size_t)b * n_max + i) * 3;
    return (cell_coord(p[0], gx) * gy + cell_coord(p[1], gy)) * gz + cell_coord(p[2], gz);
  };
  const int i = i0 + (tid >> 4), part = tid & 15;
  const int ki = i < n ? key_of(i) : 0;
  int rank = 0;
  for (int j0 = 0; j0 < n && i0 < n; j0 += kRankTile) {
    const int cnt = min(kRankTile, n - j0);
    __syncthreads();
    for (int t = tid; t < cnt; t += 1024) keys[t] = key_of(j0 + t);
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
// those that lie farther than the cutoff by their distance along one axis alone.  That bound carries a margin for the
// rounding of the distances it stands for, so the answer is the same bit.
// Where the cutoff is below half of each width, at most one image per axis passes the bound, the nearest; in wider cells (most)
// a pair then takes one distance instead of up to 27.  8 structures of 300-500 atoms, cutoff 6 Angstrom: 21 us with the loop for
// every pair.
__device__ __forceinline__ bool within_cutoff(float xi, float yi, float zi, float xj, float yj, float zj, const Cell& c,
                                              const float* width, float cutoff, float cutoff2, float margin) {
  const float dx = __fsub_rn(xi, xj), dy = __fsub_rn(yi, yj), dz = __fsub_rn(zi, zj);
  const float limit = fmaf(margin, fabsf(dx) + fabsf(dy) + fabsf(dz) + 3.f, cutoff * 1.0001f);
  if (limit < 0.4999f * fminf(fminf(width[0], width[1]), width[2])) {
    const float ox = fminf(fmaxf(-rintf(dx), -1.f), 1.f), oy = fminf(fmaxf(-rintf(dy), -1.f), 1.f), oz = fminf(fmaxf(-rintf(dz), -1.f), 1.f);
    return fabsf(__fadd_rn(dx, ox)) * width[0] <= limit && fabsf(__fadd_rn(dy, oy)) * width[1] <= limit &&
           fabsf(__fadd_rn(dz, oz)) * width[2] <= limit && image_d2(dx, dy, dz, ox, oy, oz, c) <= cutoff2;
  }
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

// One CTA per row tile I; warp r = row of the tile, lane = column of the column tile J.  The active column tiles are
// collected in shared memory and listed at the end.
constexpr int kBlockAtoms = 1024;  // one for every thread of a CTA
__global__ void __launch_bounds__(kBlockAtoms) block_list_kernel(const float* __restrict__ frac, const StructureInfo* __restrict__ info,
                                                          const int32_t* __restrict__ num_atoms, const int32_t* __restrict__ perm,
                                                          int n_max, int tiles, float cutoff, uint32_t* __restrict__ block_mask,
                                                          int32_t* __restrict__ block_count, int32_t* __restrict__ block_cols) {
  extern __shared__ uint32_t active[];  // bit J
  __shared__ float px[kBlockAtoms], py[kBlockAtoms], pz[kBlockAtoms];  // sorted atoms, kBlockAtoms at a time
  const int I = blockIdx.x, b = blockIdx.y;
  const int r = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = min(num_atoms[b], n_max);
  const float* pos = frac + (size_t)b * n_max * 3;
  const int32_t* pb = perm + (size_t)b * n_max;
  const int words = (tiles + 31) / 32;
  for (int t = threadIdx.x; t < words; t += 1024) active[t] = 0u;
  const Cell c = load_cell(info[b].cell);
  const float width[3] = {info[b].width[0], info[b].width[1], info[b].width[2]};
  float sum = 0.f;
#pragma unroll
  for (int t = 0; t < 9; ++t) sum += fabsf(info[b].cell[t]);
  const float margin = 4e-6f * sum, cutoff2 = squared_cutoff(cutoff);
  const int si = 32 * I + r;
  float xi = 0.f, yi = 0.f, zi = 0.f;
  if (si < n) {
    const int ai = pb[si];
    xi = pos[3 * ai], yi = pos[3 * ai + 1], zi = pos[3 * ai + 2];
  }
  uint32_t* mask = block_mask + ((size_t)b * tiles + I) * tiles * 32 + r;
  for (int J = 0; J < tiles; ++J) {
    const int sj = 32 * J + lane, at = sj % kBlockAtoms;
    if (32 * J % kBlockAtoms == 0) {
      __syncthreads();
      const int t = 32 * J + threadIdx.x;
      if (t < n) {
        const int aj = pb[t];
        px[threadIdx.x] = pos[3 * aj], py[threadIdx.x] = pos[3 * aj + 1], pz[threadIdx.x] = pos[3 * aj + 2];
      }
      __syncthreads();
    }
    const float xj = px[at], yj = py[at], zj = pz[at];
    const bool hit = si < n && sj < n && within_cutoff(xi, yi, zi, xj, yj, zj, c, width, cutoff, cutoff2, margin);
    const uint32_t word = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) {
      mask[(size_t)J * 32] = word;
      if (word) atomicOr(&active[J >> 5], 1u << (J & 31));
    }
  }
  __syncthreads();
  if (r == 0) {
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
  block_list_kernel<<<dim3(tiles, batch), 1024, words, s>>>(frac, info, num_atoms, perm, n_max, tiles, (float)cutoff, block_mask,
                                                            block_count, block_cols);
  MF_CHECK_LAUNCH("block_list_kernel");
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
