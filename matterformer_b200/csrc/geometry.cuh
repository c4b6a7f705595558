// Device functions shared by the periodic-geometry kernels: the fixed-order minimum-image distance and
// the grid cell of a fractional coordinate.  One definition, so every kernel (and the CPU oracle that
// repeats it operation for operation) produces the same bits.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace mf {

struct Cell {
  float l00, l10, l11, l20, l21, l22;
};

__device__ __forceinline__ Cell load_cell(const float* cell) {
  Cell c;
  c.l00 = cell[0];
  c.l10 = cell[3];
  c.l11 = cell[4];
  c.l20 = cell[6];
  c.l21 = cell[7];
  c.l22 = cell[8];
  return c;
}

// Squared minimum-image distance; see the formula in include/matterformer_b200.h.
// Explicit round-to-nearest intrinsics: the compiler may neither fuse nor reorder them.
__device__ __forceinline__ float min_image_d2(float xi, float yi, float zi, float xj, float yj, float zj,
                                              const Cell& c) {
  const float dx = __fsub_rn(xi, xj), dy = __fsub_rn(yi, yj), dz = __fsub_rn(zi, zj);
  float best = INFINITY;
#pragma unroll
  for (int ox = -1; ox <= 1; ++ox) {
    const float ax = __fadd_rn(dx, (float)ox);
    const float rx0 = __fmul_rn(ax, c.l00);
#pragma unroll
    for (int oy = -1; oy <= 1; ++oy) {
      const float ay = __fadd_rn(dy, (float)oy);
      const float rx1 = __fmaf_rn(ay, c.l10, rx0);
      const float ry0 = __fmul_rn(ay, c.l11);
#pragma unroll
      for (int oz = -1; oz <= 1; ++oz) {
        const float az = __fadd_rn(dz, (float)oz);
        const float rx = __fmaf_rn(az, c.l20, rx1);
        const float ry = __fmaf_rn(az, c.l21, ry0);
        const float rz = __fmul_rn(az, c.l22);
        const float d2 = __fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmul_rn(rx, rx)));
        if (d2 < best) best = d2;  // strict: the first minimum wins
      }
    }
  }
  return best;
}

// squared length of one image: delta + (ox, oy, oz), same operation sequence as inside min_image_d2
__device__ __forceinline__ float image_d2(float dx, float dy, float dz, float ox, float oy, float oz, const Cell& c) {
  const float ax = __fadd_rn(dx, ox), ay = __fadd_rn(dy, oy), az = __fadd_rn(dz, oz);
  const float rx = __fmaf_rn(az, c.l20, __fmaf_rn(ay, c.l10, __fmul_rn(ax, c.l00)));
  const float ry = __fmaf_rn(az, c.l21, __fmul_rn(ay, c.l11));
  const float rz = __fmul_rn(az, c.l22);
  return __fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmul_rn(rx, rx)));
}

__device__ __forceinline__ int cell_coord(float f, int g) {
  const float w = __fsub_rn(f, floorf(f));  // wrapped to [0,1]
  int c = (int)__fmul_rn(w, (float)g);
  return min(max(c, 0), g - 1);
}

// The lower-triangular cell (nine floats, rows = lattice vectors) of the latent [log a, log b, log c, cos alpha, cos beta,
// cos gamma]: operation for operation what the host-side formula does in fp32 (lattice_latent_to_cell), clamps included.
__device__ __forceinline__ void cell_from_latent(const float* lat, float* cell) {
  auto clamp = [](float x, float lo, float hi) { return x != x ? x : fminf(fmaxf(x, lo), hi); };  // NaN stays NaN
  const float a = expf(clamp(lat[0], -5.f, 5.f)), b = expf(clamp(lat[1], -5.f, 5.f)), c = expf(clamp(lat[2], -5.f, 5.f));
  const float ca = clamp(lat[3], -0.9999f, 0.9999f), cb = clamp(lat[4], -0.9999f, 0.9999f), cg = clamp(lat[5], -0.9999f, 0.9999f);
  const float sg = __fsqrt_rn(clamp(__fsub_rn(1.f, __fmul_rn(cg, cg)), 1e-8f, INFINITY));
  const float c20 = __fmul_rn(c, cb), c21 = __fdiv_rn(__fmul_rn(c, __fsub_rn(ca, __fmul_rn(cb, cg))), sg);
  const float c22 = __fsqrt_rn(__fsub_rn(__fsub_rn(__fmul_rn(c, c), __fmul_rn(c20, c20)), __fmul_rn(c21, c21)));
  cell[0] = a, cell[1] = 0.f, cell[2] = 0.f;
  cell[3] = __fmul_rn(b, cg), cell[4] = __fmul_rn(b, sg), cell[5] = 0.f;
  cell[6] = c20, cell[7] = c21, cell[8] = clamp(c22, 1e-8f, INFINITY);
}

// Volume and the perpendicular width along one axis of a cell, in double precision.
__device__ __forceinline__ double axis_width(const float* c, int axis, double* volume) {
  const double r[3][3] = {{c[0], c[1], c[2]}, {c[3], c[4], c[5]}, {c[6], c[7], c[8]}};
  const double bc[3] = {r[1][1] * r[2][2] - r[1][2] * r[2][1], r[1][2] * r[2][0] - r[1][0] * r[2][2],
                        r[1][0] * r[2][1] - r[1][1] * r[2][0]};
  const double vol = fabs(r[0][0] * bc[0] + r[0][1] * bc[1] + r[0][2] * bc[2]);
  const int u = (axis + 1) % 3, v = (axis + 2) % 3;
  const double x0 = r[u][1] * r[v][2] - r[u][2] * r[v][1], x1 = r[u][2] * r[v][0] - r[u][0] * r[v][2],
               x2 = r[u][0] * r[v][1] - r[u][1] * r[v][0];
  *volume = vol;
  return vol / fmax(sqrt(x0 * x0 + x1 * x1 + x2 * x2), 1e-12);
}

}  // namespace mf
