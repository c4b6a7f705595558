// Element-wise steps of the EDM preconditioner and sampler on padded molecules, one launch each:
//   out = a_b x + c_b (y - z) + k (p - q), zeros on padded rows, with `center` minus its mean over the molecule's real rows
// (recenter_coordinates and the updates around it, tasks/edm.py:34-81, 153-233).  As separate element-wise operations this is
// ten to sixteen launches over a few kilobytes: 25 us on the stream against 2.5 us.  A CTA per molecule; bound by the launch.
#include "common.cuh"

namespace mf {
namespace {

constexpr int kSumThreads = 128;

__device__ __forceinline__ float masked_sum_at(const MfMaskedSumArgs& p, float a, float c, size_t at) {
  float v = __fmul_rn(a, p.x[at]);
  if (p.y) v = __fadd_rn(v, __fmul_rn(c, p.z ? __fsub_rn(p.y[at], p.z[at]) : p.y[at]));
  if (p.p) v = __fadd_rn(v, __fmul_rn(p.k, __fsub_rn(p.p[at], p.q[at])));
  return v;
}

__global__ void __launch_bounds__(kSumThreads) masked_sum_kernel(const __grid_constant__ MfMaskedSumArgs p) {
  wait_for_previous();
  const int b = blockIdx.x, tid = threadIdx.x, N = p.tokens, C = p.channels;
  const float a = p.a ? p.a[b] : p.a_value, c = p.c ? p.c[b] : p.c_value;
  const uint8_t* pad = p.pad + (size_t)b * N;
  const size_t base = (size_t)b * N * C;
  if (!p.center) {
    for (int e = tid; e < N * C; e += kSumThreads) p.out[base + e] = pad[e / C] ? 0.f : masked_sum_at(p, a, c, base + e);
    return;
  }
  // three channels: a thread's rows are tid, tid + 128, ...; sums per thread, warp, CTA in a fixed order
  __shared__ float part[kSumThreads / 32][4];
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  for (int n = tid; n < N; n += kSumThreads)
    if (!pad[n]) {
#pragma unroll
      for (int d = 0; d < 3; ++d) s[d] += masked_sum_at(p, a, c, base + 3 * n + d);
      s[3] += 1.f;
    }
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    s[d] = warp_sum(s[d]);
    if ((tid & 31) == 0) part[tid >> 5][d] = s[d];
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 4; ++d) s[d] = (part[0][d] + part[1][d]) + (part[2][d] + part[3][d]);
  const float count = fmaxf(s[3], 1.f);
  for (int n = tid; n < N; n += kSumThreads)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const size_t at = base + 3 * n + d;
      p.out[at] = pad[n] ? 0.f : masked_sum_at(p, a, c, at) - s[d] / count;
    }
}

}  // namespace
}  // namespace mf

extern "C" int mf_masked_sum(const MfMaskedSumArgs* p, void* stream) {
  using namespace mf;
  MF_CHECK_ARG(p != nullptr, "mf_masked_sum: null argument struct");
  MF_CHECK_ARG(p->batch >= 0 && p->tokens >= 0 && p->channels >= 0, "mf_masked_sum: negative size");
  MF_CHECK_ARG(!p->center || p->channels == 3, "mf_masked_sum: a centred sum has three channels, got %d", (int)p->channels);
  MF_CHECK_ARG((long long)p->tokens * p->channels < (1ll << 31), "mf_masked_sum: molecule too large");
  if (p->batch == 0 || p->tokens == 0 || p->channels == 0) return MF_OK;
  MF_CHECK_ARG(p->x && p->pad && p->out && (!p->p || p->q) && (!p->z || p->y), "mf_masked_sum: null pointer argument");
  launch_dependent(masked_sum_kernel, dim3(p->batch), dim3(kSumThreads), 0, static_cast<cudaStream_t>(stream), *p);
  MF_CHECK_LAUNCH("masked_sum_kernel");
  return MF_OK;
}
