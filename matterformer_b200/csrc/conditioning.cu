// The steps around the trunk that work on a few numbers per molecule: preconditioner factors, noise-level embedding, token
// projection, padding counts, modulation vectors (EDMPreconditioner and QM9EDMModel, tasks/edm.py:34-81, models/qm9.py:509-565,
// TimeEmbedder, models/embeddings.py:9-44, AdaLNBlock, models/transformer.py:228-316).
//
// As element-wise operations they were some sixty launches of an evaluation of the denoiser, 1.0-4 us each over a few kilobytes: a
// sixth of the time of a sampling run of 64 molecules.  All are bound by their launch, the modulations and the gradient of the
// token projection of a large batch by memory.
#include <cuda_bf16.h>

#include "common.cuh"

namespace mf {
namespace {

// c_skip, c_out and c_in of the preconditioner, and the network's noise channel log(sigma) / 4: the operations of the element-wise form
__global__ void edm_scalings_kernel(const float* __restrict__ sigma, int B, float sd, float sd2, float* __restrict__ scalings,
                                    float* __restrict__ noise) {
  wait_for_previous();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const float s = sigma[b], t = __fadd_rn(__fmul_rn(s, s), sd2);
  if (scalings) {
    scalings[b] = __fmul_rn(__frcp_rn(t), sd2);
    scalings[B + b] = __fdiv_rn(__fmul_rn(s, sd), __fsqrt_rn(t));
    scalings[2 * B + b] = __frcp_rn(__fsqrt_rn(t));
  }
  if (noise) noise[b] = 0.25f * logf(s < 1e-8f ? 1e-8f : s);
}

// cos and sin of 2 pi t f for the frequencies f_i = 10000^(-i / half), twice over (the network embeds one noise level for the
// molecule and one for its atoms, and they are the same)
template <typename T>
__global__ void time_embedding_kernel(const float* __restrict__ t, int half, T* __restrict__ out) {
  wait_for_previous();
  const float at = __fmul_rn(6.283185307179586f, t[blockIdx.x]);
  T* row = out + (size_t)blockIdx.x * 4 * half;
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const float arg = __fmul_rn(at, expf(__fmul_rn(__fmul_rn(-9.210340371976184f, (float)i), __fdiv_rn(1.f, (float)half))));
    float s, c;
    sincosf(arg, &s, &c);
    row[i] = row[2 * half + i] = from_f32<T>(c);
    row[half + i] = row[3 * half + i] = from_f32<T>(s);
  }
}

// Real atoms: 1 - pad, and their number per molecule.  A warp per molecule.
__global__ void pad_counts_kernel(const uint8_t* __restrict__ pad, int B, int N, uint8_t* __restrict__ valid, int32_t* __restrict__ counts) {
  wait_for_previous();
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= B) return;
  int n = 0;
  for (int i = lane; i < N; i += 32) {
    const bool real = pad[(size_t)b * N + i] == 0;
    valid[(size_t)b * N + i] = real;
    n += real;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0) counts[b] = n;
}

// Token projection: bf16 rows W x + bias of (features, noise level) in bf16 with fp32 sums, zeros on padded rows.  A thread holds the
// weights of eight channels and walks over rows.  1 856 rows of 512 4.7 us (8.9 with the weights read where they lie and 64-bit
// divisions), 29 696 rows 18 us (62).
constexpr int kMaxTokenInputs = 8;
constexpr int kTokenThreads = 256, kTokenRows = 16;  // rows of a block of a small batch; larger ones make one wave of blocks
__device__ __forceinline__ float as_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__global__ void __launch_bounds__(kTokenThreads) token_projection_kernel(const float* __restrict__ x, const float* __restrict__ noise,
                                                                         const uint8_t* __restrict__ pad, const float* __restrict__ weight,
                                                                         const float* __restrict__ bias, long long rows, int rows_per_block,
                                                                         int N, int K, int C, __nv_bfloat16* __restrict__ out) {
  wait_for_previous();
  __shared__ __align__(16) float ws[kMaxTokenInputs * 1024];  // weights by input: a thread's own lie 8 K floats from its neighbour's in memory
  for (int i = threadIdx.x; i < C * K; i += kTokenThreads) ws[(unsigned)i % (unsigned)K * C + (unsigned)i / (unsigned)K] = as_bf16(weight[i]);
  __syncthreads();
  const int per_row = C >> 3, at_once = kTokenThreads / per_row, group = threadIdx.x / per_row, c = 8 * (threadIdx.x - group * per_row);
  if (group >= at_once) return;
  float w[8][kMaxTokenInputs], b[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) b[e] = as_bf16(bias[c + e]);
#pragma unroll
  for (int k = 0; k < kMaxTokenInputs; ++k) {
    const float4 lo = *reinterpret_cast<const float4*>(&ws[min(k, K - 1) * C + c]), hi = *reinterpret_cast<const float4*>(&ws[min(k, K - 1) * C + c + 4]);
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e][k] = k < K ? v[e] : 0.f;
  }
  const long long r1 = min(rows, (long long)(blockIdx.x + 1) * rows_per_block);
#pragma unroll 2
  for (long long r = (long long)blockIdx.x * rows_per_block + group; r < r1; r += at_once) {
    float v[8];
    const bool hidden = pad[r] != 0;
    float in[kMaxTokenInputs];
    const float level = as_bf16(noise[(unsigned)r / (unsigned)N]);
#pragma unroll
    for (int k = 0; k < kMaxTokenInputs; ++k) {  // (loaded without a condition, here and below: conditional loads are waited for one by one)
      const float* at = K > 1 ? x + r * (K - 1) + min(k, K - 2) : noise + (unsigned)r / (unsigned)N;
      const float v = as_bf16(*at);
      in[k] = k < K - 1 ? v : k == K - 1 ? level : 0.f;
    }
    uint32_t packed[4];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[e] = 0.f;
#pragma unroll
      for (int k = 0; k < kMaxTokenInputs; ++k) v[e] = fmaf(in[k], w[e][k], v[e]);
      v[e] = hidden ? 0.f : v[e] + b[e];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
      packed[e] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(out + r * C + c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  }
}

// Its weight and bias gradients: part[band] = (C, K) sums of dy x, then C sums of dy, over a band of rows; the bands are added in
// order.  A thread holds two channels.  1 024 molecules of 29 tokens: a GEMM with seven columns and a reduction took 76 + 10 us.
constexpr int kTokenChunk = 32;
__global__ void token_projection_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const float* __restrict__ x, const float* __restrict__ noise,
                                            const uint8_t* __restrict__ pad, long long rows, long long rows_per_band, int N, int K, int C,
                                            float* __restrict__ part) {
  __shared__ float in[kTokenChunk][kMaxTokenInputs + 1];
  wait_for_previous();
  const int c = 2 * threadIdx.x;
  float acc[2][kMaxTokenInputs + 1];
#pragma unroll
  for (int k = 0; k <= kMaxTokenInputs; ++k) acc[0][k] = acc[1][k] = 0.f;
  const long long lo = blockIdx.x * rows_per_band, hi = min(rows, lo + rows_per_band);
  for (long long r0 = lo; r0 < hi; r0 += kTokenChunk) {
    uint32_t g[kTokenChunk];  // all rows of the chunk are on their way together
#pragma unroll
    for (int u = 0; u < kTokenChunk; ++u) g[u] = *reinterpret_cast<const uint32_t*>(dy + min(r0 + u, rows - 1) * C + c);
    __syncthreads();
    for (int i = threadIdx.x; i < kTokenChunk * (kMaxTokenInputs + 1); i += blockDim.x) {
      const int k = i % (kMaxTokenInputs + 1);
      const long long r = r0 + i / (kMaxTokenInputs + 1), at = min(r, rows - 1);
      const bool hidden = pad[at] != 0;
      const float level = as_bf16(noise[(unsigned)at / (unsigned)N]), v = K > 1 ? as_bf16(x[at * (K - 1) + min(k, K - 2)]) : 0.f;
      // rows beyond the band and padded ones count for nothing
      in[i / (kMaxTokenInputs + 1)][k] = r >= hi || hidden ? 0.f : k == kMaxTokenInputs ? 1.f : k < K - 1 ? v : k == K - 1 ? level : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTokenChunk; ++u) {
      if (in[u][kMaxTokenInputs] == 0.f) continue;
      const float g0 = __uint_as_float(g[u] << 16), g1 = __uint_as_float(g[u] & 0xffff0000u);
#pragma unroll
      for (int k = 0; k <= kMaxTokenInputs; ++k) {
        acc[0][k] = fmaf(g0, in[u][k], acc[0][k]);
        acc[1][k] = fmaf(g1, in[u][k], acc[1][k]);
      }
    }
  }
  float* mine = part + (size_t)blockIdx.x * C * (K + 1);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
#pragma unroll
    for (int k = 0; k < kMaxTokenInputs; ++k)
      if (k < K) mine[(c + u) * K + k] = acc[u][k];
    mine[C * K + c + u] = acc[u][kMaxTokenInputs];
  }
}

// (B, G C) -> G fp32 matrices (B, C) and back: eight channels a thread.  1 024 molecules, 72 vectors of 512: as a transposing copy
// 130 us, as a concatenation and a cast 83 us.
__device__ __forceinline__ void unpack8(uint4 a, float (&v)[8]) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) v[2 * e] = __uint_as_float(w[e] << 16), v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
}
__global__ void split_modulation_kernel(const __nv_bfloat16* __restrict__ mod, int B, int G, int C, float* __restrict__ out) {
  wait_for_previous();
  const int c = 8 * threadIdx.x, g = blockIdx.x, step = gridDim.y * blockDim.y;
#pragma unroll 4
  for (int b = blockIdx.y * blockDim.y + threadIdx.y; b < B; b += step) {
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(mod + ((size_t)b * G + g) * C + c), v);
    float4* o = reinterpret_cast<float4*>(out + ((size_t)g * B + b) * C + c);
    o[0] = make_float4(v[0], v[1], v[2], v[3]), o[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}
constexpr int kMaxModulations = 128;
struct ModulationGrads {
  const float* g[kMaxModulations];
};
__global__ void merge_modulation_kernel(const __grid_constant__ ModulationGrads in, int B, int G, int C, __nv_bfloat16* __restrict__ out) {
  wait_for_previous();
  const int c = 8 * threadIdx.x, g = blockIdx.x, step = gridDim.y * blockDim.y;
  const float* src = in.g[g];
#pragma unroll 4
  for (int b = blockIdx.y * blockDim.y + threadIdx.y; b < B; b += step) {
    uint4 packed = make_uint4(0u, 0u, 0u, 0u);
    if (src) {
      const float4* p = reinterpret_cast<const float4*>(src + (size_t)b * C + c);
      const float4 x = p[0], y = p[1];
      __nv_bfloat162 h[4] = {__floats2bfloat162_rn(x.x, x.y), __floats2bfloat162_rn(x.z, x.w), __floats2bfloat162_rn(y.x, y.y),
                             __floats2bfloat162_rn(y.z, y.w)};
      packed = *reinterpret_cast<const uint4*>(h);
    }
    *reinterpret_cast<uint4*>(out + ((size_t)b * G + g) * C + c) = packed;
  }
}

int check_token_sizes(const char* name, int batch, int tokens, int inputs, int channels) {
  MF_CHECK_ARG(batch >= 0 && tokens >= 0, "%s: negative size", name);
  MF_CHECK_ARG((long long)batch * tokens < (1ll << 31), "%s: batch * tokens too large", name);
  MF_CHECK_ARG(inputs >= 1 && inputs <= kMaxTokenInputs, "%s: 1 to %d inputs, got %d", name, kMaxTokenInputs, inputs);
  MF_CHECK_ARG(channels >= 64 && channels <= 1024 && channels % 64 == 0, "%s: channels must be a multiple of 64, at most 1024, got %d", name,
               channels);
  return MF_OK;
}
int token_bands(long long rows) { return (int)min((rows + kTokenChunk - 1) / kTokenChunk, (long long)2 * 148); }

int check_modulation_sizes(const char* name, int batch, int groups, int channels) {
  MF_CHECK_ARG(batch >= 0 && groups >= 1 && groups <= kMaxModulations, "%s: 1 to %d vectors, got %d", name, kMaxModulations, groups);
  MF_CHECK_ARG(channels >= 8 && channels <= 4096 && channels % 8 == 0, "%s: channels must be a multiple of 8, at most 4096, got %d", name, channels);
  return MF_OK;
}
// threads: a row's vectors x as many rows as make a block; blocks: a few waves
void modulation_launch(int batch, int groups, int channels, dim3* grid, dim3* block) {
  const int x = channels / 8, y = max(1, 256 / x);
  const int rows = (batch + y - 1) / y;
  *block = dim3(x, y), *grid = dim3(groups, max(1, min(rows, max(1, 8 * 148 / groups))));
}

}  // namespace
}  // namespace mf

using namespace mf;

extern "C" int mf_edm_scalings(const float* sigma, int32_t batch, double sigma_data, float* scalings, float* noise, void* stream) {
  MF_CHECK_ARG(batch >= 0, "mf_edm_scalings: negative size");
  if (batch == 0) return MF_OK;
  MF_CHECK_ARG(sigma, "mf_edm_scalings: null pointer argument");
  launch_dependent(edm_scalings_kernel, dim3((batch + 127) / 128), dim3(128), 0, static_cast<cudaStream_t>(stream), sigma, batch,
                   (float)sigma_data, (float)(sigma_data * sigma_data), scalings, noise);
  MF_CHECK_LAUNCH("edm_scalings_kernel");
  return MF_OK;
}

extern "C" int mf_time_embedding(const float* t, int32_t batch, int32_t half, int32_t dtype, void* out, void* stream) {
  MF_CHECK_ARG(batch >= 0 && half >= 0, "mf_time_embedding: negative size");
  if (batch == 0 || half == 0) return MF_OK;
  MF_CHECK_ARG(t && out, "mf_time_embedding: null pointer argument");
  MF_DISPATCH_DTYPE(dtype, T, launch_dependent(time_embedding_kernel<T>, dim3(batch), dim3(128), 0, static_cast<cudaStream_t>(stream), t, half,
                                               static_cast<T*>(out)));
  MF_CHECK_LAUNCH("time_embedding_kernel");
  return MF_OK;
}

extern "C" int mf_pad_counts(const uint8_t* pad, int32_t batch, int32_t tokens, uint8_t* valid, int32_t* counts, void* stream) {
  MF_CHECK_ARG(batch >= 0 && tokens >= 0, "mf_pad_counts: negative size");
  if (batch == 0) return MF_OK;
  MF_CHECK_ARG(counts && (tokens == 0 || (pad && valid)), "mf_pad_counts: null pointer argument");
  launch_dependent(pad_counts_kernel, dim3((batch + 3) / 4), dim3(128), 0, static_cast<cudaStream_t>(stream), pad, batch, tokens, valid, counts);
  MF_CHECK_LAUNCH("pad_counts_kernel");
  return MF_OK;
}

extern "C" int mf_token_projection_fwd(const float* x, const float* noise, const uint8_t* pad, const float* weight, const float* bias,
                                       int32_t batch, int32_t tokens, int32_t inputs, int32_t channels, void* out, void* stream) {
  const int rc = check_token_sizes("mf_token_projection_fwd", batch, tokens, inputs, channels);
  if (rc != MF_OK) return rc;
  const long long rows = (long long)batch * tokens;
  if (rows == 0) return MF_OK;
  MF_CHECK_ARG((x || inputs == 1) && noise && pad && weight && bias && out, "mf_token_projection_fwd: null pointer argument");
  MF_CHECK_ALIGNED("mf_token_projection_fwd", out);
  const int per_block = (int)max((long long)kTokenRows, (rows + 2 * 148 - 1) / (2 * 148));
  launch_dependent(token_projection_kernel, dim3((unsigned)((rows + per_block - 1) / per_block)), dim3(kTokenThreads), 0,
                   static_cast<cudaStream_t>(stream), x, noise, pad, weight, bias, rows, per_block, tokens, inputs, channels,
                   static_cast<__nv_bfloat16*>(out));
  MF_CHECK_LAUNCH("token_projection_kernel");
  return MF_OK;
}

extern "C" size_t mf_token_projection_bwd_workspace_bytes(int32_t batch, int32_t tokens, int32_t inputs, int32_t channels) {
  if (batch < 0 || tokens < 0 || inputs < 1 || channels < 1) return 0;
  return (size_t)token_bands((long long)batch * tokens) * channels * (inputs + 1) * sizeof(float);
}

extern "C" int mf_token_projection_bwd(const void* dy, const float* x, const float* noise, const uint8_t* pad, int32_t batch, int32_t tokens,
                                       int32_t inputs, int32_t channels, float* grads, void* workspace, size_t workspace_bytes,
                                       void* stream) {
  const int rc = check_token_sizes("mf_token_projection_bwd", batch, tokens, inputs, channels);
  if (rc != MF_OK) return rc;
  MF_CHECK_ARG(grads, "mf_token_projection_bwd: null pointer argument");
  const long long rows = (long long)batch * tokens;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int sums = channels * (inputs + 1);
  if (rows == 0) {
    const cudaError_t e = cudaMemsetAsync(grads, 0, (size_t)sums * sizeof(float), s);
    return e == cudaSuccess ? MF_OK : cuda_error(e, "cudaMemsetAsync(mf_token_projection_bwd)");
  }
  MF_CHECK_ARG(dy && (x || inputs == 1) && noise && pad, "mf_token_projection_bwd: null pointer argument");
  MF_CHECK_ALIGNED("mf_token_projection_bwd", dy);
  const size_t need = mf_token_projection_bwd_workspace_bytes(batch, tokens, inputs, channels);
  if (!workspace || workspace_bytes < need) {
    set_error("mf_token_projection_bwd: workspace too small (%zu bytes needed)", need);
    return MF_ERR_WORKSPACE_TOO_SMALL;
  }
  const int bands = token_bands(rows);
  float* part = static_cast<float*>(workspace);
  launch_dependent(token_projection_bwd_kernel, dim3(bands), dim3(channels / 2), 0, s, static_cast<const __nv_bfloat16*>(dy), x, noise, pad,
                   rows, (rows + bands - 1) / bands, tokens, inputs, channels, part);
  MF_CHECK_LAUNCH("token_projection_bwd_kernel");
  return add_bands(part, bands, sums, grads, s);
}

extern "C" int mf_split_modulation(const void* mod, int32_t batch, int32_t groups, int32_t channels, float* out, void* stream) {
  const int rc = check_modulation_sizes("mf_split_modulation", batch, groups, channels);
  if (rc != MF_OK || batch == 0) return rc;
  MF_CHECK_ARG(mod && out, "mf_split_modulation: null pointer argument");
  MF_CHECK_ALIGNED("mf_split_modulation", mod, out);
  dim3 grid, block;
  modulation_launch(batch, groups, channels, &grid, &block);
  launch_dependent(split_modulation_kernel, grid, block, 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(mod), batch,
                   groups, channels, out);
  MF_CHECK_LAUNCH("split_modulation_kernel");
  return MF_OK;
}

extern "C" int mf_merge_modulation(const float* const* grads, int32_t batch, int32_t groups, int32_t channels, void* out, void* stream) {
  const int rc = check_modulation_sizes("mf_merge_modulation", batch, groups, channels);
  if (rc != MF_OK || batch == 0) return rc;
  MF_CHECK_ARG(grads && out, "mf_merge_modulation: null pointer argument");
  MF_CHECK_ALIGNED("mf_merge_modulation", out);
  ModulationGrads in{};
  for (int i = 0; i < groups; ++i) {
    MF_CHECK_ALIGNED("mf_merge_modulation", grads[i]);
    in.g[i] = grads[i];
  }
  dim3 grid, block;
  modulation_launch(batch, groups, channels, &grid, &block);
  launch_dependent(merge_modulation_kernel, grid, block, 0, static_cast<cudaStream_t>(stream), in, batch, groups, channels,
                   static_cast<__nv_bfloat16*>(out));
  MF_CHECK_LAUNCH("merge_modulation_kernel");
  return MF_OK;
}
