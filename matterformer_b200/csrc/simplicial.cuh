// Internal interfaces between the C-ABI layer and the simplicial-attention kernels.
#pragma once

#include <cuda_runtime.h>

#include "../../include/matterformer_b200.h"
#include "common.cuh"

namespace mf {

// fp32 CUDA-core kernels (simplicial_generic.cu)
int simplicial_generic_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream);
int simplicial_generic_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream);
size_t simplicial_generic_bwd_workspace_bytes(const MfSimplicialBwdArgs& a);

// fp32 CUDA-core kernels for small molecules without geometry operands (simplicial_f32.cu)
int simplicial_f32_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream);
int simplicial_f32_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream);

// tcgen05 tensor-core kernels (simplicial_sm100.cu)
bool simplicial_sm100_supports(int dtype, int precision, int tokens, int head_dim);
int simplicial_sm100_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream);
int simplicial_sm100_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream);
size_t simplicial_sm100_fwd_workspace_bytes(const MfSimplicialFwdArgs& a);
size_t simplicial_sm100_bwd_workspace_bytes(const MfSimplicialBwdArgs& a);

// warp-level kernels for molecules of at most 32 tokens (simplicial_small_fwd.cu, simplicial_small_res_fwd.cu, simplicial_small_bwd.cu);
// rows that are not (B,H,N,D) contiguous by `layouts` (NULL = contiguous), see RowLayout
struct TileLayouts;
constexpr int kSmallTokens = 32;
int simplicial_small_fwd(const MfSimplicialFwdArgs& a, const TileLayouts* layouts, cudaStream_t stream);
int simplicial_small_bwd(const MfSimplicialBwdArgs& a, const TileLayouts* layouts, cudaStream_t stream);
int simplicial_small_res_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream);  // with the low-rank residuals
// Workspace with which a call of them takes heavy molecules first (0 where that does not pay), and the list; all of it is optional
size_t simplicial_small_order_bytes(int batch, int heads, bool backward, bool residual);
int simplicial_small_order(const uint8_t* key_valid, int batch, int tokens, void* workspace, size_t workspace_bytes, size_t need,
                           const int32_t** order, cudaStream_t stream);

// warp-level forward kernel for 33 to 192 tokens (simplicial_warp_fwd.cu)
int simplicial_warp_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream);
size_t simplicial_warp_order_bytes(const MfSimplicialFwdArgs& a);  // 0 with the bias; optional

// trilinear tcgen05 kernels for 33 to 192 tokens with the factorized bias (simplicial_tri.cu)
int simplicial_tri_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream, BoundedWaits waits = {});
int simplicial_tri_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream, BoundedWaits waits = {});
size_t simplicial_tri_fwd_workspace_bytes(const MfSimplicialFwdArgs& a);
size_t simplicial_tri_bwd_workspace_bytes(const MfSimplicialBwdArgs& a);

// row-packed tcgen05 kernels (simplicial_rows_fwd.cu, simplicial_rows_bwd.cu); same problems as the kernels above
int simplicial_rows_fwd(const MfSimplicialFwdArgs& a, cudaStream_t stream, BoundedWaits waits = {});
int simplicial_rows_bwd(const MfSimplicialBwdArgs& a, cudaStream_t stream);
size_t simplicial_rows_bwd_workspace_bytes(const MfSimplicialBwdArgs& a);
size_t simplicial_rows_bwd_least_bytes(const MfSimplicialBwdArgs& a);  // with less the call is refused

}  // namespace mf
