// C-ABI entry points for 2-simplicial attention plus the error plumbing shared
// by every entry point of the library.
#include <stdarg.h>
#include <string.h>

#include "common.cuh"
#include "tensor_map.cuh"
#include "simplicial.cuh"
#include "simplicial_rows.cuh"

namespace mf {

static thread_local char g_error[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

int cuda_error(cudaError_t err, const char* what) {
  set_error("%s: CUDA error %d (%s)", what, (int)err, cudaGetErrorString(err));
  return MF_ERR_CUDA;
}

namespace {

template <typename Args>
int check_common(const Args* a, const char* name) {
  MF_CHECK_ARG(a != nullptr, "%s: null argument struct", name);
  MF_CHECK_ARG(a->batch >= 0 && a->heads >= 0 && a->tokens >= 0 && a->head_dim > 0, "%s: negative size", name);
  MF_CHECK_ARG(a->head_dim <= 128, "%s: only supports head_dim <= 128, got %d", name, (int)a->head_dim);
  MF_CHECK_ARG(a->dtype == MF_DTYPE_F32 || a->dtype == MF_DTYPE_BF16 || a->dtype == MF_DTYPE_F16,
               "%s: only supports float16/bfloat16/float32 inputs, got dtype code %d", name, (int)a->dtype);
  MF_CHECK_ARG(a->precision >= MF_PRECISION_BF16_TC && a->precision <= MF_PRECISION_IEEE_FP32,
               "%s: unknown precision code %d", name, (int)a->precision);
  MF_CHECK_ARG(a->backend >= MF_BACKEND_AUTO && a->backend <= MF_BACKEND_TCGEN05_TILES, "%s: unknown backend code %d",
               name, (int)a->backend);
  if (a->batch == 0 || a->heads == 0 || a->tokens == 0) return MF_OK;  // nothing to read or write
  MF_CHECK_ARG(a->q && a->k1 && a->v1 && a->k2 && a->v2, "%s: null q/k/v pointer", name);
  MF_CHECK_ARG(a->query_valid && a->pair_key_valid, "%s: null mask pointer", name);
  MF_CHECK_ARG((long long)a->batch * a->heads <= 65535, "%s: batch*heads above 65535", name);
  return MF_OK;
}

// The factorized bias comes as four tensors or not at all.
template <typename Args>
int check_bias(const Args* a, const char* name) {
  const int n = (a->u != nullptr) + (a->v_bias != nullptr) + (a->w != nullptr) + (a->gate != nullptr);
  MF_CHECK_ARG(n == 0 || n == 4, "%s: u, v_bias, w and gate must be given together (got %d of 4)", name, n);
  const int na = (a->angle_left != nullptr) + (a->angle_right != nullptr) + (a->angle_gate != nullptr);
  MF_CHECK_ARG(na == 0 || na == 3, "%s: angle_left, angle_right and angle_gate must be given together", name);
  const int nm = (a->message_left != nullptr) + (a->message_right != nullptr) + (a->message_basis != nullptr);
  MF_CHECK_ARG(nm == 0 || nm == 3, "%s: message_left, message_right and message_basis must be given together", name);
  if ((na && (a->angle_rank < 1 || a->angle_rank > 32)) || (nm && (a->message_rank < 1 || a->message_rank > 32))) {
    set_error("%s: residual ranks must be in [1, 32] (angle %d, message %d)", name, (int)a->angle_rank,
              (int)a->message_rank);
    return MF_ERR_UNSUPPORTED;
  }
  return MF_OK;
}

inline bool vectors_aligned(const MfSimplicialFwdArgs* a) {
  return aligned16(a->q) && aligned16(a->k1) && aligned16(a->v1) && aligned16(a->k2) && aligned16(a->v2) &&
         aligned16(a->out) && aligned16(a->out_cast) && aligned16(a->message_basis);
}
inline bool vectors_aligned(const MfSimplicialBwdArgs* a) {
  return aligned16(a->q) && aligned16(a->k1) && aligned16(a->v1) && aligned16(a->k2) && aligned16(a->v2) &&
         aligned16(a->grad_out) && aligned16(a->out) && aligned16(a->dq) && aligned16(a->dk1) && aligned16(a->dv1) &&
         aligned16(a->dk2) && aligned16(a->dv2) && aligned16(a->message_basis);
}

template <typename Args>
bool has_factorized_bias(const Args* a) {
  return a->u || a->v_bias || a->w || a->gate;
}

template <typename Args>
bool wants_tcgen05(const Args* a, int* rc, const char* name) {
  *rc = MF_OK;
  // The factorized bias is built into the warp-level kernels, not into the row-packed ones; the low-rank residuals into the
  // warp-level ones of at most 32 tokens, else they run on the CUDA-core kernel.
  const bool has_residual = a->angle_left || a->message_left;
  const bool bias_ok = (!has_residual || (a->backend == MF_BACKEND_AUTO && a->tokens <= kSmallTokens)) &&
                       (!has_factorized_bias(a) || a->backend != MF_BACKEND_TCGEN05);
  // the tensor-core kernels move rows with 16-byte vector accesses; tensors that do not start on a 16-byte boundary
  // (a view into the middle of another tensor) go to the CUDA-core kernel, which loads element by element
  const bool ok = bias_ok && simplicial_sm100_supports(a->dtype, a->precision, a->tokens, a->head_dim) &&
                  vectors_aligned(a);
  if (a->backend == MF_BACKEND_GENERIC) return false;
  if ((a->backend == MF_BACKEND_TCGEN05 || a->backend == MF_BACKEND_TCGEN05_TILES) && !ok) {
    set_error("%s: the tcgen05 kernels need bf16 inputs with precision bf16_tc, head_dim 64, tokens <= 192, tensors "
              "that start on 16-byte boundaries and no residual operands; the factorized bias does not run on the "
              "row-packed ones", name);
    *rc = MF_ERR_UNSUPPORTED;
    return false;
  }
  return ok;
}

// Molecules of at most 32 tokens run on the warp-level kernels, with and without the factorized bias.
template <typename Args>
bool uses_small_kernels(const Args* a) {
  return (a->backend == MF_BACKEND_AUTO || a->backend == MF_BACKEND_TCGEN05_TILES) && a->tokens <= kSmallTokens;
}

// Larger molecules with the factorized bias: the backward pass runs on the trilinear tcgen05 kernels (simplicial_tri.cu has both sides'
// times; 1.5 to 4 times as fast from one molecule on).
template <typename Args>
bool uses_tri_kernels(const Args* a) {
  return a->tokens > kSmallTokens && has_factorized_bias(a);
}
// The forward pass runs on them where a call is long enough.  A tile walks all first keys of its rows whatever the batch, up to 100
// tokens in at most 32 steps, from 101 on in up to 64 (tri_plan); the warp-level kernel spreads the queries of a small batch over
// the chip.  The host does not know how full the batch is, so the lines lie between the two extremes.  8 heads, us, trilinear |
// warp-level, all molecules full | spread, up to 96 tokens from an eighth of the tokens up, above from a third: 64 tokens x 4 molecules
// 53 | 32, 53 | 17; x 16 54 | 77, 54 | 43; x 32 98 | 136, 57 | 92.  96 x 4 54 | 60, 54 | 31; x 12 99 | 150, 60 | 87.  128 x 1 144 | 50; x 4
// 146 | 145, 142 | 82; x 8 148 | 252, 144 | 156.  192 x 1 144 | 106; x 2 146 | 207, 144 | 122.  (Above 100 tokens the line, from nine
// molecules of 128 or three of 192 on, dates from longer tiles, of up to 128 steps; it is kept, because moving it changes which rounding a
// call gets.)  On either side a molecule's result does not depend on its batch; the two sides round differently, with the same error.
// MF_BACKEND_TCGEN05_TILES stays on one side.
inline bool uses_tri_forward(const MfSimplicialFwdArgs* a) {
  if (!uses_tri_kernels(a)) return false;
  const double heads = (double)a->batch * a->heads, n = a->tokens;
  return a->backend == MF_BACKEND_TCGEN05_TILES || (n <= 100 ? heads * n >= 6144 : heads * n * n * n >= 150e6);
}
// Without the bias the forward pass runs on the warp-level kernel, unless a tcgen05 family is asked for: 64 molecules of 20-181 atoms
// take 0.64 ms on the trilinear kernel against 0.89, but 2 molecules 201 us against 105, and a molecule's result is to be the same in
// every batch; the backward pass runs on the row-packed kernel (1.98 against 2.26 ms).
inline bool uses_warp_forward(const MfSimplicialFwdArgs* a) {
  return a->tokens > kSmallTokens && (a->backend == MF_BACKEND_AUTO || has_factorized_bias(a));
}

// fp32 molecules of at most 64 tokens (two keys per lane would not fit the registers), plain attention, aligned rows.
template <typename Args>
bool uses_f32_kernels(const Args* a) {
  return a->backend == MF_BACKEND_AUTO && a->dtype == MF_DTYPE_F32 && a->tokens <= 64 && (a->head_dim == 32 || a->head_dim == 64) &&
         !has_factorized_bias(a) && !a->angle_left && !a->message_left && vectors_aligned(a);
}

}  // namespace
}  // namespace mf

using namespace mf;

extern "C" size_t mf_last_error(char* buf, size_t buf_len) {
  const size_t n = strlen(g_error);
  if (buf && buf_len > 0) {
    const size_t c = n < buf_len - 1 ? n : buf_len - 1;
    memcpy(buf, g_error, c);
    buf[c] = '\0';
  }
  return n;
}

extern "C" int mf_version(void) { return 100; }

extern "C" int mf_feature_flags(void) { return tensor_maps_available() ? MF_FEATURE_TENSOR_MAPS : 0; }

extern "C" size_t mf_simplicial_fwd_workspace_bytes(const MfSimplicialFwdArgs* a) {
  if (!a) return 0;
  int rc;
  if (!wants_tcgen05(a, &rc, "mf_simplicial_fwd")) return 0;
  if (uses_small_kernels(a)) return simplicial_small_order_bytes(a->batch, a->heads, false, a->angle_left || a->message_left);
  return uses_tri_forward(a)    ? simplicial_tri_fwd_workspace_bytes(*a)
         : uses_warp_forward(a) ? simplicial_warp_order_bytes(*a)
                                : simplicial_sm100_fwd_workspace_bytes(*a);
}

extern "C" size_t mf_simplicial_bwd_workspace_bytes(const MfSimplicialBwdArgs* a) {
  if (!a) return 0;
  int rc;
  if (wants_tcgen05(a, &rc, "mf_simplicial_bwd"))
    return uses_small_kernels(a)   ? simplicial_small_order_bytes(a->batch, a->heads, true, a->angle_left || a->message_left)
           : uses_tri_kernels(a)   ? simplicial_tri_bwd_workspace_bytes(*a)
           : a->backend == MF_BACKEND_TCGEN05_TILES ? simplicial_sm100_bwd_workspace_bytes(*a) : simplicial_rows_bwd_workspace_bytes(*a);
  return uses_f32_kernels(a) ? 0 : simplicial_generic_bwd_workspace_bytes(*a);
}

extern "C" int mf_simplicial_fwd_backend(const MfSimplicialFwdArgs* a) {
  if (!a) return MF_BACKEND_GENERIC;
  int rc;
  return wants_tcgen05(a, &rc, "mf_simplicial_fwd_backend") ? MF_BACKEND_TCGEN05 : MF_BACKEND_GENERIC;
}

extern "C" int mf_simplicial_bwd_backend(const MfSimplicialBwdArgs* a) {
  if (!a) return MF_BACKEND_GENERIC;
  int rc;
  return wants_tcgen05(a, &rc, "mf_simplicial_bwd_backend") ? MF_BACKEND_TCGEN05 : MF_BACKEND_GENERIC;
}

// The kernels of at most 32 tokens, the warp-level forward kernel and the CUDA-core kernels have no device-side waits.
extern "C" int mf_simplicial_fwd_keeps_status(const MfSimplicialFwdArgs* a) {
  if (!a) return 0;
  int rc;
  return wants_tcgen05(a, &rc, "mf_simplicial_fwd_keeps_status") && !uses_small_kernels(a) && (uses_tri_forward(a) || !uses_warp_forward(a));
}

extern "C" int mf_simplicial_bwd_keeps_status(const MfSimplicialBwdArgs* a) {
  if (!a) return 0;
  int rc;
  return wants_tcgen05(a, &rc, "mf_simplicial_bwd_keeps_status") && !uses_small_kernels(a);
}

extern "C" int mf_simplicial_bwd_needs_zeros(const MfSimplicialBwdArgs* a) {
  if (!a) return 1;
  int rc;
  return !(wants_tcgen05(a, &rc, "mf_simplicial_bwd_needs_zeros") && uses_small_kernels(a));
}

extern "C" int mf_simplicial_row_plan(int32_t n_queries, int32_t valid_keys, int32_t plan[4]) {
  MF_CHECK_ARG(plan != nullptr, "mf_simplicial_row_plan: null output pointer");
  MF_CHECK_ARG(n_queries >= 0 && valid_keys >= 0, "mf_simplicial_row_plan: negative count");
  const RowPlan rp = plan_rows(n_queries, valid_keys);
  plan[0] = rp.tiles;
  plan[1] = rp.rows_per_tile;
  plan[2] = rp.groups;
  plan[3] = rp.steps;
  return MF_OK;
}

extern "C" int mf_simplicial_fwd(const MfSimplicialFwdArgs* a, void* stream) {
  int rc = check_common(a, "mf_simplicial_fwd");
  if (rc != MF_OK) return rc;
  if (a->batch == 0 || a->heads == 0 || a->tokens == 0) return MF_OK;
  MF_CHECK_ARG(a->out && a->lse, "mf_simplicial_fwd: null output pointer");
  if ((rc = check_bias(a, "mf_simplicial_fwd")) != MF_OK) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool tc = wants_tcgen05(a, &rc, "mf_simplicial_fwd");
  if (rc != MF_OK) return rc;
  const size_t need = mf_simplicial_fwd_workspace_bytes(a);
  const bool scratch = a->workspace && a->workspace_bytes >= need;
  if (need > 0 && !scratch && !uses_small_kernels(a) && !uses_warp_forward(a)) {
    set_error("mf_simplicial_fwd: workspace of %zu bytes needed, %zu given", need, a->workspace_bytes);
    return MF_ERR_WORKSPACE_TOO_SMALL;
  }
  if (!tc) return uses_f32_kernels(a) ? simplicial_f32_fwd(*a, s) : simplicial_generic_fwd(*a, s);
  if (uses_small_kernels(a))
    return a->angle_left || a->message_left ? simplicial_small_res_fwd(*a, s) : simplicial_small_fwd(*a, nullptr, s);
  if (uses_tri_forward(a) && scratch) return simplicial_tri_fwd(*a, s);
  if (uses_warp_forward(a)) return simplicial_warp_fwd(*a, s);  // with the bias: callers that give no workspace
  return a->backend == MF_BACKEND_TCGEN05_TILES ? simplicial_sm100_fwd(*a, s) : simplicial_rows_fwd(*a, s);
}

extern "C" int mf_simplicial_bwd(const MfSimplicialBwdArgs* a, void* stream) {
  int rc = check_common(a, "mf_simplicial_bwd");
  if (rc != MF_OK) return rc;
  if (a->batch == 0 || a->heads == 0 || a->tokens == 0) return MF_OK;
  MF_CHECK_ARG(a->grad_out && a->out && a->lse, "mf_simplicial_bwd: null saved-tensor pointer");
  MF_CHECK_ARG(a->dq && a->dk1 && a->dv1 && a->dk2 && a->dv2, "mf_simplicial_bwd: null gradient pointer");
  if ((rc = check_bias(a, "mf_simplicial_bwd")) != MF_OK) return rc;
  MF_CHECK_ARG(a->u || !(a->du || a->dv_bias || a->dw || a->dgate),
               "mf_simplicial_bwd: bias gradients requested without the bias operands");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool tc = wants_tcgen05(a, &rc, "mf_simplicial_bwd");
  if (rc != MF_OK) return rc;
  const bool rows = tc && !uses_small_kernels(a) && !uses_tri_kernels(a) && a->backend != MF_BACKEND_TCGEN05_TILES;
  const size_t need = rows ? simplicial_rows_bwd_least_bytes(*a) : mf_simplicial_bwd_workspace_bytes(a);
  if (need > 0 && (!a->workspace || a->workspace_bytes < need) && !(tc && uses_small_kernels(a))) {
    set_error("mf_simplicial_bwd: workspace of %zu bytes needed, %zu given", need, a->workspace_bytes);
    return MF_ERR_WORKSPACE_TOO_SMALL;
  }
  if (!tc) return uses_f32_kernels(a) ? simplicial_f32_bwd(*a, s) : simplicial_generic_bwd(*a, s);
  if (uses_small_kernels(a)) return simplicial_small_bwd(*a, nullptr, s);
  if (uses_tri_kernels(a)) return simplicial_tri_bwd(*a, s);
  return rows ? simplicial_rows_bwd(*a, s) : simplicial_sm100_bwd(*a, s);
}

extern "C" int mf_selftest_simplicial_give_up(const MfSimplicialFwdArgs* fwd, const MfSimplicialBwdArgs* bwd, int32_t withheld,
                                              int64_t limit_cycles, void* stream) {
  const char* name = "mf_selftest_simplicial_give_up";
  MF_CHECK_ARG((fwd != nullptr) != (bwd != nullptr), "%s: one of the two argument structs", name);
  MF_CHECK_ARG(limit_cycles >= 1 && limit_cycles <= (1ll << 31), "%s: limit must be in [1, 2^31] clocks", name);
  const BoundedWaits waits{(long long)limit_cycles, withheld};
  auto run = [&](const auto* a, int kinds, size_t need, auto kernels) {
    int rc = check_common(a, name);
    if (rc != MF_OK || (rc = check_bias(a, name)) != MF_OK) return rc;
    const bool served = wants_tcgen05(a, &rc, name) && a->batch > 0 && a->heads > 0 && (uses_tri_kernels(a) || a->backend == MF_BACKEND_TCGEN05);
    MF_CHECK_ARG(served && a->workspace && a->workspace_bytes >= need, "%s: not a call of these kernels, or no workspace", name);
    MF_CHECK_ARG(withheld >= 0 && withheld < kinds, "%s: kind of hand-off %d not in [0, %d)", name, (int)withheld, kinds);
    return kernels(*a, static_cast<cudaStream_t>(stream), waits);
  };
  if (fwd) {
    MF_CHECK_ARG(fwd->out && fwd->lse, "%s: null output pointer", name);
    return has_factorized_bias(fwd) ? run(fwd, 8, simplicial_tri_fwd_workspace_bytes(*fwd), simplicial_tri_fwd)
                                    : run(fwd, 6, simplicial_sm100_fwd_workspace_bytes(*fwd), simplicial_rows_fwd);
  }
  MF_CHECK_ARG(bwd->grad_out && bwd->out && bwd->lse && bwd->dq && bwd->dk1 && bwd->dv1 && bwd->dk2 && bwd->dv2, "%s: null pointer", name);
  MF_CHECK_ARG(has_factorized_bias(bwd), "%s: a backward call needs the bias", name);
  return run(bwd, 8, simplicial_tri_bwd_workspace_bytes(*bwd), simplicial_tri_bwd);
}

// ---------------------------------------------------------------------------
// kernel timing aid
// ---------------------------------------------------------------------------
#include <vector>

#include <atomic>
#include <mutex>

namespace mf {
namespace {
std::atomic<bool> g_profile_on{false};
std::mutex g_profile_mutex;                    // guards the event lists
std::vector<cudaEvent_t> g_profile_events[2];  // begin, end, begin, end, ...
}  // namespace

void profile_mark(int which, bool begin, cudaStream_t stream) {
  if (!g_profile_on.load(std::memory_order_relaxed) || which < 0 || which > 1) return;
  std::lock_guard<std::mutex> lock(g_profile_mutex);
  std::vector<cudaEvent_t>& ev = g_profile_events[which];
  if (begin != (ev.size() % 2 == 0)) return;  // unpaired call: ignore
  cudaEvent_t e;
  if (cudaEventCreate(&e) != cudaSuccess) return;
  cudaEventRecord(e, stream);
  ev.push_back(e);
}
}  // namespace mf

extern "C" int mf_profile_enable(int32_t on) {
  g_profile_on.store(on != 0);
  return MF_OK;
}

extern "C" int mf_profile_read(int32_t which, double* total_ms, int32_t* launches) {
  MF_CHECK_ARG(which == MF_PROFILE_SIMPLICIAL_FWD || which == MF_PROFILE_SIMPLICIAL_BWD,
               "mf_profile_read: unknown kernel id %d", (int)which);
  MF_CHECK_ARG(total_ms && launches, "mf_profile_read: null output pointer");
  std::lock_guard<std::mutex> lock(g_profile_mutex);
  std::vector<cudaEvent_t>& ev = g_profile_events[which];
  double total = 0.0;
  int n = 0;
  for (size_t i = 0; i + 1 < ev.size(); i += 2) {
    cudaError_t e = cudaEventSynchronize(ev[i + 1]);
    if (e != cudaSuccess) return cuda_error(e, "mf_profile_read");
    float ms = 0.f;
    e = cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
    if (e != cudaSuccess) return cuda_error(e, "mf_profile_read");
    total += ms;
    ++n;
  }
  for (cudaEvent_t e : ev) cudaEventDestroy(e);
  ev.clear();
  *total_ms = total;
  *launches = n;
  return MF_OK;
}
