// The operators' host path in C++: argument checks, allocations, launch and, where there is one, the autograd node.
//
// A call on small tensors is bound by the host.  Through a Python autograd function and ctypes a forward + backward pass of
// simplicial attention on one small molecule took 171 us of which the kernels are 15; the backward node additionally
// competes for the interpreter lock with the thread that waits for it.  A block list (two launches of 17 us together) took 27 us
// that way and takes 20.  These functions serve calls whose operands are
// ready as they are (contiguous, on one device, of the types the kernels take) and return None for every other call, which
// then takes the Python path with its conversions and error messages.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <array>
#include <mutex>

#include "../../include/matterformer_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;
using torch::autograd::Variable;
using OptTensor = std::optional<Tensor>;

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return MF_DTYPE_F32;
    case at::kBFloat16: return MF_DTYPE_BF16;
    case at::kHalf: return MF_DTYPE_F16;
    default: return -1;
  }
}

void check(int rc) {
  if (rc == MF_OK) return;
  char msg[512];
  mf_last_error(msg, sizeof(msg));
  if (rc == MF_ERR_INVALID_ARGUMENT) throw py::value_error(msg);
  throw std::runtime_error(msg);
}

// The status word of the most recent call on kernels that keep one (see simplicial.py).
std::mutex g_status_mutex;
OptTensor g_status;
void remember_status(OptTensor workspace) {
  OptTensor word;
  if (workspace) word = at::narrow_copy(*workspace, 0, 0, 4);
  std::lock_guard<std::mutex> lock(g_status_mutex);
  g_status = std::move(word);
}
OptTensor last_status() {
  std::lock_guard<std::mutex> lock(g_status_mutex);
  return g_status;
}

const float* fptr(const Tensor& t) { return t.defined() && t.numel() ? t.const_data_ptr<float>() : nullptr; }
float* grad_ptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
Tensor bytes(int64_t n, const Tensor& like) { return n ? at::empty({n}, like.options().dtype(at::kByte)) : Tensor(); }

// The workspace that a call asks for.  On tensor-core kernels without a status word it only holds the list of heavy molecules, which
// the caller may not want.
size_t workspace_bytes(const MfSimplicialFwdArgs& a, bool heavy_first) {
  const bool leave_out = !heavy_first && mf_simplicial_fwd_backend(&a) == MF_BACKEND_TCGEN05 && !mf_simplicial_fwd_keeps_status(&a);
  return leave_out ? 0 : mf_simplicial_fwd_workspace_bytes(&a);
}
size_t workspace_bytes(const MfSimplicialBwdArgs& a, bool heavy_first) {
  const bool leave_out = !heavy_first && mf_simplicial_bwd_backend(&a) == MF_BACKEND_TCGEN05 && !mf_simplicial_bwd_keeps_status(&a);
  return leave_out ? 0 : mf_simplicial_bwd_workspace_bytes(&a);
}

// ---------------------------------------------------------------------------------------------------------------------
// 2-simplicial attention
// ---------------------------------------------------------------------------------------------------------------------
// inputs: q k1 v1 k2 v2 | query_valid key_valid pair_valid | u v w gate | al ar agate | ml mr basis   (undefined when absent)
enum { Q, K1, V1, K2, V2, QV, KV, PV, U, V, W, GATE, AL, AR, AG, ML, MR, BASIS, kInputs };

template <typename Args>
void fill_common(Args& a, const std::array<Tensor, kInputs>& t, int precision, int backend) {
  const Tensor& q = t[Q];
  a.batch = q.size(0), a.heads = q.size(1), a.tokens = q.size(2), a.head_dim = q.size(3);
  a.dtype = dtype_code(q), a.precision = precision, a.backend = backend;
  a.q = q.const_data_ptr(), a.k1 = t[K1].const_data_ptr(), a.v1 = t[V1].const_data_ptr(), a.k2 = t[K2].const_data_ptr(),
  a.v2 = t[V2].const_data_ptr();
  a.query_valid = static_cast<const uint8_t*>(t[QV].const_data_ptr());
  a.pair_key_valid = static_cast<const uint8_t*>(t[KV].const_data_ptr());
  a.pair_valid = t[PV].defined() ? static_cast<const uint8_t*>(t[PV].const_data_ptr()) : nullptr;
  a.u = fptr(t[U]), a.v_bias = fptr(t[V]), a.w = fptr(t[W]), a.gate = fptr(t[GATE]);
  a.angle_left = fptr(t[AL]), a.angle_right = fptr(t[AR]), a.angle_gate = fptr(t[AG]);
  a.message_left = fptr(t[ML]), a.message_right = fptr(t[MR]), a.message_basis = fptr(t[BASIS]);
  a.angle_rank = t[AL].defined() ? t[AL].size(4) : 0, a.message_rank = t[ML].defined() ? t[ML].size(4) : 0;
}

struct SimplicialAttention : torch::autograd::Function<SimplicialAttention> {
  static Variable forward(AutogradContext* ctx, const Tensor& q, const Tensor& k1, const Tensor& v1, const Tensor& k2,
                          const Tensor& v2, const Tensor& qv, const Tensor& kv, const OptTensor& pv, const OptTensor& u,
                          const OptTensor& v, const OptTensor& w, const OptTensor& gate, const OptTensor& al, const OptTensor& ar,
                          const OptTensor& ag, const OptTensor& ml, const OptTensor& mr, const OptTensor& basis, int64_t precision,
                          int64_t backend, bool heavy_first) {
    auto or_none = [](const OptTensor& t) { return t ? *t : Tensor(); };
    const std::array<Tensor, kInputs> t = {q, k1, v1, k2, v2, qv, kv, or_none(pv), or_none(u), or_none(v), or_none(w), or_none(gate),
                                           or_none(al), or_none(ar), or_none(ag), or_none(ml), or_none(mr), or_none(basis)};
    const c10::cuda::CUDAGuard guard(q.device());
    MfSimplicialFwdArgs a{};
    fill_common(a, t, precision, backend);
    const Tensor out32 = at::empty(q.sizes(), q.options().dtype(at::kFloat));
    const Tensor lse = at::empty(q.sizes().slice(0, 3), out32.options());
    const Tensor out = q.scalar_type() == at::kFloat ? out32 : at::empty_like(q);
    a.out = out32.data_ptr<float>(), a.lse = lse.data_ptr<float>();
    a.out_cast = out.is_same(out32) ? nullptr : out.data_ptr();
    const Tensor ws = bytes(workspace_bytes(a, heavy_first), q);
    if (ws.defined()) a.workspace = ws.data_ptr(), a.workspace_bytes = ws.numel();
    check(mf_simplicial_fwd(&a, c10::cuda::getCurrentCUDAStream().stream()));
    if (mf_simplicial_fwd_backend(&a) == MF_BACKEND_TCGEN05)
      remember_status(ws.defined() && mf_simplicial_fwd_keeps_status(&a) ? OptTensor(ws) : std::nullopt);
    ctx->saved_data["call"] = precision | backend << 8 | (int64_t)heavy_first << 16;
    tensor_list saved(t.begin(), t.end());
    saved.push_back(out32);
    saved.push_back(lse);
    ctx->save_for_backward(std::move(saved));
    return out;
  }

  static tensor_list backward(AutogradContext* ctx, tensor_list grad_out) {
    const tensor_list saved = ctx->get_saved_variables();
    std::array<Tensor, kInputs> t;
    std::copy(saved.begin(), saved.begin() + kInputs, t.begin());
    const Tensor &q = t[Q], &out32 = saved[kInputs], &lse = saved[kInputs + 1];
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor go = grad_out[0].to(q.scalar_type()).contiguous();
    MfSimplicialBwdArgs a{};
    const int64_t call = ctx->saved_data["call"].toInt();
    fill_common(a, t, call & 255, call >> 8 & 255);
    a.grad_out = go.const_data_ptr(), a.out = out32.const_data_ptr<float>(), a.lse = lse.const_data_ptr<float>();
    tensor_list g(kInputs + 3);  // (one for each argument of forward)
    for (int i = Q; i <= V2; ++i) g[i] = at::empty_like(q);
    a.dq = g[Q].data_ptr(), a.dk1 = g[K1].data_ptr(), a.dv1 = g[V1].data_ptr(), a.dk2 = g[K2].data_ptr(), a.dv2 = g[V2].data_ptr();
    // edges of the node are counted over the tensors that were given
    auto wanted = [&](int i) {
      if (!t[i].defined()) return false;
      size_t edge = 0;
      for (int j = 0; j < i; ++j) edge += t[j].defined();
      return ctx->needs_input_grad(edge);
    };
    Tensor coeff;
    if (t[U].defined() || t[AL].defined() || t[ML].defined()) {
      const bool zeros = mf_simplicial_bwd_needs_zeros(&a) != 0;
      auto make = [&](const Tensor& like) { return zeros ? at::zeros_like(like) : at::empty_like(like); };
      for (int i = U; i <= MR; ++i)
        if (wanted(i)) g[i] = make(t[i]);
      a.du = grad_ptr(g[U]), a.dv_bias = grad_ptr(g[V]), a.dw = grad_ptr(g[W]), a.dgate = grad_ptr(g[GATE]);
      a.dangle_left = grad_ptr(g[AL]), a.dangle_right = grad_ptr(g[AR]), a.dangle_gate = grad_ptr(g[AG]);
      a.dmessage_left = grad_ptr(g[ML]), a.dmessage_right = grad_ptr(g[MR]);
      if (wanted(BASIS)) {
        const std::vector<int64_t> shape = {a.batch, a.heads, a.tokens, a.message_rank};
        coeff = zeros ? at::zeros(shape, lse.options()) : at::empty(shape, lse.options());
        a.message_coeff = coeff.data_ptr<float>();
      }
    }
    const Tensor ws = bytes(workspace_bytes(a, call >> 16), q);
    if (ws.defined()) a.workspace = ws.data_ptr(), a.workspace_bytes = ws.numel();
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    check(mf_simplicial_bwd(&a, stream));
    if (mf_simplicial_bwd_backend(&a) == MF_BACKEND_TCGEN05)
      remember_status(ws.defined() && mf_simplicial_bwd_keeps_status(&a) ? OptTensor(ws) : std::nullopt);
    if (coeff.defined()) {
      g[BASIS] = at::empty_like(t[BASIS]);
      check(mf_simplicial_basis_grad(a.message_coeff, a.grad_out, a.dtype, a.batch, a.heads, a.tokens, a.message_rank, a.head_dim,
                                     g[BASIS].data_ptr<float>(), stream));
    }
    return g;
  }
};

bool ready(const Tensor& t, const Tensor& like, at::ScalarType type, at::IntArrayRef shape) {
  return t.device() == like.device() && t.scalar_type() == type && t.sizes() == shape && t.is_contiguous();
}

std::optional<Tensor> simplicial_attention(const Tensor& q, const Tensor& k1, const Tensor& v1, const Tensor& k2, const Tensor& v2,
                                           const Tensor& qv, const Tensor& kv, const OptTensor& pv, std::vector<OptTensor> bias,
                                           std::vector<OptTensor> angle, std::vector<OptTensor> message, int64_t precision,
                                           int64_t backend, int64_t max_rank, bool heavy_first) {
  if (!q.is_cuda() || q.dim() != 4 || dtype_code(q) < 0 || !q.is_contiguous()) return std::nullopt;
  for (const Tensor* t : {&k1, &v1, &k2, &v2})
    if (!ready(*t, q, q.scalar_type(), q.sizes())) return std::nullopt;
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
  if (!ready(qv, q, at::kBool, {B, N}) || !ready(kv, q, at::kBool, {B, N})) return std::nullopt;
  if (pv && !ready(*pv, q, at::kBool, {B, N, N})) return std::nullopt;
  auto complete = [](const std::vector<OptTensor>& g, size_t n) {
    if (g.size() != n) return false;
    for (const OptTensor& t : g)
      if (!t || !t->defined()) return false;
    return true;
  };
  if (!bias.empty()) {
    if (!complete(bias, 4)) return std::nullopt;
    for (int i = 0; i < 3; ++i)
      if (!ready(*bias[i], q, at::kFloat, {B, H, N, N})) return std::nullopt;
    if (!ready(*bias[3], q, at::kFloat, {B, H, N})) return std::nullopt;
  }
  if (!angle.empty()) {
    if (!complete(angle, 3) || angle[0]->dim() != 5) return std::nullopt;
    const int64_t R = angle[0]->size(4);
    if (R < 1 || R > max_rank || !ready(*angle[0], q, at::kFloat, {B, H, N, N, R}) || !ready(*angle[1], q, at::kFloat, {B, H, N, N, R}) ||
        !ready(*angle[2], q, at::kFloat, {B, H, N}))
      return std::nullopt;
  }
  if (!message.empty()) {
    if (!complete(message, 3) || message[0]->dim() != 5) return std::nullopt;
    const int64_t R = message[0]->size(4);
    if (R < 1 || R > max_rank || !ready(*message[0], q, at::kFloat, {B, H, N, N, R}) ||
        !ready(*message[1], q, at::kFloat, {B, H, N, N, R}) || !ready(*message[2], q, at::kFloat, {H, R, D}))
      return std::nullopt;
  }
  bias.resize(4), angle.resize(3), message.resize(3);
  return SimplicialAttention::apply(q, k1, v1, k2, v2, qv, kv, pv, bias[0], bias[1], bias[2], bias[3], angle[0], angle[1], angle[2],
                                    message[0], message[1], message[2], precision, backend, heavy_first);
}

// ---------------------------------------------------------------------------------------------------------------------
// Radius block-sparse and local-window attention
// ---------------------------------------------------------------------------------------------------------------------
struct SparseAttention : torch::autograd::Function<SparseAttention> {
  static void fill(MfSparseAttnArgs& a, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& n, const Tensor& count,
                   const Tensor& cols, const Tensor& mask, int64_t window, double scale, int64_t backend) {
    a.batch = q.size(0), a.heads = q.size(1), a.tokens = q.size(2), a.head_dim = q.size(3);
    a.dtype = dtype_code(q), a.window = window, a.scale = scale, a.backend = a.dtype == MF_DTYPE_BF16 ? backend : 0;
    a.q = q.const_data_ptr(), a.k = k.const_data_ptr(), a.v = v.const_data_ptr();
    a.num_atoms = n.const_data_ptr<int32_t>();
    if (window == 0) {
      a.block_count = count.const_data_ptr<int32_t>(), a.block_cols = cols.const_data_ptr<int32_t>();
      a.block_mask = reinterpret_cast<const uint32_t*>(mask.const_data_ptr<int32_t>());
    }
  }

  static Variable forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& n, const Tensor& count,
                          const Tensor& cols, const Tensor& mask, int64_t window, double scale, int64_t backend) {
    const c10::cuda::CUDAGuard guard(q.device());
    MfSparseAttnArgs a{};
    fill(a, q, k, v, n, count, cols, mask, window, scale, backend);
    const Tensor out = at::empty_like(q), lse = at::empty(q.sizes().slice(0, 3), q.options().dtype(at::kFloat));
    a.out = out.data_ptr(), a.lse = lse.data_ptr<float>();
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    check(window ? mf_local_attn_fwd(&a, stream) : mf_radius_attn_fwd(&a, stream));
    ctx->saved_data["window"] = window;
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["backend"] = backend;
    ctx->save_for_backward({q, k, v, n, count, cols, mask, out, lse});
    return out;
  }

  static tensor_list backward(AutogradContext* ctx, tensor_list grad_out) {
    const tensor_list s = ctx->get_saved_variables();
    const Tensor& q = s[0];
    const c10::cuda::CUDAGuard guard(q.device());
    const int64_t window = ctx->saved_data["window"].toInt();
    MfSparseAttnArgs a{};
    fill(a, q, s[1], s[2], s[3], s[4], s[5], s[6], window, ctx->saved_data["scale"].toDouble(), ctx->saved_data["backend"].toInt());
    const Tensor go = grad_out[0].to(q.scalar_type()).contiguous();
    a.out = s[7].data_ptr(), a.lse = s[8].data_ptr<float>(), a.grad_out = go.const_data_ptr();
    tensor_list g(10);
    for (int i = 0; i < 3; ++i) g[i] = at::empty_like(q);
    a.dq = g[0].data_ptr(), a.dk = g[1].data_ptr(), a.dv = g[2].data_ptr();
    const Tensor ws = bytes(mf_sparse_attn_bwd_workspace_bytes(&a), q);
    if (ws.defined()) a.workspace = ws.data_ptr(), a.workspace_bytes = ws.numel();
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    check(window ? mf_local_attn_bwd(&a, stream) : mf_radius_attn_bwd(&a, stream));
    return g;
  }
};

// window 0: the block list; otherwise the band.  `n` (B) int32; the caller has checked shapes and types of q, k, v.
std::optional<Tensor> sparse_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& n, const Tensor& count,
                                       const Tensor& cols, const Tensor& mask, int64_t window, double scale, int64_t backend) {
  for (const Tensor* t : {&q, &k, &v})
    if (!ready(*t, q, q.scalar_type(), q.sizes())) return std::nullopt;
  if (!ready(n, q, at::kInt, {q.size(0)})) return std::nullopt;
  if (window == 0)
    for (const Tensor* t : {&count, &cols, &mask})
      if (t->device() != q.device() || t->scalar_type() != at::kInt || !t->is_contiguous()) return std::nullopt;
  return SparseAttention::apply(q, k, v, n, count, cols, mask, window, scale, backend);
}

// ---------------------------------------------------------------------------------------------------------------------
// Neighbour lists and block lists
// ---------------------------------------------------------------------------------------------------------------------
// Positions (B, N, 3), latents (B, 6) or cells (B, 3, 3) and, if given, counts of the types and on the device that the kernels take.
bool structures_ready(const Tensor& pos, const Tensor& lattice, const OptTensor& n) {
  if (!pos.is_cuda() || pos.dim() != 3 || pos.size(2) != 3 || pos.numel() == 0 || !ready(pos, pos, at::kFloat, pos.sizes())) return false;
  const int64_t B = pos.size(0);
  if (!ready(lattice, pos, at::kFloat, {B, 6}) && !ready(lattice, pos, at::kFloat, {B, 3, 3})) return false;
  return !n || (n->numel() == B && ready(*n, pos, at::kInt, n->sizes()));
}
Tensor counts(const OptTensor& n, const Tensor& pos, const at::TensorOptions& ints) {
  return n ? *n : at::full({pos.size(0)}, pos.size(1), ints);
}

// perm, block_count, block_cols, block_mask, num_atoms
std::optional<std::array<Tensor, 5>> radius_blocks(const Tensor& pos, const Tensor& lattice, const OptTensor& num_atoms, double cutoff) {
  if (!structures_ready(pos, lattice, num_atoms)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(pos.device());
  const int64_t B = pos.size(0), N = pos.size(1), T = (N + 31) / 32;
  const auto ints = at::TensorOptions(pos.device()).dtype(at::kInt);
  const Tensor n = counts(num_atoms, pos, ints);
  const Tensor perm = at::empty({B, N}, ints), count = at::empty({B, T}, ints), cols = at::empty({B, T, T}, ints);
  const Tensor mask = at::empty({B, T, T, 32}, ints), ws = bytes(mf_radius_blocks_workspace_bytes(B, N), pos);
  check(mf_radius_blocks(pos.const_data_ptr<float>(), lattice.const_data_ptr<float>(), lattice.dim() == 3, n.const_data_ptr<int32_t>(), B, N,
                         cutoff, perm.data_ptr<int32_t>(), count.data_ptr<int32_t>(), cols.data_ptr<int32_t>(),
                         reinterpret_cast<uint32_t*>(mask.data_ptr<int32_t>()), ws.data_ptr(), ws.numel(),
                         c10::cuda::getCurrentCUDAStream().stream()));
  return std::array<Tensor, 5>{perm, count, cols, mask, n};
}

std::optional<std::array<Tensor, 2>> knn_topk(const Tensor& pos, const Tensor& lattice, const OptTensor& num_atoms, int64_t k,
                                              bool include_self) {
  if (k < 1 || k > 32 || !structures_ready(pos, lattice, num_atoms)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(pos.device());
  const int64_t B = pos.size(0), N = pos.size(1);
  const auto ints = at::TensorOptions(pos.device()).dtype(at::kInt);
  const Tensor n = counts(num_atoms, pos, ints);
  const Tensor idx = at::empty({B, N, k}, ints), d2 = at::empty({B, N, k}, ints.dtype(at::kFloat));
  const Tensor ws = bytes(mf_knn_cells_workspace_bytes(B, N), pos);
  check(mf_knn_topk_lattice(pos.const_data_ptr<float>(), lattice.const_data_ptr<float>(), lattice.dim() == 3, n.const_data_ptr<int32_t>(), B,
                            N, k, include_self, idx.data_ptr<int32_t>(), d2.data_ptr<float>(), ws.data_ptr(), ws.numel(),
                            c10::cuda::getCurrentCUDAStream().stream()));
  return std::array<Tensor, 2>{idx, d2};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("simplicial_attention", &simplicial_attention);
  m.def("sparse_attention", &sparse_attention);
  m.def("radius_blocks", &radius_blocks);
  m.def("knn_topk", &knn_topk);
  m.def("remember_status", &remember_status);
  m.def("last_status", &last_status);
}
