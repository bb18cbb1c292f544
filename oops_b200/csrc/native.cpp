// Host side of the operators: argument checks of the common case, autograd nodes, allocation and launches, in C++.
//
// The Python entry points hand their arguments to this module first.  A call it does not recognise as plain (another
// device, tensor subclasses with their own dispatch, negated or conjugated views, shapes or types that do not fit) is
// declined by returning None, and the Python code beside the entry point handles it or raises the documented error.
// What it saves is host time: a Python autograd function with its ctypes structures cost 75 us per forward call and
// 250 us per forward + reverse call, more than the kernels of calls below about 300 x 300 tokens take.
// The kernels are reached through the C ABI only (include/oops_ta.h); PyTorch provides memory, streams and autograd.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>
#include <optional>
#include <vector>

#include "oops_ta.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using MaybeTensor = std::optional<Tensor>;

PyObject* g_unsupported_error = nullptr;  // OOpsUnsupportedError, set once at import
std::atomic<bool> g_check_status{false};

[[noreturn]] void raise_unsupported(const std::string& message) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(g_unsupported_error ? g_unsupported_error : PyExc_NotImplementedError, message.c_str());
  python_error error;
  error.persist();
  throw error;
}

void check_status(int status, const char* what) {
  if (status == OOPS_TA_OK) return;
  const char* detail = oops_ta_last_error();
  std::string message = std::string(what) + " failed: " + oops_ta_status_string(status);
  if (detail && *detail) message += std::string(": ") + detail;
  TORCH_CHECK_VALUE(status != OOPS_TA_INVALID_ARGUMENT, message);
  TORCH_CHECK(status != OOPS_TA_CUDA_ERROR && status != OOPS_TA_DEVICE_TIMEOUT && status != OOPS_TA_WORKSPACE_TOO_SMALL, message);
  raise_unsupported(message);
}

// Inside `checked_device_status()` every pass ends with a synchronisation and a look at the device-side status word.
void check_device(const char* what) {
  if (!g_check_status.load(std::memory_order_relaxed)) return;
  const int status = oops_ta_device_status(1);
  TORCH_CHECK(status == OOPS_TA_OK, "triangle_attention ", what, ": a kernel recorded device status ", status, " (",
              oops_ta_status_string(status), "); its results are undefined");
}

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? OOPS_TA_F32 : t == at::kHalf ? OOPS_TA_F16 : t == at::kBFloat16 ? OOPS_TA_BF16 : -1;
}

void* current_stream(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor bytes_like(const Tensor& t, uint64_t count) {
  return at::empty({int64_t(count)}, t.options().dtype(at::kByte).requires_grad(false));
}

Tensor floats_like(const Tensor& t, at::IntArrayRef sizes) {
  return at::empty(sizes, t.options().dtype(at::kFloat).requires_grad(false));
}

bool requires_grad(const Tensor& t) { return t.defined() && t.requires_grad(); }
bool requires_grad(const MaybeTensor& t) { return t.has_value() && t->defined() && t->requires_grad(); }

void* data_of(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* data_of(const MaybeTensor& t) { return t.has_value() ? data_of(*t) : nullptr; }

// No dispatch mode, transform or tracer is active that would have to see the operations of a call.
bool plain_context() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !torch::jit::tracer::isTracing() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

bool plain_tensor(const Tensor& t) {
  static const c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::Batched,
                                            c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                            c10::DispatchKey::ZeroTensor, c10::DispatchKey::Negative,
                                            c10::DispatchKey::Conjugate});
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(special);
}

// ---------------------------------------------------------------------------------------------
// triangle attention
// ---------------------------------------------------------------------------------------------

// One uniform problem (the tensors are (B, R, C, H, D) views), or a packed ragged batch: pair tensors (cells, P, H, D),
// masks (cells, P), bias head-major (P, H, values) with a sample's block ordered (group, query, key).  `transposed`:
// the packed cell order is column-major (the ending-node form).
struct Geometry {
  bool packed = false, transposed = false;
  int64_t prefixes = 1;
  std::vector<int64_t> lengths, groups, rows;  // tokens, bias groups and bias row strides of every sample

  static Geometry decode(const std::vector<int64_t>& code) {
    Geometry g;
    if (code.empty()) return g;
    g.packed = true;
    g.prefixes = code[0];
    g.transposed = code[1] != 0;
    const int64_t count = code[2];
    const bool has_bias = code[3] != 0;
    auto at = code.begin() + 4;
    g.lengths.assign(at, at + count);
    if (has_bias) {
      g.groups.assign(at + count, at + 2 * count);
      g.rows.assign(at + 2 * count, at + 3 * count);
    }
    return g;
  }
  std::vector<int64_t> encode() const {
    if (!packed) return {};
    std::vector<int64_t> code{prefixes, transposed, int64_t(lengths.size()), !groups.empty()};
    code.insert(code.end(), lengths.begin(), lengths.end());
    code.insert(code.end(), groups.begin(), groups.end());
    code.insert(code.end(), rows.begin(), rows.end());
    return code;
  }
  size_t count() const { return packed ? lengths.size() : 1; }
  int64_t lse_size(const Tensor& query) const {
    if (!packed) return query.size(0) * query.size(1) * query.size(2) * query.size(3);
    int64_t total = 0;
    for (int64_t n : lengths) total += prefixes * n * n * query.size(2);
    return total;
  }
};

struct Sample {  // where a sample of a geometry starts
  int64_t tokens = 0, cell = 0, bias = 0, lse = 0;
};

oops_ta_pair pair_of(const Geometry& g, const Sample& s, const Tensor& t) {
  if (!t.defined()) return {nullptr, 0, 0, 0, 0};
  char* base = static_cast<char*>(t.data_ptr());
  if (!g.packed) return {base, t.stride(0), t.stride(1), t.stride(2), t.stride(3)};
  const int64_t heads = t.size(2), dim = t.size(3), minor = g.prefixes * heads * dim, major = s.tokens * minor;
  return {base + s.cell * minor * t.element_size(), heads * dim, g.transposed ? minor : major, g.transposed ? major : minor, dim};
}

void describe(oops_ta_problem& p, const Geometry& g, const Sample& s, size_t index, const Tensor& query, const Tensor& key,
              const Tensor& value, const Tensor& mask, const Tensor& bias, double scale, int64_t flags) {
  p.abi_version = OOPS_TA_ABI_VERSION;
  p.flags = uint32_t(flags);
  p.dtype = dtype_code(query.scalar_type());
  p.batch = int32_t(g.packed ? g.prefixes : query.size(0));
  p.rows = int32_t(g.packed ? s.tokens : query.size(1));
  p.cols = int32_t(g.packed ? s.tokens : query.size(2));
  p.heads = int32_t(query.size(-2));
  p.head_dim = int32_t(query.size(-1));
  p.scale = float(scale);
  p.q = pair_of(g, s, query);
  p.k = pair_of(g, s, key);
  p.v = pair_of(g, s, value);
  if (mask.defined()) {
    if (!g.packed) {
      p.mask = static_cast<const uint8_t*>(mask.data_ptr());
      p.mask_sb = mask.stride(0);
      p.mask_sr = mask.stride(1);
      p.mask_sc = mask.stride(2);
    } else {
      p.mask = static_cast<const uint8_t*>(mask.data_ptr()) + s.cell * g.prefixes;
      p.mask_sb = 1;
      p.mask_sr = g.transposed ? g.prefixes : s.tokens * g.prefixes;
      p.mask_sc = g.transposed ? s.tokens * g.prefixes : g.prefixes;
    }
  }
  p.bias_dtype = p.dtype;
  if (bias.defined()) {
    p.bias_dtype = dtype_code(bias.scalar_type());
    if (!g.packed) {
      p.bias_groups = int32_t(bias.size(1));
      p.bias = bias.data_ptr();
      p.bias_sb = bias.stride(0);
      p.bias_sg = bias.stride(1);
      p.bias_sh = bias.stride(2);
      p.bias_sq = bias.stride(3);
      p.bias_sk = bias.stride(4);
    } else {
      const int64_t heads = bias.size(1), total = bias.size(2), row = g.rows[index];
      p.bias_groups = int32_t(g.groups[index]);
      p.bias = static_cast<char*>(bias.data_ptr()) + s.bias * bias.element_size();
      p.bias_sb = heads * total;
      p.bias_sg = s.tokens * row;
      p.bias_sh = total;
      p.bias_sq = row;
      p.bias_sk = 1;
    }
  }
}

// Calls `body(problem, sample, index)` for every sample of the geometry.
template <typename F>
void for_each_sample(const Geometry& g, const Tensor& query, F&& body) {
  Sample s;
  for (size_t i = 0; i < g.count(); ++i) {
    s.tokens = g.packed ? g.lengths[i] : 0;
    body(s, i);
    if (!g.packed) return;
    s.cell += s.tokens * s.tokens;
    s.lse += g.prefixes * s.tokens * s.tokens * query.size(2);
    if (!g.groups.empty()) s.bias += g.groups[i] * s.tokens * g.rows[i];
  }
}

Tensor result_like(const Tensor& t) {
  Tensor out = at::empty_like(t);
  if (out.size(-1) != 1 && out.stride(-1) != 1) out = at::empty(t.sizes(), t.options());
  return out;
}

// `gate` and `plain` are undefined except for the gated form, whose result is the gated tensor; `into` lends the result's memory.
std::tuple<Tensor, Tensor> run_forward(const Geometry& g, const Tensor& query, const Tensor& key, const Tensor& value,
                                       const Tensor& mask, const Tensor& bias, double scale, int64_t flags, bool want_lse,
                                       const Tensor& gate = {}, const Tensor& plain = {}, const Tensor& into = {}) {
  const c10::cuda::CUDAGuard guard(query.device());
  Tensor out = into.defined() ? into : gate.defined() ? at::empty(query.sizes(), query.options()) : result_like(query);
  Tensor lse = want_lse ? floats_like(query, {g.lse_size(query)}) : Tensor();
  void* stream = current_stream(query);
  for_each_sample(g, query, [&](const Sample& s, size_t i) {
    oops_ta_problem problem{};
    describe(problem, g, s, i, query, key, value, mask, bias, scale, flags);
    check_status(oops_ta_supported(&problem), "triangle_attention forward");
    Tensor scratch;
    if (const uint64_t need = oops_ta_forward_workspace_bytes(&problem)) {
      scratch = bytes_like(query, need);
      problem.workspace = scratch.data_ptr();
      problem.workspace_bytes = need;
    }
    const oops_ta_pair out_pair = pair_of(g, s, out);
    float* lse_at = lse.defined() ? lse.data_ptr<float>() + s.lse : nullptr;
    if (gate.defined()) {
      const oops_ta_pair gate_pair = pair_of(g, s, gate), plain_pair = pair_of(g, s, plain);
      check_status(oops_ta_forward_gated(&problem, &gate_pair, &out_pair, &plain_pair, lse_at, stream),
                   "triangle_attention gated forward");
    } else {
      check_status(oops_ta_forward(&problem, &out_pair, lse_at, stream), "triangle_attention forward");
    }
  });
  check_device(gate.defined() ? "gated forward" : "forward");
  return {out, lse};
}

struct Gradients {
  Tensor dq, dk, dv, dbias;
};

// `lent` is an optional caller-owned scratch buffer; `dbias_type` overrides the type of the bias gradient.
Gradients run_backward(const Geometry& g, const Tensor& grad_out, const Tensor& query, const Tensor& key, const Tensor& value,
                       const Tensor& mask, const Tensor& bias, const Tensor& out, const Tensor& lse, double scale, int64_t flags,
                       bool need_q, bool need_k, bool need_v, bool need_b, const Tensor& lent = {},
                       std::optional<at::ScalarType> dbias_type = std::nullopt) {
  const c10::cuda::CUDAGuard guard(query.device());
  Gradients grads;
  if (need_q) grads.dq = result_like(query);
  if (need_k) grads.dk = result_like(key);
  if (need_v) grads.dv = result_like(value);
  if (need_b && bias.defined()) grads.dbias = at::empty(bias.sizes(), bias.options().dtype(dbias_type.value_or(bias.scalar_type())));
  void* stream = current_stream(query);
  for_each_sample(g, query, [&](const Sample& s, size_t i) {
    oops_ta_problem problem{};
    describe(problem, g, s, i, query, key, value, mask, bias, scale, flags);
    oops_ta_grads wanted{};
    wanted.dq = pair_of(g, s, grads.dq);
    wanted.dk = pair_of(g, s, grads.dk);
    wanted.dv = pair_of(g, s, grads.dv);
    if (grads.dbias.defined()) {
      oops_ta_problem as_bias{};  // the gradient's own strides, through the same description
      describe(as_bias, g, s, i, query, key, value, {}, grads.dbias, scale, flags);
      wanted.dbias = const_cast<void*>(as_bias.bias);
      wanted.dbias_sb = as_bias.bias_sb;
      wanted.dbias_sg = as_bias.bias_sg;
      wanted.dbias_sh = as_bias.bias_sh;
      wanted.dbias_sq = as_bias.bias_sq;
      wanted.dbias_sk = as_bias.bias_sk;
    }
    const uint64_t need = oops_ta_backward_workspace_bytes(&problem, &wanted);
    Tensor scratch = lent;
    if (need && !(lent.defined() && uint64_t(lent.numel()) >= need)) scratch = bytes_like(query, need);
    if (scratch.defined()) {
      problem.workspace = scratch.data_ptr();
      problem.workspace_bytes = uint64_t(scratch.numel());
    }
    const oops_ta_pair out_pair = pair_of(g, s, out), dout_pair = pair_of(g, s, grad_out);
    check_status(oops_ta_backward(&problem, &out_pair, &dout_pair, lse.data_ptr<float>() + s.lse, &wanted, stream),
                 "triangle_attention backward");
  });
  check_device("backward");
  return grads;
}

// Unit inner stride; 16-bit tensors additionally get 16-byte aligned rows, which the TMA kernels need.
Tensor canonical_pair(const Geometry& g, const Tensor& t) {
  if (g.packed || (t.size(-1) != 1 && t.stride(-1) != 1)) return t.contiguous();
  if (t.element_size() == 2) {
    bool aligned = reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
    for (int64_t d = 0; d + 1 < t.dim(); ++d) aligned = aligned && (t.size(d) <= 1 || (t.stride(d) > 0 && t.stride(d) % 8 == 0));
    if (!aligned) return t.contiguous();
  }
  return t;
}

struct TriangleFunction : Function<TriangleFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& query, const Tensor& key, const Tensor& value, const MaybeTensor& mask,
                        const MaybeTensor& bias, double scale, const Geometry& g, int64_t flags) {
    auto [out, lse] = run_forward(g, query, key, value, mask.value_or(Tensor()), bias.value_or(Tensor()), scale, flags, true);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({query, key, value, mask.value_or(Tensor()), bias.value_or(Tensor()), out, lse});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["geometry"] = g.encode();
    ctx->saved_data["flags"] = flags;
    return out;
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    variable_list result(8);
    if (!grad_outputs[0].defined()) return result;
    const variable_list saved = ctx->get_saved_variables();
    const Geometry g = Geometry::decode(ctx->saved_data["geometry"].toIntVector());
    // saved-tensor hooks may hand back copies with other strides; the views are rebuilt from what arrives
    Tensor query = canonical_pair(g, saved[0]), key = canonical_pair(g, saved[1]), value = canonical_pair(g, saved[2]);
    Tensor mask = saved[3], bias = saved[4], out = canonical_pair(g, saved[5]), lse = saved[6].contiguous();
    Tensor grad_out = canonical_pair(g, grad_outputs[0].resolve_neg().to(query.scalar_type()));
    if (g.packed && bias.defined()) bias = bias.contiguous();
    if (g.packed && mask.defined()) mask = mask.contiguous();
    // edges count the tensor arguments that were given
    const size_t bias_edge = mask.defined() ? 4 : 3;
    Gradients grads = run_backward(g, grad_out, query, key, value, mask, bias, out, lse, ctx->saved_data["scale"].toDouble(),
                                   ctx->saved_data["flags"].toInt(), ctx->needs_input_grad(0), ctx->needs_input_grad(1),
                                   ctx->needs_input_grad(2), bias.defined() && ctx->needs_input_grad(bias_edge));
    result[0] = grads.dq;
    result[1] = grads.dk;
    result[2] = grads.dv;
    result[4] = grads.dbias;
    return result;
  }
};

Tensor attend(const Tensor& query, const Tensor& key, const Tensor& value, const MaybeTensor& mask, const MaybeTensor& bias,
              double scale, const Geometry& g, int64_t flags) {
  if (at::GradMode::is_enabled() &&
      (query.requires_grad() || key.requires_grad() || value.requires_grad() || requires_grad(bias)))
    return TriangleFunction::apply(query, key, value, mask, bias, scale, g, flags);
  return std::get<0>(run_forward(g, query, key, value, mask.value_or(Tensor()), bias.value_or(Tensor()), scale, flags, false));
}

// Folds the leading axes of (*lead, <keep axes>) into one batch axis.
Tensor as_batch(const Tensor& t, int64_t keep) {
  const int64_t lead = t.dim() - keep;
  return lead == 1 ? t : lead == 0 ? t.unsqueeze(0) : t.flatten(0, lead - 1);
}

Tensor unit_inner(const Tensor& t) { return t.size(-1) == 1 || t.stride(-1) == 1 ? t : t.contiguous(); }

bool broadcasts_to(at::IntArrayRef own, at::IntArrayRef want) {
  if (own.size() > want.size()) return false;
  for (size_t i = 1; i <= own.size(); ++i)
    if (own[own.size() - i] != 1 && own[own.size() - i] != want[want.size() - i]) return false;
  return true;
}

// Whether the operands of a dense call are what the kernels serve (the Python checks name what is not).
bool dense_operands_fit(const Tensor& query, const Tensor& key, const Tensor& value, const MaybeTensor& mask, const MaybeTensor& bias) {
  if (!plain_context() || !plain_tensor(query) || !plain_tensor(key) || !plain_tensor(value)) return false;
  const auto type = query.scalar_type();
  if (dtype_code(type) < 0 || key.scalar_type() != type || value.scalar_type() != type) return false;
  if (query.dim() < 4 || key.sizes() != query.sizes() || value.sizes() != query.sizes()) return false;
  if (query.numel() == 0 || query.size(-1) > 256) return false;
  if (key.device() != query.device() || value.device() != query.device()) return false;
  const at::IntArrayRef pair = query.sizes().slice(0, query.dim() - 2);
  if (mask.has_value()) {
    if (!plain_tensor(*mask) || mask->device() != query.device() || mask->scalar_type() != at::kBool) return false;
    if (!broadcasts_to(mask->sizes(), pair)) return false;
  }
  if (bias.has_value()) {
    const Tensor& b = *bias;
    if (!plain_tensor(b) || b.device() != query.device() || (b.scalar_type() != type && b.scalar_type() != at::kFloat)) return false;
    const int64_t lead = query.dim() - 4, rows = query.size(lead), cols = query.size(lead + 1), heads = query.size(lead + 2);
    if (b.dim() != lead + 4 || b.sizes().slice(0, lead) != query.sizes().slice(0, lead)) return false;
    if ((b.size(lead) != 1 && b.size(lead) != rows) || b.size(lead + 1) != heads || b.size(lead + 2) != cols || b.size(lead + 3) != cols)
      return false;
  }
  return true;
}

// The values of a 16-bit (B, G, H, N, N) bias in contiguous rows of whole 16-byte words, seen as (B, G, H, N, N).
Tensor padded_bias(const Tensor& bias) {
  const c10::cuda::CUDAGuard guard(bias.device());
  const int64_t cols = bias.size(4), row = (cols + 7) / 8 * 8;
  const Tensor rows = at::empty({bias.size(0), bias.size(1), bias.size(2), cols, row}, bias.options());
  check_status(oops_ta_bias_rows(int32_t(bias.size(0)), int32_t(bias.size(1)), int32_t(bias.size(2)), int32_t(cols), bias.data_ptr(),
                                 bias.strides().data(), rows.data_ptr(), current_stream(bias)),
               "triangle_attention bias rows");
  return row == cols ? rows : rows.narrow(-1, 0, cols);
}

struct PaddedBiasFunction : Function<PaddedBiasFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& bias) {
    ctx->set_materialize_grads(false);
    return padded_bias(bias);
  }
  static variable_list backward(AutogradContext*, const variable_list& grad_outputs) { return {grad_outputs[0]}; }
};

// 16-byte aligned bias rows, which the TMA kernels need (16-bit biases: the key axis is padded); otherwise contiguous.
Tensor aligned_bias(const Tensor& bias, int64_t cols) {
  const Tensor b = as_batch(bias, 4);
  if (b.element_size() != 2) return b.contiguous();
  if (b.is_contiguous() && cols % 8 == 0) return b;
  const Tensor values = b.resolve_neg().resolve_conj();
  return at::GradMode::is_enabled() && values.requires_grad() ? PaddedBiasFunction::apply(values) : padded_bias(values);
}

std::optional<Tensor> dense_attention(const Tensor& query, const Tensor& key, const Tensor& value, const MaybeTensor& mask,
                                      const MaybeTensor& bias, std::optional<double> scale, int64_t flags) {
  if (!dense_operands_fit(query, key, value, mask, bias)) return std::nullopt;
  const int64_t lead = query.dim() - 4;
  const Tensor q5 = unit_inner(as_batch(query, 4));
  // operands that are the same object stay the same object: the kernels then read one buffer
  const Tensor k5 = key.is_same(query) ? q5 : unit_inner(as_batch(key, 4));
  const Tensor v5 = value.is_same(query) ? q5 : value.is_same(key) ? k5 : unit_inner(as_batch(value, 4));
  MaybeTensor mask3, bias5;
  if (mask.has_value()) mask3 = as_batch(mask->expand(query.sizes().slice(0, query.dim() - 2)), 2);
  if (bias.has_value()) bias5 = aligned_bias(*bias, query.size(-3));
  const double factor = scale.has_value() ? *scale : 1.0 / std::sqrt(double(query.size(-1)));
  const Tensor out = attend(q5, k5, v5, mask3, bias5, factor, Geometry(), flags);
  if (lead == 1) return out;
  return lead == 0 ? out.squeeze(0) : out.unflatten(0, query.sizes().slice(0, lead));
}

// ---------------------------------------------------------------------------------------------
// the sigmoid gate
// ---------------------------------------------------------------------------------------------

oops_ta_pair dense_pair(const Tensor& t) { return pair_of(Geometry(), Sample(), t); }

// The kernels read every operand of a gate as the attention's type and shape, on its device.
void check_gate_operands(const Tensor& attention, std::initializer_list<const Tensor*> others) {
  for (const Tensor* t : others)
    TORCH_CHECK(!t->defined() || (t->scalar_type() == attention.scalar_type() && t->sizes() == attention.sizes() && t->device() == attention.device()),
                "gate_attention_output gate kernel: operands of ", attention.scalar_type(), " ", attention.sizes(), " on ", attention.device(),
                " and ", t->scalar_type(), " ", t->sizes(), " on ", t->device());
}

// Library products inside a node keep their operands' type, whatever region the reverse pass is called from.
struct NoAutocast {
  c10::impl::ExcludeDispatchKeyGuard guard{c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)};
};

void check_gate_status(int status) {
  TORCH_CHECK(status == OOPS_TA_OK, "gate_attention_output gate kernel failed: ", oops_ta_status_string(status), ": ", oops_ta_last_error());
}

void run_gate(const Tensor& attention, const Tensor& gate, const Tensor& out) {
  check_gate_operands(attention, {&gate, &out});
  const c10::cuda::CUDAGuard guard(attention.device());
  const oops_ta_pair a = dense_pair(attention), g = dense_pair(gate), o = dense_pair(out);
  check_gate_status(oops_ta_gate_forward(dtype_code(attention.scalar_type()), attention.size(0), attention.size(1), attention.size(2),
                                    attention.size(3), attention.size(4), &a, &g, &o, current_stream(attention)));
}

void run_gate_backward(const Tensor& attention, const Tensor& gate, const Tensor& dout, const Tensor& dattention, const Tensor& dgate) {
  check_gate_operands(attention, {&gate, &dout, &dattention, &dgate});
  const c10::cuda::CUDAGuard guard(attention.device());
  const oops_ta_pair a = dense_pair(attention), g = dense_pair(gate), u = dense_pair(dout), da = dense_pair(dattention),
                     dg = dense_pair(dgate);
  check_gate_status(oops_ta_gate_backward(dtype_code(attention.scalar_type()), attention.size(0), attention.size(1), attention.size(2),
                                     attention.size(3), attention.size(4), &a, &g, &u, &da, &dg, current_stream(attention)));
}

// (B, H, Q, D) values as the C ABI's (B, 1, Q, H, D), and (B, Q, H * D) rows as the same.
Tensor head_major(const Tensor& t) { return t.defined() ? t.permute({0, 2, 1, 3}).unsqueeze(1) : t; }
Tensor token_major(const Tensor& t, int64_t heads, int64_t dim) {
  return t.defined() ? t.view({t.size(0), 1, t.size(1), heads, dim}) : t;
}

// The same without a tensor for it.
oops_ta_pair head_pair(const Tensor& t) { return {t.data_ptr(), t.stride(0), 0, t.stride(2), t.stride(1)}; }

// gated[b, q, h * D + d] = sigmoid(gate[b, q, h * D + d]) * attention[b, h, q, d]
struct GateFunction : Function<GateFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& attention_in, const Tensor& gate_in) {
    const Tensor attention = unit_inner(attention_in.resolve_neg().resolve_conj()), gate = gate_in.contiguous();
    const int64_t heads = attention.size(1), dim = attention.size(3);
    Tensor gated = at::empty_like(gate);
    run_gate(head_major(attention), token_major(gate, heads, dim), token_major(gated, heads, dim));
    ctx->save_for_backward({attention, gate});
    return gated;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor attention = unit_inner(saved[0]), gate = saved[1].contiguous();
    const int64_t heads = attention.size(1), dim = attention.size(3);
    const Tensor dout = grad_outputs[0].resolve_neg().to(gate.scalar_type()).contiguous();
    Tensor dattention, dgate;
    if (ctx->needs_input_grad(0)) dattention = at::empty(attention.sizes(), attention.options());
    if (ctx->needs_input_grad(1)) dgate = at::empty_like(gate);
    run_gate_backward(head_major(attention), token_major(gate, heads, dim), token_major(dout, heads, dim), head_major(dattention),
                      token_major(dgate, heads, dim));
    return {dattention, dgate};
  }
};

struct GatedTriangleFunction : Function<GatedTriangleFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& query, const Tensor& key, const Tensor& value, const Tensor& gate,
                        const MaybeTensor& mask, const MaybeTensor& bias, double scale, int64_t flags) {
    Tensor plain = at::empty(query.sizes(), query.options());
    auto [gated, lse] = run_forward(Geometry(), query, key, value, mask.value_or(Tensor()), bias.value_or(Tensor()), scale, flags, true,
                                    gate, plain);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({query, key, value, gate, mask.value_or(Tensor()), bias.value_or(Tensor()), plain, lse});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["flags"] = flags;
    return gated;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    variable_list result(8);
    if (!grad_outputs[0].defined()) return result;
    const variable_list saved = ctx->get_saved_variables();
    const Geometry g;
    Tensor query = canonical_pair(g, saved[0]), key = canonical_pair(g, saved[1]), value = canonical_pair(g, saved[2]);
    Tensor gate = canonical_pair(g, saved[3]), mask = saved[4], bias = saved[5], plain = canonical_pair(g, saved[6]);
    Tensor grad_gated = canonical_pair(g, grad_outputs[0].resolve_neg().to(query.scalar_type()));
    const bool need_q = ctx->needs_input_grad(0), need_k = ctx->needs_input_grad(1), need_v = ctx->needs_input_grad(2),
               need_b = bias.defined() && ctx->needs_input_grad(mask.defined() ? 5 : 4);
    // through the gate: d(attention) = d(gated) * sigmoid(gate), d(gate) = d(gated) * attention * s (1 - s)
    Tensor dplain = at::empty_like(plain), dgate = ctx->needs_input_grad(3) ? at::empty_like(gate) : Tensor();
    run_gate_backward(plain, gate, grad_gated, dplain, dgate);
    result[3] = dgate;
    if (need_q || need_k || need_v || need_b) {
      Gradients grads = run_backward(g, dplain, query, key, value, mask, bias, plain, saved[7].contiguous(),
                                     ctx->saved_data["scale"].toDouble(), ctx->saved_data["flags"].toInt(), need_q, need_k, need_v, need_b);
      result[0] = grads.dq;
      result[1] = grads.dk;
      result[2] = grads.dv;
      result[5] = grads.dbias;
    }
    return result;
  }
};

Tensor gated_attend(const Tensor& query, const Tensor& key, const Tensor& value, const Tensor& gate, const MaybeTensor& mask,
                    const MaybeTensor& bias, double scale, int64_t flags) {
  if (at::GradMode::is_enabled() && (query.requires_grad() || key.requires_grad() || value.requires_grad() || gate.requires_grad() ||
                                     requires_grad(bias)))
    return GatedTriangleFunction::apply(query, key, value, gate, mask, bias, scale, flags);
  return std::get<0>(run_forward(Geometry(), query, key, value, mask.value_or(Tensor()), bias.value_or(Tensor()), scale, flags, false, gate));
}

std::optional<Tensor> dense_gated_attention(const Tensor& query, const Tensor& key, const Tensor& value, const Tensor& gate_in,
                                            const MaybeTensor& mask, const MaybeTensor& bias, std::optional<double> scale, int64_t flags) {
  if (query.dim() != 5 || !dense_operands_fit(query, key, value, mask, bias) || !plain_tensor(gate_in)) return std::nullopt;
  Tensor gate = gate_in;
  if (gate.dim() == 4 && gate.size(-1) == query.size(-2) * query.size(-1)) gate = gate.unflatten(-1, query.sizes().slice(3, 2));
  if (gate.sizes() != query.sizes() || gate.scalar_type() != query.scalar_type() || gate.device() != query.device()) return std::nullopt;
  const Geometry g;
  const Tensor q5 = canonical_pair(g, unit_inner(query));
  const Tensor k5 = key.is_same(query) ? q5 : canonical_pair(g, unit_inner(key));
  const Tensor v5 = value.is_same(query) ? q5 : value.is_same(key) ? k5 : canonical_pair(g, unit_inner(value));
  MaybeTensor mask3, bias5;
  if (mask.has_value()) mask3 = mask->expand(query.sizes().slice(0, 3));
  if (bias.has_value()) bias5 = aligned_bias(*bias, query.size(2));
  return gated_attend(q5, k5, v5, unit_inner(gate), mask3, bias5,
                      scale.has_value() ? *scale : 1.0 / std::sqrt(double(query.size(-1))), flags);
}

// C = A B^T as the C ABI describes it; operands are contiguous matrices, or `.t()` of one, of more than one column.
oops_ta_product product(const Tensor& a, const Tensor& b, const Tensor& c, int64_t m, int64_t n, int64_t k) {
  oops_ta_product p{};
  auto operand = [](const Tensor& t, const void*& ptr, int64_t& ld, int32_t& transposed) {
    transposed = t.stride(0) == 1 && t.size(0) > 1;
    ptr = t.data_ptr();
    ld = transposed ? t.size(0) : t.size(1);
  };
  operand(a, p.a, p.a_ld, p.a_transposed);
  operand(b, p.b, p.b_ld, p.b_transposed);
  p.c = data_of(c);
  p.c_ld = n;
  p.m = int32_t(m);
  p.n = int32_t(n);
  p.k = int32_t(k);
  return p;
}

// Whether the output step's products run on this library's kernels: `rows` of `in` channels, `inner` channels between the two products,
// `out` channels behind.  What they save is launches: 31 us of host work a call in the forward pass with the library's products and
// the gate between them, 14 to 17 with these; 155 with the reverse, 91.  On the device alone, in us (library / these):
//   rows x heads x channels, in = out   forward        with the reverse
//   64 x 16 x 64, 384                   9.0 / 9.7      21.0 / 19.5
//   512 x 16 x 64, 384                  9.9 / 10.8     26.9 / 24.5
//   1024 x 16 x 64, 384                 11.0 / 11.9    31.0 / 29.9
//   1536 x 16 x 64, 384                 12.3 / 14.9    34.7 / 34.4
//   2048 x 16 x 64, 384                 13.7 / 16.2    38.9 / 43.2
//   2304 x 16 x 64, 384                 13.9 / 16.1    41.0 / 44.7
//   2560 x 16 x 64, 384                 14.8 / 20.3    42.5 / 50.9
//   8192 x 8 x 32, 384                  13.8 / 17.2    53.1 / 46.9
//   16384 x 8 x 16, 128                 11.9 / 11.5    52.5 / 40.8
//   32768 x 16 x 24, 128                36.2 / 51.4    111.9 / 133.6
//   65536 x 8 x 16, 128                 28.9 / 39.9    103.3 / 131.7
//   256 x 32 x 64, 768                  10.8 / 13.6    30.7 / 36.3
// They take a call while what they may cost a device that never waits for the host (a tenth with the reverse) is small beside what they
// save one that does; beyond, the library's larger tiles are the better ones.
constexpr int64_t kOwnProductWork = int64_t(7) << 28, kOwnProductWeights = 5 << 18, kOwnProductRows = 1 << 15;
bool own_products(at::ScalarType type, int64_t rows, int64_t in, int64_t inner, int64_t out, int64_t dim) {
  return (type == at::kBFloat16 || type == at::kHalf) && rows > 0 && in > 0 && out > 0 && in % 8 == 0 && inner % 8 == 0 && out % 8 == 0 &&
         dim % 8 == 0 && rows <= kOwnProductRows && in <= kOwnProductWeights && inner <= kOwnProductWeights && out <= kOwnProductWeights &&
         inner * std::max(in, out) <= kOwnProductWeights && rows * (in + out) <= kOwnProductWork / inner;
}
bool whole_words(const Tensor& t) {  // a matrix, or pairs, whose every eighth element starts a 16-byte word
  if ((reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) != 0) return false;
  for (int64_t i = 0; i < t.dim(); ++i)
    if (t.stride(i) != 1 && t.stride(i) % 8 != 0) return false;
  return true;
}
// What a product takes as a raw address: a whole matrix of this type and size.  Saved tensors come back through hooks, as whatever these
// return, and a gradient may be a batched one; what does not fit takes the library's products, which check their operands.
bool product_matrix(const Tensor& t, const Tensor& like, int64_t rows, int64_t cols) {
  return plain_tensor(t) && t.scalar_type() == like.scalar_type() && t.device() == like.device() && t.dim() == 2 && t.size(0) == rows &&
         t.size(1) == cols && t.is_contiguous() && whole_words(t);
}
void run_products(const Tensor& like, const oops_ta_product* list, int count) {
  check_gate_status(oops_ta_products(dtype_code(like.scalar_type()), list, count, current_stream(like)));
}

// linear(sigmoid(linear(single, gate_weight)) * attention_flat, output_weight) as one node.
struct GateOutputFunction : Function<GateOutputFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& attention, const Tensor& single, const Tensor& gate_weight,
                        const Tensor& output_weight) {
    const auto type = attention.scalar_type();
    const int64_t heads = attention.size(-3), tokens = attention.size(-2), dim = attention.size(-1);
    const Tensor values = unit_inner(attention.reshape({-1, heads, tokens, dim}));
    const Tensor rows = single.reshape({-1, single.size(-1)}), wg = gate_weight.to(type), wo = output_weight.to(type);
    std::vector<int64_t> shape = single.sizes().vec();
    shape.back() = wo.size(0);
    const int64_t count = rows.size(0), in = rows.size(1), inner = heads * dim, out_channels = wo.size(0);
    if (own_products(type, count, in, inner, out_channels, dim) && product_matrix(rows, attention, count, in) &&
        product_matrix(wg, attention, inner, in) && product_matrix(wo, attention, out_channels, inner) && whole_words(values)) {
      const c10::cuda::CUDAGuard guard(attention.device());
      const Tensor gate = at::empty({count, inner}, rows.options()), gated = at::empty({count, inner}, rows.options());
      oops_ta_product open = product(rows, wg, gate, count, inner, in);
      open.epilogue = OOPS_TA_PRODUCT_GATE;
      open.values = head_pair(values);
      open.gated = gated.data_ptr();
      open.gated_ld = inner;
      open.tokens = int32_t(tokens);
      open.dim = int32_t(dim);
      run_products(rows, &open, 1);
      if (ctx) ctx->save_for_backward({attention, single, gate_weight, output_weight, gate, gated});
      const Tensor out = at::empty(shape, rows.options());
      const oops_ta_product project = product(gated, wo, out, count, out_channels, inner);
      run_products(rows, &project, 1);
      return out;
    }
    const Tensor gate = at::linear(rows, wg), gated = at::empty_like(gate);
    auto as_pairs = [&](const Tensor& t) { return t.view({values.size(0), 1, tokens, heads, dim}); };
    run_gate(head_major(values), as_pairs(gate), as_pairs(gated));
    if (ctx) ctx->save_for_backward({attention, single, gate_weight, output_weight, gate, gated});
    return at::_unsafe_view(at::linear(gated, wo), shape);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    const NoAutocast no_autocast;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &attention = saved[0], &single = saved[1];
    const auto type = attention.scalar_type(), gate_type = saved[2].scalar_type(), output_type = saved[3].scalar_type();
    const int64_t heads = attention.size(-3), tokens = attention.size(-2), dim = attention.size(-1);
    const Tensor values = unit_inner(attention.reshape({-1, heads, tokens, dim})), rows = single.reshape({-1, single.size(-1)}),
                 wg = saved[2].to(type), wo = saved[3].to(type);
    Tensor gate = saved[4].contiguous(), gated = saved[5];
    if (at::GradMode::is_enabled()) {  // a graph of the gradients is wanted: they are products of these, which are made to have one
      gate = at::linear(rows, wg);
      gated = GateFunction::apply(values, gate.view({values.size(0), tokens, heads * dim})).view(gate.sizes());
    }
    const Tensor dout = grad_outputs[0].resolve_neg().to(type).reshape({-1, wo.size(0)});
    variable_list result(4);
    const bool need_attention = ctx->needs_input_grad(0), need_gate = ctx->needs_input_grad(1) || ctx->needs_input_grad(2);
    const int64_t count = rows.size(0), in = rows.size(1), inner = heads * dim, out_channels = wo.size(0);
    if (!at::GradMode::is_enabled() && plain_context() && own_products(type, count, in, inner, out_channels, dim) && plain_tensor(values) &&
        whole_words(values) && count == values.size(0) * tokens && product_matrix(rows, attention, count, in) &&
        product_matrix(wg, attention, inner, in) && product_matrix(wo, attention, out_channels, inner) &&
        product_matrix(dout, attention, count, out_channels) && product_matrix(gate, attention, count, inner) &&
        product_matrix(gated, attention, count, inner)) {
      // Two launches: the gradient of what lies behind the gate and what follows from it, then the gate's own product.
      const c10::cuda::CUDAGuard guard(attention.device());
      oops_ta_product list[2];
      int products = 0;
      Tensor dvalues, dgate, dsingle, dwg, dwo;
      if (ctx->needs_input_grad(3)) {
        dwo = at::empty({out_channels, inner}, rows.options());
        list[products++] = product(dout.t(), gated.t(), dwo, out_channels, inner, count);
      }
      if (need_attention || need_gate) {
        if (need_attention) dvalues = at::empty(values.sizes(), values.options());
        if (need_gate) dgate = at::empty({count, inner}, rows.options());
        oops_ta_product& p = list[products++] = product(dout, wo.t(), Tensor(), count, inner, out_channels);
        p.epilogue = OOPS_TA_PRODUCT_GATE_REVERSE;
        p.values = head_pair(values);
        if (need_attention) p.dvalues = head_pair(dvalues);
        p.gate = gate.data_ptr();
        p.gate_ld = inner;
        p.gated = data_of(dgate);
        p.gated_ld = inner;
        p.tokens = int32_t(tokens);
        p.dim = int32_t(dim);
      }
      if (products) run_products(rows, list, products);
      products = 0;
      if (ctx->needs_input_grad(2)) {
        dwg = at::empty({inner, in}, rows.options());
        list[products++] = product(dgate.t(), rows.t(), dwg, inner, in, count);
      }
      if (ctx->needs_input_grad(1)) {
        dsingle = at::empty(single.sizes(), rows.options());
        list[products++] = product(dgate, wg.t(), dsingle, count, in, inner);
      }
      if (products) run_products(rows, list, products);
      if (need_attention) result[0] = dvalues.view(attention.sizes());
      result[1] = dsingle;
      if (dwg.defined()) result[2] = dwg.to(gate_type);
      if (dwo.defined()) result[3] = dwo.to(output_type);
      return result;
    }
    if (ctx->needs_input_grad(3)) result[3] = at::mm(dout.t(), gated).to(output_type);
    if (!need_attention && !need_gate) return result;
    const Tensor dgated = at::mm(dout, wo), dgate = need_gate ? at::empty_like(gate) : Tensor();
    const Tensor dvalues = need_attention ? at::empty(values.sizes(), values.options()) : Tensor();
    auto as_pairs = [&](const Tensor& t) { return t.defined() ? t.view({values.size(0), 1, tokens, heads, dim}) : t; };
    run_gate_backward(head_major(values), as_pairs(gate), as_pairs(dgated), head_major(dvalues), as_pairs(dgate));
    if (need_attention) result[0] = dvalues.view(attention.sizes());
    if (ctx->needs_input_grad(1)) result[1] = at::mm(dgate, wg).view(single.sizes());
    if (ctx->needs_input_grad(2)) result[2] = at::mm(dgate.t(), rows).to(gate_type);
    return result;
  }
};

std::optional<Tensor> gate_output(const Tensor& attention, const Tensor& single, const Tensor& gate_weight, const Tensor& output_weight) {
  if (!plain_context() || at::autocast::is_autocast_enabled(at::kCUDA)) return std::nullopt;
  for (const Tensor* t : {&attention, &single, &gate_weight, &output_weight})
    if (!plain_tensor(*t) || t->device() != attention.device() || !t->is_floating_point()) return std::nullopt;
  const int64_t rank = attention.dim();
  if (rank < 3 || rank > 5 || single.dim() + 1 != rank || gate_weight.dim() != 2 || output_weight.dim() != 2) return std::nullopt;
  if (dtype_code(attention.scalar_type()) < 0 || single.scalar_type() != attention.scalar_type() || attention.numel() == 0) return std::nullopt;
  const int64_t channels = attention.size(-3) * attention.size(-1);
  if (single.sizes().slice(0, rank - 3) != attention.sizes().slice(0, rank - 3) || single.size(-2) != attention.size(-2)) return std::nullopt;
  if (gate_weight.size(0) != channels || gate_weight.size(1) != single.size(-1) || output_weight.size(1) != channels) return std::nullopt;
  if (at::GradMode::is_enabled() &&
      (attention.requires_grad() || single.requires_grad() || gate_weight.requires_grad() || output_weight.requires_grad()))
    return GateOutputFunction::apply(attention, single, gate_weight, output_weight);
  return GateOutputFunction::forward(nullptr, attention, single, gate_weight, output_weight);
}

// ---------------------------------------------------------------------------------------------
// token attention with a pair bias
// ---------------------------------------------------------------------------------------------

// (*prefix, S, H, N, D) operands as (B, S, N, H, D) views of the pair kernels, and results back; ranks 3 and 4 omit leading axes.
Tensor tokens_as_pairs(const Tensor& t) {
  const int64_t rank = t.dim();
  return t.reshape({-1, rank > 3 ? t.size(-4) : 1, t.size(-3), t.size(-2), t.size(-1)}).permute({0, 1, 3, 2, 4});
}
Tensor pairs_as_tokens(const Tensor& pairs, at::IntArrayRef shape) {
  return pairs.defined() ? pairs.permute({0, 1, 3, 2, 4}).reshape(shape) : pairs;
}
Tensor token_bias(const Tensor& bias) {
  const int64_t rank = bias.dim();
  return aligned_bias(bias.reshape({-1, rank > 3 ? bias.size(-4) : 1, bias.size(-3), bias.size(-2), bias.size(-1)}), bias.size(-1));
}
Tensor token_mask(const Tensor& mask, const Tensor& query) {
  if (!mask.defined()) return mask;
  const int64_t groups = query.dim() > 3 ? query.size(-4) : 1, tokens = query.size(-2);
  const Tensor rows = mask.reshape({-1, mask.dim() > 1 ? mask.size(-2) : 1, tokens});
  return rows.expand({rows.size(0), groups, tokens});
}

struct TokenFunction : Function<TokenFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& query, const Tensor& key, const Tensor& value, const MaybeTensor& mask,
                        const MaybeTensor& bias, double scale, int64_t flags) {
    const Tensor laid_bias = bias.has_value() ? token_bias(*bias) : Tensor();
    const Tensor laid_mask = token_mask(mask.value_or(Tensor()), query);
    const Tensor q = unit_inner(tokens_as_pairs(query)), k = key.is_same(query) ? q : unit_inner(tokens_as_pairs(key)),
                 v = value.is_same(query) ? q : value.is_same(key) ? k : unit_inner(tokens_as_pairs(value));
    const Tensor result = at::empty(query.sizes(), query.options());
    auto [out, lse] = run_forward(Geometry(), q, k, v, laid_mask, laid_bias, scale, flags, ctx != nullptr, {}, {}, tokens_as_pairs(result));
    if (ctx) {
      ctx->set_materialize_grads(false);
      ctx->save_for_backward({q, k, v, laid_mask, laid_bias, result, lse});
      ctx->saved_data["shape"] = query.sizes().vec();
      ctx->saved_data["bias_shape"] = bias.has_value() ? bias->sizes().vec() : std::vector<int64_t>();
      ctx->saved_data["scale"] = scale;
      ctx->saved_data["flags"] = flags;
    }
    return result;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    variable_list result(7);
    if (!grad_outputs[0].defined()) return result;
    const variable_list saved = ctx->get_saved_variables();
    const Geometry g;
    const Tensor q = canonical_pair(g, saved[0]), k = canonical_pair(g, saved[1]), v = canonical_pair(g, saved[2]), mask = saved[3],
                 bias = saved[4], out = canonical_pair(g, tokens_as_pairs(saved[5]));
    const Tensor grad_out = canonical_pair(g, tokens_as_pairs(grad_outputs[0].resolve_neg().to(q.scalar_type())));
    Gradients grads = run_backward(g, grad_out, q, k, v, mask, bias, out, saved[6].contiguous(), ctx->saved_data["scale"].toDouble(),
                                   ctx->saved_data["flags"].toInt(), ctx->needs_input_grad(0), ctx->needs_input_grad(1),
                                   ctx->needs_input_grad(2), bias.defined() && ctx->needs_input_grad(mask.defined() ? 4 : 3));
    const std::vector<int64_t> shape = ctx->saved_data["shape"].toIntVector();
    result[0] = pairs_as_tokens(grads.dq, shape);
    result[1] = pairs_as_tokens(grads.dk, shape);
    result[2] = pairs_as_tokens(grads.dv, shape);
    if (grads.dbias.defined()) result[4] = grads.dbias.reshape(ctx->saved_data["bias_shape"].toIntVector());
    return result;
  }
};

std::optional<Tensor> token_attention(const Tensor& query, const Tensor& key, const Tensor& value, const MaybeTensor& mask,
                                      const MaybeTensor& bias, std::optional<double> scale, int64_t flags) {
  if (!plain_context()) return std::nullopt;
  for (const Tensor* t : {&query, &key, &value})
    if (!plain_tensor(*t) || t->device() != query.device() || t->scalar_type() != query.scalar_type() || t->sizes() != query.sizes())
      return std::nullopt;
  const int64_t rank = query.dim();
  if (rank < 3 || dtype_code(query.scalar_type()) < 0 || query.numel() == 0 || query.size(-1) > 256) return std::nullopt;
  const int64_t groups = rank > 3 ? query.size(-4) : 1, heads = query.size(-3), tokens = query.size(-2), prefix = std::max<int64_t>(rank - 4, 0);
  if (mask.has_value()) {  // (*prefix, S|1, K)
    if (!plain_tensor(*mask) || mask->device() != query.device() || mask->scalar_type() != at::kBool || mask->dim() != rank - 2 ||
        mask->size(-1) != tokens || mask->sizes().slice(0, prefix) != query.sizes().slice(0, prefix))
      return std::nullopt;
    if (mask->dim() > 1 && mask->size(-2) != 1 && mask->size(-2) != groups) return std::nullopt;
  }
  if (bias.has_value()) {  // (*prefix, S|1, H, Q, K)
    if (!plain_tensor(*bias) || bias->device() != query.device() || bias->scalar_type() != query.scalar_type() || bias->dim() != rank ||
        bias->sizes().slice(0, prefix) != query.sizes().slice(0, prefix) || bias->size(-3) != heads || bias->size(-2) != tokens ||
        bias->size(-1) != tokens)
      return std::nullopt;
    if (rank > 3 && bias->size(-4) != 1 && bias->size(-4) != groups) return std::nullopt;
  }
  const double factor = scale.has_value() ? *scale : 1.0 / std::sqrt(double(query.size(-1)));
  if (at::GradMode::is_enabled() && (query.requires_grad() || key.requires_grad() || value.requires_grad() || requires_grad(bias)))
    return TokenFunction::apply(query, key, value, mask, bias, factor, flags);
  return TokenFunction::forward(nullptr, query, key, value, mask, bias, factor, flags);
}

// ---------------------------------------------------------------------------------------------
// layer norm
// ---------------------------------------------------------------------------------------------

// `t` as (rows, width) with contiguous rows; a view when the layout allows it.
Tensor rows_of(const Tensor& t, int64_t width) {
  Tensor flat = t.reshape({-1, width});
  if ((width > 1 && flat.stride(1) != 1) || (flat.size(0) > 1 && flat.stride(0) < width)) flat = flat.contiguous();
  return flat;
}

struct Normed {
  Tensor y, stats;  // stats: (2, rows) f32, mean and reciprocal standard deviation
};

// The result has `shape` (that of the rows, or of the tensor they are a view of).
Normed norm_forward(const Tensor& rows_in, const Tensor& weight, const Tensor& bias, double eps, bool keep_stats, at::IntArrayRef shape) {
  const c10::cuda::CUDAGuard guard(rows_in.device());
  const int64_t rows = rows_in.size(0), width = rows_in.size(1);
  Normed n{at::empty(shape, rows_in.options()), keep_stats ? floats_like(rows_in, {2, rows}) : Tensor()};
  const auto affine = weight.defined() ? weight.scalar_type() : bias.defined() ? bias.scalar_type() : rows_in.scalar_type();
  float* stats = keep_stats ? n.stats.data_ptr<float>() : nullptr;
  const int status = oops_ta_layer_norm_forward(
      dtype_code(rows_in.scalar_type()), dtype_code(affine), rows, int32_t(width), rows_in.data_ptr(), rows > 1 ? rows_in.stride(0) : width,
      data_of(weight), data_of(bias), float(eps), n.y.data_ptr(), width, stats, stats ? stats + rows : nullptr, current_stream(rows_in));
  if (status) raise_unsupported(std::string("layer_norm ") + oops_ta_status_string(status) + ": " + oops_ta_last_error());
  return n;
}

struct NormGradients {
  Tensor dx, dweight, dbias;
};

NormGradients norm_backward(const Tensor& dy, const Tensor& rows_in, const Tensor& weight, const Tensor& stats, at::ScalarType affine,
                            bool need_x, bool need_w, bool need_b) {
  const c10::cuda::CUDAGuard guard(rows_in.device());
  const int64_t rows = rows_in.size(0), width = rows_in.size(1);
  NormGradients grads;
  if (need_x) grads.dx = at::empty({rows, width}, rows_in.options());
  if (need_w) grads.dweight = at::empty({width}, rows_in.options().dtype(affine));
  if (need_b) grads.dbias = at::empty({width}, rows_in.options().dtype(affine));
  const uint64_t need = need_w || need_b ? oops_ta_layer_norm_backward_workspace_bytes(rows, int32_t(width)) : 0;
  Tensor scratch = need ? bytes_like(rows_in, need) : Tensor();
  const float* mean = stats.data_ptr<float>();
  const int status = oops_ta_layer_norm_backward(
      dtype_code(rows_in.scalar_type()), dtype_code(affine), rows, int32_t(width), dy.data_ptr(), rows > 1 ? dy.stride(0) : width,
      rows_in.data_ptr(), rows > 1 ? rows_in.stride(0) : width, data_of(weight), mean, mean + rows, data_of(grads.dx), width,
      data_of(grads.dweight), data_of(grads.dbias), data_of(scratch), need, current_stream(rows_in));
  if (status) raise_unsupported(std::string("layer_norm ") + oops_ta_status_string(status) + ": " + oops_ta_last_error());
  return grads;
}

struct LayerNormFunction : Function<LayerNormFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const MaybeTensor& weight, const MaybeTensor& bias, double eps) {
    const Tensor rows = rows_of(x, x.size(-1));
    const Tensor w = weight.has_value() ? weight->contiguous() : Tensor(), b = bias.has_value() ? bias->contiguous() : Tensor();
    Normed n = norm_forward(rows, w, b, eps, true, x.sizes());
    ctx->save_for_backward({rows, w, n.stats});
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->saved_data["affine"] = int64_t(w.defined() ? w.scalar_type() : b.defined() ? b.scalar_type() : x.scalar_type());
    ctx->saved_data["has_bias"] = b.defined();
    return n.y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor rows = rows_of(saved[0], saved[0].size(-1));
    const bool has_weight = saved[1].defined(), has_bias = ctx->saved_data["has_bias"].toBool();
    const Tensor w = has_weight ? saved[1].contiguous() : Tensor();
    const size_t bias_edge = has_weight ? 2 : 1;
    NormGradients grads = norm_backward(rows_of(grad_outputs[0].resolve_neg(), rows.size(1)), rows, w, saved[2].contiguous(),
                                        at::ScalarType(ctx->saved_data["affine"].toInt()), ctx->needs_input_grad(0),
                                        has_weight && ctx->needs_input_grad(1), has_bias && ctx->needs_input_grad(bias_edge));
    if (grads.dx.defined()) grads.dx = grads.dx.view(ctx->saved_data["shape"].toIntVector());
    return {grads.dx, grads.dweight, grads.dbias, Tensor()};
  }
};

bool norm_operands_fit(const Tensor& x, const MaybeTensor& weight, const MaybeTensor& bias, int64_t width) {
  if (!plain_tensor(x) || dtype_code(x.scalar_type()) < 0 || x.dim() < 1 || x.size(-1) != width || width < 1 || width > 8192 || x.numel() == 0)
    return false;
  std::optional<at::ScalarType> affine;
  for (const MaybeTensor* p : {&weight, &bias}) {
    if (!p->has_value()) continue;
    const Tensor& t = **p;
    if (!plain_tensor(t) || t.device() != x.device() || t.dim() != 1 || t.size(0) != width) return false;
    if (t.scalar_type() != x.scalar_type() && t.scalar_type() != at::kFloat) return false;
    if (affine.has_value() && *affine != t.scalar_type()) return false;
    affine = t.scalar_type();
  }
  return true;
}

// Without a look at the context: under a dispatch mode the allocations go through it, the launches do not.
std::optional<Tensor> layer_norm_node(const Tensor& x, int64_t width, const MaybeTensor& weight, const MaybeTensor& bias, double eps) {
  if (!norm_operands_fit(x, weight, bias, width)) return std::nullopt;
  if (at::GradMode::is_enabled() && (x.requires_grad() || requires_grad(weight) || requires_grad(bias)))
    return LayerNormFunction::apply(x, weight, bias, eps);
  const Tensor w = weight.has_value() ? weight->contiguous() : Tensor(), b = bias.has_value() ? bias->contiguous() : Tensor();
  return norm_forward(rows_of(x, width), w, b, eps, false, x.sizes()).y;
}

std::optional<Tensor> layer_norm(const Tensor& x, int64_t width, const MaybeTensor& weight, const MaybeTensor& bias, double eps) {
  return plain_context() ? layer_norm_node(x, width, weight, bias, eps) : std::nullopt;
}

// ---------------------------------------------------------------------------------------------
// triangle multiplicative update
// ---------------------------------------------------------------------------------------------

struct UpdateShape {
  int code;
  int32_t prefix, tokens, padded, hidden;
  int64_t cells() const { return int64_t(prefix) * tokens * tokens; }
};

// update[i, j] = sum_k left[i, k] right[j, k] (outgoing) or sum_k left[k, i] right[k, j], plane by plane
Tensor contract(bool outgoing, const Tensor& left, const Tensor& right) {
  return outgoing ? at::bmm(left, right.transpose(1, 2)) : at::bmm(left.transpose(1, 2), right);
}

enum { kLeftGate, kLeftValue, kRightGate, kRightValue, kOutputGate, kOutput, kProjections };

// The update from single operations, with the graph that a second differentiation needs (operands as UpdateFunction has them).
Tensor composed_update(const Tensor& pair, const Tensor& mask, bool outgoing, double in_eps, double out_eps, at::TensorList parameters,
                       const std::vector<int64_t>& bias_of) {
  const auto type = pair.scalar_type();
  MaybeTensor biases[kProjections];
  for (size_t i = 0; i < bias_of.size(); ++i) biases[bias_of[i]] = parameters[10 + i].to(type);
  auto project = [&](const Tensor& x, int which) { return at::linear(x, parameters[4 + which].to(type), biases[which]); };
  const Tensor x = LayerNormFunction::apply(pair, MaybeTensor(parameters[0]), MaybeTensor(parameters[1]), in_eps);
  const Tensor weight = mask.defined() ? mask.to(type).unsqueeze(-1) : Tensor();
  auto side = [&](int gate) {  // channel-major
    const Tensor open = at::sigmoid(project(x, gate));
    return ((weight.defined() ? weight * open : open) * project(x, gate + 1)).movedim(-1, -3);
  };
  const Tensor left = side(kLeftGate), right = side(kRightGate);
  const Tensor update = at::matmul(outgoing ? left : left.transpose(-1, -2), outgoing ? right.transpose(-1, -2) : right).movedim(-3, -1);
  const Tensor normed = LayerNormFunction::apply(update.contiguous(), MaybeTensor(parameters[2]), MaybeTensor(parameters[3]), out_eps);
  return project(normed, kOutput) * at::sigmoid(project(x, kOutputGate));
}

struct UpdateFunction : Function<UpdateFunction> {
  static constexpr size_t kFirst = 5;  // inputs: pair, mask, outgoing, in_eps, out_eps, parameters..., bias_of
  // `parameters`: the input and output norms' weight and bias, the six projection weights, then the biases that exist;
  // `bias_of` says which projection each of those belongs to.
  static Tensor forward(AutogradContext* ctx, const Tensor& pair, const MaybeTensor& mask, bool outgoing, double in_eps, double out_eps,
                        at::TensorList parameters, const std::vector<int64_t>& bias_of) {
    const auto type = pair.scalar_type();
    const int64_t channels = pair.size(-1), tokens = pair.size(-2);
    const Tensor* weights = &parameters[4];
    const int64_t hidden = weights[0].size(0);
    const UpdateShape s{dtype_code(type), int32_t(pair.numel() / (tokens * tokens * channels)), int32_t(tokens),
                        int32_t((tokens + 7) / 8 * 8), int32_t(hidden)};
    const c10::cuda::CUDAGuard guard(pair.device());
    void* stream = current_stream(pair);
    Tensor biases[kProjections];
    bool stacked_has_bias = false;
    for (size_t i = 0; i < bias_of.size(); ++i) {
      biases[bias_of[i]] = parameters[10 + i];
      stacked_has_bias = stacked_has_bias || bias_of[i] != kOutput;
    }
    // rows of the projections: left gate | left value | right gate | right value | output gate
    const Tensor stacked = at::cat({weights[0], weights[1], weights[2], weights[3], weights[4]}).to(type);
    Tensor stacked_bias;
    if (stacked_has_bias) {
      std::vector<Tensor> pieces;
      for (int i = 0; i < kOutput; ++i) pieces.push_back(biases[i].defined() ? biases[i].to(type) : at::zeros({weights[i].size(0)}, pair.options()));
      stacked_bias = at::cat(pieces);
    }
    const Tensor out_matrix = weights[kOutput].to(type);
    const Tensor rows = rows_of(pair, channels), in_w = parameters[0].contiguous(), out_w = parameters[2].contiguous();
    Normed x = norm_forward(rows, in_w, parameters[1].contiguous(), in_eps, true, rows.sizes());
    const Tensor proj = stacked_has_bias ? at::linear(x.y, stacked, stacked_bias) : at::linear(x.y, stacked);
    const int64_t ld = proj.size(1);
    const Tensor weight = mask.has_value() ? mask->to(type).expand(pair.sizes().slice(0, pair.dim() - 1)).contiguous() : Tensor();
    const Tensor planes = at::empty({2, s.prefix * hidden, s.padded, s.padded}, pair.options());
    const Tensor left = planes.select(0, 0), right = planes.select(0, 1);
    check_status(oops_ta_pair_gate_forward(s.code, s.prefix, s.tokens, s.padded, s.hidden, proj.data_ptr(), ld, data_of(weight), left.data_ptr(),
                                           right.data_ptr(), stream),
                 "triangle_multiplication pair gate");
    const Tensor update = contract(outgoing, left, right);
    const Tensor normed = at::empty({s.cells(), hidden}, pair.options()), stats = floats_like(pair, {2, s.cells()});
    check_status(oops_ta_channel_norm_forward(s.code, dtype_code(out_w.scalar_type()), s.prefix, s.tokens, s.padded, s.hidden, update.data_ptr(),
                                              out_w.data_ptr(), parameters[3].contiguous().data_ptr(), float(out_eps), normed.data_ptr(),
                                              stats.data_ptr<float>(), stats.data_ptr<float>() + s.cells(), stream),
                 "triangle_multiplication output norm");
    const Tensor values = biases[kOutput].defined() ? at::linear(normed, out_matrix, biases[kOutput].to(type)) : at::linear(normed, out_matrix);
    const Tensor out = at::empty(pair.sizes(), pair.options());
    const char* gate = static_cast<const char*>(proj.data_ptr()) + 4 * hidden * proj.element_size();
    check_status(oops_ta_output_gate_forward(s.code, s.cells(), int32_t(channels), values.data_ptr(), gate, ld, out.data_ptr(), stream),
                 "triangle_multiplication output gate");
    if (ctx) {
      ctx->set_materialize_grads(false);
      variable_list kept{pair, x.stats, x.y, stacked, proj, weight, left, right, update, stats, normed, out_matrix, values, mask.value_or(Tensor())};
      kept.insert(kept.end(), parameters.begin(), parameters.end());
      ctx->save_for_backward(kept);
      ctx->saved_data["outgoing"] = outgoing;
      ctx->saved_data["eps"] = std::vector<double>{in_eps, out_eps};
      ctx->saved_data["dims"] = std::vector<int64_t>{s.prefix, s.tokens, s.padded, s.hidden, mask.has_value()};
      ctx->saved_data["bias_of"] = bias_of;
      std::vector<int64_t> types;
      for (const Tensor& p : parameters) types.push_back(int64_t(p.scalar_type()));
      ctx->saved_data["types"] = types;
    }
    return out;
  }

  // With a graph of the gradients wanted, they come from the composed form (as far as its nodes have one themselves).
  static variable_list differentiable_backward(AutogradContext* ctx, const Tensor& dout, const variable_list& saved, size_t first,
                                               const std::vector<int64_t>& bias_of, size_t edge, variable_list result) {
    const std::vector<double> eps = ctx->saved_data["eps"].toDoubleVector();
    const variable_list parameters(saved.begin() + first, saved.end());
    const Tensor out = composed_update(saved[0], saved[first - 1], ctx->saved_data["outgoing"].toBool(), eps[0], eps[1], parameters, bias_of);
    variable_list inputs;
    std::vector<size_t> places;
    for (size_t i = 0; i <= parameters.size(); ++i) {
      if (!ctx->needs_input_grad(i == 0 ? 0 : edge + i - 1)) continue;
      inputs.push_back(i == 0 ? saved[0] : parameters[i - 1]);
      places.push_back(i == 0 ? 0 : kFirst + i - 1);
    }
    const variable_list grads = torch::autograd::grad({out}, inputs, {dout.to(out.scalar_type())}, std::nullopt, true, true);
    for (size_t i = 0; i < places.size(); ++i) result[places[i]] = grads[i];
    return result;
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& grad_outputs) {
    const NoAutocast no_autocast;
    const std::vector<int64_t> dims = ctx->saved_data["dims"].toIntVector(), bias_of = ctx->saved_data["bias_of"].toIntVector(),
                               types = ctx->saved_data["types"].toIntVector();
    variable_list result(kFirst + types.size() + 1);
    if (!grad_outputs[0].defined()) return result;
    variable_list saved = ctx->get_saved_variables();
    constexpr size_t kKept = 14;  // then the parameters
    if (at::GradMode::is_enabled()) return differentiable_backward(ctx, grad_outputs[0], saved, kKept, bias_of, dims[4] ? 2 : 1, std::move(result));
    for (size_t i = 1; i < saved.size(); ++i)
      if (saved[i].defined()) saved[i] = saved[i].contiguous();
    const Tensor &pair = saved[0], &stats1 = saved[1], &x = saved[2], &stacked = saved[3], &proj = saved[4], &weight = saved[5],
                 &left = saved[6], &right = saved[7], &update = saved[8], &stats2 = saved[9], &normed = saved[10], &out_matrix = saved[11],
                 &values = saved[12], &in_w = saved[kKept], &out_w = saved[kKept + 2];
    const UpdateShape s{dtype_code(proj.scalar_type()), int32_t(dims[0]), int32_t(dims[1]), int32_t(dims[2]), int32_t(dims[3])};
    const size_t edge = dims[4] ? 2 : 1;  // first parameter's edge: behind the pair and, when it was given, the mask
    auto need = [&](size_t parameter) { return ctx->needs_input_grad(edge + parameter); };
    auto give = [&](size_t parameter, const Tensor& grad) { result[kFirst + parameter] = grad.to(at::ScalarType(types[parameter])); };
    const int64_t hidden = s.hidden, cells = proj.size(0), ld = proj.size(1), channels = x.size(1);
    const c10::cuda::CUDAGuard guard(proj.device());
    void* stream = current_stream(proj);
    const Tensor dout = rows_of(grad_outputs[0].resolve_neg().to(proj.scalar_type()), channels).contiguous();

    const Tensor dvalues = at::empty_like(values), dproj = at::empty_like(proj);
    const int64_t gate_at = 4 * hidden * proj.element_size();
    check_status(oops_ta_output_gate_backward(s.code, cells, int32_t(channels), dout.data_ptr(), values.data_ptr(),
                                              static_cast<const char*>(proj.data_ptr()) + gate_at, ld, dvalues.data_ptr(),
                                              static_cast<char*>(dproj.data_ptr()) + gate_at, ld, stream),
                 "triangle_multiplication output gate");
    size_t output_bias = 0;
    bool other_bias = false;
    for (size_t i = 0; i < bias_of.size(); ++i) {
      if (bias_of[i] == kOutput) output_bias = 10 + i;
      else other_bias = other_bias || need(10 + i);
    }
    if (need(4 + kOutput)) give(4 + kOutput, at::mm(dvalues.t(), normed));
    if (output_bias && need(output_bias)) give(output_bias, dvalues.sum(0));
    const Tensor dnormed = at::mm(dvalues, out_matrix), dupdate = at::empty_like(update);
    const Tensor dw2 = need(2) ? at::empty_like(out_w) : Tensor(), db2 = need(3) ? at::empty_like(out_w) : Tensor();
    const uint64_t bytes = oops_ta_channel_norm_backward_workspace_bytes(s.code, s.prefix, s.tokens, s.padded, s.hidden);
    const Tensor scratch = bytes_like(proj, bytes);
    check_status(oops_ta_channel_norm_backward(s.code, dtype_code(out_w.scalar_type()), s.prefix, s.tokens, s.padded, s.hidden,
                                               dnormed.data_ptr(), update.data_ptr(), out_w.data_ptr(), stats2.data_ptr<float>(),
                                               stats2.data_ptr<float>() + cells, dupdate.data_ptr(), data_of(dw2), data_of(db2),
                                               scratch.data_ptr(), bytes, stream),
                 "triangle_multiplication output norm");
    result[kFirst + 2] = dw2;
    result[kFirst + 3] = db2;
    bool weights_wanted = false;
    for (size_t i = 0; i < size_t(kOutput); ++i) weights_wanted = weights_wanted || need(4 + i);
    const bool pair_wanted = ctx->needs_input_grad(0), norm_wanted = pair_wanted || need(0) || need(1);
    if (!weights_wanted && !other_bias && !norm_wanted) return result;

    const bool outgoing = ctx->saved_data["outgoing"].toBool();
    const Tensor dleft = outgoing ? at::bmm(dupdate, right) : at::bmm(right, dupdate.transpose(1, 2));
    const Tensor dright = outgoing ? at::bmm(dupdate.transpose(1, 2), left) : at::bmm(left, dupdate);
    check_status(oops_ta_pair_gate_backward(s.code, s.prefix, s.tokens, s.padded, s.hidden, proj.data_ptr(), ld, data_of(weight),
                                            dleft.data_ptr(), dright.data_ptr(), dproj.data_ptr(), ld, stream),
                 "triangle_multiplication pair gate");
    auto piece = [&](const Tensor& t, int64_t which) { return t.narrow(0, which * hidden, which == kOutputGate ? channels : hidden); };
    if (weights_wanted) {
      Tensor stacked_grad = at::mm(dproj.t(), x);
      // weights of one type share a conversion, of which each gets its rows
      bool same_type = true;
      for (size_t i = 5; i < 4 + size_t(kOutput); ++i) same_type = same_type && types[i] == types[4];
      if (same_type) stacked_grad = stacked_grad.to(at::ScalarType(types[4]));
      for (int64_t i = 0; i < kOutput; ++i)
        if (need(4 + i)) give(4 + i, piece(stacked_grad, i));
    }
    if (other_bias) {
      const Tensor sums = dproj.sum(0);
      for (size_t i = 0; i < bias_of.size(); ++i)
        if (bias_of[i] != kOutput && need(10 + i)) give(10 + i, piece(sums, bias_of[i]));
    }
    if (norm_wanted) {
      NormGradients grads = norm_backward(at::mm(dproj, stacked), rows_of(pair, channels), in_w, stats1, in_w.scalar_type(), pair_wanted,
                                          need(0), need(1));
      if (pair_wanted) result[0] = grads.dx.view(pair.sizes());
      result[kFirst] = grads.dweight;
      result[kFirst + 1] = grads.dbias;
    }
    return result;
  }
};

// ---------------------------------------------------------------------------------------------
// Python boundary
// ---------------------------------------------------------------------------------------------

MaybeTensor maybe_tensor(PyObject* o) { return o == Py_None ? MaybeTensor() : MaybeTensor(THPVariable_Unpack(o)); }
// The entries take tensors and parameters; a subclass, whose results are of its own kind, goes through the Python path.
bool is_tensor(PyObject* o) { return THPVariable_CheckExact(o); }
bool tensor_or_none(PyObject* o) { return o == Py_None || is_tensor(o); }
bool is_number(PyObject* o) { return PyFloat_Check(o) || PyLong_Check(o); }  // anything else is converted, or refused, in Python
double number(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
std::optional<double> maybe_number(PyObject* o) { return o == Py_None ? std::nullopt : std::optional<double>(number(o)); }
bool number_or_none(PyObject* o) { return o == Py_None || is_number(o); }

PyObject* wrap(std::optional<Tensor>&& t) {
  if (!t.has_value()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(*t));
}

// triangle_attention / pair_bias_attention(query, key, value, mask, bias, scale, flags) -> Tensor or None
template <auto Attention>
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 7, "attention takes 7 arguments");
  if (!is_tensor(a[0]) || !is_tensor(a[1]) || !is_tensor(a[2]) || !tensor_or_none(a[3]) || !tensor_or_none(a[4]) ||
      !number_or_none(a[5]))
    Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
  const MaybeTensor mask = maybe_tensor(a[3]), bias = maybe_tensor(a[4]);
  const std::optional<double> scale = maybe_number(a[5]);
  const int64_t flags = PyLong_AsLongLong(a[6]);
  std::optional<Tensor> out;
  {
    py::gil_scoped_release no_gil;
    out = Attention(q, k, v, mask, bias, scale, flags);
  }
  return wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// triangle_attention_gated(query, key, value, gate, mask, bias, scale, flags) -> Tensor or None
PyObject* py_gated_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 8, "triangle_attention_gated takes 8 arguments");
  for (int i = 0; i < 4; ++i)
    if (!is_tensor(a[i])) Py_RETURN_NONE;
  if (!tensor_or_none(a[4]) || !tensor_or_none(a[5]) || !number_or_none(a[6])) Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]), &g = THPVariable_Unpack(a[3]);
  const MaybeTensor mask = maybe_tensor(a[4]), bias = maybe_tensor(a[5]);
  const std::optional<double> scale = maybe_number(a[6]);
  const int64_t flags = PyLong_AsLongLong(a[7]);
  std::optional<Tensor> out;
  {
    py::gil_scoped_release no_gil;
    out = dense_gated_attention(q, k, v, g, mask, bias, scale, flags);
  }
  return wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// gate_attention_output(attention, single, gate_weight, output_weight) -> Tensor or None
PyObject* py_gate_output(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 4, "gate_attention_output takes 4 arguments");
  for (int i = 0; i < 4; ++i)
    if (!is_tensor(a[i])) Py_RETURN_NONE;
  std::optional<Tensor> out;
  {
    const Tensor &attention = THPVariable_Unpack(a[0]), &single = THPVariable_Unpack(a[1]), &wg = THPVariable_Unpack(a[2]),
                 &wo = THPVariable_Unpack(a[3]);
    py::gil_scoped_release no_gil;
    out = gate_output(attention, single, wg, wo);
  }
  return wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// layer_norm(x, width, weight, bias, eps) -> Tensor or None
PyObject* py_layer_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 5, "layer_norm takes 5 arguments");
  if (!is_tensor(a[0]) || !PyLong_Check(a[1]) || !tensor_or_none(a[2]) || !tensor_or_none(a[3]) || !is_number(a[4])) Py_RETURN_NONE;
  const Tensor& x = THPVariable_Unpack(a[0]);
  int overflow = 0;
  const int64_t width = PyLong_AsLongLongAndOverflow(a[1], &overflow);
  if (overflow) Py_RETURN_NONE;
  const MaybeTensor weight = maybe_tensor(a[2]), bias = maybe_tensor(a[3]);
  const double eps = number(a[4]);
  std::optional<Tensor> out;
  {
    py::gil_scoped_release no_gil;
    out = layer_norm(x, width, weight, bias, eps);
  }
  return wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef g_fast_methods[] = {
    {"triangle_attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention<dense_attention>)), METH_FASTCALL, nullptr},
    {"pair_bias_attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention<token_attention>)), METH_FASTCALL, nullptr},
    {"gate_attention_output", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_gate_output)), METH_FASTCALL, nullptr},
    {"triangle_attention_gated", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_gated_attention)), METH_FASTCALL, nullptr},
    {"layer_norm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_layer_norm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(_native, m) {
  PyModule_AddFunctions(m.ptr(), g_fast_methods);
  using NoGil = py::call_guard<py::gil_scoped_release>;
  auto or_empty = [](const MaybeTensor& t) { return t.value_or(Tensor()); };
  m.def("set_unsupported_error", [](py::object type) { g_unsupported_error = type.release().ptr(); });
  m.def("check_device_status", [](bool enabled) { return g_check_status.exchange(enabled); });
  m.def("attend", [](const Tensor& q, const Tensor& k, const Tensor& v, const MaybeTensor& mask, const MaybeTensor& bias, double scale,
                     const std::vector<int64_t>& geometry, int64_t flags) {
    return attend(q, k, v, mask, bias, scale, Geometry::decode(geometry), flags);
  }, NoGil());
  m.def("gated_attend", &gated_attend, NoGil());
  m.def("run_forward", [or_empty](const std::vector<int64_t>& geometry, const Tensor& q, const Tensor& k, const Tensor& v,
                                  const MaybeTensor& mask, const MaybeTensor& bias, double scale, int64_t flags, bool want_lse) {
    auto [out, lse] = run_forward(Geometry::decode(geometry), q, k, v, or_empty(mask), or_empty(bias), scale, flags, want_lse);
    return std::make_tuple(out, lse.defined() ? MaybeTensor(lse) : MaybeTensor());
  }, NoGil());
  m.def("run_backward", [or_empty](const std::vector<int64_t>& geometry, const Tensor& grad_out, const Tensor& q, const Tensor& k,
                                   const Tensor& v, const MaybeTensor& mask, const MaybeTensor& bias, const Tensor& out, const Tensor& lse,
                                   double scale, int64_t flags, const std::vector<bool>& need, const MaybeTensor& scratch,
                                   bool dbias_f32) {
    Gradients g = run_backward(Geometry::decode(geometry), grad_out, q, k, v, or_empty(mask), or_empty(bias), out, lse, scale, flags, need[0],
                               need[1], need[2], need[3], or_empty(scratch),
                               dbias_f32 ? std::optional<at::ScalarType>(at::kFloat) : std::nullopt);
    auto maybe = [](const Tensor& t) { return t.defined() ? MaybeTensor(t) : MaybeTensor(); };
    return std::make_tuple(maybe(g.dq), maybe(g.dk), maybe(g.dv), maybe(g.dbias));
  }, NoGil());
  m.def("sigmoid_gate", [](const Tensor& attention, const Tensor& gate) { return Tensor(GateFunction::apply(attention, gate)); }, NoGil());
  m.def("run_gate", &run_gate, NoGil());
  m.def("run_gate_backward", &run_gate_backward, NoGil());
  m.def("layer_norm_node", &layer_norm_node, NoGil());
  m.def("layer_norm_forward", [or_empty](const Tensor& x, const MaybeTensor& weight, const MaybeTensor& bias, double eps) {
    TORCH_CHECK(norm_operands_fit(x, weight, bias, x.dim() ? x.size(-1) : 0), "layer_norm operands do not fit");
    const Tensor w = or_empty(weight), b = or_empty(bias);
    Normed n = norm_forward(rows_of(x, x.size(-1)), w.defined() ? w.contiguous() : w, b.defined() ? b.contiguous() : b, eps, true, x.sizes());
    return std::make_tuple(n.y, n.stats);
  }, NoGil());
  m.def("layer_norm_backward", [or_empty](const Tensor& dy, const Tensor& x, const MaybeTensor& weight, const MaybeTensor& bias,
                                          const Tensor& stats, const std::vector<bool>& need) {
    const Tensor w = or_empty(weight), rows = rows_of(x, x.size(-1));
    const auto affine = w.defined() ? w.scalar_type() : bias.has_value() ? bias->scalar_type() : x.scalar_type();
    NormGradients g = norm_backward(rows_of(dy.resolve_neg(), x.size(-1)), rows, w.defined() ? w.contiguous() : w, stats.contiguous(), affine,
                                    need[0], need[1], need[2]);
    auto maybe = [](const Tensor& t) { return t.defined() ? MaybeTensor(t) : MaybeTensor(); };
    return std::make_tuple(g.dx.defined() ? MaybeTensor(g.dx.view(x.sizes())) : MaybeTensor(), maybe(g.dweight), maybe(g.dbias));
  }, NoGil());
  m.def("pair_update", [](const Tensor& pair_in, const MaybeTensor& mask_in, bool outgoing, double in_eps, double out_eps,
                          std::vector<Tensor> parameters, const std::vector<int64_t>& bias_of) {
    // the passes read memory, which a lazily negated view does not describe
    const Tensor pair = pair_in.resolve_neg();
    const MaybeTensor mask = mask_in.has_value() ? MaybeTensor(mask_in->resolve_neg()) : mask_in;
    for (Tensor& p : parameters) p = p.resolve_neg();
    bool wanted = pair.requires_grad();
    for (const Tensor& p : parameters) wanted = wanted || p.requires_grad();
    if (at::GradMode::is_enabled() && wanted)
      return Tensor(UpdateFunction::apply(pair, mask, outgoing, in_eps, out_eps, at::TensorList(parameters), bias_of));
    return UpdateFunction::forward(nullptr, pair, mask, outgoing, in_eps, out_eps, parameters, bias_of);
  }, NoGil());
}
