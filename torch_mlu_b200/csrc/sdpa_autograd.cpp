// Autograd formulas of the attention operators and the scaled_dot_product_attention front end, in C++: a training step on
// short sequences is bound by the host work around four kernels of a few microseconds each, and the Python versions of
// these wrappers (torch.library.register_autograd, a torch.autograd.Function, the choice function's twenty checks) took
// 200 to 300 us per step where this file takes about 20.
#include <ATen/ExpandUtils.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/library.h>

#include "torch_glue.h"

namespace b200_glue {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// An ordinary CUDA tensor, without wrappers, lazy conjugate or negative bits or a Python dispatch of its own: what the kernels
// may be handed without the dispatcher.
bool plain(const Tensor& t) {
  constexpr c10::DispatchKeySet ordinary(
      {c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA});
  return ordinary.has_all(t.key_set());
}

// Nobody wants to see the operators of this thread: no dispatch mode, functional transform, functionalisation or tracing, and
// autograd not switched off below the dispatcher.
bool dispatcher_may_be_skipped() {
  const auto tls = c10::impl::tls_local_dispatch_key_set();
  return c10::default_included_set.has_all(tls.included_) && !tls.excluded_.has(c10::DispatchKey::AutogradFunctionality) &&
         !c10::impl::TorchDispatchModeTLS::any_modes_set() && !torch::jit::tracer::isTracing();
}

// ------------------------------------------------------------------------- additive bias
int64_t ceil8(int64_t n) { return (n + 7) / 8 * 8; }

// A copy of the bias (of q's type and device) with rows padded to a multiple of 8 keys. The kernel reads `seqlen_k` keys of every row, so the
// bias must have them, or one for all.
Tensor padded_copy(const Tensor& attn_bias, const Tensor& q, int64_t seqlen_k) {
  TORCH_CHECK(attn_bias.size(-1) == 1 || attn_bias.size(-1) == seqlen_k, "attn_bias must have one key or the ", seqlen_k, " of key, it has ",
              attn_bias.size(-1));
  std::vector<int64_t> sizes(attn_bias.sizes().begin(), attn_bias.sizes().end());
  sizes.back() = ceil8(seqlen_k);
  int64_t own[4] = {1, 1, 1, seqlen_k}, strides[4] = {0, 0, 0, attn_bias.size(-1) == 1 ? 0 : attn_bias.stride(-1)};
  const int64_t d = attn_bias.dim();
  for (int64_t i = 4 - d, j = 0; i < 3; ++i, ++j) {
    own[i] = attn_bias.size(j);
    strides[i] = attn_bias.stride(j);
  }
  Tensor buf = at::detail::empty_cuda(sizes, q.scalar_type(), q.device(), c10::nullopt);
  check_status(sdpa_b200_pad_bias(attn_bias.data_ptr(), strides[0], strides[1], strides[2], strides[3], static_cast<int32_t>(own[0]),
                                  static_cast<int32_t>(own[1]), static_cast<int32_t>(own[2]), static_cast<int32_t>(seqlen_k), buf.data_ptr(),
                                  sizes.back(), at::cuda::getCurrentCUDAStream(q.get_device()).stream()),
               "sdpa_b200_pad_bias");
  return buf;
}

// The gradient of a bias of shape `sizes` out of that of its expansion: summed over what it is broadcast along.
Tensor summed_bias_gradient(const Tensor& dbias, const std::vector<int64_t>& sizes) {
  const int64_t d = static_cast<int64_t>(sizes.size());
  int64_t own[4] = {1, 1, 1, 1};
  for (int64_t i = 4 - d, j = 0; j < d; ++i, ++j) own[i] = sizes[j];
  const bool over_batch = own[0] != dbias.size(0), over_heads = own[1] != dbias.size(1);
  if (!(over_batch || over_heads) || own[2] != dbias.size(2) || own[3] != dbias.size(3)) return at::sum_to(dbias, sizes);
  c10::cuda::CUDAGuard device_guard(dbias.device());
  Tensor sum = at::detail::empty_cuda(sizes, dbias.scalar_type(), dbias.device(), c10::nullopt);
  check_status(sdpa_b200_sum_bias_grad(dbias.data_ptr(), dbias.stride(0), dbias.stride(1), dbias.stride(2), static_cast<int32_t>(dbias.size(0)),
                                       static_cast<int32_t>(dbias.size(1)), static_cast<int32_t>(dbias.size(2)), static_cast<int32_t>(dbias.size(3)),
                                       over_batch, over_heads, sum.data_ptr(), dbias.scalar_type() == at::kHalf ? SDPA_B200_F16 : SDPA_B200_BF16,
                                       at::cuda::getCurrentCUDAStream(dbias.get_device()).stream()),
               "sdpa_b200_sum_bias_grad");
  return sum;
}

// The additive bias as a [B, H, Lq, Lk] view the kernels can read: broadcast dimensions keep stride 0, rows start 16-byte
// aligned and are readable up to the next multiple of 8 keys. Undefined for a bias without that layout. `padded`: its rows are
// as long as padded_copy() and mask_bias() make them.
Tensor readable_bias(const Tensor& attn_bias, const Tensor& q, int64_t seqlen_k, bool padded) {
  TORCH_CHECK(attn_bias.scalar_type() == q.scalar_type() && attn_bias.device() == q.device(),
              "attn_bias must have the dtype and device of query");
  const int64_t full[4] = {q.size(0), q.size(1), q.size(2), seqlen_k};
  // the view at once: narrowing and expanding are two calls of a microsecond, here and in the backward
  int64_t strides[4] = {0, 0, 0, 0};
  bool ok = attn_bias.dim() >= 1 && attn_bias.size(-1) == (padded ? ceil8(seqlen_k) : seqlen_k) && attn_bias.stride(-1) == 1 &&
            (padded || seqlen_k % 8 == 0) && reinterpret_cast<uintptr_t>(attn_bias.data_ptr()) % 16 == 0;
  for (int64_t i = 4 - attn_bias.dim(), j = 0; ok && i < 4; ++i, ++j) {
    const int64_t n = attn_bias.size(j);
    strides[i] = n == 1 && i < 3 ? 0 : attn_bias.stride(j);
    ok = i == 3 || ((n == 1 || n == full[i]) && strides[i] % 8 == 0);
  }
  return ok ? attn_bias.as_strided(full, strides) : Tensor();
}

Tensor prepare_bias(const Tensor& attn_bias, const Tensor& q, int64_t seqlen_k, bool padded) {
  TORCH_CHECK(attn_bias.dim() >= 1 && attn_bias.dim() <= 4, "attn_bias must have one to four dimensions, it has ", attn_bias.dim());
  const Tensor view = readable_bias(attn_bias, q, seqlen_k, padded);
  if (view.defined()) return view;
  return readable_bias(padded_copy(padded ? attn_bias.narrow(-1, 0, seqlen_k) : attn_bias, q, seqlen_k), q, seqlen_k, true);
}

// A boolean attn_mask (true = take part) as a bias of 0 / -inf with rows padded to a multiple of 8: one kernel over the mask's
// own elements (broadcast dimensions have size 1).
Tensor mask_bias(const Tensor& mask, const Tensor& q, int64_t seqlen_k) {
  const int64_t full[4] = {q.size(0), q.size(1), q.size(2), seqlen_k};
  const Tensor m = mask.expand(full);
  int64_t own[4];
  for (int i = 0; i < 3; ++i) own[i] = m.stride(i) == 0 ? 1 : full[i];
  own[3] = ceil8(seqlen_k);
  Tensor buf = at::detail::empty_cuda(own, q.scalar_type(), q.device(), c10::nullopt);
  check_status(sdpa_b200_mask_to_bias(m.data_ptr(), m.stride(0), m.stride(1), m.stride(2), m.stride(3), static_cast<int32_t>(own[0]),
                                      static_cast<int32_t>(own[1]), static_cast<int32_t>(own[2]), static_cast<int32_t>(seqlen_k),
                                      buf.data_ptr(), own[3], q.scalar_type() == at::kHalf ? SDPA_B200_F16 : SDPA_B200_BF16,
                                      at::cuda::getCurrentCUDAStream(q.get_device()).stream()),
               "sdpa_b200_mask_to_bias");
  return buf;
}

// [B, H, Lk, Lq] view of a copy of `bias` with keys and queries exchanged, for the dK/dV kernel, whose threads own keys and
// read consecutive queries; undefined for a bias that does not depend on the query.
Tensor transposed_bias(const Tensor& bias) {
  if (bias.stride(2) == 0) return {};
  const int64_t B = bias.size(0), H = bias.size(1), Lq = bias.size(2), Lk = bias.size(3);
  const int64_t nb = bias.stride(0) == 0 ? 1 : B, nh = bias.stride(1) == 0 ? 1 : H, lq8 = ceil8(Lq);
  Tensor buf = at::detail::empty_cuda({nb, nh, Lk, lq8}, bias.scalar_type(), bias.device(), c10::nullopt);
  check_status(sdpa_b200_transpose_bias(bias.data_ptr(), bias.stride(0), bias.stride(1), bias.stride(2), static_cast<int32_t>(nb),
                                        static_cast<int32_t>(nh), static_cast<int32_t>(Lq), static_cast<int32_t>(Lk),
                                        buf.data_ptr(), lq8, at::cuda::getCurrentCUDAStream(bias.get_device()).stream()),
               "sdpa_b200_transpose_bias");
  return buf.narrow(-1, 0, Lq).expand({B, H, Lk, Lq});
}

// The backward of a dense call with a bias: dq, dk, dv and, when it is wanted, the gradient of the bias before it is summed over
// the dimensions the bias is broadcast along.
std::tuple<Tensor, Tensor, Tensor, Tensor> bias_backward(const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v,
                                                         const Tensor& bias, const Tensor& out, const Tensor& lse, bool bias_padded,
                                                         bool causal, bool want_dbias, double scale) {
  c10::cuda::CUDAGuard device_guard(q.device());
  const Tensor view = prepare_bias(bias, q, k.size(2), bias_padded);
  Tensor dbias;
  if (want_dbias) {
    const int64_t sizes[4] = {q.size(0), q.size(1), q.size(2), ceil8(k.size(2))};
    // under a causal mask zero-filled, since the kernels skip what it hides; else they write every pair
    dbias = (causal ? at::zeros(sizes, q.options()) : at::empty(sizes, q.options())).narrow(-1, 0, k.size(2));
  }
  const Tensor bias_t = transposed_bias(view);
  BackwardOptions opt;
  opt.bias = &view;
  opt.dbias = &dbias;
  opt.bias_t = &bias_t;
  auto [dq, dk, dv] = dense_backward(grad_out, q, k, v, out, lse, causal, scale, opt);
  if (!want_dbias) dbias = at::empty({0}, q.options());
  return {dq, dk, dv, dbias};
}

// ------------------------------------------------------------------------- autograd
using DenseBackwardOp = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                           const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t, double,
                                                           bool, const Tensor&, const Tensor&, c10::optional<double>);

// What a backward needs besides the incoming gradient. One form for all calls: dense, dense with an additive bias, packed.
struct BackwardCall {
  bool packed = false, causal = false, has_bias = false, bias_padded = false, want_dbias = false;
  int64_t max_q = 0, max_k = 0;
  double scale = 1.0, dropout_p = 0.0;
  std::vector<int64_t> bias_sizes;  // shape of the attn_mask argument, when its gradient is wanted
};
struct BackwardTensors {
  Tensor q, k, v, out, lse;
  Tensor cu_q, cu_k;    // packed
  Tensor seed, offset;  // without a bias
  Tensor bias;          // as saved by the node

  // those the form has, in a fixed order
  std::vector<Tensor*> used(const BackwardCall& c) {
    std::vector<Tensor*> t = {&q, &k, &v, &out, &lse};
    if (c.packed) t.insert(t.end(), {&cu_q, &cu_k});
    if (c.has_bias) t.push_back(&bias);
    else t.insert(t.end(), {&seed, &offset});
    return t;
  }
};

// Gradients of query, key, value and (with a bias) the bias, undefined where `needs` says so.
variable_list run_backward(const Tensor& go, const BackwardCall& c, const BackwardTensors& t, const std::vector<bool>& needs) {
  variable_list result(needs.size());
  if (!go.defined()) return result;
  Tensor dq, dk, dv;
  // Through the operators where somebody wants to see them: create_graph=True, dispatch modes, tracing, wrapped gradients
  bool direct = !at::GradMode::is_enabled() && dispatcher_may_be_skipped();
  for (const Tensor* x : {&go, &t.q, &t.k, &t.v, &t.out, &t.lse}) direct = direct && plain(*x);
  if (c.has_bias) {
    Tensor dbias;
    if (direct && plain(t.bias)) {
      at::AutoDispatchBelowADInplaceOrView guard;
      std::tie(dq, dk, dv, dbias) = bias_backward(go, t.q, t.k, t.v, t.bias, t.out, t.lse, c.bias_padded, c.causal, c.want_dbias, c.scale);
      if (c.want_dbias) result[3] = summed_bias_gradient(dbias, c.bias_sizes);
    } else {
      static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("b200_sdpa::_bias_attention_backward", "").typed<decltype(bias_backward)>();
      std::tie(dq, dk, dv, dbias) = op.call(go, t.q, t.k, t.v, t.bias, t.out, t.lse, c.bias_padded, c.causal, c.want_dbias, c.scale);
    }
    if (c.want_dbias && !result[3].defined()) result[3] = at::sum_to(dbias, c.bias_sizes);
  } else if (!direct) {
    if (c.packed) {
      static auto op = c10::Dispatcher::singleton()
                           .findSchemaOrThrow("b200_sdpa::_flash_attention_backward", "").typed<DenseBackwardOp>();
      std::tie(dq, dk, dv) = op.call(go, t.q, t.k, t.v, t.out, t.lse, t.cu_q, t.cu_k, c.max_q, c.max_k, c.dropout_p, c.causal, t.seed,
                                     t.offset, c.scale);
    } else {
      static auto op = c10::Dispatcher::singleton()
                           .findSchemaOrThrow("b200_sdpa::_scaled_dot_product_flash_attention_backward", "").typed<DenseBackwardOp>();
      const Tensor none = at::empty({0}, t.q.options().dtype(at::kInt));
      std::tie(dq, dk, dv) = op.call(go, t.q, t.k, t.v, t.out, t.lse, none, none, c.max_q, c.max_k, c.dropout_p, c.causal, t.seed,
                                     t.offset, c.scale);
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView guard;
    if (c.packed)
      std::tie(dq, dk, dv) = varlen_backward_with_dropout(go, t.q, t.k, t.v, t.out, t.lse, t.cu_q, t.cu_k, c.max_q, c.max_k, c.dropout_p,
                                                          c.causal, t.seed, t.offset, c.scale);
    else
      std::tie(dq, dk, dv) = dense_backward_with_dropout(go, t.q, t.k, t.v, t.out, t.lse, c.dropout_p, c.causal, t.seed, t.offset,
                                                         c.scale);
  }
  if (needs[0]) result[0] = dq;
  if (needs[1]) result[1] = dk;
  if (needs[2]) result[2] = dv;
  return result;
}

struct AttentionBackward : public torch::autograd::Node {
  SavedVariable q, k, v, out, lse, cu_q, cu_k, seed, offset;
  // dense with a bias: the caller's own tensor (a change in place before the backward is noticed), or the padded buffer made from
  // it, beside which a floating-point one is kept for the same check
  SavedVariable bias, bias_given;
  BackwardCall call;

  std::string name() const override { return "B200AttentionBackward"; }
  std::array<SavedVariable*, 11> saved() { return {&q, &k, &v, &out, &lse, &cu_q, &cu_k, &seed, &offset, &bias, &bias_given}; }

  BackwardTensors unpack() {
    bias_given.unpack();  // raises when it has been changed
    return {q.unpack(), k.unpack(), v.unpack(), out.unpack(shared_from_this()), lse.unpack(), cu_q.unpack(),
            cu_k.unpack(), seed.unpack(), offset.unpack(), bias.unpack()};
  }

  std::vector<bool> needs() const {
    std::vector<bool> n(num_outputs());
    for (size_t i = 0; i < n.size(); ++i) n[i] = task_should_compute_output(i);
    return n;
  }

  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : saved()) s->reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return variable_list(num_outputs());
    return run_backward(grads[0], call, unpack(), needs());
  }

  // Compiled autograd: everything a recorded call depends on, then the call itself, recorded as a function of the incoming
  // gradient and the saved tensors.
  void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
    for (SavedVariable* s : const_cast<AttentionBackward*>(this)->saved()) args.collect(*s, /*is_output=*/s == &out);
    args.collect(call.bias_sizes);
    for (const bool flag : {call.packed, call.causal, call.has_bias, call.bias_padded, call.want_dbias}) args.collect(flag);
    args.collect(call.max_q);
    args.collect(call.max_k);
    args.collect(call.scale);
    args.collect(call.dropout_p);
  }

  variable_list apply_with_saved(const variable_list& inputs, torch::dynamo::autograd::SwapSavedVariables& swap) override {
    namespace ca = torch::dynamo::autograd;
    for (SavedVariable* s : saved()) swap.before(*s);
    BackwardTensors tensors = unpack();
    ca::ivalue_list args;
    std::vector<at::TypePtr> types;
    for (const Tensor* t : tensors.used(call)) {
      args.push_back(ca::IValuePacker<Tensor>::pack(*t));
      types.push_back(ca::IValuePacker<Tensor>::packed_type());
    }
    auto recorded = [c = call, n = needs()](const variable_list& grads, const ca::ivalue_list& a) {
      BackwardTensors t;
      size_t i = 0;
      for (Tensor* x : t.used(c)) *x = a[i++].toTensor();
      return run_backward(grads[0], c, t, n);
    };
    const auto& compiler = ca::getPyCompilerInterface();
    const std::string fn = compiler->bind_function(swap.get_py_compiler(), name(), recorded, types, /*is_custom_function=*/true);
    variable_list result = compiler->call_function(
        swap.get_py_compiler(), "apply_functional", fn, inputs, args,
        ca::IValuePacker<std::vector<std::optional<torch::autograd::InputMetadata>>>::pack(ca::get_input_metadata(next_edges())));
    for (SavedVariable* s : saved()) swap.after(*s);
    return result;
  }
};

bool any_requires_grad(std::initializer_list<const Tensor*> tensors) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : tensors)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// There is no forward-mode formula: an input with a tangent must not lose it in silence.
void refuse_tangents(std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(/*level=*/0).defined(),
                                "forward-mode differentiation of the attention operators is not implemented");
}

// The nodes below are not made for the levels of torch.func: a second derivative would be lost.
void refuse_transforms(std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    TORCH_CHECK(!t->key_set().has(c10::DispatchKey::FuncTorchGradWrapper),
                "the attention operators cannot be differentiated with torch.func transforms (grad, vjp, jacrev, ...)");
}

// Hangs a node behind `out` (a fresh tensor). `bias_arg`: the attn_mask the caller gave, or undefined.
std::shared_ptr<AttentionBackward> new_node(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias_arg, bool causal,
                                            double scale, double dropout_p) {
  std::shared_ptr<AttentionBackward> node(new AttentionBackward(), torch::autograd::deleteNode);
  node->set_next_edges(bias_arg.defined() ? torch::autograd::collect_next_edges(q, k, v, bias_arg)
                                          : torch::autograd::collect_next_edges(q, k, v));
  node->q = SavedVariable(q, false);
  node->k = SavedVariable(k, false);
  node->v = SavedVariable(v, false);
  node->call.causal = causal;
  node->call.scale = scale;
  node->call.dropout_p = dropout_p;
  return node;
}

void finish_node(const std::shared_ptr<AttentionBackward>& node, Tensor& out, const Tensor& lse, const Tensor& seed,
                 const Tensor& offset) {
  torch::autograd::set_history(out, node);
  node->out = SavedVariable(out, true);
  node->lse = SavedVariable(lse, false);
  node->seed = SavedVariable(seed, false);
  node->offset = SavedVariable(offset, false);
}

using DenseOp = std::tuple<Tensor, Tensor, Tensor, Tensor, int64_t, int64_t, Tensor, Tensor, Tensor>(
    const Tensor&, const Tensor&, const Tensor&, double, bool, bool, c10::optional<double>);
using PackedOp = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                                    const Tensor&, int64_t, int64_t, double, bool, bool,
                                                                    c10::optional<double>);

std::tuple<Tensor, Tensor, Tensor, Tensor, int64_t, int64_t, Tensor, Tensor, Tensor> dense_with_grad(
    const Tensor& q, const Tensor& k, const Tensor& v, double dropout_p, bool is_causal, bool return_debug_mask,
    c10::optional<double> scale) {
  refuse_tangents({&q, &k, &v});
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("b200_sdpa::_scaled_dot_product_flash_attention", "").typed<DenseOp>();
  auto r = [&] {
    at::AutoDispatchBelowADInplaceOrView guard;
    return op.call(q, k, v, dropout_p, is_causal, return_debug_mask, scale);
  }();
  if (any_requires_grad({&q, &k, &v})) {
    refuse_transforms({&q, &k, &v});
    auto node = new_node(q, k, v, Tensor(), is_causal, scale_or_default(q, scale), dropout_p);
    node->call.max_q = q.size(2);
    node->call.max_k = k.size(2);
    Tensor lse = std::get<1>(r);
    if (lse.size(2) != q.size(2)) lse = lse.slice(2, 0, q.size(2)).contiguous();
    finish_node(node, std::get<0>(r), lse, std::get<6>(r), std::get<7>(r));
  }
  return r;
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> packed_with_grad(const Tensor& q, const Tensor& k, const Tensor& v,
                                                                    const Tensor& cu_q, const Tensor& cu_k, int64_t max_q,
                                                                    int64_t max_k, double dropout_p, bool is_causal,
                                                                    bool return_debug_mask, c10::optional<double> scale) {
  refuse_tangents({&q, &k, &v});
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("b200_sdpa::_flash_attention_forward", "").typed<PackedOp>();
  auto r = [&] {
    at::AutoDispatchBelowADInplaceOrView guard;
    return op.call(q, k, v, cu_q, cu_k, max_q, max_k, dropout_p, is_causal, return_debug_mask, scale);
  }();
  if (any_requires_grad({&q, &k, &v})) {
    refuse_transforms({&q, &k, &v});
    auto node = new_node(q, k, v, Tensor(), is_causal, scale_or_default(q, scale), dropout_p);
    node->call.packed = true;
    node->call.max_q = max_q;
    node->call.max_k = max_k;
    node->cu_q = SavedVariable(cu_q, false);
    node->cu_k = SavedVariable(cu_k, false);
    finish_node(node, std::get<0>(r), std::get<1>(r), std::get<2>(r), std::get<3>(r));
  }
  return r;
}

// Shapes of the backward operators' results, for recorders that call them on tensors without data
Tensor meta_like(const Tensor& t) {  // memory order of the kernels' outputs: [B, L, H, D] for a dense [B, H, L, D]
  if (t.dim() != 4) return at::empty_symint(t.sym_sizes(), t.options());
  const auto H = t.sym_size(1), L = t.sym_size(2), D = t.sym_size(3);
  return at::empty_strided_symint(t.sym_sizes(), {L * H * D, D, H * D, 1}, t.options());
}

std::tuple<Tensor, Tensor, Tensor> meta_backward(const Tensor&, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor&,
                                                 const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t, double, bool, const Tensor&,
                                                 const Tensor&, c10::optional<double>) {
  return {meta_like(q), meta_like(k), meta_like(v)};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> meta_bias_backward(const Tensor&, const Tensor& q, const Tensor& k, const Tensor& v,
                                                              const Tensor&, const Tensor&, const Tensor&, bool, bool, bool want_dbias,
                                                              double) {
  Tensor dbias = at::empty({0}, q.options());
  if (want_dbias) {
    const auto Lk = k.sym_size(2);
    dbias = at::empty_symint({q.sym_size(0), q.sym_size(1), q.sym_size(2), (Lk + 7) / 8 * 8}, q.options()).narrow_symint(-1, 0, Lk);
  }
  return {meta_like(q), meta_like(k), meta_like(v), dbias};
}

bool broadcasts_to(const Tensor& t, const int64_t (&full)[4]) {
  const int64_t d = t.dim();
  for (int64_t i = 0; i < d; ++i) {
    const int64_t n = t.size(d - 1 - i);
    if (n != 1 && n != full[3 - i]) return false;
  }
  return true;
}

}  // namespace

// The checks are those of sdp_choice.py (sdp_utils.h:99-455): a call that fails one of them, or whose answer depends on more
// than they say (autocast, wrapped tensors, dispatch modes, transforms, tracing, a top-left causal mask over unequal lengths), gets
// an undefined tensor, and the Python function goes through the whole procedure with its warnings and errors.
Tensor sdpa(const Tensor& q, const Tensor& k, const Tensor& v, const c10::optional<Tensor>& attn_mask, double dropout_p,
            bool is_causal, c10::optional<double> scale) {
  const auto& ctx = at::globalContext();
  const bool flash = ctx.userEnabledFlashSDP(), efficient = ctx.userEnabledMemEfficientSDP();
  const bool has_mask = attn_mask.has_value() && attn_mask->defined();
  if (!(efficient || (flash && !has_mask))) return {};
  if (at::autocast::is_autocast_enabled(at::kCUDA) || !dispatcher_may_be_skipped()) return {};
  for (const Tensor* t : {&q, &k, &v}) {
    if (!plain(*t) || t->dim() != 4 || t->layout() != at::kStrided || t->stride(-1) != 1 || t->scalar_type() != q.scalar_type() ||
        t->size(0) != q.size(0) || t->size(1) != q.size(1) || t->size(3) != q.size(3) || t->device() != q.device())
      return {};
  }
  const auto dtype = q.scalar_type();
  const int64_t D = q.size(3), Lq = q.size(2), Lk = k.size(2);
  if ((dtype != at::kHalf && dtype != at::kBFloat16) || D < 64 || D > 256 || D % 8 != 0 || Lq == 0 || Lk == 0 || v.size(2) != Lk ||
      q.size(0) == 0 || q.size(1) == 0 || (is_causal && Lq != Lk))
    return {};
  if (at::cuda::getDeviceProperties(q.get_device())->major != 10) return {};
  const double sc = scale_or_default(q, scale);
  refuse_tangents({&q, &k, &v});

  if (!has_mask) {
    DropoutResult r = [&] {
      at::AutoDispatchBelowADInplaceOrView guard;
      return dense_forward_with_dropout(q, k, v, dropout_p, is_causal, false, sc, /*allow_gqa=*/false);
    }();
    if (any_requires_grad({&q, &k, &v})) {
      auto node = new_node(q, k, v, Tensor(), is_causal, sc, dropout_p);
      node->call.max_q = Lq;
      node->call.max_k = Lk;
      finish_node(node, r.out, r.lse, r.seed, r.offset);
    }
    return r.out;
  }

  const Tensor& mask = *attn_mask;
  const int64_t full[4] = {q.size(0), q.size(1), Lq, Lk};
  if (!efficient || D > 128 || dropout_p != 0.0 || mask.dim() < 1 || mask.dim() > 4 || !broadcasts_to(mask, full) || mask.stride(-1) != 1 ||
      !plain(mask) || mask.device() != q.device() ||
      !(mask.scalar_type() == at::kBool || at::isFloatingType(mask.scalar_type())))
    return {};
  refuse_tangents({&mask});
  c10::cuda::CUDAGuard device_guard(q.device());
  const bool boolean = mask.scalar_type() == at::kBool;
  const Tensor bias_arg = boolean ? Tensor() : mask.to(dtype);  // (differentiable) conversion of a bias of another type
  Tensor padded, out, lse;  // `padded`: the buffer the bias is read from where the argument itself cannot be
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    Tensor bias = boolean ? Tensor() : readable_bias(bias_arg, q, Lk, false);
    if (!bias.defined()) {
      padded = boolean ? mask_bias(mask, q, Lk) : padded_copy(bias_arg, q, Lk);
      bias = readable_bias(padded, q, Lk, true);
    }
    ForwardOptions opt;
    opt.bias = &bias;
    std::tie(out, lse) = dense_forward(q, k, v, is_causal, sc, /*allow_gqa=*/false, opt);
  }
  if (any_requires_grad({&q, &k, &v, &bias_arg})) {
    auto node = new_node(q, k, v, bias_arg, is_causal, sc, 0.0);
    node->call.has_bias = true;
    node->call.bias_padded = padded.defined();
    node->bias = SavedVariable(padded.defined() ? padded : bias_arg, false);
    if (padded.defined() && !boolean) node->bias_given = SavedVariable(bias_arg, false);
    if (bias_arg.defined() && bias_arg.requires_grad()) {
      node->call.want_dbias = true;
      node->call.bias_sizes = bias_arg.sizes().vec();
    }
    finish_node(node, out, lse, Tensor(), Tensor());
  }
  return out;
}

}  // namespace b200_glue

TORCH_LIBRARY_FRAGMENT(b200_sdpa, m) {
  m.def("_bias_attention_backward(Tensor grad_out, Tensor query, Tensor key, Tensor value, Tensor bias, Tensor out, Tensor logsumexp, "
        "bool bias_padded, bool is_causal, bool want_dbias, float scale) -> (Tensor, Tensor, Tensor, Tensor)");
}

TORCH_LIBRARY_IMPL(b200_sdpa, CUDA, m) {
  m.impl("_bias_attention_backward", b200_glue::bias_backward);
}

TORCH_LIBRARY_IMPL(b200_sdpa, Meta, m) {
  m.impl("_scaled_dot_product_flash_attention_backward", b200_glue::meta_backward);
  m.impl("_flash_attention_backward", b200_glue::meta_backward);
  m.impl("_bias_attention_backward", b200_glue::meta_bias_backward);
}

TORCH_LIBRARY_IMPL(b200_sdpa, AutogradCUDA, m) {
  m.impl("_scaled_dot_product_flash_attention", b200_glue::dense_with_grad);
  m.impl("_flash_attention_forward", b200_glue::packed_with_grad);
}
