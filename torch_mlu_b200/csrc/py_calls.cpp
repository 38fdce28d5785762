// Direct Python entry points of the glue (module `libsdpa_b200_torch`), behind ops.py and sdp_choice.py: one native call from
// tensors to launched kernels. The calls these functions serve run for 5 to 20 us on the GPU when the problem is small (a
// decode step, a short prompt), and building the 90-field parameter block field by field through ctypes took the host
// 50 to 60 us per call; here a call costs 5 to 10 us, most of it the CUDA launches.
#include <ATen/PythonTorchFunctionTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>

#include "torch_glue.h"

namespace {

using at::Tensor;
using namespace b200_glue;

PyObject* g_status_error = nullptr;  // _cabi.SdpaError

const Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) throw torch::TypeError(c10::str(name, " must be a Tensor"));
  return THPVariable_Unpack(o);
}

c10::optional<Tensor> optional_tensor(PyObject* o, const char* name) {
  if (o == Py_None) return c10::nullopt;
  return tensor_arg(o, name);
}

int64_t int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}

double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}

bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}

c10::optional<double> optional_float(PyObject* o) {
  if (o == Py_None) return c10::nullopt;
  return float_arg(o);
}

void expect_args(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) throw torch::TypeError(c10::str("expected ", want, " arguments, got ", got));
}

PyObject* tuple_of(std::initializer_list<Tensor> tensors) {
  THPObjectPtr t(PyTuple_New(static_cast<Py_ssize_t>(tensors.size())));
  if (!t) throw python_error();
  Py_ssize_t i = 0;
  for (const Tensor& x : tensors) {
    PyObject* o = THPVariable_Wrap(x);
    if (o == nullptr) throw python_error();
    PyTuple_SET_ITEM(t.get(), i++, o);
  }
  return t.release();
}

// Runs `fn` (no Python inside) without the interpreter lock; a status of the C ABI becomes _cabi.SdpaError.
template <class F>
auto call(F&& fn) {
  try {
    pybind11::gil_scoped_release unlocked;
    return fn();
  } catch (const StatusError& e) {
    if (g_status_error == nullptr) throw;
    THPObjectPtr err(PyObject_CallFunction(g_status_error, "is", e.status(), e.what_without_backtrace()));
    if (err) PyErr_SetObject(g_status_error, err.get());
    throw python_error();
  }
}

// keep-masks of a call: (rows, cols, dropout_p), or None for rows
struct KeepArgs {
  KeepMasks masks;
  bool given = false;
  KeepArgs(PyObject* rows, PyObject* cols, PyObject* p) {
    if (rows == Py_None) return;
    masks.rows = tensor_arg(rows, "keep_rows");
    masks.cols = tensor_arg(cols, "keep_cols");
    masks.p = float_arg(p);
    given = true;
  }
  const KeepMasks* get() const { return given ? &masks : nullptr; }
};

// dense_forward(q, k, v, is_causal, scale, allow_gqa, kernel, num_splits, sm_margin, keep_rows, keep_cols, dropout_p, bias)
PyObject* py_dense_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 13);
  const Tensor &q = tensor_arg(a[0], "query"), &k = tensor_arg(a[1], "key"), &v = tensor_arg(a[2], "value");
  const bool causal = bool_arg(a[3]), gqa = bool_arg(a[5]);
  const double scale = scale_or_default(q, optional_float(a[4]));
  const KeepArgs keep(a[9], a[10], a[11]);
  const c10::optional<Tensor> bias = optional_tensor(a[12], "bias");
  ForwardOptions opt;
  opt.kernel = static_cast<int>(int_arg(a[6]));
  opt.num_splits = static_cast<int>(int_arg(a[7]));
  opt.sm_margin = static_cast<int>(int_arg(a[8]));
  opt.keep = keep.get();
  opt.bias = bias.has_value() ? &*bias : nullptr;
  auto r = call([&] { return dense_forward(q, k, v, causal, scale, gqa, opt); });
  return tuple_of({std::get<0>(r), std::get<1>(r)});
  END_HANDLE_TH_ERRORS
}

struct BackwardArgs {
  KeepArgs keep;
  c10::optional<Tensor> bias, dbias, bias_t;
  BackwardOptions opt;
  // keep_rows, keep_cols, dropout_p, bias, dbias, bias_t, deterministic (-1 / 0 / 1)
  explicit BackwardArgs(PyObject* const* a)
      : keep(a[0], a[1], a[2]), bias(optional_tensor(a[3], "bias")), dbias(optional_tensor(a[4], "dbias")),
        bias_t(optional_tensor(a[5], "bias_t")) {
    opt.keep = keep.get();
    opt.bias = bias.has_value() ? &*bias : nullptr;
    opt.dbias = dbias.has_value() ? &*dbias : nullptr;
    opt.bias_t = bias_t.has_value() ? &*bias_t : nullptr;
    opt.deterministic = static_cast<int>(int_arg(a[6]));
  }
};

// dense_backward(dout, q, k, v, out, lse, is_causal, scale, <BackwardArgs>)
PyObject* py_dense_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 15);
  const Tensor &dout = tensor_arg(a[0], "grad_out"), &q = tensor_arg(a[1], "query"), &k = tensor_arg(a[2], "key"),
               &v = tensor_arg(a[3], "value"), &out = tensor_arg(a[4], "out"), &lse = tensor_arg(a[5], "logsumexp");
  const bool causal = bool_arg(a[6]);
  const double scale = float_arg(a[7]);
  const BackwardArgs more(a + 8);
  auto r = call([&] { return dense_backward(dout, q, k, v, out, lse, causal, scale, more.opt); });
  return tuple_of({std::get<0>(r), std::get<1>(r), std::get<2>(r)});
  END_HANDLE_TH_ERRORS
}

// varlen_forward(q, k, v, cu_q, cu_k, max_q, max_k, is_causal, scale, keep_rows, keep_cols, dropout_p, bias)
PyObject* py_varlen_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 13);
  const Tensor &q = tensor_arg(a[0], "query"), &k = tensor_arg(a[1], "key"), &v = tensor_arg(a[2], "value"),
               &cu_q = tensor_arg(a[3], "cu_seqlens_q"), &cu_k = tensor_arg(a[4], "cu_seqlens_k");
  const int64_t max_q = int_arg(a[5]), max_k = int_arg(a[6]);
  const bool causal = bool_arg(a[7]);
  const double scale = scale_or_default(q, optional_float(a[8]));
  const KeepArgs keep(a[9], a[10], a[11]);
  const c10::optional<Tensor> bias = optional_tensor(a[12], "bias");
  ForwardOptions opt;
  opt.keep = keep.get();
  opt.bias = bias.has_value() ? &*bias : nullptr;
  auto r = call([&] { return varlen_forward(q, k, v, cu_q, cu_k, max_q, max_k, causal, scale, opt); });
  return tuple_of({std::get<0>(r), std::get<1>(r)});
  END_HANDLE_TH_ERRORS
}

// varlen_backward(dout, q, k, v, out, lse, cu_q, cu_k, max_q, max_k, is_causal, scale, <BackwardArgs>)
PyObject* py_varlen_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 19);
  const Tensor &dout = tensor_arg(a[0], "grad_out"), &q = tensor_arg(a[1], "query"), &k = tensor_arg(a[2], "key"),
               &v = tensor_arg(a[3], "value"), &out = tensor_arg(a[4], "out"), &lse = tensor_arg(a[5], "logsumexp"),
               &cu_q = tensor_arg(a[6], "cu_seqlens_q"), &cu_k = tensor_arg(a[7], "cu_seqlens_k");
  const int64_t max_q = int_arg(a[8]), max_k = int_arg(a[9]);
  const bool causal = bool_arg(a[10]);
  const double scale = float_arg(a[11]);
  const BackwardArgs more(a + 12);
  auto r = call([&] { return varlen_backward(dout, q, k, v, out, lse, cu_q, cu_k, max_q, max_k, causal, scale, more.opt); });
  return tuple_of({std::get<0>(r), std::get<1>(r), std::get<2>(r)});
  END_HANDLE_TH_ERRORS
}

// flash_attention_forward(q, k, v, cu_q, cu_k, max_q, max_k, is_causal, scale): the packed operator without dropout, with
// its five results
PyObject* py_flash_attention_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 9);
  const Tensor &q = tensor_arg(a[0], "query"), &k = tensor_arg(a[1], "key"), &v = tensor_arg(a[2], "value"),
               &cu_q = tensor_arg(a[3], "cu_seqlens_q"), &cu_k = tensor_arg(a[4], "cu_seqlens_k");
  const int64_t max_q = int_arg(a[5]), max_k = int_arg(a[6]);
  const bool causal = bool_arg(a[7]);
  const double scale = scale_or_default(q, optional_float(a[8]));
  auto r = call([&] { return varlen_forward_with_dropout(q, k, v, cu_q, cu_k, max_q, max_k, 0.0, causal, scale); });
  return tuple_of({r.out, r.lse, r.seed, r.offset, r.debug});
  END_HANDLE_TH_ERRORS
}

// sdpa(q, k, v, attn_mask, dropout_p, is_causal, scale): the output, or None when the call is not served here
PyObject* py_sdpa(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 7);
  // a subclass, or a mode with __torch_function__, sees the operators of the Python procedure
  if (at::impl::torch_function_mode_enabled()) Py_RETURN_NONE;
  for (int i = 0; i < 4; ++i)
    if (!(i == 3 && a[3] == Py_None) && !THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
  auto number = [](PyObject* o) { return PyFloat_Check(o) || PyLong_Check(o); };
  if (!number(a[4]) || (a[6] != Py_None && !number(a[6]))) Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
  const c10::optional<Tensor> mask = optional_tensor(a[3], "attn_mask");
  const double p = float_arg(a[4]);
  const bool causal = bool_arg(a[5]);
  const c10::optional<double> scale = optional_float(a[6]);
  Tensor out = call([&] { return sdpa(q, k, v, mask, p, causal, scale); });
  if (!out.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// status_word(device index): the int32 tensor the kernels launched through this module report time-outs in
PyObject* py_status_word(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect_args(n, 1);
  return THPVariable_Wrap(status_word(static_cast<int>(int_arg(a[0]))));
  END_HANDLE_TH_ERRORS
}

PyObject* py_set_status_error(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XDECREF(g_status_error);
  g_status_error = cls;
  Py_RETURN_NONE;
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    FAST("dense_forward", py_dense_forward),
    FAST("dense_backward", py_dense_backward),
    FAST("varlen_forward", py_varlen_forward),
    FAST("varlen_backward", py_varlen_backward),
    FAST("flash_attention_forward", py_flash_attention_forward),
    FAST("sdpa", py_sdpa),
    FAST("status_word", py_status_word),
    {"set_status_error", py_set_status_error, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "libsdpa_b200_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_libsdpa_b200_torch(void) { return PyModule_Create(&g_module); }
