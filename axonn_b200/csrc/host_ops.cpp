// Host paths of the operators that short calls are bound by: the same launches as the Python code beside them (ops/norm.py,
// ops/attention_cuda.py, intra_layer/fully_connected.py), with the questions asked and the tensors allocated in C++, and the
// normalisation's autograd node in C++, so that neither its backward nor the launches of a layer wait for the interpreter.
//
// A function returns None where the call is not one of those it takes; the caller then goes its general way, which accepts or
// refuses it.  Nothing is kept from one call to the next.  The kernels are those of the library that ops/_lib.py has loaded: bind()
// is given the addresses of its launchers.
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <ATen/autocast_mode.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <atomic>
#include <string>

#include "axonn_b200.h"

namespace {

using at::Tensor;
using std::optional;

// Launchers of the kernel library, of the types that its header gives them; bind() fills them in.  The header's number comes from
// the build, and a library of another one is not bound.
#define AXB_LAUNCHERS(X) \
  X(axb_norm_fwd, norm_fwd) X(axb_norm_bwd, norm_bwd) X(axb_add_norm_fwd, add_norm_fwd) X(axb_add_norm_bwd, add_norm_bwd) \
  X(axb_norm_grid, norm_grid) X(axb_gemm, gemm) X(axb_flash_attn_fwd, flash_fwd) X(axb_last_error, last_error)
#define AXB_DECLARE(symbol, name) decltype(&::symbol) name = nullptr;
AXB_LAUNCHERS(AXB_DECLARE)
PyObject *kernel_error = nullptr, *parameter_type = nullptr;
std::atomic<long long> launches{0};

struct KernelError : torch::PyTorchError {
  explicit KernelError(const std::string& what) : torch::PyTorchError(what) {}
  PyObject* python_type() override { return kernel_error; }
};

void check(int status, const char* what, int count = 1) {
  if (status != 0) {
    const char* msg = last_error();
    throw KernelError(std::string(what) + " failed (status " + std::to_string(status) + "): " + (msg ? msg : ""));
  }
  launches += count;
}

int dtype_code(const Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? 0 : t.scalar_type() == at::kHalf ? 1 : t.scalar_type() == at::kFloat ? 2 : -1;
}
const void* addr(const optional<Tensor>& t) { return t ? t->data_ptr() : nullptr; }
// The norm kernels read 16 bytes at a time.
bool on_16_bytes(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
Tensor dense(const Tensor& t) {
  const Tensor d = t.contiguous();
  return on_16_bytes(d) ? d : d.clone();
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Other Python threads run while this one allocates (the allocator may have to free blocks, which synchronises) and launches (a full
// launch queue lets the caller wait).
struct NoGil {
  PyThreadState* const state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// An ordinary CUDA tensor or parameter.
bool plain(PyObject* o) {
  return (Py_TYPE(o) == reinterpret_cast<PyTypeObject*>(THPVariableClass) || Py_TYPE(o) == reinterpret_cast<PyTypeObject*>(parameter_type)) &&
         THPVariable_Unpack(o).is_cuda();
}
// Neither a tracer nor a function transform looks at the call (the caller has asked for forward-mode levels and compilation).
bool observed() {
  const auto keys = c10::impl::tls_local_dispatch_key_set().included_;
  return keys.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || keys.has(c10::DispatchKey::FuncTorchDynamicLayerBackMode) ||
         torch::jit::tracer::isTracing();
}

// ---------------------------------------------------------------------------------------------------------------- norms
// y = norm(x), or h = x + delta and norm(h); stats [rows, 2] receives mean and reciprocal deviation of the rows.
void run_norm(const Tensor& x, const optional<Tensor>& delta, const Tensor& gamma, const optional<Tensor>& beta, double eps, bool rms,
              Tensor& h, Tensor& y, Tensor& stats) {
  const int H = static_cast<int>(x.size(-1)), rows = static_cast<int>(x.numel() / H), device = x.get_device();
  y = at::empty_like(x);
  stats = at::empty({rows, 2}, x.options().dtype(at::kFloat));
  if (delta) {
    h = at::empty_like(x);
    check(add_norm_fwd(x.data_ptr(), delta->data_ptr(), h.data_ptr(), gamma.data_ptr(), addr(beta), y.data_ptr(), stats.data_ptr<float>(),
                       rows, H, H, static_cast<float>(eps), rms, 0, dtype_code(x), device, stream()), "axb_add_norm_fwd");
  } else {
    h = x;
    check(norm_fwd(x.data_ptr(), gamma.data_ptr(), addr(beta), y.data_ptr(), stats.data_ptr<float>(), rows, H, H, static_cast<float>(eps),
                   rms, 0, dtype_code(x), device, stream()), "axb_norm_fwd");
  }
}

// Inputs: x, delta (may be missing), gamma, beta (may be missing).  Outputs: y, or h and y.
struct NormNode : torch::autograd::Function<NormNode> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const optional<Tensor>& delta,
                                                const Tensor& gamma, const optional<Tensor>& beta, double eps, bool rms) {
    Tensor h, y, stats;
    run_norm(x, delta, gamma, beta, eps, rms, h, y, stats);
    ctx->save_for_backward({h, gamma, stats});
    ctx->saved_data["rms"] = rms;
    ctx->saved_data["beta"] = beta.has_value();
    ctx->saved_data["delta"] = delta.has_value();
    if (delta) return {h, y};
    return {y};
  }
  // The kernels leave no graph: differentiating these gradients again is an error (first_derivative_only in ops/direct.py).
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    if (!at::GradMode::is_enabled()) return gradients(ctx, grads);
    torch::autograd::variable_list out, inputs = ctx->get_saved_variables();
    {
      at::AutoGradMode no_grad(false);
      out = gradients(ctx, grads);
    }
    inputs.insert(inputs.end(), grads.begin(), grads.end());
    if (!std::any_of(inputs.begin(), inputs.end(), [](const Tensor& t) { return t.defined() && t.requires_grad(); })) return out;
    const auto node = std::make_shared<torch::autograd::Error>("Norm: second derivatives are not implemented",
                                                               torch::autograd::collect_next_edges(inputs));
    for (Tensor& t : out)
      if (t.defined()) torch::autograd::set_history(t = t.detach(), node);
    return out;
  }
  static torch::autograd::variable_list gradients(torch::autograd::AutogradContext* ctx, const torch::autograd::variable_list& grads) {
    const auto saved = ctx->get_saved_variables();
    // what hooks (offloading, compression) give back may lie in another layout
    const Tensor h = dense(saved[0]), gamma = dense(saved[1]), stats = dense(saved[2]);
    const bool rms = ctx->saved_data["rms"].toBool(), delta = ctx->saved_data["delta"].toBool();
    const Tensor dy = dense(grads[delta ? 1 : 0]);
    const int H = static_cast<int>(h.size(-1)), rows = static_cast<int>(stats.size(0)), device = h.get_device();
    const int grid = norm_grid(device, rows);
    Tensor dx = at::empty_like(h), part = at::empty({2, grid, H}, stats.options()), dgamma = at::empty_like(gamma), dbeta;
    if (!rms) dbeta = at::empty_like(gamma);
    float* pa = part.data_ptr<float>();
    float* pb = pa + static_cast<size_t>(grid) * H;
    void* db = rms ? nullptr : dbeta.data_ptr();
    if (delta) {
      const Tensor dh = dense(grads[0]);
      check(add_norm_bwd(dy.data_ptr(), dh.data_ptr(), h.data_ptr(), gamma.data_ptr(), stats.data_ptr<float>(), dx.data_ptr(), nullptr, pa, pb,
                         dgamma.data_ptr(), db, rows, H, H, rms, 0, dtype_code(h), dtype_code(gamma), device, stream()),
            "axb_add_norm_bwd", 2);
    } else {
      check(norm_bwd(dy.data_ptr(), h.data_ptr(), gamma.data_ptr(), stats.data_ptr<float>(), dx.data_ptr(), nullptr, pa, pb, dgamma.data_ptr(),
                     db, rows, H, H, rms, 0, dtype_code(h), dtype_code(gamma), device, stream()), "axb_norm_bwd", 2);
    }
    return {dx, delta ? dx : Tensor(), dgamma, ctx->saved_data["beta"].toBool() ? dbeta : Tensor(), Tensor(), Tensor()};
  }
};

// norm(x, delta | None, gamma, beta | None, eps, rms) -> y, (h, y) with delta, or None
PyObject* py_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !plain(a[0]) || !plain(a[2]) || (a[1] != Py_None && !plain(a[1])) || (a[3] != Py_None && !plain(a[3])) || observed()) Py_RETURN_NONE;
  const Tensor &x = THPVariable_Unpack(a[0]), &gamma = THPVariable_Unpack(a[2]);
  optional<Tensor> delta, beta;
  if (a[1] != Py_None) delta = THPVariable_Unpack(a[1]);
  if (a[3] != Py_None) beta = THPVariable_Unpack(a[3]);
  const double eps = PyFloat_AsDouble(a[4]);
  if (eps == -1.0 && PyErr_Occurred()) return nullptr;
  const bool rms = PyObject_IsTrue(a[5]) == 1;
  const auto type = x.scalar_type();
  if (x.dim() == 0 || x.numel() == 0 || dtype_code(x) < 0 || !x.is_contiguous()) Py_RETURN_NONE;
  const int64_t H = x.size(-1);
  if (H > INT32_MAX || x.numel() / H > INT32_MAX) Py_RETURN_NONE;
  for (const Tensor* v : {&gamma, beta ? &*beta : &gamma})
    if (v->scalar_type() != type || v->dim() != 1 || v->size(0) != H || !v->is_contiguous() || v->device() != x.device() || !on_16_bytes(*v)) Py_RETURN_NONE;
  if (!on_16_bytes(x) || (delta && !on_16_bytes(*delta))) Py_RETURN_NONE;
  if (delta && (delta->sizes() != x.sizes() || delta->scalar_type() != type || !delta->is_contiguous() || delta->device() != x.device())) Py_RETURN_NONE;
  const bool grad = at::GradMode::is_enabled() && (x.requires_grad() || gamma.requires_grad() || (delta && delta->requires_grad()) ||
                                                   (beta && beta->requires_grad()));
  Tensor h, y, stats;
  {
    NoGil no_gil;
    if (grad) {
      const auto out = NormNode::apply(x, delta, gamma, beta, eps, rms);
      h = out[0];
      y = out[delta ? 1 : 0];
    } else {
      run_norm(x, delta, gamma, beta, eps, rms, h, y, stats);
    }
  }
  if (!delta) return THPVariable_Wrap(y);
  PyObject* pair = PyTuple_New(2);
  if (!pair) return nullptr;
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(h));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(y));
  return pair;
  END_HANDLE_TH_ERRORS
}

bool wants_grad(const Tensor& t) { return at::GradMode::is_enabled() && t.requires_grad(); }

// -------------------------------------------------------------------------------------------------------------- a linear layer
// linear(x, weight [n * k], bias | None, n, k, gelu) -> gelu?(x @ weight.T + bias) without a graph, or None
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !plain(a[0]) || !plain(a[1]) || (a[2] != Py_None && !plain(a[2])) || observed()) Py_RETURN_NONE;
  const Tensor &x = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]);
  optional<Tensor> b;
  if (a[2] != Py_None) b = THPVariable_Unpack(a[2]);
  const long rows_out = PyLong_AsLong(a[3]), k = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return nullptr;
  const bool gelu = PyObject_IsTrue(a[5]) == 1;
  const auto type = w.scalar_type();
  if ((type != at::kBFloat16 && type != at::kHalf) || x.scalar_type() != type || x.dim() == 0 || x.size(-1) != k || rows_out % 8 || k % 8 ||
      x.numel() == 0 || x.numel() / k > INT32_MAX || w.dim() != 1 || w.size(0) != static_cast<int64_t>(rows_out) * k || !x.is_contiguous() ||
      !w.is_contiguous() || w.device() != x.device() || wants_grad(x) || wants_grad(w) || at::autocast::is_autocast_enabled(at::kCUDA))
    Py_RETURN_NONE;
  if (b && (b->scalar_type() != type || b->device() != x.device() || !b->is_contiguous() || b->numel() != rows_out || wants_grad(*b))) Py_RETURN_NONE;
  c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = rows_out;
  const int code = type == at::kBFloat16 ? 0 : 1, epilogue = gelu ? (b ? 2 : 3) : (b ? 1 : 0);
  Tensor out;
  {
    NoGil no_gil;
    out = at::empty(shape, x.options());
    check(gemm(0, x.data_ptr(), w.data_ptr(), out.data_ptr(), addr(b), nullptr, static_cast<int>(x.numel() / k), static_cast<int>(rows_out),
               static_cast<int>(k), code, code, epilogue, 0, x.get_device(), stream()), "axb_gemm");
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------------------------ attention
// attention(qkv [B, S, G, q_per_kv + 2, D], scale) -> causal attention without a graph, or None
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !plain(a[0]) || observed()) Py_RETURN_NONE;
  const Tensor& qkv = THPVariable_Unpack(a[0]);
  const double scale = PyFloat_AsDouble(a[1]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  if (qkv.dim() != 5 || qkv.scalar_type() != at::kBFloat16 || !qkv.is_contiguous() || qkv.numel() == 0 || wants_grad(qkv)) Py_RETURN_NONE;
  const int64_t B = qkv.size(0), S = qkv.size(1), G = qkv.size(2), qpk = qkv.size(3) - 2, D = qkv.size(4);
  // 2^-100 < scale < 2^100, dense and on 16 bytes: see supported() in ops/attention_cuda.py
  if (qpk < 1 || (D != 64 && D != 128) || !(scale > 0x1p-100 && scale < 0x1p100) || reinterpret_cast<uintptr_t>(qkv.data_ptr()) % 16 ||
      std::max({B, S, G, qpk}) > INT32_MAX) Py_RETURN_NONE;
  Tensor out;
  {
    NoGil no_gil;
    out = at::empty({B, S, G * qpk, D}, qkv.options());
    const Tensor lse = at::empty({B, G * qpk, S}, qkv.options().dtype(at::kFloat));
    check(flash_fwd(qkv.data_ptr(), out.data_ptr(), lse.data_ptr<float>(), static_cast<int>(B), static_cast<int>(S), static_cast<int>(G),
                    static_cast<int>(qpk), static_cast<int>(D), static_cast<float>(scale), qkv.get_device(), stream()), "axb_flash_attn_fwd");
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// bind({launcher name: address}, KernelError, Parameter, axb_interface() of the library they are from) -> False if it is another one
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 4 && PyDict_Check(a[0]), "bind(launchers, error type, parameter type, interface)");
  if (PyLong_AsUnsignedLong(a[3]) != AXB_INTERFACE) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_FALSE;
  }
  const auto take = [&](const char* symbol, auto& fn) {
    PyObject* v = PyDict_GetItemString(a[0], symbol);
    TORCH_CHECK(v, "launcher ", symbol, " is missing");
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(PyLong_AsVoidPtr(v));
  };
#define AXB_TAKE(symbol, name) take(#symbol, name);
  AXB_LAUNCHERS(AXB_TAKE)
  Py_INCREF(a[1]); Py_INCREF(a[2]);
  kernel_error = a[1]; parameter_type = a[2];
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(launches.load()); }

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bind)), METH_FASTCALL, nullptr},
    {"norm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_norm)), METH_FASTCALL, nullptr},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_linear)), METH_FASTCALL, nullptr},
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL, nullptr},
    {"launches", py_launches, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "axonn_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_axonn_host() { return PyModule_Create(&module); }
