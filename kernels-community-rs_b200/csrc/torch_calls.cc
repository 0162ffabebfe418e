// Native front of the dense calls for torch tensors: forward, backward and the differentiable attention function,
// from the Python call to the kernel launches without Python, DLPack or dispatcher steps in between. What bounds a
// small call is this host path: through the operator library and a Python autograd function a forward took 15 us and
// a training step 162 us of host time (B1 H4 S128 D64), most of it argument conversion, tensor exchange and Python
// frames. Every function here returns None for arguments outside the plain case (other types, other layouts, anything
// that is an error): interface.py then takes the operator route, which converts, packs and raises as it always did.
//
// The semantics are those of interface.py's `fwd`, `bwd` and `flash_attn_func`
// (flash-attn2-rs/tvm-ffi-ext/flash_attn2_rs/flash_attn_interface.py in the reference).
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pycfunction_helpers.h>

#include <cmath>

#include "fa2_b200.h"

namespace {

using at::Tensor;

Tensor empty(at::IntArrayRef shape, c10::ScalarType type, c10::Device dev) {
  return Tensor(at::detail::empty_cuda(shape, type, dev, std::nullopt));
}

// Scratch memory that a call can do without: undefined when there is none left (the call then takes more time, and sums
// in another order).
Tensor scratch(int64_t bytes, c10::Device dev) {
  try {
    return empty({bytes}, at::kByte, dev);
  } catch (const c10::OutOfMemoryError&) {
    return Tensor();
  }
}

// The kernels address a tensor by TMA: 16-byte aligned base, unit last stride, outer strides multiples of 8 elements
// (of dimensions longer than 1).
bool addressable(const Tensor& t) {
  if (reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
  const auto sh = t.sizes(), st = t.strides();
  if (st[3] != 1 && sh[3] > 1) return false;
  for (int i = 0; i < 3; ++i)
    if (sh[i] > 1 && (st[i] % 8 != 0 || st[i] < 0)) return false;
  return true;
}

// `t`, or a copy that the kernels can address.
Tensor laid_out(const Tensor& t) {
  return t.is_cuda() && t.layout() == c10::kStrided && t.dim() == 4 && !addressable(t) ? t.clone(at::MemoryFormat::Contiguous) : t;
}

void strides_of(const Tensor& t, int64_t out[3]) {
  const auto sh = t.sizes(), st = t.strides();
  for (int i = 0; i < 3; ++i) out[i] = sh[i] > 1 ? st[i] : 0;  // the stride of a size-1 dimension is never used
}

struct Options {
  bool has_scale = false;
  double scale = 0.0;
  bool causal = false;
  int64_t left = -1, right = -1;
  double softcap = 0.0;
  Tensor alibi;  // undefined: none
};

// The trace of an autograd function holds what its forward does, down to an operation that made the output.
bool tracing() { return torch::jit::tracer::isTracing(); }

// Calls that only the autograd function in Python answers rightly: a tracer records that function (the output of a native
// call would be a constant to it), and it refuses function transforms and forward-mode derivatives (a native call would
// hand their wrappers' storage to the kernels, or drop them). Slopes that require grad are inputs of it, too.
bool transformed(const Tensor& q, const Tensor& k, const Tensor& v, const Options& o) {
  if (tracing() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode))
    return true;
  for (const Tensor* t : {&q, &k, &v, &o.alibi})
    if (t->defined() && t->_fw_grad(0).defined()) return true;
  return at::GradMode::is_enabled() && o.alibi.defined() && o.alibi.requires_grad();
}

// q, k, v and the slopes of a plain dense call.
bool plain(const Tensor& q, const Tensor& k, const Tensor& v, const Options& o) {
  if (!q.is_cuda() || q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return false;
  const auto dt = q.scalar_type();
  if ((dt != at::kHalf && dt != at::kBFloat16) || k.scalar_type() != dt || v.scalar_type() != dt) return false;
  if (k.device() != q.device() || v.device() != q.device() || q.layout() != c10::kStrided || q.is_neg() || k.is_neg() || v.is_neg())
    return false;
  const auto qs = q.sizes(), ks = k.sizes();
  if (ks != v.sizes() || ks[0] != qs[0] || ks[3] != qs[3]) return false;
  const int64_t d = qs[3];
  if (d < 8 || d > 256 || d % 8 != 0) return false;
  for (int i = 0; i < 3; ++i)
    if (qs[i] <= 0 || ks[i] <= 0 || qs[i] > INT32_MAX - 256 || ks[i] > INT32_MAX - 256) return false;
  if (qs[0] > 65535 || qs[2] > 65535 || qs[2] % ks[2] != 0) return false;
  if (!addressable(q) || !addressable(k) || !addressable(v)) return false;
  if (o.left < INT32_MIN || o.left > INT32_MAX || o.right < INT32_MIN || o.right > INT32_MAX) return false;
  if (o.has_scale && !std::isfinite(static_cast<float>(o.scale))) return false;
  if (o.alibi.defined()) {
    const Tensor& a = o.alibi;
    if (!a.is_cuda() || a.device() != q.device() || a.scalar_type() != at::kFloat || !a.is_contiguous()) return false;
    if (!((a.dim() == 1 && a.size(0) == qs[2]) || (a.dim() == 2 && a.size(0) == qs[0] && a.size(1) == qs[2]))) return false;
  }
  return true;
}

void check(int rc) {
  if (rc == FA2_OK) return;
  if (rc == FA2_E_TYPE) C10_THROW_ERROR(TypeError, fa2_last_error());
  if (rc == FA2_E_VALUE) C10_THROW_ERROR(ValueError, fa2_last_error());
  TORCH_CHECK(false, fa2_last_error());
}

float scale_of(const Options& o, int64_t d) {
  return static_cast<float>(o.has_scale ? o.scale : 1.0 / std::sqrt(static_cast<double>(d)));
}

// The single-query convention: one query row sees every key unless slopes make its position matter.
bool effective_causal(const Options& o, int64_t seqlen_q) { return o.causal && !(seqlen_q == 1 && !o.alibi.defined()); }

void forward(const Tensor& q, const Tensor& k, const Tensor& v, const Options& o, Tensor& out, Tensor& lse) {
  const c10::cuda::CUDAGuard guard(q.device());
  const auto qs = q.sizes(), ks = k.sizes();
  out = empty(qs, q.scalar_type(), q.device());
  lse = empty({qs[0], qs[2], qs[1]}, at::kFloat, q.device());
  fa2_fwd_args a{};
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.out = out.data_ptr();
  a.lse = static_cast<float*>(lse.data_ptr());
  if (o.alibi.defined()) {
    a.alibi_slopes = static_cast<const float*>(o.alibi.data_ptr());
    a.alibi_batch_stride = o.alibi.dim() == 2 ? static_cast<int32_t>(qs[2]) : 0;
  }
  a.dtype = q.scalar_type() == at::kBFloat16 ? FA2_BF16 : FA2_F16;
  a.batch = static_cast<int32_t>(qs[0]);
  a.seqlen_q = static_cast<int32_t>(qs[1]);
  a.seqlen_k = static_cast<int32_t>(ks[1]);
  a.heads = static_cast<int32_t>(qs[2]);
  a.heads_k = static_cast<int32_t>(ks[2]);
  a.head_dim = static_cast<int32_t>(qs[3]);
  strides_of(q, a.q_stride);
  strides_of(k, a.k_stride);
  strides_of(v, a.v_stride);
  strides_of(out, a.o_stride);
  a.softmax_scale = scale_of(o, qs[3]);
  a.causal = effective_causal(o, qs[1]);
  a.window_left = static_cast<int32_t>(o.left);
  a.window_right = static_cast<int32_t>(o.right);
  a.softcap = static_cast<float>(o.softcap);
  Tensor workspace;
  const int64_t need = fa2_fwd_workspace_bytes(&a);
  if (need > 0) workspace = scratch(need, q.device());
  check(fa2_fwd_with_workspace(&a, workspace.defined() ? workspace.data_ptr() : nullptr, need, c10::cuda::getCurrentCUDAStream(q.device().index()).stream()));
}

struct Gradients {
  Tensor dq, dk, dv, delta;
};

Gradients backward(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out,
                   const Tensor& lse, const Options& o, bool deterministic) {
  const c10::cuda::CUDAGuard guard(q.device());
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  const auto qs = q.sizes(), ks = k.sizes();
  const auto dt = q.scalar_type();
  Gradients g;
  g.delta = empty({qs[0], qs[2], (qs[1] + 127) / 128 * 128}, at::kFloat, q.device());
  g.dq = empty(qs, dt, q.device());
  g.dk = empty(ks, dt, q.device());
  g.dv = empty(ks, dt, q.device());
  fa2_bwd_args a{};
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.dout = dout.data_ptr();
  a.lse = static_cast<const float*>(lse.data_ptr());
  a.delta = static_cast<const float*>(g.delta.data_ptr());
  a.dq = g.dq.data_ptr();
  a.dk = g.dk.data_ptr();
  a.dv = g.dv.data_ptr();
  a.dtype = dt == at::kBFloat16 ? FA2_BF16 : FA2_F16;
  a.batch = static_cast<int32_t>(qs[0]);
  a.seqlen_q = static_cast<int32_t>(qs[1]);
  a.seqlen_k = static_cast<int32_t>(ks[1]);
  a.heads = static_cast<int32_t>(qs[2]);
  a.heads_k = static_cast<int32_t>(ks[2]);
  a.head_dim = static_cast<int32_t>(qs[3]);
  strides_of(q, a.q_stride);
  strides_of(k, a.k_stride);
  strides_of(v, a.v_stride);
  strides_of(dout, a.do_stride);
  if (o.alibi.defined()) {
    a.alibi_slopes = static_cast<const float*>(o.alibi.data_ptr());
    a.alibi_batch_stride = o.alibi.dim() == 2 ? static_cast<int32_t>(qs[2]) : 0;
  }
  a.softcap = static_cast<float>(o.softcap);
  a.softmax_scale = scale_of(o, qs[3]);
  a.causal = effective_causal(o, qs[1]);
  a.window_left = static_cast<int32_t>(o.left);
  a.window_right = static_cast<int32_t>(o.right);
  fa2_bwd_options opt{};
  opt.size = sizeof(opt);
  opt.out = out.data_ptr();  // the first call computes delta
  strides_of(out, opt.o_stride);
  opt.share_key_blocks = 1;
  // Bit-reproducible gradients come from the two separate calls: dQ in a fixed order, then dK and dV.
  const int calls[2] = {deterministic ? 1 : 3, deterministic ? 2 : 0};
  for (const int which : calls) {
    if (which == 0) continue;
    a.which = which;
    Tensor workspace;
    a.dq_accum = nullptr;
    a.dq_accum_bytes = fa2_bwd_workspace_bytes_with_options(&a, &opt);
    if (a.dq_accum_bytes > 0) {
      // The parts of shared key blocks can be done without, but not in calls whose bits are to be the same every time.
      if (!deterministic) workspace = scratch(a.dq_accum_bytes, q.device());
      if (!workspace.defined()) {
        opt.share_key_blocks = deterministic;
        a.dq_accum_bytes = fa2_bwd_workspace_bytes_with_options(&a, &opt);
        workspace = empty({a.dq_accum_bytes}, at::kByte, q.device());
      }
      a.dq_accum = workspace.data_ptr();
    }
    check(fa2_bwd_with_options(&a, &opt, stream));
    opt.out = nullptr;
  }
  return g;
}

// dO, O and LSE of a plain backward call.
bool plain_backward(const Tensor& dout, const Tensor& q, const Tensor& out, const Tensor& lse) {
  for (const Tensor* t : {&dout, &out})
    if (t->dim() != 4 || t->sizes() != q.sizes() || t->scalar_type() != q.scalar_type() || t->device() != q.device() ||
        t->layout() != c10::kStrided || t->is_neg() || !addressable(*t))
      return false;
  return lse.scalar_type() == at::kFloat && lse.device() == q.device() && lse.dim() == 3 && lse.is_contiguous() &&
         lse.size(0) == q.size(0) && lse.size(1) == q.size(2) && lse.size(2) == q.size(1);
}

class DenseAttention : public torch::autograd::Function<DenseAttention> {
 public:
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                        const Options& o, bool deterministic) {
    Tensor out, lse;
    ::forward(q, k, v, o, out, lse);
    ctx->save_for_backward({q, k, v, out, lse});
    auto& d = ctx->saved_data;
    if (o.has_scale) d["scale"] = o.scale;
    d["causal"] = o.causal;
    d["left"] = o.left;
    d["right"] = o.right;
    d["softcap"] = o.softcap;
    if (o.alibi.defined()) d["alibi"] = o.alibi;
    d["deterministic"] = deterministic;
    return out;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    auto& d = ctx->saved_data;
    Options o;
    if (const auto it = d.find("scale"); it != d.end()) {
      o.has_scale = true;
      o.scale = it->second.toDouble();
    }
    o.causal = d["causal"].toBool();
    o.left = d["left"].toInt();
    o.right = d["right"].toInt();
    o.softcap = d["softcap"].toDouble();
    if (const auto it = d.find("alibi"); it != d.end()) o.alibi = it->second.toTensor();
    // What saved-tensor hooks hand back is checked and laid out anew like any argument.
    const Tensor dout = laid_out(grads[0].contiguous()), q = laid_out(saved[0]), k = laid_out(saved[1]), v = laid_out(saved[2]),
                 out = laid_out(saved[3]), &lse = saved[4];
    TORCH_CHECK(plain(q, k, v, o) && plain_backward(dout, q, out, lse), "dout and the saved tensors must match the forward's shapes, dtypes and device");
    Gradients g = ::backward(dout, q, k, v, out, lse, o, d["deterministic"].toBool());
    return {g.dq, g.dk, g.dv, Tensor(), Tensor()};
  }
};

// ---------------------------------------------------------------- Python arguments
bool tensor_arg(PyObject* o, Tensor& t) {
  if (!THPVariable_CheckExact(o)) return false;
  t = THPVariable_Unpack(o);
  return true;
}
bool float_arg(PyObject* o, double& x) {
  if (PyFloat_CheckExact(o)) x = PyFloat_AS_DOUBLE(o);
  else if (PyLong_CheckExact(o)) {
    x = PyLong_AsDouble(o);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
  } else return false;
  return true;
}
bool int_arg(PyObject* o, int64_t& x) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  x = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
bool bool_arg(PyObject* o, bool& x) {
  if (!PyBool_Check(o)) return false;
  x = o == Py_True;
  return true;
}
// softmax_scale, is_causal, window_left, window_right, softcap, alibi_slopes
bool options_arg(PyObject* const* a, Options& o) {
  if (a[0] != Py_None) {
    if (!float_arg(a[0], o.scale)) return false;
    o.has_scale = true;
  }
  return bool_arg(a[1], o.causal) && int_arg(a[2], o.left) && int_arg(a[3], o.right) && float_arg(a[4], o.softcap) &&
         (a[5] == Py_None || tensor_arg(a[5], o.alibi));
}

// Allocations and launches can block (a full launch queue, a cudaMalloc): other Python threads run meanwhile. Saved-tensor
// hooks take the lock for themselves.
struct WithoutPython {
  PyThreadState* const state = PyEval_SaveThread();
  ~WithoutPython() { PyEval_RestoreThread(state); }
};

PyObject* list_of(std::initializer_list<Tensor> ts) {
  PyObject* list = PyList_New(static_cast<Py_ssize_t>(ts.size()));
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) PyList_SET_ITEM(list, i++, THPVariable_Wrap(t));
  return list;
}

// fwd(q, k, v, softmax_scale, is_causal, window_left, window_right, softcap, alibi_slopes)
// -> [out, lse, probabilities (empty), RNG state (unused)], or None
PyObject* py_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor q, k, v;
  Options o;
  if (n != 9 || !tensor_arg(args[0], q) || !tensor_arg(args[1], k) || !tensor_arg(args[2], v) || !options_arg(args + 3, o) ||
      tracing() || !plain(q, k, v, o))
    Py_RETURN_NONE;
  Tensor out, lse, probabilities, state;
  {
    const WithoutPython unlocked;
    forward(q, k, v, o, out, lse);
    probabilities = empty({0}, q.scalar_type(), q.device());
    state = empty({2}, at::kLong, q.device());
  }
  return list_of({out, lse, probabilities, state});
  END_HANDLE_TH_ERRORS
}

// bwd(dout, q, k, v, out, lse, softmax_scale, is_causal, window_left, window_right, softcap, alibi_slopes, deterministic)
// -> [dq, dk, dv, delta], or None
PyObject* py_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor dout, q, k, v, out, lse;
  Options o;
  bool deterministic;
  if (n != 13 || !tensor_arg(args[0], dout) || !tensor_arg(args[1], q) || !tensor_arg(args[2], k) || !tensor_arg(args[3], v) ||
      !tensor_arg(args[4], out) || !tensor_arg(args[5], lse) || !options_arg(args + 6, o) || !bool_arg(args[12], deterministic) ||
      !plain(q, k, v, o) || !plain_backward(dout, q, out, lse))
    Py_RETURN_NONE;
  Gradients g;
  {
    const WithoutPython unlocked;
    g = backward(dout, q, k, v, out, lse, o, deterministic);
  }
  return list_of({g.dq, g.dk, g.dv, g.delta});
  END_HANDLE_TH_ERRORS
}

// attention(q, k, v, softmax_scale, is_causal, window_left, window_right, softcap, alibi_slopes, deterministic)
// -> out with its gradient function, or None
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor q, k, v;
  Options o;
  bool deterministic;
  if (n != 10 || !tensor_arg(args[0], q) || !tensor_arg(args[1], k) || !tensor_arg(args[2], v) || !options_arg(args + 3, o) ||
      !bool_arg(args[9], deterministic) || transformed(q, k, v, o) || !plain(q, k, v, o))
    Py_RETURN_NONE;
  Tensor out, lse;
  {
    const WithoutPython unlocked;
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad()))
      out = DenseAttention::apply(q, k, v, o, deterministic);
    else
      forward(q, k, v, o, out, lse);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"fwd", castPyCFunctionFast(py_fwd), METH_FASTCALL, nullptr},
    {"bwd", castPyCFunctionFast(py_bwd), METH_FASTCALL, nullptr},
    {"attention", castPyCFunctionFast(py_attention), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fa2_torch", "Dense attention calls on torch tensors.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fa2_torch() { return PyModule_Create(&module); }
