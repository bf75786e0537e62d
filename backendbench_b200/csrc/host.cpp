// The host wrappers' common cases in native code: a Python callable per operator that checks its
// arguments, allocates the result and calls the C-ABI without the interpreter in between. What bounds a
// small call is this work and not its kernel: add of 16 x 16 took 12 us of host time (dispatcher 2-3,
// arguments and layout in Python 3, allocation 1.3, ctypes 3, the launch 2), 4.1 so; the evaluation sweep of 24 small
// cases 847 us, 327.
//
// Nothing here decides anything new. A call is served when its tensors are plain CUDA tensors of the
// current device -- no subclass, no mode, no transform, no tracing, no gradient to record -- and its
// arguments need no conversion; the entry point and arguments of the C-ABI are then those the wrapper in
// ops.py / backward.py would have passed. Every other call, and every error case, goes to the callable
// it stands in front of, and so does everything while that wrapper is replaced (a counter in a test) or
// its allocator is (guard bands).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200ops.h"

namespace {

// ---------------------------------------------------------------- the library
#define B200_ENTRIES(F)                                                                                                                                                              \
  F(b200_relu) F(b200_add) F(b200_mul) F(b200_add_scalar) F(b200_mul_scalar) F(b200_where) F(b200_softmax) F(b200_softmax_backward) F(b200_reduce_scratch_bytes) F(b200_sum)           \
  F(b200_layer_norm) F(b200_layer_norm_backward_scratch_bytes) F(b200_layer_norm_backward) F(b200_argmax) F(b200_gather_rows) F(b200_index_select) F(b200_gather)                    \
  F(b200_scatter_add_scratch_bytes) F(b200_scatter_add) F(b200_embedding_backward_scratch_bytes) F(b200_embedding_backward) F(b200_copy_pitched) F(b200_gemm)                        \
  F(b200_gemm_takes_as_is) F(b200_gemm_f32_scratch_bytes) F(b200_gemm_f32) F(b200_gemm_splitk_scratch_bytes) F(b200_gemm_splitk) F(b200_allclose)
struct Api {
#define F(name) decltype(&::name) name;
  B200_ENTRIES(F)
#undef F
} api;

// from setup(): the wrappers' module, their `check`, `_status` and thresholds
PyObject *ops_dict = nullptr, *check_fn = nullptr, *status_fn = nullptr, *allocator_key = nullptr;
long long f32_split_min_macs = 0, splitk_min_k = 0, splitk_max_outputs = 0;

constexpr int kDims = B200_MAX_DIMS;
constexpr size_t kRank = 16;  // tensors of more dimensions are left to the wrapper
using at::Tensor;

// ---------------------------------------------------------------- arguments
const Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
// None -> an undefined tensor; anything but None or a plain tensor: false
bool tensor_or_none(PyObject* o, const Tensor*& t) {
  static const Tensor none;
  t = o == Py_None ? &none : tensor(o);
  return t != nullptr;
}
bool integer(PyObject* o, int64_t& v) {
  if (!PyLong_CheckExact(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool number(PyObject* o, double& v) {
  if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
  v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool boolean(PyObject* o, bool& v) {
  v = o == Py_True;
  return o == Py_True || o == Py_False;
}
bool integers(PyObject* o, int64_t* v, size_t& n) {
  const bool list = PyList_CheckExact(o);
  if (!list && !PyTuple_Check(o)) return false;
  n = list ? PyList_GET_SIZE(o) : PyTuple_GET_SIZE(o);
  if (n > kRank) return false;
  for (size_t i = 0; i < n; ++i)
    if (!integer(list ? PyList_GET_ITEM(o, i) : PyTuple_GET_ITEM(o, i), v[i])) return false;
  return true;
}
// Positional arguments in `at`, keywords by name: `names` are the schema's, the first `required` have no default
struct Args {
  PyObject* at[8] = {};
  bool parse(PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, std::initializer_list<const char*> names, int required) {
    if (nargs > static_cast<Py_ssize_t>(names.size())) return false;
    for (Py_ssize_t i = 0; i < nargs; ++i) at[i] = args[i];
    const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    for (Py_ssize_t k = 0; k < nkw; ++k) {
      int i = 0;
      for (const char* n : names) {
        if (PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, k), n) == 0) break;
        ++i;
      }
      if (i == static_cast<int>(names.size()) || at[i]) return false;
      at[i] = args[nargs + k];
    }
    for (int i = 0; i < required; ++i)
      if (!at[i]) return false;
    return true;
  }
  PyObject* operator[](int i) const { return at[i]; }
};

int dt(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return B200_F32;
    case at::kBFloat16: return B200_BF16;
    case at::kHalf: return B200_F16;
    default: return -1;
  }
}
bool floating(const Tensor& t) { return dt(t) >= 0; }
int index_dt(const Tensor& t) { return t.scalar_type() == at::kLong ? B200_I64 : t.scalar_type() == at::kInt ? B200_I32 : -1; }
bool dimension(int64_t dim, int64_t nd, int64_t& d) {
  const int64_t lim = nd > 0 ? nd : 1;
  if (dim < -lim || dim >= lim) return false;
  d = dim < 0 ? dim + lim : dim;
  return true;
}
int64_t product(at::IntArrayRef s, int64_t from, int64_t to) {
  int64_t p = 1;
  for (int64_t i = from; i < to; ++i) p *= s[i];
  return p;
}
int64_t extent(const Tensor& t, int64_t d) { return t.dim() ? t.size(d) : 1; }

// Whether a call on these tensors may skip the dispatcher: it would end in the CUDA kernel, and nothing on
// the way there would do or record anything.
struct Plain {
  c10::DispatchKeySet keys;
  bool all = true, grad = false;
  int device = -1;
  Plain& with(const Tensor& t) {
    if (!t.defined()) return *this;
    all = all && t.is_cuda() && t.layout() == at::kStrided && t.dim() <= static_cast<int64_t>(kRank) && (device < 0 || device == t.get_device());
    if (!all) return *this;
    device = t.get_device();
    keys = keys | t.key_set();
    grad = grad || t.requires_grad() || t._fw_grad(0).defined();
    return *this;
  }
  bool ok() const {
    if (!all || device < 0 || device != c10::cuda::current_device()) return false;
    static const c10::DispatchKeySet autograd(c10::DispatchKey::AutogradCUDA);
    static const c10::DispatchKeySet allowed =
        c10::DispatchKeySet(c10::DispatchKey::CUDA) | autograd | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) | c10::DispatchKeySet(c10::DispatchKey::BackendSelect);
    const auto tls = c10::impl::tls_local_dispatch_key_set();
    const c10::DispatchKeySet all_keys = (keys | tls.included_) - tls.excluded_;
    if (all_keys.raw_repr() & ~allowed.raw_repr()) return false;
    if (grad && all_keys.has(c10::DispatchKey::AutogradCUDA)) return false;  // (also under no_grad: the wrapper knows best)
    if (at::impl::torch_function_mode_enabled() || at::hasCallbacks()) return false;
    return !at::globalContext().deterministicAlgorithms();
  }
};
template <typename... T> bool plain(const T&... t) {
  Plain p;
  (p.with(t), ...);
  return p.ok();
}

// ---------------------------------------------------------------- results, scratch, launches
Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) { return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt); }
Tensor new_like(const Tensor& t) { return new_tensor(t.sizes(), t.scalar_type(), t); }
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// Scratch is the call's own until its launches are queued: a call is several launches that rely on what the ones before have left
// there, and the interpreter lock is not held between them, so that a buffer kept per stream would be another thread's, too.
// It comes from the caching allocator and goes back in stream order; up to a megabyte from buffers of that size that earlier calls
// on the stream have laid down, 64 of them at most (layer norm backward of 278 x 50 9.2 us a call with an allocation each, 8.6 so). What
// is captured belongs to the graph. The pool is guarded by the interpreter lock; release() empties it.
class Scratch {
  struct Free {
    c10::Device device;
    void* stream;
    Tensor buffer;
  };
  static constexpr int64_t kKept = 1 << 20;
  static constexpr size_t kMost = 64;

  Tensor buffer_;
  void* stream_ = nullptr;  // where the buffer is laid down; NULL: nowhere
  bool kept_ = false;

 public:
  static std::vector<Free>& pool() {
    static auto* p = new std::vector<Free>();  // never destroyed: no CUDA calls at exit
    return *p;
  }
  Scratch(const Tensor& like, int64_t bytes) {
    if (bytes <= 0) return;
    kept_ = bytes <= kKept && c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None;
    if (kept_) {
      stream_ = stream();
      auto& p = pool();
      for (auto it = p.rbegin(); it != p.rend(); ++it)
        if (it->stream == stream_ && it->device == like.device()) {
          buffer_ = std::move(it->buffer);
          p.erase(std::next(it).base());
          return;
        }
    }
    buffer_ = new_tensor({kept_ ? kKept : bytes}, at::kByte, like);
  }
  ~Scratch() {
    if (!kept_ || !buffer_.defined()) return;
    auto& p = pool();
    Tensor oldest;  // (given back when the pool is in order again)
    if (p.size() >= kMost) {
      oldest = std::move(p.front().buffer);
      p.erase(p.begin());
    }
    p.push_back(Free{buffer_.device(), stream_, std::move(buffer_)});
  }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  void* data() const { return ptr(buffer_); }
};

// The device's status word (ops._status); nullptr with an exception set if that failed
uint32_t* status_word(const Tensor& t) {
  static auto* words = new std::vector<Tensor>();
  const size_t d = static_cast<size_t>(t.get_device());
  if (words->size() <= d) words->resize(d + 1);
  if (!(*words)[d].defined()) {
    PyObject* dev = THPDevice_New(t.device());
    PyObject* w = dev ? PyObject_CallOneArg(status_fn, dev) : nullptr;
    Py_XDECREF(dev);
    if (!w) return nullptr;
    (*words)[d] = THPVariable_Unpack(w);
    Py_DECREF(w);
  }
  return static_cast<uint32_t*>((*words)[d].data_ptr());
}

struct Unlocked {  // other threads run during the call, as they do during a ctypes call
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
template <typename Call> bool launched(const char* what, Call call) {
  int rc;
  {
    Unlocked u;
    rc = call();
  }
  if (rc == 0) return true;
  PyObject* r = PyObject_CallFunction(check_fn, "is", rc, what);  // raises
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed with code %d", what, rc);
  return false;
}
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }

// A contiguous result's shape with the operands' strides, size-1 dims dropped, jointly contiguous neighbours merged
struct Layout {
  int nd = 1;
  int64_t shape[kDims], st[3][kDims];
  bool build(at::IntArrayRef out, std::initializer_list<const Tensor*> operands) {
    bool flat = true;
    for (const Tensor* t : operands) flat = flat && t->sizes() == out && t->is_contiguous();
    if (flat) {
      shape[0] = product(out, 0, out.size());
      for (auto& s : st) s[0] = 1;
      return true;
    }
    nd = 0;
    int64_t out_stride[kRank], acc = 1, last_out = 0;
    for (int64_t d = static_cast<int64_t>(out.size()) - 1; d >= 0; --d) {
      out_stride[d] = acc;
      acc *= std::max<int64_t>(out[d], 1);
    }
    for (size_t d = 0; d < out.size(); ++d) {
      if (out[d] == 1) continue;
      int64_t s[3] = {};
      int i = 0;
      for (const Tensor* t : operands) {
        const int64_t k = static_cast<int64_t>(d) - (static_cast<int64_t>(out.size()) - t->dim());
        s[i++] = k < 0 || t->size(k) == 1 ? 0 : t->stride(k);
      }
      bool joined = nd > 0 && last_out == out_stride[d] * out[d];
      for (int j = 0; j < i && joined; ++j) joined = st[j][nd - 1] == s[j] * out[d];
      if (joined) {
        shape[nd - 1] *= out[d];
      } else {
        if (nd == kDims) return false;
        shape[nd++] = out[d];
      }
      for (int j = 0; j < i; ++j) st[j][nd - 1] = s[j];
      last_out = out_stride[d];
    }
    if (nd == 0) {
      nd = 1;
      shape[0] = 1;
      for (auto& s : st) s[0] = 0;
    }
    return true;
  }
};
bool broadcast(std::initializer_list<const Tensor*> ts, at::DimVector& out) {
  size_t nd = 0;
  for (const Tensor* t : ts) nd = std::max<size_t>(nd, t->dim());
  out.assign(nd, 1);
  for (const Tensor* t : ts) {
    const size_t off = nd - t->dim();
    for (int64_t d = 0; d < t->dim(); ++d) {
      int64_t& cur = out[off + d];
      if (cur == 1) cur = t->size(d);
      else if (t->size(d) != 1 && t->size(d) != cur) return false;
    }
  }
  return true;
}

// ---------------------------------------------------------------- operators: the result, or NULL -- with an
// exception set where one was raised, without where the wrapper has to take the call
#define ARGS PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames
typedef PyObject* (*Fast)(ARGS);

PyObject* relu(ARGS) {
  Args a;
  if (!a.parse(args, nargs, kwnames, {"self"}, 1)) return nullptr;
  const Tensor* x = tensor(a[0]);
  if (!x || !floating(*x) || !plain(*x) || x->numel() == 0) return nullptr;
  Layout l;
  if (!l.build(x->sizes(), {x})) return nullptr;
  Tensor out = new_like(*x);
  if (!launched("b200_relu", [&, st = stream()] { return api.b200_relu(ptr(*x), ptr(out), l.nd, l.shape, l.st[0], dt(*x), st); })) return nullptr;
  return wrap(std::move(out));
}

PyObject* binary(bool add, PyObject* self, PyObject* other, double alpha) {
  const Tensor *x = tensor(self), *y = tensor(other);
  if (!x || !floating(*x)) return nullptr;
  const char* what;
  if (!y) {
    double v;
    if (!number(other, v) || !plain(*x) || x->numel() == 0) return nullptr;
    Layout l;
    if (!l.build(x->sizes(), {x})) return nullptr;
    Tensor out = new_like(*x);
    what = add ? "b200_add_scalar" : "b200_mul_scalar";
    auto f = add ? api.b200_add_scalar : api.b200_mul_scalar;
    if (!launched(what, [&, st = stream()] { return f(ptr(*x), ptr(out), l.nd, l.shape, l.st[0], dt(*x), dt(*x), add ? alpha * v : v, st); })) return nullptr;
    return wrap(std::move(out));
  }
  if (x->scalar_type() != y->scalar_type() || !plain(*x, *y)) return nullptr;
  at::DimVector shape;
  if (!broadcast({x, y}, shape)) return nullptr;
  Layout l;
  if (!l.build(shape, {x, y})) return nullptr;
  Tensor out = new_tensor(shape, x->scalar_type(), *x);
  if (out.numel() == 0) return wrap(std::move(out));
  const int t = dt(*x);
  if (!launched(add ? "b200_add" : "b200_mul", [&, st = stream()] {
        return add ? api.b200_add(ptr(*x), ptr(*y), ptr(out), l.nd, l.shape, l.st[0], l.st[1], t, t, t, alpha, st)
                   : api.b200_mul(ptr(*x), ptr(*y), ptr(out), l.nd, l.shape, l.st[0], l.st[1], t, t, t, st);
      }))
    return nullptr;
  return wrap(std::move(out));
}
PyObject* add(ARGS) {
  Args a;
  double alpha = 1.0;
  if (nargs > 2 || !a.parse(args, nargs, kwnames, {"self", "other", "alpha"}, 2) || (a[2] && !number(a[2], alpha))) return nullptr;
  return binary(true, a[0], a[1], alpha);
}
PyObject* mul(ARGS) {
  Args a;
  if (!a.parse(args, nargs, kwnames, {"self", "other"}, 2)) return nullptr;
  return binary(false, a[0], a[1], 1.0);
}

PyObject* where(ARGS) {
  Args a;
  if (!a.parse(args, nargs, kwnames, {"condition", "self", "other"}, 3)) return nullptr;
  const Tensor *c = tensor(a[0]), *x = tensor(a[1]), *y = tensor(a[2]);
  if (!c || !x || !y || c->scalar_type() != at::kBool || !floating(*x) || x->scalar_type() != y->scalar_type() || !plain(*c, *x, *y)) return nullptr;
  at::DimVector shape;
  if (!broadcast({c, x, y}, shape)) return nullptr;
  Layout l;
  if (!l.build(shape, {c, x, y})) return nullptr;
  Tensor out = new_tensor(shape, x->scalar_type(), *x);
  if (out.numel() == 0) return wrap(std::move(out));
  const int t = dt(*x);
  if (!launched("b200_where", [&, st = stream()] { return api.b200_where(ptr(*c), ptr(*x), ptr(*y), ptr(out), l.nd, l.shape, l.st[0], l.st[1], l.st[2], t, t, t, st); })) return nullptr;
  return wrap(std::move(out));
}

PyObject* softmax_of(bool log, ARGS) {
  Args a;
  int64_t dim, d;
  bool wide;
  if (!a.parse(args, nargs, kwnames, {"self", "dim", "half_to_float"}, 3) || !integer(a[1], dim) || !boolean(a[2], wide) || wide) return nullptr;
  const Tensor* x = tensor(a[0]);
  if (!x || !floating(*x) || !x->is_contiguous() || x->numel() == 0 || !dimension(dim, x->dim(), d) || !plain(*x)) return nullptr;
  const int64_t outer = product(x->sizes(), 0, d), len = extent(*x, d), inner = product(x->sizes(), d + 1, x->dim());
  if (inner > 1 && len >= 128 && outer * ((inner + 127) / 128) < 592) return nullptr;  // through transposed copies
  Tensor out = new_like(*x);
  if (!launched("b200_softmax", [&, st = stream()] { return api.b200_softmax(ptr(*x), ptr(out), outer, len, inner, dt(*x), dt(*x), log ? 1 : 0, st); })) return nullptr;
  return wrap(std::move(out));
}
PyObject* softmax(ARGS) { return softmax_of(false, args, nargs, kwnames); }
PyObject* log_softmax(ARGS) { return softmax_of(true, args, nargs, kwnames); }

PyObject* softmax_backward_of(bool log, ARGS) {
  Args a;
  int64_t dim, d;
  if (!a.parse(args, nargs, kwnames, {"grad_output", "output", "dim", "input_dtype"}, 4) || !integer(a[2], dim) || !THPDtype_Check(a[3])) return nullptr;
  const Tensor *g = tensor(a[0]), *y = tensor(a[1]);
  if (!g || !y || !floating(*g) || g->scalar_type() != y->scalar_type() || reinterpret_cast<THPDtype*>(a[3])->scalar_type != g->scalar_type() || g->sizes() != y->sizes() ||
      !g->is_contiguous() || !y->is_contiguous() || g->numel() == 0 || !dimension(dim, g->dim(), d) || !plain(*g, *y))
    return nullptr;
  const int64_t outer = product(g->sizes(), 0, d), len = extent(*g, d), inner = product(g->sizes(), d + 1, g->dim());
  Tensor out = new_like(*g);
  if (!launched("b200_softmax_backward", [&, st = stream()] { return api.b200_softmax_backward(ptr(*g), ptr(*y), ptr(out), outer, len, inner, dt(*g), dt(*g), log ? 1 : 0, st); })) return nullptr;
  return wrap(std::move(out));
}
PyObject* softmax_backward(ARGS) { return softmax_backward_of(false, args, nargs, kwnames); }
PyObject* log_softmax_backward(ARGS) { return softmax_backward_of(true, args, nargs, kwnames); }

PyObject* sum(ARGS) {
  Args a;
  int64_t dims[kRank];
  size_t n = 0;
  bool keep = false;
  if (nargs > 3 || !a.parse(args, nargs, kwnames, {"self", "dim", "keepdim", "dtype"}, 1) || (a[2] && !boolean(a[2], keep)) || (a[3] && a[3] != Py_None)) return nullptr;
  const Tensor* x = tensor(a[0]);
  if (!x || !floating(*x) || !x->is_contiguous() || x->dim() == 0 || !plain(*x)) return nullptr;
  if (a[1] && a[1] != Py_None && !integers(a[1], dims, n)) return nullptr;
  bool in[kRank] = {};
  int64_t first = x->dim(), last = -1;
  if (n == 0) {
    first = 0;
    last = x->dim() - 1;
    for (int64_t d = 0; d <= last; ++d) in[d] = true;
  }
  for (size_t i = 0; i < n; ++i) {
    int64_t d;
    if (!dimension(dims[i], x->dim(), d) || in[d]) return nullptr;
    in[d] = true;
    first = std::min(first, d);
    last = std::max(last, d);
  }
  at::DimVector shape;
  for (int64_t d = 0; d < x->dim(); ++d) {
    if (d >= first && d <= last && !in[d]) return nullptr;  // not neighbours: through a permuted copy
    if (!in[d]) shape.push_back(x->size(d));
    else if (keep) shape.push_back(1);
  }
  Tensor out = new_tensor(shape, x->scalar_type(), *x);
  if (out.numel() == 0) return wrap(std::move(out));
  const int64_t outer = product(x->sizes(), 0, first), len = product(x->sizes(), first, last + 1), inner = product(x->sizes(), last + 1, x->dim());
  const int64_t need = api.b200_reduce_scratch_bytes(outer, len, inner);
  Scratch s(*x, need);
  if (!launched("b200_sum", [&, st = stream()] { return api.b200_sum(ptr(*x), ptr(out), outer, len, inner, dt(*x), dt(*x), s.data(), need, st); })) return nullptr;
  return wrap(std::move(out));
}

PyObject* argmax(ARGS) {
  Args a;
  int64_t dim, d;
  bool keep = false;
  if (!a.parse(args, nargs, kwnames, {"self", "dim", "keepdim"}, 2) || !integer(a[1], dim) || (a[2] && !boolean(a[2], keep))) return nullptr;
  const Tensor* x = tensor(a[0]);
  if (!x || !floating(*x) || !x->is_contiguous() || x->dim() == 0 || x->numel() == 0 || !dimension(dim, x->dim(), d) || !plain(*x)) return nullptr;
  at::DimVector shape;
  for (int64_t i = 0; i < x->dim(); ++i) {
    if (i != d) shape.push_back(x->size(i));
    else if (keep) shape.push_back(1);
  }
  const int64_t outer = product(x->sizes(), 0, d), inner = product(x->sizes(), d + 1, x->dim());
  Tensor out = new_tensor(shape, at::kLong, *x);
  const int64_t need = api.b200_reduce_scratch_bytes(outer, x->size(d), inner);
  Scratch s(*x, need);
  if (!launched("b200_argmax", [&, st = stream()] { return api.b200_argmax(ptr(*x), static_cast<int64_t*>(ptr(out)), outer, x->size(d), inner, dt(*x), s.data(), need, st); })) return nullptr;
  return wrap(std::move(out));
}

// the last dimensions of x are `shape`: how many lead, the rows and columns
bool normalized(const Tensor& x, PyObject* shape, int64_t* ns, size_t& k, int64_t& rows, int64_t& cols) {
  if (!integers(shape, ns, k) || k == 0 || static_cast<int64_t>(k) > x.dim()) return false;
  const at::IntArrayRef want(ns, k);
  if (x.sizes().slice(x.dim() - k) != want) return false;
  rows = product(x.sizes(), 0, x.dim() - k);
  cols = product(want, 0, k);
  return rows > 0 && cols > 0;
}
bool parameter(const Tensor& t, at::IntArrayRef shape) { return !t.defined() || (floating(t) && t.is_contiguous() && t.sizes() == shape); }

PyObject* layer_norm(ARGS) {
  Args a;
  int64_t ns[kRank], rows, cols;
  size_t k;
  double eps;
  const Tensor *w, *b;
  if (!a.parse(args, nargs, kwnames, {"input", "normalized_shape", "weight", "bias", "eps"}, 5) || !tensor_or_none(a[2], w) || !tensor_or_none(a[3], b) || !number(a[4], eps)) return nullptr;
  const Tensor* x = tensor(a[0]);
  if (!x || !floating(*x) || !x->is_contiguous() || !normalized(*x, a[1], ns, k, rows, cols) || !plain(*x, *w, *b)) return nullptr;
  if (!parameter(*w, at::IntArrayRef(ns, k)) || !parameter(*b, at::IntArrayRef(ns, k)) || (w->defined() && b->defined() && w->scalar_type() != b->scalar_type())) return nullptr;
  at::DimVector stat(x->sizes().begin(), x->sizes().end());
  for (size_t i = stat.size() - k; i < stat.size(); ++i) stat[i] = 1;
  Tensor y = new_like(*x), mean = new_tensor(stat, at::kFloat, *x), rstd = new_tensor(stat, at::kFloat, *x);
  const int wb = w->defined() ? dt(*w) : b->defined() ? dt(*b) : dt(*x);
  if (!launched("b200_layer_norm", [&, st = stream()] { return api.b200_layer_norm(ptr(*x), ptr(*w), ptr(*b), ptr(y), ptr(mean), ptr(rstd), rows, cols, eps, dt(*x), wb, B200_F32, st); }))
    return nullptr;
  return Py_BuildValue("(NNN)", wrap(std::move(y)), wrap(std::move(mean)), wrap(std::move(rstd)));
}

PyObject* layer_norm_backward(ARGS) {
  Args a;
  int64_t ns[kRank], rows, cols;
  size_t k;
  bool mask[3];
  const Tensor *w, *b;
  if (!a.parse(args, nargs, kwnames, {"grad_out", "input", "normalized_shape", "mean", "rstd", "weight", "bias", "output_mask"}, 8) || !tensor_or_none(a[5], w) || !tensor_or_none(a[6], b)) return nullptr;
  if (!PyList_CheckExact(a[7]) || PyList_GET_SIZE(a[7]) != 3) return nullptr;
  for (int i = 0; i < 3; ++i)
    if (!boolean(PyList_GET_ITEM(a[7], i), mask[i])) return nullptr;
  const Tensor *dy = tensor(a[0]), *x = tensor(a[1]), *mean = tensor(a[3]), *rstd = tensor(a[4]);
  if (!dy || !x || !mean || !rstd || !floating(*x) || dy->scalar_type() != x->scalar_type() || dy->sizes() != x->sizes() || !dy->is_contiguous() || !x->is_contiguous() || !mean->is_contiguous() ||
      !rstd->is_contiguous() || !floating(*mean) || mean->scalar_type() != rstd->scalar_type() || !normalized(*x, a[2], ns, k, rows, cols) || mean->numel() != rows || rstd->numel() != rows ||
      !plain(*dy, *x, *mean, *rstd, *w, *b))
    return nullptr;
  const at::IntArrayRef shape(ns, k);
  if (!parameter(*w, shape) || ((mask[1] || mask[2]) && !w->defined() && !(b->defined() && floating(*b)))) return nullptr;
  const at::ScalarType wb = w->defined() ? w->scalar_type() : b->defined() ? b->scalar_type() : x->scalar_type();
  const int wb_dt = wb == at::kFloat ? B200_F32 : wb == at::kBFloat16 ? B200_BF16 : wb == at::kHalf ? B200_F16 : -1;
  if (wb_dt < 0) return nullptr;
  Tensor dx, dw, db;
  if (mask[0]) dx = new_like(*x);
  if (mask[1]) dw = new_tensor(shape, wb, *x);
  if (mask[2]) db = new_tensor(shape, wb, *x);
  const int64_t need = mask[1] || mask[2] ? api.b200_layer_norm_backward_scratch_bytes(rows, cols) : 0;
  Scratch s(*x, need);
  if (!launched("b200_layer_norm_backward", [&, st = stream()] {
        return api.b200_layer_norm_backward(ptr(*dy), ptr(*x), ptr(*mean), ptr(*rstd), ptr(*w), ptr(dx), ptr(dw), ptr(db), rows, cols, dt(*x), wb_dt, dt(*mean), s.data(), need, st);
      }))
    return nullptr;
  auto or_none = [](Tensor t) { return t.defined() ? wrap(std::move(t)) : Py_NewRef(Py_None); };
  return Py_BuildValue("(NNN)", or_none(std::move(dx)), or_none(std::move(dw)), or_none(std::move(db)));
}

PyObject* embedding(ARGS) {
  Args a;
  int64_t padding;
  bool freq, sparse;  // (these three count in the gradient alone)
  if (!a.parse(args, nargs, kwnames, {"weight", "indices", "padding_idx", "scale_grad_by_freq", "sparse"}, 2) || (a[2] && !integer(a[2], padding)) || (a[3] && !boolean(a[3], freq)) ||
      (a[4] && !boolean(a[4], sparse)))
    return nullptr;
  const Tensor *w = tensor(a[0]), *idx = tensor(a[1]);
  if (!w || !idx || w->dim() < 1 || index_dt(*idx) < 0 || !w->is_contiguous() || !idx->is_contiguous() || !plain(*w, *idx)) return nullptr;
  at::DimVector shape(idx->sizes().begin(), idx->sizes().end());
  shape.append(w->sizes().begin() + 1, w->sizes().end());
  if (shape.size() > kRank) return nullptr;
  Tensor out = new_tensor(shape, w->scalar_type(), *w);
  if (out.numel() == 0) return wrap(std::move(out));
  uint32_t* status = status_word(*w);
  if (!status) return nullptr;
  const int64_t row_bytes = product(w->sizes(), 1, w->dim()) * static_cast<int64_t>(w->element_size());
  if (!launched("b200_gather_rows", [&, st = stream()] { return api.b200_gather_rows(ptr(*w), ptr(*idx), ptr(out), w->size(0), row_bytes, idx->numel(), index_dt(*idx), status, st); })) return nullptr;
  return wrap(std::move(out));
}

PyObject* embedding_backward(ARGS) {
  Args a;
  int64_t rows, padding;
  bool freq;
  if (!a.parse(args, nargs, kwnames, {"grad_output", "indices", "num_weights", "padding_idx", "scale_grad_by_freq"}, 5) || !integer(a[2], rows) || !integer(a[3], padding) || !boolean(a[4], freq) || freq)
    return nullptr;
  const Tensor *g = tensor(a[0]), *idx = tensor(a[1]);
  if (!g || !idx || !floating(*g) || index_dt(*idx) < 0 || g->dim() != idx->dim() + 1 || g->sizes().slice(0, idx->dim()) != idx->sizes() || !g->is_contiguous() || !idx->is_contiguous() || rows <= 0 ||
      !plain(*g, *idx))
    return nullptr;
  const int64_t width = g->size(g->dim() - 1), n = idx->numel();
  if (width == 0) return nullptr;
  Tensor out = new_tensor({rows, width}, g->scalar_type(), *g);
  uint32_t* status = status_word(*g);
  if (!status) return nullptr;
  const int64_t need = api.b200_embedding_backward_scratch_bytes(n, rows);
  Scratch s(*g, need);
  if (!launched("b200_embedding_backward", [&, st = stream()] { return api.b200_embedding_backward(ptr(*g), ptr(*idx), ptr(out), n, rows, width, padding, dt(*g), index_dt(*idx), s.data(), need, status, st); }))
    return nullptr;
  return wrap(std::move(out));
}

PyObject* index_select(ARGS) {
  Args a;
  int64_t dim, d;
  if (!a.parse(args, nargs, kwnames, {"self", "dim", "index"}, 3) || !integer(a[1], dim)) return nullptr;
  const Tensor *x = tensor(a[0]), *idx = tensor(a[2]);
  if (!x || !idx || idx->dim() > 1 || index_dt(*idx) < 0 || x->dim() == 0 || !x->is_contiguous() || !idx->is_contiguous() || !dimension(dim, x->dim(), d) || !plain(*x, *idx)) return nullptr;
  at::DimVector shape(x->sizes().begin(), x->sizes().end());
  shape[d] = idx->numel();
  Tensor out = new_tensor(shape, x->scalar_type(), *x);
  if (out.numel() == 0) return wrap(std::move(out));
  uint32_t* status = status_word(*x);
  if (!status) return nullptr;
  const int64_t outer = product(x->sizes(), 0, d), inner = product(x->sizes(), d + 1, x->dim());
  if (!launched("b200_index_select", [&, st = stream()] {
        return api.b200_index_select(ptr(*x), ptr(*idx), ptr(out), outer, x->size(d), inner, idx->numel(), static_cast<int>(x->element_size()), index_dt(*idx), status, st);
      }))
    return nullptr;
  return wrap(std::move(out));
}

// index no larger than self but along `dim`, and no larger than src
bool index_fits(const Tensor& self, int64_t dim, const Tensor& index, const Tensor& src) {
  if (index.scalar_type() != at::kLong || self.dim() != index.dim() || self.dim() == 0 || self.dim() > kDims || (src.defined() && src.dim() != index.dim())) return false;
  for (int64_t d = 0; d < self.dim(); ++d)
    if ((d != dim && index.size(d) > self.size(d)) || (src.defined() && index.size(d) > src.size(d))) return false;
  return true;
}

PyObject* gather(ARGS) {
  Args a;
  int64_t dim, d;
  bool sparse;  // (counts in the gradient alone)
  if (nargs > 3 || !a.parse(args, nargs, kwnames, {"self", "dim", "index", "sparse_grad"}, 3) || !integer(a[1], dim) || (a[3] && !boolean(a[3], sparse))) return nullptr;
  const Tensor *x = tensor(a[0]), *idx = tensor(a[2]);
  if (!x || !idx || !dimension(dim, x->dim(), d) || !index_fits(*x, d, *idx, Tensor()) || idx->numel() == 0 || !plain(*x, *idx)) return nullptr;
  uint32_t* status = status_word(*x);
  if (!status) return nullptr;
  Tensor out = new_tensor(idx->sizes(), x->scalar_type(), *x);
  if (!launched("b200_gather", [&, st = stream()] {
        return api.b200_gather(ptr(*x), ptr(*idx), ptr(out), static_cast<int>(idx->dim()), idx->sizes().data(), x->strides().data(), idx->strides().data(), x->size(d), static_cast<int>(d),
                               static_cast<int>(x->element_size()), status, st);
      }))
    return nullptr;
  return wrap(std::move(out));
}

PyObject* scatter_add(ARGS) {
  Args a;
  int64_t dim, d;
  if (!a.parse(args, nargs, kwnames, {"self", "dim", "index", "src"}, 4) || !integer(a[1], dim)) return nullptr;
  const Tensor *x = tensor(a[0]), *idx = tensor(a[2]), *src = tensor(a[3]);
  if (!x || !idx || !src || !floating(*x) || src->scalar_type() != x->scalar_type() || !x->is_contiguous() || x->numel() == 0 || idx->numel() == 0 || !dimension(dim, x->dim(), d) ||
      !index_fits(*x, d, *idx, *src) || !plain(*x, *idx, *src))
    return nullptr;
  uint32_t* status = status_word(*x);
  if (!status) return nullptr;
  Tensor out = new_like(*x);
  const int nd = static_cast<int>(x->dim()), t = dt(*x);
  const int64_t *ss = x->sizes().data(), *is = idx->sizes().data(), *ist = idx->strides().data(), *rst = src->strides().data();
  const int64_t need = api.b200_scatter_add_scratch_bytes(ptr(*x), ptr(*idx), ptr(*src), ptr(out), nd, ss, is, ist, rst, static_cast<int>(d), t);
  Scratch s(*x, need);
  if (!launched("b200_scatter_add",
                [&, st = stream()] { return api.b200_scatter_add(ptr(*x), ptr(*idx), ptr(*src), ptr(out), nd, ss, is, ist, rst, static_cast<int>(d), t, s.data(), need, status, st); }))
    return nullptr;
  return wrap(std::move(out));
}

// ---------------------------------------------------------------- contraction (ops._gemm)
struct Operand {
  Tensor t;
  int64_t batch, row, col;  // strides
};
bool tma_ready(const Operand& o, int64_t s_mn, int64_t s_k, int64_t batch) {
  if (reinterpret_cast<uintptr_t>(o.t.data_ptr()) % 16 || (batch > 1 && (o.batch % 8 || o.batch <= 0))) return false;
  return (s_k == 1 && s_mn % 8 == 0 && s_mn > 0) || (s_mn == 1 && s_k % 8 == 0 && s_k > 0);
}
// a copy of [batch, rows, cols] whose rows are a multiple of 8 elements apart: (batch, row) strides
bool repitch(Operand& o, int64_t batch, int64_t rows, int64_t cols, int64_t s_r, int64_t s_c, int64_t& pitch) {
  pitch = (cols + 7) / 8 * 8;
  Tensor buf = new_tensor({batch, rows, pitch}, o.t.scalar_type(), o.t);
  if (!launched("b200_copy_pitched", [&, st = stream()] {
        return api.b200_copy_pitched(ptr(o.t), ptr(buf), batch, rows, cols, o.batch, s_r, s_c, rows * pitch, pitch, static_cast<int>(o.t.element_size()), st);
      }))
    return false;
  o.t = buf;
  o.batch = rows * pitch;
  return true;
}
PyObject* gemm(Operand a, Operand b, const Tensor& bias, int64_t batch, int64_t M, int64_t N, int64_t K, double alpha, double beta, at::IntArrayRef shape) {
  const int t = dt(a.t);
  Tensor out = new_tensor(shape, a.t.scalar_type(), a.t);
  if (out.numel() == 0) return wrap(std::move(out));
  uint32_t* status = status_word(a.t);
  if (!status) return nullptr;
  if (t != B200_F32 && (M * N * K * batch >= (1 << 24) || K >= 1024) && K >= 16) {
    bool ra = tma_ready(a, a.row, a.col, batch), rb = tma_ready(b, b.col, b.row, batch);
    if (!(ra && rb) && api.b200_gemm_takes_as_is(ptr(a.t), ptr(b.t), batch, M, N, K, a.batch, a.row, a.col, b.batch, b.row, b.col, t)) ra = rb = true;
    if (!ra) {
      if (a.row != 1 || a.col == 1) {
        if (!repitch(a, batch, M, K, a.row, a.col, a.row)) return nullptr;
        a.col = 1;
      } else {
        if (!repitch(a, batch, K, M, a.col, a.row, a.col)) return nullptr;
        a.row = 1;
      }
    }
    if (!rb) {
      if (b.row != 1 || b.col == 1) {
        if (!repitch(b, batch, K, N, b.row, b.col, b.row)) return nullptr;
        b.col = 1;
      } else {
        if (!repitch(b, batch, N, K, b.col, b.row, b.col)) return nullptr;
        b.row = 1;
      }
    }
  }
  int64_t sbm = 0, sbn = 0;
  if (bias.defined()) {
    const int64_t nd = bias.dim();
    if (nd >= 1 && !(bias.size(nd - 1) == 1 && N != 1)) sbn = bias.stride(nd - 1);
    if (nd == 2 && !(bias.size(0) == 1 && M != 1)) sbm = bias.stride(0);
  }
  const int64_t macs = batch * M * N * K, tiles = batch * ((M + 127) / 128) * ((N + 255) / 256);
  bool done = false, ok = false;
  if (t == B200_F32 && macs >= f32_split_min_macs && K >= 32 && M > 64 && N > 64 && (tiles >= 8 || macs >= (1LL << 30))) {
    const int64_t need = api.b200_gemm_f32_scratch_bytes(batch, M, N, K);
    if (need > 0) {
      Scratch s(a.t, need);
      done = true;
      ok = launched("b200_gemm_f32", [&, st = stream()] {
        return api.b200_gemm_f32(ptr(a.t), ptr(b.t), ptr(bias), ptr(out), batch, M, N, K, a.batch, a.row, a.col, b.batch, b.row, b.col, sbm, sbn, alpha, beta, s.data(), need, status, st);
      });
    }
  } else if (t != B200_F32 && batch == 1 && K >= splitk_min_k && M * N <= splitk_max_outputs) {
    const int64_t need = api.b200_gemm_splitk_scratch_bytes(ptr(a.t), ptr(b.t), ptr(out), batch, M, N, K, a.batch, a.row, a.col, b.batch, b.row, b.col, t);
    if (need > 0) {
      Scratch s(a.t, need);
      done = true;
      ok = launched("b200_gemm_splitk", [&, st = stream()] {
        return api.b200_gemm_splitk(ptr(a.t), ptr(b.t), ptr(bias), ptr(out), batch, M, N, K, a.batch, a.row, a.col, b.batch, b.row, b.col, sbm, sbn, alpha, beta, t, s.data(), need, status, st);
      });
    }
  }
  if (!done)
    ok = launched("b200_gemm", [&, st = stream()] {
      return api.b200_gemm(ptr(a.t), ptr(b.t), ptr(bias), ptr(out), batch, M, N, K, a.batch, a.row, a.col, b.batch, b.row, b.col, sbm, sbn, alpha, beta, t, status, st);
    });
  return ok ? wrap(std::move(out)) : nullptr;
}
PyObject* matrices(const Tensor& a, const Tensor& b, const Tensor& bias, double alpha, double beta) {
  if (a.dim() != 2 || b.dim() != 2 || a.size(1) != b.size(0) || !floating(a) || a.scalar_type() != b.scalar_type() || !plain(a, b, bias)) return nullptr;
  const int64_t M = a.size(0), K = a.size(1), N = b.size(1), shape[2] = {M, N};
  if (bias.defined()) {
    if (bias.scalar_type() != a.scalar_type() || bias.dim() > 2) return nullptr;
    const int64_t nd = bias.dim();
    if ((nd >= 1 && bias.size(nd - 1) != 1 && bias.size(nd - 1) != N) || (nd == 2 && bias.size(0) != 1 && bias.size(0) != M)) return nullptr;
  }
  return gemm(Operand{a, 0, a.stride(0), a.stride(1)}, Operand{b, 0, b.stride(0), b.stride(1)}, bias, 1, M, N, K, alpha, beta, shape);
}
PyObject* mm(ARGS) {
  Args a;
  if (!a.parse(args, nargs, kwnames, {"self", "mat2"}, 2)) return nullptr;
  const Tensor *x = tensor(a[0]), *y = tensor(a[1]);
  return x && y ? matrices(*x, *y, Tensor(), 1.0, 0.0) : nullptr;
}
PyObject* addmm(ARGS) {
  Args a;
  double beta = 1.0, alpha = 1.0;
  if (nargs > 3 || !a.parse(args, nargs, kwnames, {"self", "mat1", "mat2", "beta", "alpha"}, 3) || (a[3] && !number(a[3], beta)) || (a[4] && !number(a[4], alpha))) return nullptr;
  const Tensor *bias = tensor(a[0]), *x = tensor(a[1]), *y = tensor(a[2]);
  return bias && x && y ? matrices(*x, *y, *bias, alpha, beta) : nullptr;
}
PyObject* bmm(ARGS) {
  Args a;
  if (!a.parse(args, nargs, kwnames, {"self", "mat2"}, 2)) return nullptr;
  const Tensor *x = tensor(a[0]), *y = tensor(a[1]);
  if (!x || !y || x->dim() != 3 || y->dim() != 3 || x->size(0) != y->size(0) || x->size(2) != y->size(1) || !floating(*x) || x->scalar_type() != y->scalar_type() || !plain(*x, *y)) return nullptr;
  const int64_t shape[3] = {x->size(0), x->size(1), y->size(2)};
  return gemm(Operand{*x, x->stride(0), x->stride(1), x->stride(2)}, Operand{*y, y->stride(0), y->stride(1), y->stride(2)}, Tensor(), shape[0], shape[1], shape[2], x->size(2), 1.0, 0.0, shape);
}

struct Entry {
  const char* name;
  Fast fast;
};
const Entry kEntries[] = {
    {"relu", relu}, {"add", add}, {"mul", mul}, {"where", where}, {"softmax", softmax}, {"log_softmax", log_softmax}, {"sum", sum}, {"layer_norm", layer_norm}, {"argmax", argmax},
    {"embedding", embedding}, {"index_select", index_select}, {"gather", gather}, {"scatter_add", scatter_add}, {"mm", mm}, {"addmm", addmm}, {"bmm", bmm},
    {"softmax_backward", softmax_backward}, {"log_softmax_backward", log_softmax_backward}, {"layer_norm_backward", layer_norm_backward}, {"embedding_backward", embedding_backward},
};

// ---------------------------------------------------------------- the callable
struct NativeOp {
  PyObject_HEAD vectorcallfunc vectorcall;
  Fast fast;
  PyObject *fallback, *module_dict, *attr, *original;  // the wrapper it stands for: module_dict[attr] while nobody has replaced it
};

PyObject* native_op_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  auto* op = reinterpret_cast<NativeOp*>(self);
  if (PyDict_GetItemWithError(ops_dict, allocator_key) == Py_None && PyDict_GetItemWithError(op->module_dict, op->attr) == op->original) {
    HANDLE_TH_ERRORS
    PyObject* r = op->fast(args, PyVectorcall_NARGS(nargsf), kwnames);
    if (r || PyErr_Occurred()) return r;
    END_HANDLE_TH_ERRORS
  }
  return PyObject_Vectorcall(op->fallback, args, nargsf, kwnames);
}
void native_op_dealloc(PyObject* self) {
  auto* op = reinterpret_cast<NativeOp*>(self);
  Py_XDECREF(op->fallback);
  Py_XDECREF(op->module_dict);
  Py_XDECREF(op->attr);
  Py_XDECREF(op->original);
  Py_TYPE(self)->tp_free(self);
}
PyTypeObject NativeOpType = [] {
  PyTypeObject t = {PyVarObject_HEAD_INIT(nullptr, 0)};
  t.tp_name = "_b200host.NativeOp";
  t.tp_basicsize = sizeof(NativeOp);
  t.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  t.tp_call = PyVectorcall_Call;
  t.tp_vectorcall_offset = offsetof(NativeOp, vectorcall);
  t.tp_dealloc = native_op_dealloc;
  return t;
}();

// setup(handle of libb200ops.so, ops module, check, F32_SPLIT_MIN_MACS, SPLITK_MIN_K, SPLITK_MAX_OUTPUTS)
PyObject* setup(PyObject*, PyObject* args) {
  unsigned long long handle;
  PyObject *ops, *check;
  if (!PyArg_ParseTuple(args, "KOOLLL", &handle, &ops, &check, &f32_split_min_macs, &splitk_min_k, &splitk_max_outputs)) return nullptr;
#define F(name)                                                                                     \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(reinterpret_cast<void*>(handle), #name));   \
  if (!api.name) return PyErr_Format(PyExc_RuntimeError, "libb200ops.so has no entry " #name);
  B200_ENTRIES(F)
#undef F
  PyObject* dict = PyModule_GetDict(ops);
  PyObject* status = PyObject_GetAttrString(ops, "_status");
  if (!dict || !status) return nullptr;
  Py_XSETREF(ops_dict, Py_NewRef(dict));
  Py_XSETREF(check_fn, Py_NewRef(check));
  Py_XSETREF(status_fn, status);
  Py_XSETREF(allocator_key, PyUnicode_InternFromString("_allocator"));
  Py_RETURN_NONE;
}

// make(name, module of the wrapper, its attribute, the wrapper, callable for everything else)
PyObject* make(PyObject*, PyObject* args) {
  const char* name;
  PyObject *module, *attr, *original, *fallback;
  if (!PyArg_ParseTuple(args, "sOUOO", &name, &module, &attr, &original, &fallback)) return nullptr;
  if (!ops_dict) return PyErr_Format(PyExc_RuntimeError, "setup() comes first");
  for (const Entry& e : kEntries) {
    if (strcmp(e.name, name) != 0) continue;
    auto* op = PyObject_New(NativeOp, &NativeOpType);
    if (!op) return nullptr;
    op->vectorcall = native_op_call;
    op->fast = e.fast;
    op->fallback = Py_NewRef(fallback);
    op->module_dict = Py_NewRef(PyModule_GetDict(module));
    op->attr = Py_NewRef(attr);
    op->original = Py_NewRef(original);
    return reinterpret_cast<PyObject*>(op);
  }
  return PyErr_Format(PyExc_KeyError, "%s", name);
}

// release(): the scratch that no call is using goes back to the allocator
PyObject* release(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  auto free = std::move(Scratch::pool());
  Scratch::pool().clear();
  free.clear();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// compare(reference, result, atol, rtol, record): the pairs of tensors are queued into the device record. False: nothing
// was done, the structures are not what this serves (tensors of one shape and floating dtype, contiguous, or a tuple of them).
PyObject* compare(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  double atol, rtol;
  const Tensor* rec = nargs == 5 ? tensor(args[4]) : nullptr;
  if (!rec || !number(args[2], atol) || !number(args[3], rtol) || rec->scalar_type() != at::kInt || rec->numel() != 8 || !rec->is_contiguous()) Py_RETURN_FALSE;
  const Tensor *ref[8], *res[8];
  size_t n = 0;
  auto pair = [&](PyObject* a, PyObject* b) {
    const Tensor *x = tensor(a), *y = tensor(b);
    if (n == 8 || !x || !y || !floating(*x) || x->scalar_type() != y->scalar_type() || x->sizes() != y->sizes() || x->numel() == 0 || !x->is_contiguous() || !y->is_contiguous()) return false;
    ref[n] = x;
    res[n++] = y;
    return true;
  };
  if (PyTuple_CheckExact(args[0]) && PyTuple_CheckExact(args[1])) {
    if (PyTuple_GET_SIZE(args[0]) == 0 || PyTuple_GET_SIZE(args[0]) != PyTuple_GET_SIZE(args[1])) Py_RETURN_FALSE;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[0]); ++i)
      if (!pair(PyTuple_GET_ITEM(args[0], i), PyTuple_GET_ITEM(args[1], i))) Py_RETURN_FALSE;
  } else if (!pair(args[0], args[1])) {
    Py_RETURN_FALSE;
  }
  Plain p;
  p.with(*rec);
  for (size_t i = 0; i < n; ++i) p.with(*ref[i]).with(*res[i]);
  p.grad = false;  // nothing is computed that a gradient could belong to
  if (!p.ok()) Py_RETURN_FALSE;
  for (size_t i = 0; i < n; ++i)
    if (!launched("b200_allclose", [&, st = stream()] { return api.b200_allclose(ptr(*ref[i]), ptr(*res[i]), ref[i]->numel(), dt(*ref[i]), rtol, atol, static_cast<b200_close_record*>(ptr(*rec)), i == 0, st); }))
      return nullptr;
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {{"setup", setup, METH_VARARGS, nullptr},
                          {"make", make, METH_VARARGS, nullptr},
                          {"release", release, METH_NOARGS, nullptr},
                          {"compare", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(compare)), METH_FASTCALL, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_b200host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200host() {
  if (PyType_Ready(&NativeOpType) < 0) return nullptr;
  return PyModule_Create(&kModule);
}
