// The per-call part of ops.py in C++: argument checks, output allocation, the current stream, and the call into the C ABI.
// In Python that part took 10.6 us of an eager call (4.7 of them in the library and the launch), which was longer than the
// kernels of the small calls take.  Every function returns None where a call is not of the ordinary form - the Python code
// then makes its own checks and reports the error or goes its way - and an integer where the library refused it.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <vector>

#include "qfg.h"

namespace {

// addresses of the library's entry points, given by ops.py (which finds the library)
struct Entries {
  decltype(&qfg_skinny_gemm_compute) skinny_gemm;
  decltype(&qfg_argmax_rows) argmax_rows;
  decltype(&qfg_dequant_compute) dequant;
  decltype(&qfg_lmhead_compute) lmhead;
  decltype(&qfg_shared_expert_down_compute) shared_expert_down;
} g_lib;

// A plain dense CUDA tensor, or null: no subclass, no wrapper of a transform, nothing without memory of its own.
const at::Tensor* Dense(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::DispatchKeySet keys = t.key_set();
  if (!t.defined() || !keys.has(c10::DispatchKey::CUDA) || keys.has(c10::DispatchKey::Python) || keys.has(c10::DispatchKey::FuncTorchBatched) ||
      keys.has(c10::DispatchKey::FuncTorchGradWrapper) || keys.has(c10::DispatchKey::Functionalize) || !t.has_storage() || !t.is_contiguous())
    return nullptr;
  return &t;
}
const at::Tensor* Bf16(PyObject* o) {
  const at::Tensor* t = Dense(o);
  return t != nullptr && t->scalar_type() == at::kBFloat16 ? t : nullptr;
}
bool Weight(PyObject* o, qfg_tensor2d* d) {
  const at::Tensor* t = Dense(o);
  if (t == nullptr || t->dim() != 2) return false;
  switch (t->scalar_type()) {
    case at::kBFloat16: d->dtype = QFG_BFLOAT16; break;
    case at::kHalf: d->dtype = QFG_FLOAT16; break;
    case at::kFloat: d->dtype = QFG_FLOAT; break;
    case at::kByte: d->dtype = QFG_UINT8; break;
    case at::kFloat8_e4m3fn: d->dtype = QFG_FLOAT8E4M3FN; break;
    default: return false;
  }
  d->data = t->data_ptr();
  d->rows = t->size(0);
  d->cols = t->size(1);
  return true;
}
void* Stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
PyObject* None() { Py_RETURN_NONE; }

// Neither a C++ exception (an allocation that failed, say) nor the error of a conversion crosses into Python with a None: the
// Python code meets it on its own way.
template <typename F>
PyObject* Guard(F&& f) {
  PyObject* r;
  try {
    r = f();
  } catch (...) {
    r = None();
  }
  if (r == Py_None) PyErr_Clear();
  return r;
}
template <typename F>
int Call(F&& f) {  // without the interpreter's lock, as a foreign call through ctypes
  int code;
  Py_BEGIN_ALLOW_THREADS;
  code = f();
  Py_END_ALLOW_THREADS;
  return code;
}

constexpr int kMaxTensors = 16;
// the elements of a list of widths
int Widths(PyObject* list, std::array<int64_t, kMaxTensors>* w) {
  if (!PyList_CheckExact(list) || PyList_GET_SIZE(list) > kMaxTensors) return -1;
  const int n = static_cast<int>(PyList_GET_SIZE(list));
  for (int i = 0; i < n; ++i) {
    (*w)[i] = PyLong_AsLongLong(PyList_GET_ITEM(list, i));
    if ((*w)[i] < 0) return -1;
  }
  return n;
}
PyObject* ListOf(const std::array<at::Tensor, kMaxTensors>& t, int n) {
  PyObject* list = PyList_New(n);
  for (int i = 0; list != nullptr && i < n; ++i) {
    PyObject* o = THPVariable_Wrap(t[i]);
    if (o == nullptr) {
      Py_DECREF(list);
      return nullptr;
    }
    PyList_SET_ITEM(list, i, o);
  }
  return list;
}
PyObject* TupleOf(std::initializer_list<at::Tensor> t) {
  PyObject* tuple = PyTuple_New(static_cast<Py_ssize_t>(t.size()));
  Py_ssize_t i = 0;
  for (const at::Tensor& v : t) {
    PyObject* o = tuple != nullptr ? THPVariable_Wrap(v) : nullptr;
    if (o == nullptr) {
      Py_XDECREF(tuple);
      return nullptr;
    }
    PyTuple_SET_ITEM(tuple, i++, o);
  }
  return tuple;
}

// skinny_gemm(handle, x, weights, widths) -> [y, ...]
PyObject* SkinnyGemm(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return Guard([&]() -> PyObject* {
    if (n_args != 4 || !PyTuple_CheckExact(a[2])) return None();
    const void* op = PyLong_AsVoidPtr(a[0]);
    const at::Tensor* x = Bf16(a[1]);
    const Py_ssize_t n_weights = PyTuple_GET_SIZE(a[2]);
    std::array<int64_t, kMaxTensors> widths;
    const int n_out = Widths(a[3], &widths);
    if (op == nullptr || x == nullptr || x->dim() < 1 || x->size(-1) < 1 || n_weights > kMaxTensors || n_out < 1) return None();
    std::array<qfg_tensor2d, kMaxTensors> w;
    for (Py_ssize_t i = 0; i < n_weights; ++i) {
      if (!Weight(PyTuple_GET_ITEM(a[2], i), &w[i])) return None();
    }
    const int64_t k = x->size(-1), m = x->numel() / k;
    std::array<at::Tensor, kMaxTensors> out;
    std::array<void*, kMaxTensors> ptr;
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    const at::TensorOptions options = x->options();
    for (int i = 0; i < n_out; ++i) {
      shape.back() = widths[i];
      out[i] = at::empty(shape, options);
      ptr[i] = out[i].data_ptr();
    }
    const void* xp = x->data_ptr();
    void* const stream = Stream();
    const int code = Call([&] {
      return g_lib.skinny_gemm(static_cast<const qfg_skinny_gemm*>(op), xp, m, k, w.data(), static_cast<int>(n_weights), ptr.data(), n_out, stream);
    });
    return code != 0 ? PyLong_FromLong(code) : ListOf(out, n_out);
  });
}

// argmax_rows(x, with_val) -> (idx, val) or idx
PyObject* ArgmaxRows(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return Guard([&]() -> PyObject* {
    const at::Tensor* x = n_args == 2 ? Dense(a[0]) : nullptr;
    if (x == nullptr || (a[1] != Py_True && a[1] != Py_False) || x->dim() < 1 || x->size(-1) < 1) return None();
    int dtype;
    switch (x->scalar_type()) {
      case at::kBFloat16: dtype = QFG_BFLOAT16; break;
      case at::kHalf: dtype = QFG_FLOAT16; break;
      case at::kFloat: dtype = QFG_FLOAT; break;
      default: return None();
    }
    const int64_t vocab = x->size(-1), rows = x->numel() / vocab;
    const at::IntArrayRef lead = x->sizes().slice(0, x->dim() - 1);
    const at::Tensor idx = at::empty(lead, x->options().dtype(at::kLong));
    at::Tensor val;
    if (a[1] == Py_True) val = at::empty(lead, x->options().dtype(at::kFloat));
    const void* xp = x->data_ptr();
    int64_t* const ip = idx.data_ptr<int64_t>();
    float* const vp = val.defined() ? val.data_ptr<float>() : nullptr;
    void* const stream = Stream();
    const int code = Call([&] { return g_lib.argmax_rows(dtype, xp, rows, vocab, ip, vp, stream); });
    if (code != 0) return PyLong_FromLong(code);
    return val.defined() ? TupleOf({idx, val}) : THPVariable_Wrap(idx);
  });
}

// dequant(handle, w, widths) -> [out, ...]
PyObject* Dequant(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return Guard([&]() -> PyObject* {
    qfg_tensor2d w;
    std::array<int64_t, kMaxTensors> widths;
    if (n_args != 3 || !Weight(a[1], &w)) return None();
    const void* op = PyLong_AsVoidPtr(a[0]);
    const int n_out = Widths(a[2], &widths);
    if (op == nullptr || n_out < 1) return None();
    std::array<at::Tensor, kMaxTensors> out;
    std::array<void*, kMaxTensors> ptr;
    const at::TensorOptions options = THPVariable_Unpack(a[1]).options().dtype(at::kBFloat16);
    for (int i = 0; i < n_out; ++i) {
      out[i] = at::empty({w.rows, widths[i]}, options);
      ptr[i] = out[i].data_ptr();
    }
    void* const stream = Stream();
    const int code = Call([&] { return g_lib.dequant(static_cast<const qfg_dequant*>(op), &w, ptr.data(), n_out, stream); });
    return code != 0 ? PyLong_FromLong(code) : ListOf(out, n_out);
  });
}

// lmhead(handle, workspace, x, w, n, col_offset) -> (idx, val, key)
PyObject* LmHead(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return Guard([&]() -> PyObject* {
    qfg_tensor2d w;
    if (n_args != 6 || !Weight(a[3], &w)) return None();
    const void* op = PyLong_AsVoidPtr(a[0]);
    const at::Tensor *space = Dense(a[1]), *x = Bf16(a[2]);
    const int64_t n = PyLong_AsLongLong(a[4]), col_offset = PyLong_AsLongLong(a[5]);
    if (PyErr_Occurred() || op == nullptr || space == nullptr || x == nullptr || x->dim() < 1 || x->size(-1) < 1) return None();
    const int64_t k = x->size(-1), m = x->numel() / k;
    const at::Tensor idx = at::empty({m}, x->options().dtype(at::kLong)), val = at::empty({m}, x->options().dtype(at::kFloat)),
                     key = at::empty({m}, x->options().dtype(at::kLong));
    const void* xp = x->data_ptr();
    void *const sp = space->data_ptr(), *const stream = Stream();
    int64_t* const ip = idx.data_ptr<int64_t>();
    float* const vp = val.data_ptr<float>();
    uint64_t* const kp = reinterpret_cast<uint64_t*>(key.data_ptr<int64_t>());
    const int code = Call([&] { return g_lib.lmhead(static_cast<const qfg_lmhead*>(op), xp, m, k, &w, n, col_offset, sp, ip, vp, kp, nullptr, stream); });
    return code != 0 ? PyLong_FromLong(code) : TupleOf({idx, val, key});
  });
}

// shared_expert_down(handle, g, u, w, gx, gw, routed) -> out
PyObject* SharedExpertDown(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  return Guard([&]() -> PyObject* {
    qfg_tensor2d w;
    if (n_args != 7 || !Weight(a[3], &w)) return None();
    const void* op = PyLong_AsVoidPtr(a[0]);
    const at::Tensor *g = Bf16(a[1]), *u = Bf16(a[2]), *gx = Bf16(a[4]), *gw = Bf16(a[5]), *routed = Bf16(a[6]);
    if (op == nullptr || g == nullptr || u == nullptr || gx == nullptr || gw == nullptr || routed == nullptr || w.rows < 1 || routed->dim() < 1 ||
        gw->dim() < 1)
      return None();
    const int64_t k = w.rows, n = routed->size(-1), m = g->numel() / k, gk = gw->numel();
    if (m < 1 || g->numel() != m * k || u->numel() != m * k || routed->numel() != m * n || gx->numel() != m * gk || gw->size(-1) != 1) return None();
    if (w.dtype == QFG_UINT8 ? n % 16 != 0 || w.cols != n * 9 / 16 : w.cols != n) return None();
    const at::Tensor out = at::empty(routed->sizes(), routed->options());
    const void *gp = g->data_ptr(), *up = u->data_ptr(), *gxp = gx->data_ptr(), *gwp = gw->data_ptr(), *rp = routed->data_ptr();
    void *const op_out = out.data_ptr(), *const stream = Stream();
    const int code = Call([&] {
      return g_lib.shared_expert_down(static_cast<const qfg_shared_expert_down*>(op), gp, up, m, k, &w, gxp, gk, gwp, rp, n, op_out, stream);
    });
    return code != 0 ? PyLong_FromLong(code) : THPVariable_Wrap(out);
  });
}

// bind(address, ...) in the order of Entries
PyObject* Bind(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  void* p[5];
  if (n_args != 5) {
    PyErr_SetString(PyExc_TypeError, "bind takes five addresses");
    return nullptr;
  }
  for (int i = 0; i < 5; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (p[i] == nullptr) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null address");
      return nullptr;
    }
  }
  g_lib.skinny_gemm = reinterpret_cast<decltype(g_lib.skinny_gemm)>(p[0]);
  g_lib.argmax_rows = reinterpret_cast<decltype(g_lib.argmax_rows)>(p[1]);
  g_lib.dequant = reinterpret_cast<decltype(g_lib.dequant)>(p[2]);
  g_lib.lmhead = reinterpret_cast<decltype(g_lib.lmhead)>(p[3]);
  g_lib.shared_expert_down = reinterpret_cast<decltype(g_lib.shared_expert_down)>(p[4]);
  Py_RETURN_NONE;
}

#define QFG_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {QFG_METHOD("bind", Bind),
                           QFG_METHOD("skinny_gemm", SkinnyGemm),
                           QFG_METHOD("argmax_rows", ArgmaxRows),
                           QFG_METHOD("dequant", Dequant),
                           QFG_METHOD("lmhead", LmHead),
                           QFG_METHOD("shared_expert_down", SharedExpertDown),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) {
  PyObject* m = PyModule_Create(&g_module);
  // the torch whose headers this was compiled against: ops.py uses the module with no other
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", QFG_TORCH_VERSION) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
