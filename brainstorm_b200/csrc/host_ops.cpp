// The host side of the router's hot operators for plain calls, in native code.
//
// An eager step enqueues three launches whose kernels take a few microseconds each at decode
// sizes, and the Python around them (argument checks, allocation, views, a foreign call with
// twenty converted arguments) took 12 to 19 us per operator, more than the GPU did.  These
// functions do the same for the calls that programs make all the time - contiguous tensors of
// the right types on the current device, sizes known - and return None for any other
// call, before anything has been enqueued: the Python operator then takes it and does the
// checking and the explaining.  They call the same entry points of the C library, and like the
// foreign calls they stand for they let other Python threads run meanwhile: an allocation may
// synchronise, a launch waits while the queue of the stream is full.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include "../../include/brt_b200.h"

namespace {

PyObject* g_dense;  // attribute name on index tensors

// A plain torch.Tensor (no subclass, no functional wrapper) with memory on the GPU.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.has_storage()) return nullptr;
  if (t.unsafeGetTensorImpl()->key_set().has_any(
          c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::Functionalize,
                               c10::DispatchKey::Negative, c10::DispatchKey::Conjugate})))
    return nullptr;
  return &t;
}
bool modes_active() {
  return c10::impl::TorchDispatchModeTLS::any_modes_set() ||
         at::impl::torch_function_mode_enabled();
}
bool int32c(const at::Tensor* t, int64_t dims) {
  return t != nullptr && t->scalar_type() == at::kInt && t->dim() == dims && t->is_contiguous();
}
int dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return BRT_F32;
    case at::kHalf: return BRT_F16;
    case at::kBFloat16: return BRT_BF16;
    default: return -1;
  }
}
at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, c10::Device device) {
  return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}

// The device all tensors of a call must be on, when it is the current one; its stream.
struct Place {
  c10::Device device;
  c10::cuda::CUDAStream stream;
  static bool of(const at::Tensor& t) { return t.get_device() == c10::cuda::current_device(); }
  explicit Place(const at::Tensor& t)
      : device(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device())) {}
  void* handle() const { return stream.stream(); }
};
bool same_device(const at::Tensor& a, const at::Tensor* b) {
  return b == nullptr || a.get_device() == b->get_device();
}

// Other Python threads run while this lives.  Everything that touches a Python object comes before
// or after; what is made inside (tensors that no Python object wraps yet) needs no lock.
struct Unlocked {
  PyThreadState* const state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
// The addresses of a call's tensors, and the memory behind them kept until the call has been
// enqueued: meanwhile another thread may drop a tensor or give it other memory.
struct Memory {
  c10::SmallVector<c10::Storage, 8> held;
  void* of(const at::Tensor* t) {
    if (t == nullptr) return nullptr;
    held.push_back(t->storage());
    return t->data_ptr();
  }
  int32_t* ints(const at::Tensor* t) { return static_cast<int32_t*>(of(t)); }
};

// The note of an index operator on the tensor it returns, see _C/router.py.
bool mark(PyObject* indices, const at::Tensor& counts) {
  PyObject* c = THPVariable_Wrap(counts);
  const bool ok = c != nullptr && PyObject_SetAttr(indices, g_dense, c) == 0;
  Py_XDECREF(c);
  return ok;
}
// A new reference or null (no error set) when there is no such attribute.
PyObject* attribute(PyObject* o, PyObject* name) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (v == nullptr) PyErr_Clear();
  return v;
}

// The dense counts noted on `indices`, or null.
const int32_t* dense_counts(PyObject* indices, int64_t paths, Memory& memory) {
  PyObject* note = attribute(indices, g_dense);
  if (note == nullptr) return nullptr;
  const at::Tensor* t = plain(note);
  const bool ok = int32c(t, 1) && t->numel() == paths &&
                  same_device(THPVariable_Unpack(indices), t);
  const int32_t* const p = ok ? memory.ints(t) : nullptr;
  Py_DECREF(note);
  return p;
}

struct Caps {
  const int32_t* ptr = nullptr;
  int num = 0;
  bool ok = true;
  Caps(PyObject* o, const at::Tensor& like, Memory& memory) {
    if (o == Py_None) return;
    const at::Tensor* t = plain(o);
    ok = int32c(t, 1) && same_device(like, t);
    if (!ok) return;
    ptr = memory.ints(t);
    num = (int)t->numel();
  }
};

// 0, 1, or -1 for an object without a truth value (no error is left set).
int truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) PyErr_Clear();
  return v;
}

// Errors keep the kind that torch gives them in Python: torch.OutOfMemoryError above all.
template <typename F>
PyObject* guarded(F&& body) {
  try {
    PyObject* r = body();
    if (r != nullptr || PyErr_Occurred()) return r;
    Py_RETURN_NONE;
  } catch (const std::exception&) {
    torch::translate_exception_to_python(std::current_exception());
  } catch (...) {
    PyErr_SetString(PyExc_RuntimeError, "unknown error in a router operator");
  }
  return nullptr;
}
void* data_or_null(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// scan(hot_mask, prefix | None, threshold | None, caps | None, capacity_padding, path_wise,
//      with_mask): seat indices; with prefix and threshold of the mask throttled on the way.
// -> (indices, loads) or (indices, loads, throttled mask | None)
PyObject* scan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 7 || modes_active() || brt_index_status() != BRT_OK) return nullptr;
    const at::Tensor* mask = plain(a[0]);
    if (!int32c(mask, 2) || mask->numel() == 0 || !Place::of(*mask)) return nullptr;
    const bool throttle = a[1] != Py_None;
    const at::Tensor *prefix = nullptr, *threshold = nullptr;
    const int64_t T = mask->size(0), E = mask->size(1);
    if (throttle) {
      prefix = plain(a[1]);
      threshold = plain(a[2]);
      if (!int32c(prefix, 1) || !int32c(threshold, 1) || prefix->numel() != E ||
          threshold->numel() != E || !same_device(*mask, prefix) ||
          !same_device(*mask, threshold))
        return nullptr;
    }
    Memory memory;
    const Caps caps(a[3], *mask, memory);
    if (!caps.ok) return nullptr;
    const int cpad = truth(a[4]), pwise = truth(a[5]), with_mask = truth(a[6]);
    if (cpad < 0 || pwise < 0 || with_mask < 0) return nullptr;
    if (throttle && E % 4 != 0) return nullptr;  // takes two launches
    const Place p(*mask);
    const int32_t* const m = memory.ints(mask);
    int32_t* const before = memory.ints(prefix);
    const int32_t* const limit = memory.ints(threshold);
    at::Tensor indices, loads, counts, throttled;
    int rc;
    {
      const Unlocked unlocked;
      indices = empty({T, E}, at::kInt, p.device);
      const at::Tensor both = empty({2, E}, at::kInt, p.device);
      loads = both.select(0, 0);
      counts = both.select(0, 1);
      if (with_mask) throttled = empty({T, E}, at::kInt, p.device);
      const int64_t bytes = (int64_t)brt_index_scratch_bytes(T, (int)E);
      const at::Tensor scratch = empty({bytes}, at::kByte, p.device);
      const auto out = static_cast<int32_t*>(indices.data_ptr());
      const auto l = static_cast<int32_t*>(loads.data_ptr());
      const auto c = static_cast<int32_t*>(counts.data_ptr());
      rc = throttle ? brt_throttle_and_generate_indices(
                          m, out, l, c, before, limit,
                          static_cast<int32_t*>(data_or_null(throttled)), T, (int)E, caps.ptr,
                          caps.num, cpad, pwise, scratch.data_ptr(), (size_t)bytes, p.handle())
                    : brt_generate_indices_and_loads(m, out, l, c, T, (int)E, caps.ptr, caps.num,
                                                     cpad, pwise, 0, scratch.data_ptr(),
                                                     (size_t)bytes, p.handle());
    }
    if (rc != BRT_OK) return nullptr;  // nothing was enqueued: the operator says why
    PyObject* i = THPVariable_Wrap(indices);
    if (i == nullptr || !mark(i, counts)) {
      Py_XDECREF(i);
      return nullptr;
    }
    if (!throttle) return Py_BuildValue("(NN)", i, THPVariable_Wrap(loads));
    if (with_mask)
      return Py_BuildValue("(NNN)", i, THPVariable_Wrap(loads), THPVariable_Wrap(throttled));
    return Py_BuildValue("(NNO)", i, THPVariable_Wrap(loads), Py_None);
  });
}

// route_scores(score, decision, top_k, threshold, residual_path, output, caps | None,
//              capacity_padding, path_wise, prefix | None, throttle_capacity | None, with_gates,
//              with_mask) -> (out, loads, gates | None, mask | None)
PyObject* route_scores(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 13 || modes_active() || brt_index_status() != BRT_OK) return nullptr;
    const at::Tensor* score = plain(a[0]);
    if (score == nullptr || score->scalar_type() != at::kFloat || score->dim() != 2 ||
        !score->is_contiguous() || score->numel() == 0 || !Place::of(*score))
      return nullptr;
    const int64_t T = score->size(0), E = score->size(1);
    if (E > 256 || E % 4 != 0) return nullptr;
    const long decision = PyLong_AsLong(a[1]), top_k = PyLong_AsLong(a[2]);
    const double threshold = PyFloat_AsDouble(a[3]);
    const long residual = PyLong_AsLong(a[4]), output = PyLong_AsLong(a[5]);
    if (PyErr_Occurred()) {  // numbers of other kinds: the operator converts them
      PyErr_Clear();
      return nullptr;
    }
    if (top_k != (int)top_k || residual != (int)residual) return nullptr;
    Memory memory;
    const Caps caps(a[6], *score, memory);
    const int cpad = truth(a[7]), pwise = truth(a[8]);
    const int with_gates = truth(a[11]), with_mask = truth(a[12]);
    if (cpad < 0 || pwise < 0 || with_gates < 0 || with_mask < 0) return nullptr;
    if (!caps.ok || (cpad != 0 && caps.num < 1)) return nullptr;
    const bool seats =
        output == BRT_ROUTE_SEAT_INDICES || output == BRT_ROUTE_THROTTLED_SEAT_INDICES;
    const bool throttles =
        output == BRT_ROUTE_THROTTLED_MASK || output == BRT_ROUTE_THROTTLED_SEAT_INDICES;
    const at::Tensor *prefix = nullptr, *limit = nullptr;
    if (throttles) {
      prefix = plain(a[9]);
      limit = plain(a[10]);
      if (!int32c(prefix, 1) || !int32c(limit, 1) || prefix->numel() != E ||
          limit->numel() != E || !same_device(*score, prefix) || !same_device(*score, limit))
        return nullptr;
    }
    if (with_mask && !seats) return nullptr;
    const Place p(*score);
    const auto s = static_cast<const float*>(memory.of(score));
    int32_t* const before = memory.ints(prefix);
    const int32_t* const room = memory.ints(limit);
    at::Tensor out, loads, counts, gates, mask;
    int rc;
    {
      const Unlocked unlocked;
      out = empty({T, E}, at::kInt, p.device);
      const at::Tensor both = empty({2, E}, at::kInt, p.device);
      loads = both.select(0, 0);
      counts = both.select(0, 1);
      if (with_gates) gates = empty({T, E}, at::kFloat, p.device);
      if (with_mask) mask = empty({T, E}, at::kInt, p.device);
      const int64_t bytes = (int64_t)brt_index_scratch_bytes(T, (int)E);
      const at::Tensor scratch = empty({bytes}, at::kByte, p.device);
      rc = brt_route_scores(
          s, T, (int)E, (int)decision, (int)top_k, (float)threshold, (int)residual, (int)output,
          static_cast<int32_t*>(out.data_ptr()), static_cast<int32_t*>(loads.data_ptr()),
          seats ? static_cast<int32_t*>(counts.data_ptr()) : nullptr, caps.ptr, caps.num, cpad,
          pwise, before, room, static_cast<float*>(data_or_null(gates)),
          static_cast<int32_t*>(data_or_null(mask)), scratch.data_ptr(), (size_t)bytes,
          p.handle());
    }
    if (rc != BRT_OK) return nullptr;
    PyObject* o = THPVariable_Wrap(out);
    if (o == nullptr || (seats && !mark(o, counts))) {
      Py_XDECREF(o);
      return nullptr;
    }
    PyObject* g = with_gates ? THPVariable_Wrap(gates) : Py_NewRef(Py_None);
    PyObject* m = with_mask ? THPVariable_Wrap(mask) : Py_NewRef(Py_None);
    return Py_BuildValue("(NNNN)", o, THPVariable_Wrap(loads), g, m);
  });
}

// dispatch(in_data, route_indices, loads, gates | None, max_path_load, total_rows): 1-D routing,
// seat indices straight out of an index operator, no tags -> the rows
PyObject* dispatch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 6 || modes_active()) return nullptr;
    const at::Tensor *x = plain(a[0]), *indices = plain(a[1]), *loads = plain(a[2]);
    if (x == nullptr || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0 ||
        !Place::of(*x) || !int32c(indices, 2) || !int32c(loads, 1) ||
        !same_device(*x, indices) || !same_device(*x, loads))
      return nullptr;
    const int dtype = dtype_of(*x);
    const int64_t T = x->size(0), E = indices->size(1);
    if (dtype < 0 || indices->size(0) != T || loads->numel() != E || E < 1 || E > 2048)
      return nullptr;
    const int64_t cell = x->numel() / T;
    if (dtype == BRT_F16 && cell % 2 != 0) return nullptr;
    const at::Tensor* gates = nullptr;
    if (a[3] != Py_None) {
      gates = plain(a[3]);
      if (gates == nullptr || gates->scalar_type() != x->scalar_type() ||
          !gates->is_contiguous() || gates->numel() != T * E || !same_device(*x, gates))
        return nullptr;
    }
    const long long mpl = PyLong_AsLongLong(a[4]), total = PyLong_AsLongLong(a[5]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return nullptr;
    }
    if (mpl < 0 || mpl > 0x7fffffffLL || total < 0) return nullptr;
    Memory memory;
    const int32_t* counts = dense_counts(a[1], E, memory);
    if (counts == nullptr) return nullptr;
    const Place p(*x);
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    shape[0] = total;
    const auto type = x->scalar_type();
    const void* const src = memory.of(x);
    const void* const g = memory.of(gates);
    const int32_t* const at_rows = memory.ints(indices);
    const int32_t* const l = memory.ints(loads);
    at::Tensor out;
    int rc;
    {
      const Unlocked unlocked;
      out = empty(shape, type, p.device);
      rc = brt_dispatch_with_indices_and_loads(src, out.data_ptr(), g, at_rows, l, nullptr, nullptr,
                                               T, cell, (int)E, (int)mpl, total, 1, 0, dtype,
                                               counts, nullptr, 0, p.handle());
    }
    if (rc != BRT_OK) return nullptr;
    return THPVariable_Wrap(out);
  });
}

// combine(in_data, route_indices, loads, gates | None, out_data | None, max_path_padding): seat
// indices, at least two cells -> the cells (out_data itself when given)
PyObject* combine(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 6 || modes_active()) return nullptr;
    const at::Tensor *x = plain(a[0]), *indices = plain(a[1]), *loads = plain(a[2]);
    if (x == nullptr || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0 ||
        !Place::of(*x) || !int32c(indices, 2) || !int32c(loads, 1) ||
        !same_device(*x, indices) || !same_device(*x, loads))
      return nullptr;
    const int dtype = dtype_of(*x);
    const int64_t T = indices->size(0), E = indices->size(1);
    if (dtype < 0 || T < 2 || E < 1 || loads->numel() != E) return nullptr;
    const int64_t rows = x->size(0), cell = x->numel() / rows;
    const at::Tensor* gates = nullptr;
    int gate_type = 0;
    if (a[3] != Py_None) {
      gates = plain(a[3]);
      if (gates == nullptr || !gates->is_contiguous() || gates->numel() != T * E ||
          !same_device(*x, gates))
        return nullptr;
      gate_type = dtype_of(*gates);
      if (gate_type != BRT_F32 && gate_type != dtype) return nullptr;
    }
    const at::Tensor* residual = nullptr;
    if (a[4] != Py_None) {
      residual = plain(a[4]);
      if (residual == nullptr || !residual->is_contiguous() || residual->numel() != T * cell ||
          residual->scalar_type() != x->scalar_type() || !same_device(*x, residual))
        return nullptr;
    }
    const int padded = truth(a[5]);
    if (padded < 0) return nullptr;
    const int64_t mpl = padded ? rows / E : 0;
    if (mpl > 0x7fffffffLL) return nullptr;
    Memory memory;
    const Place p(*x);
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    shape[0] = T;
    const auto type = x->scalar_type();
    const void* const src = memory.of(x);
    const void* const g = memory.of(gates);
    const int32_t* const at_rows = memory.ints(indices);
    const int32_t* const l = memory.ints(loads);
    void* dst = memory.of(residual);
    at::Tensor out;
    int rc;
    {
      const Unlocked unlocked;
      if (residual == nullptr) {
        out = empty(shape, type, p.device);
        dst = out.data_ptr();
      }
      rc = brt_combine_with_indices_and_loads(src, dst, g, at_rows, l, T, cell, (int)E,
                                              (int32_t)mpl, residual != nullptr, dtype, gate_type,
                                              p.handle());
    }
    if (rc != BRT_OK) return nullptr;
    return residual != nullptr ? Py_NewRef(a[4]) : THPVariable_Wrap(out);
  });
}

PyMethodDef methods[] = {
    {"scan", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(scan)), METH_FASTCALL, nullptr},
    {"route_scores", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(route_scores)),
     METH_FASTCALL, nullptr},
    {"dispatch", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(dispatch)), METH_FASTCALL,
     nullptr},
    {"combine", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(combine)), METH_FASTCALL,
     nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops() {
  g_dense = PyUnicode_InternFromString("_brt_dense_counts");
  PyObject* const m = g_dense != nullptr ? PyModule_Create(&module) : nullptr;
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
