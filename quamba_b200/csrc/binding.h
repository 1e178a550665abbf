// Shared pieces of the CPython extension (binding.cpp, binding_layers.cpp).
#pragma once

#include <Python.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <array>
#include <stdexcept>
#include <string>

#include "../../include/quamba_b200.h"

namespace qbn {

using at::Tensor;

struct PyErr {};                                             // a Python exception is already set
// Python's other threads run while the library or the allocator works: a launch waits where the queue is full, and a first call
// sets attributes or allocates.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
// A strong reference: between two launches other threads may replace what a module holds.
class Ref {
 public:
  Ref() = default;
  static Ref own(PyObject* o) { Ref r; r.o_ = o; return r; }
  static Ref share(PyObject* o) { return own(Py_XNewRef(o)); }
  Ref(const Ref& r) : o_(Py_XNewRef(r.o_)) {}
  Ref(Ref&& r) noexcept : o_(r.o_) { r.o_ = nullptr; }
  Ref& operator=(Ref r) noexcept { std::swap(o_, r.o_); return *this; }
  ~Ref() { Py_XDECREF(o_); }
  operator PyObject*() const { return o_; }

 private:
  PyObject* o_ = nullptr;
};
struct NotPlain {};                                          // the layer functions: walk the modules instead

void run_call(const char* name, int (*f)(const void*, void*), const void* args, cudaStream_t st);
#define QBN_CALL(fn, s, st) ::qbn::run_call(#fn, [](const void* qbn_p, void* qbn_st) { return fn(static_cast<const std::remove_reference_t<decltype(s)>*>(qbn_p), qbn_st); }, &(s), (st))

inline void need(bool ok, const char* msg) { if (!ok) throw std::runtime_error(msg); }
inline void need(bool ok, const std::string& msg) { if (!ok) throw std::runtime_error(msg); }
inline void cuda_i8(const Tensor& t, const char* name) {
  if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be a CUDA tensor");
  if (t.scalar_type() != at::kChar) throw std::runtime_error(std::string(name) + " must be int8");
}
inline void cuda_f32(const Tensor& t, const char* name) {
  if (!t.is_cuda() || t.scalar_type() != at::kFloat) throw std::runtime_error(std::string(name) + " must be a float32 CUDA tensor");
}
inline void on_gpu(const Tensor& t, const char* name) {      // nothing given passes
  if (t.defined() && !t.is_cuda()) throw std::runtime_error(std::string(name) + " must be a CUDA tensor");
}
inline const float* scale_of(const Tensor& t, const char* name) {
  cuda_f32(t, name);
  return static_cast<const float*>(t.data_ptr());
}
inline Tensor contiguous(const Tensor& t) {
  if (t.is_contiguous()) return t;
  const NoGil released;
  return t.contiguous();
}
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline int8_t* i8(const Tensor& t) { return static_cast<int8_t*>(ptr(t)); }
inline float* f32(const Tensor& t) { return static_cast<float*>(ptr(t)); }
inline int32_t* i32(const Tensor& t) { return static_cast<int32_t*>(ptr(t)); }
inline std::array<int64_t, 3> strides3(int64_t a, int64_t b, int64_t c) { return {a, b, c}; }

inline Tensor as_tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw std::runtime_error("expected a tensor, got " + std::string(Py_TYPE(o)->tp_name));
  return THPVariable_Unpack(o);
}
inline double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyErr{};
  return v;
}
inline long as_long(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyErr{};
  return v;
}

// Positional arguments of one call.
struct Args {
  PyObject* const* v;
  Py_ssize_t n;
  PyObject* object(int i) const {
    if (i >= n) throw std::runtime_error("missing argument " + std::to_string(i));
    return v[i];
  }
  bool is_none(int i) const { return object(i) == Py_None; }
  Tensor tensor(int i) const { return as_tensor(object(i)); }
  Tensor opt_tensor(int i) const { return is_none(i) ? Tensor() : as_tensor(v[i]); }
  double num(int i) const { return as_double(object(i)); }
  double num_or(int i, double d) const { return is_none(i) ? d : as_double(v[i]); }
  long integer(int i) const { return as_long(object(i)); }
  bool flag(int i) const {
    const int r = PyObject_IsTrue(object(i));
    if (r < 0) throw PyErr{};
    return r != 0;
  }
};

// The inputs' device made current, torch's stream on it, and outputs from its caching allocator.
struct Device {
  c10::cuda::CUDAGuard guard;
  cudaStream_t stream;
  c10::Device dev;
  explicit Device(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()), dev(t.device()) {}
  Tensor empty(at::IntArrayRef sizes, at::ScalarType t) const {
    const NoGil released;
    return Tensor(at::detail::empty_cuda(sizes, t, dev, std::nullopt));
  }
  Tensor empty_strided(at::IntArrayRef sizes, at::IntArrayRef strides, at::ScalarType t) const {
    const NoGil released;
    return Tensor(at::detail::empty_strided_cuda(sizes, strides, t, dev));
  }
};

inline PyObject* wrap(const Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); }
inline PyObject* wrap_tuple(std::initializer_list<Tensor> ts) {
  PyObject* r = PyTuple_New(ts.size());
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) PyTuple_SET_ITEM(r, i++, wrap(t));
  return r;
}
inline PyObject* wrap_list(std::initializer_list<Tensor> ts) {
  PyObject* r = PyList_New(ts.size());
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) PyList_SET_ITEM(r, i++, wrap(t));
  return r;
}

template <PyObject* (*F)(const Args&)>
PyObject* entry(PyObject*, PyObject* const* v, Py_ssize_t n) {
  try {
    return F(Args{v, n});
  } catch (const PyErr&) {
  } catch (const NotPlain&) {
    Py_RETURN_NONE;
  } catch (const c10::Error&) {
    torch::translate_exception_to_python(std::current_exception());   // torch's own types: out of memory, index, value errors
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}
#define QBN_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&::qbn::entry<::qbn::name>)), METH_FASTCALL, nullptr}

// ---- modules --------------------------------------------------------------------------------------------------------------
// Attribute names are interned once; a lookup is then a pointer-keyed dictionary probe.
#define QBN_NAME(x) ([]() -> PyObject* { static PyObject* s = PyUnicode_InternFromString(#x); return s; }())

inline const Tensor& plain(const Tensor& t, at::ScalarType type, c10::Device dev) {
  if (t.scalar_type() != type || t.device() != dev) throw NotPlain{};
  return t;
}

// A torch.nn.Module as its dictionaries: plain attributes, buffers, sub-modules.
struct Mod {
  Ref self, attrs, buffers;
  explicit Mod(PyObject* o);
  PyObject* find(PyObject* name) const {                     // borrowed, null when absent
    PyObject* r = PyDict_GetItem(attrs, name);
    return r != nullptr ? r : PyDict_GetItem(buffers, name);
  }
  PyObject* get(PyObject* name) const {
    PyObject* r = find(name);
    if (r == nullptr) throw NotPlain{};
    return r;
  }
  Tensor tensor(PyObject* name) const { return as_tensor(get(name)); }
  Tensor opt_tensor(PyObject* name) const {
    PyObject* r = get(name);
    return r == Py_None ? Tensor() : as_tensor(r);
  }
  // of the given type on the given device, as the kernels read it; anything else is for the module walk (and its errors)
  Tensor tensor_on(PyObject* name, at::ScalarType type, c10::Device dev) const { return plain(tensor(name), type, dev); }
  Tensor opt_tensor_on(PyObject* name, at::ScalarType type, c10::Device dev) const {
    const Tensor t = opt_tensor(name);
    return t.defined() ? plain(t, type, dev) : t;
  }
  double num(PyObject* name) const { return as_double(get(name)); }
  double num_or(PyObject* name, double d) const {
    PyObject* r = get(name);
    return r == Py_None ? d : as_double(r);
  }
  long integer(PyObject* name) const { return as_long(get(name)); }
  bool flag(PyObject* name) const { return PyObject_IsTrue(get(name)) == 1; }
  // the sub-module, which must be exactly of class `type` and carry no hooks
  Mod child(PyObject* name, PyTypeObject* type) const;
  void require_plain(PyTypeObject* type) const;
  void require_own(PyObject* method) const;                  // the method is the class's, not one set on the instance
};

struct Types {
  PyTypeObject *QRMSNorm, *QRMSNormGated, *Quamb2Conv1D, *Quamba2ChunkScan, *QHadamard, *QCausalConv1D, *QSScan, *W4A8B16O16Linear, *W4A8B8O8Linear,
      *W4A8B8O8LinearParallel, *W8A8B8O8Linear, *W8A8B8O8LinearParallel, *W8A8B16O16Linear;
};
extern Types g_types;
PyObject* set_types(PyObject*, PyObject* dict);              // {class name: class}

// ---- Quamba2 conv ---------------------------------------------------------------------------------------------------------
struct Conv2 {
  Tensor weight, bias, hgr, dgr, out_scale[3];               // order of the segments: x, B, C
  double in[3], w_scale[3], b_scale[3];
  int64_t x_dim, headdim, d_state, groups;
  int silu = 1;
  void check();                                              // validates ranges and scales, makes the ranges contiguous
  template <typename S>
  void fill(S& s, int64_t dim) const {
    s.weight = i8(weight); s.bias = i8(bias); s.head_group_range = i32(hgr); s.dim_group_range = i32(dgr);
    s.x_scales = f32(out_scale[0]); s.B_scales = f32(out_scale[1]); s.C_scales = f32(out_scale[2]);
    s.dim = dim; s.width = weight.size(1); s.x_dim = x_dim; s.x_headdim = headdim; s.d_state = d_state; s.n_groups = groups;
    s.nhead_groups = hgr.defined() ? hgr.size(1) : 0; s.ndim_groups = dgr.defined() ? dgr.size(2) : 0;
    s.scale_x = in[0]; s.scale_B = in[1]; s.scale_C = in[2];
    s.scale_wx = w_scale[0]; s.scale_wB = w_scale[1]; s.scale_wC = w_scale[2];
    s.scale_bx = b_scale[0]; s.scale_bB = b_scale[1]; s.scale_bC = b_scale[2];
    s.silu = silu;
  }
  qb_quamba2_conv1d_fwd_args fwd_args(int64_t dim) const { qb_quamba2_conv1d_fwd_args s{}; fill(s, dim); return s; }
  qb_quamba2_conv1d_update_args update_args(int64_t dim) const { qb_quamba2_conv1d_update_args s{}; fill(s, dim); return s; }
};

// ---- W4A8 weights ---------------------------------------------------------------------------------------------------------
struct W4Dims { int64_t n, k; bool per_channel; };
W4Dims w4_dims(PyObject* prep);
// a (m, k) int8 rows x the prepared weight -> out; picks the nibble kernel for a few rows of a per-channel weight
void w4a8_run(PyObject* prep, const W4Dims& w, const int8_t* a, int64_t lda, int64_t m, const float* s_tok, bool per_row, void* out,
              int64_t ldo, bool int8, bool transpose, cudaStream_t st);

PyObject* mamba2_layer(const Args& a);
PyObject* mamba1_layer(const Args& a);

}  // namespace qbn
