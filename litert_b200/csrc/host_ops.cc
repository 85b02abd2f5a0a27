// The calls of ops.py whose device work is a few microseconds, as a CPython extension over the C ABI: argument
// checks, workspace look-up, output allocation and the launch in native code.
//
// What bounds such a call is the host: through ctypes one FULLY_CONNECTED took 18 us to enqueue (conversion of
// eighteen arguments, five tensor property checks in Python, the stream look-up) against 5 to 9 us of kernels;
// through this module 6 us (4 with one launch), nearly all of it the kernel launches (measured, B200 host).
//
// Every function returns the result, or None when anything about the call is not the plain case: a tensor that is
// not contiguous or has another type, a workspace that is absent or too small, an error code. The caller then
// takes its general path, which converts, allocates, or raises the error.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>

#include "../../include/litert_b200.h"

namespace {

PyObject *s_packed, *s_row_sums, *s_kfsum, *s_n, *s_k, *s_blocksize, *s_zero, *s_scratch, *s_sdpa;

// An attribute of a Python object for the duration of a call.
struct Attr {
  PyObject* o;
  Attr(PyObject* of, PyObject* name) : o(PyObject_GetAttr(of, name)) {
    if (!o) PyErr_Clear();
  }
  ~Attr() { Py_XDECREF(o); }
  Attr(const Attr&) = delete;
};

bool as_int(PyObject* o, int* v) {
  if (!o || !PyLong_Check(o)) return false;
  const long t = PyLong_AsLong(o);
  if (t == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  if (t < INT32_MIN || t > INT32_MAX) return false;
  *v = (int)t;
  return true;
}

bool as_float(PyObject* o, float* v) {
  if (o == Py_None) {
    *v = 0.0f;
    return true;
  }
  const double t = PyFloat_AsDouble(o);  // also ints and numpy numbers
  if (t == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *v = (float)t;
  return true;
}

// A contiguous CUDA tensor of one type, or "absent" (None) where that is allowed.
struct In {
  const at::Tensor* t = nullptr;
  bool ok = false;
  In(PyObject* o, at::ScalarType type, bool optional = false) {
    if (!o) return;
    if (o == Py_None) {
      ok = optional;
      return;
    }
    if (!THPVariable_CheckExact(o)) return;
    t = &THPVariable_Unpack(o);
    ok = t->is_cuda() && t->scalar_type() == type && t->is_contiguous();
  }
  template <typename T>
  T* ptr() const {
    return t ? static_cast<T*>(t->data_ptr()) : nullptr;
  }
};

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// The result tensor: the caller's own, or a new one on x's device. An undefined tensor: not the plain case.
at::Tensor result(PyObject* out, at::IntArrayRef shape, at::ScalarType type, const at::Tensor& x) {
  if (out != Py_None) {
    In o(out, type);
    if (!o.ok) return {};
    int64_t n = 1;
    for (int64_t s : shape) n *= s;
    if (o.t->numel() != n) return {};
    return *o.t;
  }
  return at::Tensor(at::detail::empty_cuda(shape, type, x.device(), std::nullopt));
}

PyObject* give(PyObject* out, at::Tensor y, int rc) {
  if (rc != B200_OK) Py_RETURN_NONE;  // the general path repeats the call and raises its error
  if (out != Py_None) {
    Py_INCREF(out);
    return out;
  }
  return THPVariable_Wrap(std::move(y));
}

// What the three FULLY_CONNECTED forms have in common.
struct Fc {
  Attr packed_o, n_o, k_o, zero_o, scratch_o;
  In packed, zero, scratch;
  int n = 0, k = 0, m = 0;
  bool ok = false;
  Fc(PyObject* weights, PyObject* ws, const In& x)
      : packed_o(weights, s_packed), n_o(weights, s_n), k_o(weights, s_k), zero_o(ws, s_zero), scratch_o(ws, s_scratch),
        packed(packed_o.o, at::kByte), zero(zero_o.o, at::kByte), scratch(scratch_o.o, at::kByte) {
    if (!x.ok || !packed.ok || !zero.ok || !scratch.ok || !as_int(n_o.o, &n) || !as_int(k_o.o, &k) || k <= 0) return;
    const int64_t rows = x.t->numel() / k;
    if (rows * k != x.t->numel() || rows <= 0 || rows > INT32_MAX) return;
    m = (int)rows;
    ok = (size_t)scratch.t->numel() >= b200_fc_scratch_bytes(m, k);
  }
};

// (x, weights, bias, input_zero_point, filter_zero_point, output_zero_point, multipliers, shifts, act_min, act_max, ws, out)
PyObject* fc_int8(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 12 || a[10] == Py_None) Py_RETURN_NONE;
  try {
    In x(a[0], at::kChar);
    Fc f(a[1], a[10], x);
    if (!f.ok) Py_RETURN_NONE;
    Attr rs_o(a[1], s_row_sums);
    In rs(rs_o.o, at::kInt), bias(a[2], at::kInt, true), mult(a[6], at::kInt), shift(a[7], at::kInt);
    int in_zp, f_zp, out_zp, lo, hi;
    if (!rs.ok || !bias.ok || !mult.ok || !shift.ok || !as_int(a[3], &in_zp) || !as_int(a[4], &f_zp) ||
        !as_int(a[5], &out_zp) || !as_int(a[8], &lo) || !as_int(a[9], &hi) || in_zp == INT32_MIN || f_zp == INT32_MIN)
      Py_RETURN_NONE;
    at::Tensor y = result(a[11], std::array<int64_t, 2>{f.m, f.n}, at::kChar, *x.t);
    if (!y.defined()) Py_RETURN_NONE;
    void* s = stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_fc_int8(x.ptr<int8_t>(), f.m, f.k, f.packed.ptr<void>(), f.n, rs.ptr<int32_t>(), bias.ptr<int32_t>(), -in_zp,
                      -f_zp, out_zp, mult.ptr<int32_t>(), shift.ptr<int32_t>(), mult.t->numel() > 1 ? 1 : 0, lo, hi,
                      static_cast<int8_t*>(y.data_ptr()), f.zero.ptr<void>(), f.scratch.ptr<void>(),
                      (size_t)f.scratch.t->numel(), s);
    Py_END_ALLOW_THREADS
    return give(a[11], std::move(y), rc);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

// (x, weights, filter_scales, bias, asymmetric, activation, ws, out)
PyObject* fc_hybrid(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 8 || a[6] == Py_None) Py_RETURN_NONE;
  try {
    In x(a[0], at::kFloat);
    Fc f(a[1], a[6], x);
    if (!f.ok) Py_RETURN_NONE;
    Attr rs_o(a[1], s_row_sums);
    In rs(rs_o.o, at::kInt), scales(a[2], at::kFloat), bias(a[3], at::kFloat, true);
    int activation;
    const int asym = PyObject_IsTrue(a[4]);
    if (!rs.ok || !scales.ok || !bias.ok || asym < 0 || !as_int(a[5], &activation)) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const int64_t ns = scales.t->numel();
    if (ns != 1 && ns != f.n) Py_RETURN_NONE;
    at::Tensor y = result(a[7], std::array<int64_t, 2>{f.m, f.n}, at::kFloat, *x.t);
    if (!y.defined()) Py_RETURN_NONE;
    void* s = stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_fc_hybrid(x.ptr<float>(), f.m, f.k, f.packed.ptr<void>(), f.n, rs.ptr<int32_t>(), scales.ptr<float>(),
                        ns > 1 ? 1 : 0, bias.ptr<float>(), asym, activation, static_cast<float*>(y.data_ptr()),
                        f.zero.ptr<void>(), f.scratch.ptr<void>(), (size_t)f.scratch.t->numel(), s);
    Py_END_ALLOW_THREADS
    return give(a[7], std::move(y), rc);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

// (x, weights, bias, ws, out)
PyObject* fc_w4(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 5 || a[3] == Py_None) Py_RETURN_NONE;
  try {
    In x(a[0], at::kFloat);
    Fc f(a[1], a[3], x);
    if (!f.ok) Py_RETURN_NONE;
    Attr kf_o(a[1], s_kfsum), bs_o(a[1], s_blocksize);
    In kf(kf_o.o, at::kFloat), bias(a[2], at::kFloat, true);
    int blocksize;
    if (!kf.ok || !bias.ok || !as_int(bs_o.o, &blocksize)) Py_RETURN_NONE;
    at::Tensor y = result(a[4], std::array<int64_t, 2>{f.m, f.n}, at::kFloat, *x.t);
    if (!y.defined()) Py_RETURN_NONE;
    void* s = stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_fc_w4(x.ptr<float>(), f.m, f.k, f.packed.ptr<void>(), f.n, blocksize, kf.ptr<float>(), bias.ptr<float>(),
                    static_cast<float*>(y.data_ptr()), f.zero.ptr<void>(), f.scratch.ptr<void>(),
                    (size_t)f.scratch.t->numel(), s);
    Py_END_ALLOW_THREADS
    return give(a[4], std::move(y), rc);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

// (q, k, v, lengths, mask, scale, logit_cap, k_scale, v_scale, ws)
PyObject* sdpa_decode(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 10 || a[9] == Py_None || a[6] == Py_None) Py_RETURN_NONE;
  try {
    if (!THPVariable_CheckExact(a[0]) || !THPVariable_CheckExact(a[1])) Py_RETURN_NONE;
    const at::ScalarType qt = THPVariable_Unpack(a[0]).scalar_type(), kt = THPVariable_Unpack(a[1]).scalar_type();
    if (qt != at::kHalf && qt != at::kFloat) Py_RETURN_NONE;
    if (kt != at::kHalf && kt != at::kFloat && kt != at::kChar) Py_RETURN_NONE;
    Attr ws_o(a[9], s_sdpa);
    In q(a[0], qt), k(a[1], kt), v(a[2], kt), lengths(a[3], at::kInt, true), mask(a[4], at::kFloat, true),
        ks(a[7], at::kFloat, true), vs(a[8], at::kFloat, true), ws(ws_o.o, at::kByte);
    float scale, cap;
    if (!q.ok || !k.ok || !v.ok || !lengths.ok || !mask.ok || !ks.ok || !vs.ok || !ws.ok || !as_float(a[5], &scale) ||
        !as_float(a[6], &cap))
      Py_RETURN_NONE;
    if (q.t->dim() != 4 || k.t->dim() != 4 || q.t->size(1) != 1 || q.t->numel() == 0) Py_RETURN_NONE;
    const int b = (int)q.t->size(0), n = (int)q.t->size(2), h = (int)q.t->size(3);
    const int s_max = (int)k.t->size(1), nkv = (int)k.t->size(2);
    if ((size_t)ws.t->numel() < b200_sdpa_workspace_bytes(b, n, nkv, h, s_max)) Py_RETURN_NONE;
    at::Tensor y = result(Py_None, q.t->sizes(), qt, *q.t);
    auto code = [](at::ScalarType t) { return t == at::kHalf ? B200_DTYPE_F16 : t == at::kChar ? B200_DTYPE_I8 : B200_DTYPE_F32; };
    void* s = stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_sdpa_decode(q.ptr<void>(), k.ptr<void>(), v.ptr<void>(), ks.ptr<float>(), vs.ptr<float>(), lengths.ptr<int32_t>(),
                          mask.ptr<float>(), y.data_ptr(), b, n, nkv, h, s_max, code(qt), code(kt), scale, cap,
                          ws.ptr<void>(), (size_t)ws.t->numel(), s);
    Py_END_ALLOW_THREADS
    return give(Py_None, std::move(y), rc);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

PyMethodDef kMethods[] = {
    {"fc_int8", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fc_int8)), METH_FASTCALL, nullptr},
    {"fc_hybrid", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fc_hybrid)), METH_FASTCALL, nullptr},
    {"fc_w4", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fc_w4)), METH_FASTCALL, nullptr},
    {"sdpa_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(sdpa_decode)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops(void) {
  s_packed = PyUnicode_InternFromString("packed");
  s_row_sums = PyUnicode_InternFromString("row_sums");
  s_kfsum = PyUnicode_InternFromString("kfsum");
  s_n = PyUnicode_InternFromString("n");
  s_k = PyUnicode_InternFromString("k");
  s_blocksize = PyUnicode_InternFromString("blocksize");
  s_zero = PyUnicode_InternFromString("zero");
  s_scratch = PyUnicode_InternFromString("scratch");
  s_sdpa = PyUnicode_InternFromString("sdpa");
  return PyModule_Create(&kModule);
}
