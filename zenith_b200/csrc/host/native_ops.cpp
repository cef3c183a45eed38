// Native host path of the operators in zenith_b200/ops.py: one C++ call per operator instead of a chain of Python
// checks, torch.empty, the stream query and a ctypes call.
//
// What bounds a small operator is the host: a call took 15 - 17 us in Python (argument checks 4, output allocation 2,
// stream 1, ctypes with 14 - 24 arguments 4, launch 3 - 5) against 2 - 10 us of kernel time, so back-to-back calls left
// the GPU idle most of the time.  Every function here checks its arguments, allocates the result from torch's caching
// allocator, calls the C ABI on torch's current stream and returns the tensor.
//
// Only well-formed calls are served: exact tensors (or parameters) on the current device, the documented types, ranks
// and layouts, plain Python numbers.  Anything else, including a non-zero status of the C ABI, returns None and the
// Python function goes on with its own checks, which name the error; no message is written twice.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>
#include <cmath>
#include "../../../include/zenith_b200.h"

namespace {

using at::ScalarType;

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

inline const at::Tensor* tensor_of(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}

// A contiguous CUDA tensor of this type and rank (rank < 0: any) on device `dev`.
inline bool plain(const at::Tensor* t, int dev, ScalarType st, int rank) {
  return t && t->defined() && t->is_cuda() && t->get_device() == dev && t->scalar_type() == st &&
         (rank < 0 || t->dim() == rank) && t->is_contiguous() && t->layout() == at::kStrided;
}

// The same, with rows a caller may have strided (row views of a wider matrix).
inline bool plain_rows(const at::Tensor* t, int dev, ScalarType st) {
  if (!(t && t->defined() && t->is_cuda() && t->get_device() == dev && t->scalar_type() == st && t->dim() == 2 &&
        t->layout() == at::kStrided))
    return false;
  if (t->is_contiguous()) return true;
  return (t->size(1) <= 1 || t->stride(1) == 1) && t->stride(0) >= t->size(1);
}

// A contiguous vector of at least the n entries that a kernel reads.
inline bool vector_of(const at::Tensor* t, int dev, ScalarType st, int64_t n) { return plain(t, dev, st, 1) && t->numel() >= n; }

// None or a contiguous fp32 vector of n entries.
inline bool vector_or_none(PyObject* o, int dev, int64_t n, const float** p) {
  *p = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = tensor_of(o);
  if (!plain(t, dev, at::kFloat, 1) || t->numel() != n) return false;
  *p = static_cast<const float*>(t->const_data_ptr());
  return true;
}

inline bool number(PyObject* o, double* v) {
  if (PyFloat_CheckExact(o)) {
    *v = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (PyLong_CheckExact(o)) {
    *v = PyLong_AsDouble(o);
    if (*v == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    return true;
  }
  return false;
}

inline bool integer(PyObject* o, int* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long long x = PyLong_AsLongLongAndOverflow(o, &overflow);
  if (overflow || x < INT32_MIN || x > INT32_MAX) return false;
  *v = int(x);
  return true;
}

inline bool fits(int64_t a) { return a > 0 && a <= INT32_MAX; }

inline at::Tensor empty(at::IntArrayRef sizes, ScalarType st, int dev) {
  return at::detail::empty_cuda(sizes, st, c10::Device(c10::kCUDA, c10::DeviceIndex(dev)), std::nullopt);
}

inline void* stream_of(int dev) { return c10::cuda::getCurrentCUDAStream(c10::DeviceIndex(dev)).stream(); }

// Runs `body` (bool(at::Tensor* outs): false = not served) without the interpreter lock; None or the wrapped result(s).
template <int NOUT, typename F>
PyObject* serve(F&& body) {
  at::Tensor outs[NOUT];
  bool ok = false;
  try {
    NoGil free;
    ok = body(outs);
  } catch (const std::exception&) {
    ok = false;  // e.g. out of memory: the Python path meets it again and reports it
  }
  if (!ok) Py_RETURN_NONE;
  if (NOUT == 1 || !outs[NOUT - 1].defined()) return THPVariable_Wrap(std::move(outs[0]));
  PyObject* tup = PyTuple_New(NOUT);
  if (!tup) return nullptr;
  for (int i = 0; i < NOUT; ++i) {
    PyObject* w = THPVariable_Wrap(std::move(outs[i]));
    if (!w) {
      Py_DECREF(tup);
      return nullptr;
    }
    PyTuple_SET_ITEM(tup, i, w);
  }
  return tup;
}

inline int current_device() {
  try {
    return int(c10::cuda::current_device());
  } catch (const std::exception&) {
    return -1;  // no device: no tensor is served
  }
}

#define ARGS(n)                                                                            \
  if (nargs != (n)) {                                                                      \
    PyErr_Format(PyExc_TypeError, "%s takes %d arguments, got %zd", __func__, n, nargs);   \
    return nullptr;                                                                        \
  }                                                                                        \
  const int dev = current_device()

// ---------------------------------------------------------------------------------------------
// elementwise
// ---------------------------------------------------------------------------------------------
PyObject* gelu(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(1);
  const at::Tensor* x = tensor_of(a[0]);
  const bool f32 = plain(x, dev, at::kFloat, -1);
  if (!f32 && !plain(x, dev, at::kHalf, -1)) Py_RETURN_NONE;
  if (x->numel() == 0) Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty(x->sizes(), x->scalar_type(), dev);
    return f32 ? zen_gelu_f32(static_cast<const float*>(x->const_data_ptr()), static_cast<float*>(o[0].data_ptr()), x->numel(), stream_of(dev)) == ZEN_OK
               : zen_gelu_f16(x->const_data_ptr(), o[0].data_ptr(), x->numel(), stream_of(dev)) == ZEN_OK;
  });
}

PyObject* relu(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(1);
  const at::Tensor* x = tensor_of(a[0]);
  if (!plain(x, dev, at::kFloat, -1) || x->numel() == 0) Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty(x->sizes(), at::kFloat, dev);
    return zen_relu_f32(static_cast<const float*>(x->const_data_ptr()), static_cast<float*>(o[0].data_ptr()), x->numel(), stream_of(dev)) == ZEN_OK;
  });
}

// quantize(x, scale, zero_point, round_mode)
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(4);
  const at::Tensor* x = tensor_of(a[0]);
  const bool f32 = plain(x, dev, at::kFloat, -1);
  double scale;
  int zp, mode;
  if ((!f32 && !plain(x, dev, at::kHalf, -1)) || x->numel() == 0 || !number(a[1], &scale) || !integer(a[2], &zp) || !integer(a[3], &mode))
    Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty(x->sizes(), at::kChar, dev);
    int8_t* q = static_cast<int8_t*>(o[0].data_ptr());
    return f32 ? zen_quantize_f32(static_cast<const float*>(x->const_data_ptr()), q, x->numel(), float(scale), zp, mode, stream_of(dev)) == ZEN_OK
               : zen_quantize_f16(x->const_data_ptr(), q, x->numel(), float(scale), zp, mode, stream_of(dev)) == ZEN_OK;
  });
}

// dequantize(q, scale, zero_point)
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(3);
  const at::Tensor* q = tensor_of(a[0]);
  double scale;
  int zp;
  if (!plain(q, dev, at::kChar, -1) || q->numel() == 0 || !number(a[1], &scale) || !integer(a[2], &zp)) Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty(q->sizes(), at::kFloat, dev);
    return zen_dequantize_f32(static_cast<const int8_t*>(q->const_data_ptr()), static_cast<float*>(o[0].data_ptr()), q->numel(), float(scale), zp,
                              stream_of(dev)) == ZEN_OK;
  });
}

// ---------------------------------------------------------------------------------------------
// LayerNorm
// ---------------------------------------------------------------------------------------------
// layernorm(x, gamma, beta, eps)
PyObject* layernorm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(4);
  const at::Tensor *x = tensor_of(a[0]), *g = tensor_of(a[1]), *b = tensor_of(a[2]);
  double eps;
  const bool f32 = plain(x, dev, at::kFloat, 2);
  if ((!f32 && !plain(x, dev, at::kHalf, 2)) || !number(a[3], &eps)) Py_RETURN_NONE;
  const int64_t rows = x->size(0), hidden = x->size(1);
  if (!vector_of(g, dev, x->scalar_type(), hidden) || !vector_of(b, dev, x->scalar_type(), hidden) || !fits(rows) || !fits(hidden)) Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty(x->sizes(), x->scalar_type(), dev);
    if (f32)
      return zen_layernorm_f32(static_cast<const float*>(x->const_data_ptr()), static_cast<const float*>(g->const_data_ptr()),
                               static_cast<const float*>(b->const_data_ptr()), static_cast<float*>(o[0].data_ptr()), int(rows), int(hidden),
                               float(eps), stream_of(dev)) == ZEN_OK;
    return zen_layernorm_f16(x->const_data_ptr(), g->const_data_ptr(), b->const_data_ptr(), o[0].data_ptr(), int(rows), int(hidden),
                             float(eps), stream_of(dev)) == ZEN_OK;
  });
}

// add_layernorm(x, residual, gamma, beta, eps, out_scale or None, round_mode): y, or (y, int8 copy)
PyObject* add_layernorm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(7);
  const at::Tensor *x = tensor_of(a[0]), *r = tensor_of(a[1]), *g = tensor_of(a[2]), *b = tensor_of(a[3]);
  double eps, scale = 1.0;
  int mode;
  const bool f32 = plain(x, dev, at::kFloat, 2), want_q = a[5] != Py_None;
  if ((!f32 && !plain(x, dev, at::kHalf, 2)) || !number(a[4], &eps) || (want_q && (f32 || !number(a[5], &scale) || scale == 0.0)) ||
      !integer(a[6], &mode))
    Py_RETURN_NONE;
  const int64_t rows = x->size(0), hidden = x->size(1);
  const ScalarType st = x->scalar_type();
  if (!plain(r, dev, st, 2) || r->sizes() != x->sizes() || !vector_of(g, dev, st, hidden) || !vector_of(b, dev, st, hidden) || !fits(rows) ||
      !fits(hidden))
    Py_RETURN_NONE;
  return serve<2>([&](at::Tensor* o) {
    o[0] = empty(x->sizes(), st, dev);
    if (f32)
      return zen_add_layernorm_f32(static_cast<const float*>(x->const_data_ptr()), static_cast<const float*>(r->const_data_ptr()),
                                   static_cast<const float*>(g->const_data_ptr()), static_cast<const float*>(b->const_data_ptr()),
                                   static_cast<float*>(o[0].data_ptr()), int(rows), int(hidden), float(eps), stream_of(dev)) == ZEN_OK;
    if (want_q) o[1] = empty(x->sizes(), at::kChar, dev);
    return zen_add_layernorm_f16(x->const_data_ptr(), r->const_data_ptr(), g->const_data_ptr(), b->const_data_ptr(), o[0].data_ptr(),
                                 want_q ? static_cast<int8_t*>(o[1].data_ptr()) : nullptr, float(scale), mode, int(rows), int(hidden),
                                 float(eps), stream_of(dev)) == ZEN_OK;
  });
}

// ---------------------------------------------------------------------------------------------
// GEMMs
// ---------------------------------------------------------------------------------------------
inline int out_code(ScalarType st) {
  switch (st) {
    case at::kInt: return ZEN_DT_S32;
    case at::kFloat: return ZEN_DT_F32;
    case at::kHalf: return ZEN_DT_F16;
    case at::kChar: return ZEN_DT_S8;
    default: return -1;
  }
}

// linear_int8(xq, wq, x_scale, w_scale, bias, act, out_dtype, out_scale or None, round_mode, flags)
PyObject* linear_int8(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(10);
  const at::Tensor *x = tensor_of(a[0]), *w = tensor_of(a[1]);
  if (!plain(x, dev, at::kChar, 2) || !plain(w, dev, at::kChar, 2) || !THPDtype_Check(a[6])) Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  const ScalarType ot = reinterpret_cast<THPDtype*>(a[6])->scalar_type;
  double xs, os = 1.0;
  int act, mode, flags;
  const float *ws, *bias;
  if (w->size(1) != K || !fits(M) || !fits(N) || !fits(K) || out_code(ot) < 0 || !number(a[2], &xs) || !vector_or_none(a[3], dev, N, &ws) ||
      !vector_or_none(a[4], dev, N, &bias) || !integer(a[5], &act) || (a[7] == Py_None ? ot == at::kChar : !number(a[7], &os)) ||
      !integer(a[8], &mode) || !integer(a[9], &flags))
    Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty({M, N}, ot, dev);
    return zen_linear_i8_ex(static_cast<const int8_t*>(x->const_data_ptr()), K, static_cast<const int8_t*>(w->const_data_ptr()), K, int(M), int(N),
                            int(K), float(xs), ws, bias, act, out_code(ot), float(os), mode, o[0].data_ptr(), N, nullptr, 0, nullptr, 0,
                            unsigned(flags), stream_of(dev)) == ZEN_OK;
  });
}

// linear_fp16(x, w, bias, act, out_dtype, flags)
PyObject* linear_fp16(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(6);
  const at::Tensor *x = tensor_of(a[0]), *w = tensor_of(a[1]);
  if (!plain_rows(x, dev, at::kHalf) || !plain(w, dev, at::kHalf, 2) || !THPDtype_Check(a[4])) Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  const ScalarType ot = reinterpret_cast<THPDtype*>(a[4])->scalar_type;
  int act, flags;
  const float* bias;
  if (w->size(1) != K || !fits(M) || !fits(N) || !fits(K) || (ot != at::kHalf && ot != at::kFloat) || !vector_or_none(a[2], dev, N, &bias) ||
      !integer(a[3], &act) || !integer(a[5], &flags))
    Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty({M, N}, ot, dev);
    return zen_linear_f16_ex(x->const_data_ptr(), M > 1 ? x->stride(0) : K, w->const_data_ptr(), K, int(M), int(N), int(K), bias, act,
                             out_code(ot), o[0].data_ptr(), N, unsigned(flags), stream_of(dev)) == ZEN_OK;
  });
}

// linear_fp32(x, w, bias, act)
PyObject* linear_fp32(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(4);
  const at::Tensor *x = tensor_of(a[0]), *w = tensor_of(a[1]);
  if (!plain(x, dev, at::kFloat, 2) || !plain(w, dev, at::kFloat, 2)) Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  int act;
  const float* bias;
  if (w->size(1) != K || !fits(M) || !fits(N) || !fits(K) || !vector_or_none(a[2], dev, N, &bias) || !integer(a[3], &act)) Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty({M, N}, at::kFloat, dev);
    return zen_linear_f32(static_cast<const float*>(x->const_data_ptr()), K, static_cast<const float*>(w->const_data_ptr()), K, int(M), int(N),
                          int(K), bias, act, static_cast<float*>(o[0].data_ptr()), N, stream_of(dev)) == ZEN_OK;
  });
}

// wmma_matmul(a, b)
PyObject* wmma_matmul(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(2);
  const at::Tensor *x = tensor_of(a[0]), *y = tensor_of(a[1]);
  if (!plain(x, dev, at::kHalf, 2) || !plain(y, dev, at::kHalf, 2)) Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), N = y->size(1);
  if (y->size(0) != K || !fits(M) || !fits(N) || !fits(K)) Py_RETURN_NONE;
  return serve<1>([&](at::Tensor* o) {
    o[0] = empty({M, N}, at::kFloat, dev);
    return zen_wmma_matmul_f16(x->const_data_ptr(), y->const_data_ptr(), static_cast<float*>(o[0].data_ptr()), int(M), int(N), int(K),
                               stream_of(dev)) == ZEN_OK;
  });
}

// matmul_f32(a, b): c, or (c, kernels launched) if there were several.  Where b is transposed in front of the product, the copy lives in an allocation of
// this call (torch's allocator keeps it in stream order).
PyObject* matmul_f32(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(2);
  const at::Tensor *x = tensor_of(a[0]), *y = tensor_of(a[1]);
  if (!plain(x, dev, at::kFloat, 2) || !plain(y, dev, at::kFloat, 2)) Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), N = y->size(1);
  if (y->size(0) != K || !fits(M) || !fits(N) || !fits(K)) Py_RETURN_NONE;
  int kernels = 1;
  PyObject* c = serve<1>([&](at::Tensor* o) {
    o[0] = empty({M, N}, at::kFloat, dev);
    const float *pa = static_cast<const float*>(x->const_data_ptr()), *pb = static_cast<const float*>(y->const_data_ptr());
    float* pc = static_cast<float*>(o[0].data_ptr());
    const int st = zen_matmul_f32_direct(pa, pb, pc, int(M), int(N), int(K), stream_of(dev));
    if (st != ZEN_ERR_NEEDS_WORKSPACE) return st == ZEN_OK;
    kernels = 2;
    const size_t bytes = zen_matmul_f32_workspace_bytes(int(N), int(K));
    at::Tensor ws = empty({int64_t(bytes)}, at::kByte, dev);
    return zen_matmul_f32(pa, pb, pc, int(M), int(N), int(K), ws.data_ptr(), bytes, stream_of(dev)) == ZEN_OK;
  });
  return !c || c == Py_None || kernels == 1 ? c : Py_BuildValue("Ni", c, kernels);
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------
// flash_attention(q, k, v, causal, kv_lens or None, scale or None), [batch, heads, seq, dim], fp16 or fp32: o, or (o, kernels launched) if
// there were several
PyObject* flash_attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  ARGS(6);
  const at::Tensor *q = tensor_of(a[0]), *k = tensor_of(a[1]), *v = tensor_of(a[2]);
  const bool f32 = plain(q, dev, at::kFloat, 4);
  if (!f32 && !plain(q, dev, at::kHalf, 4)) Py_RETURN_NONE;
  const ScalarType st = q->scalar_type();
  if (!plain(k, dev, st, 4) || !plain(v, dev, st, 4) || k->sizes() != q->sizes() || v->sizes() != q->sizes()) Py_RETURN_NONE;
  const int64_t B = q->size(0), H = q->size(1), S = q->size(2), D = q->size(3);
  const int32_t* lens = nullptr;
  if (a[4] != Py_None) {
    const at::Tensor* t = tensor_of(a[4]);
    if (!vector_of(t, dev, at::kInt, B)) Py_RETURN_NONE;
    lens = static_cast<const int32_t*>(t->const_data_ptr());
  }
  double scale;
  if (!PyBool_Check(a[3]) || !fits(B) || !fits(H) || !fits(S) || !fits(D)) Py_RETURN_NONE;
  if (a[5] == Py_None) scale = 1.0 / std::sqrt(double(D));
  else if (!number(a[5], &scale)) Py_RETURN_NONE;
  const int causal = a[3] == Py_True ? 1 : 0;
  const int64_t sb = H * S * D, sh = S * D;
  int kernels = 1;
  PyObject* out = serve<1>([&](at::Tensor* o) {
    void* s = stream_of(dev);
    o[0] = empty(q->sizes(), st, dev);
    if (!f32)
      return zen_flash_attention_f16(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o[0].data_ptr(), nullptr, 1.0f, int(B), int(H),
                                     int(S), int(D), sb, sh, D, sb, sh, D, sb, sh, D, sb, sh, D, lens, causal, float(scale), s) == ZEN_OK;
    const float *pq = static_cast<const float*>(q->const_data_ptr()), *pk = static_cast<const float*>(k->const_data_ptr()),
                *pv = static_cast<const float*>(v->const_data_ptr());
    float* po = static_cast<float*>(o[0].data_ptr());
    const int one = zen_flash_attention_f32_direct(pq, pk, pv, po, int(B), int(H), int(S), int(D), lens, causal, float(scale), s);
    if (one != ZEN_ERR_NEEDS_WORKSPACE) return one == ZEN_OK;
    kernels = 2;
    const size_t bytes = zen_flash_attention_f32_workspace_bytes(int(B), int(H), int(S), int(D));
    at::Tensor ws = empty({int64_t(bytes)}, at::kByte, dev);
    return zen_flash_attention_f32(pq, pk, pv, po, int(B), int(H), int(S), int(D), lens, causal, float(scale), ws.data_ptr(), bytes, s) == ZEN_OK;
  });
  return !out || out == Py_None || kernels == 1 ? out : Py_BuildValue("Ni", out, kernels);
}

// No C++ exception leaves a function that Python calls.  Sizes and data pointers throw for tensors that have none of their
// own (inside vmap or forward-mode transforms, nested tensors): such a call is not served either.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t nargs) {
  try {
    return F(self, a, nargs);
  } catch (...) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

#define FN(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FN(gelu),        FN(relu),        FN(quantize),    FN(dequantize),  FN(layernorm),  FN(add_layernorm),
                         FN(linear_int8), FN(linear_fp16), FN(linear_fp32), FN(wmma_matmul), FN(matmul_f32), FN(flash_attention),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", "Native host path of zenith_b200.ops", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module_def); }
