// The Python package's calls, from tensors to the C ABI, in native code.
//
// A decode step is a dozen launches of a few microseconds and the attention calls of an image model are not much
// longer: reading shapes and strides through Python objects, packing a descriptor and converting a dozen arguments
// for ctypes costs 6 to 12 us a call, more than such a kernel runs.  Each function here does for well-formed
// arguments exactly what its Python twin in __init__.py does.  Whatever it does not recognise at once (another type
// than a plain CUDA tensor, shapes or strides that the twin would refuse, scratch that has to be allocated) it
// answers with None and leaves to the twin, which also words the errors.  Nothing is kept from one call to the next.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/DispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "ixk.h"

namespace {

decltype(&ixk_gemm) g_gemm;
decltype(&ixk_gemm_fp8) g_gemm_fp8;
decltype(&ixk_gemm_workspace_bytes) g_gemm_bytes;
decltype(&ixk_gemm_geglu) g_geglu;
decltype(&ixk_fmha_fwd) g_fwd;
decltype(&ixk_fmha_fwd_workspace_bytes) g_fwd_bytes;
decltype(&ixk_fmha_bwd) g_bwd;
decltype(&ixk_fmha_bwd_workspace_bytes) g_bwd_bytes;
decltype(&ixk_row_norm) g_row_norm;
decltype(&ixk_row_norm_gain) g_row_norm_gain;
decltype(&ixk_rotary_interleaved) g_rotary, g_rotary_half;
decltype(&ixk_kv_append) g_kv_append;
decltype(&ixk_residual_add) g_residual_add;

// A plain CUDA tensor, nullptr for anything else (None included; see `optional`).
const at::Tensor* tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  constexpr c10::DispatchKeySet special({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                         c10::DispatchKey::Functionalize, c10::DispatchKey::Python, c10::DispatchKey::Conjugate,
                                         c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  if (!t.defined() || !t.is_cuda() || t.layout() != c10::kStrided || t.key_set().has_any(special) ||
      t.unsafeGetTensorImpl()->has_symbolic_sizes_strides())
    return nullptr;
  return &t;
}
// An argument that may be None: false if it is neither None nor a plain CUDA tensor.
bool optional(PyObject* o, const at::Tensor** t) {
  *t = nullptr;
  return o == Py_None || (*t = tensor(o)) != nullptr;
}
void* ptr(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }
size_t size_of(const at::Tensor* t) { return t == nullptr ? 0 : t->nbytes(); }

int dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kBFloat16: return IXK_BF16;
    case at::kHalf: return IXK_F16;
    case at::kFloat: return IXK_F32;
    case at::kFloat8_e4m3fn: return IXK_F8E4M3;
    case at::kFloat8_e5m2: return IXK_F8E5M2;
    case at::kChar: return IXK_S8;
    case at::kInt: return IXK_S32;
    default: return -1;
  }
}

// A stream object, or None for torch's current stream on the current device.
bool stream_arg(PyObject* o, void** s) {
  if (o == Py_None) {
    *s = c10::cuda::getCurrentCUDAStream().stream();
    return true;
  }
  PyObject* handle = PyObject_GetAttrString(o, "cuda_stream");
  *s = handle != nullptr ? PyLong_AsVoidPtr(handle) : nullptr;
  Py_XDECREF(handle);
  if (PyErr_Occurred() == nullptr) return true;
  PyErr_Clear();
  return false;
}
bool number(PyObject* o, double* v) {
  if (PyFloat_CheckExact(o)) *v = PyFloat_AS_DOUBLE(o);
  else if (PyLong_CheckExact(o)) *v = PyLong_AsDouble(o);
  else return false;
  if (PyErr_Occurred() == nullptr) return true;
  PyErr_Clear();
  return false;
}
bool integer(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsLongLong(o);
  if (PyErr_Occurred() == nullptr) return true;
  PyErr_Clear();
  return false;
}

template <typename Call>
int unlocked(const Call& call) {   // the library's calls run without the interpreter's lock, as under ctypes
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = call();
  Py_END_ALLOW_THREADS
  return st;
}
PyObject* status(int st) { return PyLong_FromLong(st); }
// The result tensor, or the status where it is not OK.
PyObject* result(int st, PyObject* given, const at::Tensor& made) {
  if (st != IXK_OK) return status(st);
  if (given == Py_None) return THPVariable_Wrap(made);
  Py_INCREF(given);
  return given;
}

// _matrix_layout: whichever of the last two dimensions has stride 1 decides the order.
bool layout(const at::Tensor& t, ixk_matrix_layout* l) {
  const int64_t d = t.dim();
  if (d != 2 && d != 3) return false;
  const int64_t rows = t.size(d - 2), cols = t.size(d - 1), sr = t.stride(d - 2), sc = t.stride(d - 1);
  if (sc == 1 && (sr >= cols || rows == 1)) {
    l->order = IXK_ROW_MAJOR;
    l->leading_dim_stride = rows > 1 ? sr : std::max(sr, cols);
  } else if (sr == 1 && (sc >= rows || cols == 1)) {
    l->order = IXK_COL_MAJOR;
    l->leading_dim_stride = cols > 1 ? sc : std::max(sc, rows);
  } else {
    return false;
  }
  l->dtype = dtype_of(t);
  l->num_rows = rows;
  l->num_cols = cols;
  l->batch_stride = d == 3 ? t.stride(0) : rows * cols;
  return l->dtype >= 0;
}

// _require_c: C lies in memory as the result does, dimensions of one entry aside.
bool lies_alike(const at::Tensor& c, const at::Tensor& out) {
  if (c.scalar_type() != out.scalar_type() || c.numel() != out.numel()) return false;
  int64_t i = 0, j = 0;
  for (;; ++i, ++j) {
    while (i < c.dim() && c.size(i) == 1) ++i;
    while (j < out.dim() && out.size(j) == 1) ++j;
    if (i == c.dim() || j == out.dim()) break;
    if (c.size(i) != out.size(j) || c.stride(i) != out.stride(j)) break;
  }
  if (i == c.dim() && j == out.dim()) return true;
  return c.is_contiguous() && out.is_contiguous() && (c.dim() < 2 || c.size(c.dim() - 1) == out.size(out.dim() - 1));
}

#define IXK_PY_FUNCTION(name, count)                             \
  PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n) {  \
    HANDLE_TH_ERRORS                                             \
    if (n != (count)) Py_RETURN_NONE;
#define IXK_PY_END     \
  END_HANDLE_TH_ERRORS \
  }

// lhs, rhs, bias, c, out, out dtype, alpha, beta, epilogue, workspace, stream, inv_scale_a, inv_scale_b
IXK_PY_FUNCTION(py_gemm, 13)
  const at::Tensor *lhs = tensor(a[0]), *rhs = tensor(a[1]), *bias, *c, *out, *ws;
  double alpha, beta;
  int64_t epilogue;
  void* stream;
  if (lhs == nullptr || rhs == nullptr || !optional(a[2], &bias) || !optional(a[3], &c) || !optional(a[4], &out) ||
      !number(a[6], &alpha) || !number(a[7], &beta) || !integer(a[8], &epilogue) || !optional(a[9], &ws) || !stream_arg(a[10], &stream))
    Py_RETURN_NONE;
  double sa = 1.0, sb = 1.0;
  const bool fp8 = a[11] != Py_None || a[12] != Py_None;
  if (fp8 && (!number(a[11], &sa) || !number(a[12], &sb) || (out == nullptr && a[5] == Py_None))) Py_RETURN_NONE;
  ixk_gemm_desc d{};
  if (!layout(*lhs, &d.lhs) || !layout(*rhs, &d.rhs)) Py_RETURN_NONE;
  at::Tensor made;
  if (out == nullptr) {
    at::ScalarType type = lhs->scalar_type();
    if (a[5] != Py_None) {
      if (!THPDtype_Check(a[5])) Py_RETURN_NONE;
      type = reinterpret_cast<THPDtype*>(a[5])->scalar_type;
    }
    c10::SmallVector<int64_t, 3> shape(lhs->sizes().begin(), lhs->sizes().end());
    shape.back() = rhs->size(rhs->dim() - 1);
    made = at::empty(shape, at::TensorOptions().device(lhs->device()).dtype(type));
    out = &made;
  }
  if (!layout(*out, &d.output)) Py_RETURN_NONE;
  d.batch_size = out->dim() == 3 ? out->size(0) : 1;
  d.alpha = static_cast<float>(alpha);
  d.beta = static_cast<float>(beta);
  d.epilogue = static_cast<int32_t>(epilogue);
  if (c != nullptr && d.beta != 0.0f && !lies_alike(*c, *out)) Py_RETURN_NONE;
  // An fp8 call that makes its own result takes the scratch it can use as well, from the pool of the stream it was given
  // (where that is not the current one the twin does).
  at::Tensor own;
  if (fp8 && ws == nullptr && a[4] == Py_None) {
    if (const size_t need = g_gemm_bytes(&d)) {
      if (a[10] != Py_None) Py_RETURN_NONE;
      try {
        own = at::empty({static_cast<int64_t>(need)}, at::TensorOptions().device(lhs->device()).dtype(at::kByte));
        ws = &own;
      } catch (const c10::OutOfMemoryError&) {   // it runs without
      }
    }
  }
  const size_t bytes = size_of(ws);
  void *pa = ptr(lhs), *pb = ptr(rhs), *pc = ptr(c), *pbias = ptr(bias), *pd = ptr(out), *pw = ptr(ws);
  const int st = unlocked([&] {
    return fp8 ? g_gemm_fp8(&d, pa, pb, pc, pbias, pd, static_cast<float>(sa), static_cast<float>(sb), pw, bytes, stream)
               : g_gemm(&d, pa, pb, pc, pbias, pd, pw, bytes, stream);
  });
  return result(st, a[4], made);
IXK_PY_END

// x, w_gate_up, out, workspace, stream
IXK_PY_FUNCTION(py_geglu, 5)
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]), *out, *ws = tensor(a[3]);
  void* stream;
  if (x == nullptr || w == nullptr || !optional(a[2], &out) || ws == nullptr || !stream_arg(a[4], &stream)) Py_RETURN_NONE;
  ixk_gemm_desc d{};
  if (!layout(*x, &d.lhs) || !layout(*w, &d.rhs)) Py_RETURN_NONE;
  const int64_t m = x->size(x->dim() - 2), n2 = w->size(w->dim() - 1);
  at::Tensor made;
  if (out == nullptr) {
    made = at::empty({m, n2 / 2}, at::TensorOptions().device(x->device()).dtype(x->scalar_type()));
    out = &made;
  } else if (out->dim() < 2) {
    Py_RETURN_NONE;
  }
  d.output = ixk_matrix_layout{IXK_ROW_MAJOR, d.lhs.dtype, m, n2, m * n2, n2};
  d.batch_size = 1;
  d.alpha = 1.0f;
  void *px = ptr(x), *pw = ptr(w), *po = ptr(out), *scratch = ptr(ws);
  const int64_t ld = out->stride(out->dim() - 2);
  const size_t bytes = ws->nbytes();
  const int st = unlocked([&] { return g_geglu(&d, px, pw, po, ld, scratch, bytes, stream); });
  return result(st, a[2], made);
IXK_PY_END

// _fmha_desc
bool fmha_desc(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor* bias, const at::Tensor& out, double scale,
               bool causal, ixk_fmha_desc* d) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || out.dim() != 4) return false;
  const int64_t B = q.size(0), N = q.size(1), F = q.size(2), H = q.size(3), T = k.size(2);
  if (k.size(0) != B || k.size(1) != N || k.size(3) != H || v.sizes() != k.sizes() || out.sizes() != q.sizes()) return false;
  if (B > INT32_MAX || N > INT32_MAX || F > INT32_MAX || T > INT32_MAX || H > INT32_MAX) return false;
  const at::ScalarType type = q.scalar_type();
  if (k.scalar_type() != type || v.scalar_type() != type || out.scalar_type() != type) return false;
  if (H > 1 && (q.stride(3) != 1 || k.stride(3) != 1 || v.stride(3) != 1 || out.stride(3) != 1)) return false;
  *d = ixk_fmha_desc{};
  if (bias != nullptr) {
    if (bias->scalar_type() != type || bias->dim() != 4 || bias->size(3) != T || bias->size(2) != F || bias->stride(3) != 1) return false;
    d->bias_strides[0] = bias->size(0) > 1 ? bias->stride(0) : 0;
    d->bias_strides[1] = bias->size(1) > 1 ? bias->stride(1) : 0;
    d->bias_strides[2] = bias->stride(2);
  }
  d->dtype = dtype_of(q);
  if (d->dtype < 0) return false;
  d->causal = causal ? 1 : 0;
  d->num_batches = static_cast<int32_t>(B);
  d->num_heads = static_cast<int32_t>(N);
  d->head_size = static_cast<int32_t>(H);
  d->num_queries = static_cast<int32_t>(F);
  d->num_keys = static_cast<int32_t>(T);
  d->head_scale = static_cast<float>(scale);
  for (int i = 0; i < 3; ++i) {
    d->q_strides[i] = q.stride(i);
    d->k_strides[i] = k.stride(i);
    d->v_strides[i] = v.stride(i);
    d->o_strides[i] = out.stride(i);
  }
  return true;
}

// q, k, v, bias, out, log-sum-exp rows, scale, causal, workspace, stream
IXK_PY_FUNCTION(py_fmha_forward, 10)
  const at::Tensor *q = tensor(a[0]), *k = tensor(a[1]), *v = tensor(a[2]), *bias, *out = tensor(a[4]), *lse, *ws;
  double scale;
  void* stream;
  ixk_fmha_desc d;
  if (q == nullptr || k == nullptr || v == nullptr || !optional(a[3], &bias) || out == nullptr || !optional(a[5], &lse) ||
      !number(a[6], &scale) || !PyBool_Check(a[7]) || !optional(a[8], &ws) || !stream_arg(a[9], &stream) ||
      !fmha_desc(*q, *k, *v, bias, *out, scale, a[7] == Py_True, &d))
    Py_RETURN_NONE;
  const size_t bytes = size_of(ws);
  if (g_fwd_bytes(&d) > bytes) Py_RETURN_NONE;   // (the twin allocates)
  void *pq = ptr(q), *pk = ptr(k), *pv = ptr(v), *pb = ptr(bias), *po = ptr(out), *pl = ptr(lse), *pw = ptr(ws);
  return status(unlocked([&] { return g_fwd(&d, pq, pk, pv, pb, po, static_cast<float*>(pl), pw, bytes, stream); }));
IXK_PY_END

// q, k, v, out, bias, grad_out, log-sum-exp rows, dq, dk, dv, scale, causal, workspace, stream
IXK_PY_FUNCTION(py_fmha_backward, 14)
  const at::Tensor *q = tensor(a[0]), *k = tensor(a[1]), *v = tensor(a[2]), *out = tensor(a[3]), *bias, *go = tensor(a[5]),
                   *lse = tensor(a[6]), *dq = tensor(a[7]), *dk = tensor(a[8]), *dv = tensor(a[9]), *ws = tensor(a[12]);
  double scale;
  void* stream;
  ixk_fmha_bwd_desc d{};
  if (q == nullptr || k == nullptr || v == nullptr || out == nullptr || !optional(a[4], &bias) || go == nullptr || lse == nullptr ||
      dq == nullptr || dk == nullptr || dv == nullptr || !number(a[10], &scale) || !PyBool_Check(a[11]) || ws == nullptr ||
      !stream_arg(a[13], &stream) || !fmha_desc(*q, *k, *v, bias, *out, scale, a[11] == Py_True, &d.fwd))
    Py_RETURN_NONE;
  if (lse->scalar_type() != at::kFloat || !lse->is_contiguous() || lse->dim() != 3 || lse->sizes() != q->sizes().slice(0, 3)) Py_RETURN_NONE;
  const at::Tensor* grads[4] = {go, dq, dk, dv};
  const at::Tensor* like[4] = {q, q, k, v};
  int64_t* strides[4] = {d.do_strides, d.dq_strides, d.dk_strides, d.dv_strides};
  for (int i = 0; i < 4; ++i) {
    const at::Tensor& t = *grads[i];
    if (t.sizes() != like[i]->sizes() || t.scalar_type() != like[i]->scalar_type() || (t.stride(3) != 1 && t.size(3) > 1)) Py_RETURN_NONE;
    for (int j = 0; j < 3; ++j) strides[i][j] = t.stride(j);
  }
  const size_t bytes = ws->nbytes();
  if (g_bwd_bytes(&d) > bytes) Py_RETURN_NONE;
  void *pq = ptr(q), *pk = ptr(k), *pv = ptr(v), *po = ptr(out), *pb = ptr(bias), *pg = ptr(go), *pl = ptr(lse), *pdq = ptr(dq),
       *pdk = ptr(dk), *pdv = ptr(dv), *pw = ptr(ws);
  return status(unlocked([&] {
    return g_bwd(&d, pq, pk, pv, po, pb, pg, static_cast<const float*>(pl), pdq, pdk, pdv, pw, bytes, stream);
  }));
IXK_PY_END

// x, kind, eps, out, gain, gain_offset, stream
IXK_PY_FUNCTION(py_row_norm, 7)
  const at::Tensor *x = tensor(a[0]), *out, *gain;
  int64_t kind;
  double eps, offset;
  void* stream;
  if (x == nullptr || !integer(a[1], &kind) || !number(a[2], &eps) || !optional(a[3], &out) || !optional(a[4], &gain) ||
      !number(a[5], &offset) || !stream_arg(a[6], &stream) || x->dim() < 1 || !x->is_contiguous() || dtype_of(*x) < 0)
    Py_RETURN_NONE;
  const int64_t cols = x->size(x->dim() - 1), rows = cols != 0 ? x->numel() / cols : 0;
  if (gain != nullptr && (gain->dim() != 1 || gain->size(0) != cols || gain->scalar_type() != x->scalar_type() || !gain->is_contiguous()))
    Py_RETURN_NONE;
  at::Tensor made;
  if (out == nullptr) {
    made = at::empty(x->sizes(), at::TensorOptions().device(x->device()).dtype(x->scalar_type()));
    out = &made;
  } else if (out->sizes() != x->sizes() || out->scalar_type() != x->scalar_type() || !out->is_contiguous()) {
    Py_RETURN_NONE;
  }
  void *px = ptr(x), *pg = ptr(gain), *po = ptr(out);
  const int type = dtype_of(*x), k = static_cast<int>(kind);
  const float e = static_cast<float>(eps), off = static_cast<float>(offset);
  const int st = unlocked([&] {
    return gain != nullptr ? g_row_norm_gain(type, k, rows, cols, px, cols, pg, off, po, cols, e, stream)
                           : g_row_norm(type, k, rows, cols, px, cols, po, cols, e, stream);
  });
  return result(st, a[3], made);
IXK_PY_END

// x, cos, sin, seq_len, rotary_dim, half_split, stream
IXK_PY_FUNCTION(py_rotary, 7)
  const at::Tensor *x = tensor(a[0]), *cos = tensor(a[1]), *sin = tensor(a[2]);
  int64_t seq_len, dim;
  void* stream;
  if (x == nullptr || cos == nullptr || sin == nullptr || !integer(a[3], &seq_len) || !integer(a[4], &dim) || !PyBool_Check(a[5]) ||
      !stream_arg(a[6], &stream) || x->dim() != 3 || x->stride(2) != 1 || cos->scalar_type() != at::kFloat ||
      sin->scalar_type() != at::kFloat || !cos->is_contiguous() || !sin->is_contiguous() || cos->dim() != 2 ||
      cos->size(0) != seq_len || cos->size(1) != dim / 2 || sin->sizes() != cos->sizes() || dim > x->size(2) || dim < 0 || dtype_of(*x) < 0)
    Py_RETURN_NONE;
  void *px = ptr(x), *pc = ptr(cos), *ps = ptr(sin);
  const auto fn = a[5] == Py_True ? g_rotary_half : g_rotary;
  const int type = dtype_of(*x);
  const int64_t tokens = x->size(0), heads = x->size(1), s0 = x->stride(0), s1 = x->stride(1);
  return status(unlocked([&] {
    return fn(type, px, tokens, seq_len, heads, dim, s0, s1, static_cast<const float*>(pc), static_cast<const float*>(ps), stream);
  }));
IXK_PY_END

// k_cache, v_cache, k_new, v_new, position, stream
IXK_PY_FUNCTION(py_kv_append, 6)
  const at::Tensor *kc = tensor(a[0]), *vc = tensor(a[1]), *kn = tensor(a[2]), *vn = tensor(a[3]);
  int64_t position;
  void* stream;
  if (kc == nullptr || vc == nullptr || kn == nullptr || vn == nullptr || !integer(a[4], &position) || !stream_arg(a[5], &stream) ||
      kc->dim() != 4 || kn->dim() != 3 || dtype_of(*kc) < 0)
    Py_RETURN_NONE;
  const int64_t B = kc->size(0), T = kc->size(1), N = kc->size(2), H = kc->size(3);
  if (vc->sizes() != kc->sizes() || vc->strides() != kc->strides() || kn->size(0) != B || kn->size(1) != N || kn->size(2) != H ||
      vn->sizes() != kn->sizes() || vn->strides() != kn->strides() || kc->stride(3) != 1 || kn->stride(2) != 1 || position < 0 || position >= T)
    Py_RETURN_NONE;
  void *pkn = ptr(kn), *pvn = ptr(vn), *pkc = ptr(kc), *pvc = ptr(vc);
  const int type = dtype_of(*kc);
  const int64_t n0 = kn->stride(0), n1 = kn->stride(1), c0 = kc->stride(0), c1 = kc->stride(1), c2 = kc->stride(2);
  return status(unlocked([&] { return g_kv_append(type, B, N, H, pkn, pvn, n0, n1, pkc, pvc, c0, c1, c2, position, stream); }));
IXK_PY_END

// x, partial, bias, out, stream
IXK_PY_FUNCTION(py_residual_add, 5)
  const at::Tensor *x = tensor(a[0]), *p = tensor(a[1]), *bias, *out;
  void* stream;
  if (x == nullptr || p == nullptr || !optional(a[2], &bias) || !optional(a[3], &out) || !stream_arg(a[4], &stream) || x->dim() < 1 ||
      !x->is_contiguous() || !p->is_contiguous() || p->numel() != x->numel() || p->scalar_type() != x->scalar_type() || dtype_of(*x) < 0)
    Py_RETURN_NONE;
  const int64_t cols = x->size(x->dim() - 1), rows = cols != 0 ? x->numel() / cols : 0;
  if (bias != nullptr && (bias->dim() != 1 || bias->size(0) != cols || bias->scalar_type() != x->scalar_type() || !bias->is_contiguous()))
    Py_RETURN_NONE;
  at::Tensor made;
  if (out == nullptr) {
    made = at::empty(x->sizes(), at::TensorOptions().device(x->device()).dtype(x->scalar_type()));
    out = &made;
  } else if (out->numel() != x->numel() || out->scalar_type() != x->scalar_type() || !out->is_contiguous()) {
    Py_RETURN_NONE;
  }
  void *px = ptr(x), *pp = ptr(p), *pb = ptr(bias), *po = ptr(out);
  const int type = dtype_of(*x);
  const int st = unlocked([&] { return g_residual_add(type, rows, cols, px, pp, pb, po, stream); });
  return result(st, a[3], made);
IXK_PY_END

// bind(name -> address): the entry points of the library that the package has loaded
PyObject* py_bind(PyObject*, PyObject* table) {
  struct Entry {
    const char* name;
    void** slot;
  };
  const Entry entries[] = {
      {"ixk_gemm", reinterpret_cast<void**>(&g_gemm)},
      {"ixk_gemm_fp8", reinterpret_cast<void**>(&g_gemm_fp8)},
      {"ixk_gemm_workspace_bytes", reinterpret_cast<void**>(&g_gemm_bytes)},
      {"ixk_gemm_geglu", reinterpret_cast<void**>(&g_geglu)},
      {"ixk_fmha_fwd", reinterpret_cast<void**>(&g_fwd)},
      {"ixk_fmha_fwd_workspace_bytes", reinterpret_cast<void**>(&g_fwd_bytes)},
      {"ixk_fmha_bwd", reinterpret_cast<void**>(&g_bwd)},
      {"ixk_fmha_bwd_workspace_bytes", reinterpret_cast<void**>(&g_bwd_bytes)},
      {"ixk_row_norm", reinterpret_cast<void**>(&g_row_norm)},
      {"ixk_row_norm_gain", reinterpret_cast<void**>(&g_row_norm_gain)},
      {"ixk_rotary_interleaved", reinterpret_cast<void**>(&g_rotary)},
      {"ixk_rotary_half", reinterpret_cast<void**>(&g_rotary_half)},
      {"ixk_kv_append", reinterpret_cast<void**>(&g_kv_append)},
      {"ixk_residual_add", reinterpret_cast<void**>(&g_residual_add)},
  };
  for (const Entry& e : entries) {
    PyObject* address = PyDict_GetItemString(table, e.name);   // borrowed
    if (address == nullptr) {
      PyErr_SetString(PyExc_KeyError, e.name);
      return nullptr;
    }
    *e.slot = PyLong_AsVoidPtr(address);
    if (PyErr_Occurred() != nullptr) return nullptr;
  }
  Py_RETURN_NONE;
}

#define IXK_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", py_bind, METH_O, nullptr},
    IXK_METHOD("gemm", py_gemm),
    IXK_METHOD("geglu", py_geglu),
    IXK_METHOD("fmha_forward", py_fmha_forward),
    IXK_METHOD("fmha_backward", py_fmha_backward),
    IXK_METHOD("row_norm", py_row_norm),
    IXK_METHOD("rotary", py_rotary),
    IXK_METHOD("kv_append", py_kv_append),
    IXK_METHOD("residual_add", py_residual_add),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ixk_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ixk_calls() { return PyModule_Create(&module); }
