// Host side of the per-token operators in native code: the contract checks, the
// allocation of results and workspaces, and the marshalling of one library call,
// which in Python cost more than the kernels of a small decode step take (the
// same checks and ctypes calls took 40-60 us per append or attention call).
//
// Every function here is the fast path of one Python function and only ever
// answers "done" or "not mine" (None): whatever it does not serve, malformed
// arguments among it, goes through the Python path, which raises the errors.  C++
// exceptions (no memory, a tensor without storage, a device that cannot be set) leave as
// the Python exceptions that torch's own functions raise for them, and every tensor whose
// address goes to the library is held until the call returns.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "../../include/winnow_tq.h"

namespace {

PyObject *g_backend_error = nullptr;         // winnow_b200._lib.BackendError
struct Names {
  PyObject *k_pages, *k_norms, *v_pages, *v_norms, *page_table, *seq_lens, *k_quant, *v_quant, *head_dim, *Pi,
      *centroids, *boundaries, *bit_width;
} N;

// A new reference that is dropped at the end of the scope.
struct Ref {
  PyObject *o;
  explicit Ref(PyObject *p) : o(p) {
    if (!o) PyErr_Clear();
  }
  Ref(const Ref &) = delete;
  ~Ref() { Py_XDECREF(o); }
  explicit operator bool() const { return o != nullptr; }
};

// The interpreter lock is given up while the library launches (a full launch queue blocks).
struct Unlocked {
  PyThreadState *s;
  Unlocked() : s(PyEval_SaveThread()) {}
  Unlocked(const Unlocked &) = delete;
  ~Unlocked() { PyEval_RestoreThread(s); }
};

bool tensor(PyObject *o, at::Tensor &t) {
  if (o == nullptr || !THPVariable_Check(o)) return false;
  t = THPVariable_Unpack(o);
  return t.defined() && t.layout() == at::kStrided;
}
bool tensor_attr(PyObject *owner, PyObject *name, at::Tensor &t) {
  Ref a(PyObject_GetAttr(owner, name));
  return a && tensor(a.o, t);
}
bool int_attr(PyObject *owner, PyObject *name, int64_t &v) {
  Ref a(PyObject_GetAttr(owner, name));
  if (!a || !PyLong_Check(a.o)) return false;
  v = PyLong_AsLongLong(a.o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? WTQ_F32 : t == at::kHalf ? WTQ_F16 : t == at::kBFloat16 ? WTQ_BF16 : -1;
}
bool width_ok(int64_t bw, int64_t D) {
  return (bw == 2 || bw == 3 || bw == 4 || bw == 5 || bw == 6 || bw == 8) && D * bw % 8 == 0;
}

// Pages and norms of one side: (P, Hkv, S, NB) uint8 with contiguous (S, NB) rows, (P, Hkv, S) fp16.
bool side_pages(const at::Tensor &pages, const at::Tensor &norms, int64_t bw, int64_t D, wtq_side_t &s) {
  if (pages.dim() != 4 || norms.dim() != 3 || pages.scalar_type() != at::kByte || norms.scalar_type() != at::kHalf)
    return false;
  const int64_t nb = D * bw / 8;
  if (!width_ok(bw, D) || pages.size(3) != nb || pages.stride(3) != 1 || pages.stride(2) != nb || norms.stride(2) != 1)
    return false;
  for (int i = 0; i < 3; ++i)
    if (norms.size(i) != pages.size(i)) return false;
  s.pages = (uint8_t *)pages.data_ptr();
  s.norms = norms.data_ptr();
  s.page_stride = pages.stride(0);
  s.head_stride = pages.stride(1);
  s.norm_page_stride = norms.stride(0);
  s.norm_head_stride = norms.stride(1);
  s.bw = (int)bw;
  return true;
}

// The rotation and one table of a quantizer (`table`: centroids or boundaries).
struct Quant {
  int64_t bw = 0;
  at::Tensor pi, tab;
};
bool quant_table(PyObject *quant, PyObject *table, int64_t D, int64_t extra, const at::Device &dev, Quant &held,
                 const float *&Pi, const float *&values) {
  int64_t &bw = held.bw;
  at::Tensor &pi = held.pi, &tab = held.tab;
  if (!int_attr(quant, N.bit_width, bw) || bw < 1 || bw > 8 || !tensor_attr(quant, N.Pi, pi) ||
      !tensor_attr(quant, table, tab))
    return false;
  if (pi.scalar_type() != at::kFloat || pi.dim() != 2 || pi.size(0) != D || pi.size(1) != D || !pi.is_contiguous() ||
      pi.device() != dev)
    return false;
  if (tab.scalar_type() != at::kFloat || tab.numel() != ((int64_t)1 << bw) - extra || !tab.is_contiguous() ||
      tab.device() != dev)
    return false;
  Pi = pi.const_data_ptr<float>();
  values = tab.const_data_ptr<float>();
  return true;
}

bool table_and_lengths(const at::Tensor &table, const at::Tensor &lens, int64_t B, const at::Device &dev) {
  return table.dim() == 2 && table.size(0) == B && table.scalar_type() == at::kInt && table.stride(1) == 1 &&
         lens.dim() == 1 && lens.size(0) == B && lens.scalar_type() == at::kInt && lens.is_contiguous() &&
         table.device() == dev && lens.device() == dev;
}

// One layer's paged packed K/V (a PackedKV) for queries of head_dim D on `dev`.
struct Layer {
  wtq_side_t k, v;
  at::Tensor kp, kn, vp, vn, table, lens;
  Quant k_quant, v_quant;
  int64_t P, Hkv, S;
};
bool read_layer(PyObject *kv, int64_t B, int64_t D, const at::Device &dev, Layer &l) {
  int64_t head_dim = 0;
  at::Tensor &kp = l.kp, &kn = l.kn, &vp = l.vp, &vn = l.vn;
  if (!int_attr(kv, N.head_dim, head_dim) || head_dim != D || D < 1 || D > 256) return false;
  if (!tensor_attr(kv, N.k_pages, kp) || !tensor_attr(kv, N.k_norms, kn) || !tensor_attr(kv, N.v_pages, vp) ||
      !tensor_attr(kv, N.v_norms, vn) || !tensor_attr(kv, N.page_table, l.table) || !tensor_attr(kv, N.seq_lens, l.lens))
    return false;
  if (kp.device() != dev || kn.device() != dev || vp.device() != dev || vn.device() != dev ||
      !table_and_lengths(l.table, l.lens, B, dev))
    return false;
  Ref kq(PyObject_GetAttr(kv, N.k_quant)), vq(PyObject_GetAttr(kv, N.v_quant));
  l.k.bounds = l.v.bounds = nullptr;
  if (!kq || !vq || !quant_table(kq.o, N.centroids, D, 0, dev, l.k_quant, l.k.Pi, l.k.centroids) ||
      !quant_table(vq.o, N.centroids, D, 0, dev, l.v_quant, l.v.Pi, l.v.centroids))
    return false;
  if (!side_pages(kp, kn, l.k_quant.bw, D, l.k) || !side_pages(vp, vn, l.v_quant.bw, D, l.v)) return false;
  for (int i = 0; i < 3; ++i)
    if (kp.size(i) != vp.size(i)) return false;
  l.P = kp.size(0);
  l.Hkv = kp.size(1);
  l.S = kp.size(2);
  return l.P >= 1 && l.Hkv >= 1 && l.S >= 1 && l.table.size(1) >= 1;
}

bool optional_status(PyObject *o, const at::Device &dev, at::Tensor &t, int32_t *&p) {
  p = nullptr;
  if (o == Py_None) return true;
  if (!tensor(o, t) || t.scalar_type() != at::kInt || t.numel() < 1 || t.device() != dev) return false;
  p = t.mutable_data_ptr<int32_t>();
  return true;
}

PyObject *library_error(int rc) {
  PyErr_Format(g_backend_error ? g_backend_error : PyExc_RuntimeError, "libwinnow_tq error %d: %s", rc, wtq_last_error());
  return nullptr;
}

// One decode call: q (B, Hq, 1, D).  `out` / `ws` / `status_arg` may be None; without `out` the result is a new
// tensor, (B, Hq, 1, D) or, with `token_major`, (B, 1, Hq, D).
PyObject *run_decode(PyObject *q_arg, PyObject *kv, PyObject *scale_arg, long splits, PyObject *out_arg, PyObject *ws_arg,
                     PyObject *status_arg, bool token_major) {
  at::Tensor q, out, ws, status_tensor;
  if (!tensor(q_arg, q) || !q.is_cuda() || q.dim() != 4 || q.size(2) != 1 || q.stride(3) != 1) Py_RETURN_NONE;
  const int dtype = dtype_code(q.scalar_type());
  const int64_t B = q.size(0), Hq = q.size(1), D = q.size(3);
  const at::Device dev = q.device();
  Layer l;
  int32_t *status;
  if (dtype < 0 || B < 1 || Hq < 1 || !read_layer(kv, B, D, dev, l) || Hq % l.Hkv ||
      !optional_status(status_arg, dev, status_tensor, status))
    Py_RETURN_NONE;
  const double scale = PyFloat_AsDouble(scale_arg);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (out_arg != Py_None) {
    if (!tensor(out_arg, out) || out.dim() != 4 || out.size(0) != B || out.size(1) != Hq || out.size(2) != 1 ||
        out.size(3) != D || out.stride(3) != 1 || out.scalar_type() != q.scalar_type() || out.device() != dev)
      Py_RETURN_NONE;
  }
  if (ws_arg != Py_None && (!tensor(ws_arg, ws) || ws.device() != dev)) Py_RETURN_NONE;
  const c10::cuda::OptionalCUDAGuard guard(dev);
  int64_t os[2] = {Hq * D, D};
  if (out.defined()) {
    os[0] = out.stride(0);
    os[1] = out.stride(1);
  } else {
    out = token_major ? at::empty({B, 1, Hq, D}, q.options()) : at::empty({B, Hq, 1, D}, q.options());
  }
  void *stream = (void *)at::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int64_t qs[2] = {q.stride(0), q.stride(1)};
  const int W = (int)l.table.size(1), S = (int)l.S, H = (int)l.Hkv;
  int rc = WTQ_ERR_UNSUPPORTED;
  if (splits <= 0 && !ws.defined()) {
    const Unlocked u;
    rc = wtq_decode_direct(q.const_data_ptr(), dtype, qs, out.mutable_data_ptr(), os, &l.k, &l.v,
                           l.table.const_data_ptr<int32_t>(), l.table.stride(0), l.lens.const_data_ptr<int32_t>(),
                           (float)scale, (int)B, (int)Hq, H, (int)D, S, (int)l.P, W, status, stream);
  }
  if (rc == WTQ_ERR_UNSUPPORTED) {
    if (!ws.defined()) {
      ws = at::empty({(int64_t)wtq_decode_workspace_bytes((int)B, (int)Hq, H, (int)D, W, S, (int)splits)},
                     q.options().dtype(at::kByte));
      ws.narrow(0, 0, (int64_t)wtq_decode_counter_bytes((int)B, H)).zero_();
    }
    const Unlocked u;
    rc = wtq_decode(q.const_data_ptr(), dtype, qs, out.mutable_data_ptr(), os, &l.k, &l.v,
                    l.table.const_data_ptr<int32_t>(), l.table.stride(0), l.lens.const_data_ptr<int32_t>(),
                    (float)scale, (int)B, (int)Hq, H, (int)D, S, (int)l.P, W, (int)splits, ws.mutable_data_ptr(),
                    (size_t)ws.numel(), status, stream);
  }
  if (rc) return library_error(rc);
  if (out_arg != Py_None) {
    Py_INCREF(out_arg);
    return out_arg;
  }
  return THPVariable_Wrap(std::move(out));
}

// decode(q, kv, scale, num_splits, out, workspace, status) -> out, or None
PyObject *decode(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 || !PyLong_Check(a[3])) Py_RETURN_NONE;
  const long splits = PyLong_AsLong(a[3]);
  if (splits == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  return run_decode(a[0], a[1], a[2], splits, a[4], a[5], a[6], false);
  END_HANDLE_TH_ERRORS
}

// attend(q, kv, scale, status) -> (B, 1, Hq, D), the layout attention interfaces hand back, or None
PyObject *attend(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4) Py_RETURN_NONE;
  return run_decode(a[0], a[1], a[2], 0, Py_None, Py_None, a[3], true);
  END_HANDLE_TH_ERRORS
}

// append(k, v, k_pages, k_norms, v_pages, v_norms, page_table, seq_lens, k_tq, v_tq, order, status) -> True, or None
PyObject *append(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  at::Tensor k, v, kp, kn, vp, vn, table, lens, status_tensor;
  Quant k_quant, v_quant;
  if (n != 12 || !tensor(a[0], k) || !tensor(a[1], v) || !tensor(a[2], kp) || !tensor(a[3], kn) || !tensor(a[4], vp) ||
      !tensor(a[5], vn) || !tensor(a[6], table) || !tensor(a[7], lens))
    Py_RETURN_NONE;
  const at::Device dev = k.device();
  if (!k.is_cuda() || k.dim() != 4 || v.dim() != 4 || k.sizes() != v.sizes() || k.scalar_type() != v.scalar_type() ||
      k.stride(3) != 1 || v.stride(3) != 1 || v.device() != dev)
    Py_RETURN_NONE;
  const int dtype = dtype_code(k.scalar_type());
  const int64_t B = k.size(0), Hkv = k.size(1), tokens = k.size(2), D = k.size(3);
  if (dtype < 0 || B < 1 || Hkv < 1 || tokens < 1 || D < 1 || D > 256) Py_RETURN_NONE;
  wtq_side_t sk, sv;
  int32_t *status;
  sk.centroids = sv.centroids = nullptr;
  if (kp.device() != dev || kn.device() != dev || vp.device() != dev || vn.device() != dev ||
      !table_and_lengths(table, lens, B, dev) || !quant_table(a[8], N.boundaries, D, 1, dev, k_quant, sk.Pi, sk.bounds) ||
      !quant_table(a[9], N.boundaries, D, 1, dev, v_quant, sv.Pi, sv.bounds) || !side_pages(kp, kn, k_quant.bw, D, sk) ||
      !side_pages(vp, vn, v_quant.bw, D, sv) || !optional_status(a[11], dev, status_tensor, status) || kp.size(1) != Hkv ||
      table.size(1) < 1)
    Py_RETURN_NONE;
  for (int i = 0; i < 3; ++i)
    if (kp.size(i) != vp.size(i)) Py_RETURN_NONE;
  const long order = PyLong_AsLong(a[10]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const c10::cuda::OptionalCUDAGuard guard(dev);
  const int64_t ks[3] = {k.stride(0), k.stride(1), k.stride(2)}, vs[3] = {v.stride(0), v.stride(1), v.stride(2)};
  void *stream = (void *)at::cuda::getCurrentCUDAStream(dev.index()).stream();
  int rc;
  {
    const Unlocked u;
    rc = wtq_append(k.const_data_ptr(), v.const_data_ptr(), dtype, ks, vs, &sk, &sv, table.const_data_ptr<int32_t>(),
                    table.stride(0), lens.const_data_ptr<int32_t>(), (int)B, (int)Hkv, (int)tokens, (int)D,
                    (int)kp.size(2), (int)kp.size(0), (int)table.size(1), (int)order, status, stream);
  }
  if (rc) return library_error(rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// stage(dst, src, dst, src, dst, src) -> True, or None: copies of contiguous tensors of equal type and size
// (a pair of None: nothing to copy)
PyObject *stage(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  at::Tensor held[3][2];
  void *dst[3] = {};
  const void *src[3] = {};
  int64_t bytes[3] = {};
  at::Device dev(at::kCPU);
  if (n != 6) Py_RETURN_NONE;
  for (int i = 0; i < 3; ++i) {
    if (a[2 * i + 1] == Py_None) continue;
    at::Tensor &d = held[i][0], &s = held[i][1];
    if (!tensor(a[2 * i], d) || !tensor(a[2 * i + 1], s) || !d.is_cuda() || s.device() != d.device() ||
        d.scalar_type() != s.scalar_type() || d.sizes() != s.sizes() || !d.is_contiguous() || !s.is_contiguous() ||
        (dev.is_cuda() && dev != d.device()))
      Py_RETURN_NONE;
    dev = d.device();
    dst[i] = d.mutable_data_ptr();
    src[i] = s.const_data_ptr();
    bytes[i] = (int64_t)d.nbytes();
    if ((((uintptr_t)dst[i] | (uintptr_t)src[i]) & 15) != 0) Py_RETURN_NONE;
  }
  if (!dev.is_cuda()) Py_RETURN_TRUE;
  const c10::cuda::OptionalCUDAGuard guard(dev);
  void *stream = (void *)at::cuda::getCurrentCUDAStream(dev.index()).stream();
  int rc;
  {
    const Unlocked u;
    rc = wtq_stage(dst, src, bytes, stream);
  }
  if (rc) return library_error(rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyObject *set_error(PyObject *, PyObject *type) {
  Py_INCREF(type);
  Py_XSETREF(g_backend_error, type);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"decode", (PyCFunction)(void (*)(void))decode, METH_FASTCALL, "decode(q, kv, scale, num_splits, out, workspace, status)"},
    {"attend", (PyCFunction)(void (*)(void))attend, METH_FASTCALL, "attend(q, kv, scale, status)"},
    {"append", (PyCFunction)(void (*)(void))append, METH_FASTCALL,
     "append(k, v, k_pages, k_norms, v_pages, v_norms, page_table, seq_lens, k_tq, v_tq, order, status)"},
    {"stage", (PyCFunction)(void (*)(void))stage, METH_FASTCALL, "stage(dst, src, dst, src, dst, src)"},
    {"set_error", set_error, METH_O, "the exception type library errors are raised as"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host side of winnow_b200", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  N.k_pages = PyUnicode_InternFromString("k_pages");
  N.k_norms = PyUnicode_InternFromString("k_norms");
  N.v_pages = PyUnicode_InternFromString("v_pages");
  N.v_norms = PyUnicode_InternFromString("v_norms");
  N.page_table = PyUnicode_InternFromString("page_table");
  N.seq_lens = PyUnicode_InternFromString("seq_lens");
  N.k_quant = PyUnicode_InternFromString("k_quant");
  N.v_quant = PyUnicode_InternFromString("v_quant");
  N.head_dim = PyUnicode_InternFromString("head_dim");
  N.Pi = PyUnicode_InternFromString("Pi");
  N.centroids = PyUnicode_InternFromString("centroids");
  N.boundaries = PyUnicode_InternFromString("boundaries");
  N.bit_width = PyUnicode_InternFromString("bit_width");
  return PyModule_Create(&module);
}
