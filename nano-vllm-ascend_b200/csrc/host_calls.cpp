// host_calls.cpp -- the attention entry points of ops.py as one native call each.
//
// A decode call of one row takes 6.4 us on the device (in a graph) and took 17 us of Python: 25 arguments through ctypes (3.6 us), some 35
// tensor attributes (4 us); 6.4 us now, all in all (7.7 with the workspace looked up that its one launch does not take). Captured steps
// never paid it. Here the same attributes are looked at
// and the same library function is called without either. What ops.py would refuse is not judged here: the functions return None for
// any argument that is not exactly what they expect, and ops.py goes its own way, checks and errors included. An int is the library's
// status. Plain torch.Tensor with memory of its own only (subclasses, fake tensors, dispatch modes and what torch.vmap and torch.func
// wrap take ops.py's way); nothing is kept between calls.
// The interpreter lock is given up around the library's function alone: everything that can throw, addresses of tensors included,
// is read before, since an exception that left the block would be handled without the lock.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>

#include "../../include/b200attn.h"

namespace {

decltype(&b200_paged_decode_attn_windowed) g_decode = nullptr;
decltype(&b200_paged_decode_attn_fp8) g_decode_fp8 = nullptr;
decltype(&b200_prefill_varlen_attn_windowed) g_prefill = nullptr;
decltype(&b200_paged_decode_attn_few) g_decode_few = nullptr;
decltype(&b200_paged_decode_attn_fp8_few) g_decode_fp8_few = nullptr;

// a plain CUDA tensor with memory, or nullptr (the wrappers of torch.vmap, grad and jvp are torch.Tensor to Python, and have none)
const at::Tensor* cuda_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && !t.is_neg() && !t.is_conj() && t.has_storage() ? &t : nullptr;
}
int element(const at::Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? B200_DTYPE_BF16 : t.scalar_type() == at::kHalf ? B200_DTYPE_F16 : -1;
}
bool is_int(const at::Tensor& t) { return t.scalar_type() == at::kInt; }
bool heads_fit(const at::Tensor& t, int64_t width) { return t.dim() == 3 && t.stride(2) == 1 && t.stride(1) == width; }
// [blocks, block size, row] or [blocks, block size, heads, width], contiguous, with rows of `row` elements
bool cache_fits(const at::Tensor& t, int64_t row) {
  return (t.dim() == 3 || t.dim() == 4) && t.is_contiguous() && t.size(0) > 0 && t.size(1) > 0 &&
         t.size(2) * (t.dim() == 4 ? t.size(3) : 1) == row;
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
// ints that fit 64 bits (what int() would make of a float, and what ctypes would refuse, is ops.py's business)
bool ints(PyObject* const* a, int n) {
  for (int i = 0; i < n; ++i) {
    int over = 0;
    if (!PyLong_CheckExact(a[i])) return false;
    PyLong_AsLongLongAndOverflow(a[i], &over);
    if (over != 0) return false;
  }
  return true;
}
bool reals(PyObject* const* a, int n) {
  for (int i = 0; i < n; ++i)
    if (!PyFloat_CheckExact(a[i]) && !ints(a + i, 1)) return false;
  return true;
}
int64_t whole(PyObject* o) { return PyLong_AsLongLong(o); }
float real(PyObject* o) { return (float)(PyFloat_CheckExact(o) ? PyFloat_AS_DOUBLE(o) : PyLong_AsDouble(o)); }

PyObject* status(int rc, at::Tensor out) { return rc == B200_OK ? THPVariable_Wrap(std::move(out)) : PyLong_FromLong(rc); }

// decode(workspace of ops.py, q, k_cache, v_cache, block_tables, context_lens, scale, num_kv_heads, num_ctas, softcap, window, keep_first,
// chunk); decode_fp8 (.., num_ctas, k_scale, v_scale)
template <bool FP8>
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != (FP8 ? 11 : 13) || !reals(a + 6, 1) || !ints(a + 7, 2) || !reals(a + 9, FP8 ? 2 : 1) || (!FP8 && !ints(a + 10, 3)) ||
      c10::impl::TorchDispatchModeTLS::any_modes_set())
    Py_RETURN_NONE;
  const at::Tensor *q = cuda_tensor(a[1]), *k = cuda_tensor(a[2]), *v = cuda_tensor(a[3]), *bt = cuda_tensor(a[4]), *lens = cuda_tensor(a[5]);
  if (!q || !k || !v || !bt || !lens || element(*q) < 0 || q->dim() != 3) Py_RETURN_NONE;
  const int64_t B = q->size(0), H = q->size(1), D = q->size(2), kv = whole(a[7]), ctas = whole(a[8]);
  if (!heads_fit(*q, D) || !is_int(*bt) || !is_int(*lens) || bt->dim() != 2 || bt->stride(1) != 1 || !lens->is_contiguous()) Py_RETURN_NONE;
  if (!cache_fits(*k, kv * D)) Py_RETURN_NONE;
  if (FP8) {
    for (const at::Tensor* c : {k, v})
      if (c->scalar_type() != at::kByte && c->scalar_type() != at::kFloat8_e4m3fn) Py_RETURN_NONE;
  }
  at::Tensor out = at::empty({B, H * D}, q->options());
  const int64_t qs = B > 1 ? q->stride(0) : H * D;
  const float scale = real(a[6]), f9 = real(a[9]), f10 = FP8 ? real(a[10]) : 0.f;
  const int32_t window = FP8 ? 0 : (int32_t)whole(a[10]), keep_first = FP8 ? 0 : (int32_t)whole(a[11]), chunk = FP8 ? 0 : (int32_t)whole(a[12]);
  void *const to = out.data_ptr(), *const qp = q->data_ptr(), *const kp = k->data_ptr(), *const vp = v->data_ptr();
  const int32_t *const tables = (const int32_t*)bt->data_ptr(), *const rows = (const int32_t*)lens->data_ptr();
  const int32_t nb = (int32_t)k->size(0), bs = (int32_t)k->size(1), bt_stride = (int32_t)bt->stride(0);
  const int type = element(*q);
  void* const on = stream();
  int rc = B200_ERR_UNSUPPORTED;
  if (B > 0 && ctas == 0 && window == 0 && chunk == 0) { // few rows: one launch that takes no workspace
    Py_BEGIN_ALLOW_THREADS
    if constexpr (FP8)
      rc = g_decode_fp8_few(to, qp, kp, vp, tables, rows, (int32_t)B, (int32_t)H, (int32_t)kv, (int32_t)D, qs, H * D, nb, bs, bt_stride, scale,
                            f9, f10, type, on);
    else
      rc = g_decode_few(to, qp, kp, vp, tables, rows, (int32_t)B, (int32_t)H, (int32_t)kv, (int32_t)D, qs, H * D, nb, bs, bt_stride, scale, f9,
                        nullptr, type, on);
    Py_END_ALLOW_THREADS
  }
  if (rc != B200_ERR_UNSUPPORTED) return status(rc, std::move(out));
  PyObject* device = PyObject_GetAttrString(a[1], "device");
  if (device == nullptr) return nullptr;
  PyObject* held = PyObject_CallFunction(a[0], "LLLLO", (long long)B, (long long)H, (long long)kv, (long long)D, device);
  Py_DECREF(device);
  if (held == nullptr) return nullptr;
  const at::Tensor* ws = cuda_tensor(held);
  if (ws == nullptr) {
    Py_DECREF(held);
    Py_RETURN_NONE;
  }
  PyObject* got = nullptr;
  try {
    void* const wp = ws->data_ptr();
    const size_t bytes = (size_t)ws->numel();
    Py_BEGIN_ALLOW_THREADS
    if constexpr (FP8)
      rc = g_decode_fp8(to, qp, kp, vp, tables, rows, (int32_t)B, (int32_t)H, (int32_t)kv, (int32_t)D, qs, H * D, nb, bs, bt_stride, scale,
                        f9, f10, wp, bytes, (int32_t)ctas, type, on);
    else
      rc = g_decode(to, qp, kp, vp, tables, rows, (int32_t)B, (int32_t)H, (int32_t)kv, (int32_t)D, (int32_t)D, qs, H * D, nb, bs, bt_stride,
                    scale, f9, nullptr, window, keep_first, chunk, wp, bytes, (int32_t)ctas, type, on);
    Py_END_ALLOW_THREADS
    got = status(rc, std::move(out));
  } catch (...) {
    Py_DECREF(held);
    throw;
  }
  Py_DECREF(held);
  return got;
  END_HANDLE_TH_ERRORS
}

// prefill(workspace tensor or None, q, k, v, cu_seqlens_q, cu_seqlens_k, block_tables or None, max_seqlen_q, max_seqlen_k, scale, num_kv_heads,
// softcap, sink or None, window, keep_first, chunk)
PyObject* prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 16 || !ints(a + 7, 2) || !reals(a + 9, 1) || !ints(a + 10, 1) || !reals(a + 11, 1) || !ints(a + 13, 3) || c10::impl::TorchDispatchModeTLS::any_modes_set()) Py_RETURN_NONE;
  const bool paged = a[6] != Py_None;
  const at::Tensor *q = cuda_tensor(a[1]), *k = cuda_tensor(a[2]), *v = cuda_tensor(a[3]), *cq = cuda_tensor(a[4]), *ck = cuda_tensor(a[5]),
                   *bt = paged ? cuda_tensor(a[6]) : nullptr, *ws = a[0] != Py_None ? cuda_tensor(a[0]) : nullptr,
                   *sink = a[12] != Py_None ? cuda_tensor(a[12]) : nullptr;
  if (!q || !k || !v || !cq || !ck || (paged && !bt) || (a[0] != Py_None && !ws) || (a[12] != Py_None && !sink)) Py_RETURN_NONE;
  if (element(*q) < 0 || q->dim() != 3 || !is_int(*cq) || !is_int(*ck)) Py_RETURN_NONE;
  const int64_t T = q->size(0), H = q->size(1), D = q->size(2), kv = whole(a[10]);
  if (!heads_fit(*q, D)) Py_RETURN_NONE;
  if (sink && (sink->numel() != H || sink->scalar_type() != at::kFloat || !sink->is_contiguous())) Py_RETURN_NONE;
  int64_t ks = kv * D, vs = kv * D, nb = 0, bs = 0, total_k = 0;
  if (paged) {
    if (!is_int(*bt) || bt->dim() != 2 || bt->stride(1) != 1 || !cache_fits(*k, kv * D) || !cache_fits(*v, kv * D)) Py_RETURN_NONE;
    nb = k->size(0), bs = k->size(1);
  } else {
    if (!heads_fit(*k, D) || !heads_fit(*v, D)) Py_RETURN_NONE;
    total_k = k->size(0);
    if (k->size(0) > 1) ks = k->stride(0);
    if (v->size(0) > 1) vs = v->stride(0);
  }
  at::Tensor out = at::empty({T, H * D}, q->options());
  const int32_t max_q = (int32_t)whole(a[7]), max_k = (int32_t)whole(a[8]);
  const float scale = real(a[9]), softcap = real(a[11]);
  const int32_t window = (int32_t)whole(a[13]), keep_first = (int32_t)whole(a[14]), chunk = (int32_t)whole(a[15]);
  void *const to = out.data_ptr(), *const qp = q->data_ptr(), *const kp = k->data_ptr(), *const vp = v->data_ptr(),
             *const wp = ws ? ws->data_ptr() : nullptr;
  const int32_t *const cqp = (const int32_t*)cq->data_ptr(), *const ckp = (const int32_t*)ck->data_ptr(),
                *const tables = paged ? (const int32_t*)bt->data_ptr() : nullptr;
  const float* const sinks = sink ? (const float*)sink->data_ptr() : nullptr;
  const int32_t seqs = (int32_t)(cq->numel() - 1), bt_stride = paged ? (int32_t)bt->stride(0) : 0;
  const int64_t qs = T > 1 ? q->stride(0) : H * D, bytes = ws ? ws->numel() : 0;
  const int type = element(*q);
  void* const on = stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_prefill(to, qp, kp, vp, cqp, ckp, seqs, (int32_t)T, (int32_t)total_k, max_q, max_k, (int32_t)H, (int32_t)kv, (int32_t)D, (int32_t)D,
                 qs, ks, vs, H * D, tables, bt_stride, (int32_t)nb, (int32_t)bs, scale, softcap, sinks, window, keep_first, chunk, type, wp,
                 bytes, on);
  Py_END_ALLOW_THREADS
  return status(rc, std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind(addresses of the five library functions)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "bind takes five addresses");
    return nullptr;
  }
  void* p[5];
  for (int i = 0; i < 5; ++i)
    if ((p[i] = PyLong_AsVoidPtr(a[i])) == nullptr) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null address");
      return nullptr;
    }
  g_decode = (decltype(g_decode))p[0], g_decode_fp8 = (decltype(g_decode_fp8))p[1], g_prefill = (decltype(g_prefill))p[2];
  g_decode_few = (decltype(g_decode_few))p[3], g_decode_fp8_few = (decltype(g_decode_fp8_few))p[4];
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"decode", (PyCFunction)(void (*)())decode<false>, METH_FASTCALL, nullptr},
    {"decode_fp8", (PyCFunction)(void (*)())decode<true>, METH_FASTCALL, nullptr},
    {"prefill", (PyCFunction)(void (*)())prefill, METH_FASTCALL, nullptr},
    {"bind", (PyCFunction)(void (*)())bind, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200calls() { return PyModule_Create(&module); }
