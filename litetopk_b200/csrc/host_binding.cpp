// The plain calls of sparse_prefill, lite_topk and the two DSv4 operators in one step from Python: arguments, output and workspace
// tensors, the C ABI.  A call of a few tokens takes 13 to 20 us on the device; by way of ctypes, with the checks and allocations in
// Python, its host side took as long or longer and was what such calls were bound by: sparse_prefill of 2 tokens 22 us (11 this
// way), dsv4_c128a_bf16 of 24 tokens 19 (9), lite_topk and sparse_prefill of 36 tokens 48 (19).
//
// Each function takes the arguments of its operator in api.py and returns the result (True from dsv4_masked_mla_bf16_out, whose caller
// has it), the status code of a call that the library refused (lite_topk, which makes two: with the refused one's name), or None for
// whatever is not plain: then nothing has been done, and api.py goes its own way, checks and errors included.  Plain are dense CUDA tensors of the expected types, shapes and strides on the current device that
// no dispatch mode, function transform or subclass stands behind.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/litedsa_b200.h"

namespace {

using at::Tensor;

// a plain CUDA tensor on the current device, or null
const Tensor* plain(PyObject* o, int dev) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_conj() || t.is_neg() ||
      at::isTensorSubclassLike(t) || t.get_device() != dev)
    return nullptr;
  return &t;
}
bool number(PyObject* o, double* v) {      // Python's own floats and integers
  if (PyFloat_CheckExact(o)) { *v = PyFloat_AS_DOUBLE(o); return true; }
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsDouble(o);
  if (*v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
bool integer(PyObject* o, int64_t* v) {      // 0 .. 2^31 - 1
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0 && *v >= 0 && *v <= 0x7fffffff;
}
bool small(int64_t n) { return n <= 0x7fffffff; }
bool e4m3(const Tensor& t) { return t.scalar_type() == at::kByte || t.scalar_type() == at::kFloat8_e4m3fn; }
// heads per token that tile 128 rows
bool heads_ok(int64_t h) { return h > 0 && h <= 128 && 128 % h == 0 && 128 / h <= 16; }
// the current device, or -1 if a call with this first argument is not plain anyway (the runtime is not asked without a GPU)
int current_device(PyObject* first) {
  if (!THPVariable_CheckExact(first) || !THPVariable_Unpack(first).is_cuda() || c10::impl::dispatch_mode_enabled()) return -1;
  return static_cast<int>(c10::cuda::current_device());
}
void* stream_of(int dev) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream(); }
Tensor empty(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
  return at::empty(size, at::TensorOptions().dtype(type).device(like.device()));
}
PyObject* pair(const Tensor& a, const Tensor& b) {
  PyObject* pa = THPVariable_Wrap(a);
  PyObject* pb = pa ? THPVariable_Wrap(b) : nullptr;
  PyObject* r = pb ? PyTuple_Pack(2, pa, pb) : nullptr;
  Py_XDECREF(pa);
  Py_XDECREF(pb);
  return r;
}
// allocations and launches can block: other Python threads run meanwhile, as with ctypes
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
// Exceptions and warnings leave as they do from torch's own functions: a Python exception raised below a call as itself, a C++ one as
// the Python class that torch has for it.
template <class F>
PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  return f();
  END_HANDLE_TH_ERRORS
}

// (q, kv, topk_idx, sm_scale, kv_scale, q_scale, seq_space, job_tokens)
PyObject* sparse_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int dev = current_device(a[0]);
    const Tensor *q = plain(a[0], dev), *kv = plain(a[1], dev), *idx = plain(a[2], dev);
    double sm = 0, kv_scale = 1.0, q_scale = 1.0;
    int64_t space = 0, job = 0;
    if (!q || !kv || !idx || q->dim() != 3 || kv->dim() != 2 || idx->dim() != 2 || !number(a[3], &sm)) Py_RETURN_NONE;
    const int64_t T = q->size(0), h = q->size(1), k = idx->size(1), s_kv = kv->size(0);
    const bool q_bf16 = q->scalar_type() == at::kBFloat16, kv_bf16 = kv->scalar_type() == at::kBFloat16;
    if (T <= 0 || !small(T) || !heads_ok(h) || q->size(2) != 576 || T % (128 / h) != 0 || !q->is_contiguous() || !(q_bf16 || e4m3(*q)) ||
        idx->scalar_type() != at::kInt || idx->size(0) != T || k <= 0 || !small(k) || !idx->is_contiguous() || kv->size(1) != 576 ||
        kv->stride(1) != 1 || s_kv <= 0 || !small(s_kv) || !(kv_bf16 || e4m3(*kv)) || (kv_bf16 && !q_bf16))
      Py_RETURN_NONE;
    if (a[4] != Py_None && !number(a[4], &kv_scale)) Py_RETURN_NONE;
    if (a[5] != Py_None ? !number(a[5], &q_scale) : q_bf16 && !kv_bf16) Py_RETURN_NONE;
    // bf16 queries that get a pass of their own (_quantise_first in api.py)
    if (q_bf16 && !kv_bf16 && T * h / 128 > 296 && 128 / h * k <= (h == 128 ? 512 : 128)) Py_RETURN_NONE;
    if (a[6] == Py_None) space = s_kv;
    else if (!integer(a[6], &space)) Py_RETURN_NONE;
    if (a[7] == Py_None) job = T;
    else if (!integer(a[7], &job) || job < T) Py_RETURN_NONE;
    Tensor out, lse;
    int rc;
    {
      NoGil unlocked;
      out = empty({T, h, 512}, at::kBFloat16, *q);
      lse = empty({T, h}, at::kFloat, *q);
      const int64_t bytes = litedsa_sparse_prefill_job_workspace((int)T, (int)h, (int)k, kv_bf16, (int)job);
      Tensor ws = empty({bytes > 0 ? bytes : 1}, at::kByte, *q);
      rc = litedsa_sparse_prefill_job(q->data_ptr(), q_bf16, kv->data_ptr(), kv_bf16, static_cast<const int32_t*>(idx->data_ptr()), sm, q_scale,
                                      kv_scale, out.data_ptr(), static_cast<float*>(lse.data_ptr()), (int)T, (int)h, (int)k, (int)s_kv,
                                      kv->stride(0), (space + 1023) / 1024 * 1024, (int)job, ws.data_ptr(), ws.numel(), stream_of(dev));
    }
    return rc == LITEDSA_OK ? pair(out, lse) : PyLong_FromLong(rc);
  });
}

// (q, kv_compressed, kv_raw, q_pos0, sm_scale, window, ratio, attn_sink)
PyObject* dsv4_c128a_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int dev = current_device(a[0]);
    const Tensor *q = plain(a[0], dev), *kc = a[1] == Py_None ? nullptr : plain(a[1], dev), *kr = plain(a[2], dev);
    const Tensor* sink = a[7] == Py_None ? nullptr : plain(a[7], dev);
    double sm = 0;
    int64_t pos0 = 0, window = 0, ratio = 0;
    auto rows = [](const Tensor& t) {
      return t.dim() == 2 && t.scalar_type() == at::kBFloat16 && t.size(1) == 576 && t.stride(1) == 1 && t.size(0) > 0 && small(t.size(0));
    };
    if (!q || !kr || (a[1] != Py_None && !kc) || (a[7] != Py_None && !sink) || !number(a[4], &sm) || !integer(a[3], &pos0) ||
        !integer(a[5], &window) || !integer(a[6], &ratio))
      Py_RETURN_NONE;
    if (q->dim() != 3 || q->scalar_type() != at::kBFloat16 || q->size(2) != 576 || !q->is_contiguous() || !rows(*kr) || (kc && !rows(*kc)))
      Py_RETURN_NONE;
    const int64_t T = q->size(0), h = q->size(1);
    if (T <= 0 || !small(T) || !heads_ok(h) || T % (128 / h) != 0) Py_RETURN_NONE;
    if (sink && (sink->scalar_type() != at::kFloat || sink->dim() != 1 || sink->size(0) != h || !sink->is_contiguous())) Py_RETURN_NONE;
    const int ng = (int)(T * h / 128), n_comp = kc ? (int)kc->size(0) : 0;
    Tensor out, lse;
    int rc;
    {
      NoGil unlocked;
      Tensor ws;
      out = empty({T, h, 512}, at::kBFloat16, *q);
      lse = empty({T, h}, at::kFloat, *q);
      const int64_t bytes = litedsa_dsv4_workspace(ng, (int)h, n_comp, (int)pos0, (int)window, (int)ratio);
      if (bytes > 0) ws = empty({bytes}, at::kByte, *q);
      rc = litedsa_dsv4_c128a_bf16_ws(q->data_ptr(), kc ? kc->data_ptr() : nullptr, kr->data_ptr(), ng, (int)h, n_comp, (int)kr->size(0),
                                      (int)pos0, (int)window, (int)ratio, (float)sm, sink ? static_cast<const float*>(sink->data_ptr()) : nullptr,
                                      (int)h, out.data_ptr(), static_cast<float*>(lse.data_ptr()), 576, kc ? kc->stride(0) : 576,
                                      kr->stride(0), h * 576, 576, h * 512, 512, bytes > 0 ? ws.data_ptr() : nullptr, bytes, stream_of(dev));
    }
    return rc == LITEDSA_OK ? pair(out, lse) : PyLong_FromLong(rc);
  });
}

// (q, kv, indices, pref, win_lo, win_hi, counts, sm_scale, h_per_q, out, lse, attn_sink), dense packed, with run detection; True if done
PyObject* dsv4_masked_mla_bf16_out(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 12) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int dev = current_device(a[0]);
    const Tensor *q = plain(a[0], dev), *kv = plain(a[1], dev), *idx = plain(a[2], dev), *counts = plain(a[6], dev), *out = plain(a[9], dev),
                 *lse = plain(a[10], dev), *sink = a[11] == Py_None ? nullptr : plain(a[11], dev);
    const Tensor* range[3] = {plain(a[3], dev), plain(a[4], dev), plain(a[5], dev)};
    double sm = 0;
    int64_t h = 0;
    if (!q || !kv || !idx || !counts || !out || !lse || (a[11] != Py_None && !sink) || !number(a[7], &sm) || !integer(a[8], &h)) Py_RETURN_NONE;
    // [rows, d] or [rows, 1, d] with unit inner stride
    auto rows = [](const Tensor& t) {
      return (t.dim() == 2 || (t.dim() == 3 && t.size(1) == 1)) && t.stride(-1) == 1 && t.size(0) > 0 && small(t.size(0)) && small(t.size(-1));
    };
    if (q->dim() != 3 || q->scalar_type() != at::kBFloat16 || kv->scalar_type() != at::kBFloat16 || idx->scalar_type() != at::kInt ||
        !rows(*kv) || !rows(*idx) || !heads_ok(h))
      Py_RETURN_NONE;
    const int64_t ng = q->size(0), d = q->size(2);
    if (ng <= 0 || !small(ng) || q->size(1) != 128 || (d != 512 && d != 576) || kv->size(-1) != d || q->stride(2) != 1 ||
        q->stride(1) * 128 != q->stride(0) || idx->size(0) != ng)
      Py_RETURN_NONE;
    for (const Tensor* t : range)
      if (!t || t->scalar_type() != at::kInt || t->numel() != ng * (128 / h) || !t->is_contiguous()) Py_RETURN_NONE;
    if (counts->scalar_type() != at::kInt || counts->dim() != 1 || counts->size(0) != ng || !counts->is_contiguous()) Py_RETURN_NONE;
    if (out->scalar_type() != at::kBFloat16 || out->dim() != 3 || out->size(0) != ng || out->size(1) != 128 || out->size(2) != 512 ||
        !out->is_contiguous() || lse->scalar_type() != at::kFloat || lse->numel() != ng * 128 || !lse->is_contiguous())
      Py_RETURN_NONE;
    if (sink && (sink->scalar_type() != at::kFloat || sink->dim() != 1 || sink->size(0) != 128 || !sink->is_contiguous())) Py_RETURN_NONE;
    auto ints = [](const Tensor* t) { return static_cast<const int32_t*>(t->data_ptr()); };
    int rc;
    {
      NoGil unlocked;
      Tensor ws = empty({16 + 16 * ng}, at::kByte, *q);
      rc = litedsa_dsv4_masked_mla_bf16(q->data_ptr(), kv->data_ptr(), ints(idx), ints(range[0]), ints(range[1]), ints(range[2]), ints(counts),
                                        (float)sm, (int)h, out->data_ptr(), static_cast<float*>(lse->data_ptr()),
                                        sink ? static_cast<const float*>(sink->data_ptr()) : nullptr, (int)ng, (int)kv->size(0),
                                        (int)idx->size(-1), (int)d, q->stride(1), kv->stride(0), idx->stride(0), 0, 0, 0, 0, ws.data_ptr(),
                                        ws.numel(), stream_of(dev));
    }
    if (rc != LITEDSA_OK) return PyLong_FromLong(rc);
    Py_RETURN_TRUE;
  });
}

// (q_idx8, k_idx8, weights, k_scale, k, q_pos0): index logits into a workspace of this call, selection
PyObject* lite_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int dev = current_device(a[0]);
    const Tensor *q = plain(a[0], dev), *k8 = plain(a[1], dev), *w = plain(a[2], dev), *ks = a[3] == Py_None ? nullptr : plain(a[3], dev);
    int64_t k = 0, pos0 = 0;
    if (!q || !k8 || !w || (a[3] != Py_None && !ks) || !integer(a[4], &k) || !integer(a[5], &pos0)) Py_RETURN_NONE;
    if (q->dim() != 3 || k8->dim() != 2 || w->dim() != 2 || !e4m3(*q) || !e4m3(*k8) || w->scalar_type() != at::kFloat) Py_RETURN_NONE;
    const int64_t T = q->size(0), Hi = q->size(1), S = k8->size(0), ld = (S + 3) / 4 * 4;
    if (T <= 0 || S <= 0 || k <= 0 || !small(T) || !small(ld) || !small(Hi) || q->size(2) != 128 || !q->is_contiguous() || k8->size(1) != 128 ||
        k8->stride(1) != 1 || w->size(0) != T || w->size(1) != Hi || !w->is_contiguous())
      Py_RETURN_NONE;
    if (ks && (ks->scalar_type() != at::kFloat || ks->dim() != 1 || ks->size(0) != S || !ks->is_contiguous())) Py_RETURN_NONE;
    // rows start on 16-byte boundaries whatever S is: the streaming selection kernels need that
    Tensor out;
    int rc;
    const char* where = "index_logits_fp8";
    {
      NoGil unlocked;
      Tensor logits = empty({T, ld}, at::kFloat, *q);
      void* stream = stream_of(dev);
      rc = litedsa_index_logits_fp8(q->data_ptr(), k8->data_ptr(), static_cast<const float*>(w->data_ptr()),
                                    ks ? static_cast<const float*>(ks->data_ptr()) : nullptr, static_cast<float*>(logits.data_ptr()), (int)T,
                                    (int)Hi, (int)S, (int)pos0, k8->stride(0), ld, stream);
      if (rc == LITEDSA_OK) {
        where = "topk_select";
        out = empty({T, k}, at::kInt, *q);
        rc = litedsa_topk_select(static_cast<const float*>(logits.data_ptr()), nullptr, static_cast<int32_t*>(out.data_ptr()), (int)T, (int)S,
                                 (int)k, (int)pos0, ld, stream);
      }
    }
    return rc == LITEDSA_OK ? THPVariable_Wrap(out) : Py_BuildValue("(is)", rc, where);
  });
}

PyMethodDef kMethods[] = {
    {"sparse_prefill", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(sparse_prefill)), METH_FASTCALL, nullptr},
    {"dsv4_c128a_bf16", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(dsv4_c128a_bf16)), METH_FASTCALL, nullptr},
    {"dsv4_masked_mla_bf16_out", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(dsv4_masked_mla_bf16_out)), METH_FASTCALL, nullptr},
    {"lite_topk", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(lite_topk)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "litedsa_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_litedsa_host() { return PyModule_Create(&kModule); }
