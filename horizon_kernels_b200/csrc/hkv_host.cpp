// Native side of kernels.write, kernels.decode_ragged and kernels.prefill, and of the backend's cache update and decode: takes
// the callers' Python arguments as they are, checks them and calls the C ABI (include/hkv.h). What the wrappers do per call in
// Python (about forty attribute reads and checks, a device context, the conversion of 25 ctypes arguments) costs 20 to 25
// microseconds, longer than a small decode step runs on the GPU; here it costs two.
//
// Each function answers None when an argument is not of the plain form it knows (wrong type, shape or device, a tensor
// subclass, anything that throws): nothing has been launched then, and the Python path checks, raises or serves the
// call. Otherwise it answers the status of the C call. No state is kept between calls.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/Functions.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/hkv.h"

namespace {

struct Abi {                       // entry points of the loaded libhkv.so, handed over by bind()
  decltype(&hkv_write) write = nullptr;
  decltype(&hkv_write_rot) write_rot = nullptr;
  decltype(&hkv_write_k8) write_k8 = nullptr;
  decltype(&hkv_decode) decode = nullptr;
  decltype(&hkv_decode_rot) decode_rot = nullptr;
  decltype(&hkv_decode_k8) decode_k8 = nullptr;
  decltype(&hkv_prefill_scratch_bytes) prefill_scratch_bytes = nullptr;
  decltype(&hkv_prefill) prefill = nullptr;
} abi;

const at::Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

bool integer(PyObject* o, long long* v) {
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsLongLong(o);
  if (*v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool number(PyObject* o, double* v) {
  if (!PyFloat_CheckExact(o)) return false;
  *v = PyFloat_AS_DOUBLE(o);
  return true;
}
bool boolean(PyObject* o, bool* v) {
  if (!PyBool_Check(o)) return false;
  *v = o == Py_True;
  return true;
}
bool on(const at::Tensor& t, int dev) { return t.is_cuda() && t.device().index() == dev; }

struct Cache {
  void* part[4];
  int64_t strides[6];
};
bool cache_of(PyObject* flat, PyObject* strides, int dev, Cache* c) {
  if (!PyTuple_CheckExact(flat) || PyTuple_GET_SIZE(flat) != 4 || !PyTuple_CheckExact(strides) || PyTuple_GET_SIZE(strides) != 6)
    return false;
  for (int i = 0; i < 4; ++i) {
    const at::Tensor* t = tensor(PyTuple_GET_ITEM(flat, i));
    if (!t || !on(*t, dev)) return false;
    c->part[i] = t->data_ptr();
  }
  for (int i = 0; i < 6; ++i) {
    long long v;
    if (!integer(PyTuple_GET_ITEM(strides, i), &v)) return false;
    c->strides[i] = v;
  }
  return true;
}
// per-head scales and, with rotated keys, the sign vector
bool scales(const at::Tensor* gk, const at::Tensor* gv, int64_t KVH, int dev) {
  for (const at::Tensor* t : {gk, gv})
    if (!t || !on(*t, dev) || t->scalar_type() != at::kFloat || t->dim() != 1 || t->size(0) != KVH || !t->is_contiguous()) return false;
  return true;
}
bool sign_vector(PyObject* o, int64_t D, int dev, const float** p) {
  *p = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = tensor(o);
  if (!t || !on(*t, dev) || t->scalar_type() != at::kFloat || t->dim() != 1 || t->size(0) != D || !t->is_contiguous()) return false;
  *p = static_cast<const float*>(t->data_ptr());
  return true;
}

// The launches behind the checks. Cache parts and strides as in include/hkv.h.
struct Rows {                      // new keys and values
  const void *k, *v;
  int64_t k0, k1, v0, v1, KVH, D;
};
PyObject* run_write(const Rows& r, const Cache& c, int PS, const at::Tensor& slots, const at::Tensor& gk, const at::Tensor& gv, bool search,
                    const float* signs, bool k8, int dev) {
  const int64_t *sl = static_cast<const int64_t*>(slots.data_ptr()), n_slots = slots.size(0);
  const float *gkp = static_cast<const float*>(gk.data_ptr()), *gvp = static_cast<const float*>(gv.data_ptr());
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  if (k8)
    rc = abi.write_k8(r.k, r.v, r.k0, r.k1, r.v0, r.v1, c.part[0], c.part[2], c.part[3], c.strides, PS, sl, n_slots, gkp, gvp,
                      (int)r.KVH, (int)r.D, search, st);
  else if (signs)
    rc = abi.write_rot(r.k, r.v, r.k0, r.k1, r.v0, r.v1, c.part[0], c.part[1], c.part[2], c.part[3], c.strides, PS, sl, n_slots, gkp,
                       gvp, (int)r.KVH, (int)r.D, search, signs, st);
  else
    rc = abi.write(r.k, r.v, r.k0, r.k1, r.v0, r.v1, c.part[0], c.part[1], c.part[2], c.part[3], c.strides, PS, sl, n_slots, gkp, gvp,
                   (int)r.KVH, (int)r.D, search, st);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}
PyObject* run_decode(const void* q, const Cache& c, int PS, const at::Tensor& bt, const at::Tensor& lens, const at::Tensor& qsl, int64_t HQ,
                     int64_t D, double s1, double s2, const at::Tensor& gk, const at::Tensor& gv, int qlmax, void* out,
                     const at::Tensor& ws, int splits, const float* signs, bool k8, int dev) {
  const int32_t *btp = static_cast<const int32_t*>(bt.data_ptr()), *lp = static_cast<const int32_t*>(lens.data_ptr()),
                *sp = static_cast<const int32_t*>(qsl.data_ptr());
  const float *gkp = static_cast<const float*>(gk.data_ptr()), *gvp = static_cast<const float*>(gv.data_ptr());
  void* wp = ws.data_ptr();
  const size_t wsb = ws.nbytes();
  const int B = (int)bt.size(0), MP = (int)bt.size(1), KVH = (int)gk.size(0), G = (int)(HQ / KVH);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  if (k8)
    rc = abi.decode_k8(q, c.part[0], c.part[2], c.part[3], c.strides, PS, btp, MP, lp, sp, B, KVH, G, (int)D, qlmax, (float)s1,
                       (float)s2, gkp, gvp, wp, wsb, splits, out, st);
  else if (signs)
    rc = abi.decode_rot(q, c.part[0], c.part[1], c.part[2], c.part[3], c.strides, PS, btp, MP, lp, sp, B, KVH, G, (int)D, qlmax,
                        (float)s1, (float)s2, gkp, gvp, wp, wsb, splits, signs, out, st);
  else
    rc = abi.decode(q, c.part[0], c.part[1], c.part[2], c.part[3], c.strides, PS, btp, MP, lp, sp, B, KVH, G, (int)D, qlmax, (float)s1,
                    (float)s2, gkp, gvp, wp, wsb, splits, out, st);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}
// parts and strides of the logical (pages, heads, positions, slot) cache that the engine holds, as layout.slot_views /
// flat_views (K8: k8_views / k8_flat_views) give them
bool cache_of_slots(PyObject* o, int64_t KVH, int64_t D, bool k8, int dev, Cache* c, int* PS) {
  const at::Tensor* t = tensor(o);
  if (!t || !on(*t, dev) || t->scalar_type() != at::kByte || t->dim() != 4 || (D != 128 && D != 256)) return false;
  const int64_t slot = (k8 ? D : 0) + D / 2 + D / 16;
  if (t->size(1) != (k8 ? KVH : 2 * KVH) || t->size(3) != slot || t->stride(3) != 1 || t->size(2) > INT32_MAX) return false;
  uint8_t* p = static_cast<uint8_t*>(t->data_ptr());
  uint8_t* v = k8 ? p + D : p + KVH * t->stride(1);
  c->part[0] = p;
  c->part[1] = k8 ? v + D / 2 : p + D / 2;
  c->part[2] = v;
  c->part[3] = v + D / 2;
  for (int i = 0; i < 6; i += 3) {
    c->strides[i] = t->stride(0);
    c->strides[i + 1] = t->stride(2);
    c->strides[i + 2] = t->stride(1);
  }
  *PS = (int)t->size(2);
  return true;
}
// (tokens, heads * D) or (tokens, heads, D) bf16
bool token_rows(const at::Tensor& t, int64_t heads, int64_t D) {
  return t.scalar_type() == at::kBFloat16 && ((t.dim() == 2 && t.size(1) == heads * D) || (t.dim() == 3 && t.size(1) == heads && t.size(2) == D));
}

// write(key, value, flat, strides, PS, slot_mapping, gk, gv, search, signs, k8)
PyObject* write(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 11 || !abi.write) Py_RETURN_NONE;
    const at::Tensor *k = tensor(a[0]), *v = tensor(a[1]), *slots = tensor(a[5]), *gk = tensor(a[6]), *gv = tensor(a[7]);
    if (!k || !v || !slots || !k->is_cuda()) Py_RETURN_NONE;
    const int dev = k->device().index();
    long long PS;
    bool search, k8;
    const float* signs;
    Cache c;
    if (dev != c10::cuda::current_device() || !on(*v, dev) || !on(*slots, dev) || k->scalar_type() != at::kBFloat16 ||
        v->scalar_type() != at::kBFloat16 || k->dim() != 3 || v->sizes() != k->sizes() || k->stride(2) != 1 || v->stride(2) != 1 ||
        slots->scalar_type() != at::kLong || slots->dim() != 1 || !slots->is_contiguous() || slots->size(0) > k->size(0) ||
        !integer(a[4], &PS) || PS != (int)PS || !boolean(a[8], &search) || !boolean(a[10], &k8))
      Py_RETURN_NONE;
    const int64_t KVH = k->size(1), D = k->size(2);
    if (KVH > INT32_MAX || D > INT32_MAX || !scales(gk, gv, KVH, dev) || !sign_vector(a[9], D, dev, &signs) || (k8 && signs) ||
        !cache_of(a[2], a[3], dev, &c))
      Py_RETURN_NONE;
    return run_write({k->data_ptr(), v->data_ptr(), k->stride(0), k->stride(1), v->stride(0), v->stride(1), KVH, D}, c, (int)PS, *slots, *gk,
                     *gv, search, signs, k8, dev);
  } catch (...) {
    Py_RETURN_NONE;
  }
}

// decode(query, flat, strides, PS, block_tables, seq_lens, query_start_loc, bmm1_scale, bmm2_scale, gk, gv, qlmax, out,
//        workspace, splits, signs, k8)
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 17 || !abi.decode) Py_RETURN_NONE;
    const at::Tensor *q = tensor(a[0]), *bt = tensor(a[4]), *lens = tensor(a[5]), *qsl = tensor(a[6]), *gk = tensor(a[9]),
                     *gv = tensor(a[10]), *out = tensor(a[12]), *ws = tensor(a[13]);
    if (!q || !bt || !lens || !qsl || !gk || !out || !ws || !q->is_cuda() || gk->dim() != 1) Py_RETURN_NONE;
    const int dev = q->device().index();
    long long PS, qlmax, splits = 0;
    double s1, s2;
    bool k8;
    const float* signs;
    Cache c;
    if (dev != c10::cuda::current_device() || !integer(a[3], &PS) || PS != (int)PS || !number(a[7], &s1) || !number(a[8], &s2) ||
        !integer(a[11], &qlmax) || qlmax != (int)qlmax || (a[14] != Py_None && (!integer(a[14], &splits) || splits != (int)splits)) ||
        !boolean(a[16], &k8))
      Py_RETURN_NONE;
    if (q->scalar_type() != at::kBFloat16 || out->scalar_type() != at::kBFloat16 || q->dim() != 3 || out->dim() != 3 ||
        out->size(1) != q->size(1) || out->size(2) != q->size(2) || out->size(0) < q->size(0) || !q->is_contiguous() ||
        !out->is_contiguous() || bt->dim() != 2 || lens->dim() != 1 || qsl->dim() != 1 || lens->size(0) != bt->size(0) ||
        qsl->size(0) != bt->size(0) + 1 || !on(*out, dev) || !on(*ws, dev))
      Py_RETURN_NONE;
    for (const at::Tensor* t : {bt, lens, qsl})
      if (!on(*t, dev) || t->scalar_type() != at::kInt || !t->is_contiguous()) Py_RETURN_NONE;
    const int64_t B = bt->size(0), MP = bt->size(1), KVH = gk->size(0), HQ = q->size(1), D = q->size(2);
    if (KVH < 1 || HQ % KVH || B > INT32_MAX || MP > INT32_MAX || HQ > INT32_MAX || D > INT32_MAX || !scales(gk, gv, KVH, dev) ||
        !sign_vector(a[15], D, dev, &signs) || (k8 && signs) || !cache_of(a[1], a[2], dev, &c))
      Py_RETURN_NONE;
    return run_decode(q->data_ptr(), c, (int)PS, *bt, *lens, *qsl, HQ, D, s1, s2, *gk, *gv, (int)qlmax, out->data_ptr(), *ws, (int)splits, signs,
                      k8, dev);
  } catch (...) {
    Py_RETURN_NONE;
  }
}

// layer_write(key, value, kv_cache, slot_mapping, gk, gv, D, search, signs, k8)
PyObject* layer_write(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 10 || !abi.write) Py_RETURN_NONE;
    const at::Tensor *k = tensor(a[0]), *v = tensor(a[1]), *slots = tensor(a[3]), *gk = tensor(a[4]), *gv = tensor(a[5]);
    if (!k || !v || !slots || !gk || !k->is_cuda() || gk->dim() != 1) Py_RETURN_NONE;
    const int dev = k->device().index();
    const int64_t KVH = gk->size(0);
    long long D;
    bool search, k8;
    const float* signs;
    int PS;
    Cache c;
    if (dev != c10::cuda::current_device() || !on(*v, dev) || !on(*slots, dev) || !integer(a[6], &D) || !boolean(a[7], &search) ||
        !boolean(a[9], &k8) || KVH < 1 || KVH > 65536 || !cache_of_slots(a[2], KVH, D, k8, dev, &c, &PS) || !token_rows(*k, KVH, D) ||
        !token_rows(*v, KVH, D) || k->dim() != v->dim() || k->size(0) != v->size(0) || k->stride(-1) != 1 || v->stride(-1) != 1 ||
        slots->scalar_type() != at::kLong || slots->dim() != 1 || !slots->is_contiguous() || slots->size(0) > k->size(0) ||
        !scales(gk, gv, KVH, dev) || !sign_vector(a[8], D, dev, &signs) || (k8 && signs))
      Py_RETURN_NONE;
    const bool flat = k->dim() == 2;
    return run_write({k->data_ptr(), v->data_ptr(), k->stride(0), flat ? D : k->stride(1), v->stride(0), flat ? D : v->stride(1), KVH, D}, c, PS,
                     *slots, *gk, *gv, search, signs, k8, dev);
  } catch (...) {
    Py_RETURN_NONE;
  }
}

// layer_decode(query, kv_cache, block_table, seq_lens, query_start_loc, tokens, scale, v_scale, gk, gv, qlmax, output, workspace,
//              splits, heads, D, signs, k8); the first `tokens` rows of query belong to the step
PyObject* layer_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 18 || !abi.decode) Py_RETURN_NONE;
    const at::Tensor *q = tensor(a[0]), *bt = tensor(a[2]), *lens = tensor(a[3]), *qsl = tensor(a[4]), *gk = tensor(a[8]),
                     *gv = tensor(a[9]), *out = tensor(a[11]), *ws = tensor(a[12]);
    if (!q || !bt || !lens || !qsl || !gk || !out || !ws || !q->is_cuda() || gk->dim() != 1) Py_RETURN_NONE;
    const int dev = q->device().index();
    const int64_t KVH = gk->size(0);
    long long T, qlmax, splits, HQ, D;
    double s1, s2;
    bool k8;
    const float* signs;
    int PS;
    Cache c;
    if (dev != c10::cuda::current_device() || !integer(a[5], &T) || !number(a[6], &s1) || !number(a[7], &s2) || !integer(a[10], &qlmax) ||
        qlmax != (int)qlmax || !integer(a[13], &splits) || splits != (int)splits || !integer(a[14], &HQ) || HQ != (int)HQ ||
        !integer(a[15], &D) || !boolean(a[17], &k8) || KVH < 1 || KVH > 65536 || HQ < 1 || HQ % KVH)
      Py_RETURN_NONE;
    if (!cache_of_slots(a[1], KVH, D, k8, dev, &c, &PS) || !token_rows(*q, HQ, D) || !token_rows(*out, HQ, D) || !q->is_contiguous() ||
        !out->is_contiguous() || T < 0 || q->size(0) < T || out->size(0) < T || bt->dim() != 2 || lens->dim() != 1 || qsl->dim() != 1 ||
        lens->size(0) != bt->size(0) || qsl->size(0) != bt->size(0) + 1 || !on(*out, dev) || !on(*ws, dev) || bt->size(0) > INT32_MAX ||
        bt->size(1) > INT32_MAX || !scales(gk, gv, KVH, dev) || !sign_vector(a[16], D, dev, &signs) || (k8 && signs))
      Py_RETURN_NONE;
    for (const at::Tensor* t : {bt, lens, qsl})
      if (!on(*t, dev) || t->scalar_type() != at::kInt || !t->is_contiguous()) Py_RETURN_NONE;
    return run_decode(q->data_ptr(), c, PS, *bt, *lens, *qsl, HQ, D, s1, s2, *gk, *gv, (int)qlmax, out->data_ptr(), *ws, (int)splits, signs,
                      k8, dev);
  } catch (...) {
    Py_RETURN_NONE;
  }
}

// prefill(query, flat, strides, PS, block_tables, rows, qk_scale, out_scale, KVH, out, chunk, signs, k8, workspace)
PyObject* prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 14 || !abi.prefill) Py_RETURN_NONE;
    const at::Tensor *q = tensor(a[0]), *bt = tensor(a[4]), *out = tensor(a[9]), *ws = a[13] == Py_None ? nullptr : tensor(a[13]);
    if (!q || !bt || !out || (!ws && a[13] != Py_None) || !q->is_cuda() || !PyList_CheckExact(a[5])) Py_RETURN_NONE;
    const int dev = q->device().index();
    long long PS, KVH, chunk;
    double s1, s2;
    bool k8;
    const float* signs;
    Cache c;
    if (dev != c10::cuda::current_device() || !integer(a[3], &PS) || PS < 1 || PS != (int)PS || !number(a[6], &s1) ||
        !number(a[7], &s2) || !integer(a[8], &KVH) || KVH < 1 || KVH != (int)KVH || !integer(a[10], &chunk) ||
        !boolean(a[12], &k8))
      Py_RETURN_NONE;
    const bool out_f32 = out->scalar_type() == at::kFloat;
    if (q->scalar_type() != at::kBFloat16 || (out->scalar_type() != at::kBFloat16 && !out_f32) || q->dim() != 3 || out->dim() != 3 ||
        out->size(1) != q->size(1) || out->size(2) != q->size(2) || out->size(0) < q->size(0) || !q->is_contiguous() ||
        !out->is_contiguous() || !on(*out, dev) || !on(*bt, dev) || bt->scalar_type() != at::kInt || bt->dim() != 2 ||
        !bt->is_contiguous() || (ws && (!on(*ws, dev) || ws->nbytes() < 64)))
      Py_RETURN_NONE;
    const int64_t B = bt->size(0), MP = bt->size(1), NT = q->size(0), HQ = q->size(1), D = q->size(2);
    if (HQ % KVH || B > INT32_MAX || MP > INT32_MAX || NT > INT32_MAX || HQ > INT32_MAX || D > INT32_MAX ||
        !sign_vector(a[11], D, dev, &signs) || (k8 && signs) || !cache_of(a[1], a[2], dev, &c))
      Py_RETURN_NONE;
    const Py_ssize_t n_rows = PyList_GET_SIZE(a[5]);
    if (n_rows > INT32_MAX) Py_RETURN_NONE;
    std::vector<int32_t> rows(4 * n_rows);
    for (Py_ssize_t i = 0; i < n_rows; ++i) {
      PyObject* t = PyList_GET_ITEM(a[5], i);
      long long v[4];
      if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 4) Py_RETURN_NONE;
      for (int k = 0; k < 4; ++k)
        if (!integer(PyTuple_GET_ITEM(t, k), &v[k])) Py_RETURN_NONE;
      if (v[3] > MP * PS || v[0] < 0 || v[0] >= B || v[1] < 0 || v[1] >= v[2] || v[2] > NT || v[3] < 1 || v[3] > INT32_MAX)
        Py_RETURN_NONE;
      for (int k = 0; k < 4; ++k) rows[4 * i + k] = (int32_t)v[k];
    }
    const int G = (int)(HQ / KVH);
    const size_t nb = abi.prefill_scratch_bytes(rows.data(), (int)n_rows, (int)NT, (int)KVH, G, (int)D, chunk, signs != nullptr);
    const void* qp = q->data_ptr();
    const int32_t* btp = static_cast<const int32_t*>(bt->data_ptr());
    void *op = out->data_ptr(), *wp = ws ? ws->data_ptr() : nullptr;
    const at::Tensor scratch = at::empty({(int64_t)(nb ? nb : 1)}, q->options().dtype(at::kByte));
    void* sp = scratch.data_ptr();
    void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = abi.prefill(qp, 0, c.part[0], c.part[1], c.part[2], c.part[3], c.strides, (int)PS, btp, (int)B, (int)MP,
                     rows.data(), (int)n_rows, (int)NT, (int)KVH, G, (int)D, (float)s1, (float)s2, signs, k8, chunk, sp, nb, op,
                     out_f32, wp, st);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
  } catch (...) {
    Py_RETURN_NONE;
  }
}

// bind(addresses of the entry points in the order of Abi)
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long p[8];
  if (!PyArg_ParseTuple(args, "KKKKKKKK", &p[0], &p[1], &p[2], &p[3], &p[4], &p[5], &p[6], &p[7])) return nullptr;
  abi.write = reinterpret_cast<decltype(abi.write)>(p[0]);
  abi.write_rot = reinterpret_cast<decltype(abi.write_rot)>(p[1]);
  abi.write_k8 = reinterpret_cast<decltype(abi.write_k8)>(p[2]);
  abi.decode = reinterpret_cast<decltype(abi.decode)>(p[3]);
  abi.decode_rot = reinterpret_cast<decltype(abi.decode_rot)>(p[4]);
  abi.decode_k8 = reinterpret_cast<decltype(abi.decode_k8)>(p[5]);
  abi.prefill_scratch_bytes = reinterpret_cast<decltype(abi.prefill_scratch_bytes)>(p[6]);
  abi.prefill = reinterpret_cast<decltype(abi.prefill)>(p[7]);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, "hands over the addresses of the C entry points"},
    {"write", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(write)), METH_FASTCALL, "status, or None: not the plain form"},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(decode)), METH_FASTCALL, "status, or None: not the plain form"},
    {"layer_write", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer_write)), METH_FASTCALL, "status, or None: not the plain form"},
    {"layer_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer_decode)), METH_FASTCALL, "status, or None: not the plain form"},
    {"prefill", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(prefill)), METH_FASTCALL, "status, or None: not the plain form"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "hkv_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hkv_host(void) {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "torch_version", HKV_TORCH_VERSION) != 0) {   // the torch it is compiled against
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
