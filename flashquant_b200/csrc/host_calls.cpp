// Extension module `_host`: the host side of the package's calls for arguments that need no
// conversion.
//
// A call through ctypes costs about 20 us of interpreter time (a dozen tensor look-ups, twenty
// boxed arguments, the stream object) in front of a launch of 2-4 us, more than the GPU needs for a small
// decode step.  Here the tensors are looked at in C++ and the C ABI is called directly
// (1 x 900-token decode step, append and decode: host time 42 -> 9 us).  Every function returns
// None when an argument is not exactly what the kernels take (another type, device, layout or
// a wrong shape): the caller in kernels.py then converts it or raises.  A failing native call
// returns its status as an int.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAFunctions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "flashquant_b200.h"

namespace {

using at::Tensor;
using Args = PyObject* const*;

// A tensor argument as the kernels take it: on `dev`, contiguous.  Null if it is anything else.
const Tensor* raw_tensor(PyObject* o) {
  return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}
// Device of the call: that of its first tensor, if that is the current device; else -1.
int call_device(PyObject* o) {
  const Tensor* t = raw_tensor(o);
  if (!t || !t->is_cuda()) return -1;
  const int dev = t->get_device();
  return dev == c10::cuda::current_device() ? dev : -1;
}
const Tensor* on_device(PyObject* o, int dev) {
  const Tensor* t = raw_tensor(o);
  return t && t->is_cuda() && t->get_device() == dev ? t : nullptr;
}
const Tensor* dense(PyObject* o, int dev) {
  const Tensor* t = on_device(o, dev);
  return t && t->is_contiguous() ? t : nullptr;
}
const Tensor* dense(PyObject* o, int dev, at::ScalarType st) {
  const Tensor* t = dense(o, dev);
  return t && t->scalar_type() == st ? t : nullptr;
}
const Tensor* f32(PyObject* o, int dev) { return dense(o, dev, at::kFloat); }

// -1: not a type the kernels read
int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return FQ_F32;
    case at::kHalf: return FQ_F16;
    case at::kBFloat16: return FQ_BF16;
    default: return -1;
  }
}
fq_stream_t stream_of(int dev) {
  return reinterpret_cast<fq_stream_t>(at::cuda::getCurrentCUDAStream(dev).stream());
}
PyObject* none() { Py_RETURN_NONE; }
PyObject* done(int rc, const Tensor& out) {
  return rc == FQ_OK ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
}
PyObject* done(int rc) { return PyLong_FromLong(rc); }

bool as_int(PyObject* o, int64_t& v) {
  if (!PyLong_Check(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return v >= INT32_MIN && v <= INT32_MAX;
}
// None: 1 / sqrt(head_dim)
bool as_scale(PyObject* o, int64_t head_dim, float& v) {
  if (o == Py_None) {
    v = float(1.0 / std::sqrt(double(head_dim)));
    return head_dim > 0;
  }
  if (!PyFloat_Check(o)) return false;
  v = float(PyFloat_AS_DOUBLE(o));
  return true;
}
template <typename T = float>
T* data(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }

// ------------------------------------------------------------------------------------
// Workspaces: one per (device, stream, use), zero at first use, grown on demand.  Calls on
// different streams may overlap on the GPU and must not share counters or partial rows.  None is given
// back: a call recorded in a CUDA graph keeps the address, so a workspace that was outgrown stays too
// (each is at least twice its predecessor, all of them together less than twice the last).
// ------------------------------------------------------------------------------------
struct Workspace {
  std::vector<Tensor> kept;  // the last one is in use
  std::mutex calls;          // held while a call that uses it is enqueued
};
std::mutex g_ws_mutex;
std::map<std::tuple<int, const void*, int>, Workspace>& workspaces() {
  static auto* m = new std::map<std::tuple<int, const void*, int>, Workspace>();
  return *m;  // never destroyed: the CUDA context may be gone at exit
}
// `calls`: receives the lock of the workspace's calls
Tensor workspace(int dev, int use, size_t bytes, std::mutex** calls = nullptr) {
  const auto key = std::make_tuple(dev, static_cast<const void*>(stream_of(dev)), use);
  size_t have = size_t(1) << 19;
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    Workspace& w = workspaces()[key];
    if (calls) *calls = &w.calls;
    if (!w.kept.empty()) {
      have = size_t(w.kept.back().numel());
      if (have >= bytes) return w.kept.back();
    }
  }
  // (not under the lock: an allocation may run Python code, which may pass the interpreter on)
  Tensor t = at::zeros({int64_t(std::max(bytes, 2 * have))},
                       at::TensorOptions().device(at::kCUDA, dev).dtype(at::kByte));
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  auto& kept = workspaces()[key].kept;
  if (kept.empty() || size_t(kept.back().numel()) < size_t(t.numel())) kept.push_back(t);
  return kept.back();
}
// The native call without the interpreter lock (a full launch queue makes it wait), and alone among the
// calls that use the same workspace: it may be several launches.
struct WithoutInterpreter {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutInterpreter() { PyEval_RestoreThread(state); }
};
template <typename F>
int native(std::mutex* calls, F call) {
  WithoutInterpreter released;
  std::unique_lock<std::mutex> lock;
  if (calls) lock = std::unique_lock<std::mutex>(*calls);
  return call();
}
enum { kDecode = 0, kAttention = 1 };

// Bytes for one call: what a call writes and reads back within itself is not shared with another one.
Tensor call_bytes(int dev, size_t bytes, bool zero) {
  const auto options = at::TensorOptions().device(at::kCUDA, dev).dtype(at::kByte);
  return zero ? at::zeros({int64_t(bytes)}, options) : at::empty({int64_t(bytes)}, options);
}

// (device_index, use) -> the workspaces of all streams
PyObject* py_workspaces(PyObject*, Args a, Py_ssize_t n) {
  int64_t dev, use;
  if (n != 2 || !as_int(a[0], dev) || !as_int(a[1], use)) {
    PyErr_SetString(PyExc_TypeError, "workspaces(device_index, use)");
    return nullptr;
  }
  std::vector<Tensor> found;
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    for (const auto& [key, w] : workspaces())
      if (std::get<0>(key) == dev && std::get<2>(key) == use)
        found.insert(found.end(), w.kept.begin(), w.kept.end());
  }
  PyObject* list = PyList_New(0);
  for (const Tensor& t : found) {
    PyObject* o = list ? THPVariable_Wrap(t) : nullptr;
    if (!o || PyList_Append(list, o)) Py_CLEAR(list);
    Py_XDECREF(o);
  }
  return list;
}

PyObject* py_workspace(PyObject*, Args a, Py_ssize_t n) {
  int64_t dev, use;
  if (n != 3 || !as_int(a[0], dev) || !as_int(a[1], use) || !PyLong_Check(a[2])) {
    PyErr_SetString(PyExc_TypeError, "workspace(device_index, use, bytes)");
    return nullptr;
  }
  try {
    return THPVariable_Wrap(workspace(int(dev), int(use), PyLong_AsSize_t(a[2])));
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// ------------------------------------------------------------------------------------
// compress-on-append
// ------------------------------------------------------------------------------------
struct Append {
  const Tensor *key, *value, *cache, *slots;
  int dt, h, d;
  int64_t n, stride, num_slots;
};
bool append_args(PyObject* k, PyObject* v, PyObject* cache, PyObject* slots, int dev, Append& p) {
  p.key = on_device(k, dev);
  p.value = on_device(v, dev);
  p.cache = dense(cache, dev, at::kByte);
  p.slots = dense(slots, dev);
  if (!p.key || !p.value || !p.cache || !p.slots) return false;
  const Tensor &key = *p.key, &val = *p.value;
  if (key.dim() != 3 || val.sizes() != key.sizes() || val.scalar_type() != key.scalar_type())
    return false;
  p.dt = dtype_code(key);
  p.n = key.size(0);
  p.h = int(key.size(1));
  p.d = int(key.size(2));
  p.stride = key.stride(0);
  if (p.dt < 0 || key.stride(2) != 1 || key.stride(1) != p.d || p.stride % 4 != 0 ||
      val.stride(2) != 1 || val.stride(1) != p.d || val.stride(0) != p.stride)
    return false;
  if (p.cache->dim() != 3 || p.cache->size(2) != int64_t(p.h) * (p.d + 8)) return false;
  const auto st = p.slots->scalar_type();
  if (st != at::kLong && st != at::kInt) return false;
  p.num_slots = p.cache->size(0) * p.cache->size(1);
  return true;
}

// (key, value, kv_cache, slot_mapping, rotation, boundaries_k, boundaries_v or None)
PyObject* compress_append(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 7 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  Append p;
  const Tensor *rot = f32(a[4], dev), *bk = f32(a[5], dev);
  const Tensor* bv = a[6] == Py_None ? bk : f32(a[6], dev);
  if (!rot || !bk || !bv || !append_args(a[0], a[1], a[2], a[3], dev, p)) return none();
  return done(native(nullptr, [&] {
    return fq_tq4_compress_append(
      p.key->data_ptr(), p.value->data_ptr(), fq_dtype(p.dt), p.n, p.h, p.d, p.stride, data(*rot),
      data(*bk), int(bk->numel()), data(*bv), int(bv->numel()), data<uint8_t>(*p.cache),
      p.num_slots, p.slots->data_ptr(), p.slots->scalar_type() == at::kLong, stream_of(dev));
  }));
}

// (key, value, kv_cache, kq_cache, slot_mapping, rotation, boundaries_k, centroids_k,
//  boundaries_v, qjl_matrix)
PyObject* compress_append_qjl(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 10 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  Append p;
  const Tensor* plane = dense(a[3], dev, at::kByte);
  const Tensor *rot = f32(a[5], dev), *bk = f32(a[6], dev), *ck = f32(a[7], dev),
               *bv = f32(a[8], dev), *s = f32(a[9], dev);
  if (!plane || !rot || !bk || !ck || !bv || !s || !append_args(a[0], a[1], a[2], a[4], dev, p))
    return none();
  if (plane->dim() != 3 || plane->size(2) != int64_t(p.h) * (p.d / 8 + 4) ||
      plane->size(0) * plane->size(1) != p.num_slots || s->dim() != 2 || s->size(0) != p.d ||
      s->size(1) != p.d || ck->numel() != bk->numel() + 1)
    return none();
  return done(native(nullptr, [&] {
    return fq_tq4_compress_append_qjl(
      p.key->data_ptr(), p.value->data_ptr(), fq_dtype(p.dt), p.n, p.h, p.d, p.stride, data(*rot),
      data(*bk), int(bk->numel()), data(*ck), data(*bv), int(bv->numel()), data(*s),
      data<uint8_t>(*p.cache), data<uint8_t>(*plane), p.num_slots, p.slots->data_ptr(),
      p.slots->scalar_type() == at::kLong, stream_of(dev));
  }));
}

// ------------------------------------------------------------------------------------
// paged decode
// ------------------------------------------------------------------------------------
struct Decode {
  const Tensor *q, *cache, *table, *lens, *ck, *cv, *rot;
  int dt, hq, hkv, d, bs, splits;
  float scale;
};
// q, kv_cache, block_table, seq_lens, centroids_k, centroids_v, rotation, num_kv_heads, head_dim,
// block_size, sm_scale, num_splits; `dims` dimensions of q (the last two: heads, head_dim)
bool decode_args(Args a, PyObject* scale, PyObject* splits, int dev, int dims, Decode& p) {
  p.q = dense(a[0], dev);
  p.cache = dense(a[1], dev, at::kByte);
  p.table = on_device(a[2], dev);
  p.lens = dense(a[3], dev, at::kInt);
  p.ck = f32(a[4], dev);
  p.cv = f32(a[5], dev);
  p.rot = f32(a[6], dev);
  int64_t hkv, d, bs, sp;
  if (!p.q || !p.cache || !p.table || !p.lens || !p.ck || !p.cv || !p.rot || !as_int(a[7], hkv) ||
      !as_int(a[8], d) || !as_int(a[9], bs) || !as_int(splits, sp) || !as_scale(scale, d, p.scale))
    return false;
  p.dt = dtype_code(*p.q);
  if (p.dt < 0 || p.q->dim() != dims || p.q->size(dims - 1) != d) return false;
  if (p.table->dim() != 2 || p.table->scalar_type() != at::kInt || p.table->stride(1) != 1)
    return false;
  if (p.cache->dim() != 3 || p.cache->size(1) != bs || p.cache->size(2) != hkv * (d + 8))
    return false;
  p.hq = int(p.q->size(dims - 2));
  p.hkv = int(hkv);
  p.d = int(d);
  p.bs = int(bs);
  p.splits = int(sp);
  return true;
}
// `out` argument: None makes a new tensor like q
bool decode_out(PyObject* o, const Tensor& q, int dev, Tensor& out) {
  if (o == Py_None) {
    out = at::empty(q.sizes(), q.options());
    return true;
  }
  const Tensor* t = dense(o, dev, q.scalar_type());
  if (!t || t->sizes() != q.sizes()) return false;
  out = *t;
  return true;
}

// (q, kv_cache, block_table, seq_lens, centroids_k, centroids_v, rotation, num_kv_heads, head_dim,
//  block_size, sm_scale, out, num_splits)
PyObject* paged_decode(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 13 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  Decode p;
  Tensor out;
  if (!decode_args(a, a[10], a[12], dev, 3, p) || !decode_out(a[11], *p.q, dev, out)) return none();
  const int seqs = int(p.q->size(0));
  std::mutex* calls;
  Tensor ws = workspace(dev, kDecode,
                        fq_paged_decode_workspace_bytes(seqs, p.hq, p.hkv, p.d, p.splits), &calls);
  return done(native(calls, [&] {
    return fq_split_k_paged_decode(
                  p.q->data_ptr(), fq_dtype(p.dt), data<uint8_t>(*p.cache), data<int32_t>(*p.table),
                  p.table->stride(0), data<int32_t>(*p.lens), data(*p.ck), int(p.ck->numel()),
                  data(*p.cv), int(p.cv->numel()), data(*p.rot), seqs, p.hq, p.hkv, p.d, p.bs,
                  p.cache->size(0), p.scale, out.data_ptr(), p.splits, ws.data_ptr(),
                  size_t(ws.numel()), stream_of(dev));
  }),
              out);
}

// (..., sm_scale, out, num_splits, kq_cache, qjl_matrix)
PyObject* paged_decode_qjl(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 15 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  Decode p;
  Tensor out;
  const Tensor *plane = dense(a[13], dev, at::kByte), *s = f32(a[14], dev);
  if (!plane || !s || !decode_args(a, a[10], a[12], dev, 3, p) ||
      !decode_out(a[11], *p.q, dev, out))
    return none();
  if (plane->dim() != 3 || plane->size(0) != p.cache->size(0) || plane->size(1) != p.bs ||
      plane->size(2) != int64_t(p.hkv) * (p.d / 8 + 4) || s->dim() != 2 || s->size(0) != p.d ||
      s->size(1) != p.d)
    return none();
  const int seqs = int(p.q->size(0));
  std::mutex* calls;
  Tensor ws = workspace(dev, kDecode,
                        fq_paged_decode_workspace_bytes(seqs, p.hq, p.hkv, p.d, p.splits), &calls);
  return done(native(calls, [&] {
    return fq_split_k_paged_decode_qjl(
                  p.q->data_ptr(), fq_dtype(p.dt), data<uint8_t>(*p.cache), data<uint8_t>(*plane),
                  data<int32_t>(*p.table), p.table->stride(0), data<int32_t>(*p.lens), data(*p.ck),
                  int(p.ck->numel()), data(*p.cv), int(p.cv->numel()), data(*p.rot), data(*s), seqs,
                  p.hq, p.hkv, p.d, p.bs, p.cache->size(0), p.scale, out.data_ptr(), p.splits,
                  ws.data_ptr(), size_t(ws.numel()), stream_of(dev));
  }),
              out);
}

// (q (num_seqs, n_q, H, D), ..., sm_scale, num_splits)
PyObject* paged_decode_multi(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 12 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  Decode p;
  if (!decode_args(a, a[10], a[11], dev, 4, p)) return none();
  const int seqs = int(p.q->size(0)), n_q = int(p.q->size(1));
  if (seqs == 0 || n_q == 0) return none();
  Tensor out = at::empty(p.q->sizes(), p.q->options());
  const int max_blocks = int(p.table->size(1));
  std::mutex* calls;
  Tensor ws = workspace(dev, kDecode,
                        std::max(fq_split_k_paged_decode_multi_workspace_bytes(
                                     seqs, n_q, p.hq, p.hkv, p.d, p.splits),
                                 fq_paged_decode_workspace_bytes(seqs * n_q, p.hq, p.hkv, p.d,
                                                                 p.splits)),
                        &calls);
  Tensor scratch = call_bytes(
      dev, std::max<size_t>(fq_split_k_paged_decode_multi_scratch_bytes(seqs, n_q, max_blocks), 16),
      false);
  return done(native(calls, [&] {
    return fq_split_k_paged_decode_multi(
                  p.q->data_ptr(), fq_dtype(p.dt), data<uint8_t>(*p.cache), data<int32_t>(*p.table),
                  p.table->stride(0), max_blocks, data<int32_t>(*p.lens), data(*p.ck),
                  int(p.ck->numel()), data(*p.cv), int(p.cv->numel()), data(*p.rot), seqs, n_q,
                  p.hq, p.hkv, p.d, p.bs, p.cache->size(0), p.scale, out.data_ptr(), p.splits,
                  ws.data_ptr(), size_t(ws.numel()), scratch.data_ptr(), size_t(scratch.numel()),
                  stream_of(dev));
  }),
              out);
}

// (q, kv_cache, block_table, seq_lens, centroids_k, centroids_v, rotation, num_kv_heads, head_dim,
//  block_size, sm_scale, out, cu_seqlens_q, max_q_len)
PyObject* paged_prefill(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 14 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  Decode p;
  Tensor out;
  int64_t max_q;
  static PyObject* zero = PyLong_FromLong(0);
  const Tensor* cu = dense(a[12], dev, at::kInt);
  if (!cu || !as_int(a[13], max_q) || !decode_args(a, a[10], zero, dev, 3, p) ||
      !decode_out(a[11], *p.q, dev, out) || cu->numel() != p.lens->numel() + 1)
    return none();
  const int total = int(p.q->size(0));
  Tensor ws = call_bytes(dev, fq_paged_tq4_prefill_workspace_bytes(total, p.hq, p.d), true);
  return done(native(nullptr, [&] {
    return fq_paged_tq4_prefill(
                  p.q->data_ptr(), fq_dtype(p.dt), data<uint8_t>(*p.cache), data<int32_t>(*p.table),
                  p.table->stride(0), data<int32_t>(*p.lens), data<int32_t>(*cu), data(*p.ck),
                  int(p.ck->numel()), data(*p.cv), int(p.cv->numel()), data(*p.rot),
                  int(p.lens->numel()), total, int(max_q), p.hq, p.hkv, p.d, p.bs,
                  p.cache->size(0), p.scale, out.data_ptr(), ws.data_ptr(), size_t(ws.numel()),
                  stream_of(dev));
  }),
              out);
}

// ------------------------------------------------------------------------------------
// contiguous form
// ------------------------------------------------------------------------------------
// (x (N, H, D), rotation_T_even, rotation_T_odd, boundaries) -> (packed, norms)
PyObject* compress(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 4 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  const Tensor *x = dense(a[0], dev), *even = f32(a[1], dev), *odd = f32(a[2], dev),
               *bnd = f32(a[3], dev);
  if (!x || !even || !odd || !bnd || x->dim() != 3 || dtype_code(*x) < 0) return none();
  const int64_t nt = x->size(0), h = x->size(1), d = x->size(2);
  Tensor packed = at::empty({nt, h, d / 2}, x->options().dtype(at::kByte));
  Tensor norms = at::empty({nt, h, 1}, x->options().dtype(at::kFloat));
  const int rc = native(nullptr, [&] {
    return fq_tq4_compress(x->data_ptr(), fq_dtype(dtype_code(*x)), data(*even), data(*odd),
                                 data(*bnd), int(bnd->numel()), data<uint8_t>(packed), data(norms),
                                 nt * h, int(d), stream_of(dev));
  });
  if (rc != FQ_OK) return done(rc);
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(packed));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(norms));
  return t;
}

// Tokens between the (batch, head) rows of the buffers that codes and norms are [:, :, :n] views
// of (n where there is one row); 0 if they are not.  Strides of dimensions of size one say nothing.
int64_t view_capacity(const Tensor& codes, const Tensor& norms) {
  const int64_t b = codes.size(0), h = codes.size(1), n = codes.size(2), half = codes.size(3);
  if (n == 0 || half == 0 || norms.dim() != 4 || norms.size(0) != b || norms.size(1) != h ||
      norms.size(2) != n || norms.size(3) != 1)
    return 0;
  const int64_t cap = b * h == 1 ? n : codes.stride(h > 1 ? 1 : 0) / half;
  const auto laid_out = [&](const Tensor& t, int64_t unit) {
    const int64_t want[4] = {h * cap * unit, cap * unit, unit, 1};
    for (int i = 0; i < 4; ++i)
      if (t.size(i) > 1 && t.stride(i) != want[i]) return false;
    return true;
  };
  return cap >= n && laid_out(codes, half) && laid_out(norms, 1) ? cap : 0;
}

// (q, k_packed, k_norms, v_packed, v_norms, centroids_k, centroids_v, rotation_k, rotation_v,
//  sm_scale, is_causal)
PyObject* attention(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 11 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  const Tensor* q = dense(a[0], dev);
  const Tensor* kv[4];
  for (int i = 0; i < 4; ++i) {
    kv[i] = on_device(a[1 + i], dev);
    if (!kv[i] || kv[i]->dim() != 4 || kv[i]->scalar_type() != (i & 1 ? at::kFloat : at::kByte))
      return none();
  }
  const Tensor *ck = f32(a[5], dev), *cv = f32(a[6], dev), *rk = f32(a[7], dev), *rv = f32(a[8], dev);
  float scale;
  if (!q || q->dim() != 4 || dtype_code(*q) < 0 || !ck || !cv || !rk || !rv ||
      !as_scale(a[9], q->size(3), scale) || !PyBool_Check(a[10]))
    return none();
  const int b = int(q->size(0)), hq = int(q->size(1)), nq = int(q->size(2)), d = int(q->size(3));
  const int hkv = int(kv[0]->size(1)), nkv = int(kv[0]->size(2));
  if (kv[0]->size(0) != b || kv[0]->size(3) * 2 != d || kv[2]->sizes() != kv[0]->sizes())
    return none();
  const int64_t cap = view_capacity(*kv[0], *kv[1]);
  if (cap == 0 || view_capacity(*kv[2], *kv[3]) != cap) return none();
  Tensor out = at::empty(q->sizes(), q->options());
  std::mutex* calls;
  Tensor ws = workspace(dev, kAttention, fq_fused_tq_attention_workspace_bytes(b, hq, nq, d), &calls);
  return done(native(calls, [&] {
    return fq_fused_tq_attention_kv(
                  q->data_ptr(), fq_dtype(dtype_code(*q)), data<uint8_t>(*kv[0]), data(*kv[1]),
                  data<uint8_t>(*kv[2]), data(*kv[3]), data(*ck), int(ck->numel()), data(*cv),
                  int(cv->numel()), data(*rk), data(*rv), b, hq, hkv, nq, nkv, cap, d, scale,
                  a[10] == Py_True, out.data_ptr(), ws.data_ptr(), size_t(ws.numel()),
                  stream_of(dev));
  }),
              out);
}

// (key, value, tables_k, tables_v, k_packed, k_norms, v_packed, v_norms, position, k_out, v_out,
//  out_position, workspace)
PyObject* cache_update(PyObject*, Args a, Py_ssize_t n) {
  const int dev = n == 13 ? call_device(a[0]) : -1;
  if (dev < 0) return none();
  const Tensor *key = dense(a[0], dev), *val = dense(a[1], dev);
  if (!key || !val || key->dim() != 4 || dtype_code(*key) < 0 || val->sizes() != key->sizes() ||
      val->scalar_type() != key->scalar_type() || !PyTuple_Check(a[2]) || !PyTuple_Check(a[3]) ||
      PyTuple_GET_SIZE(a[2]) != 5 || PyTuple_GET_SIZE(a[3]) != 5)
    return none();
  const Tensor *tk[5], *tv[5];  // Pi^T even, Pi^T odd, boundaries, centroids, Pi
  for (int i = 0; i < 5; ++i) {
    tk[i] = f32(PyTuple_GET_ITEM(a[2], i), dev);
    tv[i] = f32(PyTuple_GET_ITEM(a[3], i), dev);
    if (!tk[i] || !tv[i]) return none();
  }
  const int64_t b = key->size(0), h = key->size(1), s = key->size(2), d = key->size(3);
  const Tensor* buf[4];
  for (int i = 0; i < 4; ++i) {
    buf[i] = dense(a[4 + i], dev, i & 1 ? at::kFloat : at::kByte);
    if (!buf[i] || buf[i]->dim() != 4) return none();
    const int64_t cap = buf[0]->size(2);
    if (buf[i]->size(0) != b || buf[i]->size(1) != h || buf[i]->size(2) != cap ||
        buf[i]->size(3) != (i & 1 ? 1 : d / 2))
      return none();
  }
  int64_t at, out_at;
  if (!as_int(a[8], at) || !as_int(a[11], out_at)) return none();
  const Tensor *ko = nullptr, *vo = nullptr, *ws = nullptr;
  int64_t out_cap = 0;
  size_t need = 0;
  if (a[9] != Py_None) {
    ko = dense(a[9], dev, key->scalar_type());
    vo = dense(a[10], dev, key->scalar_type());
    if (!ko || !vo || ko->dim() != 4 || ko->sizes() != vo->sizes() || ko->size(0) != b ||
        ko->size(1) != h || ko->size(3) != d)
      return none();
    out_cap = ko->size(2);
    need = fq_cache_update_workspace_bytes(b * h, s, int(d));
    if (need) {
      ws = dense(a[12], dev, at::kByte);
      if (!ws || size_t(ws->numel()) < need) return none();
    }
  } else if (a[10] != Py_None) {
    return none();
  }
  return done(native(nullptr, [&] {
    return fq_cache_update(
      key->data_ptr(), val->data_ptr(), fq_dtype(dtype_code(*key)), data(*tk[0]), data(*tk[1]),
      data(*tk[4]), data(*tv[0]), data(*tv[1]), data(*tv[4]), data(*tk[2]), int(tk[2]->numel()),
      data(*tk[3]), int(tk[3]->numel()), data<uint8_t>(*buf[0]), data(*buf[1]),
      data<uint8_t>(*buf[2]), data(*buf[3]), b * h, s, buf[0]->size(2), at,
      ko ? ko->data_ptr() : nullptr, vo ? vo->data_ptr() : nullptr, out_cap, out_at, int(d),
      ws ? ws->data_ptr() : nullptr, need, stream_of(dev));
  }));
}

// C++ exceptions (an allocation that fails) become Python ones
PyObject* g_oom = nullptr;  // torch.OutOfMemoryError
template <PyObject* (*F)(PyObject*, Args, Py_ssize_t)>
PyObject* guarded(PyObject* self, Args a, Py_ssize_t n) {
  try {
    return F(self, a, n);
  } catch (const c10::OutOfMemoryError& e) {
    PyErr_SetString(g_oom ? g_oom : PyExc_MemoryError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

#define FQ_METHOD(f) \
  { #f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<f>)), METH_FASTCALL, nullptr }
PyMethodDef kMethods[] = {
    FQ_METHOD(compress_append), FQ_METHOD(compress_append_qjl), FQ_METHOD(paged_decode),
    FQ_METHOD(paged_decode_qjl), FQ_METHOD(paged_decode_multi), FQ_METHOD(paged_prefill),
    FQ_METHOD(compress), FQ_METHOD(attention), FQ_METHOD(cache_update),
    {"workspaces", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&py_workspaces)),
     METH_FASTCALL, nullptr},
    {"workspace", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&py_workspace)),
     METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host",
                       "host side of the package's calls for arguments that need no conversion",
                       -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  if (PyObject* torch = PyImport_ImportModule("torch")) {
    g_oom = PyObject_GetAttrString(torch, "OutOfMemoryError");
    Py_DECREF(torch);
  }
  if (PyErr_Occurred()) return nullptr;
  return PyModule_Create(&kModule);
}
