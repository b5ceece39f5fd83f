// Host side of the operators: argument checks, scratch lookup, output allocation and the call into
// the C ABI, as a CPython module over torch's tensors.
//
// A decode step of a small model is a chain of calls whose kernels take 2 to 15 us each; done in
// Python (tensor attribute reads, ctypes conversion of 20 arguments, context managers) the host
// side of one layer took 40 us and of a step's index arrays 62 to 97 us, i.e. such a step was bound
// by the host.  Here a call costs its launch and one allocation.
//
// Contract with the Python wrappers: a call whose arguments are not what the operator takes, or
// whose tensors live on a device that is not current, returns None and launches nothing; the
// wrapper then names the fault (or makes the device current and calls again).  An error of the C
// ABI is raised as RuntimeError with the library's message, and what C++ throws as the exception that
// torch raises for it (see `guarded`).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <algorithm>
#include <cmath>
#include <deque>
#include <mutex>
#include <string>

#include "../../include/msgl_b200.h"

namespace {

using at::Tensor;

// ------------------------------------------------------------------ scratch
// Address and size of the scratch of a stream's operators, as the Python side made it; asked for again
// (which grows it) when a call needs more.
enum Kind { kDecode = 0, kPrefill = 1 };
const char* const kKindNames[] = {"decode", "prefill"};

struct StreamScratch {
  int device;
  int64_t stream;
  // Held while a call queues its launches.  An attention call can be several of them that hand data over
  // through the scratch (slot ids or counters written in front, partials merged behind), and other Python
  // threads run while it queues them: two calls in turn keep each its own.
  std::mutex launches;
  void* ptr[2] = {};
  size_t bytes[2] = {};
  StreamScratch(int d, int64_t s) : device(d), stream(s) {}
};
// guarded by the GIL, but for `launches`; entries keep their place and are never destroyed (a thread may hold one at exit)
std::deque<StreamScratch>& g_scratch = *new std::deque<StreamScratch>;
PyObject* g_make_workspace = nullptr;  // Python: (nbytes, device index, stream handle, kind) -> tensor
PyObject* g_make_pages = nullptr;      // Python: (nbytes, device index, stream handle) -> tensor or None

// The scratch a call got: it stays valid when the stream's scratch grows meanwhile (the Python side keeps
// outgrown buffers).
struct Scratch {
  StreamScratch* of;
  void* ptr;
  size_t bytes;
};

bool scratch_for(int device, int64_t stream, int kind, size_t need, Scratch* out) {
  StreamScratch* found = nullptr;
  for (StreamScratch& s : g_scratch)
    if (s.stream == stream && s.device == device) {
      found = &s;
      break;
    }
  if (found == nullptr) found = &g_scratch.emplace_back(device, stream);
  if (found->bytes[kind] < need) {
    THPObjectPtr t(PyObject_CallFunction(g_make_workspace, "niLs", static_cast<Py_ssize_t>(need), device,
                                         static_cast<long long>(stream), kKindNames[kind]));
    if (!t) return false;
    const Tensor& ws = THPVariable_Unpack(t.get());
    found->ptr[kind] = ws.data_ptr();
    found->bytes[kind] = static_cast<size_t>(ws.numel());
  }
  *out = Scratch{found, found->ptr[kind], found->bytes[kind]};
  return true;
}

// Memory of one call for the pages of its K/V rows, asked for after the call's output and given back when the call
// has queued its launches.  Without it (no memory, or none made) the attention kernel gathers the rows itself.
struct Pages {
  THPObjectPtr tensor;
  void* ptr = nullptr;
  size_t bytes = 0;
};
bool pages_for(int device, int64_t stream, size_t bytes, Pages* out) {
  if (bytes == 0 || g_make_pages == nullptr) return true;
  out->tensor = PyObject_CallFunction(g_make_pages, "niL", static_cast<Py_ssize_t>(bytes), device,
                                      static_cast<long long>(stream));
  if (!out->tensor) return false;
  if (out->tensor.get() == Py_None) return true;
  const Tensor& t = THPVariable_Unpack(out->tensor.get());
  out->ptr = t.data_ptr();
  out->bytes = static_cast<size_t>(t.numel());
  return true;
}

// ------------------------------------------------------------------ arguments
int dtype_code(const Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? 0 : t.scalar_type() == at::kHalf ? 1 : -1;
}

inline bool is_tensor(PyObject* o) { return THPVariable_Check(o); }

inline bool index_ok(const Tensor& t, const c10::Device& dev) {
  return t.dim() == 1 && t.scalar_type() == at::kInt && t.is_contiguous() && t.device() == dev;
}

const int32_t* i32(const Tensor& t) { return static_cast<const int32_t*>(t.data_ptr()); }

// A call of the C ABI without the GIL: a launch waits when the stream's queue is full.  (Its error
// message is per thread.)  The GIL is taken back however the call ends.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
template <typename F>
int unlocked(F&& call) {
  NoGil no_gil;
  return call();
}
// The same for a call whose launches share scratch: calls on one stream take turns.  (Waited for without the
// GIL, which the thread whose turn it is wants back at its end.)
template <typename F>
int in_turn(const Scratch& ws, F&& call) {
  NoGil no_gil;
  std::lock_guard<std::mutex> turn(ws.of->launches);
  return call();
}

// The form in which a function of this module is handed to Python: torch turns what it throws into the
// Python exception.  Above all an allocation that finds no memory is torch.OutOfMemoryError, which a
// serving loop answers by giving cache back and calling again: every function allocates before its first
// launch, so the call that failed has changed nothing.  (Left alone, a C++ exception that leaves a
// CPython function ends the process.)
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}

PyObject* raise_status(int rc) {
  PyErr_Format(PyExc_RuntimeError, "%s [msgl status %d]", msgl_last_error_string(), rc);
  return nullptr;
}

// Stream handle: None = torch's current stream of the device.
bool stream_of(PyObject* o, int device, int64_t* out) {
  if (o == Py_None) {
    *out = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream());
    return true;
  }
  *out = PyLong_AsLongLong(o);
  return !(*out == -1 && PyErr_Occurred());
}

// What the attention operators' q and pools must be; fills the sizes.
struct Shapes {
  int n, hq, hkv, d, dtype, device;
  int64_t num_slots;
};
bool attention_shapes(const Tensor& q, const Tensor& kc, const Tensor& vc, Shapes* s) {
  if (q.dim() != 3 || kc.dim() != 3 || vc.dim() != 3 || !q.is_cuda()) return false;
  s->dtype = dtype_code(q);
  if (s->dtype < 0 || kc.scalar_type() != q.scalar_type() || vc.scalar_type() != q.scalar_type()) return false;
  const c10::Device dev = q.device();
  if (kc.device() != dev || vc.device() != dev || !q.is_contiguous() || !kc.is_contiguous() ||
      !vc.is_contiguous() || kc.sizes() != vc.sizes() || kc.size(2) != q.size(2))
    return false;
  s->n = static_cast<int>(q.size(0));
  s->hq = static_cast<int>(q.size(1));
  s->d = static_cast<int>(q.size(2));
  s->num_slots = kc.size(0);
  s->hkv = static_cast<int>(kc.size(1));
  s->device = dev.index();
  return c10::cuda::current_device() == s->device;
}

// gate: None or a tensor like q
bool gate_ptr(PyObject* o, const Tensor& q, const void** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  if (!is_tensor(o)) return false;
  const Tensor& g = THPVariable_Unpack(o);
  if (g.sizes() != q.sizes() || g.scalar_type() != q.scalar_type() || g.device() != q.device() ||
      !g.is_contiguous())
    return false;
  *out = g.data_ptr();
  return true;
}

// An output like q (below autograd's dispatch layers: nothing here is differentiable).
Tensor empty_like_rows(const Tensor& q) {
  at::AutoDispatchBelowADInplaceOrView below;
  return at::empty(q.sizes(), at::TensorOptions().dtype(q.scalar_type()).device(q.device()));
}

#define ALL_TENSORS(args, n)                                   \
  do {                                                         \
    for (int i_ = 0; i_ < (n); ++i_)                           \
      if (!is_tensor((args)[i_])) Py_RETURN_NONE;              \
  } while (0)
#define ARG_INT(var, o)                                        \
  const long long var = PyLong_AsLongLong(o);                  \
  if (var == -1 && PyErr_Occurred()) return nullptr
#define ARG_FLOAT(var, o)                                      \
  const double var = PyFloat_AsDouble(o);                      \
  if (var == -1.0 && PyErr_Occurred()) return nullptr

// ------------------------------------------------------------------ attention operators
// (q, k_cache, v_cache, kv_indptr, kv_indices, num_kv_splits, sm_scale, max_kv_splits, gate, stream)
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10) return PyErr_Format(PyExc_TypeError, "decode takes 10 arguments");
  ALL_TENSORS(a, 6);
  const Tensor &q = THPVariable_Unpack(a[0]), &kc = THPVariable_Unpack(a[1]), &vc = THPVariable_Unpack(a[2]),
               &indptr = THPVariable_Unpack(a[3]), &indices = THPVariable_Unpack(a[4]),
               &splits = THPVariable_Unpack(a[5]);
  Shapes s;
  const void* gate;
  if (!attention_shapes(q, kc, vc, &s) || !index_ok(indptr, q.device()) || !index_ok(indices, q.device()) ||
      !index_ok(splits, q.device()) || indptr.numel() != s.n + 1 || splits.numel() != s.n ||
      !gate_ptr(a[8], q, &gate))
    Py_RETURN_NONE;
  ARG_FLOAT(scale, a[6]);
  ARG_INT(max_splits, a[7]);
  int64_t stream;
  Scratch ws;
  if (!stream_of(a[9], s.device, &stream) ||
      !scratch_for(s.device, stream, kDecode,
                   msgl_decode_workspace_bytes_full(s.n, s.hq, s.hkv, s.d, static_cast<int>(max_splits),
                                                    indices.numel()),
                   &ws))
    return nullptr;
  Tensor out = empty_like_rows(q);
  const int rc = in_turn(ws, [&] {
    return msgl_paged_decode_attention_sized(
      q.data_ptr(), kc.data_ptr(), vc.data_ptr(), i32(indptr), i32(indices), gate, out.data_ptr(), ws.ptr, ws.bytes,
      s.n, s.hq, s.hkv, s.d, s.num_slots, s.dtype, static_cast<float>(scale), static_cast<int>(max_splits),
      indices.numel(), reinterpret_cast<void*>(stream));
  });
  return rc ? raise_status(rc) : THPVariable_Wrap(std::move(out));
}

// (q, k_cache, v_cache, page_indptr, page_indices, kv_lens, num_kv_splits, sm_scale, max_kv_splits,
//  page_size, gate, stream)
PyObject* decode_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 12) return PyErr_Format(PyExc_TypeError, "decode_paged takes 12 arguments");
  ALL_TENSORS(a, 7);
  const Tensor &q = THPVariable_Unpack(a[0]), &kc = THPVariable_Unpack(a[1]), &vc = THPVariable_Unpack(a[2]),
               &indptr = THPVariable_Unpack(a[3]), &pages = THPVariable_Unpack(a[4]),
               &lens = THPVariable_Unpack(a[5]), &splits = THPVariable_Unpack(a[6]);
  Shapes s;
  const void* gate;
  if (!attention_shapes(q, kc, vc, &s) || !index_ok(indptr, q.device()) || !index_ok(pages, q.device()) ||
      !index_ok(lens, q.device()) || !index_ok(splits, q.device()) || indptr.numel() != s.n + 1 ||
      lens.numel() != s.n || splits.numel() != s.n || !gate_ptr(a[10], q, &gate))
    Py_RETURN_NONE;
  ARG_FLOAT(scale, a[7]);
  ARG_INT(max_splits, a[8]);
  ARG_INT(page_size, a[9]);
  if (page_size <= 0) Py_RETURN_NONE;
  const int64_t total_pages = pages.numel();
  const size_t need =
      (msgl_decode_workspace_bytes_full(s.n, s.hq, s.hkv, s.d, static_cast<int>(max_splits),
                                        total_pages * page_size) + 255) / 256 * 256 +
      msgl_page_index_workspace_bytes(s.n, total_pages, static_cast<int>(page_size));
  int64_t stream;
  Scratch ws;
  if (!stream_of(a[11], s.device, &stream) || !scratch_for(s.device, stream, kDecode, need, &ws))
    return nullptr;
  Tensor out = empty_like_rows(q);
  const int rc = in_turn(ws, [&] {
    return msgl_paged_decode_attention_p16(
      q.data_ptr(), kc.data_ptr(), vc.data_ptr(), i32(indptr), i32(pages), i32(lens), i32(splits), gate,
      out.data_ptr(), ws.ptr, ws.bytes, s.n, s.hq, s.hkv, s.d, s.num_slots, s.dtype, static_cast<float>(scale),
      static_cast<int>(max_splits), static_cast<int>(page_size), total_pages, reinterpret_cast<void*>(stream));
  });
  return rc ? raise_status(rc) : THPVariable_Wrap(std::move(out));
}

// (q, k_cache, v_cache, qo_indptr, kv_indptr, kv_indices, prefix_lens, sm_scale, max_len_extend,
//  is_cross_attention, sliding_window_size, gate, stream)
PyObject* prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 13) return PyErr_Format(PyExc_TypeError, "prefill takes 13 arguments");
  ALL_TENSORS(a, 7);
  const Tensor &q = THPVariable_Unpack(a[0]), &kc = THPVariable_Unpack(a[1]), &vc = THPVariable_Unpack(a[2]),
               &qo = THPVariable_Unpack(a[3]), &indptr = THPVariable_Unpack(a[4]),
               &indices = THPVariable_Unpack(a[5]), &prefix = THPVariable_Unpack(a[6]);
  Shapes s;
  const void* gate;
  if (!attention_shapes(q, kc, vc, &s) || !index_ok(qo, q.device()) || !index_ok(indptr, q.device()) ||
      !index_ok(indices, q.device()) || !index_ok(prefix, q.device()) || qo.numel() < 2 ||
      indptr.numel() != qo.numel() || prefix.numel() + 1 != qo.numel() || !gate_ptr(a[11], q, &gate))
    Py_RETURN_NONE;
  ARG_FLOAT(scale, a[7]);
  ARG_INT(max_ext, a[8]);
  ARG_INT(window, a[10]);
  const int cross = PyObject_IsTrue(a[9]);
  if (cross < 0) return nullptr;
  const int batch = static_cast<int>(prefix.numel());
  const int64_t total_kv = indices.numel();
  int64_t stream;
  Scratch ws;
  Pages pages;
  if (!stream_of(a[12], s.device, &stream) ||
      !scratch_for(s.device, stream, kPrefill,
                   msgl_prefill_workspace_bytes(batch, s.n, total_kv, s.hq, s.hkv, s.d, static_cast<int>(max_ext),
                                                static_cast<int>(window)),
                   &ws))
    return nullptr;
  Tensor out = empty_like_rows(q);
  if (!pages_for(s.device, stream,
                 msgl_prefill_kv_pages_bytes(batch, s.n, total_kv, s.hq, s.hkv, s.d, static_cast<int>(max_ext),
                                             static_cast<int>(window)),
                 &pages))
    return nullptr;
  const int rc = in_turn(ws, [&] {
    return msgl_prefill_layer_pages(
      nullptr, q.data_ptr(), kc.data_ptr(), vc.data_ptr(), i32(qo), i32(indptr), i32(indices), nullptr, i32(prefix),
      gate, out.data_ptr(), ws.ptr, ws.bytes, pages.ptr, pages.bytes, batch, s.n, s.hq, s.hkv, s.d, s.num_slots,
      s.dtype, static_cast<float>(scale), static_cast<int>(max_ext), cross, static_cast<int>(window), 1, total_kv,
      reinterpret_cast<void*>(stream));
  });
  return rc ? raise_status(rc) : THPVariable_Wrap(std::move(out));
}

// (q, k_cache, v_cache, qo_indptr, page_indptr, page_indices, kv_lens, prefix_lens, sm_scale,
//  max_len_extend, page_size, is_cross_attention, sliding_window_size, gate, stream)
PyObject* prefill_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 15) return PyErr_Format(PyExc_TypeError, "prefill_paged takes 15 arguments");
  ALL_TENSORS(a, 8);
  const Tensor &q = THPVariable_Unpack(a[0]), &kc = THPVariable_Unpack(a[1]), &vc = THPVariable_Unpack(a[2]),
               &qo = THPVariable_Unpack(a[3]), &indptr = THPVariable_Unpack(a[4]),
               &pages = THPVariable_Unpack(a[5]), &lens = THPVariable_Unpack(a[6]),
               &prefix = THPVariable_Unpack(a[7]);
  Shapes s;
  const void* gate;
  if (!attention_shapes(q, kc, vc, &s) || !index_ok(qo, q.device()) || !index_ok(indptr, q.device()) ||
      !index_ok(pages, q.device()) || !index_ok(lens, q.device()) || !index_ok(prefix, q.device()) ||
      qo.numel() < 2 || indptr.numel() != qo.numel() || lens.numel() + 1 != qo.numel() ||
      prefix.numel() + 1 != qo.numel() || !gate_ptr(a[13], q, &gate))
    Py_RETURN_NONE;
  ARG_FLOAT(scale, a[8]);
  ARG_INT(max_ext, a[9]);
  ARG_INT(page_size, a[10]);
  ARG_INT(window, a[12]);
  const int cross = PyObject_IsTrue(a[11]);
  if (cross < 0) return nullptr;
  if (page_size <= 0) Py_RETURN_NONE;
  const int batch = static_cast<int>(prefix.numel());
  const int64_t total_pages = pages.numel();
  int64_t stream;
  Scratch ws;
  if (!stream_of(a[14], s.device, &stream) ||
      !scratch_for(s.device, stream, kPrefill,
                   msgl_prefill_workspace_bytes_p16(batch, s.n, total_pages, static_cast<int>(page_size), s.hq,
                                                    s.hkv, s.d, static_cast<int>(max_ext),
                                                    static_cast<int>(window)),
                   &ws))
    return nullptr;
  Tensor out = empty_like_rows(q);
  const int rc = in_turn(ws, [&] {
    return msgl_paged_prefill_attention_p16(
      q.data_ptr(), kc.data_ptr(), vc.data_ptr(), i32(qo), i32(indptr), i32(pages), i32(lens), i32(prefix), gate,
      out.data_ptr(), ws.ptr, ws.bytes, batch, s.n, s.hq, s.hkv, s.d, s.num_slots, s.dtype, static_cast<float>(scale),
      static_cast<int>(max_ext), cross, static_cast<int>(window), static_cast<int>(page_size), total_pages,
      reinterpret_cast<void*>(stream));
  });
  return rc ? raise_status(rc) : THPVariable_Wrap(std::move(out));
}

// ------------------------------------------------------------------ rows into the pool
inline bool rows_dense(const Tensor& t, int64_t d) { return t.stride(2) == 1 && t.stride(1) == d; }

// (k_cache, v_cache, indices, k, v, stream)
PyObject* store_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "store_kv takes 6 arguments");
  ALL_TENSORS(a, 5);
  const Tensor &kc = THPVariable_Unpack(a[0]), &vc = THPVariable_Unpack(a[1]), &idx = THPVariable_Unpack(a[2]),
               &k = THPVariable_Unpack(a[3]), &v = THPVariable_Unpack(a[4]);
  if (kc.dim() != 3 || !kc.is_cuda() || vc.sizes() != kc.sizes() || k.dim() != 3 || v.sizes() != k.sizes())
    Py_RETURN_NONE;
  const c10::Device dev = kc.device();
  const int dt = dtype_code(kc);
  const int64_t hkv = kc.size(1), d = kc.size(2), len = k.size(0);
  if (dt < 0 || d % 4 != 0 || vc.scalar_type() != kc.scalar_type() || k.scalar_type() != kc.scalar_type() ||
      v.scalar_type() != kc.scalar_type() || !index_ok(idx, dev) || idx.numel() != len || k.size(1) != hkv ||
      k.size(2) != d || vc.device() != dev || k.device() != dev || v.device() != dev || !rows_dense(kc, d) ||
      !rows_dense(vc, d) || !rows_dense(k, d) || !rows_dense(v, d) || k.stride(0) != v.stride(0) ||
      kc.stride(0) != vc.stride(0) || c10::cuda::current_device() != dev.index())
    Py_RETURN_NONE;
  int64_t stream;
  Scratch ws;
  if (!stream_of(a[5], dev.index(), &stream) || !scratch_for(dev.index(), stream, kDecode, 256, &ws))
    return nullptr;
  const int rc = unlocked([&] {
    return msgl_store_kv_cache(kc.data_ptr(), vc.data_ptr(), i32(idx), k.data_ptr(), v.data_ptr(),
                                     static_cast<int>(len), static_cast<int>(hkv), static_cast<int>(d), kc.size(0),
                                     kc.stride(0), k.stride(0), dt, ws.ptr, reinterpret_cast<void*>(stream));
  });
  if (rc) return raise_status(rc);
  Py_RETURN_TRUE;
}

// (q, k, v, q_weight, k_weight, positions, out_loc, k_cache, v_cache, rope_base, eps, rotary_dim, stream)
PyObject* qk_norm_rope_store(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 13) return PyErr_Format(PyExc_TypeError, "qk_norm_rope_store takes 13 arguments");
  for (int i = 0; i < 9; ++i)
    if (!is_tensor(a[i]) && !((i == 3 || i == 4) && a[i] == Py_None)) Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]),
               &pos = THPVariable_Unpack(a[5]), &loc = THPVariable_Unpack(a[6]), &kc = THPVariable_Unpack(a[7]),
               &vc = THPVariable_Unpack(a[8]);
  if (q.dim() != 3 || k.dim() != 3 || v.sizes() != k.sizes() || kc.dim() != 3 || vc.sizes() != kc.sizes() ||
      !q.is_cuda())
    Py_RETURN_NONE;
  const c10::Device dev = q.device();
  const int dt = dtype_code(q);
  const int64_t nt = q.size(0), hq = q.size(1), d = q.size(2), hkv = k.size(1);
  if (dt < 0 || k.size(0) != nt || k.size(2) != d || kc.size(1) != hkv || kc.size(2) != d ||
      c10::cuda::current_device() != dev.index())
    Py_RETURN_NONE;
  for (const Tensor* t : {&q, &k, &v, &kc, &vc})
    if (t->scalar_type() != q.scalar_type() || t->device() != dev || !rows_dense(*t, d)) Py_RETURN_NONE;
  if (kc.stride(0) != vc.stride(0) || !index_ok(pos, dev) || !index_ok(loc, dev) || pos.numel() != nt ||
      loc.numel() != nt)
    Py_RETURN_NONE;
  const void* wt[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; ++i) {
    if (a[3 + i] == Py_None) continue;
    const Tensor& w = THPVariable_Unpack(a[3 + i]);
    if (w.scalar_type() != q.scalar_type() || w.device() != dev || w.dim() != 1 || w.size(0) != d ||
        !w.is_contiguous())
      Py_RETURN_NONE;
    wt[i] = w.data_ptr();
  }
  ARG_FLOAT(base, a[9]);
  ARG_FLOAT(eps, a[10]);
  const long long rd = a[11] == Py_None ? d : PyLong_AsLongLong(a[11]);
  if (rd == -1 && PyErr_Occurred()) return nullptr;
  int64_t stream;
  if (!stream_of(a[12], dev.index(), &stream)) return nullptr;
  const int rc = unlocked([&] {
    return msgl_qk_norm_rope_store(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), wt[0], wt[1], i32(pos), i32(loc), kc.data_ptr(), vc.data_ptr(),
      static_cast<int>(nt), static_cast<int>(hq), static_cast<int>(hkv), static_cast<int>(d), static_cast<int>(rd),
      static_cast<float>(base), static_cast<float>(eps), kc.size(0), q.stride(0), k.stride(0), v.stride(0),
      kc.stride(0), dt, reinterpret_cast<void*>(stream));
  });
  if (rc) return raise_status(rc);
  Py_RETURN_TRUE;
}

// ------------------------------------------------------------------ a layer's new tokens, store and attention
// k, v, out_loc and projection (None, or (q_weight, k_weight, positions, rope_base, eps, rotary_dim or
// None)) of a layer call -> *rows.  1: fine, 0: not what the native call takes, -1: a Python error.
int new_rows(PyObject* ko, PyObject* vo, PyObject* loco, PyObject* proj, const Tensor& q, const Shapes& s,
             msgl_new_rows* r) {
  if (!is_tensor(ko) || !is_tensor(vo) || !is_tensor(loco)) return 0;
  const Tensor &k = THPVariable_Unpack(ko), &v = THPVariable_Unpack(vo), &loc = THPVariable_Unpack(loco);
  const c10::Device dev = q.device();
  if (k.dim() != 3 || v.sizes() != k.sizes() || k.size(1) != s.hkv || k.size(2) != s.d ||
      k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type() || k.device() != dev ||
      v.device() != dev || !rows_dense(k, s.d) || !rows_dense(v, s.d) || !index_ok(loc, dev) ||
      loc.numel() != k.size(0))
    return 0;
  *r = msgl_new_rows{};
  r->k = k.data_ptr();
  r->v = v.data_ptr();
  r->out_loc = i32(loc);
  r->n_tokens = static_cast<int>(k.size(0));
  r->k_token_stride = k.stride(0);
  r->v_token_stride = v.stride(0);
  if (proj == Py_None) return r->k_token_stride == r->v_token_stride ? 1 : 0;
  if (!PyTuple_Check(proj) || PyTuple_GET_SIZE(proj) != 6 || k.size(0) != s.n) return 0;
  r->project = 1;
  const void** weights[2] = {&r->q_weight, &r->k_weight};
  for (int i = 0; i < 2; ++i) {
    PyObject* o = PyTuple_GET_ITEM(proj, i);
    if (o == Py_None) continue;
    if (!is_tensor(o)) return 0;
    const Tensor& w = THPVariable_Unpack(o);
    if (w.scalar_type() != q.scalar_type() || w.device() != dev || w.dim() != 1 || w.size(0) != s.d ||
        !w.is_contiguous())
      return 0;
    *weights[i] = w.data_ptr();
  }
  if (!is_tensor(PyTuple_GET_ITEM(proj, 2))) return 0;
  const Tensor& pos = THPVariable_Unpack(PyTuple_GET_ITEM(proj, 2));
  if (!index_ok(pos, dev) || pos.numel() != s.n) return 0;
  r->positions = i32(pos);
  r->rope_base = static_cast<float>(PyFloat_AsDouble(PyTuple_GET_ITEM(proj, 3)));
  r->eps = static_cast<float>(PyFloat_AsDouble(PyTuple_GET_ITEM(proj, 4)));
  PyObject* rd = PyTuple_GET_ITEM(proj, 5);
  r->rotary_dim = rd == Py_None ? s.d : static_cast<int>(PyLong_AsLong(rd));
  return PyErr_Occurred() ? -1 : 1;
}

// (q, k, v, k_cache, v_cache, out_loc, projection, indptr, indices, kv_lens or None, sm_scale,
//  max_kv_splits, page_size, gate)
PyObject* decode_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 14) return PyErr_Format(PyExc_TypeError, "decode_layer takes 14 arguments");
  if (!is_tensor(a[0]) || !is_tensor(a[3]) || !is_tensor(a[4]) || !is_tensor(a[7]) || !is_tensor(a[8]))
    Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(a[0]), &kc = THPVariable_Unpack(a[3]), &vc = THPVariable_Unpack(a[4]),
               &indptr = THPVariable_Unpack(a[7]), &indices = THPVariable_Unpack(a[8]);
  Shapes s;
  const void* gate;
  if (!attention_shapes(q, kc, vc, &s) || !index_ok(indptr, q.device()) || !index_ok(indices, q.device()) ||
      indptr.numel() != s.n + 1 || !gate_ptr(a[13], q, &gate))
    Py_RETURN_NONE;
  const int32_t* lens = nullptr;
  if (a[9] != Py_None) {
    if (!is_tensor(a[9])) Py_RETURN_NONE;
    const Tensor& t = THPVariable_Unpack(a[9]);
    if (!index_ok(t, q.device()) || t.numel() != s.n) Py_RETURN_NONE;
    lens = i32(t);
  }
  msgl_new_rows rows;
  const int fine = new_rows(a[1], a[2], a[5], a[6], q, s, &rows);
  if (fine < 0) return nullptr;
  if (fine == 0) Py_RETURN_NONE;
  ARG_FLOAT(scale, a[10]);
  ARG_INT(max_splits, a[11]);
  ARG_INT(page_size, a[12]);
  const int64_t total = indices.numel();
  int64_t stream;
  Scratch ws;
  if (!stream_of(Py_None, s.device, &stream) ||
      !scratch_for(s.device, stream, kDecode,
                   msgl_decode_workspace_bytes_full(s.n, s.hq, s.hkv, s.d, static_cast<int>(max_splits),
                                                    lens ? total * page_size : total),
                   &ws))
    return nullptr;
  Tensor out = empty_like_rows(q);
  const int rc = in_turn(ws, [&] {
    return msgl_decode_layer(&rows, q.data_ptr(), kc.data_ptr(), vc.data_ptr(), i32(indptr), i32(indices),
                                   lens, gate, out.data_ptr(), ws.ptr, ws.bytes, s.n, s.hq, s.hkv, s.d, s.num_slots,
                                   s.dtype, static_cast<float>(scale), static_cast<int>(max_splits),
                                   static_cast<int>(page_size), total, reinterpret_cast<void*>(stream));
  });
  return rc ? raise_status(rc) : THPVariable_Wrap(std::move(out));
}

// (q, k, v, k_cache, v_cache, out_loc, projection, qo_indptr, indptr, indices, kv_lens or None,
//  prefix_lens, sm_scale, max_len_extend, page_size, is_cross_attention, sliding_window_size, gate)
PyObject* prefill_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 18) return PyErr_Format(PyExc_TypeError, "prefill_layer takes 18 arguments");
  for (int i : {0, 3, 4, 7, 8, 9, 11})
    if (!is_tensor(a[i])) Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(a[0]), &kc = THPVariable_Unpack(a[3]), &vc = THPVariable_Unpack(a[4]),
               &qo = THPVariable_Unpack(a[7]), &indptr = THPVariable_Unpack(a[8]),
               &indices = THPVariable_Unpack(a[9]), &prefix = THPVariable_Unpack(a[11]);
  Shapes s;
  const void* gate;
  if (!attention_shapes(q, kc, vc, &s) || !index_ok(qo, q.device()) || !index_ok(indptr, q.device()) ||
      !index_ok(indices, q.device()) || !index_ok(prefix, q.device()) || qo.numel() < 2 ||
      indptr.numel() != qo.numel() || prefix.numel() + 1 != qo.numel() || !gate_ptr(a[17], q, &gate))
    Py_RETURN_NONE;
  const int batch = static_cast<int>(prefix.numel());
  const int32_t* lens = nullptr;
  if (a[10] != Py_None) {
    if (!is_tensor(a[10])) Py_RETURN_NONE;
    const Tensor& t = THPVariable_Unpack(a[10]);
    if (!index_ok(t, q.device()) || t.numel() != batch) Py_RETURN_NONE;
    lens = i32(t);
  }
  msgl_new_rows rows;
  const int fine = new_rows(a[1], a[2], a[5], a[6], q, s, &rows);
  if (fine < 0) return nullptr;
  if (fine == 0) Py_RETURN_NONE;
  ARG_FLOAT(scale, a[12]);
  ARG_INT(max_ext, a[13]);
  ARG_INT(page_size, a[14]);
  ARG_INT(window, a[16]);
  const int cross = PyObject_IsTrue(a[15]);
  if (cross < 0) return nullptr;
  const int64_t total = indices.numel();
  int64_t stream;
  Scratch ws;
  Pages pages;
  const int64_t tokens = lens ? total * page_size : total;
  if (!stream_of(Py_None, s.device, &stream) ||
      !scratch_for(s.device, stream, kPrefill,
                   msgl_prefill_workspace_bytes(batch, s.n, tokens, s.hq, s.hkv, s.d, static_cast<int>(max_ext),
                                                static_cast<int>(window)),
                   &ws))
    return nullptr;
  Tensor out = empty_like_rows(q);
  if (!pages_for(s.device, stream,
                 lens ? 0 : msgl_prefill_kv_pages_bytes(batch, s.n, tokens, s.hq, s.hkv, s.d, static_cast<int>(max_ext),
                                                        static_cast<int>(window)),
                 &pages))
    return nullptr;
  const int rc = in_turn(ws, [&] {
    return msgl_prefill_layer_pages(
      &rows, q.data_ptr(), kc.data_ptr(), vc.data_ptr(), i32(qo), i32(indptr), i32(indices), lens, i32(prefix), gate,
      out.data_ptr(), ws.ptr, ws.bytes, pages.ptr, pages.bytes, batch, s.n, s.hq, s.hkv, s.d, s.num_slots, s.dtype,
      static_cast<float>(scale), static_cast<int>(max_ext), cross, static_cast<int>(window),
      static_cast<int>(page_size), total, reinterpret_cast<void*>(stream));
  });
  return rc ? raise_status(rc) : THPVariable_Wrap(std::move(out));
}

// ------------------------------------------------------------------ index arrays of a step
PyObject *g_s_row, *g_s_cached, *g_s_device, *g_s_extend;   // interned attribute names

bool attr_int(PyObject* o, PyObject* name, long long* out) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (v == nullptr) return false;
  *out = PyLong_AsLongLong(v);
  Py_DECREF(v);
  return !(*out == -1 && PyErr_Occurred());
}

// (reqs, extend_lens or None, kv_lens or None, decode, page_size)
//   -> (packed, total_q, total_kv, total_pages, max_extend, max_kv)
// packed: bytes of (3, batch) int32: new tokens, KV lengths, page-table rows.  A decode row's new
// tokens are everything behind what the request has cached.
PyObject* collect_lens(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) return PyErr_Format(PyExc_TypeError, "collect_lens takes 5 arguments");
  const int decode_step = PyObject_IsTrue(a[3]);
  ARG_INT(ps, a[4]);
  if (decode_step < 0) return nullptr;
  if (ps <= 0) return PyErr_Format(PyExc_ValueError, "page_size must be > 0");
  PyObject* seq[3] = {PySequence_Fast(a[0], "reqs must be a sequence"), nullptr, nullptr};
  if (seq[0] == nullptr) return nullptr;
  const Py_ssize_t b = PySequence_Fast_GET_SIZE(seq[0]);
  PyObject* packed = nullptr;
  long long tq = 0, tkv = 0, tp = 0, me = 0, mk = 0;
  bool ok = true;
  for (int i = 1; i < 3 && ok; ++i) {
    if (a[i] == Py_None) continue;
    seq[i] = PySequence_Fast(a[i], "lengths must be a sequence");
    ok = seq[i] != nullptr;
    if (ok && PySequence_Fast_GET_SIZE(seq[i]) != b) {
      PyErr_SetString(PyExc_ValueError, "one length per request");
      ok = false;
    }
  }
  if (ok) packed = PyBytes_FromStringAndSize(nullptr, b * 3 * static_cast<Py_ssize_t>(sizeof(int32_t)));
  ok = packed != nullptr;
  int32_t* rec = ok ? reinterpret_cast<int32_t*>(PyBytes_AS_STRING(packed)) : nullptr;
  for (Py_ssize_t i = 0; i < b && ok; ++i) {
    PyObject* r = PySequence_Fast_GET_ITEM(seq[0], i);
    long long e = 0, kv = 0, row = 0, cached = 0;
    ok = attr_int(r, g_s_row, &row);
    if (ok && seq[2] != nullptr) {
      kv = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq[2], i));
      ok = !(kv == -1 && PyErr_Occurred());
    } else if (ok) {
      ok = attr_int(r, g_s_device, &kv);
    }
    if (ok && seq[1] != nullptr) {
      e = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq[1], i));
      ok = !(e == -1 && PyErr_Occurred());
    } else if (ok && decode_step) {
      ok = attr_int(r, g_s_cached, &cached);
      e = std::max(1LL, std::min(kv, kv - cached));
    } else if (ok) {
      ok = attr_int(r, g_s_extend, &e);
    }
    if (ok && (e < INT32_MIN || e > INT32_MAX || kv < INT32_MIN || kv > INT32_MAX || row < INT32_MIN ||
               row > INT32_MAX)) {
      PyErr_SetString(PyExc_OverflowError, "a request's length or row does not fit 32 bits");
      ok = false;
    }
    if (!ok) break;
    rec[i] = static_cast<int32_t>(e);
    rec[b + i] = static_cast<int32_t>(kv);
    rec[2 * b + i] = static_cast<int32_t>(row);
    tq += e;
    tkv += kv;
    tp += (kv + ps - 1) / ps;
    me = i == 0 ? e : std::max(me, e);
    mk = i == 0 ? kv : std::max(mk, kv);
  }
  for (PyObject* s : seq) Py_XDECREF(s);
  if (!ok) {
    Py_XDECREF(packed);
    return nullptr;
  }
  return Py_BuildValue("(NLLLLL)", packed, tq, tkv, tp, me, mk);
}

// Elements [off, off + n) of a 1-D tensor as a tensor of its own that shares its storage (a slice
// without the dispatcher: a step makes nine of them).
PyObject* piece(const Tensor& buf, int64_t off, int64_t n) {
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buf.storage()), buf.key_set(), buf.dtype());
  t.unsafeGetTensorImpl()->set_sizes_contiguous(c10::IntArrayRef(n));
  t.unsafeGetTensorImpl()->set_storage_offset(off);
  return THPVariable_Wrap(std::move(t));
}

// (packed, page_table, total_q, total_kv, total_pages, page_size, split_chunk, max_kv_splits,
//  per_token_ids, stream)
//   -> (qo_indptr, kv_indptr, prefix_lens, num_kv_splits, positions, kv_lens, kv_indices or None,
//       page_indptr or None, page_indices or None), or None where the batch is too large to travel
//       with the launch.
PyObject* index_arrays(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10) return PyErr_Format(PyExc_TypeError, "index_arrays takes 10 arguments");
  if (!PyBytes_Check(a[0]) || !is_tensor(a[1])) Py_RETURN_NONE;
  const Tensor& table = THPVariable_Unpack(a[1]);
  const int64_t batch = PyBytes_GET_SIZE(a[0]) / static_cast<int64_t>(3 * sizeof(int32_t));
  if (table.dim() != 2 || table.scalar_type() != at::kInt || !table.is_cuda() || table.stride(1) != 1 ||
      c10::cuda::current_device() != table.device().index() || batch < 1 || batch > MSGL_METADATA_HOST_MAX)
    Py_RETURN_NONE;
  ARG_INT(tq, a[2]);
  ARG_INT(tkv, a[3]);
  ARG_INT(tp, a[4]);
  ARG_INT(ps, a[5]);
  ARG_INT(chunk, a[6]);
  ARG_INT(max_splits, a[7]);
  const int per_token = PyObject_IsTrue(a[8]);
  if (per_token < 0) return nullptr;
  if (tq < 0 || tkv < 0 || tp < 0) Py_RETURN_NONE;
  const int dev = table.device().index();
  int64_t stream;
  Scratch ws;
  if (!stream_of(a[9], dev, &stream) || !scratch_for(dev, stream, kDecode, 256, &ws)) return nullptr;
  const bool paged = ps > 1;
  const int64_t size[9] = {batch + 1, batch + 1, batch, batch, tq, batch, per_token ? tkv : 0,
                           paged ? batch + 1 : 0, paged ? tp : 0};
  int64_t off[10] = {0};
  for (int i = 0; i < 9; ++i) off[i + 1] = off[i] + size[i];
  Tensor buf;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    buf = at::empty({off[9]}, at::TensorOptions().dtype(at::kInt).device(table.device()));
  }
  int32_t* p = static_cast<int32_t*>(buf.data_ptr());
  const int rc = unlocked([&] {
    return msgl_build_attn_metadata_host(
      reinterpret_cast<const int32_t*>(PyBytes_AS_STRING(a[0])), i32(table), table.stride(0), table.size(0),
      table.size(1), static_cast<int>(batch), static_cast<int>(ps), static_cast<int>(chunk),
      static_cast<int>(max_splits), tq, tkv, paged ? tp : 0, p + off[0], p + off[1], p + off[2], p + off[3],
      tq ? p + off[4] : nullptr, p + off[5], size[6] ? p + off[6] : nullptr, paged ? p + off[7] : nullptr,
      size[8] ? p + off[8] : nullptr, ws.ptr, reinterpret_cast<void*>(stream));
  });
  if (rc) return raise_status(rc);
  THPObjectPtr out(PyTuple_New(9));
  if (!out) return nullptr;
  for (int i = 0; i < 9; ++i) {
    PyObject* t;
    if ((i == 6 && !per_token) || (i >= 7 && !paged)) {
      t = Py_None;
      Py_INCREF(t);
    } else {
      t = piece(buf, off[i], size[i]);
      if (t == nullptr) return nullptr;
    }
    PyTuple_SET_ITEM(out.get(), i, t);
  }
  return out.release();
}

// (callable): how scratch is made, see g_make_workspace and g_make_pages
template <PyObject** MAKER>
PyObject* set_maker(PyObject*, PyObject* fn) {
  Py_INCREF(fn);
  Py_XDECREF(*MAKER);
  *MAKER = fn;
  Py_RETURN_NONE;
}

#define FAST(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(decode),       FAST(decode_paged),       FAST(prefill),
                          FAST(prefill_paged), FAST(store_kv),          FAST(qk_norm_rope_store),
                          FAST(decode_layer), FAST(prefill_layer),     FAST(collect_lens),
                          FAST(index_arrays),
                          {"set_workspace_maker", set_maker<&g_make_workspace>, METH_O, nullptr},
                          {"set_pages_maker", set_maker<&g_make_pages>, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Host side of the operators.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  g_s_row = PyUnicode_InternFromString("table_idx");
  g_s_cached = PyUnicode_InternFromString("cached_len");
  g_s_device = PyUnicode_InternFromString("device_len");
  g_s_extend = PyUnicode_InternFromString("extend_len");
  if (!g_s_row || !g_s_cached || !g_s_device || !g_s_extend) return nullptr;
  return PyModule_Create(&kModule);
}
