// The host side of the path's hot calls: argument checks, output allocation and the C-ABI call in one crossing from
// Python.  A decode step of a few rows keeps the GPU busy for ~10 us; the same steps in Python (tensor views and
// conversions, environment look-ups, a foreign-function call of 25 arguments) took 45-55 us per call.
//
// Every function takes tensors as they come from the caller and serves the regular case only: CUDA tensors on one
// device, int32 metadata, contiguous operands of the expected dtypes.  Anything else returns None and launches
// nothing; the caller then takes the Python route, which converts what can be converted and raises what must be
// raised, so that errors and results are the same whichever route a call takes.
//
// The entry points of libnvj_b200.so are resolved from the handle that Python has loaded.  Workspaces and status words
// belong to Python (one per device and stream); this module keeps references to them.

#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <structmember.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../../include/nvj_b200.h"

namespace {

// ---- what Python hands over once ------------------------------------------------------------------------------

struct Library {
  decltype(&nvj_paged_decode_fused_append) fused_append;
  decltype(&nvj_paged_decode_window) window;
  decltype(&nvj_kv_append) append;
  decltype(&nvj_kv_append_mapped) append_mapped;
  decltype(&nvj_paged_prefill_packed_counted) prefill;
  decltype(&nvj_qk_norm_rope_kv_append) norm_rope;
  decltype(&nvj_compute_slot_mapping) slot_mapping;
  decltype(&nvj_copy_blocks) copy_blocks;
  decltype(&nvj_copy_many_async) copy_many;
  decltype(&nvj_stage_in) stage_in;
  decltype(&nvj_hybrid_snapshot_host_slots) snapshot;
  decltype(&nvj_hybrid_restore_host_slots) restore;
};
Library lib;
PyObject* cb_workspace;  // (device index, rows): makes Python create the workspace and hand it over
PyObject* cb_status;     // (device index): the same for the status word
PyObject* cb_failed;     // (status, name): raises
PyObject* cb_strict;     // (device index, stream, name, check workspace, check status word): reads the device status back

struct Workspace {
  int device;
  void* stream;
  at::Tensor buf;
  long long max_batch;
};
struct StatusWord {
  int device;
  void* stream;
  at::Tensor word;
};
// A handful of entries (one per stream in use), guarded by the interpreter lock.
std::vector<Workspace>& workspaces() { static auto* v = new std::vector<Workspace>; return *v; }
std::vector<StatusWord>& status_words() { static auto* v = new std::vector<StatusWord>; return *v; }

bool env_is(const char* name, const char* value) {
  const char* v = std::getenv(name);
  return v && std::strcmp(v, value) == 0;
}

const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kBFloat16: return NVJ_BF16;
    case at::kHalf: return NVJ_F16;
    case at::kFloat: return NVJ_F32;
    default: return -1;
  }
}

bool on(const at::Tensor& t, int device) { return t.is_cuda() && t.get_device() == device; }
bool meta(const at::Tensor& t, int device) { return on(t, device) && t.scalar_type() == at::kInt && t.is_contiguous(); }
const int32_t* i32(const at::Tensor& t) { return static_cast<const int32_t*>(t.data_ptr()); }

void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

// The workspace of (device, current stream) with room for `rows` rows; null with a Python error set.
const Workspace* workspace_for(int device, void* stream, long long rows) {
  for (int turn = 0; turn < 2; ++turn) {
    for (const Workspace& w : workspaces())
      if (w.device == device && w.stream == stream && w.max_batch >= rows) return &w;
    PyObject* r = PyObject_CallFunction(cb_workspace, "iL", device, rows);
    if (!r) return nullptr;
    Py_DECREF(r);
  }
  PyErr_SetString(PyExc_RuntimeError, "no workspace for this stream");
  return nullptr;
}

int32_t* status_for(int device, void* stream) {
  for (int turn = 0; turn < 2; ++turn) {
    for (const StatusWord& w : status_words())
      if (w.device == device && w.stream == stream) return static_cast<int32_t*>(w.word.data_ptr());
    PyObject* r = PyObject_CallFunction(cb_status, "i", device);
    if (!r) return nullptr;
    Py_DECREF(r);
  }
  PyErr_SetString(PyExc_RuntimeError, "no status word for this stream");
  return nullptr;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, int device) {
  return at::detail::empty_cuda(sizes, dtype, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt);
}

// A float32 output; NVJ_POISON_OUTPUT=1 (tests) starts it as NaN.
at::Tensor output(at::IntArrayRef sizes, int device) {
  at::Tensor t = empty(sizes, at::kFloat, device);
  if (env_is("NVJ_POISON_OUTPUT", "1")) t.fill_(std::nan(""));
  return t;
}

// After a call: a failure raises; NVJ_CHECK_STATUS=1 (tests) reads the device status back.  False: Python error set.
bool finished(int rc, const char* what, int device, void* stream, bool workspace, bool word) {
  if (rc != NVJ_OK) {
    PyObject* r = PyObject_CallFunction(cb_failed, "is", rc, what);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, what);
    return false;
  }
  if (env_is("NVJ_CHECK_STATUS", "1")) {
    PyObject* r = PyObject_CallFunction(cb_strict, "iKsii", device, reinterpret_cast<unsigned long long>(stream), what, workspace ? 1 : 0, word ? 1 : 0);
    if (!r) return false;
    Py_DECREF(r);
  }
  return true;
}

#define NVJ_NONE() do { Py_RETURN_NONE; } while (0)
#define NVJ_CALL(rc, call) do { Py_BEGIN_ALLOW_THREADS rc = (call); Py_END_ALLOW_THREADS } while (0)

bool args_are(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
  return false;
}

// A layer of a pair of 5-D caches [L, NB, bs, Hkv, D].
struct Layer {
  bool ok = false;
  int device, dtype, block_size, hkv, d;
  long long blocks;
  char *k, *v;
};
Layer cache_layer(const at::Tensor* k, const at::Tensor* v, long long layer) {
  Layer l;
  if (!k || !v || !k->is_cuda() || k->dim() != 5 || v->dim() != 5 || k->sizes() != v->sizes() || k->dtype() != v->dtype()) return l;
  l.device = k->get_device();
  l.dtype = dtype_code(*k);
  if (l.dtype < 0 || !on(*v, l.device) || !k->is_contiguous() || !v->is_contiguous() || layer < 0 || layer >= k->size(0)) return l;
  l.blocks = k->size(1);
  l.block_size = (int)k->size(2);
  l.hkv = (int)k->size(3);
  l.d = (int)k->size(4);
  const size_t bytes = (size_t)l.blocks * l.block_size * l.hkv * l.d * k->element_size();
  l.k = static_cast<char*>(k->data_ptr()) + layer * bytes;
  l.v = static_cast<char*>(v->data_ptr()) + layer * bytes;
  l.ok = true;
  return l;
}

// ---- the calls ----------------------------------------------------------------------------------------------------

// fused_decode(query, new_k, new_v, k_cache, v_cache, block_tables, seq_lens, positions | None, layer, block_size, scale,
//              groups, variant, out | None, stream | None) -> out [B, 1, Hq * D] float32.  A given `out` may lie in pinned host
// memory (the kernels only write it), which spares the caller a copy; a given stream must have its workspace already.
PyObject* fused_decode(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 15)) return nullptr;
  const at::Tensor *q = tensor(a[0]), *nk = tensor(a[1]), *nv = tensor(a[2]), *tab = tensor(a[5]), *len = tensor(a[6]);
  const at::Tensor* pos = a[7] == Py_None ? nullptr : tensor(a[7]);
  const long long layer = PyLong_AsLongLong(a[8]), bs = PyLong_AsLongLong(a[9]), groups = PyLong_AsLongLong(a[11]);
  const double scale = PyFloat_AsDouble(a[10]);
  const long long variant = PyLong_AsLongLong(a[12]);
  void* given = a[14] == Py_None ? nullptr : reinterpret_cast<void*>(PyLong_AsUnsignedLongLong(a[14]));
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  const Layer l = cache_layer(tensor(a[3]), tensor(a[4]), layer);
  if (!l.ok || !q || !nk || !nv || !tab || !len || (!pos && a[7] != Py_None)) NVJ_NONE();
  if (q->dim() != 4 || q->size(1) != 1 || nk->dim() != 4 || nk->size(1) != 1 || nk->sizes() != nv->sizes()) NVJ_NONE();
  const long long batch = q->size(0), hq = q->size(2), d = q->size(3);
  const int qdt = dtype_code(*q);
  if (batch == 0 || l.block_size != bs || d != l.d || hq != l.hkv * groups || nk->size(0) != batch || nk->size(2) != l.hkv ||
      nk->size(3) != l.d || (qdt != NVJ_F32 && qdt != l.dtype) || dtype_code(*nk) != l.dtype || dtype_code(*nv) != l.dtype)
    NVJ_NONE();
  if (!on(*q, l.device) || !on(*nk, l.device) || !on(*nv, l.device) || !q->is_contiguous() || !nk->is_contiguous() ||
      !nv->is_contiguous() || !meta(*tab, l.device) || !meta(*len, l.device) || tab->dim() != 2 || tab->size(0) != batch ||
      len->dim() != 1 || len->size(0) != batch || (pos && (!meta(*pos, l.device) || pos->numel() != batch)))
    NVJ_NONE();
  void* stream = given ? given : stream_of(l.device);
  const Workspace* ws = workspace_for(l.device, stream, batch);
  if (!ws) return nullptr;
  at::Tensor out;
  if (a[13] == Py_None) {
    out = output({batch, 1, hq * d}, l.device);
  } else {
    const at::Tensor* o = tensor(a[13]);
    if (!o || o->scalar_type() != at::kFloat || !o->is_contiguous() || o->numel() != batch * hq * d || !(on(*o, l.device) || (o->is_cpu() && o->is_pinned()))) NVJ_NONE();
    out = *o;
    if (env_is("NVJ_POISON_OUTPUT", "1")) out.fill_(std::nan(""));
  }
  void* wp = ws->buf.data_ptr();
  const size_t wb = (size_t)ws->buf.numel();
  int rc;
  NVJ_CALL(rc, lib.fused_append(q->data_ptr(), qdt, nk->data_ptr(), nv->data_ptr(), pos ? i32(*pos) : nullptr, l.k, l.v, l.dtype,
                                l.blocks, l.block_size, l.hkv, l.d, (int)hq, i32(*tab), (int)tab->size(1), i32(*len), (int)batch,
                                (float)scale, static_cast<float*>(out.data_ptr()), wp, wb, (int)variant, stream));
  if (!finished(rc, "nvj_paged_decode_fused_append", l.device, stream, true, false)) return nullptr;
  return THPVariable_Wrap(std::move(out));
}

// window_decode(query [B, T, Hq, D], k_cache, v_cache, block_tables, seq_lens, positions [B, T] | None, layer, block_size,
//               scale, groups, max_kv_len | None) -> out [B, T, Hq * D] float32
PyObject* window_decode(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 11)) return nullptr;
  const at::Tensor *q = tensor(a[0]), *tab = tensor(a[3]), *len = tensor(a[4]);
  const at::Tensor* pos = a[5] == Py_None ? nullptr : tensor(a[5]);
  const long long layer = PyLong_AsLongLong(a[6]), bs = PyLong_AsLongLong(a[7]), groups = PyLong_AsLongLong(a[9]);
  const double scale = PyFloat_AsDouble(a[8]);
  long long max_len = a[10] == Py_None ? -1 : PyLong_AsLongLong(a[10]);
  if (a[10] != Py_None && max_len < 1) { PyErr_Clear(); NVJ_NONE(); }
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  const Layer l = cache_layer(tensor(a[1]), tensor(a[2]), layer);
  if (!l.ok || !q || !tab || !len || (!pos && a[5] != Py_None) || q->dim() != 4) NVJ_NONE();
  const long long batch = q->size(0), width = q->size(1), hq = q->size(2), d = q->size(3);
  const int qdt = dtype_code(*q);
  if (batch == 0 || width < 1 || width > 16 || l.block_size != bs || d != l.d || hq != l.hkv * groups || qdt < 0) NVJ_NONE();
  if (width > 1 && !(pos && qdt == NVJ_BF16 && l.dtype == NVJ_BF16 && hq == 8 && d == 256 && bs == 16 && l.hkv == 2)) NVJ_NONE();
  if (!on(*q, l.device) || !q->is_contiguous() || !meta(*tab, l.device) || !meta(*len, l.device) || tab->dim() != 2 ||
      tab->size(0) != batch || len->dim() != 1 || len->size(0) != batch ||
      (pos && (!meta(*pos, l.device) || pos->dim() != 2 || pos->size(0) != batch || pos->size(1) != width)))
    NVJ_NONE();
  const long long span = tab->size(1) * bs;
  if (max_len < 0) max_len = span;
  if (max_len < 1 || max_len > span || max_len > l.blocks * bs || max_len > 0x7fffffffLL) NVJ_NONE();
  void* stream = stream_of(l.device);
  const Workspace* ws = workspace_for(l.device, stream, batch);
  if (!ws) return nullptr;
  at::Tensor out = output({batch, width, hq * d}, l.device);
  void* wp = ws->buf.data_ptr();
  const size_t wb = (size_t)ws->buf.numel();
  int rc;
  NVJ_CALL(rc, lib.window(q->data_ptr(), qdt, l.k, l.v, l.dtype, l.blocks, l.block_size, l.hkv, l.d, (int)hq, i32(*tab),
                          (int)tab->size(1), i32(*len), pos ? i32(*pos) : nullptr, (int)batch, (int)width, (int)max_len,
                          (float)scale, static_cast<float*>(out.data_ptr()), wp, wb, stream));
  if (rc == NVJ_ERR_UNSUPPORTED) NVJ_NONE();
  if (!finished(rc, "nvj_paged_decode_window", l.device, stream, true, false)) return nullptr;
  return THPVariable_Wrap(std::move(out));
}

// stage_in(targets, sources, on_first, streams (3), events (2), by kernel) -> True: copies sources[i] -> targets[i] and makes the
// third stream wait for them: in one kernel on the first stream if so asked and the sources are pinned, else the first
// `on_first` pairs by the copy engines on the first stream and the rest on the second.  None, and nothing issued, when a source
// differs from its target in dtype or size or is not contiguous.
PyObject* stage_in(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 6)) return nullptr;
  const long long split = PyLong_AsLongLong(a[2]);
  unsigned long long st[3], ev[2];
  if (PyErr_Occurred() || !PyTuple_Check(a[0]) || !PyTuple_Check(a[1]) || !PyArg_ParseTuple(a[3], "KKK", &st[0], &st[1], &st[2]) ||
      !PyArg_ParseTuple(a[4], "KK", &ev[0], &ev[1]))
    return nullptr;
  constexpr Py_ssize_t kMost = 16;
  void* dst[kMost];
  const void* src[kMost];
  size_t bytes[kMost];
  const Py_ssize_t pairs = PyTuple_GET_SIZE(a[0]);
  if (pairs != PyTuple_GET_SIZE(a[1]) || pairs > kMost || split < 0 || split > pairs) NVJ_NONE();
  for (Py_ssize_t i = 0; i < pairs; ++i) {
    const at::Tensor *d = tensor(PyTuple_GET_ITEM(a[0], i)), *s = tensor(PyTuple_GET_ITEM(a[1], i));
    if (!d || !s || d->dtype() != s->dtype() || d->numel() != s->numel() || !d->is_contiguous() || !s->is_contiguous()) NVJ_NONE();
    dst[i] = d->data_ptr();
    src[i] = s->data_ptr();
    bytes[i] = d->nbytes();
  }
  auto stream = [&](int i) { return reinterpret_cast<cudaStream_t>(st[i]); };
  auto event = [&](int i) { return reinterpret_cast<cudaEvent_t>(ev[i]); };
  const bool by_kernel = PyObject_IsTrue(a[5]) == 1;
  int rc = NVJ_ERR_UNSUPPORTED, streams = 1;
  cudaError_t e = cudaSuccess;
  Py_BEGIN_ALLOW_THREADS
  if (by_kernel) rc = lib.stage_in(dst, src, bytes, (int)pairs, stream(0));
  if (rc == NVJ_ERR_UNSUPPORTED) {
    streams = 2;
    rc = lib.copy_many(dst, src, bytes, (int)split, stream(0));
    if (rc == NVJ_OK) rc = lib.copy_many(dst + split, src + split, bytes + split, (int)(pairs - split), stream(1));
  }
  for (int i = 0; i < streams && e == cudaSuccess; ++i) {
    e = cudaEventRecord(event(i), stream(i));
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream(2), event(i), 0);
  }
  Py_END_ALLOW_THREADS
  if (rc == NVJ_OK && e != cudaSuccess) rc = NVJ_ERR_LAUNCH;
  if (rc != NVJ_OK && !finished(rc, "nvj_stage_in or nvj_copy_many_async", 0, nullptr, false, false)) return nullptr;
  Py_RETURN_TRUE;
}

// append(new_k, new_v, k_cache, v_cache, layer, slot_mapping | None, positions, block_tables, token_row_ids | None,
//        query_start_loc, block_size of the tables) -> True: token rows [rows, cols, Hkv, D] go to their slots; without a slot mapping the slots of
// a rectangular batch are made from positions and tables in the same launch.
PyObject* append(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 11)) return nullptr;
  const at::Tensor *nk = tensor(a[0]), *nv = tensor(a[1]), *qsl = tensor(a[9]);
  const long long layer = PyLong_AsLongLong(a[4]), bs = PyLong_AsLongLong(a[10]);
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  const Layer l = cache_layer(tensor(a[2]), tensor(a[3]), layer);
  if (!l.ok || !nk || !nv || !qsl || nk->dim() != 4 || nk->sizes() != nv->sizes() || nk->size(2) != l.hkv || nk->size(3) != l.d) NVJ_NONE();
  const long long rows = nk->size(0), cols = nk->size(1);
  const int dt = dtype_code(*nk);
  if (rows * cols == 0 || dt < 0 || nv->dtype() != nk->dtype() || !on(*nk, l.device) || !on(*nv, l.device) || !nk->is_contiguous() ||
      !nv->is_contiguous() || !meta(*qsl, l.device) || qsl->numel() < 1)
    NVJ_NONE();
  const bool packed = a[8] != Py_None;
  const long long num_slots = l.blocks * l.block_size;
  void* stream = stream_of(l.device);
  int rc;
  const char* what;
  if (a[5] != Py_None) {
    const at::Tensor* slots = tensor(a[5]);
    if (!slots || !meta(*slots, l.device) || slots->dim() != 2 || slots->size(0) != rows || slots->size(1) != cols) NVJ_NONE();
    int32_t* st = status_for(l.device, stream);
    if (!st) return nullptr;
    what = "nvj_kv_append";
    NVJ_CALL(rc, lib.append(nk->data_ptr(), nv->data_ptr(), dt, i32(*slots), nullptr, i32(*qsl), (int)qsl->numel() - 1, packed ? 1 : 0,
                            (int)rows, (int)cols, l.k, l.v, l.dtype, num_slots, l.hkv, l.d, st, stream));
  } else {
    const at::Tensor *pos = tensor(a[6]), *tab = tensor(a[7]);
    if (packed || !pos || !tab || !meta(*pos, l.device) || !meta(*tab, l.device) || pos->dim() != 2 || pos->size(0) != rows || pos->size(1) != cols ||
        tab->dim() != 2 || tab->size(0) != rows || tab->size(1) == 0 || bs != l.block_size)
      NVJ_NONE();
    int32_t* st = status_for(l.device, stream);
    if (!st) return nullptr;
    what = "nvj_kv_append_mapped";
    NVJ_CALL(rc, lib.append_mapped(nk->data_ptr(), nv->data_ptr(), dt, i32(*pos), i32(*tab), nullptr, (int)tab->size(0),
                                   (int)tab->size(1), l.block_size, i32(*qsl), (int)qsl->numel() - 1, 0, (int)rows, (int)cols,
                                   l.k, l.v, l.dtype, num_slots, l.hkv, l.d, st, stream));
  }
  if (!finished(rc, what, l.device, stream, false, true)) return nullptr;
  Py_RETURN_TRUE;
}

// packed_prefill(query [1, T, Hq, D], k_cache, v_cache, block_tables, kv_lens, positions, query_start_loc, layer, block_size,
//                scale, groups, decode_rows | None, tile_pairs | None) -> out [1, T, Hq * D] float32
PyObject* packed_prefill(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 13)) return nullptr;
  const at::Tensor *q = tensor(a[0]), *tab = tensor(a[3]), *len = tensor(a[4]), *pos = tensor(a[5]), *qsl = tensor(a[6]);
  const long long layer = PyLong_AsLongLong(a[7]), bs = PyLong_AsLongLong(a[8]), groups = PyLong_AsLongLong(a[10]);
  const double scale = PyFloat_AsDouble(a[9]);
  const long long decode_rows = a[11] == Py_None ? -1 : PyLong_AsLongLong(a[11]);
  const long long pairs = a[12] == Py_None ? -1 : PyLong_AsLongLong(a[12]);
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  const Layer l = cache_layer(tensor(a[1]), tensor(a[2]), layer);
  if (!l.ok || !q || !tab || !len || !pos || !qsl || q->dim() != 4 || q->size(0) != 1) NVJ_NONE();
  const long long tokens = q->size(1), hq = q->size(2), d = q->size(3);
  const int qdt = dtype_code(*q);
  if (tokens == 0 || l.block_size != bs || d != l.d || hq != l.hkv * groups || qdt < 0 || !on(*q, l.device) || !q->is_contiguous()) NVJ_NONE();
  if (!meta(*tab, l.device) || !meta(*len, l.device) || !meta(*pos, l.device) || !meta(*qsl, l.device) || tab->dim() != 2) NVJ_NONE();
  const long long rows = tab->size(0);
  if (len->dim() != 1 || len->size(0) != rows || pos->dim() != 2 || pos->size(0) != 1 || pos->size(1) != tokens || qsl->numel() != rows + 1) NVJ_NONE();
  const char* env = std::getenv("NVJ_PREFILL_VARIANT");
  const int variant = env ? std::atoi(env) : 0;
  const bool model_shape = l.dtype == NVJ_BF16 && bs == 16 && l.hkv == 2 && d == 256 && hq == 8 && (qdt == NVJ_BF16 || qdt == NVJ_F32);
  // decode rows and tiles side by side on two streams: the Python route forks and joins
  if (model_shape && (variant == 0 || variant == 4 || variant == 5) && decode_rows > 0 && decode_rows < rows &&
      !env_is("NVJ_MIXED_SIDE_BY_SIDE", "0") &&
      (env_is("NVJ_MIXED_SIDE_BY_SIDE", "1") ||
       c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None))
    NVJ_NONE();
  void* stream = stream_of(l.device);
  int32_t* st = status_for(l.device, stream);
  if (!st) return nullptr;
  const bool tiles_only = model_shape && variant != 1 && decode_rows == 0;  // a workspace lent to the tiles lets them split key ranges
  const Workspace* ws = nullptr;
  if (tiles_only ? !env_is("NVJ_PREFILL_KEY_SPLITS", "0") : decode_rows != 0) {
    ws = workspace_for(l.device, stream, rows);
    if (!ws) return nullptr;
  }
  void* wp = ws ? ws->buf.data_ptr() : nullptr;
  const size_t wb = ws ? (size_t)ws->buf.numel() : 0;
  at::Tensor out = output({1, tokens, hq * d}, l.device);
  int rc;
  // (the count is of rows of several tokens: it holds when a row of one is served by the decode kernel, or there is none)
  const long long counted = decode_rows >= 0 && pairs >= 0 ? pairs : -1;
  NVJ_CALL(rc, lib.prefill(q->data_ptr(), qdt, l.k, l.v, l.dtype, l.blocks, l.block_size, l.hkv, l.d, (int)hq, i32(*tab), (int)tab->size(1),
                           i32(*len), i32(*pos), i32(*qsl), (int)rows, (int)tokens, (float)scale, static_cast<float*>(out.data_ptr()), st, wp,
                           wb, variant, tiles_only ? 3 : 0, (int)counted, stream));
  if (!finished(rc, "nvj_paged_prefill_packed", l.device, stream, ws != nullptr, true)) return nullptr;
  return THPVariable_Wrap(std::move(out));
}

// norm_rope(query, k, v, q_weight, k_weight, positions, slot_mapping, k_layer, v_layer, query_start_loc | None, packed, eps,
//           inv_freq | None, rotary_dim) -> query for attention; text positions [rows, cols], cache layers [..., Hkv, D]
PyObject* norm_rope(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 14)) return nullptr;
  const at::Tensor *q = tensor(a[0]), *k = tensor(a[1]), *v = tensor(a[2]), *qw = tensor(a[3]), *kw = tensor(a[4]), *pos = tensor(a[5]),
                   *slots = tensor(a[6]), *kl = tensor(a[7]), *vl = tensor(a[8]);
  const at::Tensor *qsl = a[9] == Py_None ? nullptr : tensor(a[9]), *inv = a[12] == Py_None ? nullptr : tensor(a[12]);
  const int packed = PyObject_IsTrue(a[10]);
  const double eps = PyFloat_AsDouble(a[11]);
  const long long rotary = PyLong_AsLongLong(a[13]);
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  if (!q || !k || !v || !qw || !kw || !pos || !slots || !kl || !vl || (!qsl && a[9] != Py_None) || (!inv && rotary > 0)) NVJ_NONE();
  if (!q->is_cuda() || q->dim() != 4 || k->dim() != 4 || k->sizes() != v->sizes() || q->size(0) != k->size(0) || q->size(1) != k->size(1)) NVJ_NONE();
  const int dev = q->get_device();
  const long long rows = q->size(0), cols = q->size(1), hq = q->size(2), d = q->size(3), hkv = k->size(2);
  if (rows * cols == 0 || k->size(3) != d || kl->dim() < 3 || kl->sizes() != vl->sizes() || kl->size(-2) != hkv || kl->size(-1) != d) NVJ_NONE();
  const int dt = dtype_code(*q), wdt = dtype_code(*qw);
  if (dt < 0 || k->dtype() != q->dtype() || v->dtype() != q->dtype() || wdt < 0 || kw->dtype() != qw->dtype() || qw->numel() != d || kw->numel() != d ||
      !qw->is_contiguous() || !kw->is_contiguous() || kl->dtype() != vl->dtype() || dtype_code(*kl) < 0 || !kl->is_contiguous() || !vl->is_contiguous())
    NVJ_NONE();
  for (const at::Tensor* t : {k, v, qw, kw, kl, vl}) if (!on(*t, dev)) NVJ_NONE();
  if (inv && (!on(*inv, dev) || inv->scalar_type() != at::kFloat || inv->numel() * 2 < rotary)) NVJ_NONE();
  if (!meta(*pos, dev) || !meta(*slots, dev) || pos->dim() != 2 || pos->numel() != rows * cols || slots->numel() != rows * cols || (qsl && !meta(*qsl, dev))) NVJ_NONE();
  // tokens evenly spaced: one stride serves rows and columns (the query may be a view of a wider projection)
  auto token_stride = [&](const at::Tensor& t, long long* stride) {
    if (t.stride(3) != 1 || (rows > 1 && cols > 1 && t.stride(0) != t.stride(1) * cols)) return false;
    *stride = cols > 1 ? t.stride(1) : (rows > 1 ? t.stride(0) : t.size(2) * d);
    return true;
  };
  long long qs;
  long long ks;
  long long vs;
  if (!token_stride(*q, &qs) || !token_stride(*k, &ks) || !token_stride(*v, &vs) || k->stride(2) != d || v->stride(2) != d) NVJ_NONE();
  void* stream = stream_of(dev);
  int32_t* st = status_for(dev, stream);
  if (!st) return nullptr;
  at::Tensor out = empty({rows, cols, hq, d}, q->scalar_type(), dev);
  int rc;
  NVJ_CALL(rc, lib.norm_rope(q->data_ptr(), qs, q->stride(2), k->data_ptr(), ks, v->data_ptr(), vs, dt, qw->data_ptr(), kw->data_ptr(), wdt,
                             (float)eps, inv ? static_cast<const float*>(inv->data_ptr()) : nullptr, (int)rotary, i32(*pos), 1, nullptr, i32(*slots),
                             nullptr, qsl ? i32(*qsl) : nullptr, qsl ? (int)qsl->numel() - 1 : 0, packed, (int)rows, (int)cols, kl->data_ptr(),
                             vl->data_ptr(), dtype_code(*kl), kl->numel() / (hkv * d), (int)hq, (int)hkv, (int)d, out.data_ptr(), st, stream));
  if (!finished(rc, "nvj_qk_norm_rope_kv_append", dev, stream, false, true)) return nullptr;
  return THPVariable_Wrap(std::move(out));
}

// copy_blocks(k_cache, v_cache, src_ids, dst_ids) -> True
PyObject* copy_blocks(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 4)) return nullptr;
  const at::Tensor *k = tensor(a[0]), *v = tensor(a[1]), *src = tensor(a[2]), *dst = tensor(a[3]);
  const Layer l = cache_layer(k, v, 0);
  if (!l.ok || !src || !dst || !meta(*src, l.device) || !meta(*dst, l.device) || src->dim() != 1 || src->sizes() != dst->sizes()) NVJ_NONE();
  const long long block = (long long)l.block_size * l.hkv * l.d * k->element_size();
  void* stream = stream_of(l.device);
  int32_t* st = status_for(l.device, stream);
  if (!st) return nullptr;
  int rc;
  NVJ_CALL(rc, lib.copy_blocks(l.k, l.v, (int)k->size(0), l.blocks, block, l.blocks * block, i32(*src), i32(*dst), (int)src->numel(), st, stream));
  if (!finished(rc, "nvj_copy_blocks", l.device, stream, false, true)) return nullptr;
  Py_RETURN_TRUE;
}

// hybrid_copy(conv_table | None, rec_table | None, conv_pool | None, rec_pool | None, table_slots, pool_slots, restore) -> True,
// for slot lists of at most NVJ_HYBRID_HOST_SLOTS entries in host memory
PyObject* hybrid_copy(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 7)) return nullptr;
  const at::Tensor* t[4];
  const at::Tensor* some = nullptr;
  for (int i = 0; i < 4; ++i) {
    t[i] = a[i] == Py_None ? nullptr : tensor(a[i]);
    if (a[i] != Py_None && (!t[i] || !t[i]->is_cuda() || !t[i]->is_contiguous() || t[i]->dim() < 1 || t[i]->size(0) < 1)) NVJ_NONE();
    if (t[i]) some = t[i];
  }
  if (!some || (t[0] == nullptr) != (t[2] == nullptr) || (t[1] == nullptr) != (t[3] == nullptr) || !PyList_Check(a[4]) || !PyList_Check(a[5])) NVJ_NONE();
  const int device = some->get_device();
  long long bytes[4] = {0, 0, 0, 0};
  for (int i = 0; i < 4; ++i)
    if (t[i]) {
      if (t[i]->get_device() != device) NVJ_NONE();
      bytes[i] = t[i]->numel() / t[i]->size(0) * t[i]->element_size();
    }
  const Py_ssize_t pairs = PyList_GET_SIZE(a[4]);
  if (bytes[0] != bytes[2] || bytes[1] != bytes[3] || pairs != PyList_GET_SIZE(a[5]) || pairs > NVJ_HYBRID_HOST_SLOTS) NVJ_NONE();
  int32_t slots[2][NVJ_HYBRID_HOST_SLOTS];
  for (int side = 0; side < 2; ++side)
    for (Py_ssize_t i = 0; i < pairs; ++i) {
      const long long v = PyLong_AsLongLong(PyList_GET_ITEM(a[4 + side], i));
      if (PyErr_Occurred() || v < INT32_MIN || v > INT32_MAX) { PyErr_Clear(); NVJ_NONE(); }
      slots[side][i] = (int32_t)v;
    }
  const int restore = PyObject_IsTrue(a[6]);
  void* stream = stream_of(device);
  int32_t* st = status_for(device, stream);
  if (!st) return nullptr;
  auto ptr = [&](int i) { return t[i] ? t[i]->data_ptr() : nullptr; };
  const long long table_rows = (t[1] ? t[1] : t[0])->size(0), pool_rows = (t[3] ? t[3] : t[2])->size(0);
  int rc;
  if (restore) NVJ_CALL(rc, lib.restore(ptr(0), ptr(2), bytes[0], ptr(1), ptr(3), bytes[1], table_rows, pool_rows, slots[0], slots[1], (int)pairs, st, stream));
  else NVJ_CALL(rc, lib.snapshot(ptr(0), ptr(2), bytes[0], ptr(1), ptr(3), bytes[1], table_rows, pool_rows, slots[0], slots[1], (int)pairs, st, stream));
  if (!finished(rc, restore ? "nvj_hybrid_restore" : "nvj_hybrid_snapshot", device, stream, false, true)) return nullptr;
  Py_RETURN_TRUE;
}

// decode_shape(positions [B, T], block_tables [B, W], seq_lens [B]) -> (B, T, W), or None unless they are CUDA tensors that agree
PyObject* decode_shape(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 3)) return nullptr;
  const at::Tensor *pos = tensor(a[0]), *tab = tensor(a[1]), *len = tensor(a[2]);
  if (!pos || !tab || !len || pos->dim() != 2 || tab->dim() != 2 || len->dim() != 1 || !pos->is_cuda() || !tab->is_cuda() || !len->is_cuda() ||
      pos->size(0) != tab->size(0) || pos->size(0) != len->size(0))
    NVJ_NONE();
  return Py_BuildValue("LLL", (long long)pos->size(0), (long long)pos->size(1), (long long)tab->size(1));
}

// The int32 slots [rows, cols] of positions, from the rows' block tables: 1, or 0 when an operand has to be converted or complained
// about, or -1 with a Python error set.
int make_slots(const at::Tensor* pos, const at::Tensor* tab, const at::Tensor* rid, long long bs, at::Tensor* out) {
  if (!pos || !tab || !pos->is_cuda() || pos->dim() != 2 || tab->dim() != 2 || bs < 1) return 0;
  const int dev = pos->get_device();
  if (!meta(*pos, dev) || !meta(*tab, dev) || tab->size(0) < 1 || tab->size(1) < 1) return 0;
  if (rid ? (!meta(*rid, dev) || rid->sizes() != pos->sizes()) : pos->size(0) > tab->size(0)) return 0;
  void* stream = stream_of(dev);
  *out = empty(pos->sizes(), at::kInt, dev);
  int rc;
  NVJ_CALL(rc, lib.slot_mapping(i32(*pos), i32(*tab), rid ? i32(*rid) : nullptr, (int)pos->size(0), (int)pos->size(1), (int)tab->size(0),
                                (int)tab->size(1), (int)bs, static_cast<int32_t*>(out->data_ptr()), stream));
  return finished(rc, "nvj_compute_slot_mapping", dev, stream, false, false) ? 1 : -1;
}

// slot_mapping(positions [rows, cols], block_tables, block_size, token_row_ids | None) -> int32 [rows, cols]
PyObject* slot_mapping(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 4)) return nullptr;
  const at::Tensor* rid = a[3] == Py_None ? nullptr : tensor(a[3]);
  const long long bs = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  if (!rid && a[3] != Py_None) NVJ_NONE();
  at::Tensor out;
  const int made = make_slots(tensor(a[0]), tensor(a[1]), rid, bs, &out);
  if (made < 0) return nullptr;
  if (made == 0) NVJ_NONE();
  return THPVariable_Wrap(std::move(out));
}

// prefill_slots(positions [rows, cols], block_tables, seq_lens, block_size, token_row_ids | None) -> (slots, rows, cols) of a prefill
// batch whose shapes agree
PyObject* prefill_slots(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 5)) return nullptr;
  const at::Tensor *pos = tensor(a[0]), *tab = tensor(a[1]), *len = tensor(a[2]), *rid = a[4] == Py_None ? nullptr : tensor(a[4]);
  const long long bs = PyLong_AsLongLong(a[3]);
  if (PyErr_Occurred()) { PyErr_Clear(); NVJ_NONE(); }
  if (!pos || !tab || !len || (!rid && a[4] != Py_None) || pos->dim() != 2 || tab->dim() != 2 || len->dim() != 1 ||
      len->size(0) != tab->size(0) || (!rid && pos->size(0) != tab->size(0)))
    NVJ_NONE();
  at::Tensor out;
  const int made = make_slots(pos, tab, rid, bs, &out);
  if (made < 0) return nullptr;
  if (made == 0) NVJ_NONE();
  return Py_BuildValue("NLL", THPVariable_Wrap(std::move(out)), (long long)pos->size(0), (long long)pos->size(1));
}

// ---- prefix hashes --------------------------------------------------------------------------------------------------

// XXH64 (seed 0) over 64-bit words, after the published specification of the xxHash family: four lanes over stripes of four
// words, the words left over, an avalanche.  Blocks are whole words, so the specification's byte tail never occurs.
class WordHash {
  static constexpr uint64_t kP1 = 0x9E3779B185EBCA87ull, kP2 = 0xC2B2AE3D27D4EB4Full, kP3 = 0x165667B19E3779F9ull,
                            kP4 = 0x85EBCA77C2B2AE63ull, kP5 = 0x27D4EB2F165667C5ull;
  static uint64_t rotate(uint64_t x, int r) { return (x << r) | (x >> (64 - r)); }
  static uint64_t mix(uint64_t lane, uint64_t word) { return rotate(lane + word * kP2, 31) * kP1; }

 public:
  static uint64_t of(const uint64_t* w, size_t n) {
    uint64_t h = kP5;
    size_t i = 0;
    if (n >= 4) {
      uint64_t lane[4] = {kP1 + kP2, kP2, 0, 0 - kP1};
      for (; i + 4 <= n; i += 4)
        for (int k = 0; k < 4; ++k) lane[k] = mix(lane[k], w[i + k]);
      h = rotate(lane[0], 1) + rotate(lane[1], 7) + rotate(lane[2], 12) + rotate(lane[3], 18);
      for (uint64_t v : lane) h = (h ^ mix(0, v)) * kP1 + kP4;
    }
    h += 8 * n;
    for (; i < n; ++i) h = rotate(h ^ mix(0, w[i]), 27) * kP1 + kP4;
    h = (h ^ (h >> 33)) * kP2;
    h = (h ^ (h >> 29)) * kP3;
    return h ^ (h >> 32);
  }
};

// The value of a plain int of machine size; false for anything else.  (Token ids are one digit: no call.)
inline bool int_of(PyObject* o, long long* v) {
  if (!PyLong_CheckExact(o)) return false;
#if PY_VERSION_HEX >= 0x030C0000
  const PyLongObject* i = reinterpret_cast<const PyLongObject*>(o);
  if (PyUnstable_Long_IsCompact(i)) { *v = PyUnstable_Long_CompactValue(i); return true; }
#endif
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return !overflow;
}

// The chained digests of a token list's blocks, one at a time.
class HashChain {
  PyObject* tokens_;
  long long bs_;
  std::vector<uint64_t> words_;  // [predecessor's digest, the block's tokens]
  bool chained_ = false;

 public:
  HashChain(PyObject* tokens, long long block_size) : tokens_(tokens), bs_(block_size), words_((size_t)block_size + 1) {}
  void start_from(uint64_t digest) { words_[0] = digest; chained_ = true; }
  // Digest of block b, the one behind the last asked for; false when its tokens are not machine-size integers.
  bool next(long long b, uint64_t* h) {
    for (long long i = 0; i < bs_; ++i) {
      long long v;
      if (!int_of(PyList_GET_ITEM(tokens_, (Py_ssize_t)(b * bs_ + i)), &v)) return false;
      words_[(size_t)i + 1] = (uint64_t)v;
    }
    *h = chained_ ? WordHash::of(words_.data(), words_.size()) : WordHash::of(words_.data() + 1, words_.size() - 1);
    start_from(*h);
    return true;
  }
};

// hash_chain(token_ids, block_size, blocks, prefix | -1) -> digests of the first `blocks` full blocks of a token list, each
// over its predecessor's digest (the first over `prefix` if there is one) and its own tokens as int64.  None when the
// tokens are not a list of machine-size integers.
PyObject* hash_chain(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 4)) return nullptr;
  const long long bs = PyLong_AsLongLong(a[1]), blocks = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (!PyList_CheckExact(a[0]) || !PyLong_CheckExact(a[3]) || bs < 1 || blocks < 0 || blocks > PyList_GET_SIZE(a[0]) / bs) NVJ_NONE();
  int overflow = 0;
  HashChain chain(a[0], bs);
  if (PyLong_AsLongLongAndOverflow(a[3], &overflow) != -1 || overflow) chain.start_from(PyLong_AsUnsignedLongLongMask(a[3]));
  PyObject* out = PyList_New((Py_ssize_t)blocks);
  for (long long b = 0; out && b < blocks; ++b) {
    uint64_t h;
    if (!chain.next(b, &h)) { Py_DECREF(out); NVJ_NONE(); }
    PyObject* d = PyLong_FromUnsignedLongLong(h);
    if (!d) { Py_DECREF(out); return nullptr; }
    PyList_SET_ITEM(out, (Py_ssize_t)b, d);
  }
  return out;
}

// ---- the block manager's walks ----------------------------------------------------------------------------------------

// A block's attributes.  Blocks are objects with __slots__: where the type has a plain slot of that name it is read and
// written in place (15 ns less per access; a 96-block sequence has some 500 of them), else through the attribute.
enum BlockField { kRefCount, kHash, kTokenIds, kBlockFields };
PyObject* block_field_names[kBlockFields];

class BlockSlots {
  PyTypeObject* type_ = nullptr;
  Py_ssize_t at_[kBlockFields];

  PyObject** slot(PyObject* block, BlockField f) {
    if (Py_TYPE(block) != type_) {
      Py_INCREF(Py_TYPE(block));
      Py_XDECREF(type_);
      type_ = Py_TYPE(block);
      for (int k = 0; k < kBlockFields; ++k) {
        PyObject* d = PyObject_GetAttr(reinterpret_cast<PyObject*>(type_), block_field_names[k]);
        at_[k] = -1;
        if (d && Py_IS_TYPE(d, &PyMemberDescr_Type)) {
          const PyMemberDef* m = reinterpret_cast<PyMemberDescrObject*>(d)->d_member;
          if (m->type == T_OBJECT_EX && !(m->flags & READONLY)) at_[k] = m->offset;
        }
        if (!d) PyErr_Clear();
        Py_XDECREF(d);
      }
    }
    return at_[f] < 0 ? nullptr : reinterpret_cast<PyObject**>(reinterpret_cast<char*>(block) + at_[f]);
  }

 public:
  PyObject* get(PyObject* block, BlockField f) {  // a new reference
    PyObject** p = slot(block, f);
    if (!p || !*p) return PyObject_GetAttr(block, block_field_names[f]);
    Py_INCREF(*p);
    return *p;
  }
  bool set(PyObject* block, BlockField f, PyObject* v) {
    PyObject** p = slot(block, f);
    if (!p) return PyObject_SetAttr(block, block_field_names[f], v) == 0;
    PyObject* old = *p;
    Py_INCREF(v);
    *p = v;
    Py_XDECREF(old);
    return true;
  }
} block_slots;

PyObject* block_at(PyObject* blocks, PyObject* id) {  // borrowed; IndexError outside the pool
  const long long at = PyLong_AsLongLong(id);
  if (at >= 0 && at < PyList_GET_SIZE(blocks)) return PyList_GET_ITEM(blocks, (Py_ssize_t)at);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_IndexError, "block outside the pool");
  return nullptr;
}

int same_token(PyObject* x, PyObject* y) {
  long long u, v;
  if (x == y) return 1;
  return int_of(x, &u) && int_of(y, &v) ? u == v : PyObject_RichCompareBool(x, y, Py_EQ);
}

// Whether a block holds exactly the tokens [at, at + bs) of the list under this digest: 1, 0, or -1 with a Python error set.
int holds(PyObject* block, PyObject* digest, PyObject* tokens, long long at, long long bs) {
  PyObject *hash = block_slots.get(block, kHash), *held = block_slots.get(block, kTokenIds);
  int same = hash && held ? PyObject_RichCompareBool(hash, digest, Py_EQ) : -1;
  if (same == 1) same = PyList_Check(held) && PyList_GET_SIZE(held) == bs ? 1 : 0;
  for (long long k = 0; same == 1 && k < bs; ++k)
    same = same_token(PyList_GET_ITEM(held, (Py_ssize_t)k), PyList_GET_ITEM(tokens, (Py_ssize_t)(at + k)));
  Py_XDECREF(hash);
  Py_XDECREF(held);
  return same;
}

// cached_run(token_ids, digests | None, block_size, full blocks, published {digest: block id}, blocks, cacheable digests |
// None, used ids) -> (ids of the published blocks of the longest reusable prefix, its digest | None, how many of them are in
// use): a block counts when it holds exactly these tokens.  Digests are taken as the walk needs them when none are given;
// None when that meets tokens which are not machine-size integers.
PyObject* cached_run(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 8)) return nullptr;
  const long long bs = PyLong_AsLongLong(a[2]), full = PyLong_AsLongLong(a[3]);
  if (PyErr_Occurred()) return nullptr;
  const bool lazy = a[1] == Py_None;
  if (!PyList_Check(a[0]) || (!lazy && (!PyList_Check(a[1]) || PyList_GET_SIZE(a[1]) < full)) || !PyDict_Check(a[4]) ||
      !PyList_Check(a[5]) || !PyAnySet_Check(a[7]) || bs < 1 || full > PyList_GET_SIZE(a[0]) / bs) {
    PyErr_SetString(PyExc_TypeError, "cached_run: lists, a dict and a set expected");
    return nullptr;
  }
  HashChain chain(a[0], bs);
  PyObject *hits = PyList_New(0), *best_digest = nullptr;
  Py_ssize_t best = 0;
  long long live = 0, best_live = 0;
  bool ok = hits != nullptr, whole = true;
  for (long long i = 0; ok && i < full; ++i) {
    PyObject* digest;
    if (lazy) {
      uint64_t h;
      if (!(whole = chain.next(i, &h))) break;
      digest = PyLong_FromUnsignedLongLong(h);
      if (!(ok = digest != nullptr)) break;
    } else {
      digest = PyList_GET_ITEM(a[1], (Py_ssize_t)i);
      Py_INCREF(digest);
    }
    PyObject* id = PyDict_GetItemWithError(a[4], digest);  // borrowed
    PyObject* block = id ? block_at(a[5], id) : nullptr;
    ok = block || (!id && !PyErr_Occurred());
    const int same = block ? holds(block, digest, a[0], i * bs, bs) : 0;
    if (same == 1) {
      const int used = PySet_Contains(a[7], id), usable = a[6] == Py_None ? 1 : PySequence_Contains(a[6], digest);
      ok = ok && used >= 0 && usable >= 0 && PyList_Append(hits, id) == 0;
      live += used > 0;
      if (ok && usable) {
        best = (Py_ssize_t)i + 1;
        best_live = live;
        Py_XDECREF(best_digest);
        Py_INCREF(digest);
        best_digest = digest;
      }
    }
    Py_DECREF(digest);
    ok = ok && same >= 0;
    if (same != 1) break;
  }
  ok = ok && PyList_SetSlice(hits, best, PyList_GET_SIZE(hits), nullptr) == 0;
  PyObject* out = nullptr;
  if (ok && !whole) { Py_INCREF(Py_None); out = Py_None; }
  else if (ok) out = Py_BuildValue("OOL", hits, best_digest ? best_digest : Py_None, best_live);
  Py_XDECREF(hits);
  Py_XDECREF(best_digest);
  return out;
}

// add_owner(blocks, ids, used) -> those of the ids that are not in use, which stay as they are
PyObject* add_owner(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 3)) return nullptr;
  if (!PyList_Check(a[0]) || !PyList_Check(a[1]) || !PyAnySet_Check(a[2])) {
    PyErr_SetString(PyExc_TypeError, "add_owner: lists and a set expected");
    return nullptr;
  }
  PyObject* idle = PyList_New(0);
  for (Py_ssize_t k = 0; idle && k < PyList_GET_SIZE(a[1]); ++k) {
    PyObject* id = PyList_GET_ITEM(a[1], k);
    const int used = PySet_Contains(a[2], id);
    bool ok = used == 0 ? PyList_Append(idle, id) == 0 : used == 1;
    if (used == 1) {
      PyObject* block = block_at(a[0], id);
      PyObject* owners = block ? block_slots.get(block, kRefCount) : nullptr;
      PyObject* more = owners ? PyLong_FromLongLong(PyLong_AsLongLong(owners) + 1) : nullptr;
      ok = more && !PyErr_Occurred() && block_slots.set(block, kRefCount, more);
      Py_XDECREF(owners);
      Py_XDECREF(more);
    }
    if (!ok) Py_CLEAR(idle);
  }
  return idle;
}

// Block `id` becomes a sequence's: owned once, with its digest and the tokens [at, at + bs) when it is a full block (else `digest` is
// null); what it published before is withdrawn.  False: Python error set.
bool fresh_block(PyObject* blocks, PyObject* id, PyObject* published, PyObject* no_hash, PyObject* one, PyObject* digest, PyObject* tokens,
                 long long at, long long bs) {
  PyObject* block = block_at(blocks, id);
  if (!block) return false;
  PyObject *owners = block_slots.get(block, kRefCount), *old = block_slots.get(block, kHash);
  bool ok = owners && old;
  if (ok && PyObject_IsTrue(owners) != 0) {
    PyErr_SetString(PyExc_AssertionError, "a free block has an owner");
    ok = false;
  }
  const int had = ok ? PyObject_RichCompareBool(old, no_hash, Py_NE) : 0;
  if (had == 1) {  // its old content is about to be overwritten
    PyObject* holder = PyDict_GetItemWithError(published, old);
    const int mine = holder ? PyObject_RichCompareBool(holder, id, Py_EQ) : 0;
    if (mine == 1) ok = PyDict_DelItem(published, old) == 0;
    else ok = mine == 0 && !PyErr_Occurred();
  } else if (had < 0) {
    ok = false;
  }
  Py_XDECREF(owners);
  Py_XDECREF(old);
  PyObject* held = ok ? (digest ? PyList_GetSlice(tokens, (Py_ssize_t)at, (Py_ssize_t)(at + bs)) : PyList_New(0)) : nullptr;
  ok = ok && held && block_slots.set(block, kRefCount, one) && block_slots.set(block, kHash, digest ? digest : no_hash) &&
       block_slots.set(block, kTokenIds, held);
  Py_XDECREF(held);
  return ok;
}

// take_fresh(blocks, ids, first, digests, token_ids, block_size, published, no_hash): block ids[k] becomes block first + k of
// a sequence: owned once, with its digest and tokens when it is a full block; what it published before is withdrawn.
PyObject* take_fresh(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 8)) return nullptr;
  const long long first = PyLong_AsLongLong(a[2]), bs = PyLong_AsLongLong(a[5]);
  if (PyErr_Occurred()) return nullptr;
  if (!PyList_Check(a[0]) || !PyList_Check(a[1]) || !PyList_Check(a[3]) || !PyList_Check(a[4]) || !PyDict_Check(a[6])) {
    PyErr_SetString(PyExc_TypeError, "take_fresh: lists and a dict expected");
    return nullptr;
  }
  PyObject* one = PyLong_FromLong(1);
  bool ok = one != nullptr;
  for (Py_ssize_t k = 0; ok && k < PyList_GET_SIZE(a[1]); ++k) {
    const long long index = first + k;
    PyObject* digest = index < PyList_GET_SIZE(a[3]) ? PyList_GET_ITEM(a[3], (Py_ssize_t)index) : nullptr;
    ok = fresh_block(a[0], PyList_GET_ITEM(a[1], k), a[6], a[7], one, digest, a[4], index * bs, bs);
  }
  Py_XDECREF(one);
  if (!ok) return nullptr;
  Py_RETURN_NONE;
}

PyObject* name_num_cached;

// allocate(seq, token_ids, block_size, full blocks, blocks in all, published, blocks, cacheable digests | None, used ids, whether published
// blocks are shared, the sequence's table, take(n), take_cached(id), no_hash) -> (digest of the reused prefix | None,): a sequence's
// blocks in one pass over its tokens, the published ones of its longest reusable prefix (cached_run, add_owner), then fresh ones (take_fresh).
// None, and nothing changed, when the tokens are not machine-size integers.
PyObject* allocate(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 14)) return nullptr;
  PyObject *tokens = a[1], *published = a[5], *blocks = a[6], *used = a[8], *table = a[10];
  const long long bs = PyLong_AsLongLong(a[2]), full = PyLong_AsLongLong(a[3]), want = PyLong_AsLongLong(a[4]);
  const int share = PyObject_IsTrue(a[9]);
  if (PyErr_Occurred()) return nullptr;
  if (!PyList_CheckExact(tokens) || !PyDict_Check(published) || !PyList_Check(blocks) || !PySet_Check(used) || !PyList_Check(table) || bs < 1 ||
      full < 0 || full > PyList_GET_SIZE(tokens) / bs)
    NVJ_NONE();
  HashChain chain(tokens, bs);
  std::vector<uint64_t> digests((size_t)full);
  PyObject *hits = PyList_New(0), *best_digest = nullptr;
  Py_ssize_t best = 0;
  bool ok = hits != nullptr, whole = true, run = share != 0;
  for (long long i = 0; ok && i < full; ++i) {
    if (!(whole = chain.next(i, &digests[(size_t)i]))) break;
    if (!run) continue;
    PyObject* digest = PyLong_FromUnsignedLongLong(digests[(size_t)i]);
    PyObject* id = digest ? PyDict_GetItemWithError(published, digest) : nullptr;  // borrowed
    PyObject* block = id ? block_at(blocks, id) : nullptr;
    ok = digest && (block || (!id && !PyErr_Occurred()));
    const int same = block ? holds(block, digest, tokens, i * bs, bs) : 0;
    if (same == 1) {
      const int usable = a[7] == Py_None ? 1 : PySequence_Contains(a[7], digest);
      ok = ok && usable >= 0 && PyList_Append(hits, id) == 0;
      if (ok && usable) {
        best = (Py_ssize_t)i + 1;
        Py_XDECREF(best_digest);
        Py_INCREF(digest);
        best_digest = digest;
      }
    }
    Py_XDECREF(digest);
    ok = ok && same >= 0;
    run = same == 1;
  }
  ok = ok && PyList_SetSlice(hits, best, PyList_GET_SIZE(hits), nullptr) == 0;
  if (!ok || !whole) {
    Py_XDECREF(hits);
    Py_XDECREF(best_digest);
    if (!ok) return nullptr;
    NVJ_NONE();
  }
  // the shared ones: owned once more, those that nobody holds taken back from the free list
  PyObject* owner_args[3] = {blocks, hits, used};
  PyObject* idle = add_owner(owner_args, 3);
  ok = idle != nullptr;
  for (Py_ssize_t k = 0; ok && k < PyList_GET_SIZE(idle); ++k) {
    PyObject* r = PyObject_CallOneArg(a[12], PyList_GET_ITEM(idle, k));
    ok = r != nullptr;
    Py_XDECREF(r);
  }
  Py_XDECREF(idle);
  ok = ok && PyList_SetSlice(table, PyList_GET_SIZE(table), PyList_GET_SIZE(table), hits) == 0;
  PyObject* cached = ok ? PyLong_FromLongLong((long long)best * bs) : nullptr;
  ok = cached && PyObject_SetAttr(a[0], name_num_cached, cached) == 0;
  Py_XDECREF(cached);
  Py_DECREF(hits);
  // the rest
  PyObject* rest = ok ? PyLong_FromLongLong(want - best) : nullptr;
  PyObject* fresh = rest ? PyObject_CallOneArg(a[11], rest) : nullptr;
  Py_XDECREF(rest);
  PyObject* one = PyLong_FromLong(1);
  ok = fresh && one && PyList_Check(fresh);
  for (Py_ssize_t k = 0; ok && k < PyList_GET_SIZE(fresh); ++k) {
    const long long index = (long long)best + k;
    PyObject* digest = index < full ? PyLong_FromUnsignedLongLong(digests[(size_t)index]) : nullptr;
    ok = (digest || index >= full) && fresh_block(blocks, PyList_GET_ITEM(fresh, k), published, a[13], one, digest, tokens, index * bs, bs);
    Py_XDECREF(digest);
  }
  for (Py_ssize_t k = 0; ok && k < PyList_GET_SIZE(fresh); ++k) ok = PySet_Add(used, PyList_GET_ITEM(fresh, k)) == 0;
  ok = ok && PyList_SetSlice(table, PyList_GET_SIZE(table), PyList_GET_SIZE(table), fresh) == 0;
  Py_XDECREF(one);
  Py_XDECREF(fresh);
  PyObject* out = ok ? PyTuple_Pack(1, best_digest ? best_digest : Py_None) : nullptr;
  Py_XDECREF(best_digest);
  if (!out && !PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "allocate: take() has to return a list");
  return out;
}

// drop_owner(blocks, table) -> ids that have no owner left, last block of the table first
PyObject* drop_owner(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 2)) return nullptr;
  if (!PyList_Check(a[0]) || !PyList_Check(a[1])) { PyErr_SetString(PyExc_TypeError, "drop_owner: lists expected"); return nullptr; }
  PyObject* gone = PyList_New(0);
  for (Py_ssize_t k = PyList_GET_SIZE(a[1]); gone && k-- > 0;) {
    PyObject* id = PyList_GET_ITEM(a[1], k);
    PyObject* block = block_at(a[0], id);
    PyObject* owners = block ? block_slots.get(block, kRefCount) : nullptr;
    const long long left = owners ? PyLong_AsLongLong(owners) - 1 : 0;
    PyObject* fewer = owners && !PyErr_Occurred() ? PyLong_FromLongLong(left) : nullptr;
    const bool ok = fewer && block_slots.set(block, kRefCount, fewer) && (left != 0 || PyList_Append(gone, id) == 0);
    Py_XDECREF(owners);
    Py_XDECREF(fewer);
    if (!ok) Py_CLEAR(gone);
  }
  return gone;
}

// ---- a batch's host arrays ------------------------------------------------------------------------------------------

// One int32 out of a Python integer (anything with __index__); false with OverflowError or TypeError set.
bool as_i32(PyObject* o, int32_t* v) {
  long long x;
  if (!int_of(o, &x)) {
    x = PyLong_AsLongLong(o);
    if (x == -1 && PyErr_Occurred()) return false;
  }
  if (x < INT32_MIN || x > INT32_MAX) {
    PyErr_SetString(PyExc_OverflowError, "a batch entry does not fit 32 bits");
    return false;
  }
  *v = (int32_t)x;
  return true;
}

bool fill_i32(PyObject* list, int32_t* to) {
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i)
    if (!as_i32(PyList_GET_ITEM(list, i), to + i)) return false;
  return true;
}

// The block tables `rows`, padded with zeros to `width`: as int32 to `to` (zeros already), as a tuple of tuples in return.
PyObject* fill_tables(PyObject* rows, Py_ssize_t width, int32_t* to) {
  PyObject *zero = PyLong_FromLong(0), *out = PyTuple_New(PyList_GET_SIZE(rows));
  for (Py_ssize_t r = 0; out && r < PyList_GET_SIZE(rows); ++r, to += width) {
    PyObject* list = PySequence_Fast(PyList_GET_ITEM(rows, r), "a block table is a sequence");
    PyObject* row = list && PySequence_Fast_GET_SIZE(list) <= width ? PyTuple_New(width) : nullptr;
    if (!row) {
      if (!PyErr_Occurred())
        PyErr_Format(PyExc_ValueError, "scheduled block table needs %zd blocks but bucket has %zd", PySequence_Fast_GET_SIZE(list), width);
      Py_XDECREF(list);
      Py_CLEAR(out);
      break;
    }
    PyTuple_SET_ITEM(out, r, row);
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(list);
    bool ok = true;
    for (Py_ssize_t i = 0; ok && i < len; ++i) {
      PyObject* item = PySequence_Fast_GET_ITEM(list, i);
      if (!(ok = as_i32(item, to + i))) break;
      if (PyLong_CheckExact(item)) Py_INCREF(item);
      else ok = (item = PyLong_FromLong(to[i])) != nullptr;
      PyTuple_SET_ITEM(row, i, item);
    }
    for (Py_ssize_t i = len; ok && i < width; ++i) {
      Py_INCREF(zero);
      PyTuple_SET_ITEM(row, i, zero);
    }
    Py_DECREF(list);
    if (!ok) Py_CLEAR(out);
  }
  Py_XDECREF(zero);
  return out;
}

// pack_batch(parts, rows, width, device index | -1) -> ([a tensor per part], the [len(rows), width] table, the same table as a
// tuple of tuples).  A part is (list of ints, shape); what the list does not fill of its shape is zero.  All of it is written
// into one staging buffer (pinned for a GPU) and crosses in one copy; the tensors are views of the one device buffer.
PyObject* pack_batch(PyObject* const* a, Py_ssize_t n) {
  if (!args_are(n, 4)) return nullptr;
  const long long width = PyLong_AsLongLong(a[2]), device = PyLong_AsLongLong(a[3]);
  if (PyErr_Occurred()) return nullptr;
  if (!PyList_Check(a[0]) || !PyList_Check(a[1]) || width < 0) {
    PyErr_SetString(PyExc_TypeError, "pack_batch: lists expected");
    return nullptr;
  }
  struct Part { PyObject* list; int64_t shape[2], at; int dims; };
  std::vector<Part> parts((size_t)PyList_GET_SIZE(a[0]));
  int64_t total = 0;
  for (size_t k = 0; k < parts.size(); ++k) {
    Part& p = parts[k];
    PyObject *entry = PyList_GET_ITEM(a[0], (Py_ssize_t)k), *shape;
    if (!PyArg_ParseTuple(entry, "O!O!", &PyList_Type, &p.list, &PyTuple_Type, &shape)) return nullptr;
    p.dims = (int)PyTuple_GET_SIZE(shape);
    p.at = total;
    int64_t count = 1;
    for (int d = 0; d < p.dims && d < 2; ++d) {
      p.shape[d] = PyLong_AsLongLong(PyTuple_GET_ITEM(shape, d));
      if (PyErr_Occurred()) return nullptr;
      count *= p.shape[d];
    }
    if (p.dims < 1 || p.dims > 2 || count < PyList_GET_SIZE(p.list)) {
      PyErr_SetString(PyExc_ValueError, "pack_batch: a part is longer than its shape");
      return nullptr;
    }
    total += count;
  }
  const int64_t rows = PyList_GET_SIZE(a[1]), rows_at = total;
  total += rows * width;
  at::AutoDispatchBelowADInplaceOrView plain;  // integers: nothing here is differentiable
  at::Tensor stage = at::empty({total > 0 ? total : 1}, at::TensorOptions(at::kInt).pinned_memory(device >= 0));
  int32_t* words = static_cast<int32_t*>(stage.data_ptr());
  std::memset(words, 0, (size_t)total * sizeof(int32_t));
  for (const Part& p : parts)
    if (!fill_i32(p.list, words + p.at)) return nullptr;
  PyObject* host = fill_tables(a[1], (Py_ssize_t)width, words + rows_at);
  if (!host) return nullptr;
  at::Tensor dev = stage;
  if (device >= 0) {
    dev = empty(stage.sizes(), at::kInt, (int)device);
    dev.copy_(stage, /*non_blocking=*/true);
  }
  PyObject* views = PyList_New((Py_ssize_t)parts.size());
  for (size_t k = 0; views && k < parts.size(); ++k) {
    const Part& p = parts[k];
    const int64_t strides[2] = {p.dims == 2 ? p.shape[1] : 1, 1};
    PyList_SET_ITEM(views, (Py_ssize_t)k, THPVariable_Wrap(dev.as_strided({p.shape, (size_t)p.dims}, {strides, (size_t)p.dims}, p.at)));
  }
  PyObject* out = views ? Py_BuildValue("NNN", views, THPVariable_Wrap(dev.as_strided({rows, width}, {width, 1}, rows_at)), host) : nullptr;
  if (!views) Py_DECREF(host);
  return out;
}

// ---- set-up ---------------------------------------------------------------------------------------------------------

// init(library handle, workspace, status, failed, strict)
PyObject* init(PyObject*, PyObject* args) {
  unsigned long long handle;
  PyObject *ws, *st, *failed, *strict;
  if (!PyArg_ParseTuple(args, "KOOOO", &handle, &ws, &st, &failed, &strict)) return nullptr;
  void* h = reinterpret_cast<void*>(handle);
  const char* missing = nullptr;
  auto get = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(h, name));
    if (!fn) missing = name;
  };
  get(lib.fused_append, "nvj_paged_decode_fused_append");
  get(lib.window, "nvj_paged_decode_window");
  get(lib.append, "nvj_kv_append");
  get(lib.append_mapped, "nvj_kv_append_mapped");
  get(lib.prefill, "nvj_paged_prefill_packed_counted");
  get(lib.norm_rope, "nvj_qk_norm_rope_kv_append");
  get(lib.slot_mapping, "nvj_compute_slot_mapping");
  get(lib.copy_many, "nvj_copy_many_async");
  get(lib.stage_in, "nvj_stage_in");
  get(lib.copy_blocks, "nvj_copy_blocks");
  get(lib.snapshot, "nvj_hybrid_snapshot_host_slots");
  get(lib.restore, "nvj_hybrid_restore_host_slots");
  if (missing) {
    PyErr_Format(PyExc_ImportError, "libnvj_b200.so does not export %s", missing);
    return nullptr;
  }
  for (PyObject* o : {ws, st, failed, strict}) Py_INCREF(o);
  cb_workspace = ws; cb_status = st; cb_failed = failed; cb_strict = strict;
  Py_RETURN_NONE;
}

// set_workspace(device index, stream, buffer, max_batch): replaces the one of that (device, stream)
PyObject* set_workspace(PyObject*, PyObject* args) {
  int device;
  unsigned long long stream;
  PyObject* buf;
  long long max_batch;
  if (!PyArg_ParseTuple(args, "iKOL", &device, &stream, &buf, &max_batch)) return nullptr;
  const at::Tensor* t = tensor(buf);
  if (!t) { PyErr_SetString(PyExc_TypeError, "buffer must be a tensor"); return nullptr; }
  void* s = reinterpret_cast<void*>(stream);
  for (Workspace& w : workspaces())
    if (w.device == device && w.stream == s) { w.buf = *t; w.max_batch = max_batch; Py_RETURN_NONE; }
  workspaces().push_back({device, s, *t, max_batch});
  Py_RETURN_NONE;
}

PyObject* set_status_word(PyObject*, PyObject* args) {
  int device;
  unsigned long long stream;
  PyObject* word;
  if (!PyArg_ParseTuple(args, "iKO", &device, &stream, &word)) return nullptr;
  const at::Tensor* t = tensor(word);
  if (!t) { PyErr_SetString(PyExc_TypeError, "word must be a tensor"); return nullptr; }
  void* s = reinterpret_cast<void*>(stream);
  for (StatusWord& w : status_words())
    if (w.device == device && w.stream == s) { w.word = *t; Py_RETURN_NONE; }
  status_words().push_back({device, s, *t});
  Py_RETURN_NONE;
}

// C++ exceptions become the Python ones that torch's own functions raise (out of memory among them).
template <PyObject* (*Fn)(PyObject* const*, Py_ssize_t)>
PyObject* entry(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return Fn(a, n);
  END_HANDLE_TH_ERRORS
}
#define NVJ_FAST(fn, doc) {#fn, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<fn>)), METH_FASTCALL, doc}
PyMethodDef methods[] = {
    NVJ_FAST(fused_decode, "append + decode of one token per row, or None"),
    NVJ_FAST(window_decode, "decode attention over a window, or None"),
    NVJ_FAST(append, "append of new K/V rows, or None"),
    NVJ_FAST(packed_prefill, "ragged packed attention, or None"),
    NVJ_FAST(norm_rope, "norm + rope + append, or None"),
    NVJ_FAST(decode_shape, "batch, query length and table width of a decode batch, or None"),
    NVJ_FAST(cached_run, "published blocks of a sequence's longest reusable prefix"),
    NVJ_FAST(add_owner, "a sequence shares blocks that are in use"),
    NVJ_FAST(take_fresh, "free blocks become a sequence's"),
    NVJ_FAST(allocate, "a sequence's blocks, shared and fresh, or None"),
    NVJ_FAST(drop_owner, "a sequence gives its blocks up"),
    NVJ_FAST(hash_chain, "chained digests of a token list's blocks, or None"),
    NVJ_FAST(stage_in, "a step's operands to the device, or None"),
    NVJ_FAST(copy_blocks, "cache[:, dst] = cache[:, src], or None"),
    NVJ_FAST(hybrid_copy, "snapshot or restore of GDN state rows, or None"),
    NVJ_FAST(pack_batch, "a batch's lists on the device"),
    NVJ_FAST(slot_mapping, "flat cache slots of positions, or None"),
    NVJ_FAST(prefill_slots, "flat cache slots of a prefill batch and its shape, or None"),
    {"init", init, METH_VARARGS, "resolve the library's entry points and keep the callbacks"},
    {"set_workspace", set_workspace, METH_VARARGS, "hand over a (device, stream)'s workspace"},
    {"set_status_word", set_status_word, METH_VARARGS, "hand over a (device, stream)'s status word"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_nvj_host", "Host side of the hot calls.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nvj_host(void) {
  const char* names[kBlockFields] = {"ref_count", "hash", "token_ids"};
  for (int k = 0; k < kBlockFields; ++k)
    if (!(block_field_names[k] = PyUnicode_InternFromString(names[k]))) return nullptr;
  if (!(name_num_cached = PyUnicode_InternFromString("num_cached_tokens"))) return nullptr;
  return PyModule_Create(&module);
}
