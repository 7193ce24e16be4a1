// Python entry points of the calls a decode loop makes every step, on the C ABI of libanna_b200_kv.so, the uploads of small arrays
// (fused_ops.py) and the loops over page ids behind the allocators (pools.py).
//
// A ctypes call converts some forty arguments one by one, and every address, size and stride among them costs a Python
// call of its own: two thirds of the 18 us of host time of a decode call, whose GPU work for a few short rows takes no
// longer.  The functions here take the tensors themselves.  They serve the ordinary call only: where an argument is not
// what they expect they return None before anything has happened, and the caller takes the general path, which converts
// or rejects it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/Functions.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "anna_b200_kv.h"

namespace {

const at::Tensor* tensor(PyObject* obj) {
  return THPVariable_Check(obj) ? &THPVariable_Unpack(obj) : nullptr;
}
// a tensor or None; *ok turns false for anything else
const at::Tensor* optional_tensor(PyObject* obj, bool* ok) {
  if (obj == Py_None) return nullptr;
  const at::Tensor* t = tensor(obj);
  if (t == nullptr) *ok = false;
  return t;
}
void* address(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }
const float* floats(const at::Tensor* t) { return static_cast<const float*>(address(t)); }

bool dtype_code(at::ScalarType type, int* code) {
  switch (type) {
    case at::kFloat: *code = ANNA_DTYPE_F32; return true;
    case at::kHalf: *code = ANNA_DTYPE_F16; return true;
    case at::kBFloat16: *code = ANNA_DTYPE_BF16; return true;
    default: return false;
  }
}
bool plain(const at::Tensor& t, c10::Device device, int64_t dims) {
  return t.device() == device && t.layout() == at::kStrided && t.dim() == dims;
}
bool on(const at::Tensor* t, c10::Device device) { return t == nullptr || t->device() == device; }

// Split-K scratch of a problem, as split_scratch and query_scratch of fused_ops.py hand it out; dropped by
// forget_scratch(), which they call whenever a buffer behind it is replaced.  Guarded by the interpreter lock; never
// destroyed, so that no CUDA memory is freed after the runtime is gone.
struct Scratch {
  at::Tensor stats, values, counters, frags;
  int capacity = 0;
};
using ScratchKey = std::tuple<int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t>;
std::map<ScratchKey, Scratch>& scratch_table() {
  static auto* table = new std::map<ScratchKey, Scratch>();
  return *table;
}
constexpr size_t kMaxScratch = 256;
PyObject* scratch_source = nullptr;  // (device, batch, heads, dim, kv_heads, max_len, (max_blocks, block, window) | None)

// false with a Python error set when the scratch cannot be had.  The query's device must be current.
bool scratch_of(const at::Tensor& query, int64_t stream, int64_t kv_heads, int64_t max_len, int64_t max_blocks, int64_t block,
                int64_t window, Scratch* out) {
  const ScratchKey key(query.device().index(), stream, query.size(0), query.size(1), query.size(3), kv_heads, max_len, block,
                       window);
  auto& table = scratch_table();
  const auto found = table.find(key);
  if (found != table.end()) {
    *out = found->second;
    return true;
  }
  if (scratch_source == nullptr) {
    PyErr_SetString(PyExc_RuntimeError, "anna_b200: no scratch source");
    return false;
  }
  PyObject* device = THPDevice_New(query.device());
  PyObject* got = window > 0
                      ? PyObject_CallFunction(scratch_source, "NLLLLL(LLL)", device, (long long)query.size(0),
                                              (long long)query.size(1), (long long)query.size(3), (long long)kv_heads,
                                              (long long)max_len, (long long)max_blocks, (long long)block, (long long)window)
                      : PyObject_CallFunction(scratch_source, "NLLLLLO", device, (long long)query.size(0),
                                              (long long)query.size(1), (long long)query.size(3), (long long)kv_heads,
                                              (long long)max_len, Py_None);
  if (got == nullptr) return false;
  Scratch s;
  bool ok = PyTuple_Check(got) && PyTuple_GET_SIZE(got) == 5;
  if (ok) {
    const at::Tensor* parts[4] = {tensor(PyTuple_GET_ITEM(got, 0)), tensor(PyTuple_GET_ITEM(got, 1)),
                                  tensor(PyTuple_GET_ITEM(got, 3)), optional_tensor(PyTuple_GET_ITEM(got, 4), &ok)};
    s.capacity = (int)PyLong_AsLong(PyTuple_GET_ITEM(got, 2));
    ok = ok && parts[0] != nullptr && parts[1] != nullptr && parts[2] != nullptr;
    if (ok) {
      s.stats = *parts[0];
      s.values = *parts[1];
      s.counters = *parts[2];
      if (parts[3] != nullptr) s.frags = *parts[3];
    }
  }
  Py_DECREF(got);
  if (!ok) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "anna_b200: bad scratch");
    return false;
  }
  if (table.size() >= kMaxScratch) table.clear();
  table[key] = s;
  *out = std::move(s);
  return true;
}

PyObject* failed(const char* what, int status) {
  return PyErr_Format(PyExc_RuntimeError, "%s failed (status %d): %s", what, status, anna_kv_last_error());
}

bool int_args(PyObject* const* args, int count, int64_t* out) {
  for (int i = 0; i < count; ++i) {
    out[i] = PyLong_AsLongLong(args[i]);
    if (out[i] == -1 && PyErr_Occurred()) return false;
  }
  return true;
}

// set_scratch_source(callable)
PyObject* set_scratch_source(PyObject*, PyObject* callable) {
  Py_INCREF(callable);
  Py_XSETREF(scratch_source, callable);
  Py_RETURN_NONE;
}

PyObject* forget_scratch(PyObject*, PyObject*) {
  scratch_table().clear();
  Py_RETURN_NONE;
}

// tq_decode(query, gate | None, packed_pages | None, table | None, window, slots, lengths, signs1, signs2, centroids, scaling,
//           kv_heads, block_size, residual_len, bits, value_group, num_pages) -> output | None
PyObject* tq_decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 17) return PyErr_Format(PyExc_TypeError, "tq_decode takes 17 arguments");
  const at::Tensor* query = tensor(args[0]);
  bool ok = true;
  const at::Tensor* gate = optional_tensor(args[1], &ok);
  const at::Tensor* pages = optional_tensor(args[2], &ok);
  const at::Tensor* table = optional_tensor(args[3], &ok);
  const at::Tensor* fixed[6];
  for (int i = 0; i < 6; ++i) {
    fixed[i] = tensor(args[4 + i]);
    ok = ok && fixed[i] != nullptr;
  }
  int code = 0;
  int64_t n[6];  // kv_heads, block_size, residual_len, bits, value_group, num_pages
  const double scaling = PyFloat_AsDouble(args[10]);
  if (scaling == -1.0 && PyErr_Occurred()) return nullptr;
  if (!int_args(args + 11, 6, n)) return nullptr;
  if (!ok || query == nullptr || !query->is_cuda() || !plain(*query, query->device(), 4) || query->size(2) != 1 ||
      query->stride(3) != 1 || query->size(0) == 0 || n[0] <= 0 || query->size(1) % n[0] != 0 ||
      !dtype_code(query->scalar_type(), &code))
    Py_RETURN_NONE;
  const c10::Device device = query->device();
  if (gate != nullptr && (!plain(*gate, device, 4) || gate->stride(3) != 1 || gate->scalar_type() != query->scalar_type() ||
                          gate->sizes() != query->sizes()))
    Py_RETURN_NONE;
  if (fixed[0]->scalar_type() != query->scalar_type() || fixed[0]->dim() != 5 || fixed[0]->size(2) != n[0] ||
      fixed[0]->size(4) != query->size(3))
    Py_RETURN_NONE;
  for (const at::Tensor* t : fixed)
    if (!on(t, device)) Py_RETURN_NONE;
  if (!on(pages, device) || !on(table, device)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  const int64_t max_blocks = table == nullptr ? 0 : table->size(1);
  Scratch s;
  if (!scratch_of(*query, reinterpret_cast<int64_t>(stream), n[0], max_blocks * n[1] + n[2], max_blocks, n[1], n[2], &s))
    return nullptr;
  at::Tensor out = at::empty(query->sizes(), query->options());
  const int64_t q_sb = query->stride(0), q_sh = query->stride(1), g_sb = gate ? gate->stride(0) : 0,
                g_sh = gate ? gate->stride(1) : 0;
  const int batch = (int)query->size(0), heads = (int)query->size(1), dim = (int)query->size(3);
  int status;
  {
    pybind11::gil_scoped_release unlocked;
    status = anna_tq_paged_decode(
        query->data_ptr(), q_sb, q_sh, static_cast<const uint8_t*>(address(pages)), static_cast<const int32_t*>(address(table)),
        table == nullptr ? 0 : table->stride(0), address(fixed[0]), static_cast<const int64_t*>(address(fixed[1])),
        static_cast<const int64_t*>(address(fixed[2])), floats(fixed[3]), floats(fixed[4]), floats(fixed[5]), address(gate),
        g_sb, g_sh, out.data_ptr(), out.stride(0), out.stride(1), static_cast<float*>(s.stats.data_ptr()),
        static_cast<float*>(s.values.data_ptr()), s.capacity, 0, static_cast<int32_t*>(s.counters.data_ptr()),
        s.frags.defined() ? s.frags.data_ptr() : nullptr, s.frags.defined() ? (size_t)s.frags.numel() : 0, batch, heads,
        (int)n[0], dim, (int)n[1], (int)n[2], (int)n[3], (int)n[4], n[5], max_blocks, (float)scaling, code, stream);
  }
  if (status != 0) return failed("anna_tq_paged_decode", status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// tq_append(keys, values, packed_pages | None, table | None, window, slots, past, new_lengths | None, signs1, signs2, centroids,
//           boundaries, status | None, block_size, residual_len, bits, value_group, num_pages) -> True | None
PyObject* tq_append(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 18) return PyErr_Format(PyExc_TypeError, "tq_append takes 18 arguments");
  const at::Tensor *keys = tensor(args[0]), *values = tensor(args[1]);
  bool ok = keys != nullptr && values != nullptr;
  const at::Tensor* pages = optional_tensor(args[2], &ok);
  const at::Tensor* table = optional_tensor(args[3], &ok);
  const at::Tensor* window = tensor(args[4]);
  const at::Tensor* slots = tensor(args[5]);
  const at::Tensor* past = tensor(args[6]);
  const at::Tensor* fresh = optional_tensor(args[7], &ok);
  const at::Tensor* fixed[4];
  for (int i = 0; i < 4; ++i) {
    fixed[i] = tensor(args[8 + i]);
    ok = ok && fixed[i] != nullptr;
  }
  const at::Tensor* word = optional_tensor(args[12], &ok);
  int64_t n[5];  // block_size, residual_len, bits, value_group, num_pages
  if (!int_args(args + 13, 5, n)) return nullptr;
  int code = 0;
  if (!ok || window == nullptr || slots == nullptr || past == nullptr || !keys->is_cuda() || !plain(*keys, keys->device(), 4) ||
      !plain(*values, keys->device(), 4) || keys->stride(3) != 1 || keys->sizes() != values->sizes() ||
      keys->strides() != values->strides() || keys->scalar_type() != values->scalar_type() || keys->numel() == 0 ||
      window->dim() != 5 || window->scalar_type() != keys->scalar_type() || window->size(2) != keys->size(1) ||
      window->size(4) != keys->size(3) || !dtype_code(keys->scalar_type(), &code))
    Py_RETURN_NONE;
  const c10::Device device = keys->device();
  for (const at::Tensor* t : {pages, table, window, slots, past, fresh, fixed[0], fixed[1], fixed[2], fixed[3], word})
    if (!on(t, device)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  int status;
  {
    pybind11::gil_scoped_release unlocked;
    status = anna_tq_append(
        keys->data_ptr(), values->data_ptr(), keys->stride(0), keys->stride(1), keys->stride(2),
        static_cast<uint8_t*>(address(pages)), static_cast<const int32_t*>(address(table)),
        table == nullptr ? 0 : table->stride(0), nullptr, 0, address(window), static_cast<const int64_t*>(address(slots)),
        static_cast<const int64_t*>(address(past)), static_cast<int64_t*>(address(fresh)), floats(fixed[0]), floats(fixed[1]),
        floats(fixed[2]), floats(fixed[3]), (int)keys->size(0), (int)keys->size(1), (int)keys->size(2), (int)keys->size(3),
        (int)n[0], (int)n[1], (int)n[2], (int)n[3], n[4], table == nullptr ? 0 : table->size(1), code,
        static_cast<int32_t*>(address(word)), stream);
  }
  if (status != 0) return failed("anna_tq_append", status);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// paged_decode(query, key_pages, value_pages, page_table, visible_lengths, scaling, gate | None) -> output | None
PyObject* paged_decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 7) return PyErr_Format(PyExc_TypeError, "paged_decode takes 7 arguments");
  const at::Tensor* t[5];
  for (int i = 0; i < 5; ++i)
    if ((t[i] = tensor(args[i])) == nullptr) Py_RETURN_NONE;
  const at::Tensor &query = *t[0], &keys = *t[1], &values = *t[2], &table = *t[3], &lengths = *t[4];
  bool ok = true;
  const at::Tensor* gate = optional_tensor(args[6], &ok);
  const double scaling = PyFloat_AsDouble(args[5]);
  if (scaling == -1.0 && PyErr_Occurred()) return nullptr;
  int code = 0;
  if (!ok || !query.is_cuda() || !plain(query, query.device(), 4) || query.size(2) != 1 || query.stride(3) != 1 ||
      !dtype_code(query.scalar_type(), &code))
    Py_RETURN_NONE;
  const c10::Device device = query.device();
  if (!plain(keys, device, 4) || !plain(values, device, 4) || !plain(table, device, 2) || !plain(lengths, device, 1) ||
      keys.sizes() != values.sizes() || !keys.is_contiguous() || !values.is_contiguous() ||
      keys.scalar_type() != query.scalar_type() || values.scalar_type() != query.scalar_type() ||
      table.scalar_type() != at::kInt || lengths.scalar_type() != at::kLong || table.stride(1) != 1 || lengths.stride(0) != 1)
    Py_RETURN_NONE;
  const int64_t batch = query.size(0), heads = query.size(1), dim = query.size(3), kv_heads = keys.size(1),
                block = keys.size(2), max_blocks = table.size(1);
  if (keys.numel() == 0 || batch == 0 || heads == 0 || heads % kv_heads != 0 || dim != keys.size(3) || table.size(0) != batch ||
      lengths.size(0) != batch || max_blocks == 0)
    Py_RETURN_NONE;
  int64_t g_sb = 0, g_sh = 0;
  if (gate != nullptr) {
    if (gate->device() != device || gate->layout() != at::kStrided || gate->scalar_type() != query.scalar_type() ||
        gate->dim() < 3 || gate->size(0) != batch)
      Py_RETURN_NONE;
    if (gate->dim() == 4 && gate->sizes() == query.sizes() && gate->stride(3) == 1) {
      g_sb = gate->stride(0);
      g_sh = gate->stride(1);
    } else if (gate->dim() == 3 && gate->size(1) == 1 && gate->size(2) == heads * dim && gate->stride(2) == 1) {
      g_sb = gate->stride(0);
      g_sh = dim;
    } else {
      Py_RETURN_NONE;
    }
  }
  const c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  Scratch s;
  if (!scratch_of(query, reinterpret_cast<int64_t>(stream), kv_heads, max_blocks * block, 0, block, 0, &s)) return nullptr;
  at::Tensor out = at::empty(query.sizes(), query.options());
  int status;
  {
    pybind11::gil_scoped_release unlocked;
    status = anna_paged_gqa_decode(
        query.data_ptr(), query.stride(0), query.stride(1), keys.data_ptr(), values.data_ptr(),
        static_cast<const int32_t*>(table.data_ptr()), table.stride(0), static_cast<const int64_t*>(lengths.data_ptr()),
        address(gate), g_sb, g_sh, out.data_ptr(), heads * dim, dim, static_cast<float*>(s.stats.data_ptr()),
        static_cast<float*>(s.values.data_ptr()), s.capacity, 0, static_cast<int32_t*>(s.counters.data_ptr()), (int)batch,
        (int)heads, (int)kv_heads, (int)dim, (int)block, keys.size(0), max_blocks, (float)scaling, code, stream);
  }
  if (status != 0) return failed("paged_gqa_decode_fused", status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// prefill(query, keys, values, key_lengths | None, scaling, causal) -> output | None
PyObject* prefill(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 6) return PyErr_Format(PyExc_TypeError, "prefill takes 6 arguments");
  const at::Tensor* t[3];
  for (int i = 0; i < 3; ++i)
    if ((t[i] = tensor(args[i])) == nullptr) Py_RETURN_NONE;
  const at::Tensor &query = *t[0], &keys = *t[1], &values = *t[2];
  bool ok = true;
  const at::Tensor* lengths = optional_tensor(args[3], &ok);
  const double scaling = PyFloat_AsDouble(args[4]);
  if (scaling == -1.0 && PyErr_Occurred()) return nullptr;
  const int causal = PyObject_IsTrue(args[5]);
  if (causal < 0) return nullptr;
  int code = 0;
  if (!ok || !query.is_cuda() || !plain(query, query.device(), 4) || !dtype_code(query.scalar_type(), &code) ||
      code == ANNA_DTYPE_F32)
    Py_RETURN_NONE;
  const c10::Device device = query.device();
  const int64_t batch = query.size(0), heads = query.size(1), tokens = query.size(2), dim = query.size(3);
  if (!plain(keys, device, 4) || !plain(values, device, 4) || keys.sizes() != values.sizes() ||
      keys.strides() != values.strides() || keys.scalar_type() != query.scalar_type() ||
      values.scalar_type() != query.scalar_type() || keys.numel() == 0 || query.numel() == 0 || keys.size(0) != batch ||
      keys.size(3) != dim || heads % keys.size(1) != 0 || (dim != 64 && dim != 128 && dim != 256))
    Py_RETURN_NONE;
  if (lengths != nullptr && (!plain(*lengths, device, 1) || lengths->scalar_type() != at::kLong || lengths->size(0) != batch ||
                             lengths->stride(0) != 1))
    Py_RETURN_NONE;
  for (const at::Tensor* x : t) {  // what 16-byte copies need
    if (x->stride(3) != 1 || reinterpret_cast<uintptr_t>(x->data_ptr()) % 16 != 0) Py_RETURN_NONE;
    for (int i = 0; i < 3; ++i)
      if (x->stride(i) % 8 != 0) Py_RETURN_NONE;
  }
  const c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  at::Tensor out = at::empty(query.sizes(), query.options());
  int status;
  {
    pybind11::gil_scoped_release unlocked;
    status = anna_gqa_prefill(query.data_ptr(), query.stride(0), query.stride(1), query.stride(2), keys.data_ptr(),
                              values.data_ptr(), keys.stride(0), keys.stride(1), keys.stride(2),
                              static_cast<const int64_t*>(address(lengths)), out.data_ptr(), out.stride(0), out.stride(1),
                              out.stride(2), (int)batch, (int)heads, (int)keys.size(1), (int)tokens, keys.size(2), (int)dim,
                              (float)scaling, causal, code, stream);
  }
  if (status != 0) return failed("anna_gqa_prefill", status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// ---- uploads: small integer arrays go to the GPU through a ring of pinned host buffers, one asynchronous copy each ---------

// The buffers of one device.  They are handed out in turn, under the interpreter lock; a buffer whose last copy is still under way
// (sixteen uploads back: normally long done) is waited for without the lock, and is out of the ring for other threads meanwhile.
// A slot that has no event or too small a buffer gets it when its turn comes: a failure in between leaves the others as they are.
struct UploadRing {
  static constexpr int kSlots = 16;
  struct Slot {
    at::Tensor buffer;
    cudaEvent_t done = nullptr;
    bool taken = false;
  };
  Slot slots[kSlots];
  int64_t capacity = 8192;  // bytes of a buffer that is made now
  int next = 0;
};
std::map<int64_t, UploadRing>& upload_rings() {
  static auto* rings = new std::map<int64_t, UploadRing>();
  return *rings;
}

// Host copies for uploads that a graph captures: every replay reads its copy again, so the graph owns it.  One whose graph is gone
// serves a later capture (a graph's last reference may end on a thread of the driver, which may not free it).
struct CapturedBytes {
  void* data;
  size_t size;
};
std::mutex captured_free_lock;
std::vector<CapturedBytes*>& captured_free() {
  static auto* list = new std::vector<CapturedBytes*>();
  return *list;
}
void captured_give_back(void* bytes) {
  const std::lock_guard<std::mutex> lock(captured_free_lock);
  captured_free().push_back(static_cast<CapturedBytes*>(bytes));
}
CapturedBytes* captured_take(size_t size) {
  {
    const std::lock_guard<std::mutex> lock(captured_free_lock);
    auto& list = captured_free();
    for (size_t i = 0; i < list.size(); ++i) {
      if (list[i]->size < size) continue;
      CapturedBytes* found = list[i];
      list.erase(list.begin() + (std::ptrdiff_t)i);
      return found;
    }
  }
  size_t rounded = 256;
  while (rounded < size) rounded *= 2;
  void* data = nullptr;
  C10_CUDA_CHECK(cudaHostAlloc(&data, rounded, cudaHostAllocPortable));
  return new CapturedBytes{data, rounded};
}

// Copies the `bytes` at `data` to `out`, as part of the graph that `stream` captures.
void upload_captured(void* out, const void* data, size_t bytes, cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream, &status, &id, &graph, nullptr, nullptr));
  TORCH_CHECK(status == cudaStreamCaptureStatusActive, "anna_b200: upload under a graph capture that has failed");
  CapturedBytes* kept = captured_take(bytes);
  cudaUserObject_t owner = nullptr;
  const cudaError_t made = cudaUserObjectCreate(&owner, kept, captured_give_back, 1, cudaUserObjectNoDestructorSync);
  if (made != cudaSuccess) captured_give_back(kept);
  C10_CUDA_CHECK(made);
  const cudaError_t moved = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
  if (moved != cudaSuccess) (void)cudaUserObjectRelease(owner, 1);  // gives the copy back
  C10_CUDA_CHECK(moved);
  std::memcpy(kept->data, data, bytes);
  C10_CUDA_CHECK(cudaMemcpyAsync(out, kept->data, bytes, cudaMemcpyHostToDevice, stream));
}

// A tensor of `sizes` with the `bytes` at `data` on the device, ordered on its current stream (the device must be current).
at::Tensor upload_bytes(c10::DeviceIndex device, const void* data, int64_t bytes, at::IntArrayRef sizes, at::ScalarType type) {
  at::Tensor out = at::empty(sizes, at::TensorOptions().dtype(type).device(c10::Device(c10::kCUDA, device)));
  if (bytes == 0) return out;
  // waiting for an event and making pinned memory would end any thread's capture otherwise
  const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
    upload_captured(out.data_ptr(), data, (size_t)bytes, stream);
    return out;
  }
  UploadRing& ring = upload_rings()[device];
  UploadRing::Slot* slot = nullptr;
  while (slot == nullptr) {
    for (int i = 0; i < UploadRing::kSlots && slot == nullptr; ++i) {
      const int candidate = (ring.next + i) % UploadRing::kSlots;
      if (ring.slots[candidate].taken) continue;
      slot = &ring.slots[candidate];
      ring.next = (candidate + 1) % UploadRing::kSlots;
    }
    if (slot == nullptr) pybind11::gil_scoped_release others;  // as many threads wait for a buffer each
  }
  struct Taken {
    bool* flag;
    explicit Taken(bool* f) : flag(f) { *flag = true; }
    ~Taken() { *flag = false; }
  } taken(&slot->taken);
  if (slot->done == nullptr) {
    C10_CUDA_CHECK(cudaEventCreateWithFlags(&slot->done, cudaEventDisableTiming));
  } else if (cudaEventQuery(slot->done) != cudaSuccess) {
    (void)cudaGetLastError();
    pybind11::gil_scoped_release waiting;
    C10_CUDA_CHECK(cudaEventSynchronize(slot->done));
  }
  if (slot->buffer.numel() < bytes) {
    if (ring.capacity < bytes) ring.capacity = 2 * bytes;
    auto grow = [&](UploadRing::Slot& small) {
      if (small.buffer.numel() < ring.capacity)
        small.buffer = at::empty({ring.capacity}, at::TensorOptions().dtype(at::kByte).pinned_memory(true));
    };
    grow(*slot);
    // and those whose copies are done, so that the next uploads of this size find theirs
    for (UploadRing::Slot& other : ring.slots) {
      if (other.taken) continue;
      if (other.done == nullptr || cudaEventQuery(other.done) == cudaSuccess) grow(other);
      else (void)cudaGetLastError();
    }
  }
  std::memcpy(slot->buffer.data_ptr(), data, (size_t)bytes);
  C10_CUDA_CHECK(cudaMemcpyAsync(out.data_ptr(), slot->buffer.data_ptr(), (size_t)bytes, cudaMemcpyHostToDevice, stream));
  C10_CUDA_CHECK(cudaEventRecord(slot->done, stream));
  return out;
}

// Rows that are lists or tuples of ints and of one length, one after the other; false for all others.  Nothing here runs code of
// the objects (an __index__ could shorten the very lists that are being read).
bool plain_rows(PyObject* rows, std::vector<int64_t>* values, int64_t* count, int64_t* width) {
  if (!PyList_CheckExact(rows) && !PyTuple_CheckExact(rows)) return false;
  *count = PySequence_Fast_GET_SIZE(rows);
  for (Py_ssize_t r = 0; r < *count; ++r) {
    PyObject* row = PySequence_Fast_GET_ITEM(rows, r);
    if (!PyList_CheckExact(row) && !PyTuple_CheckExact(row)) return false;
    const Py_ssize_t entries = PySequence_Fast_GET_SIZE(row);
    if (r == 0) {
      *width = entries;
      values->reserve((size_t)(*count * entries));
    }
    if (entries != *width) return false;
    for (Py_ssize_t i = 0; i < entries; ++i) {
      PyObject* entry = PySequence_Fast_GET_ITEM(row, i);
      if (!PyLong_CheckExact(entry)) return false;
      int overflow = 0;
      values->push_back(PyLong_AsLongLongAndOverflow(entry, &overflow));
      if (overflow != 0) return false;
    }
  }
  return *count > 0;
}

// upload(device index, rows) -> int64 [len(rows), len(rows[0])] on the device | None
PyObject* upload(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2) return PyErr_Format(PyExc_TypeError, "upload(device, rows)");
  const long device = PyLong_AsLong(args[0]);
  if (device == -1 && PyErr_Occurred()) return nullptr;
  std::vector<int64_t> values;
  int64_t count = 0, width = 0;
  if (!plain_rows(args[1], &values, &count, &width)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  return THPVariable_Wrap(upload_bytes((c10::DeviceIndex)device, values.data(), (int64_t)values.size() * 8, {count, width}, at::kLong));
  END_HANDLE_TH_ERRORS
}

// upload_i32(device index, buffer), upload_i64(device index, buffer) -> the buffer's entries, flat, on the device | None unless it is
// contiguous and of that type
PyObject* upload_buffer(PyObject* const* args, Py_ssize_t nargs, at::ScalarType type) {
  HANDLE_TH_ERRORS
  if (nargs != 2) return PyErr_Format(PyExc_TypeError, "upload of a buffer: (device, buffer)");
  const long device = PyLong_AsLong(args[0]);
  if (device == -1 && PyErr_Occurred()) return nullptr;
  struct View {
    Py_buffer view{};
    bool held = false;
    ~View() {
      if (held) PyBuffer_Release(&view);
    }
  } buffer;
  buffer.held = PyObject_GetBuffer(args[1], &buffer.view, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) == 0;
  if (!buffer.held) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const char* format = buffer.view.format == nullptr ? "" : buffer.view.format;
  const bool fits = type == at::kInt ? std::strcmp(format, "i") == 0 : std::strcmp(format, "l") == 0 || std::strcmp(format, "q") == 0;
  if (!fits) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  return THPVariable_Wrap(upload_bytes((c10::DeviceIndex)device, buffer.view.buf, buffer.view.len,
                                       {(int64_t)(buffer.view.len / buffer.view.itemsize)}, type));
  END_HANDLE_TH_ERRORS
}
PyObject* upload_i32(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return upload_buffer(args, nargs, at::kInt); }
PyObject* upload_i64(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return upload_buffer(args, nargs, at::kLong); }

// tq_gather_dense(packed_pages | None, table | None, window, slots, lengths, signs1, signs2, centroids, max_len, block_size,
//                 residual_len, bits, value_group, num_pages) -> (keys, values) | None
PyObject* tq_gather_dense(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 14) return PyErr_Format(PyExc_TypeError, "tq_gather_dense takes 14 arguments");
  bool ok = true;
  const at::Tensor* pages = optional_tensor(args[0], &ok);
  const at::Tensor* table = optional_tensor(args[1], &ok);
  const at::Tensor* fixed[6];  // window, slots, lengths, signs1, signs2, centroids
  for (int i = 0; i < 6; ++i) {
    fixed[i] = tensor(args[2 + i]);
    ok = ok && fixed[i] != nullptr;
  }
  int64_t n[6];  // max_len, block_size, residual_len, bits, value_group, num_pages
  if (!int_args(args + 8, 6, n)) return nullptr;
  int code = 0;
  if (!ok || !fixed[0]->is_cuda() || !plain(*fixed[0], fixed[0]->device(), 5) || !dtype_code(fixed[0]->scalar_type(), &code) ||
      fixed[2]->dim() != 1 || fixed[2]->size(0) == 0 || fixed[1]->sizes() != fixed[2]->sizes() || n[0] <= 0)
    Py_RETURN_NONE;
  const c10::Device device = fixed[0]->device();
  for (const at::Tensor* t : fixed)
    if (!on(t, device)) Py_RETURN_NONE;
  if (!on(pages, device) || !on(table, device)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  const int64_t batch = fixed[2]->size(0), kv_heads = fixed[0]->size(2), dim = fixed[0]->size(4);
  at::Tensor keys = at::empty({batch, kv_heads, n[0], dim}, fixed[0]->options());
  at::Tensor values = at::empty(keys.sizes(), keys.options());
  int status;
  {
    pybind11::gil_scoped_release unlocked;
    status = anna_tq_gather_dense(
        static_cast<const uint8_t*>(address(pages)), static_cast<const int32_t*>(address(table)),
        table == nullptr ? 0 : table->stride(0), address(fixed[0]), static_cast<const int64_t*>(address(fixed[1])),
        static_cast<const int64_t*>(address(fixed[2])), floats(fixed[3]), floats(fixed[4]), floats(fixed[5]), keys.data_ptr(),
        values.data_ptr(), keys.stride(0), keys.stride(1), keys.stride(2), (int)batch, (int)kv_heads, (int)dim, (int)n[1],
        (int)n[2], (int)n[3], (int)n[4], n[5], table == nullptr ? 0 : table->size(1), n[0], code, stream);
  }
  if (status != 0) return failed("anna_tq_gather_dense", status);
  PyObject* pair = PyTuple_New(2);
  if (pair == nullptr) return nullptr;
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(keys)));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(values)));
  if (PyTuple_GET_ITEM(pair, 0) == nullptr || PyTuple_GET_ITEM(pair, 1) == nullptr) Py_CLEAR(pair);
  return pair;
  END_HANDLE_TH_ERRORS
}

// ---- page book: free pages are a list of ints, last in first out; owners are int32 counts by page id --------------------

struct Ints {  // a writable int32 buffer
  Py_buffer view{};
  bool held = false;
  explicit Ints(PyObject* obj) { held = PyObject_GetBuffer(obj, &view, PyBUF_WRITABLE | PyBUF_ND) == 0; }
  ~Ints() {
    if (held) PyBuffer_Release(&view);
  }
  int32_t* data() const { return static_cast<int32_t*>(view.buf); }
  Py_ssize_t size() const { return view.len / (Py_ssize_t)sizeof(int32_t); }
  Ints(const Ints&) = delete;
  Ints& operator=(const Ints&) = delete;
};

// The list itself, or a new one of plain ints where entries are other integers (numpy's); nullptr with an error set for
// anything that is no integer.  A new reference.
PyObject* plain_ints(PyObject* list) {
  const Py_ssize_t n = PyList_GET_SIZE(list);
  Py_ssize_t plain = 0;
  while (plain < n && PyLong_Check(PyList_GET_ITEM(list, plain))) ++plain;
  if (plain == n) {
    Py_INCREF(list);
    return list;
  }
  PyObject* ints = PyList_GetSlice(list, 0, n);
  for (Py_ssize_t i = plain; ints != nullptr && i < n; ++i) {
    PyObject* id = PyNumber_Index(PyList_GET_ITEM(ints, i));
    if (id == nullptr) Py_CLEAR(ints);
    else PyList_SetItem(ints, i, id);
  }
  return ints;
}
// of a plain int; -1, which is no page either, where it fits no Py_ssize_t
Py_ssize_t page_id(PyObject* list, Py_ssize_t i) {
  const Py_ssize_t id = PyLong_AsSsize_t(PyList_GET_ITEM(list, i));
  if (id == -1) PyErr_Clear();
  return id;
}

// take_pages(free, counts, count) -> the last `count` ids of `free`, last one first; they leave `free` with one owner each
PyObject* take_pages(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3 || !PyList_Check(args[0])) return PyErr_Format(PyExc_TypeError, "take_pages(list, counts, count)");
  PyObject* free_list = args[0];
  const Py_ssize_t have = PyList_GET_SIZE(free_list), count = PyLong_AsSsize_t(args[2]);
  if (count < 0 || count > have) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "take_pages: more pages than are free");
    return nullptr;
  }
  Ints counts(args[1]);
  PyObject* out = counts.held ? PyList_New(count) : nullptr;
  if (out == nullptr) return nullptr;
  bool ok = true;
  for (Py_ssize_t i = 0; ok && i < count; ++i) {
    PyObject* id = PyList_GET_ITEM(free_list, have - 1 - i);
    if (PyLong_CheckExact(id)) {
      Py_INCREF(id);
    } else {
      id = PyNumber_Index(id);
      ok = id != nullptr && PyList_GET_SIZE(free_list) == have;  // (an entry's __index__ may have done anything)
      if (!ok && !PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "take_pages: the free list has changed");
    }
    if (id != nullptr) PyList_SET_ITEM(out, i, id);
    if (!ok) break;
    const Py_ssize_t page = page_id(out, i);
    ok = page >= 0 && page < counts.size() && counts.data()[page] == 0;
    if (!ok)
      PyErr_Format(PyExc_RuntimeError, "Invariant violated: free list page %zd %s.", page,
                   page >= 0 && page < counts.size() ? "has non-zero refcount" : "does not exist");
  }
  for (Py_ssize_t i = 0; ok && i < count; ++i) counts.data()[page_id(out, i)] = 1;
  if (!ok || PyList_SetSlice(free_list, have - count, have, nullptr) != 0) {
    Py_DECREF(out);
    return nullptr;
  }
  return out;
}

// release_pages(ids, counts) -> (ids that lost their last owner, in order; pages that are no longer shared): every id loses
// one owner, ids without one are passed over
PyObject* release_pages(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2 || !PyList_Check(args[0])) return PyErr_Format(PyExc_TypeError, "release_pages(list, counts)");
  PyObject* ids = plain_ints(args[0]);
  if (ids == nullptr) return nullptr;
  Ints counts(args[1]);
  const Py_ssize_t n = PyList_GET_SIZE(ids);
  PyObject* freed = counts.held ? PyList_New(n) : nullptr;
  if (freed == nullptr) {
    Py_DECREF(ids);
    return nullptr;
  }
  Py_ssize_t last = 0, unshared = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const Py_ssize_t page = page_id(ids, i);
    if (page < 0 || page >= counts.size() || counts.data()[page] <= 0) continue;
    const int32_t left = --counts.data()[page];
    if (left == 1) ++unshared;
    if (left > 0) continue;
    PyObject* id = PyList_GET_ITEM(ids, i);
    Py_INCREF(id);
    PyList_SET_ITEM(freed, last++, id);
  }
  Py_DECREF(ids);
  if (last < n) {  // the rest of the new list is empty slots
    PyObject* part = PyList_GetSlice(freed, 0, last);
    Py_DECREF(freed);
    freed = part;
    if (freed == nullptr) return nullptr;
  }
  return Py_BuildValue("Nn", freed, unshared);
}

// copy_pages(ids, first, last, target): ids[first:last] of a list or another sequence to the same places of an int32 buffer
PyObject* copy_pages(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4) return PyErr_Format(PyExc_TypeError, "copy_pages(ids, first, last, target)");
  const Py_ssize_t first = PyLong_AsSsize_t(args[1]), last = PyLong_AsSsize_t(args[2]);
  if (PyErr_Occurred()) return nullptr;
  PyObject* ids = PySequence_Fast(args[0], "copy_pages: page ids must be a sequence");
  if (ids == nullptr) return nullptr;
  Ints target(args[3]);
  bool ok = target.held;
  if (ok && (first < 0 || last < first || last > PySequence_Fast_GET_SIZE(ids) || last > target.size())) {
    PyErr_SetString(PyExc_ValueError, "copy_pages: out of range");
    ok = false;
  }
  for (Py_ssize_t i = first; ok && i < last; ++i) {
    PyObject* obj = PySequence_Fast_GET_ITEM(ids, i);
    const long id = PyLong_AsLong(obj);
    target.data()[i] = (int32_t)id;
    if (id == (int32_t)id && id != -1 && PyLong_CheckExact(obj)) continue;
    ok = !(id == -1 && PyErr_Occurred());
    if (ok && id != (int32_t)id) {
      PyErr_SetString(PyExc_OverflowError, "copy_pages: page id does not fit 32 bits");
      ok = false;
    } else if (ok && PySequence_Fast_GET_SIZE(ids) < last) {  // an entry's __index__ may have shortened the list
      PyErr_SetString(PyExc_ValueError, "copy_pages: out of range");
      ok = false;
    }
  }
  Py_DECREF(ids);
  if (!ok) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"take_pages", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(take_pages)), METH_FASTCALL, nullptr},
    {"release_pages", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(release_pages)), METH_FASTCALL, nullptr},
    {"copy_pages", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(copy_pages)), METH_FASTCALL, nullptr},
    {"set_scratch_source", set_scratch_source, METH_O, nullptr},
    {"forget_scratch", forget_scratch, METH_NOARGS, nullptr},
    {"tq_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(tq_decode)), METH_FASTCALL, nullptr},
    {"tq_append", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(tq_append)), METH_FASTCALL, nullptr},
    {"paged_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(paged_decode)), METH_FASTCALL, nullptr},
    {"upload", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(upload)), METH_FASTCALL, nullptr},
    {"upload_i64", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(upload_i64)), METH_FASTCALL, nullptr},
    {"upload_i32", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(upload_i32)), METH_FASTCALL, nullptr},
    {"tq_gather_dense", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(tq_gather_dense)), METH_FASTCALL, nullptr},
    {"prefill", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(prefill)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_launch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launch() {
  PyObject* self = PyModule_Create(&module);
  if (self != nullptr && PyModule_AddStringConstant(self, "built_for", ANNA_BUILT_FOR) != 0) Py_CLEAR(self);
  return self;
}
