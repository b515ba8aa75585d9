// Per-call host path of the cache as a CPython extension: append and decode calls go from the Python tensor objects
// straight into the C ABI.  One generation step makes two such calls per layer, each of a few microseconds of GPU
// work, so what the host does per call decides the step time of small batches; reading a tensor's fields from
// Python and converting ctypes arguments cost 15-25 us per call, a call here 3 us for an append (one launch) and 7 us
// for a decode (two launches and the output tensor).
//
// Every function answers "not for me" (kSlowPath / None) for anything out of the ordinary -- other devices, odd
// strides, wrong shapes, pools that have to grow -- before it launches anything; the Python code then takes its
// full path, which also raises the errors.  HANDLE_TH_ERRORS turns a C++ exception (out of memory, a tensor without
// storage) into a Python one at every entry.

#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/dartkv_b200.h"

namespace {

constexpr long kSlowPath = -100;

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return DARTKV_F32;
    case at::kHalf: return DARTKV_F16;
    case at::kBFloat16: return DARTKV_BF16;
    default: return -1;
  }
}

bool on_current_device(const at::Tensor& t) {
  return t.is_cuda() && t.device().index() == c10::cuda::current_device();
}

// Device index of the cache's pools: the last argument of append() and decode().  A caller that leaves it out vouches
// that the tensors are on the cache's device.
long device_argument(PyObject* const* args, Py_ssize_t n, Py_ssize_t at, const at::Tensor& t) {
  return n > at ? PyLong_AsLong(args[at]) : (long)t.device().index();
}

// The interpreter stays unlocked as long as one of these lives.  Every launch runs so: one that waits for room in the queue must
// not stop the other Python threads.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
template <class Call>
auto unlocked(Call call) {
  const Unlocked scope;
  return call();
}
// the tensor itself where it is contiguous, else a copy
at::Tensor dense_of(const at::Tensor& t) {
  if (t.is_contiguous()) return t;
  const Unlocked scope;
  return t.detach().contiguous();
}

void* stream_of(const at::Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// append(keys, values, desc, lifecycle_config, lifecycle_state, plan, nonfinite[, device]) -> return code or kSlowPath
PyObject* append(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 && n != 8) { PyErr_SetString(PyExc_TypeError, "append takes 7 or 8 arguments"); return nullptr; }
  if (!THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) return PyLong_FromLong(kSlowPath);
  const at::Tensor& k = THPVariable_Unpack(args[0]);
  const at::Tensor& v = THPVariable_Unpack(args[1]);
  auto* desc = static_cast<const dartkv_cache_desc*>(PyLong_AsVoidPtr(args[2]));
  auto* cfg = static_cast<const dartkv_lifecycle_config*>(PyLong_AsVoidPtr(args[3]));
  auto* state = static_cast<dartkv_lifecycle_state*>(PyLong_AsVoidPtr(args[4]));
  auto* plan = static_cast<dartkv_append_plan*>(PyLong_AsVoidPtr(args[5]));
  auto* nonfinite = static_cast<int32_t*>(PyLong_AsVoidPtr(args[6]));
  const long device = device_argument(args, n, 7, k);
  if (PyErr_Occurred()) return nullptr;
  if (k.dim() != 4 || v.dim() != 4 || k.sizes() != v.sizes() || k.scalar_type() != v.scalar_type() ||
      dtype_code(k.scalar_type()) != desc->dtype || !on_current_device(k) || k.device().index() != device ||
      v.device() != k.device() ||
      k.size(0) != desc->batch || k.size(1) != desc->kv_heads || k.size(3) != desc->head_dim || k.size(2) < 1 ||
      k.size(2) > 32768)
    return PyLong_FromLong(kSlowPath);
  // one set of strides serves both tensors; the stride of a dimension of size one says nothing
  int64_t stride[3];
  for (int i = 0; i < 3; ++i) {
    stride[i] = k.stride(i);
    if (k.size(i) != 1 && v.stride(i) != stride[i]) return PyLong_FromLong(kSlowPath);
    if (k.size(i) == 1) stride[i] = 0;
  }
  if (k.stride(3) != 1 || v.stride(3) != 1) return PyLong_FromLong(kSlowPath);
  const void *kp = k.data_ptr(), *vp = v.data_ptr();
  void* stream = stream_of(k);
  const int chunk = (int)k.size(2);
  return PyLong_FromLong(unlocked([&] {
    return dartkv_cache_append_step(desc, cfg, state, kp, vp, chunk, stride[0], stride[1], stride[2], nullptr, nonfinite, plan, stream);
  }));
  END_HANDLE_TH_ERRORS
}

// decode(query, desc, workspace, workspace_bytes, query_heads, tokens, scale, flavour, row_start | None[, device[, stream]])
//   -> output tensor shaped like the query ([B,Hq,D] or [B,Hq,1,D]), a negative return code, or None (slow path)
// stream: the one the workspace belongs to; a call on another stream is not for this workspace.
PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 9 || n > 11) { PyErr_SetString(PyExc_TypeError, "decode takes 9 to 11 arguments"); return nullptr; }
  if (!THPVariable_Check(args[0])) Py_RETURN_NONE;
  const at::Tensor& q = THPVariable_Unpack(args[0]);
  auto* desc = static_cast<const dartkv_cache_desc*>(PyLong_AsVoidPtr(args[1]));
  void* workspace = PyLong_AsVoidPtr(args[2]);
  const long long workspace_bytes = PyLong_AsLongLong(args[3]);
  const long query_heads = PyLong_AsLong(args[4]);
  const long tokens = PyLong_AsLong(args[5]);
  const double scale = PyFloat_AsDouble(args[6]);
  const long flavour = PyLong_AsLong(args[7]);
  const long device = device_argument(args, n, 9, q);
  const void* owner = n > 10 ? PyLong_AsVoidPtr(args[10]) : nullptr;
  if (PyErr_Occurred()) return nullptr;
  const int64_t dims = q.dim();
  const int code = dtype_code(q.scalar_type());
  if ((dims != 3 && dims != 4) || code < 0 || !on_current_device(q) || q.device().index() != device ||
      q.size(0) != desc->batch || q.size(1) != query_heads || q.size(dims - 1) != desc->head_dim || (dims == 4 && q.size(2) != 1) ||
      query_heads % desc->kv_heads != 0 || tokens < 1)
    Py_RETURN_NONE;
  void* stream = stream_of(q);
  if (n > 10 && stream != owner) Py_RETURN_NONE;
  const long rep = query_heads / desc->kv_heads;
  if (rep > 4 && rep > dartkv_decode_rows_limit(desc, code, (int)flavour, (int)tokens)) Py_RETURN_NONE;
  const int32_t* row_start = nullptr;
  if (args[8] != Py_None) {
    if (!THPVariable_Check(args[8])) Py_RETURN_NONE;
    const at::Tensor& r = THPVariable_Unpack(args[8]);
    if (r.dim() != 1 || r.size(0) != desc->batch || r.scalar_type() != at::kInt || r.device() != q.device() ||
        !r.is_contiguous())
      Py_RETURN_NONE;
    row_start = r.data_ptr<int32_t>();
  }
  // the kernels read the query two channels at a time: a 16-bit view from an odd element on is copied too
  at::Tensor dense = dense_of(q);
  if ((uintptr_t)dense.data_ptr() % 4) dense = unlocked([&] { return q.detach().clone(); });
  const void* qp = dense.data_ptr();
  at::Tensor out = at::empty(q.sizes(), q.options().requires_grad(false).memory_format(at::MemoryFormat::Contiguous));
  void* op = out.data_ptr();
  const int rc = unlocked([&] {
    return (rep > 4 ? dartkv_decode_attention_rows : dartkv_decode_attention_padded)(
        desc, qp, code, (int)query_heads, (float)scale, (int)flavour, (int)tokens, row_start, workspace, workspace_bytes, op, stream);
  });
  if (rc != 0) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

at::ScalarType scalar_type(int code) {
  return code == DARTKV_F32 ? at::kFloat : code == DARTKV_F16 ? at::kHalf : at::kBFloat16;
}

// `count` integers of a one-dimensional tensor from element `first` on, without the dispatches of narrow() and select().
at::Tensor integers_of(const at::Tensor& all, int64_t first, int64_t count) {
  at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(all.storage()), all.key_set(), all.dtype());
  t.unsafeGetTensorImpl()->set_storage_offset(first);
  t.unsafeGetTensorImpl()->set_sizes_contiguous({count});
  return t;
}

// allocate(desc, device_index, key_pages, value_rows): the pools of a new cache, in the order of `kPoolNames` on the
// Python side, with the descriptor's pointers set; None when the device is not the current one.  Only the state words
// and the finite-input flag start at zero (one launch for both); everything else is written before it is read.  What a
// reorder replaces and what segments are views of is an allocation of its own each, so that none of them holds memory of
// another.  A new cache with its first append: 32.7 us of host time with at::empty, narrow() and a fill kernel, 24.8 so, 23.3 with
// the pools in three allocations.
PyObject* allocate(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4) { PyErr_SetString(PyExc_TypeError, "allocate takes 4 arguments"); return nullptr; }
  auto* d = static_cast<dartkv_cache_desc*>(PyLong_AsVoidPtr(args[0]));
  const long device = PyLong_AsLong(args[1]), pages = PyLong_AsLong(args[2]), rows = PyLong_AsLong(args[3]);
  if (PyErr_Occurred()) return nullptr;
  if (device != c10::cuda::current_device()) Py_RETURN_NONE;
  try {
    const int64_t b = d->batch, h = d->kv_heads, hd = d->head_dim, sinks = d->sink_tokens > 0 ? d->sink_tokens : 1;
    const auto dense = scalar_type(d->dtype), ints = at::kInt, bytes = at::kByte;
    const at::Device here(at::kCUDA, (c10::DeviceIndex)device);
    auto empty = [&](at::IntArrayRef shape, at::ScalarType type) { return at::detail::empty_cuda(shape, type, here, std::nullopt); };
    const int64_t second = (pages + 63) / 64 * 64;   // of the two columns of the page table: from a multiple of 256 bytes on, like the flag
    const at::Tensor words = empty({65}, ints), table = empty({second + pages}, ints);
    at::Tensor pools[] = {
        empty({b, h, sinks, hd}, dense), empty({b, h, sinks, hd}, dense),
        empty({b, h, d->ring_tokens, hd}, dense), empty({b, h, d->ring_tokens, hd}, dense),
        integers_of(words, 0, 32), integers_of(words, 64, 1),
        empty({b, h, pages, d->key_page_bytes}, bytes), integers_of(table, 0, pages), integers_of(table, second, pages),
        empty({b, h, rows, d->value_row_bytes}, bytes),
        empty({b, h, rows, 2, d->value_groups}, scalar_type(d->md_dtype))};
    d->k_sink = pools[0].data_ptr(); d->v_sink = pools[1].data_ptr();
    d->k_ring = pools[2].data_ptr(); d->v_ring = pools[3].data_ptr();
    d->state = (int32_t*)pools[4].data_ptr();
    d->k_pages = (uint8_t*)pools[6].data_ptr();
    d->page_start = (int32_t*)pools[7].data_ptr(); d->page_tokens = (int32_t*)pools[8].data_ptr();
    d->v_codes = (uint8_t*)pools[9].data_ptr(); d->v_meta = pools[10].data_ptr();
    d->max_key_pages = (int32_t)pages; d->max_value_tokens = (int32_t)rows;
    auto* flag = (int32_t*)pools[5].data_ptr();
    void* stream = stream_of(pools[4]);
    if (unlocked([&] { return dartkv_cache_clear(d, flag, stream); }) != 0) Py_RETURN_NONE;   // Python allocates again, or raises
    constexpr int kPools = sizeof(pools) / sizeof(pools[0]);
    PyObject* out = PyTuple_New(kPools);
    if (!out) return nullptr;
    for (int i = 0; i < kPools; ++i) PyTuple_SET_ITEM(out, i, THPVariable_Wrap(pools[i]));
    return out;
  } catch (const c10::OutOfMemoryError&) {
    Py_RETURN_NONE;   // the Python path allocates the same pools and raises torch's own error
  }
  END_HANDLE_TH_ERRORS
}

// scratch(bytes, device_index): decode scratch with its first 16 bytes (status word and counters) zero, the rest as it
// comes; None when the device is not the current one.
PyObject* scratch(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) { PyErr_SetString(PyExc_TypeError, "scratch takes 2 arguments"); return nullptr; }
  const int64_t bytes = PyLong_AsLongLong(args[0]);
  const long device = PyLong_AsLong(args[1]);
  if (PyErr_Occurred()) return nullptr;
  if (bytes < 16 || device != c10::cuda::current_device()) Py_RETURN_NONE;
  at::Tensor buffer = at::empty({bytes}, at::TensorOptions().dtype(at::kByte).device(at::Device(at::kCUDA, (c10::DeviceIndex)device)));
  void *at = buffer.data_ptr(), *stream = stream_of(buffer);
  const cudaError_t err = unlocked([&] { return cudaMemsetAsync(at, 0, 16, (cudaStream_t)stream); });
  if (err != cudaSuccess) {
    PyErr_Format(PyExc_RuntimeError, "CUDA error while clearing decode scratch: %s", cudaGetErrorString(err));
    return nullptr;
  }
  return THPVariable_Wrap(std::move(buffer));
  END_HANDLE_TH_ERRORS
}

// Finite-input flag of a synchronous call: one pinned word per thread that the kernels write through its device
// mapping.  Such a call ends with a wait for its own stream anyway; the word saves the fill kernel before it and the
// copy after it.
struct HostFlag {
  int32_t* word = nullptr;
  HostFlag() {
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) word = static_cast<int32_t*>(p);
  }
  ~HostFlag() {
    if (word) cudaFreeHost(word);
  }
};
int32_t* host_flag() {
  thread_local HostFlag flag;
  if (flag.word) *reinterpret_cast<volatile int32_t*>(flag.word) = 0;
  return flag.word;
}

// What a call with a finite-input check returns: the tuple, a return code, or False where the input was not finite.
PyObject* finish(PyObject* tuple, int rc, const int32_t* flag, void* stream) {
  if (rc == 0 && flag) {
    const cudaError_t err = unlocked([&] { return cudaStreamSynchronize((cudaStream_t)stream); });
    if (err != cudaSuccess) {
      Py_DECREF(tuple);
      PyErr_Format(PyExc_RuntimeError, "CUDA error while waiting for the finite-input check: %s", cudaGetErrorString(err));
      return nullptr;
    }
    if (*reinterpret_cast<const volatile int32_t*>(flag)) {
      Py_DECREF(tuple);
      Py_RETURN_FALSE;
    }
  }
  if (rc != 0) {
    Py_DECREF(tuple);
    return PyLong_FromLong(rc);
  }
  return tuple;
}

PyObject* tensors(std::initializer_list<at::Tensor> list) {
  PyObject* out = PyTuple_New((Py_ssize_t)list.size());
  Py_ssize_t i = 0;
  for (const at::Tensor& t : list) PyTuple_SET_ITEM(out, i++, THPVariable_Wrap(t));
  return out;
}

// get(desc, tokens, device_index) -> (keys, values): the whole cache materialized; None when the device is not the current one.
PyObject* get(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3) { PyErr_SetString(PyExc_TypeError, "get takes 3 arguments"); return nullptr; }
  auto* d = static_cast<const dartkv_cache_desc*>(PyLong_AsVoidPtr(args[0]));
  const int64_t tokens = PyLong_AsLongLong(args[1]);
  const long device = PyLong_AsLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  if (device != c10::cuda::current_device()) Py_RETURN_NONE;
  const auto options = at::TensorOptions().dtype(scalar_type(d->dtype)).device(at::Device(at::kCUDA, (c10::DeviceIndex)device));
  at::Tensor keys = at::empty({d->batch, d->kv_heads, tokens, d->head_dim}, options), values = at::empty(keys.sizes(), options);
  void *kp = keys.data_ptr(), *vp = values.data_ptr(), *stream = stream_of(keys);
  const int rc = unlocked([&] { return dartkv_cache_materialize_both(d, 0, (int32_t)tokens, DARTKV_DEQUANT_PER_OP, kp, vp, d->dtype, stream); });
  if (rc != 0) return PyLong_FromLong(rc);
  return tensors({keys, values});
  END_HANDLE_TH_ERRORS
}

// the shape in a Python tuple of integers; false when it is not one
bool shape_of(PyObject* tuple, at::SmallVector<int64_t, 6>& shape) {
  if (!PyTuple_Check(tuple)) return false;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(tuple); ++i) {
    shape.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(tuple, i)));
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
  }
  return true;
}

// dequantize(values, scale, zero, original shape, axis, bits, group, flavour, output dtype code) -> tensor
PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9) { PyErr_SetString(PyExc_TypeError, "dequantize takes 9 arguments"); return nullptr; }
  at::SmallVector<int64_t, 6> shape;
  for (int i = 0; i < 3; ++i)
    if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
  const at::Tensor &values_given = THPVariable_Unpack(args[0]), &scale_given = THPVariable_Unpack(args[1]), &zero_given = THPVariable_Unpack(args[2]);
  if (!shape_of(args[3], shape)) Py_RETURN_NONE;
  int64_t axis = PyLong_AsLongLong(args[4]);
  const int bits = (int)PyLong_AsLong(args[5]);
  const int64_t group = PyLong_AsLongLong(args[6]);
  const int flavour = (int)PyLong_AsLong(args[7]), code = (int)PyLong_AsLong(args[8]);
  if (PyErr_Occurred()) return nullptr;
  const int64_t dims = (int64_t)shape.size();
  if (axis < 0) axis += dims;
  const int md = dtype_code(scale_given.scalar_type());
  if (code < DARTKV_F32 || code > DARTKV_BF16 || md < 0 || zero_given.scalar_type() != scale_given.scalar_type() || axis < 0 || axis >= dims ||
      group < 1 || group > INT32_MAX || values_given.scalar_type() != at::kByte || !on_current_device(values_given) ||
      !on_current_device(scale_given) || !on_current_device(zero_given))
    Py_RETURN_NONE;
  const at::Tensor values = dense_of(values_given), scale = dense_of(scale_given), zero = dense_of(zero_given);
  int64_t outer = 1, inner = 1;
  for (int64_t i = 0; i < axis; ++i) outer *= shape[i];
  for (int64_t i = axis + 1; i < dims; ++i) inner *= shape[i];
  const int64_t len = shape[axis];
  at::Tensor out = at::empty(shape, values.options().dtype(scalar_type(code)).requires_grad(false));
  const void *vp = values.data_ptr(), *sp = scale.data_ptr(), *zp = zero.data_ptr();
  void *op = out.data_ptr(), *stream = stream_of(values);
  const int rc = unlocked([&] {
    return dartkv_dequantize((const uint8_t*)vp, sp, zp, md, outer, len, inner, bits, (int)group, flavour, op, code, len * inner, inner, 1, stream);
  });
  if (rc != 0) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// dequantize_mixed(low, high, indices, scale, zero, original shape, group, flavour, output dtype code) -> tensor
PyObject* dequantize_mixed(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9) { PyErr_SetString(PyExc_TypeError, "dequantize_mixed takes 9 arguments"); return nullptr; }
  at::SmallVector<int64_t, 6> shape;
  for (int i = 0; i < 5; ++i)
    if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
  const at::Tensor* given[5];
  for (int i = 0; i < 5; ++i) given[i] = &THPVariable_Unpack(args[i]);
  if (!shape_of(args[5], shape) || shape.size() != 4) Py_RETURN_NONE;
  const int64_t group = PyLong_AsLongLong(args[6]);
  const int flavour = (int)PyLong_AsLong(args[7]), code = (int)PyLong_AsLong(args[8]);
  if (PyErr_Occurred()) return nullptr;
  const int md = dtype_code(given[3]->scalar_type());
  if (code < DARTKV_F32 || code > DARTKV_BF16 || md < 0 || given[4]->scalar_type() != given[3]->scalar_type() || group < 1 || group > INT32_MAX ||
      given[0]->scalar_type() != at::kByte || given[1]->scalar_type() != at::kByte || given[2]->scalar_type() != at::kInt || given[2]->dim() < 1)
    Py_RETURN_NONE;
  for (const at::Tensor* t : given)
    if (!on_current_device(*t)) Py_RETURN_NONE;
  const at::Tensor low = dense_of(*given[0]), high = dense_of(*given[1]), index = dense_of(*given[2]), scale = dense_of(*given[3]),
                   zero = dense_of(*given[4]);
  const int64_t promoted = index.size(-1);
  at::Tensor out = at::empty(shape, low.options().dtype(scalar_type(code)).requires_grad(false));
  const void *lp = low.data_ptr(), *hp = promoted ? high.data_ptr() : nullptr, *ip = promoted ? index.data_ptr() : nullptr;
  const void *sp = scale.data_ptr(), *zp = zero.data_ptr();
  void *op = out.data_ptr(), *stream = stream_of(low);
  const int rc = unlocked([&] {
    return dartkv_dequantize_key_mixed((const uint8_t*)lp, (const uint8_t*)hp, (const int32_t*)ip, sp, zp, md, shape[0] * shape[1], shape[2], shape[3],
                                       (int)group, (int)promoted, flavour, op, code, stream);
  });
  if (rc != 0) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// quantize(data, bits, group, axis, metadata dtype code (-1: the data's own, or fp32), division, check) -> (values, scale, zero);
// data of any strides, as for the other functional calls: a strided one that came back to Python to be copied there would cross twice
PyObject* quantize(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7) { PyErr_SetString(PyExc_TypeError, "quantize takes 7 arguments"); return nullptr; }
  if (!THPVariable_Check(args[0])) Py_RETURN_NONE;
  for (int i = 1; i < 7; ++i)
    if (!PyLong_Check(args[i])) Py_RETURN_NONE;
  const at::Tensor& given = THPVariable_Unpack(args[0]);
  const int64_t bits_asked = PyLong_AsLongLong(args[1]);
  const int64_t group = PyLong_AsLongLong(args[2]);
  int64_t axis = PyLong_AsLongLong(args[3]);
  int md = (int)PyLong_AsLong(args[4]);
  const int division = (int)PyLong_AsLong(args[5]), wanted = (int)PyLong_AsLong(args[6]);
  if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }   // a number that no C integer holds
  const int code = dtype_code(given.scalar_type());
  if (code < 0 || !on_current_device(given) || given.numel() == 0 || group < 1 || group > INT32_MAX || md < -1 || division < 0 ||
      (bits_asked != 2 && bits_asked != 4 && bits_asked != 8) || axis < -given.dim() || axis >= given.dim())
    Py_RETURN_NONE;
  const at::Tensor x = dense_of(given);
  const int bits = (int)bits_asked;
  if (axis < 0) axis += x.dim();
  if (md < 0) md = code;   // fp16 and bf16 keep their own, fp32 data fp32
  int64_t outer = 1, inner = 1;
  at::SmallVector<int64_t, 6> shape;
  for (int64_t i = 0; i < x.dim(); ++i) {
    if (i < axis) outer *= x.size(i);
    if (i > axis) inner *= x.size(i);
    if (i != axis) shape.push_back(x.size(i));
  }
  const int64_t len = x.size(axis), groups = (len + group - 1) / group, vpb = 8 / bits;
  shape.push_back((groups * group + vpb - 1) / vpb);
  const auto options = x.options().requires_grad(false);
  at::Tensor values = at::empty(shape, options.dtype(at::kByte));
  shape.back() = groups;
  at::Tensor scale = at::empty(shape, options.dtype(scalar_type(md))), zero = at::empty(shape, options.dtype(scalar_type(md)));
  int32_t* flag = wanted ? host_flag() : nullptr;
  if (wanted && !flag) Py_RETURN_NONE;
  void* stream = stream_of(x);
  const void* xp = x.data_ptr();
  void *vp = values.data_ptr(), *sp = scale.data_ptr(), *zp = zero.data_ptr();
  const int rc = unlocked([&] {
    return dartkv_quantize(xp, code, outer, len, inner, len * inner, inner, 1, bits, (int)group, md, division, (uint8_t*)vp, sp, zp, flag, stream);
  });
  return finish(tensors({values, scale, zero}), rc, flag, stream);
  END_HANDLE_TH_ERRORS
}

// quantize_mixed(keys, group, promoted count, metadata dtype code, indices | None, check)
//   -> (low, high, indices, scale, zero); keys [B,H,T,D], indices int32 contiguous
PyObject* quantize_mixed(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6) { PyErr_SetString(PyExc_TypeError, "quantize_mixed takes 6 arguments"); return nullptr; }
  if (!THPVariable_Check(args[0])) Py_RETURN_NONE;
  const at::Tensor& given = THPVariable_Unpack(args[0]);
  const int64_t group = PyLong_AsLongLong(args[1]), count = PyLong_AsLongLong(args[2]);
  const int md = (int)PyLong_AsLong(args[3]), wanted = (int)PyLong_AsLong(args[5]);
  if (PyErr_Occurred()) return nullptr;
  const int code = dtype_code(given.scalar_type());
  if (code < 0 || !on_current_device(given) || given.dim() != 4 || given.numel() == 0 || group > INT32_MAX) Py_RETURN_NONE;
  const at::Tensor k = dense_of(given);
  const int64_t b = k.size(0), h = k.size(1), t = k.size(2), d = k.size(3), groups = (t + group - 1) / group, packed = (group + 3) / 4;
  const auto options = k.options().requires_grad(false);
  void* stream = stream_of(k);
  at::Tensor index;
  int rc = 0;
  if (args[4] != Py_None) {
    if (!THPVariable_Check(args[4])) Py_RETURN_NONE;
    index = THPVariable_Unpack(args[4]);
    if (index.scalar_type() != at::kInt || !index.is_contiguous() || !on_current_device(index)) Py_RETURN_NONE;
  } else {
    index = at::empty({b, h, count}, options.dtype(at::kInt));
    const void* kp = k.data_ptr();
    auto* ip = (int32_t*)index.data_ptr();
    auto promote = [&](void* scores) {
      return unlocked([&] { return dartkv_promote_channels(kp, code, b * h, t, d, t * d, d, (int)count, scores, ip, stream); });
    };
    rc = promote(nullptr);   // enough where one launch does it
    if (rc == DARTKV_ELIMIT) rc = promote(at::empty({b, h, d}, options).data_ptr());
    if (rc) return PyLong_FromLong(rc);
  }
  const int64_t promoted = index.size(-1);
  at::Tensor low = at::empty({b, h, d, groups, packed}, options.dtype(at::kByte));
  at::Tensor high = at::empty({b, h, promoted, groups, packed}, options.dtype(at::kByte));
  at::Tensor scale = at::empty({b, h, d, groups}, options.dtype(scalar_type(md)));
  at::Tensor zero = at::empty({b, h, d, groups}, options.dtype(scalar_type(md)));
  int32_t* flag = wanted ? host_flag() : nullptr;
  if (wanted && !flag) Py_RETURN_NONE;
  const void *kp = k.data_ptr(), *ip = promoted ? index.data_ptr() : nullptr;
  void *lp = low.data_ptr(), *hp = promoted ? high.data_ptr() : nullptr, *sp = scale.data_ptr(), *zp = zero.data_ptr();
  rc = unlocked([&] {
    return dartkv_quantize_key_mixed(kp, code, b * h, t, d, t * d, d, (int)group, (const int32_t*)ip, (int)promoted, md, (uint8_t*)lp, (uint8_t*)hp,
                                     sp, zp, flag, stream);
  });
  return finish(tensors({low, high, index, scale, zero}), rc, flag, stream);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"get", (PyCFunction)(void (*)(void))get, METH_FASTCALL, "keys and values of a whole cache"},
    {"dequantize", (PyCFunction)(void (*)(void))dequantize, METH_FASTCALL, "group-wise dequantizer"},
    {"dequantize_mixed", (PyCFunction)(void (*)(void))dequantize_mixed, METH_FASTCALL, "mixed key dequantizer"},
    {"quantize", (PyCFunction)(void (*)(void))quantize, METH_FASTCALL, "group-wise quantizer"},
    {"quantize_mixed", (PyCFunction)(void (*)(void))quantize_mixed, METH_FASTCALL, "mixed key quantizer"},
    {"allocate", (PyCFunction)(void (*)(void))allocate, METH_FASTCALL, "the pools of a new cache"},
    {"scratch", (PyCFunction)(void (*)(void))scratch, METH_FASTCALL, "decode scratch"},
    {"append", (PyCFunction)(void (*)(void))append, METH_FASTCALL, "one append step of a cache"},
    {"decode", (PyCFunction)(void (*)(void))decode, METH_FASTCALL, "one decode attention call on a cache"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dartkv_host", "host path of the packed KV cache", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dartkv_host(void) {
  PyObject* m = PyModule_Create(&module);
  if (m) PyModule_AddIntConstant(m, "SLOW_PATH", kSlowPath);
  return m;
}
