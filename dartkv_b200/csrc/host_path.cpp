// Per-call host path of the cache as a CPython extension: append and decode calls go from the Python tensor objects
// straight into the C ABI.  One generation step makes two such calls per layer, each of a few microseconds of GPU
// work, so what the host does per call decides the step time of small batches; reading a tensor's fields from
// Python and converting ctypes arguments cost 15-25 us per call, this file about one (B200 host, 128-token appends:
// 26 -> 15 us per call, the three kernel launches included).
//
// Every function answers "not for me" (kSlowPath / None) for anything out of the ordinary -- other devices, odd
// strides, wrong shapes, pools that have to grow -- before it launches anything; the Python code then takes its
// full path, which also raises the errors.

#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
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

void* stream_of(const at::Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// append(keys, values, desc, lifecycle_config, lifecycle_state, plan, nonfinite) -> return code or kSlowPath
PyObject* append(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) { PyErr_SetString(PyExc_TypeError, "append takes 7 arguments"); return nullptr; }
  if (!THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) return PyLong_FromLong(kSlowPath);
  const at::Tensor& k = THPVariable_Unpack(args[0]);
  const at::Tensor& v = THPVariable_Unpack(args[1]);
  auto* desc = static_cast<const dartkv_cache_desc*>(PyLong_AsVoidPtr(args[2]));
  auto* cfg = static_cast<const dartkv_lifecycle_config*>(PyLong_AsVoidPtr(args[3]));
  auto* state = static_cast<dartkv_lifecycle_state*>(PyLong_AsVoidPtr(args[4]));
  auto* plan = static_cast<dartkv_append_plan*>(PyLong_AsVoidPtr(args[5]));
  auto* nonfinite = static_cast<int32_t*>(PyLong_AsVoidPtr(args[6]));
  if (PyErr_Occurred()) return nullptr;
  if (k.dim() != 4 || v.dim() != 4 || k.sizes() != v.sizes() || k.scalar_type() != v.scalar_type() ||
      dtype_code(k.scalar_type()) != desc->dtype || !on_current_device(k) || v.device() != k.device() ||
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
  int rc;
  const void *kp = k.data_ptr(), *vp = v.data_ptr();
  void* stream = stream_of(k);
  const int chunk = (int)k.size(2);
  Py_BEGIN_ALLOW_THREADS
  rc = dartkv_cache_append_step(desc, cfg, state, kp, vp, chunk, stride[0], stride[1], stride[2], nullptr, nonfinite,
                                plan, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// decode(query, desc, workspace, workspace_bytes, query_heads, tokens, scale, flavour, row_start | None)
//   -> output tensor shaped like the query ([B,Hq,D] or [B,Hq,1,D]), a negative return code, or None (slow path)
PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 9) { PyErr_SetString(PyExc_TypeError, "decode takes 9 arguments"); return nullptr; }
  if (!THPVariable_Check(args[0])) Py_RETURN_NONE;
  const at::Tensor& q = THPVariable_Unpack(args[0]);
  auto* desc = static_cast<const dartkv_cache_desc*>(PyLong_AsVoidPtr(args[1]));
  void* workspace = PyLong_AsVoidPtr(args[2]);
  const long long workspace_bytes = PyLong_AsLongLong(args[3]);
  const long query_heads = PyLong_AsLong(args[4]);
  const long tokens = PyLong_AsLong(args[5]);
  const double scale = PyFloat_AsDouble(args[6]);
  const long flavour = PyLong_AsLong(args[7]);
  if (PyErr_Occurred()) return nullptr;
  const int64_t dims = q.dim();
  const int code = dtype_code(q.scalar_type());
  if ((dims != 3 && dims != 4) || code < 0 || !on_current_device(q) || q.size(0) != desc->batch ||
      q.size(1) != query_heads || q.size(dims - 1) != desc->head_dim || (dims == 4 && q.size(2) != 1) ||
      query_heads % desc->kv_heads != 0 || query_heads / desc->kv_heads > 4 || tokens < 1)
    Py_RETURN_NONE;
  const int32_t* row_start = nullptr;
  if (args[8] != Py_None) {
    if (!THPVariable_Check(args[8])) Py_RETURN_NONE;
    const at::Tensor& r = THPVariable_Unpack(args[8]);
    if (r.dim() != 1 || r.size(0) != desc->batch || r.scalar_type() != at::kInt || r.device() != q.device() ||
        !r.is_contiguous())
      Py_RETURN_NONE;
    row_start = r.data_ptr<int32_t>();
  }
  at::Tensor dense = q.is_contiguous() ? at::Tensor() : q.detach().contiguous();
  const void* qp = dense.defined() ? dense.data_ptr() : q.data_ptr();
  at::Tensor out = at::empty(q.sizes(), q.options().requires_grad(false).memory_format(at::MemoryFormat::Contiguous));
  void* op = out.data_ptr();
  void* stream = stream_of(q);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = dartkv_decode_attention_padded(desc, qp, code, (int)query_heads, (float)scale, (int)flavour, (int)tokens, row_start,
                                      workspace, workspace_bytes, op, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
}

PyMethodDef methods[] = {
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
