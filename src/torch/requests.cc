// One dense request from Python in one native call.
//
// A small request costs the GPU about 2 us and its launch and completion some 9; the Python
// statements and the ctypes conversion in front of them cost another 2.  This function checks the
// tensors, looks up the current stream and hands the request to the worker
// (ps_capi_bworker_request_on, src/capi/ps_nvl_c_api.h).
#include <ATen/cuda/CUDAContext.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include "ps/device/psdev.h"

namespace {

using RequestFn = int (*)(void*, void*, int, int, const uint64_t*, size_t, const void*, size_t,
                          void*, size_t, int, int);

// What is fixed for a declared tensor.
struct Target {
  RequestFn request;
  void* worker;
  const uint64_t* keys;
  size_t nkeys;
  int64_t n;
  at::ScalarType grad_type, out_type;
  size_t grad_size, out_size;
  void* grad;    // the tensor's own buffers
  void* weight;
  c10::DeviceIndex device;
};
constexpr const char* kName = "psb200.target";

// The address of `obj`'s values, or `own` for None; false with a Python error set.
bool values_of(PyObject* obj, const Target& t, at::ScalarType type, void* own, const char* wrong,
               void** at) {
  if (obj == Py_None) {
    *at = own;
    return true;
  }
  if (!THPVariable_Check(obj)) {
    PyErr_SetString(PyExc_TypeError, "a tensor or None is expected");
    return false;
  }
  const at::Tensor& x = THPVariable_Unpack(obj);
  if (x.numel() != t.n || x.scalar_type() != type || !x.is_contiguous()) {
    PyErr_SetString(PyExc_ValueError, wrong);
    return false;
  }
  *at = x.data_ptr();
  return true;
}

// request(target, push, pull, value, out, cmd, priority) -> timestamp, negative after an error
PyObject* request(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 7) {
    PyErr_SetString(PyExc_TypeError, "request takes 7 arguments");
    return nullptr;
  }
  auto* t = static_cast<Target*>(PyCapsule_GetPointer(args[0], kName));
  if (!t) return nullptr;
  const bool push = args[1] == Py_True, pull = args[2] == Py_True;
  void *vals = nullptr, *outs = nullptr;
  HANDLE_TH_ERRORS
  if (push && !values_of(args[3], *t, t->grad_type, t->grad,
                         "pushed values must be a contiguous tensor of the declared length and "
                         "gradient dtype", &vals))
    return nullptr;
  if (pull && !values_of(args[4], *t, t->out_type, t->weight,
                         "the output must be a contiguous tensor of the declared length and "
                         "weight dtype", &outs))
    return nullptr;
  const long cmd = PyLong_AsLong(args[5]), priority = PyLong_AsLong(args[6]);
  if (PyErr_Occurred()) return nullptr;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(t->device).stream();
  int ts;
  Py_BEGIN_ALLOW_THREADS
  ts = t->request(t->worker, stream, push, pull, t->keys, t->nkeys, vals,
                  push ? static_cast<size_t>(t->n) * t->grad_size : 0, outs,
                  pull ? static_cast<size_t>(t->n) * t->out_size : 0, static_cast<int>(cmd),
                  static_cast<int>(priority));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(ts);
  END_HANDLE_TH_ERRORS
}

// ---- keyed tables ----
using KeyedFn = int (*)(void*, void*, int, int, const uint64_t*, size_t, const void*, size_t, void*,
                        size_t, const int*, int*, int);
struct KeyedTarget {
  KeyedFn request;
  KeyedFn request_here;  // all arrays on the table's GPU
  void* worker;
  int64_t max_keys;
  bool var_len;
  c10::DeviceIndex device;
};
constexpr const char* kKeyedName = "psb200.keyed_target";

// A device tensor of `type`, or NULL for None; false with a Python error set.
bool device_tensor(PyObject* obj, at::ScalarType type, const char* what, const at::Tensor** x) {
  *x = nullptr;
  if (obj == Py_None) return true;
  if (!THPVariable_Check(obj)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor", what);
    return false;
  }
  const at::Tensor& t = THPVariable_Unpack(obj);
  if (!t.is_cuda() || !t.is_contiguous() || t.scalar_type() != type) {
    PyErr_Format(PyExc_ValueError, "%s must be a contiguous torch.%s tensor on the device", what,
                 type == at::kLong ? "int64" : type == at::kInt ? "int32" : "float32");
    return false;
  }
  *x = &t;
  return true;
}

// keyed_request(target, keys, vals, out, lens, lens_out) -> timestamp, negative after an error
PyObject* keyed_request(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 6) {
    PyErr_SetString(PyExc_TypeError, "keyed_request takes 6 arguments");
    return nullptr;
  }
  auto* t = static_cast<KeyedTarget*>(PyCapsule_GetPointer(args[0], kKeyedName));
  if (!t) return nullptr;
  HANDLE_TH_ERRORS
  const at::Tensor *keys, *vals, *out, *lens, *lens_out;
  if (!device_tensor(args[1], at::kLong, "keys", &keys) ||
      !device_tensor(args[2], at::kFloat, "vals", &vals) ||
      !device_tensor(args[3], at::kFloat, "out", &out) ||
      !device_tensor(args[4], at::kInt, "lens", &lens) ||
      !device_tensor(args[5], at::kInt, "lens_out", &lens_out))
    return nullptr;
  const char* wrong = nullptr;
  const int64_t n = keys ? keys->numel() : 0;
  if (!vals && !out) wrong = "nothing to do: give vals, out or both";
  else if (!keys) wrong = "a request names its keys";
  else if (n > t->max_keys) wrong = "more keys than max_keys";
  else if (vals && t->var_len && (!lens || lens->numel() != n))
    wrong = "a push to a table with lengths names one length per key";
  else if (!t->var_len && (lens || lens_out)) wrong = "this table holds fixed-width values";
  else if (lens_out && lens_out->numel() != n) wrong = "lens_out needs one entry per key";
  if (wrong) {
    PyErr_SetString(PyExc_ValueError, wrong);
    return nullptr;
  }
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(t->device).stream();
  const void* kp = keys->data_ptr();
  const void* vp = vals ? vals->data_ptr() : nullptr;
  void* op = out ? out->data_ptr() : nullptr;
  const int* lp = vals && lens ? static_cast<const int*>(lens->data_ptr()) : nullptr;
  int* lo = out && !vals && lens_out ? static_cast<int*>(lens_out->data_ptr()) : nullptr;
  const size_t vb = vals ? vals->numel() * 4 : 0, ob = out ? out->numel() * 4 : 0;
  auto here = [&](const at::Tensor* x) { return !x || x->get_device() == t->device; };
  const bool all = here(keys) && here(vals) && here(out) && here(lens) && here(lens_out);
  int ts;
  Py_BEGIN_ALLOW_THREADS
  ts = (all ? t->request_here : t->request)(
      t->worker, stream, vals != nullptr, out != nullptr, static_cast<const uint64_t*>(kp),
      static_cast<size_t>(n), vp, vb, op, ob, lp, lo, 0);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(ts);
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"keyed_request",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&keyed_request)), METH_FASTCALL,
     "keyed_request(target, keys, vals, out, lens, lens_out) -> timestamp"},
    {"request", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&request)), METH_FASTCALL,
     "request(target, push, pull, value, out, cmd, priority) -> timestamp"},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

void add_requests(py::module& m) {
  m.def("target", [](uint64_t fn, uint64_t worker, uint64_t keys, size_t nkeys, int64_t n,
                     py::object grad_type, py::object out_type, uint64_t grad, uint64_t weight,
                     int device) {
    auto type_of = [](const py::object& o) {
      TORCH_CHECK(THPDtype_Check(o.ptr()), "a dtype is expected");
      return reinterpret_cast<THPDtype*>(o.ptr())->scalar_type;
    };
    auto* t = new Target{reinterpret_cast<RequestFn>(fn), reinterpret_cast<void*>(worker),
                         reinterpret_cast<const uint64_t*>(keys), nkeys, n, type_of(grad_type),
                         type_of(out_type), 0, 0, reinterpret_cast<void*>(grad),
                         reinterpret_cast<void*>(weight), static_cast<c10::DeviceIndex>(device)};
    t->grad_size = c10::elementSize(t->grad_type);
    t->out_size = c10::elementSize(t->out_type);
    return py::capsule(t, kName, [](void* p) { delete static_cast<Target*>(p); });
  });
  m.def("keyed_target", [](uint64_t fn, uint64_t here_fn, uint64_t worker, int64_t max_keys,
                           bool var_len, int device) {
    auto* t = new KeyedTarget{reinterpret_cast<KeyedFn>(fn), reinterpret_cast<KeyedFn>(here_fn),
                              reinterpret_cast<void*>(worker), max_keys, var_len,
                              static_cast<c10::DeviceIndex>(device)};
    return py::capsule(t, kKeyedName, [](void* p) { delete static_cast<KeyedTarget*>(p); });
  });
  PyModule_AddFunctions(m.ptr(), kMethods);
}
