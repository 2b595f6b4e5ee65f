// Native forms of the Python calls whose kernels take a few microseconds: argument checks, output
// allocation, the current stream and the library call in one function each.  A Python statement
// costs about 0.1 us and a ctypes call with a dozen arguments 1.5 us; a launch costs 2.5 us.
#include <ATen/ATen.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/GradMode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include "ps/device/psdev.h"

namespace {

using GemmFn = int (*)(const void*, const void*, void*, int64_t, int64_t, int64_t, int, uint64_t,
                       void*);
using PullGemmFn = int (*)(const psdev_world_t*, const psdev_table_t*, int64_t, const void*, void*,
                           int64_t, int64_t, int64_t, int, int, uint64_t, void*);
using DenseFn = int (*)(const psdev_world_t*, const psdev_table_t*, int, int64_t, int64_t,
                        const psdev_opt_t*, int, int, uint64_t, int, void*);
using SparseFn = int (*)(const psdev_world_t*, const psdev_sparse_t*, int64_t, const uint64_t*,
                         const float*, int64_t, const int32_t*, float*, int64_t, int32_t*, void*);

using UniqueBytesFn = size_t (*)(int64_t, int);
using UniqueSortFn = int (*)(const uint64_t*, const float*, int64_t, int, void*, size_t, int64_t*,
                             void*);
using UniqueWriteFn = int (*)(const void*, int64_t, int, int64_t, uint64_t*, float*, void*);

// (time limits wrap like a C integer: a negative one is a very long one)
template <typename T>
T address(PyObject* o) {
  return reinterpret_cast<T>(PyLong_AsUnsignedLongLong(o));
}
cudaStream_t stream_on(c10::DeviceIndex device) {
  return c10::cuda::getCurrentCUDAStream(device).stream();
}
// A launch may wait for room in the stream: other Python threads run meanwhile.
template <typename F>
int without_gil(F&& f) {
  py::gil_scoped_release no_gil;  // (taken back on the way of an exception as well)
  return f();
}
bool is_bf16(PyObject* o) {
  return THPVariable_Check(o) && THPVariable_Unpack(o).scalar_type() == at::kBFloat16;
}
// `out`, or a new tensor with the leading sizes of `x` and `cols` columns.
at::Tensor output_for(PyObject* out, const at::Tensor& x, int64_t cols) {
  if (out != Py_None) return THPVariable_Unpack(out);
  at::DimVector sizes(x.sizes());
  sizes.back() = cols;
  return at::empty(sizes, x.options().requires_grad(false));
}

// linear(fn, x, w, out, num_ctas, timeout_ns) -> tensor, or the library's error code
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "linear takes 6 arguments");
  HANDLE_TH_ERRORS
  bool ok = is_bf16(a[1]) && is_bf16(a[2]) && (a[3] == Py_None || THPVariable_Check(a[3]));
  if (ok) {
    const at::Tensor &x = THPVariable_Unpack(a[1]), &w = THPVariable_Unpack(a[2]);
    ok = x.is_cuda() && w.is_cuda() && x.is_contiguous() && w.is_contiguous() && x.dim() > 0 &&
         w.dim() > 0 && x.size(-1) == w.size(-1) &&
         (a[3] == Py_None || THPVariable_Unpack(a[3]).is_cuda());
  }
  if (!ok) {
    PyErr_SetString(PyExc_AssertionError,
                    "x and w must be contiguous bf16 tensors on the device whose last sizes agree, "
                    "and the output must be on the device");
    return nullptr;
  }
  const at::Tensor &x = THPVariable_Unpack(a[1]), &w = THPVariable_Unpack(a[2]);
  const int64_t K = x.size(-1), M = K ? x.numel() / K : 0, N = w.size(0);
  at::Tensor out = output_for(a[3], x, N);
  const long ctas = PyLong_AsLong(a[4]);
  const uint64_t timeout = PyLong_AsUnsignedLongLongMask(a[5]);
  const auto fn = address<GemmFn>(a[0]);
  if (PyErr_Occurred()) return nullptr;
  const int rc = without_gil([&] {
    return fn(x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, static_cast<int>(ctas), timeout,
              stream_on(x.get_device()));
  });
  if (rc) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// pull_linear(fn, world, table, w_offset, n_out, x, out, copy_ctas, num_ctas, timeout_ns)
PyObject* pull_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10) return PyErr_Format(PyExc_TypeError, "pull_linear takes 10 arguments");
  HANDLE_TH_ERRORS
  if (!is_bf16(a[5]) || !THPVariable_Unpack(a[5]).is_contiguous() ||
      THPVariable_Unpack(a[5]).dim() == 0 || !THPVariable_Unpack(a[5]).is_cuda() ||
      (a[6] != Py_None &&
       !(THPVariable_Check(a[6]) && THPVariable_Unpack(a[6]).is_cuda()))) {
    PyErr_SetString(PyExc_AssertionError,
                    "x must be a contiguous bf16 tensor on the device, like the output");
    return nullptr;
  }
  const at::Tensor& x = THPVariable_Unpack(a[5]);
  const int64_t K = x.size(-1), M = K ? x.numel() / K : 0, N = PyLong_AsLongLong(a[4]);
  const int64_t off = PyLong_AsLongLong(a[3]);
  const long copy = PyLong_AsLong(a[7]), ctas = PyLong_AsLong(a[8]);
  const uint64_t timeout = PyLong_AsUnsignedLongLongMask(a[9]);
  const auto fn = address<PullGemmFn>(a[0]);
  const auto* world = address<const psdev_world_t*>(a[1]);
  const auto* table = address<const psdev_table_t*>(a[2]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor out = output_for(a[6], x, N);
  const int rc = without_gil([&] {
    return fn(world, table, off, x.data_ptr(), out.data_ptr(), M, N, K, static_cast<int>(copy),
              static_cast<int>(ctas), timeout, stream_on(x.get_device()));
  });
  if (rc) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// Whether what is done to `t` is followed: by a graph, a tangent or a transform of torch.func.
bool followed(const at::Tensor& t) {
  return (t.requires_grad() && c10::GradMode::is_enabled()) || at::isTensorSubclassLike(t) ||
         t._fw_grad(/*level=*/0).defined();
}

// unique_sum(bytes_fn, sort_fn, write_fn, keys, vals, key_bits) -> (keys, sums), None where this
// form does not apply (other types; a key of more than key_bits bits), or an error code
PyObject* unique_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "unique_sum takes 6 arguments");
  HANDLE_TH_ERRORS
  const long bits = PyLong_AsLong(a[5]);
  const auto bytes_fn = address<UniqueBytesFn>(a[0]);
  const auto sort_fn = address<UniqueSortFn>(a[1]);
  const auto write_fn = address<UniqueWriteFn>(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (!THPVariable_Check(a[3]) || !THPVariable_Check(a[4])) Py_RETURN_NONE;
  const at::Tensor &k_in = THPVariable_Unpack(a[3]), &v_in = THPVariable_Unpack(a[4]);
  const int64_t count = k_in.numel();
  if (k_in.scalar_type() != at::kLong || v_in.scalar_type() != at::kFloat || k_in.dim() != 1 ||
      v_in.dim() != 1 || v_in.numel() != count || count <= 0 || count >= (int64_t{1} << 30) ||
      !k_in.is_cuda() || v_in.device() != k_in.device() || followed(v_in) ||
      at::isTensorSubclassLike(k_in) || v_in.is_neg())
    Py_RETURN_NONE;
  const at::Tensor k = k_in.contiguous(), v = v_in.contiguous();
  void* stream = stream_on(k.get_device());
  const size_t bytes = bytes_fn(count, static_cast<int>(bits));
  const auto plain = k.options().requires_grad(false);
  at::Tensor scratch = at::empty({static_cast<int64_t>(bytes)}, plain.dtype(at::kByte));
  int64_t unique = 0;
  int rc = without_gil([&] {
    return sort_fn(static_cast<const uint64_t*>(k.data_ptr()),
                   static_cast<const float*>(v.data_ptr()), count, static_cast<int>(bits),
                   scratch.data_ptr(), bytes, &unique, stream);
  });
  if (rc == PSDEV_ERR_ARG) Py_RETURN_NONE;
  if (rc) return PyLong_FromLong(rc);
  at::Tensor keys = at::empty({unique}, plain), sums = at::empty({unique}, plain.dtype(at::kFloat));
  rc = without_gil([&] {
    return write_fn(scratch.data_ptr(), count, static_cast<int>(bits), unique,
                    static_cast<uint64_t*>(keys.data_ptr()), static_cast<float*>(sums.data_ptr()),
                    stream);
  });
  if (rc) return PyLong_FromLong(rc);
  PyObject* pair = PyTuple_New(2);
  if (!pair) return nullptr;
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(keys)));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(sums)));
  return pair;
  END_HANDLE_TH_ERRORS
}

// dense_op(fn, world, table, op, begin, end, opt, channel, num_ctas, timeout_ns, sync, stream)
PyObject* dense_op(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 12) return PyErr_Format(PyExc_TypeError, "dense_op takes 12 arguments");
  HANDLE_TH_ERRORS
  const auto fn = address<DenseFn>(a[0]);
  const auto* world = address<const psdev_world_t*>(a[1]);
  const auto* table = address<const psdev_table_t*>(a[2]);
  const long op = PyLong_AsLong(a[3]);
  const int64_t begin = PyLong_AsLongLong(a[4]), end = PyLong_AsLongLong(a[5]);
  const auto* opt = address<const psdev_opt_t*>(a[6]);
  const long channel = PyLong_AsLong(a[7]), ctas = PyLong_AsLong(a[8]);
  const uint64_t timeout = PyLong_AsUnsignedLongLongMask(a[9]);
  const long sync = PyLong_AsLong(a[10]);
  void* stream = address<void*>(a[11]);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromLong(without_gil([&] {
    return fn(world, table, static_cast<int>(op), begin, end, opt, static_cast<int>(channel),
              static_cast<int>(ctas), timeout, static_cast<int>(sync), stream);
  }));
  END_HANDLE_TH_ERRORS
}

// A keyed table of one rank.
struct SparseTarget {
  SparseFn fn;
  const psdev_world_t* world;
  const psdev_sparse_t* table;
  at::Tensor out;
  int64_t max_keys, max_vals, width;
  bool var_len;
  c10::DeviceIndex device;
};
constexpr const char* kSparseName = "psb200.sparse_target";

// (what is elsewhere, or negated by torch on reading, is copied into the table's buffers)
bool plain(const at::Tensor& t, at::ScalarType type, c10::DeviceIndex device) {
  return t.is_cuda() && t.get_device() == device && t.scalar_type() == type &&
         t.is_contiguous() && !t.is_neg();
}

// sparse_push_pull(target, keys, grads, lens): the pulled values (a view of the table's output),
// or None when the request is not one that the kernel can take as it is.
PyObject* sparse_push_pull(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4) return PyErr_Format(PyExc_TypeError, "sparse_push_pull takes 4 arguments");
  auto* t = static_cast<SparseTarget*>(PyCapsule_GetPointer(a[0], kSparseName));
  if (!t) return nullptr;
  HANDLE_TH_ERRORS
  if (!THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) Py_RETURN_NONE;
  const at::Tensor &keys = THPVariable_Unpack(a[1]), &grads = THPVariable_Unpack(a[2]);
  const int64_t nk = keys.numel(), nv = grads.numel();
  if (!(plain(keys, at::kLong, t->device) || plain(keys, at::kUInt64, t->device)) ||
      !plain(grads, at::kFloat, t->device) || nk > t->max_keys)
    Py_RETURN_NONE;
  const int32_t* lens = nullptr;
  if (t->var_len) {
    if (!THPVariable_Check(a[3])) Py_RETURN_NONE;
    const at::Tensor& l = THPVariable_Unpack(a[3]);
    if (!plain(l, at::kInt, t->device) || l.numel() != nk || nv > t->max_vals) Py_RETURN_NONE;
    lens = static_cast<const int32_t*>(l.data_ptr());
  } else if (nv != nk * t->width) {
    Py_RETURN_NONE;
  }
  // values inside the output buffer, other than at its start, would be overwritten while read
  auto* out = static_cast<float*>(t->out.data_ptr());
  const auto* vals = static_cast<const float*>(grads.data_ptr());
  if (vals < out + t->max_vals && out < vals + nv && vals != out) Py_RETURN_NONE;
  const int rc = without_gil([&] {
    return t->fn(t->world, t->table, nk, static_cast<const uint64_t*>(keys.data_ptr()), vals, nv,
                 lens, out, t->max_vals, nullptr, stream_on(t->device));
  });
  if (rc) return PyLong_FromLong(rc);
  return THPVariable_Wrap(t->out.narrow(0, 0, nv));
  END_HANDLE_TH_ERRORS
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f));
}
PyMethodDef kMethods[] = {
    {"linear", fast(&linear), METH_FASTCALL, "linear(fn, x, w, out, num_ctas, timeout_ns)"},
    {"pull_linear", fast(&pull_linear), METH_FASTCALL,
     "pull_linear(fn, world, table, w_offset, n_out, x, out, copy_ctas, num_ctas, timeout_ns)"},
    {"unique_sum", fast(&unique_sum), METH_FASTCALL,
     "unique_sum(bytes_fn, sort_fn, write_fn, keys, vals, key_bits)"},
    {"dense_op", fast(&dense_op), METH_FASTCALL,
     "dense_op(fn, world, table, op, begin, end, opt, channel, num_ctas, timeout_ns, sync, "
     "stream)"},
    {"sparse_push_pull", fast(&sparse_push_pull), METH_FASTCALL,
     "sparse_push_pull(target, keys, grads, lens)"},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

void add_calls(py::module& m) {
  m.def("sparse_target", [](uint64_t fn, uint64_t world, uint64_t table, at::Tensor out,
                            int64_t max_keys, int64_t max_vals, int64_t width, bool var_len) {
    auto* t = new SparseTarget{reinterpret_cast<SparseFn>(fn),
                               reinterpret_cast<const psdev_world_t*>(world),
                               reinterpret_cast<const psdev_sparse_t*>(table),
                               out, max_keys, max_vals, width, var_len, out.device().index()};
    return py::capsule(t, kSparseName, [](void* p) { delete static_cast<SparseTarget*>(p); });
  });
  PyModule_AddFunctions(m.ptr(), kMethods);
}
