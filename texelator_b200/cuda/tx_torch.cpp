// The operator call as Python makes it: argument checks, the output tensor and the launch in one native step.
//
// What bounds a small linear is the host: a 256 x 2048 matrix runs 3.2 us on the GPU, and the same call written
// in Python (tensor attribute reads, torch.empty, a stream object, ctypes conversions) cost 12.5 us of host time
// per call.  Here the tensor is read through its C++ object, the output comes straight from the caching allocator
// and the C-ABI entry point is called through its address: 5.1 us a call with the module's own Python on top.
//
// The module holds no CUDA code and links no library of this package: every handle is remembered with the addresses
// of the C-ABI functions (include/texelator_b200.h) of the library that packed it, so several loaded libraries keep
// to their own handles.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <unordered_map>

namespace {

using LinearFn = int (*)(uint64_t, const void *, void *, int, int, void *);
using ErrorFn = const char *(*)();

struct Shape {
  int64_t m, k;
  int device;
  LinearFn linear;
  ErrorFn last_error;
};

std::unordered_map<uint64_t, Shape> g_shapes;   // every access holds the GIL

PyObject *raise(const char *message) {
  PyErr_SetString(PyExc_RuntimeError, message);
  return nullptr;
}

// positional or keyword arguments called `names[0..count)`; false with an exception set when they do not fit
bool take_arguments(PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames, const char *const *names, int count, PyObject **out) {
  for (int i = 0; i < count; ++i) out[i] = i < nargs ? args[i] : nullptr;
  bool fits = nargs <= count;
  if (kwnames && fits) {
    for (Py_ssize_t j = 0; j < PyTuple_GET_SIZE(kwnames); ++j) {
      int at = -1;
      for (int i = 0; i < count; ++i)
        if (PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, j), names[i]) == 0) at = i;
      if (at < 0 || out[at]) fits = false;
      else out[at] = args[nargs + j];
    }
  }
  for (int i = 0; i < count; ++i) fits = fits && out[i];
  if (!fits) PyErr_SetString(PyExc_TypeError, count == 2 ? "linear(handle, x)" : "linear_out(handle, x, y)");
  return fits;
}

// A fake tensor (shape propagation under torch.compile and its kin) calls itself a CUDA tensor but owns no memory, and
// a view of one has its offset for an address: nothing may be launched on it.
bool has_memory(const at::Tensor &t) { return t.numel() == 0 || (t.has_storage() && t.storage().data() != nullptr); }

// the checks of texelator_cuda.cu:1332-1337; null with an exception set when one fails
const Shape *check_input(PyObject *handle_object, PyObject *x_object, uint64_t *handle, const at::Tensor **x) {
  // any integer (NumPy's too); what is none, or does not fit, names no handle
  PyObject *number = PyNumber_Index(handle_object);
  *handle = number ? PyLong_AsUnsignedLongLong(number) : 0;
  Py_XDECREF(number);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    *handle = 0;
  }
  auto found = g_shapes.find(*handle);
  if (found == g_shapes.end()) {
    raise("null Texelator handle");
    return nullptr;
  }
  if (!THPVariable_Check(x_object)) {
    PyErr_SetString(PyExc_TypeError, "input must be a tensor");
    return nullptr;
  }
  *x = &THPVariable_Unpack(x_object);
  const at::Tensor &t = **x;
  if (!t.is_cuda() || (t.scalar_type() != at::kBFloat16 && t.scalar_type() != at::kHalf) || !t.is_contiguous()) {
    raise("input must be contiguous CUDA FP16 or BF16");
    return nullptr;
  }
  if (!has_memory(t)) {
    raise("input must be contiguous CUDA FP16 or BF16");
    return nullptr;
  }
  if (t.dim() < 1 || t.size(-1) != found->second.k || t.get_device() != found->second.device) {
    raise("input shape/device mismatch");
    return nullptr;
  }
  return &found->second;
}

bool launch(uint64_t handle, const at::Tensor &x, const at::TensorBase &y, const Shape &shape) {
  const int64_t tokens = x.numel() / shape.k;
  if (tokens == 0) return true;
  if (tokens > INT32_MAX) {
    raise("input shape/device mismatch");
    return false;
  }
  void *stream = c10::cuda::getCurrentCUDAStream(c10::DeviceIndex(shape.device)).stream();
  const void *in = x.const_data_ptr();
  void *out = y.mutable_data_ptr();
  const int dtype = x.scalar_type() == at::kBFloat16 ? 1 : 0;
  int status;
  Py_BEGIN_ALLOW_THREADS   // a launch can wait for room in the stream's queue
  status = shape.linear(handle, in, out, int(tokens), dtype, stream);
  Py_END_ALLOW_THREADS
  if (status != 0) {
    const char *message = shape.last_error();
    raise(message && message[0] ? message : "texelator_b200 call failed");
    return false;
  }
  return true;
}

PyObject *linear(PyObject *, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  HANDLE_TH_ERRORS
  static const char *const names[] = {"handle", "x"};
  PyObject *given[2];
  if (!take_arguments(args, nargs, kwnames, names, 2, given)) return nullptr;
  uint64_t handle;
  const at::Tensor *x;
  const Shape *found = check_input(given[0], given[1], &handle, &x);
  if (!found) return nullptr;
  const Shape shape = *found;
  c10::SmallVector<int64_t, 5> sizes(x->sizes().begin(), x->sizes().end());
  sizes.back() = shape.m;
  at::Tensor y(at::detail::empty_cuda(sizes, x->scalar_type(), x->device(), std::nullopt));
  if (!launch(handle, *x, y, shape)) return nullptr;
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyObject *linear_out(PyObject *, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  HANDLE_TH_ERRORS
  static const char *const names[] = {"handle", "x", "y"};
  PyObject *given[3];
  if (!take_arguments(args, nargs, kwnames, names, 3, given)) return nullptr;
  uint64_t handle;
  const at::Tensor *x;
  const Shape *found = check_input(given[0], given[1], &handle, &x);
  if (!found) return nullptr;
  if (!THPVariable_Check(given[2])) {
    PyErr_SetString(PyExc_TypeError, "output must be a tensor");
    return nullptr;
  }
  const at::Tensor &y = THPVariable_Unpack(given[2]);
  const Shape shape = *found;
  if (y.numel() != x->numel() / shape.k * shape.m || y.scalar_type() != x->scalar_type() || !y.is_contiguous() || y.device() != x->device() ||
      !has_memory(y))
    return raise("input shape/device mismatch");
  if (x->numel() == 0) return raise("input must be contiguous CUDA FP16 or BF16");   // tx_linear refuses a null activation pointer
  if (!launch(handle, *x, y, shape)) return nullptr;
  return Py_NewRef(given[2]);
  END_HANDLE_TH_ERRORS
}

PyObject *remember(PyObject *, PyObject *args) {
  unsigned long long handle, linear_address, error_address;
  long long m, k;
  int device;
  if (!PyArg_ParseTuple(args, "KLLiKK", &handle, &m, &k, &device, &linear_address, &error_address)) return nullptr;
  HANDLE_TH_ERRORS
  g_shapes[handle] = Shape{m, k, device, reinterpret_cast<LinearFn>(linear_address), reinterpret_cast<ErrorFn>(error_address)};
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject *forget(PyObject *, PyObject *args) {
  unsigned long long handle;
  if (!PyArg_ParseTuple(args, "K", &handle)) return nullptr;
  g_shapes.erase(handle);
  Py_RETURN_NONE;
}

#define TX_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL | METH_KEYWORDS
PyMethodDef methods[] = {
    {"linear", TX_FAST(linear), "linear(handle, x) -> tensor [..., M]"},
    {"linear_out", TX_FAST(linear_out), "linear_out(handle, x, y) -> y, for outputs the caller keeps (CUDA graphs)"},
    {"remember", remember, METH_VARARGS, "remember(handle, m, k, device, address of tx_linear, address of tx_last_error)"},
    {"forget", forget, METH_VARARGS, "forget(handle)"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tx_torch", nullptr, -1, methods};

}  // namespace

// Tensors are read through inlined C++ accessors, which hold for one torch only; the loader compares this text.
#ifndef TX_BUILT_FOR
#define TX_BUILT_FOR "unknown"
#endif
PyMODINIT_FUNC PyInit__tx_torch() {
  PyObject *self = PyModule_Create(&module);
  if (self && PyModule_AddStringConstant(self, "built_for", TX_BUILT_FOR) != 0) Py_CLEAR(self);
  return self;
}
