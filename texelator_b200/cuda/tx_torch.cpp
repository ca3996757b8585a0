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
using StagedFn = int (*)(uint64_t, const void *, void *, int, void *);
using TakesFn = int (*)(uint64_t, int);
using BytesFn = size_t (*)(int, int);

struct Shape {
  int64_t m, k;
  int device;
  LinearFn linear;
  ErrorFn last_error;
  StagedFn staged;   // null where the library has none
  TakesFn takes;
  BytesFn bytes;
};

std::unordered_map<uint64_t, Shape> g_shapes;   // every access holds the GIL

PyObject *raise(const char *message) {
  PyErr_SetString(PyExc_RuntimeError, message);
  return nullptr;
}

// positional or keyword arguments called `names[0..count)`; false with an exception set when they do not fit
bool take_arguments(PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames, const char *const *names, int count, PyObject **out, const char *usage) {
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
  if (!fits) PyErr_SetString(PyExc_TypeError, usage);
  return fits;
}

// A fake tensor (shape propagation under torch.compile and its kin) calls itself a CUDA tensor but owns no memory, and
// a view of one has its offset for an address: nothing may be launched on it.
bool has_memory(const at::Tensor &t) { return t.numel() == 0 || (t.has_storage() && t.storage().data() != nullptr); }

// null where no handle of that number is known
const Shape *find(PyObject *handle_object, uint64_t *handle) {
  // any integer (NumPy's too); what is none, or does not fit, names no handle
  PyObject *number = PyNumber_Index(handle_object);
  *handle = number ? PyLong_AsUnsignedLongLong(number) : 0;
  Py_XDECREF(number);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    *handle = 0;
  }
  auto found = g_shapes.find(*handle);
  return found == g_shapes.end() ? nullptr : &found->second;
}

// the checks of texelator_cuda.cu:1332-1337; null with an exception set when one fails
const Shape *check_input(PyObject *handle_object, PyObject *x_object, uint64_t *handle, const at::Tensor **x) {
  const Shape *found = find(handle_object, handle);
  if (!found) {
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
  if (t.dim() < 1 || t.size(-1) != found->k || t.get_device() != found->device) {
    raise("input shape/device mismatch");
    return nullptr;
  }
  return found;
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
  if (!take_arguments(args, nargs, kwnames, names, 2, given, "linear(handle, x)")) return nullptr;
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
  if (!take_arguments(args, nargs, kwnames, names, 3, given, "linear_out(handle, x, y)")) return nullptr;
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

// Short prompts wait for the host: with this call and the question below in Python a prompt of 58 tokens through five layers of the 2048-wide model took 605 us,
// 520 with rows and their staging launches.
PyObject *linear_staged(PyObject *, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  HANDLE_TH_ERRORS
  static const char *const names[] = {"handle", "staged", "y"};
  PyObject *given[3];
  if (!take_arguments(args, nargs, kwnames, names, 3, given, "linear_staged(handle, staged, y)")) return nullptr;
  uint64_t handle;
  const Shape *found = find(given[0], &handle);
  if (!found || !found->staged || !found->bytes) return raise("null Texelator handle");
  const Shape shape = *found;
  if (!THPVariable_Check(given[1]) || !THPVariable_Check(given[2])) {
    PyErr_SetString(PyExc_TypeError, "staged activations and output must be tensors");
    return nullptr;
  }
  const at::Tensor &staged = THPVariable_Unpack(given[1]), &y = THPVariable_Unpack(given[2]);
  const int64_t tokens = y.numel() / shape.m;
  if (!y.is_cuda() || y.scalar_type() != at::kBFloat16 || !y.is_contiguous() || y.get_device() != shape.device || y.numel() != tokens * shape.m || tokens > INT32_MAX)
    return raise("input shape/device mismatch");
  if (!staged.is_cuda() || staged.scalar_type() != at::kByte || !staged.is_contiguous() || staged.get_device() != shape.device)
    return raise("staged activations are a contiguous uint8 tensor on the CUDA device of the rows");
  if (size_t(staged.numel()) < shape.bytes(int(shape.k), int(tokens))) return raise("the staged buffer is too small");
  if (!has_memory(staged) || !has_memory(y)) return raise("input shape/device mismatch");
  void *stream = c10::cuda::getCurrentCUDAStream(c10::DeviceIndex(shape.device)).stream();
  const void *in = staged.const_data_ptr();
  void *out = y.mutable_data_ptr();
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = shape.staged(handle, in, out, int(tokens), stream);
  Py_END_ALLOW_THREADS
  if (status != 0) {
    const char *message = shape.last_error();
    return raise(message && message[0] ? message : "texelator_b200 call failed");
  }
  return Py_NewRef(given[2]);
  END_HANDLE_TH_ERRORS
}

PyObject *takes_staged(PyObject *, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  static const char *const names[] = {"handle", "tokens"};
  PyObject *given[2];
  if (!take_arguments(args, nargs, kwnames, names, 2, given, "takes_staged(handle, tokens)")) return nullptr;
  const long tokens = PyLong_AsLong(given[1]);
  if (tokens == -1 && PyErr_Occurred()) return nullptr;
  uint64_t handle;
  const Shape *found = find(given[0], &handle);
  return PyBool_FromLong(found && tokens > 0 && tokens <= INT32_MAX && found->takes && found->takes(handle, int(tokens)) == 1);
}

PyObject *remember(PyObject *, PyObject *args) {
  unsigned long long handle, linear_address, error_address, staged_address, takes_address, bytes_address;
  long long m, k;
  int device;
  if (!PyArg_ParseTuple(args, "KLLiKKKKK", &handle, &m, &k, &device, &linear_address, &error_address, &staged_address, &takes_address, &bytes_address)) return nullptr;
  HANDLE_TH_ERRORS
  g_shapes[handle] = Shape{m, k, device, reinterpret_cast<LinearFn>(linear_address), reinterpret_cast<ErrorFn>(error_address),
                           reinterpret_cast<StagedFn>(staged_address), reinterpret_cast<TakesFn>(takes_address), reinterpret_cast<BytesFn>(bytes_address)};
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
    {"linear_staged", TX_FAST(linear_staged), "linear_staged(handle, staged, y) -> y, rows that the kernel in front left in staged form"},
    {"takes_staged", TX_FAST(takes_staged), "takes_staged(handle, tokens) -> bool"},
    {"remember", remember, METH_VARARGS,
     "remember(handle, m, k, device, addresses of tx_linear, tx_last_error, tx_linear_staged, tx_linear_takes_staged and tx_staged_prompt_bytes)"},
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
