// The common form of QuantizedLinear.__call__ (a prepared weight, no gate, residual, adapter, output buffer or scratch) in
// native code, as the CPython module mflux_b200._host. A call of a few rows is bound by the host: through Python and
// ctypes (thirty attribute reads, a struct filled field by field) it took 12.8 us beside a kernel of 4.4 us.
// linear() takes a call only when it would do exactly what ops.qlinear does with it; for everything else, and for every
// error, it returns None and the Python path decides and raises. The library's functions come by address from the
// loaded libmfx.so (bind()), so this module links against torch only. The interpreter lock is held for looking at the
// arguments only: allocation and launch may wait for the device, and other threads run meanwhile.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string.h>

#include "mfx.h"

namespace {

using QlinearFn = int (*)(const mfx_qlinear_args*, void*);
using ScratchFn = size_t (*)(int64_t, int64_t, int64_t, int64_t, int);
using PreparedFn = size_t (*)(int64_t, int64_t, int, int);
QlinearFn qlinear_fn = nullptr;
ScratchFn scratch_fn = nullptr;
PreparedFn prepared_fn = nullptr;

// A plain, strided CUDA tensor with memory of its own kind: no subclass that overrides operations, no functorch wrapper.
const at::Tensor* plain_cuda(PyObject* o) {
  if (!THPVariable_CheckExact(o) && Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(ParameterClass)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_inference()) return nullptr;
  if (t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                               c10::DispatchKey::Functionalize, c10::DispatchKey::Python})))
    return nullptr;
  return &t;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MFX_F32;
    case at::kBFloat16: return MFX_BF16;
    case at::kHalf: return MFX_F16;
    default: return -1;
  }
}

// The six numbers nn.QuantizedLinear.prepared() keys its blob with: address and version of weight, scales and biases.
bool same_weight(PyObject* key, const at::Tensor* const (&t)[3]) {
  if (!PyTuple_CheckExact(key) || PyTuple_GET_SIZE(key) != 6) return false;
  for (int i = 0; i < 3; ++i) {
    const unsigned long long ptr = PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(key, 2 * i));
    const long long version = PyLong_AsLongLong(PyTuple_GET_ITEM(key, 2 * i + 1));
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    if (ptr != reinterpret_cast<unsigned long long>(t[i]->data_ptr()) ||
        version != static_cast<long long>(t[i]->unsafeGetTensorImpl()->version_counter().current_version()))
      return false;
  }
  return true;
}

// Lets other Python threads run while it lives.
struct WithoutInterpreterLock {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutInterpreterLock() { PyEval_RestoreThread(state); }
};

// linear(x, weight, scales, biases, bias, prepared, bits, group_size, epilogue) -> Tensor or None
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 9) {
    PyErr_SetString(PyExc_TypeError, "linear() takes nine arguments");
    return nullptr;
  }
  if (qlinear_fn == nullptr || !PyTuple_CheckExact(args[5]) || PyTuple_GET_SIZE(args[5]) != 2) Py_RETURN_NONE;
  if (at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set()) Py_RETURN_NONE;
  const at::Tensor* x = plain_cuda(args[0]);
  const at::Tensor* w[3] = {plain_cuda(args[1]), plain_cuda(args[2]), plain_cuda(args[3])};
  const at::Tensor* blob = plain_cuda(PyTuple_GET_ITEM(args[5], 1));
  if (!x || !w[0] || !w[1] || !w[2] || !blob) Py_RETURN_NONE;
  if (!same_weight(PyTuple_GET_ITEM(args[5], 0), w)) Py_RETURN_NONE;
  const long bits = PyLong_AsLong(args[6]), group_size = PyLong_AsLong(args[7]), epilogue = PyLong_AsLong(args[8]);
  if (PyErr_Occurred()) return nullptr;
  if (epilogue == MFX_EPI_GATE_RESIDUAL || epilogue == MFX_EPI_PEER_SCATTER) Py_RETURN_NONE;

  const int64_t dims = x->dim();
  if (x->scalar_type() != at::kBFloat16 || dims < 1 || dims > 3 || x->stride(dims - 1) != 1) Py_RETURN_NONE;
  if (bits <= 0 || w[0]->dim() != 2) Py_RETURN_NONE;
  const int64_t n = w[0]->size(0), k = x->size(dims - 1);
  if (w[0]->size(1) * 32 / bits != k) Py_RETURN_NONE;
  mfx_qlinear_args a;
  memset(&a, 0, sizeof(a));
  a.rows = dims == 1 ? 1 : x->size(dims - 2);
  a.batch = dims == 3 ? x->size(0) : 1;
  a.x_row_stride = dims == 1 ? k : x->stride(dims - 2);
  a.x_batch_stride = dims == 3 ? x->stride(0) : 0;
  if (a.rows <= 0 || a.batch <= 0) Py_RETURN_NONE;
  if (blob->scalar_type() != at::kByte ||
      static_cast<size_t>(blob->numel()) != prepared_fn(n, k, static_cast<int>(bits), static_cast<int>(group_size)))
    Py_RETURN_NONE;
  if (scratch_fn(a.rows, a.batch, n, k, static_cast<int>(bits)) != 0) Py_RETURN_NONE;   // a call that wants scratch
  a.K = k;
  a.N = n;
  a.bits = static_cast<int>(bits);
  a.group_size = static_cast<int>(group_size);
  a.x = x->data_ptr();
  a.prepared = blob->data_ptr();
  if (args[4] != Py_None) {
    const at::Tensor* bias = plain_cuda(args[4]);
    if (!bias || !bias->is_contiguous()) Py_RETURN_NONE;
    a.bias_dtype = dtype_code(bias->scalar_type());
    if (a.bias_dtype < 0) Py_RETURN_NONE;
    a.bias = bias->data_ptr();
  }
  a.epilogue = static_cast<int>(epilogue);
  const int64_t n_out = epilogue == MFX_EPI_SWIGLU ? n / 2 : n;
  at::DimVector shape(x->sizes().begin(), x->sizes().end());
  shape[dims - 1] = n_out;
  const at::TensorOptions options = x->options().requires_grad(false);
  at::Tensor y;
  int status;
  a.y_dtype = MFX_BF16;
  a.y_row_stride = n_out;
  a.y_batch_stride = dims == 3 ? a.rows * n_out : 0;
  {
    // No Python object is touched in here, and none of the arguments' tensors (another thread may replace their data):
    // what the call needs was copied out above, and the caller's references keep the objects.
    WithoutInterpreterLock unlocked;
    y = at::empty(shape, options);
    a.y = y.data_ptr();
    status = qlinear_fn(&a, c10::cuda::getCurrentCUDAStream(c10::cuda::current_device()).stream());
  }
  if (status != MFX_OK) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// bind(address of mfx_qlinear_ex, of mfx_qlinear_scratch_bytes_batch, of mfx_qlinear_prepared_bytes)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "bind() takes three addresses");
    return nullptr;
  }
  void* fn[3];
  for (int i = 0; i < 3; ++i) {
    fn[i] = PyLong_AsVoidPtr(args[i]);
    if (PyErr_Occurred()) return nullptr;
  }
  scratch_fn = reinterpret_cast<ScratchFn>(fn[1]);
  prepared_fn = reinterpret_cast<PreparedFn>(fn[2]);
  qlinear_fn = reinterpret_cast<QlinearFn>(fn[0]);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear)), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  PyObject* m = PyModule_Create(&module);
  if (m != nullptr && PyModule_AddStringConstant(m, "BUILT_FOR", MFX_BUILT_FOR) != 0) Py_CLEAR(m);
  return m;
}
