// The operators' way from torch tensors to the C ABI, for plain tensors: what the raw-pointer entry points cannot see (types,
// shapes, strides, devices) is checked here, and the launch goes to the current stream of the tensors' device.
//
// In Python the same checks, four data_ptr() and two ctypes calls took 4.4 of the 7.1 us of a batch-1 call whose kernel takes 4.6.
//
// True: launched.  False: nothing was done, and the caller takes the general path, which names the error where there is one. That
// path also takes everything that is not a plain tensor: subclasses, wrapped tensors (vmap, grad transforms, functionalisation),
// lazily conjugated, negated or zero tensors, and any call under a torch-function mode.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200_q4f16.h"

namespace {

// The library that the package has loaded (its own or the one that the environment names).
struct Entry {
  decltype(&b200_set_stream) set_stream = nullptr;
  decltype(&b200_q4f16_matmul) matmul = nullptr;
  decltype(&b200_q4f16_matmul_layout) matmul_layout = nullptr;
  decltype(&b200_q4f16_dequantize) dequantize = nullptr;
} g_entry;

const at::Tensor* plain_matrix(PyObject* o, at::ScalarType type) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
                                            c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                            c10::DispatchKey::Functionalize, c10::DispatchKey::ZeroTensor,
                                            c10::DispatchKey::Conjugate, c10::DispatchKey::Negative});
  if (!t.defined() || t.key_set().has_any(special) || !t.is_cuda() || t.layout() != c10::kStrided || !t.has_storage()) return nullptr;
  if (t.scalar_type() != type || t.dim() != 2 || !t.is_contiguous()) return nullptr;
  return &t;
}

// The tensors' device if it is everyone's and the current one, else -1.
int common_device(std::initializer_list<const at::Tensor*> ts) {
  const int dev = (*ts.begin())->get_device();
  for (const at::Tensor* t : ts)
    if (t->get_device() != dev) return -1;
  return c10::cuda::current_device() == dev ? dev : -1;
}

PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "matmul(x, wq, scales, out, layout)");
    return nullptr;
  }
  // -1: no layout given.  Any other number that is no layout is for the general path, which refuses it.
  int overflow = 0;
  const long layout = PyLong_AsLongAndOverflow(args[4], &overflow);
  if (layout == -1 && PyErr_Occurred()) return nullptr;
  if (overflow != 0 || layout < -1 || layout > INT32_MAX) Py_RETURN_FALSE;
  try {
    if (!g_entry.matmul || at::impl::torch_function_mode_enabled()) Py_RETURN_FALSE;
    const at::Tensor *x = plain_matrix(args[0], at::kHalf), *wq = plain_matrix(args[1], at::kUInt32),
                     *scales = plain_matrix(args[2], at::kHalf), *out = plain_matrix(args[3], at::kHalf);
    if (!x || !wq || !scales || !out) Py_RETURN_FALSE;
    const int dev = common_device({x, wq, scales, out});
    const int64_t M = x->size(0), K = x->size(1), N = wq->size(0);
    if (dev < 0 || K % 32 != 0 || wq->size(1) * 8 != K || scales->size(0) != N || scales->size(1) != K / 32 || out->size(0) != M ||
        out->size(1) != N)
      Py_RETURN_FALSE;
    void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    const void *px = x->const_data_ptr(), *pw = wq->const_data_ptr(), *ps = scales->const_data_ptr();
    void* py = out->mutable_data_ptr();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    g_entry.set_stream(stream);
    rc = layout < 0 ? g_entry.matmul(px, pw, ps, py, M, N, K, stream)
                    : g_entry.matmul_layout(px, pw, ps, py, M, N, K, (int32_t)layout, stream);
    Py_END_ALLOW_THREADS
    return PyBool_FromLong(rc == 0);
  } catch (const std::exception&) {
    Py_RETURN_FALSE;
  }
}

PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "dequantize(wq, scales, out)");
    return nullptr;
  }
  try {
    if (!g_entry.dequantize || at::impl::torch_function_mode_enabled()) Py_RETURN_FALSE;
    const at::Tensor *wq = plain_matrix(args[0], at::kUInt32), *scales = plain_matrix(args[1], at::kHalf), *out = plain_matrix(args[2], at::kHalf);
    if (!wq || !scales || !out) Py_RETURN_FALSE;
    const int dev = common_device({wq, scales, out});
    const int64_t N = wq->size(0), K = wq->size(1) * 8;
    if (dev < 0 || K % 32 != 0 || scales->size(0) != N || scales->size(1) != K / 32 || out->size(0) != N || out->size(1) != K) Py_RETURN_FALSE;
    void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    const void *pw = wq->const_data_ptr(), *ps = scales->const_data_ptr();
    void* po = out->mutable_data_ptr();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    g_entry.set_stream(stream);
    rc = g_entry.dequantize(pw, ps, po, N, K, stream);
    Py_END_ALLOW_THREADS
    return PyBool_FromLong(rc == 0);
  } catch (const std::exception&) {
    Py_RETURN_FALSE;
  }
}

// bind(set_stream, matmul, matmul_layout, dequantize): addresses of the loaded library's entry points.
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  void* p[4] = {};
  for (Py_ssize_t i = 0; n == 4 && i < n; ++i) p[i] = PyLong_AsVoidPtr(args[i]);
  if (PyErr_Occurred()) return nullptr;
  if (n != 4 || !p[0] || !p[1] || !p[2] || !p[3]) {
    PyErr_SetString(PyExc_TypeError, "bind() takes the addresses of four entry points");
    return nullptr;
  }
  g_entry.set_stream = reinterpret_cast<decltype(g_entry.set_stream)>(p[0]);
  g_entry.matmul = reinterpret_cast<decltype(g_entry.matmul)>(p[1]);
  g_entry.matmul_layout = reinterpret_cast<decltype(g_entry.matmul_layout)>(p[2]);
  g_entry.dequantize = reinterpret_cast<decltype(g_entry.dequantize)>(p[3]);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(matmul)), METH_FASTCALL, nullptr},
    {"dequantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(dequantize)), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_call", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_call() { return PyModule_Create(&kModule); }
