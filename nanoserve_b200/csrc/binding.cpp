// The host side of ops.Kernels.w4_linear and w4_quantize as one native call each.  Through ctypes an eager one-token call spent
// more time in Python (argument conversion, torch.empty with keywords, the tensors' properties) than its launch takes; here the
// same steps run on the tensors' C++ objects (512 x 3584 at one token 8.6 -> 4.8 us a call).
//
// w4_linear(fn, x, Wq, S, group, flags, out): `fn` is the address of b2_w4_linear in whatever library the caller has loaded.
// w4_quantize(fn, W, group): likewise of ns_w4_quantize.  They take exactly torch.Tensor (or Parameter) arguments on a CUDA
// device, x and W matrices; for anything else -- a subclass, a tensor on the host, an active dispatch or function mode, other
// argument types -- they return NotImplemented before they have done anything, and the caller takes its own path, which then
// answers or refuses as ever.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

using LinearFn = int (*)(const void*, const void*, const void*, void*, int, int, int, int, int, void*);
using QuantizeFn = int (*)(const void*, void*, void*, int, int, int, void*);

bool plain(PyObject* o) { return THPVariable_CheckExact(o); }

bool modes_active() {
  return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() ||
         c10::impl::tls_is_dispatch_key_included(at::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

bool as_int(PyObject* o, int* out) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow || v < INT32_MIN || v > INT32_MAX) return false;
  *out = (int)v;
  return true;
}

PyObject* w4_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int group = 0, flags = 0;
  if (n != 7 || !PyLong_CheckExact(a[0]) || !plain(a[1]) || !plain(a[2]) || !plain(a[3]) || !as_int(a[4], &group) ||
      !as_int(a[5], &flags) || !(a[6] == Py_None || plain(a[6])) || modes_active())
    Py_RETURN_NOTIMPLEMENTED;
  const at::Tensor& x0 = THPVariable_Unpack(a[1]);
  const at::Tensor& wq = THPVariable_Unpack(a[2]);
  const at::Tensor& s = THPVariable_Unpack(a[3]);
  if (!x0.is_cuda() || !wq.is_cuda() || !s.is_cuda() || x0.dim() != 2 || wq.dim() < 1 || x0.size(0) > INT32_MAX ||
      x0.size(1) > INT32_MAX || wq.size(0) > INT32_MAX || !x0.has_storage() || !wq.has_storage() || !s.has_storage())
    Py_RETURN_NOTIMPLEMENTED;
  if (a[6] != Py_None && (!THPVariable_Unpack(a[6]).is_cuda() || !THPVariable_Unpack(a[6]).has_storage()))
    Py_RETURN_NOTIMPLEMENTED;
  const at::Tensor x = x0.is_contiguous() ? x0 : x0.contiguous();
  const int M = (int)x.size(0), K = (int)x.size(1), N = (int)wq.size(0);
  const at::Tensor y = a[6] != Py_None ? THPVariable_Unpack(a[6])
                                       : at::empty({M, N}, at::TensorOptions().dtype(at::kBFloat16).device(x.device()));
  const auto fn = reinterpret_cast<LinearFn>(PyLong_AsVoidPtr(a[0]));
  const void *xp = x.const_data_ptr(), *wp = wq.const_data_ptr(), *sp = s.const_data_ptr();
  void* const yp = y.mutable_data_ptr();
  void* const stream = c10::cuda::getCurrentCUDAStream().stream();
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(xp, wp, sp, yp, M, N, K, group, flags, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyErr_Format(PyExc_RuntimeError, "ns_w4_linear failed with code %d", rc);
    return nullptr;
  }
  if (a[6] != Py_None) {
    Py_INCREF(a[6]);
    return a[6];
  }
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* w4_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int group = 0;
  if (n != 3 || !PyLong_CheckExact(a[0]) || !plain(a[1]) || !as_int(a[2], &group) || group < 1 || modes_active())
    Py_RETURN_NOTIMPLEMENTED;
  const at::Tensor& w0 = THPVariable_Unpack(a[1]);
  if (!w0.is_cuda() || w0.dim() != 2 || w0.size(0) > INT32_MAX || w0.size(1) > INT32_MAX || !w0.has_storage())
    Py_RETURN_NOTIMPLEMENTED;
  const int64_t N = w0.size(0), K = w0.size(1);
  const at::Tensor wq = at::empty({N, K / 8}, at::TensorOptions().dtype(at::kInt).device(w0.device()));
  const at::Tensor s = at::empty({N, K / group}, at::TensorOptions().dtype(at::kBFloat16).device(w0.device()));
  const at::Tensor w = w0.is_contiguous() ? w0 : w0.contiguous();
  const auto fn = reinterpret_cast<QuantizeFn>(PyLong_AsVoidPtr(a[0]));
  const void* const wp = w.const_data_ptr();
  void *const qp = wq.mutable_data_ptr(), *const sp = s.mutable_data_ptr();
  void* const stream = c10::cuda::getCurrentCUDAStream().stream();
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(wp, qp, sp, (int)N, (int)K, group, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyErr_Format(PyExc_RuntimeError, "ns_w4_quantize failed with code %d", rc);
    return nullptr;
  }
  PyObject* const q = THPVariable_Wrap(wq);
  PyObject* const t = q ? THPVariable_Wrap(s) : nullptr;
  if (!t) {
    Py_XDECREF(q);
    return nullptr;
  }
  PyObject* const both = PyTuple_Pack(2, q, t);
  Py_DECREF(q);
  Py_DECREF(t);
  return both;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"w4_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(w4_linear)), METH_FASTCALL, nullptr},
    {"w4_quantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(w4_quantize)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "nanoserve_call", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit_nanoserve_call(void) { return PyModule_Create(&kModule); }
