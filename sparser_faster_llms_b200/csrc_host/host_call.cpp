// The host side of an eager fused-MLP call in native code: argument checks, scratch from torch's allocator
// and the call into the C ABI.  In Python these take 12 to 16 us of a call of 18 to 28 us whose kernels take
// 12 to 20, so small layers waited for the host.
//
// Only the plain case is handled: dense CUDA tensors of the right shapes on the current device, without
// dispatch or function modes.  Everything else (None is returned) goes through the Python path, which
// also raises the errors.  Nothing is kept between calls.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstddef>
#include <cstdint>

namespace {

using ScratchFn = size_t (*)(int64_t, int64_t, int64_t, int, uint32_t);
using GatedFn = int (*)(const void*, const void*, const float*, const void*, const void*, void*, void*,
                        int64_t, int64_t, int64_t, int, uint32_t, void*, size_t, void*, size_t, void*);
using PlainFn = int (*)(const void*, const void*, const void*, void*, void*, int64_t, int64_t, int64_t,
                        int, int, void*, size_t, void*, size_t, void*);

// The tensor behind `o` if it is an ordinary CUDA tensor (no subclass that dispatches, no functorch or
// functionalisation wrapper, no lazy conjugate), contiguous, of this type and rank.
const at::Tensor* plain(PyObject* o, at::ScalarType type, int64_t dim) {
  static const c10::DispatchKeySet ordinary =
      c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
      c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) |
      c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA);
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !ordinary.isSupersetOf(t.key_set())) return nullptr;
  if (t.scalar_type() != type || t.dim() != dim || !t.is_contiguous()) return nullptr;
  return &t;
}

bool is_matrix(const at::Tensor* t, int64_t rows, int64_t cols) {
  return t != nullptr && t->size(0) == rows && t->size(1) == cols;
}

// call(fn, scratch_fn, A, first, bias, up, down, packed, out, cf, option, workspace, workspace_bytes,
//      scratch_from): the status of the C call, or None where the Python path has to serve.
// up is None for the non-gated MLP; option: flags (gated) or num_splits.
PyObject* call(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 14) {
    PyErr_SetString(PyExc_TypeError, "call takes 14 arguments");
    return nullptr;
  }
  const bool gated = v[5] != Py_None;
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled())
    Py_RETURN_NONE;
  const at::Tensor* x = plain(v[2], at::kBFloat16, 2);
  const at::Tensor* first = plain(v[3], at::kBFloat16, 2);
  const at::Tensor* down = plain(v[6], at::kBFloat16, 2);
  const at::Tensor* packed = plain(v[7], at::kUInt32, 2);
  const at::Tensor* out = plain(v[8], at::kBFloat16, 2);
  const at::Tensor* up = gated ? plain(v[5], at::kBFloat16, 2) : first;
  const at::Tensor* bias = v[4] == Py_None ? nullptr : plain(v[4], at::kFloat, 1);
  if (x == nullptr || first == nullptr || (v[4] != Py_None && bias == nullptr)) Py_RETURN_NONE;
  const long cf = PyLong_AsLong(v[9]), option = PyLong_AsLong(v[10]);
  if (PyErr_Occurred()) {  // no number, or one beyond a long: the Python path decides
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int64_t m = x->size(0), d = x->size(1), h = first->size(0);
  if ((cf != 2 && cf != 4 && cf != 8) || h % 256 != 0) Py_RETURN_NONE;
  if (first->size(1) != d || !is_matrix(up, h, d) || !is_matrix(down, h, d) || !is_matrix(out, m, d) ||
      !is_matrix(packed, m, h / cf) || (bias != nullptr && bias->size(0) != h))
    Py_RETURN_NONE;
  const c10::Device dev = x->device();
  if (first->device() != dev || up->device() != dev || down->device() != dev ||
      packed->device() != dev || out->device() != dev || (bias != nullptr && bias->device() != dev) ||
      dev.index() != c10::cuda::current_device())
    Py_RETURN_NONE;

  void* fn = PyLong_AsVoidPtr(v[0]);
  auto scratch_fn = reinterpret_cast<ScratchFn>(PyLong_AsVoidPtr(v[1]));
  void* workspace = v[11] == Py_None ? nullptr : PyLong_AsVoidPtr(v[11]);
  const size_t workspace_bytes = PyLong_AsSize_t(v[12]);
  const long scratch_from = PyLong_AsLong(v[13]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor scratch;
  size_t scratch_bytes = 0;
  if (m >= scratch_from)
    scratch_bytes = scratch_fn(m, d, h, gated, (gated ? (uint32_t)option : 0u) | (uint32_t)cf << 8);
  if (scratch_bytes != 0)
    scratch = at::empty({(int64_t)scratch_bytes}, at::TensorOptions().dtype(at::kByte).device(dev));
  void* scratch_ptr = scratch_bytes != 0 ? scratch.data_ptr() : nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const void *px = x->const_data_ptr(), *pf = first->const_data_ptr(), *pd = down->const_data_ptr();
  const void* pu = up->const_data_ptr();
  const float* pb = bias != nullptr ? static_cast<const float*>(bias->const_data_ptr()) : nullptr;
  void *pp = packed->data_ptr(), *po = out->data_ptr();
  int status;
  Py_BEGIN_ALLOW_THREADS;
  if (gated)
    status = reinterpret_cast<GatedFn>(fn)(px, pf, pb, pu, pd, pp, po, m, d, h, (int)cf, (uint32_t)option,
                                           workspace, workspace_bytes, scratch_ptr, scratch_bytes, stream);
  else
    status = reinterpret_cast<PlainFn>(fn)(px, pf, pd, pp, po, m, d, h, (int)cf, (int)option, workspace,
                                           workspace_bytes, scratch_ptr, scratch_bytes, stream);
  Py_END_ALLOW_THREADS;
  return PyLong_FromLong(status);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call)), METH_FASTCALL,
     "One fused-MLP call; None where the Python path has to serve."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_call", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_call() { return PyModule_Create(&module); }
