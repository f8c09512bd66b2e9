// Python extension `sparsetir_b200._pycall`: packs torch tensors into the operator boundary's
// argument arrays (TVMValue / type codes / DLTensor) and makes the packed call.
//
// What bounds a call of a few microseconds is the host: packed through ctypes, a call cost about
// 5 us per tensor (a 4096-row csrmm 35 us around a 5 us kernel, hyb_spmm with ten buckets 220 us
// around a 22 us kernel).  Here a tensor costs a few dozen nanoseconds: its DLTensor lives on the
// stack and points at the sizes and strides that the tensor itself holds.
//
// The module does not link against the operator library; the Python side passes the addresses of
// the entry points it resolved, so that another build of the library can be loaded.
#include <Python.h>

#if SPTIR_TORCH_CUDA
#include <c10/cuda/CUDAStream.h>
#endif
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "sparsetir_b200.h"

namespace {

using PackedFn = int (*)(TVMValue*, int*, int, TVMValue*, int*, void*);
using SetStreamFn = int (*)(int, void*);

bool dl_type(at::ScalarType t, DLDataType* out) {
  out->lanes = 1;
  switch (t) {
    case at::kFloat: out->code = kDLFloat; out->bits = 32; return true;
    case at::kHalf: out->code = kDLFloat; out->bits = 16; return true;
    case at::kDouble: out->code = kDLFloat; out->bits = 64; return true;
    case at::kInt: out->code = kDLInt; out->bits = 32; return true;
    case at::kLong: out->code = kDLInt; out->bits = 64; return true;
    case at::kByte: out->code = kDLUInt; out->bits = 8; return true;
    default: return false;
  }
}

// Without the GIL, taken again whichever way the scope is left.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// Runs the call without the GIL on torch's current stream of `device` (-1: no device argument).
int run(PackedFn fn, SetStreamFn set_stream, TVMValue* values, int* codes, int n, int device) {
  TVMValue ret;
  int ret_code = 0;
  ret.v_int64 = 0;
#if SPTIR_TORCH_CUDA  // without it torch has no CUDA tensors
  if (device >= 0) {
    void* st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    if (set_stream(device, st) != 0) return -1;
  }
#else
  (void)set_stream;
  (void)device;
#endif
  const NoGil no_gil;
  return fn(values, codes, n, &ret, &ret_code, nullptr);
}

// C++ exceptions end at the functions below: a tensor without storage (inside torch.vmap, torch.func.jvp or
// FakeTensorMode) throws from data_ptr(), and an exception that reached the interpreter's C frames would
// end the process.

// invoke(fn, set_stream, args) -> return code, or None when an argument is of a kind that only the
// general packing on the Python side takes (or refuses with its message).
PyObject* invoke(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  HANDLE_TH_ERRORS
  if (argc != 3 || !PyTuple_Check(argv[2])) {
    PyErr_SetString(PyExc_TypeError, "invoke(fn, set_stream, args)");
    return nullptr;
  }
  const auto fn = reinterpret_cast<PackedFn>(PyLong_AsVoidPtr(argv[0]));
  const auto set_stream = reinterpret_cast<SetStreamFn>(PyLong_AsVoidPtr(argv[1]));
  if (fn == nullptr || set_stream == nullptr) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point");
    return nullptr;
  }
  constexpr int kInline = 48;
  const int n = static_cast<int>(PyTuple_GET_SIZE(argv[2]));
  TVMValue values_s[kInline];
  int codes_s[kInline];
  DLTensor dl_s[kInline];
  std::vector<TVMValue> values_v;
  std::vector<int> codes_v;
  std::vector<DLTensor> dl_v;
  TVMValue* values = values_s;
  int* codes = codes_s;
  DLTensor* dl = dl_s;
  if (n > kInline) {
    values_v.resize(n);
    codes_v.resize(n);
    dl_v.resize(n);
    values = values_v.data();
    codes = codes_v.data();
    dl = dl_v.data();
  }
  int device = -1;
  for (int i = 0; i < n; ++i) {
    PyObject* o = PyTuple_GET_ITEM(argv[2], i);
    if (THPVariable_Check(o)) {
      const at::Tensor& t = THPVariable_Unpack(o);
      DLTensor& d = dl[i];
      if (t.layout() != c10::kStrided || !(t.is_cuda() || t.is_cpu()) || !dl_type(t.scalar_type(), &d.dtype))
        Py_RETURN_NONE;
      d.data = t.numel() > 0 ? t.data_ptr() : nullptr;
      d.ndim = static_cast<int32_t>(t.dim());
      d.shape = const_cast<int64_t*>(t.sizes().data());
      d.strides = t.is_contiguous() ? nullptr : const_cast<int64_t*>(t.strides().data());
      d.byte_offset = 0;
      if (t.is_cuda()) {
        d.device = DLDevice{kDLCUDA, t.get_device()};
        if (device < 0) device = t.get_device();
      } else {
        d.device = DLDevice{kDLCPU, 0};
      }
      values[i].v_handle = &d;
      codes[i] = kTVMDLTensorHandle;
    } else if (PyLong_Check(o)) {
      int overflow = 0;
      values[i].v_int64 = PyLong_AsLongLongAndOverflow(o, &overflow);
      if (overflow != 0) Py_RETURN_NONE;
      codes[i] = kTVMArgInt;
    } else if (PyFloat_Check(o)) {
      values[i].v_float64 = PyFloat_AS_DOUBLE(o);
      codes[i] = kTVMArgFloat;
    } else if (o == Py_None) {
      values[i].v_handle = nullptr;
      codes[i] = kTVMNullptr;
    } else {
      Py_RETURN_NONE;
    }
  }
  return PyLong_FromLong(run(fn, set_stream, values, codes, n, device));
  END_HANDLE_TH_ERRORS
}

// invoke_packed(fn, set_stream, values, codes, n, device): the call of argument arrays packed before
// (addresses of the arrays; device -1: no device argument).
PyObject* invoke_packed(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  HANDLE_TH_ERRORS
  if (argc != 6) {
    PyErr_SetString(PyExc_TypeError, "invoke_packed(fn, set_stream, values, codes, n, device)");
    return nullptr;
  }
  const auto fn = reinterpret_cast<PackedFn>(PyLong_AsVoidPtr(argv[0]));
  const auto set_stream = reinterpret_cast<SetStreamFn>(PyLong_AsVoidPtr(argv[1]));
  auto* values = static_cast<TVMValue*>(PyLong_AsVoidPtr(argv[2]));
  auto* codes = static_cast<int*>(PyLong_AsVoidPtr(argv[3]));
  const long n = PyLong_AsLong(argv[4]);
  const long device = PyLong_AsLong(argv[5]);
  if (PyErr_Occurred()) return nullptr;
  if (fn == nullptr || set_stream == nullptr || values == nullptr || codes == nullptr) {
    PyErr_SetString(PyExc_ValueError, "null address");
    return nullptr;
  }
  return PyLong_FromLong(run(fn, set_stream, values, codes, static_cast<int>(n), static_cast<int>(device)));
  END_HANDLE_TH_ERRORS
}

// flatten(list): replaces every tensor of the list that is not one-dimensional by its flat view
// (or copy, as Tensor.reshape(-1) decides), in place; returns the list.
PyObject* flatten(PyObject*, PyObject* list) {
  HANDLE_TH_ERRORS
  if (!PyList_Check(list)) {
    PyErr_SetString(PyExc_TypeError, "flatten(list)");
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
    PyObject* o = PyList_GET_ITEM(list, i);
    if (!THPVariable_Check(o) || THPVariable_Unpack(o).dim() == 1) continue;
    PyObject* flat = PyObject_CallMethod(o, "reshape", "i", -1);
    if (flat == nullptr) return nullptr;
    if (PyList_SetItem(list, i, flat) != 0) return nullptr;
  }
  Py_INCREF(list);
  return list;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"invoke", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(invoke)), METH_FASTCALL, nullptr},
    {"invoke_packed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(invoke_packed)), METH_FASTCALL, nullptr},
    {"flatten", flatten, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall() {
  PyObject* m = PyModule_Create(&module);
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", SPTIR_TORCH_VERSION) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
