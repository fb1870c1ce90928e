// The calls from Python into the compiled launchers: a prompt step of a small model is some 300 of them, and with ctypes and checks
// written in Python each cost more than the driver's launch (a launcher of seven arguments 5.0 us, 2.2 of them the launch).
//
//   Launcher  one extern "C" function with its declared argument types.  A pointer takes None, a tensor's address as an int, or the
//             tensor itself; integers are cut to their width and floats rounded, as ctypes does.  The interpreter's lock is released
//             while the function runs.
//   ptr       a tensor's address (None: None)
//   stream    the current stream's handle
//   need      a tensor's device, type and layout; what does not hold goes on to the Python check, which says what is wrong
//   mm        out = x . w^T in bfloat16 by the vendor library, called as `torch.mm` calls it (the same handle, workspace, stream,
//             algorithm and math mode), without the dispatcher's 4 us; False for what only `torch.mm` should decide
//
// The table of argument types is generated from launchers.py when this file is compiled.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/Context.h>
#include <ATen/cuda/CUDAContext.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <tuple>
#include <utility>

namespace {

bool take(PyObject* o, void** v) {
  if (o == Py_None) {
    *v = nullptr;
    return true;
  }
  if (PyLong_Check(o)) {
    *v = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(o));
    return !PyErr_Occurred();
  }
  if (THPVariable_Check(o)) {
    *v = THPVariable_Unpack(o).data_ptr();
    return true;
  }
  PyErr_Format(PyExc_TypeError, "a pointer argument is None, an address or a tensor, not %s", Py_TYPE(o)->tp_name);
  return false;
}
bool whole(PyObject* o, unsigned long long* v) {
  if (!PyLong_Check(o)) {
    PyErr_Format(PyExc_TypeError, "an integer argument is an int, not %s", Py_TYPE(o)->tp_name);
    return false;
  }
  *v = PyLong_AsUnsignedLongLongMask(o);
  return !(*v == ~0ull && PyErr_Occurred());
}
bool take(PyObject* o, int* v) {
  unsigned long long w;
  if (!whole(o, &w)) return false;
  *v = static_cast<int>(w);
  return true;
}
bool take(PyObject* o, long long* v) {
  unsigned long long w;
  if (!whole(o, &w)) return false;
  *v = static_cast<long long>(w);
  return true;
}
bool take(PyObject* o, float* v) {
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) return false;
  *v = static_cast<float>(d);
  return true;
}

using Call = PyObject* (*)(void*, PyObject* const*, Py_ssize_t);

template <class R, class... A, std::size_t... N>
PyObject* invoke(void* fn, PyObject* const* args, std::index_sequence<N...>) {
  std::tuple<A...> v;
  if (!(take(args[N], &std::get<N>(v)) && ...)) return nullptr;
  if constexpr (std::is_void_v<R>) {
    Py_BEGIN_ALLOW_THREADS
    reinterpret_cast<R (*)(A...)>(fn)(std::get<N>(v)...);
    Py_END_ALLOW_THREADS
    Py_RETURN_NONE;
  } else {
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = reinterpret_cast<R (*)(A...)>(fn)(std::get<N>(v)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong(r);
  }
}
template <class R, class... A>
PyObject* call(void* fn, PyObject* const* args, Py_ssize_t n) {
  if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
    PyErr_Format(PyExc_TypeError, "this launcher takes %zd arguments (%zd given)", static_cast<Py_ssize_t>(sizeof...(A)), n);
    return nullptr;
  }
  return invoke<R, A...>(fn, args, std::index_sequence_for<A...>{});
}

using P = void*;
using I = int;
using F = float;
using LL = long long;
struct Entry {
  const char* name;
  Call call;
};
const Entry table[] = {
#include "native_table.inc"
};

struct Launcher {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Call call;
  void* fn;
};

PyObject* launcher_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  if (kwnames != nullptr && PyTuple_GET_SIZE(kwnames) != 0) {
    PyErr_SetString(PyExc_TypeError, "a launcher takes no keyword arguments");
    return nullptr;
  }
  Launcher* l = reinterpret_cast<Launcher*>(self);
  return l->call(l->fn, args, PyVectorcall_NARGS(nargsf));
}

PyTypeObject LauncherType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* slow_need = nullptr;  // the Python check

PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "bind(name, address)");
    return nullptr;
  }
  const char* name = PyUnicode_AsUTF8(args[0]);
  if (name == nullptr) return nullptr;
  void* fn = PyLong_AsVoidPtr(args[1]);
  if (fn == nullptr) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: no address");
    return nullptr;
  }
  for (const Entry& e : table)
    if (std::strcmp(e.name, name) == 0) {
      Launcher* l = PyObject_New(Launcher, &LauncherType);
      if (l == nullptr) return nullptr;
      l->vectorcall = launcher_call;
      l->call = e.call;
      l->fn = fn;
      return reinterpret_cast<PyObject*>(l);
    }
  PyErr_Format(PyExc_KeyError, "no launcher %s in the table this module was built with", name);
  return nullptr;
}

PyObject* ptr(PyObject*, PyObject* o) {
  if (o == Py_None) Py_RETURN_NONE;
  if (!THPVariable_Check(o)) return PyObject_CallMethod(o, "data_ptr", nullptr);
  return PyLong_FromVoidPtr(THPVariable_Unpack(o).data_ptr());
}

PyObject* stream(PyObject*, PyObject*) {
  try {
    return PyLong_FromVoidPtr(at::cuda::getCurrentCUDAStream().stream());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

PyObject* set_slow_need(PyObject*, PyObject* o) {
  Py_INCREF(o);
  Py_XSETREF(slow_need, o);
  Py_RETURN_NONE;
}

// need(tensor, name, dtype=None, contiguous=True)
PyObject* need(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) {
  const Py_ssize_t named = kwnames == nullptr ? 0 : PyTuple_GET_SIZE(kwnames);
  if (n >= 2 && n + named <= 4 && THPVariable_Check(args[0])) {
    PyObject* dtype = n > 2 ? args[2] : Py_None;
    PyObject* contiguous = n > 3 ? args[3] : Py_True;
    bool known = true;
    for (Py_ssize_t i = 0; i < named; ++i) {
      PyObject* k = PyTuple_GET_ITEM(kwnames, i);
      if (n <= 2 && PyUnicode_CompareWithASCIIString(k, "dtype") == 0) dtype = args[n + i];
      else if (n <= 3 && PyUnicode_CompareWithASCIIString(k, "contiguous") == 0) contiguous = args[n + i];
      else known = false;
    }
    if (known && (dtype == Py_None || THPDtype_Check(dtype))) {
      const at::Tensor& t = THPVariable_Unpack(args[0]);
      const int dense = PyObject_IsTrue(contiguous);
      if (dense < 0) return nullptr;
      if (t.is_cuda() && (dtype == Py_None || t.scalar_type() == reinterpret_cast<THPDtype*>(dtype)->scalar_type) &&
          (!dense || t.is_contiguous()))
        Py_RETURN_NONE;
    }
  }
  return PyObject_Vectorcall(slow_need, args, n, kwnames);
}

// mm(x, w, out): out [M, N] (bfloat16 or float32) = x [M, K] . w [N, K]^T in bfloat16
PyObject* mm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1]) || !THPVariable_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "mm(x, w, out): three tensors");
    return nullptr;
  }
  const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]), &out = THPVariable_Unpack(args[2]);
  if (x.dim() != 2 || w.dim() != 2 || out.dim() != 2 || !x.is_cuda() || !w.is_cuda() || !out.is_cuda()) Py_RETURN_FALSE;
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  const bool wide = out.scalar_type() == at::kFloat;
  if (M < 2 || N < 2 || K < 2 || M > INT_MAX || N > INT_MAX || K > INT_MAX || w.size(1) != K || out.size(0) != M || out.size(1) != N ||
      x.scalar_type() != at::kBFloat16 || w.scalar_type() != at::kBFloat16 || !(wide || out.scalar_type() == at::kBFloat16) ||
      !x.is_contiguous() || !w.is_contiguous() || !out.is_contiguous() || x.get_device() != w.get_device() ||
      x.get_device() != out.get_device() || x.get_device() != at::cuda::current_device() || x.requires_grad() || w.requires_grad() ||
      out.requires_grad())
    Py_RETURN_FALSE;
  at::Context& context = at::globalContext();
  if (context.allowBF16ReductionCuBLAS() != at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK ||
      context.deterministicAlgorithms())
    Py_RETURN_FALSE;
  cublasStatus_t rc;
  try {
    cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
    const float one = 1.f, zero = 0.f;
    Py_BEGIN_ALLOW_THREADS
    rc = cublasGemmEx(handle, CUBLAS_OP_T, CUBLAS_OP_N, static_cast<int>(N), static_cast<int>(M), static_cast<int>(K), &one,
                      w.data_ptr(), CUDA_R_16BF, static_cast<int>(K), x.data_ptr(), CUDA_R_16BF, static_cast<int>(K), &zero,
                      out.data_ptr(), wide ? CUDA_R_32F : CUDA_R_16BF, static_cast<int>(N), CUBLAS_COMPUTE_32F,
                      CUBLAS_GEMM_DEFAULT_TENSOR_OP);
    Py_END_ALLOW_THREADS
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  if (rc != CUBLAS_STATUS_SUCCESS) {
    PyErr_Format(PyExc_RuntimeError, "cublasGemmEx (%lld x %lld . %lld x %lld) answered %d", static_cast<long long>(M),
                 static_cast<long long>(K), static_cast<long long>(N), static_cast<long long>(K), static_cast<int>(rc));
    return nullptr;
  }
  Py_RETURN_TRUE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, "the Launcher of a function's name and address"},
    {"ptr", ptr, METH_O, "a tensor's address"},
    {"need", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(need)), METH_FASTCALL | METH_KEYWORDS, "checks a tensor"},
    {"stream", stream, METH_NOARGS, "the current stream's handle on the current device"},
    {"set_slow_need", set_slow_need, METH_O, "the check that `need` falls back to"},
    {"mm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(mm)), METH_FASTCALL, "a bfloat16 product by the vendor library"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "ullm_b200_native", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_ullm_b200_native() {
  LauncherType.tp_name = "ullm_b200_native.Launcher";
  LauncherType.tp_basicsize = sizeof(Launcher);
  LauncherType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  LauncherType.tp_vectorcall_offset = offsetof(Launcher, vectorcall);
  LauncherType.tp_call = PyVectorcall_Call;
  LauncherType.tp_dealloc = [](PyObject* o) { PyObject_Free(o); };
  if (PyType_Ready(&LauncherType) < 0) return nullptr;
  return PyModule_Create(&module);
}
