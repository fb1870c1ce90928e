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
//   record / recorded / alike / replay
//             the launches of a layer as a list, and the same list run for another layer of the same make: two layers are recorded as
//             they launch, `alike` finds every argument equal but for addresses inside the layers' own tensors, and `replay` runs the
//             list with those addresses moved to a third layer's.  A list lives as long as the step that recorded it.
//
// The table of argument types is generated from launchers.py when this file is compiled.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/Context.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/tunable/Tunable.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <exception>
#include <tuple>
#include <utility>
#include <vector>

namespace {

// What a function called from Python answers where C++ threw (a tensor without storage, the library's handle): Python's exception for it.
PyObject* thrown(const std::exception_ptr& e = std::current_exception()) {
  try {
    std::rethrow_exception(e);
  } catch (const std::exception&) {
    torch::translate_exception_to_python(e);
  } catch (...) {
    PyErr_SetString(PyExc_RuntimeError, "an unknown C++ exception");
  }
  return nullptr;
}

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

// ---- lists of launches ----------------------------------------------------------------------------------------------------------
constexpr int MAX_ARGS = 48;
struct Value {
  unsigned long long bits = 0;
  bool address = false;
};
Value value(void* p) { return {reinterpret_cast<unsigned long long>(p), true}; }
Value value(int i) { return {static_cast<unsigned long long>(static_cast<long long>(i)), false}; }
Value value(long long i) { return {static_cast<unsigned long long>(i), false}; }
Value value(float f) {
  unsigned u;
  std::memcpy(&u, &f, 4);
  return {u, false};
}
void back(unsigned long long bits, void** v) { *v = reinterpret_cast<void*>(bits); }
void back(unsigned long long bits, int* v) { *v = static_cast<int>(bits); }
void back(unsigned long long bits, long long* v) { *v = static_cast<long long>(bits); }
void back(unsigned long long bits, float* v) {
  const unsigned u = static_cast<unsigned>(bits);
  std::memcpy(v, &u, 4);
}
using Again = long long (*)(void*, const unsigned long long*);
struct Launch {
  Again again;
  void* fn;
  int n;
  Value v[MAX_ARGS];
};
struct Moved {  // argument `arg` of launch `launch` lies `offset` bytes into tensor `tensor` of the layer
  int launch, arg, tensor;
  unsigned long long offset;
};
struct Span {  // a layer's tensor; `bytes` 0: not in one piece
  unsigned long long at, bytes;
  int type, device;
  bool like(const Span& o) const { return bytes == o.bytes && type == o.type && device == o.device; }
};
struct Tape {
  PyObject_HEAD
  std::vector<Launch>* launches;
  std::vector<Moved>* moved;               // null: not compared yet
  std::vector<Span>* make;                 // of the compared layers' tensors: how long they are, and of what
  bool whole;                              // nothing ran that is not in the list
};
thread_local Tape* recording = nullptr;

template <class R, class... A, std::size_t... N>
long long again_as(void* fn, const unsigned long long* bits, std::index_sequence<N...>) {
  std::tuple<A...> v;
  (back(bits[N], &std::get<N>(v)), ...);
  if constexpr (std::is_void_v<R>) {
    reinterpret_cast<R (*)(A...)>(fn)(std::get<N>(v)...);
    return 0;
  } else {
    return static_cast<long long>(reinterpret_cast<R (*)(A...)>(fn)(std::get<N>(v)...));
  }
}
template <class R, class... A>
long long again(void* fn, const unsigned long long* bits) {
  return again_as<R, A...>(fn, bits, std::index_sequence_for<A...>{});
}
template <class... A>
void note(Again how, void* fn, const A&... args) {
  static_assert(sizeof...(A) <= MAX_ARGS, "a launcher's arguments fit the list");
  Launch l = {how, fn, static_cast<int>(sizeof...(A)), {}};
  int i = 0;
  ((l.v[i++] = value(args)), ...);
  recording->launches->push_back(l);
}

using Call = PyObject* (*)(void*, PyObject* const*, Py_ssize_t);

// LISTED: launches and settings, not questions
template <bool LISTED, class R, class... A, std::size_t... N>
PyObject* invoke(void* fn, PyObject* const* args, std::index_sequence<N...>) try {
  std::tuple<A...> v;
  if (!(take(args[N], &std::get<N>(v)) && ...)) return nullptr;
  if (LISTED && recording != nullptr) note(again<R, A...>, fn, std::get<N>(v)...);
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
    if (LISTED && recording != nullptr && r != 0) recording->whole = false;  // (what follows depends on it)
    return PyLong_FromLongLong(r);
  }
} catch (...) {
  return thrown();  // (of the arguments: a launcher throws nothing)
}
template <bool LISTED, class R, class... A>
PyObject* call(void* fn, PyObject* const* args, Py_ssize_t n) {
  if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
    PyErr_Format(PyExc_TypeError, "this launcher takes %zd arguments (%zd given)", static_cast<Py_ssize_t>(sizeof...(A)), n);
    return nullptr;
  }
  return invoke<LISTED, R, A...>(fn, args, std::index_sequence_for<A...>{});
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

PyObject* ptr(PyObject*, PyObject* o) try {
  if (o == Py_None) Py_RETURN_NONE;
  if (!THPVariable_Check(o)) return PyObject_CallMethod(o, "data_ptr", nullptr);
  return PyLong_FromVoidPtr(THPVariable_Unpack(o).data_ptr());
} catch (...) {
  return thrown();
}

PyObject* stream(PyObject*, PyObject*) try {
  return PyLong_FromVoidPtr(at::cuda::getCurrentCUDAStream().stream());
} catch (...) {
  return thrown();
}

PyObject* set_slow_need(PyObject*, PyObject* o) {
  Py_INCREF(o);
  Py_XSETREF(slow_need, o);
  Py_RETURN_NONE;
}

// need(tensor, name, dtype=None, contiguous=True)
PyObject* need(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) try {
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
} catch (...) {
  return thrown();
}

// out [M, N] (bfloat16, or float32 where `wide`) = x [M, K] . w [N, K]^T, on the current stream; the library's status
int product(void* x, void* w, void* out, int M, int N, int K, int wide) {
  const float one = 1.f, zero = 0.f;
  return cublasGemmEx(at::cuda::getCurrentCUDABlasHandle(), CUBLAS_OP_T, CUBLAS_OP_N, N, M, K, &one, w, CUDA_R_16BF, K, x, CUDA_R_16BF,
                      K, &zero, out, wide ? CUDA_R_32F : CUDA_R_16BF, N, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
}

// As a list runs it: a launcher's codes are 0 and above, the library's status counts down from there.
int listed_product(void* x, void* w, void* out, int M, int N, int K, int wide) { return -product(x, w, out, M, N, K, wide); }

// Whether `torch.mm` would be this product and nothing besides: nobody watches or replaces torch's operations (profilers, dispatch and
// function modes, subclasses, transforms), and no setting picks another library or algorithm.
bool plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.has_storage() && !t.key_set().has(c10::DispatchKey::Python) && !t.requires_grad() && !t._fw_grad(0).defined();
}
bool as_torch_does() {
  if (at::hasCallbacks() || c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled()) return false;
  at::Context& context = at::globalContext();
  const at::BlasBackend library = context.blasPreferredBackend();
  return (library == at::BlasBackend::Default || library == at::BlasBackend::Cublas) &&
         context.allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK &&
         !context.deterministicAlgorithms() && !at::cuda::tunable::getTuningContext()->IsTunableOpEnabled();
}

// mm(x, w, out): the product, False for what only `torch.mm` should decide
PyObject* mm(PyObject*, PyObject* const* args, Py_ssize_t n) try {
  if (n != 3 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1]) || !THPVariable_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "mm(x, w, out): three tensors");
    return nullptr;
  }
  const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]), &out = THPVariable_Unpack(args[2]);
  if (!plain(args[0]) || !plain(args[1]) || !plain(args[2])) Py_RETURN_FALSE;
  if (x.dim() != 2 || w.dim() != 2 || out.dim() != 2 || !x.is_cuda() || !w.is_cuda() || !out.is_cuda()) Py_RETURN_FALSE;
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  const bool wide = out.scalar_type() == at::kFloat;
  if (M < 2 || N < 2 || K < 2 || M > INT_MAX || N > INT_MAX || K > INT_MAX || w.size(1) != K || out.size(0) != M || out.size(1) != N ||
      x.scalar_type() != at::kBFloat16 || w.scalar_type() != at::kBFloat16 || !(wide || out.scalar_type() == at::kBFloat16) ||
      !x.is_contiguous() || !w.is_contiguous() || !out.is_contiguous() || x.get_device() != w.get_device() ||
      x.get_device() != out.get_device() || x.get_device() != at::cuda::current_device() || !as_torch_does())
    Py_RETURN_FALSE;
  void *px = x.data_ptr(), *pw = w.data_ptr(), *po = out.data_ptr();
  const int m = static_cast<int>(M), nn = static_cast<int>(N), k = static_cast<int>(K), f = wide ? 1 : 0;
  if (recording != nullptr)
    note(again<int, void*, void*, void*, int, int, int, int>, reinterpret_cast<void*>(listed_product), px, pw, po, m, nn, k, f);
  int rc = 0;
  std::exception_ptr failed;
  Py_BEGIN_ALLOW_THREADS
  try {
    rc = product(px, pw, po, m, nn, k, f);
  } catch (...) {
    failed = std::current_exception();
  }
  Py_END_ALLOW_THREADS
  if (failed || rc != 0) {
    if (recording != nullptr) recording->whole = false;
    if (failed) return thrown(failed);
    PyErr_Format(PyExc_RuntimeError, "cublasGemmEx (%d x %d . %d x %d) answered %d", m, k, nn, k, rc);
    return nullptr;
  }
  Py_RETURN_TRUE;
} catch (...) {
  return thrown();
}

// ---- record, compare, run again ---------------------------------------------------------------------------------------------------
PyTypeObject TapeType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* record(PyObject*, PyObject*) {
  Tape* t = PyObject_New(Tape, &TapeType);
  if (t == nullptr) return nullptr;
  t->launches = new std::vector<Launch>;
  t->launches->reserve(32);
  t->moved = nullptr;
  t->make = nullptr;
  t->whole = true;
  Py_XDECREF(reinterpret_cast<PyObject*>(recording));
  recording = t;
  Py_RETURN_NONE;
}
// work that is not in the list is about to run
PyObject* unlisted(PyObject*, PyObject*) {
  if (recording != nullptr) recording->whole = false;
  Py_RETURN_NONE;
}
// ends the recording: the list, or None where something ran beside it
PyObject* recorded(PyObject*, PyObject*) {
  Tape* t = recording;
  recording = nullptr;
  if (t == nullptr) Py_RETURN_NONE;
  if (!t->whole || t->launches->empty()) {
    Py_DECREF(reinterpret_cast<PyObject*>(t));
    Py_RETURN_NONE;
  }
  return reinterpret_cast<PyObject*>(t);
}

bool spans(PyObject* tensors, std::vector<Span>* out) {
  if (!PyTuple_Check(tensors)) {
    PyErr_SetString(PyExc_TypeError, "a layer's tensors are a tuple");
    return false;
  }
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(tensors); ++i) {
    PyObject* o = PyTuple_GET_ITEM(tensors, i);
    if (!THPVariable_Check(o)) {
      PyErr_SetString(PyExc_TypeError, "a layer's tensors are tensors");
      return false;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    out->push_back({reinterpret_cast<unsigned long long>(t.data_ptr()), t.is_contiguous() ? static_cast<unsigned long long>(t.nbytes()) : 0,
                    static_cast<int>(t.scalar_type()), t.is_cuda() ? t.get_device() : -1});
  }
  return true;
}
bool is_tape(PyObject* o) {
  if (Py_TYPE(o) == &TapeType) return true;
  PyErr_SetString(PyExc_TypeError, "not a recorded list");
  return false;
}

// alike(a, a's tensors, b, b's tensors): whether b's list is a's with the addresses moved; b can then be replayed
PyObject* alike(PyObject*, PyObject* const* args, Py_ssize_t n) try {
  if (n != 4) {
    PyErr_SetString(PyExc_TypeError, "alike(a, tensors of a, b, tensors of b)");
    return nullptr;
  }
  if (!is_tape(args[0]) || !is_tape(args[2])) return nullptr;
  Tape *a = reinterpret_cast<Tape*>(args[0]), *b = reinterpret_cast<Tape*>(args[2]);
  std::vector<Span> sa, sb;
  if (!spans(args[1], &sa) || !spans(args[3], &sb)) return nullptr;
  if (sa.size() != sb.size() || a->launches->size() != b->launches->size()) Py_RETURN_FALSE;
  for (size_t i = 0; i < sa.size(); ++i)
    if (!sa[i].like(sb[i]) || sa[i].bytes == 0) Py_RETURN_FALSE;
  std::vector<Moved> moved;
  for (size_t l = 0; l < a->launches->size(); ++l) {
    const Launch &x = (*a->launches)[l], &y = (*b->launches)[l];
    if (x.fn != y.fn || x.again != y.again || x.n != y.n) Py_RETURN_FALSE;
    for (int i = 0; i < x.n; ++i) {
      int tensor = -1;
      if (y.v[i].address)
        for (size_t t = 0; t < sb.size() && tensor < 0; ++t)
          if (y.v[i].bits >= sb[t].at && y.v[i].bits < sb[t].at + sb[t].bytes) tensor = static_cast<int>(t);
      if (tensor < 0) {
        if (x.v[i].bits != y.v[i].bits) Py_RETURN_FALSE;  // (what differs has to lie in a tensor of the layer's)
        continue;
      }
      const unsigned long long offset = y.v[i].bits - sb[tensor].at;
      if (x.v[i].bits != sa[tensor].at + offset) Py_RETURN_FALSE;
      moved.push_back({static_cast<int>(l), i, tensor, offset});
    }
  }
  delete b->moved;
  delete b->make;
  b->moved = new std::vector<Moved>(std::move(moved));
  b->make = new std::vector<Span>(std::move(sb));
  Py_RETURN_TRUE;
} catch (...) {
  return thrown();
}

// replay(list, tensors of another layer): runs it there; the first launch's code that is not 0 (below it: the library's status,
// negated), else 0
PyObject* replay(PyObject*, PyObject* const* args, Py_ssize_t n) try {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "replay(list, tensors)");
    return nullptr;
  }
  if (!is_tape(args[0])) return nullptr;
  Tape* t = reinterpret_cast<Tape*>(args[0]);
  if (t->moved == nullptr) {
    PyErr_SetString(PyExc_ValueError, "replay: a list that has not been compared");
    return nullptr;
  }
  std::vector<Span> to;
  if (!spans(args[1], &to)) return nullptr;
  bool same = to.size() == t->make->size();  // (the launches take sizes and types from the layer that was recorded)
  for (size_t i = 0; same && i < to.size(); ++i) same = to[i].like((*t->make)[i]);
  if (!same) {
    PyErr_SetString(PyExc_ValueError, "replay: tensors of another make");
    return nullptr;
  }
  long long code = 0;
  std::exception_ptr failed;
  Py_BEGIN_ALLOW_THREADS
  try {
    size_t at = 0;
    for (size_t l = 0; l < t->launches->size() && code == 0; ++l) {
      const Launch& launch = (*t->launches)[l];
      unsigned long long bits[MAX_ARGS];
      for (int i = 0; i < launch.n; ++i) bits[i] = launch.v[i].bits;
      for (; at < t->moved->size() && (*t->moved)[at].launch == static_cast<int>(l); ++at)
        bits[(*t->moved)[at].arg] = to[(*t->moved)[at].tensor].at + (*t->moved)[at].offset;
      code = launch.again(launch.fn, bits);
    }
  } catch (...) {
    failed = std::current_exception();
  }
  Py_END_ALLOW_THREADS
  if (failed) return thrown(failed);
  return PyLong_FromLongLong(code);
} catch (...) {
  return thrown();
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, "the Launcher of a function's name and address"},
    {"ptr", ptr, METH_O, "a tensor's address"},
    {"need", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(need)), METH_FASTCALL | METH_KEYWORDS, "checks a tensor"},
    {"stream", stream, METH_NOARGS, "the current stream's handle on the current device"},
    {"set_slow_need", set_slow_need, METH_O, "the check that `need` falls back to"},
    {"mm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(mm)), METH_FASTCALL, "a bfloat16 product by the vendor library"},
    {"record", record, METH_NOARGS, "begins a list of this thread's launches"},
    {"unlisted", unlisted, METH_NOARGS, "work that the list cannot hold is about to run"},
    {"recorded", recorded, METH_NOARGS, "the list, or None"},
    {"alike", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(alike)), METH_FASTCALL, "whether two lists differ by their tensors alone"},
    {"replay", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(replay)), METH_FASTCALL, "runs a list with other tensors"},
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
  TapeType.tp_name = "ullm_b200_native.Tape";
  TapeType.tp_basicsize = sizeof(Tape);
  TapeType.tp_flags = Py_TPFLAGS_DEFAULT;
  TapeType.tp_dealloc = [](PyObject* o) {
    delete reinterpret_cast<Tape*>(o)->launches;
    delete reinterpret_cast<Tape*>(o)->moved;
    delete reinterpret_cast<Tape*>(o)->make;
    PyObject_Free(o);
  };
  if (PyType_Ready(&LauncherType) < 0 || PyType_Ready(&TapeType) < 0) return nullptr;
  return PyModule_Create(&module);
}
