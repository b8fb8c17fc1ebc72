// The entry points of the C ABI as Python callables that convert their arguments in C++ (module dromos_b200._calls).
//
// A decode step is hundreds of calls of 10 to 17 arguments whose kernels take a few microseconds each; a GEMV's 15 arguments took ctypes
// 5.1 us, here it is 0.9. What is converted: ints, floats, None, c_void_p objects and
// abi.WeightRef, which is what this package passes. A call with anything else goes, as it is, to the ctypes function that is kept
// behind the callable, so it is accepted, refused or converted as it always was. That function also stands in for the callable as an
// argument of ctypes (cast), and once one of its attributes is set (errcheck, restype) it takes all calls. The interpreter lock is
// released during a call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "dromos_b200.h"

namespace {

PyObject* g_void_p = nullptr;      // ctypes.c_void_p
PyObject* g_weight_ref = nullptr;  // abi.WeightRef
PyObject *g_value = nullptr, *g_address = nullptr;  // the names "value" and "address"

struct Function {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* fn;
  PyObject* slow;
  bool plain;  // an attribute of `slow` has been set: what it does to calls is for ctypes to do
};

// An address from an int; false for anything else (no Python error is left set).
bool address_of(PyObject* o, void*& out) {
  if (!PyLong_CheckExact(o)) return false;
  const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
  if (v == ~0ull && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  out = reinterpret_cast<void*>(static_cast<uintptr_t>(v));
  return true;
}
bool address_attribute(PyObject* o, PyObject* name, void*& out) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (!v) {
    PyErr_Clear();
    return false;
  }
  bool ok = true;
  if (v == Py_None) out = nullptr;
  else ok = address_of(v, out);
  Py_DECREF(v);
  return ok;
}

template <typename T>
bool take(PyObject* o, T& out) {
  using Pointee = std::remove_cv_t<std::remove_pointer_t<T>>;
  if constexpr (std::is_pointer_v<T> && std::is_same_v<Pointee, lx_weight>) {
    void* p = nullptr;
    if (reinterpret_cast<PyObject*>(Py_TYPE(o)) != g_weight_ref || !address_attribute(o, g_address, p)) return false;
    out = static_cast<T>(p);
    return true;
  } else if constexpr (std::is_pointer_v<T>) {
    void* p = nullptr;
    if (o != Py_None && !(reinterpret_cast<PyObject*>(Py_TYPE(o)) == g_void_p ? address_attribute(o, g_value, p) : address_of(o, p))) return false;
    out = static_cast<T>(p);
    return true;
  } else if constexpr (std::is_floating_point_v<T>) {
    if (!PyFloat_CheckExact(o)) return false;
    out = static_cast<T>(PyFloat_AS_DOUBLE(o));
    return true;
  } else {
    if (!PyLong_CheckExact(o)) return false;
    int overflow = 0;
    const long long v = PyLong_AsLongLongAndOverflow(o, &overflow);
    if (overflow) return false;
    out = static_cast<T>(v);
    return true;
  }
}

template <typename Fn>
struct Call;
template <typename R, typename... A>
struct Call<R(A...)> {
  template <size_t... I>
  static bool convert(PyObject* const* args, std::tuple<A...>& to, std::index_sequence<I...>) {
    return (take(args[I], std::get<I>(to)) && ...);
  }
  static PyObject* run(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
    auto* f = reinterpret_cast<Function*>(self);
    std::tuple<A...> to;
    if (f->plain || names || PyVectorcall_NARGS(nargsf) != static_cast<Py_ssize_t>(sizeof...(A)) || !convert(args, to, std::index_sequence_for<A...>{}))
      return PyObject_Vectorcall(f->slow, args, nargsf, names);
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = std::apply(reinterpret_cast<R (*)(A...)>(f->fn), to);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong(static_cast<long long>(r));
  }
};

struct Entry {
  const char* name;
  vectorcallfunc call;
};
#define ENTRY(f) {#f, &Call<std::remove_pointer_t<decltype(&f)>>::run}
const Entry kEntries[] = {
    ENTRY(lx_gemv_w),
    ENTRY(lx_gemm_w),
    ENTRY(lx_gemm_workspace_bytes),
    ENTRY(lx_gemm_skinny),
    ENTRY(lx_dequantize_weight),
    ENTRY(lx_bf16x_row_bytes),
    ENTRY(lx_bf16x_bytes),
    ENTRY(lx_bf16x_encode),
    ENTRY(lx_bf16x_decode),
    ENTRY(lx_moe_route),
    ENTRY(lx_moe_experts_grouped),
    ENTRY(lx_moe_grouped_workspace_bytes),
    ENTRY(lx_moe_experts_decode),
    ENTRY(lx_moe_decode_workspace_bytes),
};
#undef ENTRY

void function_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<Function*>(self)->slow);
  Py_TYPE(self)->tp_free(self);
}
PyObject* function_getattro(PyObject* self, PyObject* name) {  // restype, argtypes and the like: the ctypes function's
  PyObject* slow = reinterpret_cast<Function*>(self)->slow;
  if (PyUnicode_Check(name) && PyUnicode_CompareWithASCIIString(name, "_as_parameter_") == 0) return Py_NewRef(slow);
  return PyObject_GetAttr(slow, name);
}
int function_setattro(PyObject* self, PyObject* name, PyObject* value) {
  auto* f = reinterpret_cast<Function*>(self);
  if (PyObject_SetAttr(f->slow, name, value) != 0) return -1;
  f->plain = true;
  return 0;
}

PyTypeObject g_function_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

bool ready_function_type() {
  PyTypeObject& t = g_function_type;
  t.tp_name = "dromos_b200._calls.Function";
  t.tp_basicsize = sizeof(Function);
  t.tp_dealloc = function_dealloc;
  t.tp_vectorcall_offset = offsetof(Function, vectorcall);
  t.tp_call = PyVectorcall_Call;
  t.tp_getattro = function_getattro;
  t.tp_setattro = function_setattro;
  t.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  t.tp_doc = "An entry point; calls with unusual arguments go to the ctypes function it was made from.";
  return PyType_Ready(&t) == 0;
}

// bind(name, address, ctypes function) -> callable, or the ctypes function itself where there is none for that name
PyObject* bind(PyObject*, PyObject* args) {
  const char* name;
  unsigned long long address;
  PyObject* slow;
  if (!PyArg_ParseTuple(args, "sKO", &name, &address, &slow)) return nullptr;
  for (const Entry& e : kEntries) {
    if (std::strcmp(e.name, name) != 0) continue;
    Function* f = PyObject_New(Function, &g_function_type);
    if (!f) return nullptr;
    f->vectorcall = e.call;
    f->fn = reinterpret_cast<void*>(static_cast<uintptr_t>(address));
    f->slow = Py_NewRef(slow);
    f->plain = false;
    return reinterpret_cast<PyObject*>(f);
  }
  return Py_NewRef(slow);
}

// setup(c_void_p, WeightRef)
PyObject* setup(PyObject*, PyObject* args) {
  PyObject *v, *w;
  if (!PyArg_ParseTuple(args, "OO", &v, &w)) return nullptr;
  Py_XSETREF(g_void_p, Py_NewRef(v));
  Py_XSETREF(g_weight_ref, Py_NewRef(w));
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"bind", bind, METH_VARARGS, "bind(name, address, ctypes function)"},
                          {"setup", setup, METH_VARARGS, "setup(c_void_p, WeightRef)"},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", "The C ABI's entry points with arguments converted in C++.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  if (!ready_function_type()) return nullptr;
  if (!(g_value = PyUnicode_InternFromString("value")) || !(g_address = PyUnicode_InternFromString("address"))) return nullptr;
  return PyModule_Create(&kModule);
}
