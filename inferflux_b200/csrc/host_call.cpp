// Calls of the kernel library's C entry points from Python, in place of ctypes: a small layer's launches take the GPU a few microseconds
// each, and ctypes an object an argument and as long a call.
//
//   Function(address, wide, tensor_type, signature)(...)    integers, floats (as float32), None (null) and tensors (their data_ptr());
//                                                           also objects with a `value` of those (ctypes' own)
//
// signature: a letter an argument, p pointer, i int, l long long, f float.  A call with another count of arguments or with an argument of
// another kind raises TypeError; a pointer may be an integer, and an integer in the place of a float is passed as a float.  (Without a
// signature arguments are passed as what they are.)
//
// The entry points take pointers, integers and up to eight floats.  By the System V convention of x86-64 the first six integers and
// pointers go to general registers, floats to vector registers and further integers to the stack, eight bytes each and in order, so one
// signature with room for all of them reaches every such function: what is too much is not read.  The interpreter's lock is let go for
// the call, as ctypes does.
//
// A call of 14 arguments costs the host 0.3 us beside its launch; through ctypes and an object an argument it was 7.0.  Layers that the host
// bounds, us: a feed-forward of few rows 50.7 -> 39.5, a recurrence of 60 tokens 92.6 -> 73.7, a mixture of few 56.0 -> 43.7.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstdint>
#include <cstring>

#if !defined(__x86_64__) || !defined(__linux__)
#error "host_call.cpp is written for the System V calling convention of x86-64 (build.py leaves it out elsewhere)"
#endif

namespace {

constexpr int kRegisters = 6, kFloats = 8, kFew = 16, kMost = 48;

struct Function {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* address;
  PyObject* tensor_type;
  PyObject* signature;                                     // ASCII, or null
  int wide;                                                // returns long long, not int
};

struct Arguments {
  uint64_t integers[kRegisters + kMost] = {};
  double floats[kFloats] = {};
  int integer = 0, real = 0;
};

PyObject* g_data_ptr = nullptr;
PyObject* g_value = nullptr;

bool add_integer(Arguments& a, PyObject* v) {
  if (a.integer == kRegisters + kMost) {
    PyErr_SetString(PyExc_TypeError, "too many arguments");
    return false;
  }
  const uint64_t x = PyLong_AsUnsignedLongLongMask(v);
  if (x == (uint64_t)-1 && PyErr_Occurred()) return false;
  a.integers[a.integer++] = x;
  return true;
}

bool add_float(Arguments& a, double v) {
  if (a.real == kFloats) {
    PyErr_SetString(PyExc_TypeError, "more than eight floats");
    return false;
  }
  const float f = (float)v;
  std::memcpy(&a.floats[a.real++], &f, sizeof f);
  return true;
}

bool refuse(PyObject* v, char kind) {
  PyErr_Format(PyExc_TypeError, "cannot pass a %s as %s", Py_TYPE(v)->tp_name, kind == 'p' ? "a pointer" : kind == 'f' ? "a float" : "an integer");
  return false;
}

// kind: a signature's letter, or 0
bool add(Arguments& a, PyObject* v, PyObject* tensor_type, char kind, int depth) {
  if (v == Py_None) return kind == 0 || kind == 'p' ? add_integer(a, Py_False) : refuse(v, kind);
  if (PyLong_Check(v)) {
    if (kind != 'f') return add_integer(a, v);
    const double x = PyLong_AsDouble(v);
    return x == -1.0 && PyErr_Occurred() ? false : add_float(a, x);
  }
  if (PyFloat_Check(v)) return kind == 0 || kind == 'f' ? add_float(a, PyFloat_AS_DOUBLE(v)) : refuse(v, kind);
  PyObject* inner;
  if (PyObject_TypeCheck(v, (PyTypeObject*)tensor_type)) {
    if (kind != 0 && kind != 'p') return refuse(v, kind);
    PyObject* self[1] = {v};
    inner = PyObject_VectorcallMethod(g_data_ptr, self, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
  } else {
    inner = depth == 0 ? PyObject_GetAttr(v, g_value) : nullptr;
    if (!inner && !PyErr_Occurred()) PyErr_Format(PyExc_TypeError, "cannot pass a %s", Py_TYPE(v)->tp_name);
  }
  if (!inner) return false;
  const bool ok = add(a, inner, tensor_type, kind, 1);
  Py_DECREF(inner);
  return ok;
}

#define IFX_R uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t
#define IFX_F double, double, double, double, double, double, double, double
#define IFX_8 uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t
using Few = int64_t (*)(IFX_R, IFX_F, IFX_8, IFX_8);
using Most = int64_t (*)(IFX_R, IFX_F, IFX_8, IFX_8, IFX_8, IFX_8, IFX_8, IFX_8);
#define IFX_S(i) s[i], s[i + 1], s[i + 2], s[i + 3], s[i + 4], s[i + 5], s[i + 6], s[i + 7]

int64_t invoke(void* address, const Arguments& a) {
  const uint64_t *r = a.integers, *s = r + kRegisters;
  const double* f = a.floats;
  if (a.integer <= kRegisters + kFew)
    return reinterpret_cast<Few>(address)(r[0], r[1], r[2], r[3], r[4], r[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], IFX_S(0), IFX_S(8));
  return reinterpret_cast<Most>(address)(r[0], r[1], r[2], r[3], r[4], r[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], IFX_S(0), IFX_S(8),
                                         IFX_S(16), IFX_S(24), IFX_S(32), IFX_S(40));
}

PyObject* call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* names) {
  const Function* self = reinterpret_cast<Function*>(callable);
  if (names && PyTuple_GET_SIZE(names)) {
    PyErr_SetString(PyExc_TypeError, "no keyword arguments");
    return nullptr;
  }
  Arguments a;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  const char* kinds = nullptr;
  if (self->signature) {
    kinds = reinterpret_cast<const char*>(PyUnicode_1BYTE_DATA(self->signature));
    if (n != PyUnicode_GET_LENGTH(self->signature)) {
      PyErr_Format(PyExc_TypeError, "%zd arguments instead of %zd", n, PyUnicode_GET_LENGTH(self->signature));
      return nullptr;
    }
  }
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!add(a, args[i], self->tensor_type, kinds ? kinds[i] : 0, 0)) return nullptr;
  int64_t result;
  Py_BEGIN_ALLOW_THREADS
  result = invoke(self->address, a);
  Py_END_ALLOW_THREADS
  return PyLong_FromLongLong(self->wide ? result : (int64_t)(int32_t)result);
}

PyObject* make(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long address;
  int wide;
  PyObject *tensor_type, *signature = nullptr;
  if (!PyArg_ParseTuple(args, "KpO!|U", &address, &wide, &PyType_Type, &tensor_type, &signature)) return nullptr;
  if (signature && !PyUnicode_IS_ASCII(signature)) {
    PyErr_SetString(PyExc_ValueError, "a signature has the letters p, i, l and f");
    return nullptr;
  }
  Function* self = reinterpret_cast<Function*>(type->tp_alloc(type, 0));
  if (!self) return nullptr;
  self->vectorcall = call;
  self->address = reinterpret_cast<void*>((uintptr_t)address);
  self->wide = wide;
  Py_INCREF(tensor_type);
  self->tensor_type = tensor_type;
  Py_XINCREF(signature);
  self->signature = signature;
  return reinterpret_cast<PyObject*>(self);
}

void drop(PyObject* o) {
  Py_XDECREF(reinterpret_cast<Function*>(o)->tensor_type);
  Py_XDECREF(reinterpret_cast<Function*>(o)->signature);
  Py_TYPE(o)->tp_free(o);
}

PyTypeObject function_type = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_ifx_host", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ifx_host(void) {
  function_type.tp_name = "_ifx_host.Function";
  function_type.tp_basicsize = sizeof(Function);
  function_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  function_type.tp_vectorcall_offset = offsetof(Function, vectorcall);
  function_type.tp_call = PyVectorcall_Call;
  function_type.tp_new = make;
  function_type.tp_dealloc = drop;
  if (PyType_Ready(&function_type) < 0) return nullptr;
  g_data_ptr = PyUnicode_InternFromString("data_ptr");
  g_value = PyUnicode_InternFromString("value");
  PyObject* m = PyModule_Create(&module_def);
  if (!m || !g_data_ptr || !g_value) return nullptr;
  Py_INCREF(&function_type);
  if (PyModule_AddObject(m, "Function", reinterpret_cast<PyObject*>(&function_type)) < 0) return nullptr;
  return m;
}
