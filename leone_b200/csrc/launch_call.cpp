// Calls of the kernels' C entry points from Python without libffi.
//
// A step makes hundreds of launches; ctypes takes 2 us to convert the 25 to 35 arguments of one, and the objects that it wants
// for pointers and floats take as long again to make.  `bind(address)` gives a callable that reads the arguments where they are:
// a tensor stands for its data pointer, None for a null pointer, an int for an integer or a pointer, a float for a C float.
// The entry points take pointers, integers and floats (no double, no structure) and return an int.
//
// One prototype serves them all: by the System V ABI of x86-64 and the procedure call standard of 64-bit Arm, integers and pointers
// go to the integer registers in their order and then to 8-byte places on the stack, and up to eight floats to vector registers,
// whatever stands between them.  Places past a function's arguments are not read.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cstddef>
#include <cstring>

#define EIGHT(X, o) X(o), X(o + 1), X(o + 2), X(o + 3), X(o + 4), X(o + 5), X(o + 6), X(o + 7)
#if defined(__x86_64__)
#define LEONE_INT_REGISTERS 6
#define REGISTERS(X) X(0), X(1), X(2), X(3), X(4), X(5)
#elif defined(__aarch64__) && !defined(__APPLE__)
#define LEONE_INT_REGISTERS 8
#define REGISTERS(X) EIGHT(X, 0)
#else
#error "argument passing of this platform is not described here"
#endif
#define TYPE(k) L
#define VALUE(k) i[k]
#define PLACE(k) s[k]
#define FLOAT(k) float
#define FLOAT_VALUE(k) f[k]

namespace {

constexpr int kMostFloats = 8, kMostInts = LEONE_INT_REGISTERS + 40;
typedef long long L;

struct Entry {
  PyObject_HEAD
  vectorcallfunc call;
  void* address;
};

PyObject* g_data_ptr = nullptr;      // the name "data_ptr"

// -1: an error is set
int take(PyObject* a, L* ints, int& ni, float* floats, int& nf) {
  if (PyFloat_Check(a)) {
    if (nf == kMostFloats) { PyErr_SetString(PyExc_TypeError, "too many float arguments"); return -1; }
    floats[nf++] = (float)PyFloat_AS_DOUBLE(a);
    return 0;
  }
  if (ni == kMostInts) { PyErr_SetString(PyExc_TypeError, "too many integer arguments"); return -1; }
  if (a == Py_None) {
    ints[ni++] = 0;
    return 0;
  }
  PyObject* number = nullptr;
  if (!PyLong_Check(a)) {
    number = PyObject_CallMethodNoArgs(a, g_data_ptr);
    if (number == nullptr) return -1;
    a = number;
  }
  int overflow = 0;
  L v = PyLong_AsLongLongAndOverflow(a, &overflow);
  if (overflow > 0) v = (L)PyLong_AsUnsignedLongLong(a);       // an address in the upper half
  Py_XDECREF(number);
  if (overflow < 0) PyErr_SetString(PyExc_OverflowError, "an argument does not fit 64 bits");
  if ((overflow != 0 || v == -1) && PyErr_Occurred()) return -1;
  ints[ni++] = v;
  return 0;
}

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
  if (names != nullptr && PyTuple_GET_SIZE(names) != 0) {
    PyErr_SetString(PyExc_TypeError, "an entry point takes no named arguments");
    return nullptr;
  }
  L i[kMostInts];
  float f[kMostFloats];
  memset(i, 0, sizeof(i));
  memset(f, 0, sizeof(f));
  int ni = 0, nf = 0;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  for (Py_ssize_t k = 0; k < n; ++k)
    if (take(args[k], i, ni, f, nf) != 0) return nullptr;
  void* const p = ((Entry*)self)->address;
  const L* s = i + LEONE_INT_REGISTERS;
  int r;
  Py_BEGIN_ALLOW_THREADS                                        // (as a call through ctypes does)
  if (ni <= LEONE_INT_REGISTERS + 16)
    r = ((int (*)(REGISTERS(TYPE), EIGHT(FLOAT, 0), EIGHT(TYPE, 0), EIGHT(TYPE, 8)))p)(REGISTERS(VALUE), EIGHT(FLOAT_VALUE, 0),
                                                                                       EIGHT(PLACE, 0), EIGHT(PLACE, 8));
  else
    r = ((int (*)(REGISTERS(TYPE), EIGHT(FLOAT, 0), EIGHT(TYPE, 0), EIGHT(TYPE, 8), EIGHT(TYPE, 16), EIGHT(TYPE, 24), EIGHT(TYPE, 32)))p)(
        REGISTERS(VALUE), EIGHT(FLOAT_VALUE, 0), EIGHT(PLACE, 0), EIGHT(PLACE, 8), EIGHT(PLACE, 16), EIGHT(PLACE, 24), EIGHT(PLACE, 32));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(r);
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* bind(PyObject*, PyObject* address) {
  void* p = PyLong_AsVoidPtr(address);
  if (p == nullptr) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "a null address");
    return nullptr;
  }
  Entry* e = PyObject_New(Entry, &EntryType);
  if (e == nullptr) return nullptr;
  e->call = entry_call;
  e->address = p;
  return (PyObject*)e;
}

PyMethodDef methods[] = {{"bind", bind, METH_O, "A callable for the C function at this address."}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "libleone_call", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_libleone_call(void) {
  EntryType.tp_name = "libleone_call.Entry";
  EntryType.tp_basicsize = sizeof(Entry);
  EntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  EntryType.tp_vectorcall_offset = offsetof(Entry, call);
  EntryType.tp_call = PyVectorcall_Call;
  if (PyType_Ready(&EntryType) < 0) return nullptr;
  g_data_ptr = PyUnicode_InternFromString("data_ptr");
  if (g_data_ptr == nullptr) return nullptr;
  return PyModule_Create(&module);
}
