// Calls of the C ABI from Python without ctypes: an Entry is a callable with the address and the argument kinds of one function of
// libb200ops.so. ctypes converts an argument of a call in 60 - 100 ns and needs 0.4 us around them, 2 us for an entry point of 18 arguments,
// as long as the launch takes the driver; an Entry 0.2 us.
//
// Kinds: 'i' an integer of up to 64 bits (wrapped, as ctypes does), 'p' a pointer (an integer or None), 'f' a float. Whatever else
// comes (ctypes objects, another number of arguments, keywords) goes to the ctypes function that the Entry was made with, and so do errors.
//
// One function type serves every entry point: by the System V ABI of x86-64 integers and pointers take the six integer registers and then
// eight-byte slots of the stack in their own order, floats the vector registers in theirs (up to eight), and a callee looks at no
// more than it declares. Elsewhere (or with more arguments) no Entry is made.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#if !defined(__x86_64__) || defined(_WIN32)
#error "System V x86-64 only"
#endif

namespace {

constexpr int kInts = 32, kFloats = 8;
typedef uint64_t u;
typedef int (*Fn)(u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, float, float, float, float, float,
                  float, float, float);

struct Entry {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Fn fn;
  PyObject* slow;
  int n;
  char kinds[kInts + kFloats + 1];
};

PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  const Entry* e = reinterpret_cast<const Entry*>(self);
  if (PyVectorcall_NARGS(nargsf) != e->n || (kwnames && PyTuple_GET_SIZE(kwnames))) return PyObject_Vectorcall(e->slow, args, nargsf, kwnames);
  u a[kInts] = {0};
  float f[kFloats] = {0};
  int na = 0, nf = 0;
  for (int i = 0; i < e->n; ++i) {
    PyObject* x = args[i];
    if (e->kinds[i] == 'f') {
      if (PyFloat_Check(x)) f[nf++] = (float)PyFloat_AS_DOUBLE(x);
      else if (PyLong_Check(x)) {
        const double d = PyLong_AsDouble(x);
        if (d == -1.0 && PyErr_Occurred()) return nullptr;
        f[nf++] = (float)d;
      } else return PyObject_Vectorcall(e->slow, args, nargsf, kwnames);
    } else if (PyLong_Check(x)) a[na++] = PyLong_AsUnsignedLongLongMask(x);
    else if (x == Py_None && e->kinds[i] == 'p') a[na++] = 0;
    else return PyObject_Vectorcall(e->slow, args, nargsf, kwnames);
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = e->fn(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17], a[18], a[19], a[20],
             a[21], a[22], a[23], a[24], a[25], a[26], a[27], a[28], a[29], a[30], a[31], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

int traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<Entry*>(self)->slow);
  return 0;
}
int clear(PyObject* self) {
  Py_CLEAR(reinterpret_cast<Entry*>(self)->slow);
  return 0;
}
void dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  clear(self);
  Py_TYPE(self)->tp_free(self);
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// make(address, kinds, slow) -> Entry, or None where one cannot be made
PyObject* make(PyObject*, PyObject* args) {
  unsigned long long address;
  const char* kinds;
  PyObject* slow;
  if (!PyArg_ParseTuple(args, "KsO", &address, &kinds, &slow)) return nullptr;
  int ints = 0, floats = 0;
  for (const char* k = kinds; *k; ++k) {
    if (*k == 'f') ++floats;
    else if (*k == 'i' || *k == 'p') ++ints;
    else Py_RETURN_NONE;
  }
  if (!address || ints > kInts || floats > kFloats) Py_RETURN_NONE;
  Entry* e = PyObject_GC_New(Entry, &EntryType);
  if (!e) return nullptr;
  e->vectorcall = call;
  e->fn = reinterpret_cast<Fn>(static_cast<uintptr_t>(address));
  Py_INCREF(slow);
  e->slow = slow;
  e->n = ints + floats;
  memset(e->kinds, 0, sizeof(e->kinds));
  strcpy(e->kinds, kinds);
  PyObject_GC_Track(reinterpret_cast<PyObject*>(e));
  return reinterpret_cast<PyObject*>(e);
}

PyMethodDef methods[] = {{"make", make, METH_VARARGS, "make(address, kinds, slow) -> callable or None"}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200_fastcall(void) {
  EntryType.tp_name = "_b200_fastcall.Entry";
  EntryType.tp_basicsize = sizeof(Entry);
  EntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL;
  EntryType.tp_vectorcall_offset = offsetof(Entry, vectorcall);
  EntryType.tp_call = PyVectorcall_Call;
  EntryType.tp_traverse = traverse;
  EntryType.tp_clear = clear;
  EntryType.tp_dealloc = dealloc;
  EntryType.tp_free = PyObject_GC_Del;
  if (PyType_Ready(&EntryType) < 0) return nullptr;
  return PyModule_Create(&module);
}
