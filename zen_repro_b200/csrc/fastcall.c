/* Calls into the native library without ctypes' marshalling.
 *
 * Every exported function of libzen_b200.so takes integers, pointers and floats and returns an int.  Under the System V x86-64
 * convention integer and pointer arguments fill the integer registers and then 8-byte stack slots in order, floats fill the
 * vector registers in order, whatever their order in the prototype; a callee ignores what it does not declare.  So one call
 * form (all integers, then all floats) reaches every function, and a call costs the conversion of its Python numbers: about
 * 0.2 us for 20 arguments, where ctypes took 4 to 5 us, which an eager training step pays about a hundred times.
 *
 * Arguments: int (also bool; pointers are ints), float, None (null pointer), and the ctypes objects that describe structures:
 * byref(x), arrays and structures are passed by address, simple values by value. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <structmember.h>
#include <stdint.h>

#define MAX_INTS 28
#define MAX_FLOATS 8

typedef struct {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* fn;
} FastFn;

typedef int (*any_fn)(int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                      int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                      int64_t, int64_t, int64_t, int64_t, float, float, float, float, float, float, float, float);

/* The address of a ctypes object.  Anything else with a buffer is refused, as ctypes itself does: a NumPy integer has one too, and
 * its address would pass for its value. */
static int address_of(PyObject* o, int64_t* out) {
  Py_buffer view;
  PyObject* owner = PyObject_GetAttrString(o, "_b_needsfree_");
  if (!owner) {
    PyErr_Format(PyExc_TypeError, "native call: cannot pass %.100s", Py_TYPE(o)->tp_name);
    return -1;
  }
  Py_DECREF(owner);
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) return -1;
  *out = (int64_t)(intptr_t)view.buf;     /* the object outlives the call: the caller's argument list holds it */
  PyBuffer_Release(&view);
  return 0;
}

static int convert_other(PyObject* a, int64_t* iv, int* ni, float* fv, int* nf) {
  PyObject* x = PyObject_GetAttrString(a, "_obj");                 /* ctypes.byref */
  if (x) {
    const int rc = address_of(x, &iv[(*ni)++]);
    Py_DECREF(x);
    return rc;
  }
  PyErr_Clear();
  x = PyObject_GetAttrString(a, "value");                          /* c_int, c_float, c_void_p, ... */
  if (x) {
    int rc = 0;
    if (PyFloat_Check(x)) fv[(*nf)++] = (float)PyFloat_AS_DOUBLE(x);
    else if (PyLong_Check(x)) iv[(*ni)++] = (int64_t)PyLong_AsUnsignedLongLongMask(x);
    else if (x == Py_None) iv[(*ni)++] = 0;
    else rc = -1;
    Py_DECREF(x);
    if (rc) PyErr_SetString(PyExc_TypeError, "native call: unsupported ctypes value");
    return rc;
  }
  PyErr_Clear();
  return address_of(a, &iv[(*ni)++]);
}

static PyObject* fast_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kw) {
  FastFn* f = (FastFn*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  int64_t iv[MAX_INTS + 1] = {0};
  float fv[MAX_FLOATS + 1] = {0};
  int ni = 0, nf = 0, rc;
  if (kw && PyTuple_GET_SIZE(kw)) {
    PyErr_SetString(PyExc_TypeError, "native call: no keyword arguments");
    return NULL;
  }
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* a = args[i];
    if (ni >= MAX_INTS || nf >= MAX_FLOATS) {
      PyErr_SetString(PyExc_TypeError, "native call: too many arguments");
      return NULL;
    }
    if (PyLong_Check(a)) iv[ni++] = (int64_t)PyLong_AsUnsignedLongLongMask(a);
    else if (PyFloat_Check(a)) fv[nf++] = (float)PyFloat_AS_DOUBLE(a);
    else if (a == Py_None) iv[ni++] = 0;
    else if (convert_other(a, iv, &ni, fv, &nf) != 0) return NULL;
  }
  Py_BEGIN_ALLOW_THREADS
  rc = ((any_fn)f->fn)(iv[0], iv[1], iv[2], iv[3], iv[4], iv[5], iv[6], iv[7], iv[8], iv[9], iv[10], iv[11], iv[12], iv[13], iv[14],
                       iv[15], iv[16], iv[17], iv[18], iv[19], iv[20], iv[21], iv[22], iv[23], iv[24], iv[25], iv[26], iv[27], fv[0],
                       fv[1], fv[2], fv[3], fv[4], fv[5], fv[6], fv[7]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyMemberDef fast_members[] = {{"__vectorcalloffset__", T_PYSSIZET, offsetof(FastFn, vectorcall), READONLY, NULL}, {NULL, 0, 0, 0, NULL}};
static PyType_Slot fast_slots[] = {{Py_tp_call, (void*)PyVectorcall_Call}, {Py_tp_members, fast_members}, {0, NULL}};
static PyType_Spec fast_spec = {"zen_fastcall.Function", sizeof(FastFn), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL, fast_slots};
static PyTypeObject* fast_type = NULL;

static PyObject* make(PyObject* m, PyObject* args) {
  unsigned long long addr;
  (void)m;
  if (!PyArg_ParseTuple(args, "K", &addr)) return NULL;
  FastFn* f = PyObject_New(FastFn, fast_type);
  if (!f) return NULL;
  f->vectorcall = fast_call;
  f->fn = (void*)(uintptr_t)addr;
  return (PyObject*)f;
}

static PyMethodDef methods[] = {{"function", make, METH_VARARGS, "function(address)"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef mod = {PyModuleDef_HEAD_INIT, "zen_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_zen_fastcall(void) {
  fast_type = (PyTypeObject*)PyType_FromSpec(&fast_spec);
  if (!fast_type) return NULL;
  return PyModule_Create(&mod);
}
