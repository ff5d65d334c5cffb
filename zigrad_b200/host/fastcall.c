/* Calls into the device library's C ABI without ctypes.
 *
 * ctypes builds a libffi call description for every call: 1 to 3 us for an op of ten arguments, about what the kernel
 * launch itself costs, and more than a short kernel.  Here a function of the ABI is an object that converts its
 * arguments by a signature string and calls the address directly (zg_bmm: 3.2 -> 0.6 us).
 *
 * Signature characters: i integer (any width), b bool, p untyped pointer (int, None, bytes or a ctypes array), a pointer to
 * a given ctypes type (None or an array of it), s a given struct of one pointer (a ctypes structure), d double; return v
 * nothing, i int, u unsigned long, p pointer.
 * Under the x86-64 System V convention integers and one-pointer structs take rdi .. r9 and then the stack in order, doubles
 * xmm0 .. xmm7, independently of how they are interleaved, so one call through a prototype with six integers, eight
 * doubles and the rest of the integers serves every signature with at most eight doubles.
 *
 * What an argument's type does not fit goes to the fallback (the ctypes function), which converts it or raises. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>

#if !defined(__x86_64__) || !defined(__linux__)
#error "the call below is written for the x86-64 System V calling convention"
#endif

#define MAX_INTS 26
#define MAX_ARGS 34

typedef struct {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* address;
  PyObject* fallback;
  int n;
  char ret;
  char sig[MAX_ARGS];
  PyObject* types[MAX_ARGS]; /* the struct of an s, the element type of an a */
} Function;

typedef uint64_t (*Generic)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, double, double, double, double, double, double, double, double,
                            uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                            uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t);

/* Only what stands for its own memory: a c_void_p or a POINTER object has a buffer too, but holds the address to pass. */
static PyTypeObject* array_type;  /* ctypes.Array */
static PyObject* type_name;       /* "_type_" */

/* Whether `o` has the memory that argument `a` takes: what is nothing of the kind is for ctypes to convert or to refuse. */
static int stands(const Function* f, Py_ssize_t a, PyObject* o) {
  switch (f->sig[a]) {
    case 's': return PyObject_TypeCheck(o, (PyTypeObject*)f->types[a]);
    case 'p': return PyBytes_Check(o) || PyObject_TypeCheck(o, array_type);
    case 'a': {
      if (!PyObject_TypeCheck(o, array_type)) return 0;
      PyObject* t = PyObject_GetAttr((PyObject*)Py_TYPE(o), type_name);
      if (!t) PyErr_Clear();
      Py_XDECREF(t);
      return t == f->types[a];
    }
  }
  return 0;
}

static PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Function* f = (Function*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != f->n || kwnames) return PyObject_Vectorcall(f->fallback, args, nargsf, kwnames);
  uint64_t x[MAX_INTS] = {0};
  double d[8] = {0};
  Py_buffer held[8];
  int ni = 0, nd = 0, nh = 0, fits = 1;
  for (Py_ssize_t a = 0; a < n && fits; ++a) {
    PyObject* o = args[a];
    const char c = f->sig[a];
    if (c == 'd') {
      d[nd] = PyFloat_CheckExact(o) ? PyFloat_AS_DOUBLE(o) : PyFloat_AsDouble(o);
      if (d[nd] == -1.0 && PyErr_Occurred()) { PyErr_Clear(); fits = 0; }
      ++nd;
    } else if ((c == 'i' || c == 'p') && PyLong_Check(o)) {
      x[ni++] = PyLong_AsUnsignedLongLongMask(o);
      if (PyErr_Occurred()) { PyErr_Clear(); fits = 0; }
    } else if (c == 'b' && PyLong_Check(o)) {
      x[ni++] = (uint64_t)PyObject_IsTrue(o);
    } else if ((c == 'p' || c == 'a') && o == Py_None) {
      x[ni++] = 0;
    } else if (nh < 8 && stands(f, a, o)) {
      if (PyObject_GetBuffer(o, &held[nh], PyBUF_SIMPLE) != 0) { PyErr_Clear(); fits = 0; break; }
      const Py_buffer* b = &held[nh++];
      if (c != 's') x[ni++] = (uint64_t)(uintptr_t)b->buf;
      else if (b->len == (Py_ssize_t)sizeof(void*)) x[ni++] = *(const uint64_t*)b->buf;
      else fits = 0;
    } else {
      fits = 0;
    }
  }
  if (!fits) {
    while (nh) PyBuffer_Release(&held[--nh]);
    return PyObject_Vectorcall(f->fallback, args, nargsf, NULL);
  }
  uint64_t r;
  const Generic g = (Generic)f->address;
  Py_BEGIN_ALLOW_THREADS
  r = g(x[0], x[1], x[2], x[3], x[4], x[5], d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], x[6], x[7], x[8], x[9], x[10], x[11], x[12], x[13], x[14],
        x[15], x[16], x[17], x[18], x[19], x[20], x[21], x[22], x[23], x[24], x[25]);
  Py_END_ALLOW_THREADS
  while (nh) PyBuffer_Release(&held[--nh]);
  switch (f->ret) {
    case 'i': return PyLong_FromLong((int)r);
    case 'u': return PyLong_FromUnsignedLong((unsigned long)r);
    case 'p': if (r) return PyLong_FromUnsignedLongLong(r);  /* fall through: NULL is None */
    default: Py_RETURN_NONE;
  }
}

static void dealloc(PyObject* self) {
  Py_XDECREF(((Function*)self)->fallback);
  for (int a = 0; a < ((Function*)self)->n; ++a) Py_XDECREF(((Function*)self)->types[a]);
  Py_TYPE(self)->tp_free(self);
}

static PyObject* getattro(PyObject* self, PyObject* name) {  /* argtypes, restype, __name__, .. of the ctypes function */
  return PyObject_GetAttr(((Function*)self)->fallback, name);
}

static PyTypeObject FunctionType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "zigrad_b200._fastcall.Function",
    .tp_basicsize = sizeof(Function),
    .tp_dealloc = dealloc,
    .tp_vectorcall_offset = offsetof(Function, vectorcall),
    .tp_call = PyVectorcall_Call,
    .tp_getattro = getattro,
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
};

/* function(address, signature, return, fallback, types): a type or None per argument */
static PyObject* make(PyObject* module, PyObject* args) {
  (void)module;
  unsigned long long address;
  const char *sig, *ret;
  PyObject *fallback, *types;
  if (!PyArg_ParseTuple(args, "KssOO!", &address, &sig, &ret, &fallback, &PyTuple_Type, &types)) return NULL;
  size_t n = strlen(sig), doubles = 0;
  for (size_t i = 0; i < n; ++i) {
    if (!strchr("ibpasd", sig[i])) return PyErr_Format(PyExc_ValueError, "signature %s", sig);
    doubles += sig[i] == 'd';
    if (i >= (size_t)PyTuple_GET_SIZE(types) || (strchr("as", sig[i]) && !PyType_Check(PyTuple_GET_ITEM(types, (Py_ssize_t)i))))
      return PyErr_Format(PyExc_ValueError, "signature %s: no type for argument %zu", sig, i);
  }
  if (n > MAX_ARGS || doubles > 8 || n - doubles > MAX_INTS || strlen(ret) != 1 || !strchr("viup", ret[0]))
    return PyErr_Format(PyExc_ValueError, "signature %s -> %s", sig, ret);
  Function* f = PyObject_New(Function, &FunctionType);
  if (!f) return NULL;
  f->vectorcall = call;
  f->address = (void*)(uintptr_t)address;
  f->fallback = Py_NewRef(fallback);
  f->n = (int)n;
  f->ret = ret[0];
  memcpy(f->sig, sig, n);
  for (size_t i = 0; i < n; ++i) f->types[i] = Py_NewRef(PyTuple_GET_ITEM(types, (Py_ssize_t)i));
  return (PyObject*)f;
}

static PyMethodDef methods[] = {{"function", make, METH_VARARGS, "A callable for one function of the C ABI."}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
  if (PyType_Ready(&FunctionType) < 0) return NULL;
  PyObject* ctypes = PyImport_ImportModule("ctypes");
  if (!ctypes) return NULL;
  array_type = (PyTypeObject*)PyObject_GetAttrString(ctypes, "Array");
  type_name = PyUnicode_InternFromString("_type_");
  Py_DECREF(ctypes);
  if (!array_type || !type_name) return NULL;
  return PyModule_Create(&module_def);
}
