/* hostpath.c — the marshalling half of run_vectors (spoc_b200/plugin.py) as a CPython extension.
 *
 * A launch of a short kernel spends most of its time above the C ABI: walking the arguments, expanding every vector to
 * (buffer, int32 length) as the reference does (sarek/sarek/Execute.ml:197-216), filling the argument table.  Interpreted,
 * that took 12 us of a 17 us launch; here it takes under 1 us.  Only the case a running program meets every time is
 * handled: all vectors already on the device, nothing on its way back or to be sent back behind the launch, plain Python scalars.  Everything else
 * returns None and takes the interpreted path, which also raises the errors.
 *
 * The library is not linked: bind() receives the address of sb200_kernel_launch from the ctypes binding. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "../../include/sb200.h"

typedef int (*launch_fn)(uint64_t, const sb200_arg *, int, const uint32_t *, const uint32_t *, uint32_t, uint64_t);

#define MAX_ARGS 64
#define SEND_BACK_BYTES (16u << 20) /* Vector.PIN_MIN_BYTES */

static launch_fn g_launch;
static PyObject *g_vector_type;              /* plugin.Vector */
static PyObject *g_cpu, *g_both, *g_stale;   /* its location constants */
static PyObject *s_buffer, *s_location, *s_pinned, *s_prefetch, *s_host, *s_ptr, *s_x, *s_y, *s_z;

static int same_text(PyObject *a, PyObject *b) { return a == b || (PyUnicode_Check(a) && PyUnicode_Compare(a, b) == 0); }

/* A non-negative integer attribute; -1 when it is missing, no int, or out of range. */
static long long int_attr(PyObject *o, PyObject *name) {
  PyObject *v = PyObject_GetAttr(o, name);
  if (!v) {
    PyErr_Clear();
    return -1;
  }
  int over = 0;
  long long r = PyLong_CheckExact(v) ? PyLong_AsLongLongAndOverflow(v, &over) : -1;
  Py_DECREF(v);
  if (PyErr_Occurred()) PyErr_Clear();
  return over ? -1 : r;
}

static int dims(PyObject *d, uint32_t out[3]) {
  const long long x = int_attr(d, s_x), y = int_attr(d, s_y), z = int_attr(d, s_z);
  if (x < 0 || y < 0 || z < 0 || x > UINT32_MAX || y > UINT32_MAX || z > UINT32_MAX) return 0;
  out[0] = (uint32_t)x;
  out[1] = (uint32_t)y;
  out[2] = (uint32_t)z;
  return 1;
}

/* Appends (buffer, length) of a vector whose device copy is the valid one; 0 when the vector is in any other state.
 * *both is set when the host copy is valid too. */
static int push_vector(PyObject *v, sb200_arg *args, int *n, int *both) {
  int ok = 0;
  PyObject *buffer = NULL, *location = NULL, *pinned = NULL, *prefetch = NULL, *host = NULL;
  if (!(buffer = PyObject_GetAttr(v, s_buffer)) || buffer == Py_None) goto out;
  if (!(location = PyObject_GetAttr(v, s_location)) || same_text(location, g_cpu)) goto out;
  if (!(pinned = PyObject_GetAttr(v, s_pinned)) || (pinned != Py_False && pinned != Py_True)) goto out;
  if (!(prefetch = PyObject_GetAttr(v, s_prefetch)) || prefetch != Py_None) goto out;
  if (!(host = PyObject_GetAttr(v, s_host))) goto out;
  {
    PyObject *ptr = PyObject_GetAttr(buffer, s_ptr);
    const Py_ssize_t len = PyObject_Size(host);
    if (!ptr) goto out;
    if (pinned == Py_True && (uint64_t)len * 4 >= SEND_BACK_BYTES) { /* its result would follow the launch to the host */
      Py_DECREF(ptr);
      goto out;
    }
    const unsigned long long address = PyLong_CheckExact(ptr) ? PyLong_AsUnsignedLongLong(ptr) : 0;
    Py_DECREF(ptr);
    if (PyErr_Occurred() || address == 0 || len < 0 || len > INT32_MAX) goto out;
    args[*n].tag = SB200_ARG_BUFFER;
    args[*n].reserved = 0;
    args[*n].v.buffer = address;
    args[*n + 1].tag = SB200_ARG_I32;
    args[*n + 1].reserved = 0;
    args[*n + 1].v.buffer = 0;
    args[*n + 1].v.i32 = (int32_t)len;
    *n += 2;
    *both = same_text(location, g_both);
    ok = 1;
  }
out:
  if (PyErr_Occurred()) PyErr_Clear();
  Py_XDECREF(buffer);
  Py_XDECREF(location);
  Py_XDECREF(pinned);
  Py_XDECREF(prefetch);
  Py_XDECREF(host);
  return ok;
}

/* Appends a ("int32" | "int64" | "float32" | "float64", value) pair with a plain Python number. */
static int push_scalar(PyObject *pair, sb200_arg *a) {
  if (!PyTuple_CheckExact(pair) || PyTuple_GET_SIZE(pair) != 2) return 0;
  PyObject *kind = PyTuple_GET_ITEM(pair, 0), *value = PyTuple_GET_ITEM(pair, 1);
  if (!PyUnicode_Check(kind)) return 0;
  a->reserved = 0;
  a->v.buffer = 0;
  if (PyUnicode_CompareWithASCIIString(kind, "int32") == 0 || PyUnicode_CompareWithASCIIString(kind, "int64") == 0) {
    int over = 0;
    if (!PyLong_CheckExact(value)) return 0;
    const long long i = PyLong_AsLongLongAndOverflow(value, &over);
    if (over) return 0;
    if (PyUnicode_CompareWithASCIIString(kind, "int32") == 0) {
      if (i < INT32_MIN || i > INT32_MAX) return 0;
      a->tag = SB200_ARG_I32;
      a->v.i32 = (int32_t)i;
    } else {
      a->tag = SB200_ARG_I64;
      a->v.i64 = i;
    }
    return 1;
  }
  if (!PyFloat_CheckExact(value)) return 0;
  const double f = PyFloat_AS_DOUBLE(value);
  if (PyUnicode_CompareWithASCIIString(kind, "float32") == 0) {
    a->tag = SB200_ARG_F32;
    a->v.f32 = (float)f;
    return 1;
  }
  if (PyUnicode_CompareWithASCIIString(kind, "float64") == 0) {
    a->tag = SB200_ARG_F64;
    a->v.f64 = f;
    return 1;
  }
  return 0;
}

/* launch(kernel_handle, args, block, grid, shared_mem) -> status of sb200_kernel_launch, or None when the arguments are
 * not all of the simple kind (nothing has been launched then).  On success every vector whose host copy was valid is
 * marked stale (Execute.ml:321-335). */
static PyObject *hp_launch(PyObject *self, PyObject *const *a, Py_ssize_t na) {
  (void)self;
  if (na != 5 || !g_launch) {
    PyErr_SetString(PyExc_TypeError, "launch(handle, args, block, grid, shared_mem) after bind()");
    return NULL;
  }
  const unsigned long long handle = PyLong_AsUnsignedLongLong(a[0]);
  const long shared = PyLong_AsLong(a[4]);
  uint32_t block[3], grid[3];
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (!dims(a[2], block) || !dims(a[3], grid) || shared < 0) Py_RETURN_NONE;
  if (!PyList_CheckExact(a[1]) && !PyTuple_CheckExact(a[1])) Py_RETURN_NONE;
  const Py_ssize_t count = PySequence_Fast_GET_SIZE(a[1]);
  if (2 * count > MAX_ARGS) Py_RETURN_NONE;
  sb200_arg args[MAX_ARGS];
  PyObject *items[MAX_ARGS / 2];
  uint32_t both_mask = 0;
  int n = 0;
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject *item = PySequence_Fast_GET_ITEM(a[1], i);
    items[i] = item;
    if ((PyObject *)Py_TYPE(item) == g_vector_type) {
      int both = 0;
      if (!push_vector(item, args, &n, &both)) Py_RETURN_NONE;
      if (both) both_mask |= 1u << i;
    } else {
      if (!push_scalar(item, &args[n])) Py_RETURN_NONE;
      ++n;
    }
  }
  int rc;
  for (Py_ssize_t i = 0; i < count; ++i) Py_INCREF(items[i]); /* the caller's list may change while the lock is away */
  Py_BEGIN_ALLOW_THREADS
  rc = g_launch(handle, args, n, grid, block, (uint32_t)shared, 0);
  Py_END_ALLOW_THREADS
  int failed = 0;
  for (Py_ssize_t i = 0; i < count; ++i) {
    if (rc == 0 && (both_mask >> i & 1u) && !failed) failed = PyObject_SetAttr(items[i], s_location, g_stale) != 0;
    Py_DECREF(items[i]);
  }
  if (failed) return NULL;
  return PyLong_FromLong(rc);
}

/* bind(address of sb200_kernel_launch, Vector) */
static PyObject *hp_bind(PyObject *self, PyObject *args) {
  (void)self;
  unsigned long long address;
  PyObject *vector_type, *cpu, *both, *stale;
  if (!PyArg_ParseTuple(args, "KO", &address, &vector_type)) return NULL;
  cpu = PyObject_GetAttrString(vector_type, "CPU");
  both = PyObject_GetAttrString(vector_type, "BOTH");
  stale = PyObject_GetAttrString(vector_type, "STALE_CPU");
  if (!cpu || !both || !stale) {
    Py_XDECREF(cpu);
    Py_XDECREF(both);
    Py_XDECREF(stale);
    return NULL;
  }
  Py_INCREF(vector_type);
  g_vector_type = vector_type; /* kept for the life of the process, as are the constants and names */
  g_cpu = cpu;
  g_both = both;
  g_stale = stale;
  g_launch = (launch_fn)(uintptr_t)address;
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"launch", (PyCFunction)(void (*)(void))hp_launch, METH_FASTCALL, "launch a kernel on vectors that are on the device"},
    {"bind", hp_bind, METH_VARARGS, "address of sb200_kernel_launch and the Vector class"},
    {NULL, NULL, 0, NULL}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hostpath", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__hostpath(void) {
  s_buffer = PyUnicode_InternFromString("buffer");
  s_location = PyUnicode_InternFromString("location");
  s_pinned = PyUnicode_InternFromString("_pinned");
  s_prefetch = PyUnicode_InternFromString("_prefetch_dev");
  s_host = PyUnicode_InternFromString("host");
  s_ptr = PyUnicode_InternFromString("ptr");
  s_x = PyUnicode_InternFromString("x");
  s_y = PyUnicode_InternFromString("y");
  s_z = PyUnicode_InternFromString("z");
  return PyModule_Create(&module);
}
