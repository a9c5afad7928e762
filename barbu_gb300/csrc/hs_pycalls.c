/* hs_pycalls.c -- the per-frame calls of the Python binding without ctypes.
 *
 * A ctypes call costs about 0.6 us before the library sees it (argument
 * objects, conversions) and an array's address 0.3 us more, where a small
 * groom's whole frame takes the GPU a few microseconds. Each function here
 * takes the C function's address, the groom's handle (a c_void_p, or None for
 * NULL) and the Python arguments, and returns the call's status; it returns
 * None, having called nothing, for arguments it does not take (a dt that is
 * not a float, an array that is not contiguous native float32 or has another
 * size), which the binding's general path converts or refuses. Measured,
 * three states in turn: class Hair on 448 strands 5.4 -> 3.5 us a frame (two
 * calls), 4,096 strands x 16 with a transform and a sphere 7.0 -> 4.8 us
 * (three). The GIL is released during the call, as ctypes does.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <string.h>

static PyObject* str_value;

/* A c_void_p's pointer; 0 (no Python error set) if `o` is something else. */
static int pointer_of(PyObject* o, void** out) {
  *out = NULL;
  if (o == Py_None) return 1;
  PyObject* v = PyObject_GetAttr(o, str_value);
  if (!v) {
    PyErr_Clear();
    return 0;
  }
  int ok = 1;
  if (v != Py_None) {
    ok = PyLong_CheckExact(v);
    if (ok) *out = PyLong_AsVoidPtr(v);
  }
  Py_DECREF(v);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    ok = 0;
  }
  return ok;
}

/* A C-contiguous buffer of native floats; 0 (no error set) otherwise. */
static int floats_of(PyObject* o, Py_buffer* b) {
  if (PyObject_GetBuffer(o, b, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) != 0) {
    PyErr_Clear();
    return 0;
  }
  if (b->itemsize == sizeof(float) && b->format && strcmp(b->format, "f") == 0) return 1;
  PyBuffer_Release(b);
  return 0;
}

static void* address_of(PyObject* o) {
  void* p = PyLong_CheckExact(o) ? PyLong_AsVoidPtr(o) : NULL;
  if (PyErr_Occurred()) PyErr_Clear();
  return p;
}

/* frame(f, handle, dt): int f(void*, float). */
static PyObject* frame(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void* h;
  int (*f)(void*, float) = n == 3 ? (int (*)(void*, float))address_of(args[0]) : NULL;
  if (!f || !PyFloat_CheckExact(args[2]) || !pointer_of(args[1], &h)) Py_RETURN_NONE;
  const float dt = (float)PyFloat_AS_DOUBLE(args[2]);
  int st;
  Py_BEGIN_ALLOW_THREADS;
  st = f(h, dt);
  Py_END_ALLOW_THREADS;
  return PyLong_FromLong(st);
}

/* floats(f, handle, array, count): int f(void*, const float*), an array of
 * exactly `count` floats. */
static PyObject* floats(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void* h;
  Py_buffer b;
  int (*f)(void*, const float*) = n == 4 ? (int (*)(void*, const float*))address_of(args[0]) : NULL;
  if (!f || !pointer_of(args[1], &h) || !floats_of(args[2], &b)) Py_RETURN_NONE;
  if (b.len != (Py_ssize_t)sizeof(float) * PyLong_AsSsize_t(args[3])) {
    PyErr_Clear();
    PyBuffer_Release(&b);
    Py_RETURN_NONE;
  }
  int st;
  Py_BEGIN_ALLOW_THREADS;
  st = f(h, (const float*)b.buf);
  Py_END_ALLOW_THREADS;
  PyBuffer_Release(&b);
  return PyLong_FromLong(st);
}

/* rows(f, handle, array, width): int f(void*, const float*, uint32_t), an
 * array of whole rows of `width` floats. */
static PyObject* rows(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void* h;
  Py_buffer b;
  int (*f)(void*, const float*, uint32_t) =
      n == 4 ? (int (*)(void*, const float*, uint32_t))address_of(args[0]) : NULL;
  if (!f || !pointer_of(args[1], &h) || !floats_of(args[2], &b)) Py_RETURN_NONE;
  const Py_ssize_t bytes = (Py_ssize_t)sizeof(float) * PyLong_AsSsize_t(args[3]);
  if (bytes <= 0 || b.len % bytes != 0 || b.len / bytes > (Py_ssize_t)UINT32_MAX) {
    PyErr_Clear();
    PyBuffer_Release(&b);
    Py_RETURN_NONE;
  }
  int st;
  Py_BEGIN_ALLOW_THREADS;
  st = f(h, (const float*)b.buf, (uint32_t)(b.len / bytes));
  Py_END_ALLOW_THREADS;
  PyBuffer_Release(&b);
  return PyLong_FromLong(st);
}

static PyMethodDef methods[] = {{"frame", (PyCFunction)(void (*)(void))frame, METH_FASTCALL, "frame(f, handle, dt)"},
                                {"floats", (PyCFunction)(void (*)(void))floats, METH_FASTCALL,
                                 "floats(f, handle, array, count)"},
                                {"rows", (PyCFunction)(void (*)(void))rows, METH_FASTCALL,
                                 "rows(f, handle, array, width)"},
                                {NULL, NULL, 0, NULL}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hscalls", "Per-frame calls without ctypes.", -1, methods,
                                    NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__hscalls(void) {
  str_value = PyUnicode_InternFromString("value");
  return str_value ? PyModule_Create(&module) : NULL;
}
