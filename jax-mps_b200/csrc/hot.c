/* The calls a Python program makes over and over (execute, host array in, host array out, a buffer's end), as a CPython
 * extension over the C ABI. Through ctypes a call with three arguments and two results cost 4 us of building argument
 * arrays and wrapping results and every buffer 0.6 us at its end; here both are well under half a microsecond. Everything
 * else of the Python face stays ctypes. The functions are handed over as addresses by b200/__init__.py, which owns the
 * library handle. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>
#include <stdint.h>
#include <string.h>

#include "../../include/b200_core.h"

static struct {
  b200_error* (*execute)(b200_executable*, b200_buffer* const*, size_t, b200_buffer**, b200_event**, const b200_execute_options*);
  b200_error* (*from_host)(b200_client*, const void*, b200_dtype, const int64_t*, size_t, const int64_t*, b200_buffer**, b200_event**);
  b200_error* (*to_host)(b200_buffer*, void*, size_t*, b200_event**);
  b200_error* (*destroy)(b200_buffer*);
  void (*error_destroy)(b200_error*);
  void* (*host_alloc)(size_t);
  void (*host_free)(void*);
} api;
static PyObject *raise_error, *buffer_class;

/* ---- a buffer's handle; b200.Buffer derives from it ---- */
typedef struct {
  PyObject_HEAD
  void* h;
  PyObject *client, *host;
} Handle;

/* Without the interpreter: the client's lock may be held by a thread that waits for the device. */
static void destroy(void* h) {
  Py_BEGIN_ALLOW_THREADS
  b200_error* e = api.destroy((b200_buffer*)h);
  if (e) api.error_destroy(e);
  Py_END_ALLOW_THREADS
}
static void drop(Handle* self) {
  void* h = self->h;
  self->h = NULL;
  if (h && api.destroy) destroy(h);
}
static int handle_traverse(PyObject* o, visitproc visit, void* arg) {
  Py_VISIT(((Handle*)o)->client);
  Py_VISIT(((Handle*)o)->host);
  return 0;
}
static int handle_clear(PyObject* o) {
  Py_CLEAR(((Handle*)o)->client);
  Py_CLEAR(((Handle*)o)->host);
  return 0;
}
static void handle_dealloc(PyObject* o) {
  PyTypeObject* t = Py_TYPE(o);
  PyObject_GC_UnTrack(o);
  drop((Handle*)o);
  handle_clear(o);
  t->tp_free(o);
}
static int handle_init(PyObject* o, PyObject* args, PyObject* kw) {
  Handle* self = (Handle*)o;
  PyObject *client, *h;
  if (!PyArg_ParseTuple(args, "OO", &client, &h)) return -1;
  if (h != Py_None) {
    self->h = PyLong_AsVoidPtr(h);
    if (!self->h && PyErr_Occurred()) return -1;
  }
  Py_INCREF(client);
  Py_XSETREF(self->client, client);
  return 0;
}
static PyObject* handle_get(PyObject* o, void* unused) {
  void* h = ((Handle*)o)->h;
  if (!h) Py_RETURN_NONE;
  return PyLong_FromVoidPtr(h);
}
static PyGetSetDef handle_getset[] = {{"_h", handle_get, NULL, NULL, NULL}, {NULL}};
static PyMemberDef handle_members[] = {{"client", T_OBJECT_EX, offsetof(Handle, client), 0, NULL},
                                       {"_host", T_OBJECT, offsetof(Handle, host), 0, NULL},
                                       {NULL}};
static PyTypeObject HandleType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "b200._hot.Handle",
    .tp_basicsize = sizeof(Handle),
    .tp_dealloc = handle_dealloc,
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC,
    .tp_traverse = handle_traverse,
    .tp_clear = handle_clear,
    .tp_members = handle_members,
    .tp_getset = handle_getset,
    .tp_init = handle_init,
    .tp_new = PyType_GenericNew,
};

static PyObject* wrap(void* h, PyObject* client) {
  PyTypeObject* t = (PyTypeObject*)buffer_class;
  Handle* b = (Handle*)t->tp_alloc(t, 0);
  if (!b) {
    destroy(h);
    return NULL;
  }
  b->h = h;
  Py_INCREF(client);
  b->client = client;
  return (PyObject*)b;
}

static PyObject* failed(b200_error* e) {
  PyObject* r = PyObject_CallFunction(raise_error, "n", (Py_ssize_t)(intptr_t)e);      /* raises and frees the error */
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "b200 error");
  return NULL;
}

/* execute(handle, args, num_outputs, donate, want_event, client) -> (buffers, event address or 0) */
static PyObject* hot_execute(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "execute takes 6 arguments");
  void* exe = PyLong_AsVoidPtr(a[0]);
  if (!exe) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_ValueError, "the executable has been destroyed");
  /* a tuple of our own: the caller's list may change in another thread while the call runs without the interpreter */
  PyObject* seq = PySequence_Tuple(a[1]);
  if (!seq) return NULL;
  const Py_ssize_t num_args = PyTuple_GET_SIZE(seq), num_out = PyLong_AsSsize_t(a[2]);
  void *small_in[64], *small_out[64];
  void** in = num_args <= 64 ? small_in : PyMem_Malloc(sizeof(void*) * (size_t)num_args);
  void** out = num_out <= 64 ? small_out : PyMem_Malloc(sizeof(void*) * (size_t)num_out);
  PyObject* result = NULL;
  if (!in || !out) { PyErr_NoMemory(); goto done; }
  for (Py_ssize_t k = 0; k < num_args; k++) {
    PyObject* o = PyTuple_GET_ITEM(seq, k);
    if (!PyObject_TypeCheck(o, &HandleType)) {
      PyErr_Format(PyExc_TypeError, "argument %zd is not a buffer", k);
      goto done;
    }
    in[k] = ((Handle*)o)->h;
  }
  memset(out, 0, sizeof(void*) * (size_t)num_out);
  b200_execute_options opts;
  memset(&opts, 0, sizeof opts);
  opts.struct_size = sizeof opts;
  opts.donate_arguments = PyObject_IsTrue(a[3]);
  const int want_event = PyObject_IsTrue(a[4]);
  b200_event* event = NULL;
  b200_error* err;
  Py_BEGIN_ALLOW_THREADS
  err = api.execute((b200_executable*)exe, (b200_buffer* const*)in, (size_t)num_args, (b200_buffer**)out, want_event ? &event : NULL, &opts);
  Py_END_ALLOW_THREADS
  if (err) { failed(err); goto done; }
  PyObject* bufs = PyList_New(num_out);
  if (!bufs) goto done;
  for (Py_ssize_t k = 0; k < num_out; k++) {
    PyObject* b = wrap(out[k], a[5]);
    if (!b) {
      for (Py_ssize_t q = k + 1; q < num_out; q++) destroy(out[q]);
      Py_DECREF(bufs);
      goto done;
    }
    PyList_SET_ITEM(bufs, k, b);
  }
  if (!want_event) result = bufs;
  else {
    result = Py_BuildValue("(Nn)", bufs, (Py_ssize_t)(intptr_t)event);
  }
done:
  if (in && in != small_in) PyMem_Free(in);
  if (out && out != small_out) PyMem_Free(out);
  Py_DECREF(seq);
  return result;
}

/* b200_dtype of a buffer-protocol format, 0 when it has none here */
static int dtype_of(const char* f, Py_ssize_t size) {
  if (!f) return B200_U8;
  if (*f == '@' || *f == '=') f++;
  if (!f[0] || f[1]) return 0;
  switch (*f) {
    case '?': return B200_PRED;
    case 'b': case 'h': case 'i': case 'l': case 'q': return size == 1 ? B200_S8 : size == 2 ? B200_S16 : size == 4 ? B200_S32 : size == 8 ? B200_S64 : 0;
    case 'B': case 'H': case 'I': case 'L': case 'Q': return size == 1 ? B200_U8 : size == 2 ? B200_U16 : size == 4 ? B200_U32 : size == 8 ? B200_U64 : 0;
    case 'e': return B200_F16;
    case 'f': return B200_F32;
    case 'd': return B200_F64;
    default: return 0;
  }
}

/* from_host(client handle, array, client) -> buffer, or None for an array this does not read (the caller converts it) */
static PyObject* hot_from_host(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 3) return PyErr_Format(PyExc_TypeError, "from_host takes 3 arguments");
  void* client = PyLong_AsVoidPtr(a[0]);
  if (!client) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_ValueError, "the client is closed");
  Py_buffer v;
  if (PyObject_GetBuffer(a[1], &v, PyBUF_STRIDED_RO | PyBUF_FORMAT) != 0) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int dt = dtype_of(v.format, v.itemsize);
  if (!dt || v.ndim > 32) {
    PyBuffer_Release(&v);
    Py_RETURN_NONE;
  }
  int64_t dims[33], strides[33];
  for (int k = 0; k < v.ndim; k++) { dims[k] = v.shape[k]; strides[k] = v.strides[k]; }
  b200_buffer* out = NULL;
  b200_error* err;
  Py_BEGIN_ALLOW_THREADS
  err = api.from_host((b200_client*)client, v.len ? v.buf : NULL, (b200_dtype)dt, dims, (size_t)v.ndim, strides, &out, NULL);
  Py_END_ALLOW_THREADS
  PyBuffer_Release(&v);
  if (err) return failed(err);
  PyObject* b = wrap(out, a[2]);
  if (b) { Py_INCREF(a[1]); ((Handle*)b)->host = a[1]; }        /* pinned memory is read asynchronously */
  return b;
}

/* ---- pinned memory that an array of results lives in ---- */
typedef struct {
  PyObject_HEAD
  void* ptr;
  Py_ssize_t size;
} Block;
static void block_dealloc(PyObject* o) {
  void* ptr = ((Block*)o)->ptr;
  if (ptr) {
    Py_BEGIN_ALLOW_THREADS                       /* giving page-locked memory back may wait for the device */
    api.host_free(ptr);
    Py_END_ALLOW_THREADS
  }
  Py_TYPE(o)->tp_free(o);
}
static int block_buffer(PyObject* o, Py_buffer* v, int flags) {
  return PyBuffer_FillInfo(v, o, ((Block*)o)->ptr, ((Block*)o)->size, 0, flags);
}
static PyBufferProcs block_as_buffer = {block_buffer, NULL};
static PyTypeObject BlockType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "b200._hot.Block",
    .tp_basicsize = sizeof(Block),
    .tp_dealloc = block_dealloc,
    .tp_as_buffer = &block_as_buffer,
    .tp_flags = Py_TPFLAGS_DEFAULT,
};

/* to_block(buffer, bytes) -> the buffer's contents in pinned memory, or None when there is none to be had */
static PyObject* hot_to_block(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyObject_TypeCheck(a[0], &HandleType)) return PyErr_Format(PyExc_TypeError, "to_block takes a buffer and its size");
  const Py_ssize_t bytes = PyLong_AsSsize_t(a[1]);
  if (bytes < 0) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_ValueError, "negative size");
  void* ptr;
  Py_BEGIN_ALLOW_THREADS
  ptr = api.host_alloc((size_t)bytes);
  Py_END_ALLOW_THREADS
  if (!ptr) Py_RETURN_NONE;
  Block* b = PyObject_New(Block, &BlockType);
  if (!b) { api.host_free(ptr); return NULL; }
  b->ptr = ptr;
  b->size = bytes;
  void* h = ((Handle*)a[0])->h;
  size_t size = (size_t)bytes;
  b200_error* err;
  Py_BEGIN_ALLOW_THREADS
  err = api.to_host((b200_buffer*)h, ptr, &size, NULL);
  Py_END_ALLOW_THREADS
  if (err) { Py_DECREF(b); return failed(err); }
  return (PyObject*)b;
}

/* bind(addresses in the order of `api`, function that raises an error by its address, buffer class) */
static PyObject* hot_bind(PyObject* self, PyObject* args) {
  PyObject *seq, *raise, *cls;
  if (!PyArg_ParseTuple(args, "OOO", &seq, &raise, &cls)) return NULL;
  void** to = (void**)&api;
  const Py_ssize_t count = (Py_ssize_t)(sizeof api / sizeof(void*));
  if (PySequence_Size(seq) != count) return PyErr_Format(PyExc_ValueError, "bind wants %zd addresses", count);
  for (Py_ssize_t k = 0; k < count; k++) {
    PyObject* o = PySequence_GetItem(seq, k);
    to[k] = o ? PyLong_AsVoidPtr(o) : NULL;
    Py_XDECREF(o);
    if (!to[k]) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_ValueError, "null address");
  }
  if (!PyType_Check(cls) || !PyType_IsSubtype((PyTypeObject*)cls, &HandleType)) return PyErr_Format(PyExc_TypeError, "the buffer class derives from Handle");
  Py_INCREF(raise);
  Py_XSETREF(raise_error, raise);
  Py_INCREF(cls);
  Py_XSETREF(buffer_class, cls);
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {{"execute", (PyCFunction)(void (*)(void))hot_execute, METH_FASTCALL, NULL},
                                {"from_host", (PyCFunction)(void (*)(void))hot_from_host, METH_FASTCALL, NULL},
                                {"to_block", (PyCFunction)(void (*)(void))hot_to_block, METH_FASTCALL, NULL},
                                {"bind", hot_bind, METH_VARARGS, NULL},
                                {NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hot", NULL, -1, methods};

PyMODINIT_FUNC PyInit__hot(void) {
  if (PyType_Ready(&HandleType) < 0 || PyType_Ready(&BlockType) < 0) return NULL;
  PyObject* m = PyModule_Create(&module);
  if (!m) return NULL;
  Py_INCREF(&HandleType);
  PyModule_AddObject(m, "Handle", (PyObject*)&HandleType);
  return m;
}
