/* The host side of the smallest calls, in C: row-wise / point-wise operators and streaming decode attention.
 *
 * On a small tensor these calls are bound by the host. Of 8.3 us for an RMSNorm of 4 x 512 the launch took 2.6, the allocation of the
 * result 1.3, converting fifteen ctypes arguments 1.4, and Python code the rest. Here the ordinary case (plain tensors, contiguous, on the
 * GPU) is checked and launched in one call. Whatever is not ordinary, errors among it, is answered with None, and the caller goes
 * on with the general path in Python, which stays the only place that raises. Nothing is kept from one call to the next but the
 * functions handed to setup().
 *
 * CPython API only: no torch headers, and no link to the library either (setup() gets the entry points' addresses).
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

typedef int (*elementwise_fn)(int, const void*, const void*, const void*, void*, int, int, int, int, int, float, float, int, int, void*);
typedef int (*attention_fn)(const void*, const void*, const void*, void*, void*, int, int, int, int, int, long long, long long, float, void*);
typedef unsigned long long (*scratch_fn)(int);

static PyTypeObject *g_tensor, *g_param;
static PyObject *g_codes, *g_empty_like, *g_empty, *g_device, *g_stream, *g_f32, *g_m1;
static elementwise_fn g_elementwise;
static attention_fn g_attention;
static scratch_fn g_scratch;
static PyObject *s_is_cuda, *s_dtype, *s_is_contiguous, *s_numel, *s_size, *s_data_ptr, *s_shape, *s_stride, *s_device, *s_kw;

static int plain(PyObject* t) { return Py_TYPE(t) == g_tensor || Py_TYPE(t) == g_param; }

/* 1 / 0, or -1 with an exception set */
static int truth_of(PyObject* o) {
  if (!o) return -1;
  const int r = PyObject_IsTrue(o);
  Py_DECREF(o);
  return r;
}
static int contiguous(PyObject* t) { return truth_of(PyObject_CallMethodNoArgs(t, s_is_contiguous)); }
static int on_gpu(PyObject* t) { return truth_of(PyObject_GetAttr(t, s_is_cuda)); }
static long long int_of(PyObject* o, int* bad) {
  if (!o) { *bad = 1; return 0; }
  const long long v = PyLong_AsLongLong(o);
  Py_DECREF(o);
  if (v == -1 && PyErr_Occurred()) *bad = 1;
  return v;
}
static void* pointer(PyObject* t, int* bad) {
  PyObject* o = PyObject_CallMethodNoArgs(t, s_data_ptr);
  if (!o) { *bad = 1; return NULL; }
  void* p = PyLong_AsVoidPtr(o);
  Py_DECREF(o);
  if (!p && PyErr_Occurred()) *bad = 1;
  return p;
}
static int dtype_code(PyObject* t, int* bad) {           /* -1: not one of the library's */
  PyObject* d = PyObject_GetAttr(t, s_dtype);
  if (!d) { *bad = 1; return -1; }
  PyObject* c = PyDict_GetItemWithError(g_codes, d);     /* borrowed */
  Py_DECREF(d);
  if (!c) { if (PyErr_Occurred()) *bad = 1; return -1; }
  return (int)PyLong_AsLong(c);
}
/* 1, or 0 for what float() may still take (a text) or refuse: the general path's to say */
static int number(PyObject* o, double* v) {
  *v = PyFloat_AsDouble(o);
  if (*v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  return 1;
}
static void* current_stream(int* bad) {
  PyObject* d = PyObject_CallNoArgs(g_device);
  if (!d) { *bad = 1; return NULL; }
  PyObject* s = PyObject_CallOneArg(g_stream, d);
  Py_DECREF(d);
  if (!s) { *bad = 1; return NULL; }
  void* p = PyLong_AsVoidPtr(s);
  Py_DECREF(s);
  if (!p && PyErr_Occurred()) *bad = 1;
  return p;
}

/* elementwise(kind, x, in1 | None, in2 | None, out | None, f0, f1) -> result, an int (the library's error code), or None */
static PyObject* py_elementwise(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  (void)self;
  if (n != 7) { PyErr_SetString(PyExc_TypeError, "elementwise: seven arguments"); return NULL; }
  PyObject* x = a[1];
  for (int i = 1; i < 5; ++i)
    if ((i == 1 || a[i] != Py_None) && !plain(a[i])) Py_RETURN_NONE;
  int bad = 0, ok = on_gpu(x);
  for (int i = 1; i < 5 && ok == 1; ++i)
    if (a[i] != Py_None) ok = contiguous(a[i]);
  if (ok < 0) return NULL;
  if (!ok) Py_RETURN_NONE;
  const int dt = dtype_code(x, &bad);
  if (bad) return NULL;
  const long long numel = dt < 0 ? 0 : int_of(PyObject_CallMethodNoArgs(x, s_numel), &bad);
  if (bad) return NULL;
  if (numel <= 0) Py_RETURN_NONE;
  PyObject* size = PyObject_CallMethodOneArg(x, s_size, g_m1);
  if (!size) { PyErr_Clear(); Py_RETURN_NONE; }         /* (no dimensions) */
  const long long cols = int_of(size, &bad);
  const long kind = PyLong_AsLong(a[0]);
  if (bad || PyErr_Occurred()) return NULL;
  double f0, f1;
  if (!number(a[5], &f0) || !number(a[6], &f1)) Py_RETURN_NONE;
  PyObject* out = a[4];
  if (out == Py_None) {
    out = PyObject_CallOneArg(g_empty_like, x);
    if (!out) return NULL;
  } else {
    Py_INCREF(out);
  }
  const void* px = pointer(x, &bad);
  const void* p1 = !bad && a[2] != Py_None ? pointer(a[2], &bad) : NULL;
  const void* p2 = !bad && a[3] != Py_None ? pointer(a[3], &bad) : NULL;
  void* po = !bad ? pointer(out, &bad) : NULL;
  void* st = !bad ? current_stream(&bad) : NULL;
  if (bad) { Py_DECREF(out); return NULL; }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_elementwise((int)kind, px, p1, p2, po, (int)(numel / cols), (int)cols, dt, (int)cols, (int)cols, (float)f0, (float)f1, 0, 0, st);
  Py_END_ALLOW_THREADS
  if (rc == 0) return out;
  Py_DECREF(out);
  return PyLong_FromLong(rc);
}

/* A tuple attribute or method result of n integers: 1, 0 (another length) or -1. */
static int ints_of(PyObject* t, long long* v, Py_ssize_t n) {
  if (!t) return -1;
  int r = PyTuple_Check(t) && PyTuple_GET_SIZE(t) == n;
  for (Py_ssize_t i = 0; r == 1 && i < n; ++i) {
    v[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(t, i));
    if (v[i] == -1 && PyErr_Occurred()) r = -1;
  }
  Py_DECREF(t);
  return r;
}
/* (batch, head) strides of a cache whose rows are contiguous; a dimension of size 1 counts as contiguous. */
static int kv_strides(const long long* sh, const long long* st, long long* batch, long long* head) {
  if ((sh[3] > 1 && st[3] != 1) || (sh[2] > 1 && st[2] != sh[3])) return 0;
  *head = sh[1] > 1 ? st[1] : sh[2] * sh[3];
  *batch = sh[0] > 1 ? st[0] : sh[1] * *head;
  return 1;
}

/* attention(q, k, v, out | None, scale) -> result, an int, or None */
static PyObject* py_attention(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  (void)self;
  if (n != 5) { PyErr_SetString(PyExc_TypeError, "attention: five arguments"); return NULL; }
  PyObject *q = a[0], *k = a[1], *v = a[2];
  if (!plain(q) || !plain(k) || !plain(v) || (a[3] != Py_None && !plain(a[3]))) Py_RETURN_NONE;
  long long sq[3], sk[4], sv[4], tk[4], tv[4], kb, kh, vb, vh;
  int bad = 0, ok = on_gpu(q);
  if (ok == 1) ok = contiguous(q);
  if (ok == 1 && a[3] != Py_None) ok = contiguous(a[3]);
  if (ok == 1) ok = ints_of(PyObject_GetAttr(q, s_shape), sq, 3);
  if (ok == 1) ok = ints_of(PyObject_GetAttr(k, s_shape), sk, 4);
  if (ok == 1) ok = ints_of(PyObject_GetAttr(v, s_shape), sv, 4);
  if (ok == 1) ok = ints_of(PyObject_CallMethodNoArgs(k, s_stride), tk, 4);
  if (ok == 1) ok = ints_of(PyObject_CallMethodNoArgs(v, s_stride), tv, 4);
  if (ok < 0) return NULL;
  if (!ok) Py_RETURN_NONE;
  for (int i = 0; i < 4; ++i) if (sk[i] != sv[i]) Py_RETURN_NONE;
  if (sq[2] != 128 || sk[3] != 128 || sk[0] < sq[0] || sq[0] < 1 || sk[1] < 1 || sk[2] < 1 || sq[1] < 1 || sq[1] % sk[1] != 0 || sq[1] / sk[1] > 8)
    Py_RETURN_NONE;
  if (!kv_strides(sk, tk, &kb, &kh) || !kv_strides(sv, tv, &vb, &vh) || kb != vb || kh != vh) Py_RETURN_NONE;
  const int dt = dtype_code(q, &bad);
  if (bad) return NULL;
  double scale;
  if (dt < 0 || !number(a[4], &scale)) Py_RETURN_NONE;
  PyObject* dev = PyObject_GetAttr(q, s_device);
  if (!dev) return NULL;
  PyObject* words = PyLong_FromUnsignedLongLong(g_scratch((int)(sq[1] / sk[1])) / 4);
  PyObject* call[3] = {words, g_f32, dev};
  PyObject* scratch = words ? PyObject_Vectorcall(g_empty, call, 1, s_kw) : NULL;
  Py_XDECREF(words);
  Py_DECREF(dev);
  if (!scratch) return NULL;
  PyObject* out = a[3];
  if (out == Py_None) {
    out = PyObject_CallOneArg(g_empty_like, q);
    if (!out) { Py_DECREF(scratch); return NULL; }
  } else {
    Py_INCREF(out);
  }
  const void *pq = pointer(q, &bad), *pk = !bad ? pointer(k, &bad) : NULL, *pv = !bad ? pointer(v, &bad) : NULL;
  void *po = !bad ? pointer(out, &bad) : NULL, *ps = !bad ? pointer(scratch, &bad) : NULL, *st = !bad ? current_stream(&bad) : NULL;
  int rc = 0;
  if (!bad) {
    Py_BEGIN_ALLOW_THREADS
    rc = g_attention(pq, pk, pv, po, ps, (int)sq[0], (int)sq[1], (int)sk[1], (int)sk[2], dt, kb, kh, (float)scale, st);
    Py_END_ALLOW_THREADS
  }
  Py_DECREF(scratch);                                    /* (freed in stream order by torch's allocator) */
  if (!bad && rc == 0) return out;
  Py_DECREF(out);
  if (bad) return NULL;
  if (rc == -2) Py_RETURN_NONE;
  return PyLong_FromLong(rc);
}

/* setup(Tensor, Parameter, dtype codes, empty_like, empty, current device, raw stream, float32, three addresses) */
static PyObject* py_setup(PyObject* self, PyObject* args) {
  (void)self;
  PyObject *t, *p, *codes, *el, *em, *dev, *st, *f32;
  unsigned long long fe, fa, fs;
  if (!PyArg_ParseTuple(args, "OOOOOOOOKKK", &t, &p, &codes, &el, &em, &dev, &st, &f32, &fe, &fa, &fs)) return NULL;
  if (!PyType_Check(t) || !PyType_Check(p) || !PyDict_Check(codes)) { PyErr_SetString(PyExc_TypeError, "setup: types and a dict"); return NULL; }
  Py_INCREF(t); Py_INCREF(p); Py_INCREF(codes); Py_INCREF(el); Py_INCREF(em); Py_INCREF(dev); Py_INCREF(st); Py_INCREF(f32);
  g_tensor = (PyTypeObject*)t; g_param = (PyTypeObject*)p; g_codes = codes; g_empty_like = el; g_empty = em; g_device = dev; g_stream = st; g_f32 = f32;
  g_elementwise = (elementwise_fn)(uintptr_t)fe; g_attention = (attention_fn)(uintptr_t)fa; g_scratch = (scratch_fn)(uintptr_t)fs;
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"setup", py_setup, METH_VARARGS, "Hands over the types, functions and entry points that the calls use."},
    {"elementwise", (PyCFunction)(void (*)(void))py_elementwise, METH_FASTCALL, "A row-wise or point-wise operator; None: not an ordinary call."},
    {"attention", (PyCFunction)(void (*)(void))py_attention, METH_FASTCALL, "Streaming decode attention; None: not an ordinary call."},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "maco_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_maco_fastcall(void) {
  s_is_cuda = PyUnicode_InternFromString("is_cuda"); s_dtype = PyUnicode_InternFromString("dtype");
  s_is_contiguous = PyUnicode_InternFromString("is_contiguous"); s_numel = PyUnicode_InternFromString("numel");
  s_size = PyUnicode_InternFromString("size"); s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_shape = PyUnicode_InternFromString("shape"); s_stride = PyUnicode_InternFromString("stride");
  s_device = PyUnicode_InternFromString("device"); g_m1 = PyLong_FromLong(-1);
  s_kw = Py_BuildValue("(ss)", "dtype", "device");
  return PyModule_Create(&module);
}
