/* The per-layer calls of AttnEngine without ctypes: reads pointers and strides from the tensors and calls the C ABI.
 *
 * A decode step is one call per layer, and while the GPU spends 6 to 10 us on a layer of a short context, ctypes' conversion of
 * 18 arguments, the tensors' accessors as Python calls and the stream object took 7 us of host time before the library
 * was entered.  Here the accessors are vectorcalls on interned names and the arguments plain C values.
 * Conversions are ctypes': integers wrap to their width, the GIL is released for the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <stdlib.h>

#include "../../include/pooled_attn.h"

typedef int (*fn_attn_layer)(pa_layer*, uint32_t, uint32_t, uint32_t, int, const void*, uint64_t, uint64_t, const void*, const void*, uint64_t, const void*,
                             uint64_t, uint64_t, const float*, void*, uint64_t, void*);
typedef int (*fn_attn_items)(pa_layer*, const pa_item*, uint32_t, const void*, uint64_t, uint64_t, const void*, const void*, uint64_t, const void*, uint64_t,
                             uint64_t, void*, uint64_t, int, void*);
typedef int (*fn_rope_append)(pa_layer*, uint32_t, uint32_t, uint32_t, const void*, uint64_t, uint64_t, const void*, const void*, uint64_t, const float*, float*,
                              void*);
typedef int (*fn_decode_gather)(pa_layer*, uint32_t, uint32_t, const uint32_t*, uint32_t, const void*, int, uint64_t, uint64_t, const void*, uint64_t,
                                uint64_t, void*, uint64_t, void*);
/* Every call names the entry point (its address in the library the engine loaded) as its first argument: the module keeps
 * nothing of its own. */
static PyObject *s_data_ptr, *s_stride, *s_size, *i_zero;

static int ptr_of(PyObject* t, void** p) {
  if (t == Py_None) { *p = NULL; return 0; }
  PyObject* r = PyObject_VectorcallMethod(s_data_ptr, &t, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, NULL);
  if (!r) return -1;
  *p = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(r);
  Py_DECREF(r);
  return PyErr_Occurred() ? -1 : 0;
}
static int stride0(PyObject* t, uint64_t* s) {
  PyObject* a[2] = {t, i_zero};
  PyObject* r = PyObject_VectorcallMethod(s_stride, a, 2 | PY_VECTORCALL_ARGUMENTS_OFFSET, NULL);
  if (!r) return -1;
  *s = (uint64_t)PyLong_AsUnsignedLongLongMask(r);
  Py_DECREF(r);
  return PyErr_Occurred() ? -1 : 0;
}
static int u64_of(PyObject* o, uint64_t* v) { *v = PyLong_AsUnsignedLongLongMask(o); return PyErr_Occurred() ? -1 : 0; }
static int u32_of(PyObject* o, uint32_t* v) { *v = (uint32_t)PyLong_AsUnsignedLongMask(o); return PyErr_Occurred() ? -1 : 0; }
static int rows_of(PyObject* t, uint32_t* n) {
  PyObject* a[2] = {t, i_zero};
  PyObject* r = PyObject_VectorcallMethod(s_size, a, 2 | PY_VECTORCALL_ARGUMENTS_OFFSET, NULL);
  if (!r) return -1;
  *n = (uint32_t)PyLong_AsUnsignedLongMask(r);
  Py_DECREF(r);
  return PyErr_Occurred() ? -1 : 0;
}
static int args_are(Py_ssize_t n, Py_ssize_t want, const char* who) {
  if (n == want) return 0;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", who, want, n);
  return -1;
}

/* attn_layer(entry, layer, seq, pos, mode, q, q_head_stride, k, v, gate, gate_head_stride, cs_table, out, stream) -> status */
static PyObject* attn_layer(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  uint64_t fn, layer, qcs, qhs, kcs, gcs = 0, ghs = 0, ocs, stream;
  uint32_t seq, pos, mode, cols;
  void *q, *k, *v, *g, *cs, *out;
  (void)self;
  if (args_are(n, 14, "attn_layer") || u64_of(a[0], &fn) || u64_of(a[1], &layer) || u32_of(a[2], &seq) || u32_of(a[3], &pos) || u32_of(a[4], &mode) || rows_of(a[5], &cols) ||
      ptr_of(a[5], &q) || stride0(a[5], &qcs) || u64_of(a[6], &qhs) || ptr_of(a[7], &k) || stride0(a[7], &kcs) || ptr_of(a[8], &v) || ptr_of(a[9], &g) ||
      (a[9] != Py_None && (stride0(a[9], &gcs) || u64_of(a[10], &ghs))) || ptr_of(a[11], &cs) || ptr_of(a[12], &out) || stride0(a[12], &ocs) ||
      u64_of(a[13], &stream))
    return NULL;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = ((fn_attn_layer)(uintptr_t)fn)((pa_layer*)(uintptr_t)layer, seq, pos, cols, (int)mode, q, qcs, qhs, k, v, kcs, g, gcs, ghs, (const float*)cs, out, ocs,
                    (void*)(uintptr_t)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

/* attn_items(entry, layer, [(seq, pos)], q, q_head_stride, k, v, gate, gate_head_stride, out, exchange, stream) -> status */
static PyObject* attn_items(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  uint64_t fn, layer, qcs, qhs, kcs, gcs = 0, ghs = 0, ocs, stream;
  uint32_t exch;
  void *q, *k, *v, *g, *out;
  (void)self;
  if (args_are(n, 12, "attn_items") || u64_of(a[0], &fn) || u64_of(a[1], &layer) || ptr_of(a[3], &q) || stride0(a[3], &qcs) || u64_of(a[4], &qhs) || ptr_of(a[5], &k) ||
      stride0(a[5], &kcs) || ptr_of(a[6], &v) || ptr_of(a[7], &g) || (a[7] != Py_None && (stride0(a[7], &gcs) || u64_of(a[8], &ghs))) || ptr_of(a[9], &out) ||
      stride0(a[9], &ocs) || u32_of(a[10], &exch) || u64_of(a[11], &stream))
    return NULL;
  PyObject* list = PySequence_Fast(a[2], "the items are a sequence of (seq, pos) pairs");
  if (!list) return NULL;
  const Py_ssize_t cnt = PySequence_Fast_GET_SIZE(list);
  pa_item* items = (pa_item*)calloc((size_t)(cnt ? cnt : 1), sizeof(pa_item));
  if (!items) { Py_DECREF(list); return PyErr_NoMemory(); }
  for (Py_ssize_t i = 0; i < cnt; ++i) {
    PyObject* pr = PySequence_Fast(PySequence_Fast_GET_ITEM(list, i), "an item is a (seq, pos) pair");
    int bad = !pr;
    if (pr && PySequence_Fast_GET_SIZE(pr) != 2) { PyErr_SetString(PyExc_ValueError, "an item is a (seq, pos) pair"); bad = 1; }
    bad = bad || u32_of(PySequence_Fast_GET_ITEM(pr, 0), &items[i].seq) || u32_of(PySequence_Fast_GET_ITEM(pr, 1), &items[i].pos);
    Py_XDECREF(pr);
    if (bad) { free(items); Py_DECREF(list); return NULL; }
    items[i].n_cols = 1;
  }
  Py_DECREF(list);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = ((fn_attn_items)(uintptr_t)fn)((pa_layer*)(uintptr_t)layer, items, (uint32_t)cnt, q, qcs, qhs, k, v, kcs, g, gcs, ghs, out, ocs, (int)exch, (void*)(uintptr_t)stream);
  Py_END_ALLOW_THREADS
  free(items);
  return PyLong_FromLong(rc);
}

/* rope_append(entry, layer, seq, pos, q, q_head_stride, k, v, cs_table, q_rot, stream) -> status */
static PyObject* rope_append(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  uint64_t fn, layer, qcs, qhs, kcs, stream;
  uint32_t seq, pos, cols;
  void *q, *k, *v, *cs, *qr;
  (void)self;
  if (args_are(n, 11, "rope_append") || u64_of(a[0], &fn) || u64_of(a[1], &layer) || u32_of(a[2], &seq) || u32_of(a[3], &pos) || rows_of(a[4], &cols) || ptr_of(a[4], &q) ||
      stride0(a[4], &qcs) || u64_of(a[5], &qhs) || ptr_of(a[6], &k) || stride0(a[6], &kcs) || ptr_of(a[7], &v) || ptr_of(a[8], &cs) || ptr_of(a[9], &qr) ||
      u64_of(a[10], &stream))
    return NULL;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = ((fn_rope_append)(uintptr_t)fn)((pa_layer*)(uintptr_t)layer, seq, pos, cols, q, qcs, qhs, k, v, kcs, (const float*)cs, (float*)qr, (void*)(uintptr_t)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

/* decode_gather(entry, layer, seq, lists, list_stride, q, q_dtype, q_head_stride, gate, gate_head_stride, out, stream) -> status */
static PyObject* decode_gather(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  uint64_t fn, layer, qcs, qhs, gcs = 0, ghs = 0, ocs, stream;
  uint32_t seq, list_stride, cols, qdt;
  void *lists, *q, *g, *out;
  (void)self;
  if (args_are(n, 12, "decode_gather") || u64_of(a[0], &fn) || u64_of(a[1], &layer) || u32_of(a[2], &seq) || ptr_of(a[3], &lists) || u32_of(a[4], &list_stride) ||
      rows_of(a[5], &cols) || ptr_of(a[5], &q) || u32_of(a[6], &qdt) || stride0(a[5], &qcs) || u64_of(a[7], &qhs) || ptr_of(a[8], &g) ||
      (a[8] != Py_None && (stride0(a[8], &gcs) || u64_of(a[9], &ghs))) || ptr_of(a[10], &out) || stride0(a[10], &ocs) || u64_of(a[11], &stream))
    return NULL;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = ((fn_decode_gather)(uintptr_t)fn)((pa_layer*)(uintptr_t)layer, seq, cols, (const uint32_t*)lists, list_stride, q, (int)qdt, qcs, qhs, g, gcs, ghs, out, ocs,
                       (void*)(uintptr_t)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {
    {"attn_layer", (PyCFunction)(void (*)(void))attn_layer, METH_FASTCALL, "pa_attn_layer on tensors"},
    {"attn_items", (PyCFunction)(void (*)(void))attn_items, METH_FASTCALL, "pa_attn_items on tensors"},
    {"rope_append", (PyCFunction)(void (*)(void))rope_append, METH_FASTCALL, "pa_rope_append on tensors"},
    {"decode_gather", (PyCFunction)(void (*)(void))decode_gather, METH_FASTCALL, "pa_decode_gather on tensors"},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pa_call", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__pa_call(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_stride = PyUnicode_InternFromString("stride");
  s_size = PyUnicode_InternFromString("size");
  i_zero = PyLong_FromLong(0);
  if (!s_data_ptr || !s_stride || !s_size || !i_zero) return NULL;
  return PyModule_Create(&module);
}
