// CPython entry points for rknn_query_batch with buffer-protocol inputs (numpy
// arrays of int32 query ids and k values), rknn_query, rknn_serve_submit and
// rknn_serve_wait.  The ctypes route costs microseconds a call in Python (a
// pointer object per array, conversion of up to nine arguments), a large share
// of the host time of a 1000-query call and most of a served request's; these
// parse the arguments in C and release the interpreter lock around the call.
// rknn.py uses them when they were built (the CPython headers are needed) and
// ctypes otherwise: both call the same C entry points.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "rknn_gpu.h"

// query_batch(index, q, k, mode, out_ids, cap, offsets) -> status
//   index, out_ids, offsets: addresses (int); q, k: C-contiguous int32
//   buffers of equal length; cap: the capacity of out_ids in ids.
static PyObject* query_batch(PyObject* self, PyObject* args)
{
    (void)self;
    unsigned long long h = 0, out = 0, off = 0;
    long long cap = 0;
    int mode = 0;
    Py_buffer qb, kb;
    if (!PyArg_ParseTuple(args, "Ky*y*iKLK", &h, &qb, &kb, &mode, &out, &cap, &off)) return NULL;
    rknn_status rc = RKNN_ERR_ARG;
    if (qb.len % 4 == 0 && kb.len == qb.len && qb.len / 4 <= INT32_MAX) {
        Py_BEGIN_ALLOW_THREADS
        rc = rknn_query_batch((rknn_index*)(uintptr_t)h, (const int32_t*)qb.buf, (const int32_t*)kb.buf,
                              (int32_t)(qb.len / 4), (int32_t)mode, (int32_t*)(uintptr_t)out, (int64_t)cap,
                              (int64_t*)(uintptr_t)off, NULL);
        Py_END_ALLOW_THREADS
    }
    PyBuffer_Release(&qb);
    PyBuffer_Release(&kb);
    return PyLong_FromLong((long)rc);
}

// (Integers wider than the C arguments keep their low bits, as in ctypes.)
//
// query(index, q, k, mode, out) -> (status, n)
//   index: address; out: a writable int32 buffer, n: the result's size.
static PyObject* query(PyObject* self, PyObject* args)
{
    (void)self;
    unsigned long long h = 0;
    unsigned long q = 0, k = 0, mode = 0;
    Py_buffer ob;
    if (!PyArg_ParseTuple(args, "Kkkkw*", &h, &q, &k, &mode, &ob)) return NULL;
    rknn_status rc;
    int64_t n = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = rknn_query((rknn_index*)(uintptr_t)h, (int32_t)q, (int32_t)k, (int32_t)mode, (int32_t*)ob.buf,
                    (int64_t)(ob.len / 4), &n, NULL);
    Py_END_ALLOW_THREADS
    PyBuffer_Release(&ob);
    return Py_BuildValue("iL", (int)rc, (long long)n);
}

// serve_submit(server, q, k, mode) -> (status, ticket)
static PyObject* serve_submit(PyObject* self, PyObject* args)
{
    (void)self;
    unsigned long long h = 0;
    unsigned long q = 0, k = 0, mode = 0;
    if (!PyArg_ParseTuple(args, "Kkkk", &h, &q, &k, &mode)) return NULL;
    rknn_status rc;
    uint64_t t = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = rknn_serve_submit((rknn_server*)(uintptr_t)h, (int32_t)q, (int32_t)k, (int32_t)mode, &t);
    Py_END_ALLOW_THREADS
    return Py_BuildValue("iK", (int)rc, (unsigned long long)t);
}

// serve_wait(server, ticket, timeout_ms, out) -> (status, n, latency_ms)
static PyObject* serve_wait(PyObject* self, PyObject* args)
{
    (void)self;
    unsigned long long h = 0, t = 0;
    unsigned long timeout = 0;
    Py_buffer ob;
    if (!PyArg_ParseTuple(args, "KKkw*", &h, &t, &timeout, &ob)) return NULL;
    rknn_status rc;
    int64_t n = 0;
    double lat = 0.0;
    Py_BEGIN_ALLOW_THREADS
    rc = rknn_serve_wait((rknn_server*)(uintptr_t)h, (uint64_t)t, (int32_t)timeout, (int32_t*)ob.buf,
                         (int64_t)(ob.len / 4), &n, &lat);
    Py_END_ALLOW_THREADS
    PyBuffer_Release(&ob);
    return Py_BuildValue("iLd", (int)rc, (long long)n, lat);
}

static PyMethodDef methods[] = {
    {"query_batch", query_batch, METH_VARARGS, "rknn_query_batch on int32 buffers; returns the status"},
    {"query", query, METH_VARARGS, "rknn_query into an int32 buffer; returns (status, n)"},
    {"serve_submit", serve_submit, METH_VARARGS, "rknn_serve_submit; returns (status, ticket)"},
    {"serve_wait", serve_wait, METH_VARARGS, "rknn_serve_wait into an int32 buffer; returns (status, n, latency_ms)"},
    {NULL, NULL, 0, NULL},
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_rknn_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__rknn_call(void) { return PyModule_Create(&module); }
