// CPython entry to ribn_gemv, the one call a host program makes once per projection.
//
// A projection of a few megabytes takes the GPU less time than the ctypes route to it took the host: converting ten
// arguments and asking both tensors for their type and length cost 2.3 us of the 5.4 us between two eager calls of one
// row, 1024 x 4096.  Here the tensors' attributes are read through the C API and the function is called by its address.
//
//   gemv(address of ribn_gemv, context, value type, weight descriptor, input, output, members) -> status
//   set_dtypes(torch.float32, torch.bfloat16): the type objects that inputs and outputs may have
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "../../include/ribn_b200.h"

typedef int (*gemv_function)(ribn_ctx*, uint32_t, const ribn_qweight*, const void*, int, uint64_t, void*, int, uint64_t, uint32_t);

static PyObject *name_data_ptr, *name_numel, *name_dtype;
static PyObject *type_f32, *type_bf16;

typedef struct {
    void* data;
    int dtype;
    uint64_t length;
} tensor_view;

static int call_for_number(PyObject* object, PyObject* method, unsigned long long* out) {
    PyObject* value = PyObject_CallMethodNoArgs(object, method);
    if (value == NULL) return -1;
    *out = PyLong_AsUnsignedLongLong(value);
    Py_DECREF(value);
    return PyErr_Occurred() ? -1 : 0;
}

static int view(PyObject* tensor, tensor_view* out) {
    PyObject* dtype = PyObject_GetAttr(tensor, name_dtype);
    if (dtype == NULL) return -1;
    const int known = dtype == type_f32 || dtype == type_bf16;
    out->dtype = dtype == type_bf16 ? RIBN_BF16 : RIBN_F32;
    if (!known) PyErr_Format(PyExc_TypeError, "activations must be float32 or bfloat16, got %S", dtype);
    Py_DECREF(dtype);
    if (!known) return -1;
    unsigned long long pointer = 0, length = 0;
    if (call_for_number(tensor, name_data_ptr, &pointer) != 0 || call_for_number(tensor, name_numel, &length) != 0) return -1;
    out->data = (void*)(uintptr_t)pointer;
    out->length = length;
    return 0;
}

static PyObject* gemv(PyObject* self, PyObject* const* args, Py_ssize_t count) {
    (void)self;
    if (count != 7) {
        PyErr_SetString(PyExc_TypeError, "gemv takes 7 arguments");
        return NULL;
    }
    const gemv_function function = (gemv_function)PyLong_AsVoidPtr(args[0]);
    ribn_ctx* context = (ribn_ctx*)PyLong_AsVoidPtr(args[1]);
    const unsigned long type = PyLong_AsUnsignedLong(args[2]);
    const ribn_qweight* weight = (const ribn_qweight*)PyLong_AsVoidPtr(args[3]);
    const unsigned long members = PyLong_AsUnsignedLongMask(args[6]);
    if (PyErr_Occurred()) return NULL;
    tensor_view x, y;
    if (view(args[4], &x) != 0 || view(args[5], &y) != 0) return NULL;
    int status;
    Py_BEGIN_ALLOW_THREADS   // a launch waits when the stream's queue is full
    status = function(context, (uint32_t)type, weight, x.data, x.dtype, x.length, y.data, y.dtype, y.length, (uint32_t)members);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

static PyObject* set_dtypes(PyObject* self, PyObject* const* args, Py_ssize_t count) {
    (void)self;
    if (count != 2) {
        PyErr_SetString(PyExc_TypeError, "set_dtypes takes 2 arguments");
        return NULL;
    }
    Py_XSETREF(type_f32, Py_NewRef(args[0]));
    Py_XSETREF(type_bf16, Py_NewRef(args[1]));
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"gemv", (PyCFunction)(void (*)(void))gemv, METH_FASTCALL, NULL},
    {"set_dtypes", (PyCFunction)(void (*)(void))set_dtypes, METH_FASTCALL, NULL},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__call(void) {
    name_data_ptr = PyUnicode_InternFromString("data_ptr");
    name_numel = PyUnicode_InternFromString("numel");
    name_dtype = PyUnicode_InternFromString("dtype");
    if (name_data_ptr == NULL || name_numel == NULL || name_dtype == NULL) return NULL;
    return PyModule_Create(&module);
}
