// Addresses and lengths of a list of bytes objects for the Python binding, in one pass: 6,000 objects take some 0.05 ms, three
// passes of the interpreter over them (types, addresses, lengths) took 0.48.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>

// addresses(list, address of n uint64 for the texts' addresses, address of n uint64 for their lengths)
//   -> how many objects at the beginning of the list are bytes objects; the rows of those are filled
static PyObject* addresses(PyObject* self, PyObject* args) {
    PyObject* list;
    unsigned long long ptrs, lens;
    if (!PyArg_ParseTuple(args, "O!KK", &PyList_Type, &list, &ptrs, &lens)) return NULL;
    uint64_t *p = (uint64_t*)(uintptr_t)ptrs, *l = (uint64_t*)(uintptr_t)lens;
    const Py_ssize_t n = PyList_GET_SIZE(list);
    Py_ssize_t i = 0;
    for (; i < n; i++) {
        PyObject* x = PyList_GET_ITEM(list, i);
        if (!PyBytes_CheckExact(x)) break;
        p[i] = (uint64_t)(uintptr_t)PyBytes_AS_STRING(x);
        l[i] = (uint64_t)PyBytes_GET_SIZE(x);
    }
    return PyLong_FromSsize_t(i);
}
static PyMethodDef methods[] = {{"addresses", addresses, METH_VARARGS, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_texts", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__texts(void) { return PyModule_Create(&module); }
