/* Host helpers that need the interpreter's own view of an object (libwf_py.<ABI>.so, called through ctypes.PyDLL with the GIL held). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#ifdef Py_GIL_DISABLED
#error "another thread may change the list meanwhile: left out, numpy does it"
#endif
#include <stdint.h>

/* The n entries of a list as 32-bit integers; 0, and out in part written, when the object is not a list of n plain ints that fit.  A prompt of 2048 token ids: 9 us,
 * 54 as numpy.array(list). */
int wf_py_i32(PyObject* list, int32_t* out, Py_ssize_t n) {
    if (!PyList_CheckExact(list) || PyList_GET_SIZE(list) != n) return 0;
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* v = PyList_GET_ITEM(list, i);
        if (!PyLong_CheckExact(v)) return 0;
        int over = 0;
        const long x = PyLong_AsLongAndOverflow(v, &over);
        if (over || x < INT32_MIN || x > INT32_MAX) return 0;
        out[i] = (int32_t)x;
    }
    return 1;
}
