// What a sampled step reads out of Python's lists, in native code: the penalties' windows (64 rows of 64 token ids take 19 us
// instead of 76 through array.fromlist) and the seeds and step numbers of its random draws.  Called with the
// interpreter's lock held (ctypes.PyDLL); nothing here runs Python code or keeps an object, and whatever is not an exact
// list of exact integers that fit is left to the caller's own way.
#include <Python.h>

#include <cstdint>
#include <cstring>

#define IBH_EXPORT extern "C" __attribute__((visibility("default")))

// Row r of out [rows, width] receives -1 if pending[r], then the last window[r] - pending[r] entries of list r (fewer if it
// is shorter), then -1 up to the width; counts[r] is how many places were filled.  A row with window[r] == 0 stays blank.
// 0: done; -1: something is not what this function takes (out is then undefined).
IBH_EXPORT int ibh_windows(PyObject* lists, const int* window, const int* pending, int rows, int width, int* out, int* counts) {
    if (!PyList_CheckExact(lists) || PyList_GET_SIZE(lists) < rows) return -1;
    for (int r = 0; r < rows; ++r) {
        int* dst = out + (size_t)r * width;
        int n = 0;
        if (window[r] > 0) {
            PyObject* list = PyList_GET_ITEM(lists, r);
            if (!PyList_CheckExact(list)) return -1;
            if (pending[r]) {
                if (width < 1) return -1;
                dst[n++] = -1;
            }
            const Py_ssize_t size = PyList_GET_SIZE(list), known = window[r] - pending[r];
            Py_ssize_t take = known < size ? known : size;
            if (take < 0) take = 0;
            if (n + take > width) return -1;
            for (Py_ssize_t i = size - take; i < size; ++i) {
                PyObject* v = PyList_GET_ITEM(list, i);
                if (!PyLong_CheckExact(v)) return -1;
                int over = 0;
                const long x = PyLong_AsLongAndOverflow(v, &over);
                if (over || x < INT32_MIN || x > INT32_MAX) return -1;
                dst[n++] = (int)x;
            }
        }
        counts[r] = n;
        for (int i = n; i < width; ++i) dst[i] = -1;
    }
    return 0;
}

// The low 64 bits of every entry of a list (as Python's & 2^64 - 1).  0: done; -1: not a list of exact integers.
IBH_EXPORT int ibh_low_words(PyObject* list, int n, uint64_t* out) {
    if (!PyList_CheckExact(list) || PyList_GET_SIZE(list) != n) return -1;
    for (int i = 0; i < n; ++i) {
        PyObject* v = PyList_GET_ITEM(list, i);
        if (!PyLong_CheckExact(v)) return -1;
        out[i] = (uint64_t)PyLong_AsUnsignedLongLongMask(v);
    }
    if (PyErr_Occurred()) { PyErr_Clear(); return -1; }
    return 0;
}
