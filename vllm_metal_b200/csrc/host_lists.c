/* Lists of Python integers -> rows of int32, for the metadata that a step stages in pinned memory.  A decode step of 64 requests at
 * 4096 tokens hands over 64 lists of 257 page numbers; NumPy converts them at some 40 ns a number.  Called with the interpreter's
 * lock held (ctypes.PyDLL).  -1: something other than exact lists of integers that fit, or too long a row -- the caller's general
 * conversion then accepts or refuses it. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

static int fill(PyObject* list, int32_t* dst, Py_ssize_t room) {
  if (!PyList_CheckExact(list)) return -1;
  const Py_ssize_t n = PyList_GET_SIZE(list);
  if (n > room) return -1;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* v = PyList_GET_ITEM(list, i);
    if (!PyLong_CheckExact(v)) return -1;
    int over = 0;
    const long x = PyLong_AsLongAndOverflow(v, &over);
    if (over || x < INT32_MIN || x > INT32_MAX) return -1;
    dst[i] = (int32_t)x;
  }
  return 0;
}

int b200_host_fill_row(PyObject* list, int32_t* dst, int64_t room) { return fill(list, dst, (Py_ssize_t)room); }

int b200_host_fill_rows(PyObject* lists, int32_t* dst, int64_t stride, int64_t rows) {
  if (!PyList_CheckExact(lists) || PyList_GET_SIZE(lists) > rows) return -1;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(lists); ++i)
    if (fill(PyList_GET_ITEM(lists, i), dst + i * stride, (Py_ssize_t)stride) != 0) return -1;
  return 0;
}
