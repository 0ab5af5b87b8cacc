// Python integers as int32, for any Python 3.
#pragma once
#include <Python.h>

#include <cstdint>

// An int that CPython holds in one digit.  Most symbols are such ints, and their value is read
// without a call (16 000 symbols of a batch: 18 us, 45 through PyLong_AsLong).
inline bool CompactValue(PyObject *x, long *value) {
#if PY_VERSION_HEX >= 0x030C0000
  if (PyLong_CheckExact(x) && PyUnstable_Long_IsCompact(reinterpret_cast<PyLongObject *>(x))) {
    *value = (long)PyUnstable_Long_CompactValue(reinterpret_cast<PyLongObject *>(x));
    return true;
  }
#endif
  return false;
}

// The n items of a list or tuple; false when one is not an integer of 32 bits.
inline bool Int32sOf(PyObject *items, Py_ssize_t n, int32_t *out) {
  PyObject **at = PySequence_Fast_ITEMS(items);
  for (Py_ssize_t k = 0; k < n; ++k) {
    long v;
    if (!CompactValue(at[k], &v)) {
      PyObject *index = PyLong_Check(at[k]) ? nullptr : PyNumber_Index(at[k]);
      if (index == nullptr && !PyLong_Check(at[k])) {
        PyErr_Clear();
        return false;
      }
      v = PyLong_AsLong(index == nullptr ? at[k] : index);
      Py_XDECREF(index);
      if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
      }
    }
    if (v != (int32_t)v) return false;
    out[k] = (int32_t)v;
  }
  return true;
}
