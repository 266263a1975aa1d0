// What a step's host side does with Python's lists: their numbers go into the int32 arrays that the kernels read.  numpy and array
// take 25 to 35 ns a number (4,131 earlier tokens of sixteen chat requests: 147 us of a 227 us draw), this loop 4.
//
// Called through ctypes.PyDLL, so with the interpreter's lock held; the functions of its C interface that are needed are
// declared here, so that the library builds without Python's headers and works with the interpreter that loads it.
#include <limits.h>
#include <stddef.h>

struct _object;
extern "C" {
struct _object* PyList_GetItem(struct _object*, ptrdiff_t);
ptrdiff_t PyList_Size(struct _object*);
long PyLong_AsLongAndOverflow(struct _object*, int*);
struct _object* PyErr_Occurred(void);
void PyErr_Clear(void);
}

// The numbers of a list into dst[0 .. n).  1, or 0 where the list has not n items (any more) or one of them is no int (nor has an index) of
// 32 bits: the caller then goes the slow way, which says what is wrong or takes it.
extern "C" __attribute__((visibility("default"))) int q25_host_ints(struct _object* list, ptrdiff_t n, int* dst) {
  if (PyList_Size(list) != n) {
    PyErr_Clear();
    return 0;
  }
  for (ptrdiff_t i = 0; i < n; ++i) {
    struct _object* item = PyList_GetItem(list, i);        // looks at the length again: an item's __index__ may shorten the list
    int over = 0;
    const long v = item ? PyLong_AsLongAndOverflow(item, &over) : -1;
    if (over || v > INT_MAX || v < INT_MIN || (v == -1 && PyErr_Occurred())) {
      PyErr_Clear();
      return 0;
    }
    dst[i] = (int)v;
  }
  return 1;
}
