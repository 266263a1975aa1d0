"""Python's lists into the int32 arrays that the kernels read, natively (``csrc/host.cpp``)."""

from __future__ import annotations

import ctypes

from .build import build_library

_fill = None


def host_ints(numbers: list, n: int, address: int) -> bool:
    """The list's ``n`` numbers as int32 at ``address``.  False where one of them is no int of 32 bits, or the list has
    another length: what is there is then not to be used, and the caller goes the way that takes other numbers or says what is wrong."""
    global _fill
    if _fill is None:
        fill = ctypes.PyDLL(build_library("host")).q25_host_ints
        fill.argtypes, fill.restype = [ctypes.py_object, ctypes.c_ssize_t, ctypes.c_void_p], ctypes.c_int
        _fill = fill
    return _fill(numbers, n, address) == 1
