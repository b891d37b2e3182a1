"""Lists of Python integers into int32 rows, by ``csrc/host_lists.c`` where that was built and applies."""

from __future__ import annotations

import ctypes
from functools import cache

import numpy as np


@cache
def _lib():
    from .metal.build import host_library_path

    try:
        lib = ctypes.PyDLL(str(host_library_path()))
    except OSError:
        return None
    lib.b200_host_fill_row.argtypes = [ctypes.py_object, ctypes.c_void_p, ctypes.c_int64]
    lib.b200_host_fill_rows.argtypes = [ctypes.py_object, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64]
    return lib


def _rows_of_int32(dst: np.ndarray) -> bool:
    return dst.dtype == np.int32 and dst.strides[-1] == 4 and dst.flags.writeable


def fill_rows(dst: np.ndarray, rows) -> None:
    """``dst[i, : len(rows[i])] = rows[i]`` for int32 ``dst [R, C]``."""
    lib = _lib()
    if (lib is not None and type(rows) is list and _rows_of_int32(dst) and dst.strides[0] == 4 * dst.shape[1]
            and lib.b200_host_fill_rows(rows, dst.ctypes.data, dst.shape[1], dst.shape[0]) == 0):
        return
    for i, row in enumerate(rows):
        dst[i, : len(row)] = row


def native_int32(values) -> np.ndarray | None:
    """A list of Python integers that fit as int32; ``None`` for anything else, which the caller's general conversion then takes
    or refuses."""
    lib = _lib()
    if lib is not None and type(values) is list and values:
        out = np.empty(len(values), dtype=np.int32)
        if lib.b200_host_fill_row(values, out.ctypes.data, len(values)) == 0:
            return out
    return None
