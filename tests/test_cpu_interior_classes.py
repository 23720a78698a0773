"""Subdomains with the same interior system share one factor (SIGMA_SMOOTHER.cpp
factors every subdomain's): the classes are exactly the equal systems."""
import ctypes as C

import numpy as np
import pytest

from hierarchicaldd_b200 import domains
from shim_ffi import load_shim


def _matrix(shim, h, level, sub):
    shape = (C.c_int * 3)()
    assert shim.shim_matrix_shape(h, 1, level, sub, shape) == 0
    rows, cols, nnz = shape
    ptr, col, val = np.zeros(rows + 1, np.int32), np.zeros(nnz, np.int32), np.zeros(nnz)
    ip = C.POINTER(C.c_int)
    assert shim.shim_matrix_get(h, 1, level, sub, ptr.ctypes.data_as(ip), col.ctypes.data_as(ip),
                                val.ctypes.data_as(C.POINTER(C.c_double))) == 0
    return rows, cols, ptr.tobytes(), col.tobytes(), val.tobytes()


@pytest.mark.parametrize("n,sub,radius", [(32, 8, 6), ((33, 40, 24), 8, 5), (48, 16, 0), (16, 16, 0)])
def test_classes_are_the_equal_interior_systems(n, sub, radius):
    d = domains.small(n, sub, radius)
    shim = load_shim()
    err = C.create_string_buffer(512)
    flags = np.ascontiguousarray(d.flags, np.uint32)
    h = shim.shim_build((C.c_int * 3)(*d.size), (C.c_int * 3)(*d.sub_size), 3, 2,
                        flags.ctypes.data_as(C.POINTER(C.c_uint32)), err, 512)
    assert h, err.value
    try:
        ns = shim.shim_num_subdomains(h)
        for level in range(2):
            rep = (C.c_int * ns)()
            shim.shim_interior_classes(h, level, rep)
            m = [_matrix(shim, h, level, i) for i in range(ns)]
            for i in range(ns):
                assert rep[i] <= i and rep[rep[i]] == rep[i] and m[rep[i]] == m[i], (level, i)
                # A system equal to an earlier one is of its class, unless the
                # ordering positions differ (the same cells at another offset
                # have the same relative positions in these domains).
                assert rep[i] == next(j for j in range(i + 1) if m[j] == m[i]), (level, i)
    finally:
        shim.shim_free(h)
