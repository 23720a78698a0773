"""The schedules of the one-CTA-per-tree solves (sn_streams.cpp), walked on the
CPU operation by operation as sn_resident.cu runs them: against the host walk of
the same fronts, from a CTA's array that holds NaN everywhere (a system that
broke down may have left it so: nothing a solve has not written itself may reach
its result), with every index in range and no entry written by one warp that
another warp reads or writes before the next barrier.

Tolerance as for the kernels: FP64 sums in another order, rounded to FP32 once,
one ulp (1.2e-7) of the largest entry.
"""
import ctypes as C

import numpy as np
import pytest

from shim_ffi import load_shim
from sn_routes import ROUTES, domain

RTOL = 1.2e-7

# Bytes of a domain's streams over those of the distinct coefficients they hold
# (once per direction): the padding of small fronts, headers and indices.
PADDING = {"one tree": 4.6, "pairs": 4.1, "quads": 3.7, "fronts in pairs": 3.7, "slots in memory": 3.2,
           "cut factors": 3.4, "equal cut factors": 3.9, "ragged": 4.5, "forest": 15.2}


def _fp(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


# Interface solves of each domain that take the route it is named for: (kind, level)
# and {field of the walk's info: value}; whole 0, trees per CTA 1, threads 2,
# slots in global memory 3, CTAs 4, fronts above the cut 5.
TAKES = {"one tree": {(0, 0): {0: 1, 4: 1}},
         "pairs": {(1, 0): {0: 1, 1: 2, 2: 128}, (0, 0): {0: 0, 2: 512}},
         "quads": {(1, 0): {0: 1, 1: 4, 2: 128}, (0, 0): {0: 0, 2: 256}},
         "fronts in pairs": {(1, 0): {0: 1, 1: 2, 2: 512, 3: 0}, (0, 0): {0: 0}},
         "slots in memory": {(1, 0): {0: 1, 1: 1, 2: 512, 3: 1}},
         "cut factors": {(1, 0): {0: 0}},
         "equal cut factors": {(1, 0): {0: 0}},
         "ragged": {(1, 0): {0: 1, 1: 1}, (0, 0): {0: 0}},
         "forest": {(0, 1): {0: 0, 5: 0}, (1, 0): {0: 1, 1: 4}}}


def _unknowns(shim, h, kind, level):
    shape = (C.c_int * 3)()
    subs = range(shim.shim_num_subdomains(h)) if kind else [0]
    return sum(shape[0] for i in subs if shim.shim_matrix_shape(h, kind, level, i, shape) == 0)


@pytest.mark.parametrize("name", ROUTES)
def test_schedules_read_nothing_but_their_own_system(name):
    d, levels = domain(name)
    shim = load_shim()
    err = C.create_string_buffer(512)
    flags = np.ascontiguousarray(d.flags, np.uint32)
    h = shim.shim_build((C.c_int * 3)(*d.size), (C.c_int * 3)(*d.sub_size), d.meta["vlevels"], levels,
                        flags.ctypes.data_as(C.POINTER(C.c_uint32)), err, 512)
    assert h, err.value
    rng = np.random.default_rng(3)
    stream = coefficients = 0.0
    try:
        for level in range(levels):
            for kind in (0, 1):
                n = _unknowns(shim, h, kind, level)
                if n == 0:
                    continue
                b = rng.uniform(-1, 1, n).astype(np.float32)
                x, xe = np.full(n, np.nan, np.float32), np.zeros(n, np.float32)
                info, by, co = (C.c_int * 11)(), C.c_double(), C.c_double()
                assert shim.shim_stream_walk(h, kind, level, _fp(b), _fp(x), info, C.byref(by), C.byref(co)) == 0
                assert shim.shim_plan_emulate(h, kind, level, _fp(b), _fp(xe)) == 0
                assert info[6] == 0 and info[7] == 0, (level, kind, "out of range, races", info[6], info[7])
                assert np.all(np.isfinite(x)), (level, kind, "NaN from outside the system")
                diff = float(np.max(np.abs(x.astype(np.float64) - xe)))
                assert diff <= RTOL * float(np.max(np.abs(xe))), (level, kind, diff)
                for i, v in TAKES[name].get((kind, level), {}).items():
                    assert info[i] == v, (name, kind, level, list(info))
                if name == "equal cut factors" and kind == 1 and level == 0:
                    assert info[0] == 0 and 2 * info[10] <= info[4], list(info)
                stream += by.value
                coefficients += co.value
        assert stream <= PADDING[name] * coefficients, stream / coefficients
    finally:
        shim.shim_free(h)


@pytest.mark.parametrize("trees,members", [(1, 1), (2700, 160), (2700, 320), (3400, 2)])
def test_small_trees_keep_their_slots_in_shared_memory(trees, members):
    # CTAs of four warps have no kernel with slots in global memory: thousands
    # of tiny fronts, a few trees to a CTA, around the edge of shared memory and
    # (3400) beyond four warps' coefficients.
    shim = load_shim()
    info = (C.c_int * 10)()
    e = shim.shim_forest_walk(trees, members, info)
    km, threads, in_memory = info[1], info[2], info[3]
    assert 0 <= e <= 1.2e-7 and info[6] == 0 and info[7] == 0, (e, list(info))
    assert threads == (128 if 3 * trees <= 8192 else 512)
    assert not (threads == 128 and in_memory), (km, threads, in_memory)
