"""The routes of a supernodal solve plan (sn_resident.cu, sn_solve.cu), each at
shapes where it can go wrong: one CTA for the only tree; one CTA per tree, and
per 2 or 4 trees with the same factor; slots in shared or global memory; lower
trees plus tasks above them, of one factor and of several; trees alone (a
forest of small ones); test_cpu_sn_streams.py checks that the domains take these
routes.  Against the host walk of the same fronts, and batches
against single solves.

Tolerance: the kernels' products are exact in FP64 and their sums differ from
the host's only in order (1e-16 of the terms), so results differ by at most the
final rounding to FP32, one ulp: 1.2e-7 of the largest entry.
"""
import ctypes as C

import numpy as np
import pytest

from hierarchicaldd_b200 import domains
from shim_ffi import load_shim
from sn_routes import ROUTES, domain

pytestmark = pytest.mark.gpu

RTOL = 1.2e-7


def _fp(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


@pytest.mark.parametrize("name", ROUTES)
def test_every_route_matches_the_host_walk_and_its_batches(name):
    from hierarchicaldd_b200 import _lib
    from hierarchicaldd_b200.solver import SPGrid_Domain_Decomposition_Solver
    d, levels = domain(name)
    m = dict(d.meta)
    shim = load_shim()
    err = C.create_string_buffer(512)
    flags = np.ascontiguousarray(d.flags, np.uint32)
    h = shim.shim_build((C.c_int * 3)(*d.size), (C.c_int * 3)(*d.sub_size), m["vlevels"], levels,
                        flags.ctypes.data_as(C.POINTER(C.c_uint32)), err, 512)
    assert h, err.value
    s = SPGrid_Domain_Decomposition_Solver()
    lib = _lib.load()
    rng = np.random.default_rng(11)
    checked = 0
    try:
        s.Set_Domain(d.flags, d.rhs)
        s.Initialize_Preconditioner(m["vlevels"], d.size, d.sub_size, levels, m["nVcycles"],
                                    m["interior_smoothing"], m["boundary_smoothing"], m["sigma_smoothing"],
                                    m["sigma_mg"])
        for level in range(levels):
            for kind in (0, 1):
                nn = C.c_int()
                assert lib.hdd_interface_solve(s.h, kind, level, None, None, C.byref(nn)) == 0
                if nn.value == 0:
                    continue
                b = rng.uniform(-1, 1, (4, nn.value)).astype(np.float32)
                x = np.full((4, nn.value), np.nan, np.float32)
                st = [lib.hdd_interface_solve(s.h, kind, level, _fp(b[k]), _fp(x[k]), C.byref(nn)) for k in range(4)]
                if st[0] == 5 and level == levels - 1:
                    continue  # the coarsest level is solved as a whole
                assert st == [0] * 4, lib.hdd_last_error(s.h)
                xe = np.zeros(nn.value, np.float32)
                assert shim.shim_plan_emulate(h, kind, level, _fp(b[0]), _fp(xe)) == 0
                diff = float(np.max(np.abs(x[0].astype(np.float64) - xe)))
                assert diff <= RTOL * float(np.max(np.abs(xe))), (level, kind, diff)
                for nrhs in (2, 4):
                    xb = np.full((nrhs, nn.value), np.nan, np.float32)
                    assert lib.hdd_interface_solve_batch(s.h, kind, level, nrhs, _fp(b), _fp(xb), C.byref(nn)) == 0
                    assert np.array_equal(xb, x[:nrhs]), (level, kind, nrhs)
                checked += 1
        assert checked >= 2
    finally:
        s.close()
        shim.shim_free(h)


def test_large_fronts_take_batches():
    # A front of more than 6240 rows (140^3 of 8^3 subdomains: about 6500) is no
    # reason to refuse right-hand sides side by side.
    from hierarchicaldd_b200 import _lib
    from hierarchicaldd_b200.solver import SPGrid_Domain_Decomposition_Solver
    d = domains.small(140, 8, 5, seed=1)
    m = d.meta
    s = SPGrid_Domain_Decomposition_Solver()
    lib = _lib.load()
    try:
        s.Set_Domain(d.flags, d.rhs)
        s.Initialize_Preconditioner(m["vlevels"], d.size, d.sub_size, 2, m["nVcycles"], m["interior_smoothing"],
                                    m["boundary_smoothing"], m["sigma_smoothing"], m["sigma_mg"])
        nn = C.c_int()
        assert lib.hdd_interface_solve(s.h, 0, 0, None, None, C.byref(nn)) == 0
        rng = np.random.default_rng(5)
        b = rng.uniform(-1, 1, (4, nn.value)).astype(np.float32)
        x, xb = np.zeros_like(b), np.zeros_like(b)
        for k in range(4):
            assert lib.hdd_interface_solve(s.h, 0, 0, _fp(b[k]), _fp(x[k]), C.byref(nn)) == 0
        assert lib.hdd_interface_solve_batch(s.h, 0, 0, 4, _fp(b), _fp(xb), C.byref(nn)) == 0, lib.hdd_last_error(s.h)
        assert np.array_equal(xb, x)
    finally:
        s.close()
