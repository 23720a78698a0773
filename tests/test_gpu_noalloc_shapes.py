"""The allocation-free operator against the tiled Laplacian for every tile edge
and for boxes whose last tiles hold one plane, one row or a part of a unit
(8 planes by up to 8, 16 rows) on each axis: y bit for bit (the same FP64 face
sums in the same order), the dot within 1e-12 (the same FP32 products summed
in FP64, at most 2^21 terms of relative rounding 2^-53 each)."""
import ctypes as C

import numpy as np
import pytest

from hierarchicaldd_b200 import domains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,sub,radius", [
    ((16, 23, 17), 8, 3), ((15, 16, 40), 8, 4), ((32, 31, 33), 16, 6), ((17, 48, 32), 16, 4),
    ((64, 63, 65), 32, 10), ((33, 40, 95), 32, 8)])
def test_noalloc_equals_tiled_laplacian(cells, sub, radius):
    import torch
    from hierarchicaldd_b200 import _lib
    from hierarchicaldd_b200.solver import SPGrid_Domain_Decomposition_Solver

    d = domains.small(cells, sub, radius, seed=3)
    m = d.meta
    s = SPGrid_Domain_Decomposition_Solver()
    try:
        s.Set_Domain(d.flags, d.rhs)
        s.Initialize_Preconditioner(m["vlevels"], d.size, d.sub_size, m["sigma_levels"], m["nVcycles"],
                                    m["interior_smoothing"], m["boundary_smoothing"], m["sigma_smoothing"],
                                    m["sigma_mg"])
        x = np.random.default_rng(5).standard_normal(d.size).astype(np.float32)
        want = s.Multiply(x)
        xd = torch.from_numpy(x).cuda()
        yd = torch.full(d.size, 7.5, dtype=torch.float32, device="cuda")
        dot = torch.zeros(1, dtype=torch.float64, device="cuda")
        p = C.c_void_p
        st = _lib.load().hdd_multiply_dot_dense_device_noalloc(
            s.h, p(xd.data_ptr()), p(yd.data_ptr()), p(dot.data_ptr()), p(torch.cuda.current_stream().cuda_stream))
        assert st == _lib.HDD_OK
        y = yd.cpu().numpy()
        stored = y != np.float32(7.5)  # cells outside the stored tiles are left alone
        assert np.array_equal(y[stored], want[stored])
        assert np.all(want[~stored] == 0)
        ref = float(np.sum((x * want)[stored].astype(np.float64)))
        assert abs(float(dot.item()) - ref) <= 1e-12 * abs(ref) + 1e-12 * float(np.sum(np.abs((x * want)[stored]), dtype=np.float64))
    finally:
        s.close()
