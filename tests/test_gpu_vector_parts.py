"""The PCG vector kernels (project_dot, update_s, update_xr and the residual
kernels of kernels_pcg.cu; CONJUGATE_GRADIENT.cpp:30-75) work on parts of 2048
cells of the tiles' array: arrays shorter than a part, with a remainder of one,
two and three 8^3 tiles, and whole parts, in both precision forms.

After a few iterations the reported residual of the returned iterate equals
b - A x formed here in FP64 up to the FP32 rounding of A x (reference form,
2^-24 of its largest entry, and of b) or of r (precision form), and the
recursive residual differs from it by no more than the roundings of the FP32
updates: per iteration half an ulp of x through the seven coefficients of A
(their magnitudes add up to 12) and half an ulp each of q and r.
"""
import numpy as np
import pytest

from hierarchicaldd_b200 import domains
from hierarchicaldd_b200.domains import ACTIVE, INTERFACE
from hierarchicaldd_b200.solver import SPGrid_Domain_Decomposition_Solver

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def _residual(d, x):
    """b - A x at Active cells (FP64), A x, with A from the domain's flags: six
    faces, a neighbour outside the Active cells counting as zero."""
    act = (d.flags & ACTIVE) != 0
    bits = domains.face_bits(d.flags)
    ax = np.zeros(x.shape)
    xp = np.pad(np.where(act, x, 0.0), 1)
    k = 0
    for axis in range(3):
        for step in (-1, 1):
            nb = xp[tuple(slice(1 + (step if a == axis else 0), 1 + (step if a == axis else 0) + x.shape[a])
                          for a in range(3))]
            on = act & ((bits & (domains.FACE_MX << k)) != 0)
            ax[on] += (x - nb)[on]
            k += 1
    return np.where(act, d.rhs.astype(np.float64) - ax, 0.0), ax


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("cells,sub", [((8, 8, 8), 8), ((16, 8, 8), 8), ((24, 8, 8), 8), ((40, 8, 8), 8),
                                       ((32, 16, 8), 8), ((16, 16, 32), 16), ((32, 32, 32), 32)])
def test_residual_of_the_iterate(cells, sub, mixed):
    d = domains.small(cells, sub, 0, seed=21)
    m = dict(d.meta)
    its = 3
    s = SPGrid_Domain_Decomposition_Solver()
    try:
        s.Set_Domain(d.flags, d.rhs)
        s.Initialize_Preconditioner(m["vlevels"], d.size, d.sub_size, m["sigma_levels"], m["nVcycles"],
                                    m["interior_smoothing"], m["boundary_smoothing"], m["sigma_smoothing"],
                                    m["sigma_mg"], tol=1e-12, precision_mode=mixed, max_iters=its)
        res = s.Solve(allow_not_converged=True)
        x = s.Solution_F64()
    finally:
        s.close()
    assert res["iterations"] == its
    r, ax = _residual(d, x)
    b, rmax = np.abs(d.rhs).max(), np.abs(r).max()
    assert abs(res["b_inf"] - b) <= U * b
    tol = 2 * U * rmax if mixed else U * (np.abs(ax).max() + 2 * b) + 2 * U * rmax
    assert abs(res["true_residual_inf"] * b - rmax) <= tol, (res["true_residual_inf"], rmax)  # relative to b
    drift = its * U * (12 * np.abs(x).max() + 4 * b) * 2 + tol
    assert abs(res["final_norm"] - rmax) <= drift, (res["final_norm"], rmax)
    l2 = np.linalg.norm(r) / np.linalg.norm(d.rhs.astype(np.float64))
    assert abs(res["true_residual_l2"] - l2) <= tol / b * np.sqrt(r.size) + 4 * U * l2, (res["true_residual_l2"], l2)
