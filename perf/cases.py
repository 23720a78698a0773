"""The work that users of this solver have it do, as measurable cases.

A user's program describes a Poisson domain (cell flags), sets the solver up
once and then solves right-hand side after right-hand side on it: a pass of a
"solve" case is Set_RHS + Solve + Solution (or the page forms of the same) on
host arrays, as those entry points take them.  A "serve" case is a burst of
requests to the serving front end with its domains resident.  An "operator"
case is the allocation-free Laplacian + dot product on the caller's device
arrays.  Domains, sizes and settings are those of the repository's own
workloads (hierarchicaldd_b200/domains.py), benchmark and tests.
"""
from __future__ import annotations

import ctypes
import functools
import random

import numpy as np
import torch

from hierarchicaldd_b200 import _lib, domains
from hierarchicaldd_b200.server import SolveServer, make_options
from hierarchicaldd_b200.solver import SPGrid_Domain_Decomposition_Solver

# Fewest PCG iterations a solve to 1e-6 takes on these domains; used for the
# work a solve cannot do without (measured counts are 7 to 40).
ITERATIONS = 7


def _case(kind, name, cells, sub, vlevels, smoothing, sigma_levels, precision=0, exact_coarse=False, multilevel=False,
          domain="sphere", geometry=0, source="noise", requests=0):
    nx, ny, nz = cells
    c = dict(kind=kind, name=name, nx=nx, ny=ny, nz=nz, sub=sub, vlevels=vlevels, interior=smoothing[0],
             boundary=smoothing[1], sigma_levels=sigma_levels, precision=precision, exact_coarse=exact_coarse,
             multilevel=multilevel, domain=domain, geometry=geometry, source=source, requests=requests)
    if not name:
        del c["name"]
    return c


def listed():
    return [
        # The operator alone, for a caller's own Krylov loop on device arrays:
        # the regular case of the 32^3-subdomain workloads ...
        _case("operator", "operator 128 sub 32", (128, 128, 128), 32, 4, (4, 4), 3),
        # ... and a ragged box whose last subdomains are partial.
        _case("operator", "operator 75x93x61 sub 16", (75, 93, 61), 16, 3, (3, 3), 3),
        # The smallest solve (the tests' and smoke run's domain): latency.
        _case("solve", "solve 16 sub 8", (16, 16, 16), 8, 3, (3, 3), 2),
        # Ragged small box, delta source.
        _case("solve", "solve 40x36x44 sub 8", (40, 36, 44), 8, 3, (3, 3), 2, source="deltas"),
        # The 64^3 workload at its own settings, reference precision.
        _case("solve", "solve 64 sub 16", (64, 64, 64), 16, 3, (3, 3), 3, source="deltas"),
        # The reference generator's own domain (Neumann bubble), which runs the
        # whole-grid V-cycle.
        _case("solve", "solve bubble 48 sub 16", (48, 48, 48), 16, 3, (3, 3), 3, domain="bubble", source="deltas"),
        # Serving-mix domain with the precision form, random spheres.
        _case("solve", "solve 128 sub 32 mixed", (128, 128, 128), 32, 4, (4, 4), 3, precision=1, exact_coarse=True,
              domain="spheres", geometry=4, source="deltas"),
        # Sparse sphere union handed over as SPGrid pages (an eighth of the
        # 1024^3 workload's edge), precision form.
        _case("solve", "solve sparse 128 sub 32", (128, 128, 128), 32, 5, (3, 3), 4, precision=1, domain="union",
              source="noise"),
        # Two-level DD at the two-level demo's default options.
        _case("solve", "solve two-level 128x64x64", (128, 64, 64), 64, 3, (1, 3), 3, multilevel=True),
        # The headline workload's settings (32^3 subdomains, reference
        # precision) on 192^3 cells, the largest size of the serving mix: its
        # set-up, which is repeated for each measured state, stays within
        # seconds, and its solve plans are several times the L2 cache, as at 256^3.
        _case("solve", "solve 192 sub 32", (192, 192, 192), 32, 4, (4, 4), 4, source="noise+delta"),
        # A burst of requests on a resident 96^3 domain of the serving mix.
        _case("serve", "serve 96 sub 16, 4 requests", (96, 96, 96), 16, 3, (3, 3), 3, precision=1, exact_coarse=True,
              domain="spheres", geometry=5, source="deltas", requests=4),
    ]


def _edge(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng: random.Random):
    """One more case: an operator, a solve or a burst of requests on a box whose
    edges are log-uniform over the listed range, odd ones among them."""
    kind = rng.choice(["operator", "operator", "solve", "solve", "solve", "serve"])
    top = {"operator": 128, "solve": 160, "serve": 96}[kind]
    a = _edge(rng, 16, top)
    # The other edges within a factor of two, as simulation boxes are.
    cells = (a,) + tuple(max(12, min(top, int(round(a * 2 ** rng.uniform(-0.8, 0.5))))) for _ in range(2))
    big = max(cells)
    # Subdomain sizes as the serving mix picks them, 8 for the smallest boxes.
    sub = 8 if big < 32 else (16 if big < 112 else 32)
    if sub == 32:
        vlevels, smoothing, sigma_levels = 4, (4, 4), 3
    else:
        vlevels, smoothing, sigma_levels = 3, (3, 3), (2 if sub == 8 else 3)
    precision = 1 if kind == "serve" else rng.randint(0, 1)
    return _case(kind, "", cells, sub, vlevels, smoothing, sigma_levels, precision=precision,
                 exact_coarse=bool(precision), domain=rng.choice(["sphere", "spheres"]),
                 geometry=rng.randrange(1 << 16), source=rng.choice(["noise", "deltas", "noise+delta"]),
                 requests=rng.randint(2, 6) if kind == "serve" else 0)


# -- inputs -------------------------------------------------------------------


@functools.lru_cache(maxsize=2)
def _flags(kind, nx, ny, nz, geometry):
    size = (nx + 1, ny + 1, nz + 1)
    small = min(nx, ny, nz)
    if kind == "bubble":
        return domains.reference_generator(size, (1 + nx // 16, ny // 2, nz // 2)).flags
    if kind == "union":
        return domains.config5(1024 // nx).flags
    if kind == "sphere":
        return domains.box_with_spheres(size, [((nx // 2, ny // 2, nz // 2), small * 3 // 16)])
    # 1-4 spheres of radius U[0.05, 0.2] of the smallest edge, as the serving mix.
    rng = np.random.Generator(np.random.Philox(geometry))
    spheres = []
    for _ in range(int(rng.integers(1, 5))):
        centre = tuple(int(rng.integers(1, n)) for n in (nx, ny, nz))
        spheres.append((centre, float(rng.uniform(0.05, 0.2)) * small))
    return domains.box_with_spheres(size, spheres)


def _case_flags(case):
    return _flags(case["domain"], case["nx"], case["ny"], case["nz"], case["geometry"])


def _rhs(case, flags, rng):
    active = (flags & domains.ACTIVE) != 0
    rhs = np.zeros(flags.shape, np.float32)
    if "noise" in case["source"]:
        # Zero-mean source on every Active cell (small beside the delta, where there is one).
        amp = 1e-3 if "delta" in case["source"] else 1.0
        rhs = rng.random(flags.shape, dtype=np.float32)
        rhs -= 0.5
        rhs *= 2 * amp
        rhs *= active
    if "delta" in case["source"]:
        cells = np.flatnonzero(active)
        n = 1 if case["source"] == "noise+delta" else int(rng.integers(1, 4))
        rhs.reshape(-1)[cells[rng.integers(0, len(cells), n)]] += np.float32(1.0)
    return rhs


def _rhs_all(case, flags, seed):
    """The seed's right-hand sides: one, or one per request."""
    rng = np.random.Generator(np.random.Philox(int(seed)))
    return [_rhs(case, flags, rng) for _ in range(max(1, case["requests"]))]


def prepare(case, seed):
    flags = _case_flags(case)
    rhs = _rhs_all(case, flags, seed)
    args = dict(precision_mode=case["precision"], coarse_solve=1 if case["exact_coarse"] else 0)
    if case["kind"] == "serve":
        server = SolveServer(slots=4)
        domain = server.add_domain(flags, make_options(
            flags.shape, (case["sub"],) * 3, vlevels=case["vlevels"], interior_smoothing=case["interior"],
            boundary_smoothing=case["boundary"], sigma_levels=case["sigma_levels"], **args))
        server.wait_domain(domain)
        return dict(case=case, server=server, domain=domain, rhs=rhs)
    s = SPGrid_Domain_Decomposition_Solver(device=0)
    pages = None
    if case["domain"] == "union":
        pages = domains.to_pages(flags, rhs[0])
        s.Set_Domain_Pages(*pages)
    else:
        s.Set_Domain(flags, rhs[0])
    s.Initialize_Preconditioner(case["vlevels"], flags.shape, (case["sub"],) * 3, case["sigma_levels"], 1,
                                case["interior"], case["boundary"], 3, 1, multilevel=case["multilevel"], **args)
    state = dict(case=case, solver=s, rhs=rhs, pages=pages)
    if case["kind"] == "operator":
        state["x"] = torch.from_numpy(_operand(case, flags, seed)).cuda()
        state["y"] = torch.zeros(flags.shape, dtype=torch.float32, device="cuda")
        state["dot"] = torch.zeros(1, dtype=torch.float64, device="cuda")
    return state


def _operand(case, flags, seed):
    x = np.random.Generator(np.random.Philox(int(seed) + 1)).standard_normal(flags.shape, dtype=np.float32)
    return x * ((flags & domains.ACTIVE) != 0)


# -- one pass -----------------------------------------------------------------


def run(state):
    kind = state["case"]["kind"]
    if kind == "operator":
        s, p = state["solver"], ctypes.c_void_p
        status = _lib.load().hdd_multiply_dot_dense_device_noalloc(
            s.h, p(state["x"].data_ptr()), p(state["y"].data_ptr()), p(state["dot"].data_ptr()),
            p(torch.cuda.current_stream().cuda_stream))
        if status != 0:
            raise _lib.HddError(status, "hdd_multiply_dot_dense_device_noalloc")
        return [state["y"], state["dot"]]
    if kind == "serve":
        server, domain = state["server"], state["domain"]
        ids = [server.submit(domain, b) for b in state["rhs"]]
        out = []
        for i in ids:
            status, _, x, _ = server.poll(i, domain)
            if status != 0:
                raise _lib.HddError(status, "request %d" % i)
            out.append(x)
        return out
    s = state["solver"]
    if state["pages"] is not None:
        origin, _, rhs = state["pages"]
        s.Set_RHS_Pages(origin, rhs)
        s.Solve()
        return s.Solution_Pages(origin)
    s.Set_RHS(state["rhs"][0])
    s.Solve()
    return s.Solution()


# -- what a pass cannot do without, and how far outputs may be off --------------


def work(case):
    cells = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if case["domain"] == "union":
        cells = cells // 8
    if case["kind"] == "operator":
        # x and the 2-byte flags in, y out; 6 differences, 6 sums and the dot's 2.
        return {"bytes": 10.0 * cells, "flops": 14.0 * cells}
    # Per PCG iteration: the Laplacian and the vector updates read or write
    # each of x, r, s, q, z about twice; two V-cycle passes of
    # 2 (2 boundary + interior) sweeps (each about 15 operations on half the
    # cells) and a residual.
    sweeps = 2 * 2 * (2 * case["boundary"] + case["interior"]) * 0.5 + 2
    per = {"bytes": 50.0 * cells, "flops": (15.0 * sweeps + 30.0) * cells}
    n = ITERATIONS * max(1, case["requests"])
    return {k: v * n for k, v in per.items()}


def tolerance(case):
    if case["kind"] == "operator":
        # FP64 face sums rounded to FP32 once; the dot in FP64.
        return {"rel": 1e-6}
    # PCG stops at a relative residual of 1e-6: its distance from the exact
    # solution (see exact) is up to 7e-4 here (4e-8 to 2e-4 on the smaller
    # domains), and a correct solve whose interface solves sum in another order
    # may stop an iteration earlier or later and be as far off on the other side.
    return {"rel": 2e-3}


def exact(case, seed):
    """The same outputs in 64 bits: the operator by shifted sums, the solves by
    a Jacobi-preconditioned conjugate gradient to 1e-12 on dense arrays."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    flags = _case_flags(case)
    f = torch.from_numpy(flags.astype(np.int64)).to(dev)
    unknown = ((f & domains.ACTIVE) != 0).double()
    faces = sum(((f & (domains.FACE_MX << k)) != 0).double() for k in range(6)) * unknown

    def neighbours(u):
        out = torch.zeros_like(u)
        for a in range(3):
            n = u.shape[a]
            out.narrow(a, 1, n - 1).add_(u.narrow(a, 0, n - 1))
            out.narrow(a, 0, n - 1).add_(u.narrow(a, 1, n - 1))
        return out

    if case["kind"] == "operator":
        x = torch.from_numpy(_operand(case, flags, seed)).to(dev).double()
        y = (faces * x - neighbours(x)) * unknown  # minus the sum of the differences
        return [y, (x * y).sum().reshape(1)]

    inv = torch.where(faces > 0, 1.0 / faces.clamp(min=1.0), torch.zeros_like(faces))

    def solve(b):
        b = torch.from_numpy(b).to(dev).double() * unknown
        x = torch.zeros_like(b)
        r = b.clone()
        z = inv * r
        p = z.clone()
        rz = (r * z).sum()
        stop = 1e-12 * float(r.abs().max())
        for it in range(20000):
            q = (faces * p - neighbours(p)) * unknown
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            if it % 16 == 15 and float(r.abs().max()) <= stop:
                break
            z = inv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x

    xs = [solve(b) for b in _rhs_all(case, flags, seed)]
    if case["kind"] == "serve":
        return xs
    x = xs[0].cpu().numpy()
    if case["domain"] == "union":
        return domains.to_pages(flags, x)[2]
    return x
