"""The momentum solve by Jacobi sweeps (csrc/momsweep.h) where its branches
differ: extrapolated outlets meeting at edges and corners (their outer rows
are resolved axis by axis), every kind of outer row, a body cut by the
boundary (ghosts beside outer cells, ghost stencils reading them), a body
inside, and a time step whose diffusion numbers leave the solve to BiCGSTAB.

Both sides solve to a relative residual of 1e-12 (the oracle to 1e-13); the
rows' condition is below 10 (diagonal dominance by 1 / (1 + 2 rho), ghost
rows near 1), so the velocities agree to 1e-10, with the two pressure solves
to 1e-9 as in the fixtures' tests."""
import importlib
import os
import sys

import numpy as np
import pytest

from conftest import ROOT, rel_l2

pytestmark = pytest.mark.gpu

INFLOW = ["W vel 1 0.2 0.1", "E press 0", "S slip", "N press 0.1", "D wall", "U press 0"]
MIXED = ["W velper 0.5", "E velper 0", "S press 0", "N vel 0.2 -0.1 0", "D sym", "U slip"]
PERIODIC = ["W per", "E per", "S press 0", "N wall", "D per", "U per"]


def _state(shape, seed):
    rng = np.random.default_rng(seed)
    pad = tuple(n + 4 for n in shape)
    return [0.5 + 0.1 * rng.standard_normal(pad), 0.1 * rng.standard_normal(pad), 0.1 * rng.standard_normal(pad),
            np.zeros(pad)]


def _check(ibm, case, modes=("FP64", "MIXED")):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    orc = importlib.import_module("oracle")
    shape = tuple(len(case[k]) - 1 for k in ("xf", "yf", "zf"))
    state = _state(shape, sum(shape))
    o = orc.Oracle(dict(case, tol=1e-13))
    o.init(*state)
    o.iterate(2)
    iters = []
    for mode in modes:
        s = wl.build_solver(ibm, case, tol=1e-12)
        s.set_precision(getattr(ibm, mode))
        s.init_flow_array(*state)
        s.iterate(2)
        iters.append(max(s.stats()["iters_u"]))
        for f in ("u1", "u2", "u3", "u1star", "u2star", "u3star"):
            a, b = s.get_field(f), o.get(f)
            if not f.endswith("star"):
                assert np.array_equal(np.isnan(a), np.isnan(b)), (mode, f)
            assert rel_l2(a, b) < 1e-9, (mode, f, rel_l2(a, b))
        s.close()
    return iters


def _faces(shape, size=1.0):
    out = []
    for q, n in enumerate(shape):
        w = 1.0 + 0.3 * np.sin(np.arange(n) * (q + 2.0))
        f = np.concatenate([[0.0], np.cumsum(w)])
        out.append(f / f[-1] * size)
    return out


@pytest.mark.parametrize("bc", [INFLOW, MIXED, PERIODIC], ids=["outlets", "mixed", "periodic"])
@pytest.mark.parametrize("shape", [(9, 8, 33), (16, 17, 7)])
def test_outer_rows(ibm, shape, bc):
    xf, yf, zf = _faces(shape)
    if bc is PERIODIC:
        xf, zf = np.linspace(0, 1, shape[0] + 1), np.linspace(0, 1, shape[2] + 1)
    if bc is MIXED:
        xf = np.linspace(0, 1, shape[0] + 1)
    _check(ibm, dict(xf=xf, yf=yf, zf=zf, re=200.0, dt=1e-3, bc=bc))


@pytest.mark.parametrize("lo,hi", [((0.31, 0.33, -0.4), (0.68, 0.71, 0.52)), ((0.31, 0.33, 0.28), (0.68, 0.71, 0.63))],
                         ids=["cut", "inside"])
def test_body(ibm, lo, hi):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    n = (26, 24, 22)
    stl = wl._body_stl("boxes", dict(boxes=[(lo, hi)]), ("boxes", "momsweep", lo, hi))
    case = dict(xf=np.linspace(0, 1, n[0] + 1), yf=np.linspace(0, 1, n[1] + 1), zf=np.linspace(0, 1, n[2] + 1),
                re=150.0, dt=1e-3, bc=["W vel 1 0 0", "E press 0", "S slip", "N slip", "D wall", "U slip"], stl=stl)
    _check(ibm, case)


def test_large_diffusion_numbers_take_bicgstab(ibm):
    """dt / (2 Re h^2) of about 1 per axis: rho > 0.5."""
    n = (12, 10, 14)
    case = dict(xf=np.linspace(0, 1, n[0] + 1), yf=np.linspace(0, 1, n[1] + 1), zf=np.linspace(0, 1, n[2] + 1), re=1.0,
                dt=1e-2, bc=["W wall", "E wall", "S wall", "N wall", "D wall", "U vel 1 0 0"])
    _check(ibm, case)
