"""The fast-diagonalisation preconditioner of the pressure solve
(csrc/fastpoisson.cu) over the grids and boundary conditions that choose its
branches: the tridiagonal axis (x, y, or none where both wrap), pinned and
pressure-bounded problems, axes at the edges of the transform tiles (32, 64),
of the tridiagonal segments (16 rows, 256-cell blocks) and odd ones, and a
body with its near-body sweeps.

Without a body the preconditioner is the inverse of the pressure rows up to
rounding (FP32 in the mixed modes: about 1e-7 times the growth of the 1-D
problems' condition, below 1e-3; FP64: below 1e-11), and one BiCGSTAB
iteration applies it twice.  So at a relative tolerance of 1e-8 a solve takes
at most three iterations with the FP32 one, and at 1e-10 at most two with the
FP64 one, where the multigrid needs 7 to 50.  The fields are held to the
oracle's (its solves to 1e-13) at the tolerance of the solve times the
pressure's loss of three digits."""
import importlib
import os
import sys

import numpy as np
import pytest

from conftest import ROOT, rel_l2

pytestmark = pytest.mark.gpu

WALLS = ["W wall", "E wall", "S wall", "N wall", "D wall", "U vel 1 0 0"]
OPEN = ["W vel 1 0 0", "E press 0", "S slip", "N slip", "D slip", "U slip"]
XZ = ["W per", "E per", "S wall", "N wall", "D per", "U per"]
XY = ["W per", "E per", "S per", "N per", "D wall", "U vel 1 0 0"]
Y = ["W vel 1 0 0", "E press 0", "S per", "N per", "D slip", "U press 0"]
VP = ["W velper 1", "E velper 0", "S wall", "N wall", "D slip", "U slip"]
GRIDS = [
    ((32, 32, 32), WALLS), ((33, 31, 17), WALLS), ((16, 65, 64), WALLS), ((64, 63, 5), OPEN), ((3, 4, 3), WALLS),
    ((257, 9, 10), OPEN), ((9, 272, 11), XZ), ((15, 16, 33), XZ), ((20, 12, 18), XY), ((31, 7, 9), XY),
    ((17, 18, 19), Y), ((24, 13, 14), VP), ((130, 6, 7), VP),
]


def _case(shape, bc):
    """Stretched faces on the axes that do not wrap, a smooth flow with
    seeded noise."""
    rng = np.random.default_rng(sum(shape))
    faces = []
    for n, side in zip(shape, "WSD"):
        w = rng.uniform(0.7, 1.3, n) if f"{side} per" not in bc else np.ones(n)
        f = np.concatenate([[0.0], np.cumsum(w)])
        faces.append(f / f[-1] * (0.5 + n / 32))
    pad = tuple(n + 4 for n in shape)
    state = [1.0 + 0.1 * rng.standard_normal(pad), 0.1 * rng.standard_normal(pad), 0.1 * rng.standard_normal(pad),
             np.zeros(pad)]
    return dict(xf=faces[0], yf=faces[1], zf=faces[2], re=100.0, dt=2e-3, bc=bc), state


def _run(ibm, wl, case, state, mode, tol):
    s = wl.build_solver(ibm, case, tol=tol)
    s.set_precision(getattr(ibm, mode))
    s.init_flow_array(*state)
    s.iterate(2)
    st = s.stats()
    out = {f: s.get_field(f) for f in ("u1", "u2", "u3", "p")}
    s.close()
    return out, st


@pytest.fixture(scope="module")
def orc():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    return importlib.import_module("oracle")


@pytest.mark.parametrize("shape,bc", GRIDS, ids=["x".join(map(str, g[0])) for g in GRIDS])
def test_solves_in_few_iterations_and_matches_the_oracle(ibm, orc, shape, bc):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    case, state = _case(shape, bc)
    o = orc.Oracle(dict(case, tol=1e-13))
    o.init(*state)
    o.iterate(2)
    for mode, tol, most in (("FP64", 1e-10, 2), ("MIXED_MG", 1e-8, 3)):
        out, st = _run(ibm, wl, case, state, mode, tol)
        assert st["iters_p_total"] <= 2 * most, (mode, st["iters_p_total"])
        for f, a in out.items():
            assert rel_l2(a, o.get(f)) < 1e3 * tol, (mode, f, rel_l2(a, o.get(f)))


@pytest.mark.parametrize("shape", [(40, 32, 33), (70, 37, 36)])
def test_body_sweeps_match_the_oracle(ibm, orc, shape):
    """A sphere: the solve no longer inverts the rows, the sweeps near the
    body keep the iterations far below the unswept solve's hundreds."""
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    case = wl.sphere(*shape, subdivisions=3)
    state = wl.initial_state(case)
    o = orc.Oracle(dict(case, tol=1e-13))
    o.init(*state)
    o.iterate(2)
    out, st = _run(ibm, wl, case, state, "MIXED_MG", 1e-9)
    assert st["iters_p_total"] <= 2 * 12, st["iters_p_total"]
    for f, a in out.items():
        ref = o.get(f)
        assert np.array_equal(np.isnan(a), np.isnan(ref))
        assert rel_l2(a, ref) < 1e-6, (f, rel_l2(a, ref))
