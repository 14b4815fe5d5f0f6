"""Fast diagonalisation with a body that reaches the domain's faces: the
partners of outer rows are then solid cells, which the launch that solves the
outer rows also writes (csrc/fastpoisson.cu, k_fp_edges).  Equal runs give
bitwise equal fields and counts, and the fields are the FP64 solve's."""
import importlib

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["FP64", "MIXED_MG", "MIXED32"])
@pytest.mark.parametrize("lo,hi", [((0.31, -0.4, -0.4), (0.68, 0.52, 0.47)), ((-0.4, -0.4, -0.4), (0.22, 1.4, 0.61))],
                         ids=["edge", "corner"])
def test_equal_runs_are_equal(ibm, lo, hi, mode):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    stl = wl._body_stl("boxes", dict(boxes=[(lo, hi)]), ("boxes", "faces", lo, hi))
    n = (26, 24, 22)
    case = dict(xf=np.linspace(0, 1, n[0] + 1), yf=np.linspace(0, 1, n[1] + 1), zf=np.linspace(0, 1, n[2] + 1),
                re=150.0, dt=1e-3, bc=["W vel 1 0 0", "E press 0", "S slip", "N slip", "D wall", "U slip"], stl=stl)
    pad = tuple(q + 4 for q in n)
    rng = np.random.default_rng(3)
    state = [0.5 + 0.1 * rng.standard_normal(pad), 0.1 * rng.standard_normal(pad), 0.1 * rng.standard_normal(pad),
             np.zeros(pad)]

    def run(precision, tol):
        s = wl.build_solver(ibm, case, tol=tol)
        s.set_precision(getattr(ibm, precision))
        s.init_flow_array(*state)
        s.iterate(3)
        out = {f: s.get_field(f) for f in ("u1", "u2", "u3", "p", "pprime")}
        count = s.stats()["iters_p_total"]
        s.close()
        return out, count

    first, k = run(mode, 1e-9)
    for _ in range(3):
        again, q = run(mode, 1e-9)
        assert q == k
        for f in first:
            assert np.array_equal(first[f], again[f], equal_nan=True), f
    ref, _ = run("FP64", 1e-12)
    for f in ("u1", "u2", "u3"):
        assert np.array_equal(np.isnan(first[f]), np.isnan(ref[f]))
        # FP32 stages: the rounding of O(dt) increments (~1e-7 relative).
        assert rel_l2(first[f], ref[f]) < 1e-6, (f, rel_l2(first[f], ref[f]))
