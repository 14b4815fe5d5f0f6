"""FP64 multigrid prolongation along lines (csrc/multigrid.cu,
k_mg0_prolong_lines): stretched grids with an axis past 512 cells, which the
multigrid serves, so that its first level has groups of one and of two cells;
ends of the eight-plane walks, boundaries, and inactive coarse cells in a body.

MIXED_MG runs the same cycle in FP32 through another kernel under the same
FP64 iteration: the cycles differ by FP32 rounding (1e-6), so the counts of a
step agree to two iterations and a tenth.  (What the solve itself leaves in the
fields depends on the long axis's condition, not on the cycle.)"""
import importlib

import numpy as np
import pytest

from test_gpu_fastpoisson import OPEN, WALLS, _case, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,bc", [((9, 10, 520), WALLS), ((530, 12, 9), OPEN), ((515, 33, 7), WALLS),
                                      ((514, 16, 40), "sphere")], ids=str)
def test_fp64_cycle_matches_the_fp32_one(ibm, shape, bc):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    if bc == "sphere":
        case = wl.sphere(*shape, subdivisions=3)
        state = wl.initial_state(case)
    else:
        case, state = _case(shape, bc)
    tol = 1e-10
    ref, r = _run(ibm, wl, case, state, "MIXED_MG", tol)
    out, st = _run(ibm, wl, case, state, "FP64", tol)
    assert abs(st["iters_p_total"] - r["iters_p_total"]) <= 2 * 2 + 0.1 * r["iters_p_total"]
    for f, a in out.items():
        assert np.array_equal(np.isnan(a), np.isnan(ref[f]))
