"""FP64 multigrid prolongation (csrc/multigrid.cu, k_mg0_prolong_lines) against the
FP32 one, which blends each cell by itself.  FP64 and MIXED_MG steps from rest
solve the same FP64 momentum rows in the same way, so their pressure right-hand
sides are equal, and one BiCGSTAB iteration with one V-cycle per direction
leaves p' and a residual that differ by the cycles' arithmetic alone: FP32
rounding through some hundred operations per cell and level, below 1e-3, where
a wrong weight or neighbour changes both by tenths.  Stretched grids (groups of
one and two cells), ends of the eight-plane walks and of the 32 x 8 tiles, and
inactive coarse cells in a body."""
import importlib

import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_fastpoisson import OPEN, WALLS, _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,bc", [((9, 10, 35), WALLS), ((16, 33, 31), OPEN), ((17, 8, 64), WALLS),
                                      ((8, 7, 33), OPEN), ((40, 32, 33), "sphere"), ((57, 40, 24), "sphere")], ids=str)
def test_one_iteration_agrees(ibm, shape, bc):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    if bc == "sphere":
        case = wl.sphere(*shape, subdivisions=3)
        state = wl.initial_state(case)
    else:
        case, state = _case(shape, bc)
    out, res = [], []
    for mode in ("FP64", "MIXED_MG"):
        s = wl.build_solver(ibm, case, tol=1e-12, coarsening=ibm.COARSEN_SPACING)
        s.set_precision(getattr(ibm, mode))
        s.set_warm_start(False)
        s.set_max_iters(200, 1)
        s.init_flow_array(*state)
        s.iterate(1)
        out.append((s.get_field("u1star"), s.get_field("pprime")))
        res.append(s.stats()["res_p"])
        assert s.stats()["iters_p"] == 1
        s.close()
    (u0, p0), (u1, p1) = out
    assert np.array_equal(u0, u1, equal_nan=True)
    assert 0 < res[0] < 0.5 and abs(res[1] - res[0]) < 1e-3 * res[0], res
    assert rel_l2(p1, p0) < 1e-3, rel_l2(p1, p0)
