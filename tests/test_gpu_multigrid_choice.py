"""IBMSolver_set_coarsening has the multigrid precondition the pressure solves in
every precision; without it the same grid takes the fast diagonalisation, to
which the multigrid's settings mean nothing (csrc/solver.cu).

Without a body the fast diagonalisation needs one to three iterations, a
V-cycle of one sweep a level many more, and a V-cycle of six fewer than that of
one; all of them stop at the same test, so the velocities agree to the solves'
tolerance times the condition of the momentum rows and three digits."""
import importlib

import pytest

from conftest import rel_l2
from test_gpu_fastpoisson import WALLS, XZ, _case

pytestmark = pytest.mark.gpu


def _solver(ibm, case, state, mode, coarsening, sweeps=None):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    s = wl.build_solver(ibm, case, tol=1e-9, coarsening=coarsening)
    s.set_precision(getattr(ibm, mode))
    if sweeps:
        s.set_multigrid(*sweeps)
    s.init_flow_array(*state)
    s.iterate(2)
    return s


@pytest.mark.parametrize("mode", ["FP64", "MIXED", "MIXED_MG", "MIXED32"])
@pytest.mark.parametrize("bc", [WALLS, XZ], ids=["walls", "xz"])
def test_the_caller_chooses_the_multigrid(ibm, mode, bc):
    case, state = _case((24, 21, 26), bc)
    count, u = {}, {}
    for key, coarsening, sweeps in (("fast", None, None), ("fast1", None, (1, 1, 1, 1, 8)),
                                    ("mg1", ibm.COARSEN_SPACING, (1, 1, 1, 1, 8)),
                                    ("mg6", ibm.COARSEN_HALVE, (6, 6, 2, 2, 16))):
        s = _solver(ibm, case, state, mode, coarsening, sweeps)
        count[key], u[key] = s.stats()["iters_p_total"], s.get_field("u1")
        s.close()
    assert count["fast"] == count["fast1"] <= 2 * 3 * (2 if mode == "MIXED" else 1), count
    assert count["mg1"] > count["mg6"] > count["fast"], count
    for key in u:
        assert rel_l2(u[key], u["fast"]) < 1e-6, (key, rel_l2(u[key], u["fast"]))


def test_the_tuner_tunes_the_multigrid_alone(ibm):
    case, state = _case((24, 21, 26), WALLS)
    s = _solver(ibm, case, state, "MIXED32", None, (2, 3, 1, 2, 7))
    ms, best = s.autotune(steps=1)
    assert ms > 0 and list(best) == [2, 3, 1, 2, 7]      # nothing to choose: the setting stays
    s.close()
    s = _solver(ibm, case, state, "MIXED32", ibm.COARSEN_SPACING, (1, 1, 1, 1, 1))
    ms, best = s.autotune(steps=1)
    assert ms > 0 and list(best) != [1, 1, 1, 1, 1]      # not among its candidates
    s.close()
