"""The pressure preconditioner is set up for the precision that runs, once, and
by whichever call needs it first (csrc/solver.cu, ready_preconditioner): the
tables of the other precision take memory only when it is chosen, and the steps
do not depend on which call came first."""
import importlib

import numpy as np
import pytest

from test_gpu_fastpoisson import WALLS, _case

pytestmark = pytest.mark.gpu

FIELDS = ("u1", "u2", "u3", "p")


def _solver(ibm, shape=(64, 60, 62)):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    case, state = _case(shape, WALLS)
    return wl.build_solver(ibm, case, tol=1e-8), state


def _step(s, state):
    s.init_flow_array(*state)
    s.iterate(2)
    return {f: s.get_field(f) for f in FIELDS}


def _equal(a, b):
    return all(np.array_equal(a[f], b[f], equal_nan=True) for f in FIELDS)


def test_tables_of_the_other_precision_on_demand(ibm):
    s, state = _solver(ibm)
    s.set_precision(ibm.MIXED32)
    mixed, small = _step(s, state), s.device_bytes()
    s.set_precision(ibm.FP64)
    # Two of the FP64 tables' three grid arrays at least (freed chunks of the
    # allocator may serve the rest).
    assert s.device_bytes() - small >= 2 * 8 * 64 * 60 * 62
    fp64 = _step(s, state)
    both = s.device_bytes()
    s.set_precision(ibm.MIXED32)
    assert _equal(_step(s, state), mixed) and s.device_bytes() == both
    s.close()
    t, _ = _solver(ibm)
    assert _equal(_step(t, state), fp64)   # no set_precision: FP64, set up with the state
    t.close()


@pytest.mark.parametrize("mode", ["FP64", "MIXED32"])
def test_steps_do_not_depend_on_the_first_call(ibm, mode):
    out = []
    for first in ("state", "time_kernel", "autotune", "bytes", "batch"):
        s, state = _solver(ibm, (20, 18, 22))
        if mode != "FP64":
            s.set_precision(getattr(ibm, mode))
        if first == "time_kernel":
            assert s.time_kernel("mg_color", reps=1)[0] > 0
        elif first == "autotune":
            s.autotune(steps=1)
        elif first == "bytes":
            assert s.device_bytes() > 0
        if first == "batch":
            b = ibm.Batch([s])
            s.init_flow_array(*state)
            b.iterate(2)
            out.append({f: s.get_field(f) for f in FIELDS})
            del b
        else:
            out.append(_step(s, state))
        s.close()
    assert all(_equal(out[0], o) for o in out[1:])
