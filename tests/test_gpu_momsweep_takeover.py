"""Momentum sweeps that reach their limit hand the solve to BiCGSTAB
(csrc/momsweep.h), which has IBMSolver_set_max_iters' cap for itself.

Equal cells with sum k = 2/3: a sweep gains a factor 0.4, so a cap of 20 leaves
1e-8 of the residual where the solves stop at 1e-12.  BiCGSTAB from there needs
a handful of iterations (condition 2.3: a factor of 20 each), so it stays far
below the cap; the step ends converged, its count past the sweeps', and equal
to the uncapped one to the tolerance times the condition.  In FP32 a cap of 6
leaves 4e-3; the residual of a row is rounded to some 5e-7 of it, so the solve
is asked for 1e-5 and the fields are only compared between the two paths.
Recorded and host-sequenced steps agree bit for bit."""
import importlib

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

FIELDS = ("u1", "u2", "u3", "p", "u1star", "u2star", "u3star")


def _run(ibm, mode, tol, cap, graphs, dt, re):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    n = (16, 14, 18)
    case = dict(xf=np.arange(n[0] + 1) / 16, yf=np.arange(n[1] + 1) / 16, zf=np.arange(n[2] + 1) / 16, re=re, dt=dt,
                bc=["W wall", "E wall", "S wall", "N wall", "D wall", "U vel 1 0 0"])
    s = wl.build_solver(ibm, case, tol=tol)
    s.set_precision(getattr(ibm, mode))
    s.set_graphs(graphs)
    if cap:
        s.set_max_iters(cap, 1000)
    rng = np.random.default_rng(1)
    s.init_flow_array(*[0.3 * rng.standard_normal(tuple(q + 4 for q in n)) for _ in range(3)],
                      np.zeros(tuple(q + 4 for q in n)))
    s.iterate(2)
    out, st = {f: s.get_field(f) for f in FIELDS}, s.stats()
    s.close()
    return out, st


@pytest.mark.parametrize("mode,tol,cap", [("FP64", 1e-12, 20), ("MIXED", 1e-12, 20), ("MIXED32", 1e-5, 6)],
                         ids=["FP64", "MIXED", "MIXED32"])
def test_bicgstab_takes_over_with_its_own_cap(ibm, capfd, mode, tol, cap):
    dt = 2.0 * 10.0 / 16 ** 2 / 9
    ref, _ = _run(ibm, mode, tol, 0, True, dt, 10.0)
    out, st = _run(ibm, mode, tol, cap, True, dt, 10.0)
    host, sh = _run(ibm, mode, tol, cap, False, dt, 10.0)
    assert "did not converge" not in capfd.readouterr().err
    assert max(st["res_u"]) < tol and min(st["iters_u"]) > cap and max(st["iters_u"]) <= 2 * cap
    assert st["iters_u"] == sh["iters_u"]
    for f in FIELDS:
        assert np.array_equal(out[f], host[f], equal_nan=True), f
        if mode != "MIXED32" and f != "p":
            assert rel_l2(out[f], ref[f]) < 1e-9, (f, rel_l2(out[f], ref[f]))


def test_large_diffusion_numbers_go_to_bicgstab_at_once(ibm):
    """sum k = 7.7: a sweep would gain 12 %, so any count from sweeps is past
    their limit of 60."""
    _, st = _run(ibm, "FP64", 1e-7, 0, True, 1e-2, 1.0)
    assert max(st["res_u"]) < 1e-7 and max(st["iters_u"]) < 60
