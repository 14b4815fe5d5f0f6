"""A momentum solve whose right-hand side is zero (csrc/momsweep.h): the first
sweep ends it.  Recorded steps launch the sweeps that stand before the loop all
the same, and none of them may touch u*: the second buffer still holds an
earlier solve's iterate.  A box between resting walls marches, is reset to rest
and takes one step: u* is zero at every cell, ghosts beside ghosts included,
with graphs on and off."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALLS = [f"{s} wall" for s in "WESNDU"]


@pytest.mark.parametrize("graphs", [True, False], ids=["graphs", "host"])
@pytest.mark.parametrize("mode", ["FP64", "MIXED", "MIXED32"])
def test_rest_after_motion(ibm, mode, graphs):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    lo, hi = (0.31, 0.33, 0.28), (0.68, 0.71, 0.63)
    stl = wl._body_stl("boxes", dict(boxes=[(lo, hi)]), ("boxes", "momsweep", lo, hi))
    n = (22, 20, 24)
    case = dict(xf=np.linspace(0, 1, n[0] + 1), yf=np.linspace(0, 1, n[1] + 1), zf=np.linspace(0, 1, n[2] + 1),
                re=150.0, dt=1e-3, bc=WALLS, stl=stl)
    s = wl.build_solver(ibm, case, tol=1e-10)
    s.set_precision(getattr(ibm, mode))
    s.set_graphs(graphs)
    pad = tuple(q + 4 for q in n)
    rng = np.random.default_rng(5)
    zero = np.zeros(pad)
    s.init_flow_array(*[0.5 * rng.standard_normal(pad) for _ in range(3)], zero)
    s.iterate(2)
    assert max(np.abs(s.get_field(f"u{l}star")).max() for l in (1, 2, 3)) > 0.1
    s.init_flow_array(zero, zero, zero, zero)
    s.iterate(1)
    for l in (1, 2, 3):
        assert not np.any(np.nan_to_num(s.get_field(f"u{l}star"))), (mode, graphs, l)
    assert max(s.stats()["iters_u"]) == 0
    s.close()
