"""Which preconditioner serves a body (csrc/fastpoisson.h, FP_NEAR;
csrc/solver.cu, kBodyOps).  A caller who sets the default coarsening has the
multigrid, so a solver left to itself takes bitwise the same steps exactly where
the rule picks the multigrid: near cells past FP_NEAR of the fluid ones on a
large enough grid, FP64 transforms past kBodyOps."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E = 0.013


def _duct(tmp_path):
    """A square duct along x in a block that fills the rest of the domain."""
    geo = importlib.import_module("2020researchproject_gb300.geometry")
    v, f = geo.box_union([((-1, -1, -1), (4, 2, 2))])
    w, g = geo.box_union([((-0.5, 0.28 + E, 0.26 + E), (3.5, 0.71 + E, 0.73 + E))])
    path = str(tmp_path / "duct.stl")
    geo.write_stl(path, np.vstack([v, w]), np.vstack([f, np.asarray(g)[:, ::-1] + len(v)]))
    return path


def _case(shape, body, tmp_path):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    if body == "sphere":
        return wl.sphere(*shape, subdivisions=3)
    stl = _duct(tmp_path)
    if body == "box":
        boxes = [((0.7 + E, 0.35 + E, 0.35 + E), (1.0 + E, 0.65 + E, 0.65 + E))]
        stl = wl._body_stl("boxes", dict(boxes=boxes), ("boxes", "rule"))
    x, y, z = (np.linspace(0, size, n + 1) for size, n in zip((2, 1, 1), shape))
    return dict(xf=x, yf=y, zf=z, re=200.0, dt=0.05 / shape[1], stl=stl, init=(1.0, 0.0, 0.0, 0.0),
                bc=["W vel 1 0 0", "E press 0", "S slip", "N slip", "D slip", "U slip"])


@pytest.mark.parametrize("shape,body,mode,multigrid", [
    ((72, 48, 48), "duct", "FP64", True), ((48, 32, 32), "duct", "FP64", False), ((72, 48, 48), "box", "FP64", False),
    ((72, 48, 48), "duct", "MIXED32", False), ((122, 72, 72), "duct", "MIXED32", True),
    ((122, 72, 72), "box", "MIXED32", False), ((136, 100, 100), "sphere", "FP64", True),
    ((112, 88, 88), "sphere", "FP64", False), ((136, 100, 100), "sphere", "MIXED32", False)], ids=str)
def test_rule(ibm, tmp_path, shape, body, mode, multigrid):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    case = _case(shape, body, tmp_path)
    out = []
    for coarsening in (None, ibm.COARSEN_SPACING):
        s = wl.build_solver(ibm, case, tol=1e-8, coarsening=coarsening)
        s.set_precision(getattr(ibm, mode))
        s.init_flow_array(*wl.initial_state(case))
        s.iterate(2)
        out.append({f: s.get_field(f) for f in ("u1", "p")})
        s.close()
    assert all(np.array_equal(out[0][f], out[1][f], equal_nan=True) for f in out[0]) == multigrid
