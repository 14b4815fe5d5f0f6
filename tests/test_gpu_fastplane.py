"""The slice kernels of the FP32 fast diagonalisation (csrc/fastplane.cuh): a
slice's rows and z lines up to the tile (32 rows of either parity by 64
columns) and past it, where the general kernels take over, mirror-symmetric
(wrapped axes here) or not, rows along y and along x, and slices next to a
body.

The FP64 mode takes the general transforms, so its fields are the reference.
The preconditioner is the rows' inverse up to FP32 rounding, and an iteration
applies it twice: without a body a solve to 1e-8 takes at most three
iterations, and the fields agree to that tolerance times the pressure's loss
of three digits; with a body both modes stop at 1e-9 and the fields agree to
1e-6."""
import importlib

import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_fastpoisson import OPEN, WALLS, XY, XZ, VP, Y, _case, _run

pytestmark = pytest.mark.gpu

SHAPES = [
    # rows along y: 32 | 33 unfolded, 63 | 64 | 65 folded
    ((33, 32, 64), WALLS), ((34, 33, 64), WALLS), ((65, 31, 16), OPEN), ((66, 65, 12), WALLS), ((12, 64, 31), Y),
    ((11, 65, 32), Y), ((10, 63, 33), Y), ((9, 128, 20), Y),
    # z: 64 | 65 unfolded, 63 | 64 | 65 | 128 folded
    ((14, 12, 65), WALLS), ((13, 12, 64), WALLS), ((13, 12, 128), WALLS), ((12, 10, 64), VP), ((12, 10, 3), VP),
    # rows along x (x wraps), and all three axes transformed
    ((64, 70, 63), XZ), ((128, 9, 128), XZ), ((63, 9, 65), XZ), ((64, 9, 64), XZ), ((40, 64, 9), XY), ((6, 33, 40), XY),
]


@pytest.mark.parametrize("shape,bc", SHAPES, ids=["x".join(map(str, s[0])) for s in SHAPES])
def test_slices_match_the_general_transforms(ibm, shape, bc):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    case, state = _case(shape, bc)
    ref, _ = _run(ibm, wl, case, state, "FP64", 1e-12)
    for mode in ("MIXED_MG", "MIXED"):
        out, st = _run(ibm, wl, case, state, mode, 1e-8)
        assert st["iters_p_total"] <= 2 * 3, (mode, st["iters_p_total"])
        for f, a in out.items():
            assert rel_l2(a, ref[f]) < 1e-5, (mode, f, rel_l2(a, ref[f]))


@pytest.mark.parametrize("shape", [(40, 24, 24), (48, 70, 40)])
def test_slices_beside_a_body(ibm, shape):
    wl = importlib.import_module("2020researchproject_gb300.workloads")
    case = wl.sphere(*shape, subdivisions=3)
    state = wl.initial_state(case)
    ref, _ = _run(ibm, wl, case, state, "FP64", 1e-12)
    out, st = _run(ibm, wl, case, state, "MIXED_MG", 1e-9)
    assert st["iters_p_total"] <= 2 * 12, st["iters_p_total"]
    for f, a in out.items():
        assert np.array_equal(np.isnan(a), np.isnan(ref[f]))
        assert rel_l2(a, ref[f]) < 1e-6, (f, rel_l2(a, ref[f]))
