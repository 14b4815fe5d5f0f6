"""reduce_partials (csrc/common.cuh) against sums and maxima on the host, exact in
any order, from one block to many more than one warp folds at once."""
import importlib
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_sums_and_maxima(tmp_path):
    build = importlib.import_module("2020researchproject_gb300.build")
    exe = str(tmp_path / "reduce_driver")
    src = os.path.join(ROOT, "tests", "drivers", "reduce_driver.cu")
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-o", exe, src], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "equal\n", r.stdout + r.stderr
