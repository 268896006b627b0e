"""The autotuner's four candidates are four different grids of the PCG for every
block order, below the device's block count.  On the host."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from xara_gb300 import gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    if not os.path.exists(gpu.LIB):
        pytest.skip("libxara_gpu.so not built")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = str(tmp_path_factory.mktemp("shapes") / "libshapes_driver.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-w", "-I" + inc,
                        os.path.join(ROOT, "tests", "launch_shapes", "shapes_driver.cpp"), "-o", out,
                        gpu.LIB, "-Wl,-rpath," + os.path.dirname(gpu.LIB)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return C.CDLL(out)


@pytest.mark.parametrize("kb", [0, 1, 2, 3, 6])
def test_pcg_grids(shapes, kb):
    nodes = 3000
    n = nodes * max(kb, 1)
    grids = [shapes.grid_of(n, nodes, kb, r, 152) for r in (32, 64, 128, 256)]
    assert grids == [-(-3000 // r) for r in (32, 64, 128, 256)]
    assert shapes.grid_of(n, nodes, kb, 0, 152) == (47 if kb == 0 else 94)
    assert shapes.grid_of(40 * n, 40 * nodes, kb, 32, 152) == 152
