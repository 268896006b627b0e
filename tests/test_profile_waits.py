"""The LDL's waits between blocks: the limit is for one hand-off, however long the
factorisation is.  An envelope of 4,000 tile columns, one neighbour each, that
ends in twelve full tile rows leaves the row blocks of the last ones idle from
the launch on, for the 35 ms and more that the columns before take one after
another (9 us at least each), four times the limit given."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from xara_gb300 import gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_idle_row_blocks_outlast_the_limit(tmp_path):
    sp = pytest.importorskip("scipy.sparse")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    out = str(tmp_path / "libwaits_driver.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-w",
                        "-I" + os.path.join(cuda, "include"),
                        os.path.join(ROOT, "tests", "profile_waits", "waits_driver.cpp"), "-o", out,
                        gpu.LIB, "-L" + os.path.join(cuda, "lib64"), "-lcudart",
                        "-Wl,-rpath," + os.path.dirname(gpu.LIB)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    gpu.lib()
    n, full = 4000 * 32, 12 * 32
    e = np.full(full, 1e-3)
    A = sp.diags([np.full(n, 4.0), np.full(n - 1, 1.0), np.full(n - 1, 1.0)], [0, 1, -1]).tocsr()
    A = (A + sp.block_diag([sp.csr_matrix((n - full, n - full)),
                            sp.csr_matrix(np.outer(e, e) + 1e-3)])).tocsr()
    A.sort_indices()
    b = np.random.default_rng(3).normal(size=n)
    x = np.zeros(n)
    vp = C.c_void_p
    args = [np.ascontiguousarray(a) for a in (A.indptr.astype(np.int32), A.indices.astype(np.int32),
                                              A.data, b)]
    f = C.CDLL(out).solve_with_limit
    f.argtypes = [C.c_int, vp, vp, vp, vp, vp, C.c_double]
    assert f(n, *[a.ctypes.data_as(vp) for a in args], x.ctypes.data_as(vp), 8.0) == 0
    assert np.linalg.norm(b - A @ x) <= 1e-13 * np.linalg.norm(b)
