"""The PCG's matrix stream (xg_block_stream.h) on the host, with bulk copies
that arrive when they are waited for: every group comes in its order, pass
after pass, and a copy that never comes ends the stream -- no record is read
from its stage, no second wait, no stage filled while a copy to it is on its
way -- with the copies in flight waited for before the block ends."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def stream(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    out = str(tmp_path_factory.mktemp("stream") / "libstream_driver.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-w", "-I" + inc,
                        os.path.join(ROOT, "tests", "block_stream", "stream_driver.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return C.CDLL(out)


@pytest.mark.parametrize("kb,sp,one", [(1, 1, 0), (1, 8, 1), (2, 1, 0), (2, 4, 1), (3, 1, 0),
                                       (3, 2, 1), (3, 8, 1), (6, 1, 0), (6, 4, 1)])
def test_stream(stream, kb, sp, one):
    for seed in range(8):
        ns, stride = (1, 1) if one else (1 + seed % 7, 1 + seed % 3)
        for lose in [-1, 0, 1, 2, 3, 4, 5, 6, 9, 14, 23, 40]:
            assert stream.stream_errors(kb, sp, one, ns, stride, 4, lose, seed) == 0, (seed, lose)
