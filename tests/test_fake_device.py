"""The host side of the solvers on devices that are not at hand, under a stand-in
for the CUDA runtime (fake_cuda/fake_cuda.c: nothing is run, launches are accepted
or refused as a device would).  In child processes on the CPU."""
import os
import subprocess
import sys
import textwrap

import pytest

from xara_gb300 import gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SETUP = """
import ctypes as C
import numpy as np
from xara_gb300 import gpu
def solve(n, band, system):
    i, j = np.nonzero(np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= band)
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    with gpu.LinearSystem(rp, j.astype(np.int32), system=system) as s:
        s.add_a(np.eye(n), np.arange(n))
        s.set_b(np.ones(n))
        s.solve(maxit=1)
def code(*a):
    try:
        solve(*a)
        return 0, ""
    except gpu.XaraGpuError as e:
        return e.code, str(e)
LDL, PCG = gpu.XG_SYSTEM_PROFILE_SPD, gpu.XG_SYSTEM_BJPCG
gpu.lib()
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not os.path.exists(gpu.LIB):
        pytest.skip("libxara_gpu.so not built")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cuda.so")
    r = subprocess.run(["gcc", "-O1", "-fPIC", "-shared", "-w", "-o", so,
                        os.path.join(HERE, "fake_cuda", "fake_cuda.c")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def child(code, **env):
        r = subprocess.run([sys.executable, "-c", SETUP + textwrap.dedent(code)], text=True,
                           capture_output=True, timeout=120, cwd=os.path.dirname(HERE),
                           env=dict(os.environ, LD_PRELOAD=so, **{k: str(v) for k, v in env.items()}))
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout
    return child


def test_each_device_gets_its_attributes(run):
    """A second device of the process has none of the first one's attributes."""
    run("""
        rt = C.CDLL(None)
        for dev in (0, 1, 0):
            rt.cudaSetDevice(dev)
            assert code(300, 40, LDL) == (0, ""), code(300, 40, LDL)
    """)


@pytest.mark.parametrize("sms", [8, 9, 12, 20, 59, 60, 132])
def test_small_devices_factor_too(run, sms):
    """One block a SM and one at least for the list, whatever the envelope: one
    tile, one neighbour, 25 and 29 tile rows below the diagonal, a long row's."""
    run(f"""
        for n, band in ((20, 5), (300, 20), (1000, 24 * 32), (1000, 29 * 32), (1000, 999)):
            assert code(n, band, LDL) == (0, ""), (n, band, code(n, band, LDL))
    """, FAKE_SMS=sms)


def test_too_small_a_device_is_named(run):
    run("""
        c, text = code(300, 100, LDL)
        assert c < 0 and "needs 8 SMs" in text and "has 7" in text, (c, text)
    """, FAKE_SMS=7)


@pytest.mark.parametrize("system,launch", [("LDL", 1), ("LDL", 2), ("PCG", 1)])
def test_a_refused_launch_is_no_failed_solve(run, system, launch):
    """XG_ECUDA (-2) with its own text, not XG_ESOLVE (-4) or a wait that timed out."""
    run(f"""
        c, text = code(300, 40, {system})
        assert c == -2 and "timed out" not in text and "pivot" not in text, (c, text)
        assert "CUDA" in text, text
    """, FAKE_REFUSE=launch)
