"""The reciprocal of the tile LDL's pivots (xg_rcp.h wide_reciprocal): on the
host with the nearest and the outermost seeds within the hardware's stated error
(2^-23 of the value), and on the device, both against the correctly rounded
quotient.  The seed's error and the 24 leading bits in place of all of d leave
|e| below 2^-22 + 2^-45; the cubic step leaves e^3 < 2^-65 and the fixed point's
discarded parts 2^-59: less than 0.02 ulp beyond the rounding's half, so that
the result is within 0.52 ulp of 1/d, and at most one off the rounded quotient."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from xara_gb300 import gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _significands(n):
    rng = np.random.default_rng(5)
    m = [np.uint64(1) << np.uint64(52)]
    near = np.arange(64, dtype=np.uint64)
    step = np.uint64(1) << np.uint64(29)          # the 24th leading bit
    one, two = np.uint64(1) << np.uint64(52), np.uint64(1) << np.uint64(53)
    parts = [one + near, two - np.uint64(1) - near, one + near * step, two - (near + np.uint64(1)) * step,
             two - np.uint64(1) - near * step, one + near * step + rng.integers(0, 1 << 29, 64).astype(np.uint64),
             two - step + rng.integers(0, 1 << 29, 64).astype(np.uint64),
             rng.integers(1 << 52, 1 << 53, n).astype(np.uint64)]
    return np.concatenate([m] + parts)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    out = str(tmp_path_factory.mktemp("rcp") / "librcp_driver.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-w", "-I" + inc,
                        os.path.join(ROOT, "tests", "reciprocal", "rcp_driver.cpp"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return C.CDLL(out)


@pytest.mark.parametrize("off", [-1, 0, 1])
def test_every_allowed_seed(host, off):
    M = _significands(4000)
    rng = np.random.default_rng(8)
    be = rng.integers(1, 2045, len(M)).astype(np.uint64)
    sign = rng.integers(0, 2, len(M)).astype(np.uint64)
    d = ((sign << np.uint64(63)) | (be << np.uint64(52)) |
         (M & np.uint64((1 << 52) - 1))).view(np.float64)
    lead = (M >> np.uint64(29)).astype(np.float64) / 2.0 ** 23
    x = (1.0 / lead) * (1.0 + off * 2.0 ** -23)
    seed = x.astype(np.float32)
    if off:                              # the outermost one allowed, not beyond it
        beyond = seed < x if off < 0 else seed > x
        seed = np.where(beyond, np.nextafter(seed, np.float32(1 - off)), seed).astype(np.float32)
    seed = seed.view(np.uint32)
    y = np.zeros(len(M))
    vp = C.c_void_p
    host.reciprocals(len(M), d.ctypes.data_as(vp), seed.ctypes.data_as(vp), y.ctypes.data_as(vp))
    for k in range(len(M)):
        # y = Y 2^(e-52) against 1/d exactly, in integers: |y d - 1| in units of the result
        Y, e = int(np.frexp(abs(y[k]))[0] * 2 ** 53), int(np.frexp(abs(y[k]))[1])
        assert (y[k] < 0) == (d[k] < 0)
        x = int(M[k])                                   # |d| = x 2^(be-1075)
        s = 53 - e - (int(be[k]) - 1075)                # y d = Y x 2^-s
        err = abs(Y * x - (1 << s)) / x                 # ulps of Y
        assert err <= 0.52, (k, hex(x), off, err)


@pytest.mark.gpu
def test_on_the_device():
    M = _significands(200_000)
    rng = np.random.default_rng(9)
    be = rng.integers(1, 2045, len(M)).astype(np.uint64)
    be[:200] = np.resize([1, 2, 1022, 1023, 1024, 2043, 2044], 200)
    sign = rng.integers(0, 2, len(M)).astype(np.uint64)
    d = ((sign << np.uint64(63)) | (be << np.uint64(52)) |
         (M & np.uint64((1 << 52) - 1))).view(np.float64)
    d = np.concatenate([d, [2.0 ** -1040, -2.0 ** -1074, 2.0 ** 1023, -1.5 * 2.0 ** 1023]])
    y, yrn = np.zeros_like(d), np.zeros_like(d)
    vp = C.c_void_p
    f = gpu.lib().xg_pivot_reciprocal_check
    f.argtypes = [C.c_int, vp, vp, vp]
    assert f(d.size, d.ctypes.data_as(vp), y.ctypes.data_as(vp), yrn.ctypes.data_as(vp)) == 0
    with np.errstate(over="ignore"):
        assert np.array_equal(yrn, 1.0 / d)
    inside = np.isfinite(yrn)
    assert np.array_equal(y[~inside], yrn[~inside])
    assert (np.abs(y[inside] - yrn[inside]) <= np.spacing(np.abs(yrn[inside]))).all()
