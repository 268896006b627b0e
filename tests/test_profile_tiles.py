"""The tiled LDL' of `system ProfileSPD` (32 x 32 tiles, the trailing
products as exact digit products on the tensor cores, the substitutions over
the tiles' coupling matrices) at the sizes where a tile scheme can go wrong:
one tile and less, exact multiples of the tile edge and one more or less,
envelopes of zero, one and many tiles, decoupled tile rows, rows of widely
different magnitude, negative pivots, and entries that are not finite."""
import numpy as np
import pytest

from xara_gb300 import gpu

EPS = np.finfo(np.float64).eps


def _matrix(n, band, seed, kind):
    """L D L' with a random unit lower L of the given band: well conditioned,
    so the solution's error is the factorisation's."""
    r = np.random.default_rng(seed)
    L = np.eye(n)
    for k in range(1, min(band, n - 1) + 1):
        i = np.arange(n - k)
        L[i + k, i] = r.normal(size=n - k) * 0.4 / np.sqrt(band) * (r.random(n - k) < 0.7)
    d = r.uniform(0.5, 2.0, n)
    if kind == "indefinite":
        d[1:][r.random(n - 1) < 0.1] *= -1.0
    if kind == "blocks":                      # tile rows 0-1 decoupled from the rest
        L[64:, :64] = 0.0
    A = L @ np.diag(d) @ L.T
    A = (A + A.T) / 2
    if kind == "scaled":                      # equations in very different units
        s = 2.0 ** r.integers(-10, 30, n)
        A = A * s[:, None] * s[None, :]
    return A


def _system(A):
    m = A != 0
    np.fill_diagonal(m, True)
    rp = np.concatenate([[0], np.cumsum(m.sum(1))]).astype(np.int32)
    s = gpu.LinearSystem(rp, np.nonzero(m)[1].astype(np.int32),
                         system=gpu.XG_SYSTEM_PROFILE_SPD)
    s.add_a(A, np.arange(len(A)))
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("n,band,kind", [
    (1, 0, "plain"), (31, 5, "plain"), (32, 31, "plain"), (33, 1, "plain"), (64, 63, "plain"),
    (65, 40, "plain"), (97, 96, "indefinite"), (200, 0, "plain"), (300, 33, "blocks"),
    (350, 349, "plain"), (640, 90, "scaled"), (900, 130, "indefinite"), (1500, 300, "scaled")])
def test_solution_error(n, band, kind):
    """Energy-scaled error against a refined solution.  The computed factors
    satisfy |A - L D L'| <= 3 n u |L||D||L'| entry by entry (Higham, Accuracy
    and Stability of Numerical Algorithms, ch. 10-11; the digit products add
    less than a rounding), so the error in the scaling by sqrt(|a_ii|) is at
    most 3 n u g with g the norm of the scaled |A^-1| times |L||D||L'|."""
    A = _matrix(n, band, 3 * n + band, kind)
    sc = np.sqrt(np.abs(np.diag(A)))
    b = np.random.default_rng(n).normal(size=n) * sc
    with _system(A) as s:
        s.set_b(b)
        x, _, _ = s.solve()
        s.set_b(2.0 * b)                      # the same factors again
        x2, _, _ = s.solve()
    assert np.allclose(x2, 2.0 * x, rtol=1e-13, atol=0)
    As = A / sc[:, None] / sc[None, :]
    y = np.linalg.solve(As, b / sc).astype(np.longdouble)
    for _ in range(3):
        y += np.linalg.solve(As, np.asarray(b / sc - As.astype(np.longdouble) @ y, np.float64))
    L, D = np.eye(n), np.zeros(n)             # LDL' in plain FP64, for |L||D||L'|
    T = As.copy()
    for c in range(n):
        D[c] = T[c, c]
        L[c + 1:, c] = T[c + 1:, c] / D[c]
        T[c + 1:, c + 1:] -= np.outer(L[c + 1:, c], T[c + 1:, c])
    g = np.linalg.norm(np.abs(np.linalg.inv(As)) @ (np.abs(L) @ np.diag(np.abs(D)) @ np.abs(L).T), 2)
    err = float(np.linalg.norm(x * sc - y) / np.linalg.norm(y))
    assert err <= 3 * n * EPS * g, (err, 3 * n * EPS * g)


@pytest.mark.gpu
def test_not_finite_entries_and_pivots():
    """A NaN in the matrix leaves no finite answer behind and ends; a zero
    pivot is refused with its equation."""
    A = _matrix(200, 60, 1, "plain")
    A[150, 130] = A[130, 150] = np.nan
    with _system(A) as s:
        s.set_b(np.ones(200))
        x, _, _ = s.solve()
        assert not np.isfinite(x).all()
    A = _matrix(200, 60, 1, "plain")
    A[99, :] = A[:, 99] = 0.0
    with _system(A) as s:
        s.set_b(np.ones(200))
        with pytest.raises(gpu.XaraGpuError, match="pivot 99"):
            s.solve()
