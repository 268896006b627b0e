"""The tiled LDL' on weakly coupled parts: tile rows 2 and 3 hang on different
halves of tile 0's equations and meet only through couplings of delta, so that
the fill between them is delta of the rows' sizes and row 3's answer to a load on
row 2 is nothing but that fill.  It has to come out to a relative accuracy of its
own, as the plain FP64 products give it, however small delta is."""
import numpy as np
import pytest

from test_profile_tiles import EPS, _system

T = 32


def _matrix(delta, scale, seed):
    r = np.random.default_rng(seed)
    A = np.zeros((4 * T, 4 * T))
    two, three = slice(2 * T, 3 * T), slice(3 * T, 4 * T)
    for rows, cols, w in ((two, slice(0, 16), 0.2), (two, slice(16, 32), 0.2 * delta),
                          (three, slice(16, 32), 0.2), (three, slice(0, 16), 0.2 * delta)):
        m = r.normal(size=(T, 16)) * w
        A[rows, cols] = m
        A[cols, rows] = m.T
    A[np.diag_indices(4 * T)] = 4.0 + r.random(4 * T)
    s = np.ones(4 * T)
    if scale:
        s = 2.0 ** r.integers(-20, 20, 4 * T)
    return A * s[:, None] * s[None, :], s


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [False, True])
@pytest.mark.parametrize("delta", [1.0, 1e-4, 1e-7, 1e-9, 1e-12, 1e-16, 1e-24, 1e-40])
def test_small_fill_keeps_its_digits(delta, scale):
    """With S the Schur complement of tile 0 (in the unscaled matrix), x3 =
    -S33^-1 S32 x2.  Each entry of a product or factor is off by at most 3 n u
    of the sum of its terms' magnitudes, so x3 is off by at most 3 n u times
    |S33^-1| (|P3||L2|' |x2| + |S33||x3|), and by what x2's own error, 3 n u
    |S22^-1||S22||x2|, passes on."""
    A, s = _matrix(delta, scale, 3)
    n, two, three = len(A), slice(2 * T, 3 * T), slice(3 * T, 4 * T)
    b = np.zeros(n)
    b[two] = np.random.default_rng(4).normal(size=T)
    with _system(A) as h:
        h.set_b(b * s)
        x = h.solve()[0] * s
    M, y = (A / s[:, None] / s[None, :]).astype(np.longdouble), b.astype(np.longdouble)
    S = None
    for k in range(n):
        if k == T:
            S = M.astype(np.float64)
        f = M[k + 1:, k] / M[k, k]
        M[k + 1:] -= np.outer(f, M[k])
        y[k + 1:] -= f * y[k]
    e = np.zeros(n, np.longdouble)
    for k in range(n - 1, -1, -1):
        e[k] = (y[k] - M[k, k + 1:] @ e[k + 1:]) / M[k, k]
    a2, a3 = np.abs(e[two]).astype(float), np.abs(e[three]).astype(float)
    U = (A / s[:, None] / s[None, :])
    i0 = np.abs(np.linalg.inv(U[:T, :T]))
    S32 = np.abs(U[three, :T]) @ i0 @ np.abs(U[:T, two])
    i3, i2 = np.abs(np.linalg.inv(S[three, three])), np.abs(np.linalg.inv(S[two, two]))
    g = i3 @ (S32 @ a2 + np.abs(S[three, three]) @ a3) + i3 @ S32 @ (i2 @ np.abs(S[two, two]) @ a2)
    err = np.abs(x[three] - e[three]).astype(float).max()
    assert err <= 3 * n * EPS / 2 * g.max(), (err / a3.max(), 1.5 * n * EPS * g.max() / a3.max())
