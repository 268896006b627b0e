"""The LDL's row blocks over their assignment: a row far longer than the others
(a constraint's), several of them, tile rows without a neighbour, an envelope of
exactly 28 rows below the diagonal tile (every row keeps its blocks) and of 29
(only the two next to it do).  The error bound is that of
test_profile_tiles.test_solution_error."""
import numpy as np
import pytest

from test_profile_tiles import EPS, _system


def _matrix(n, band, rows, seed):
    r = np.random.default_rng(seed)
    L = np.eye(n)
    for k in range(1, min(band, n - 1) + 1):
        i = np.arange(n - k)
        L[i + k, i] = r.normal(size=n - k) * 0.4 / np.sqrt(band) * (r.random(n - k) < 0.7)
    for i, first in rows:
        L[i, first:i] = r.normal(size=i - first) * 0.4 / np.sqrt(i - first)
    d = r.uniform(0.5, 2.0, n)
    A = L @ np.diag(d) @ L.T
    return (A + A.T) / 2


@pytest.mark.gpu
@pytest.mark.parametrize("n,band,rows", [
    (700, 40, [(500, 3)]), (700, 33, [(699, 0), (350, 40), (351, 41), (600, 320)]),
    (640, 10, [(300, 0), (639, 64)]), (29 * 32, 29 * 32 - 1, []), (29 * 32 + 1, 29 * 32, []),
    (1300, 960, [(1290, 5)])])
def test_row_blocks(n, band, rows):
    A = _matrix(n, band, rows, n + band)
    sc = np.sqrt(np.abs(np.diag(A)))
    b = np.random.default_rng(n).normal(size=n) * sc
    with _system(A) as s:
        s.set_b(b)
        x = s.solve()[0]
        again = s.solve()[0]
    assert (x == again).all()
    As = A / sc[:, None] / sc[None, :]
    y = np.linalg.solve(As, b / sc).astype(np.longdouble)
    for _ in range(3):
        y += np.linalg.solve(As, np.asarray(b / sc - As.astype(np.longdouble) @ y, np.float64))
    L, D, M = np.eye(n), np.zeros(n), As.copy()
    for k in range(n):
        D[k] = M[k, k]
        L[k + 1:, k] = M[k + 1:, k] / D[k]
        M[k + 1:, k + 1:] -= np.outer(L[k + 1:, k], M[k, k + 1:])
    g = np.linalg.norm(np.abs(np.linalg.inv(As)) @ (np.abs(L) * np.abs(D)) @ np.abs(L).T, np.inf)
    err = float(np.max(np.abs(x * sc - y)) / np.max(np.abs(y)))
    assert err <= 3 * n * EPS / 2 * g
