"""The PCG's answer on systems that take hundreds to thousands of iterations: a
grid of conductances that jump between 1 and 1,000, and one 10,000 times weaker
along one axis than along the other, with the nodes' blocks of 1, 2, 3 and 6
equations.  The solver looks at b - A x in FP64 and accepts up to 1.05 of the
tolerance; its own product of a row of at most six terms is off by at most 7 u
of |A||x| + |b|, and once more that much for the sums and the scaling."""
import numpy as np
import pytest

from xara_gb300 import gpu

RTOL = 1e-12


def _grid(nx, kb, jump, weak, seed):
    rng = np.random.default_rng(seed)
    k = np.where(rng.random((nx, nx)) < 0.5, 1.0, jump)
    node = np.arange(nx * nx).reshape(nx, nx)
    pairs = [(node[:-1].ravel(), node[1:].ravel(), 2 / (1 / k[:-1] + 1 / k[1:]).ravel()),
             (node[:, :-1].ravel(), node[:, 1:].ravel(),
              weak * 2 / (1 / k[:, :-1] + 1 / k[:, 1:]).ravel())]
    i, j, c = (np.concatenate(a) for a in zip(*pairs))
    e = [[p * kb + d, q * kb + d] for p, q in zip(i, j) for d in range(kb)]
    e += [[d, -1] for d in range(nx * kb)]                      # one side held
    return nx * nx * kb, np.array(e, np.int32), np.concatenate([np.repeat(c, kb), np.ones(nx * kb)])


@pytest.mark.gpu
@pytest.mark.parametrize("nx,kb,jump,weak", [
    (60, 1, 1e3, 1.0), (60, 1, 1.0, 1e-4), (50, 2, 1.0, 1e-4), (45, 3, 1.0, 1e-4),
    (130, 3, 1.0, 1e-4), (30, 6, 1.0, 1e-4)])
def test_true_residual(nx, kb, jump, weak):
    sp = pytest.importorskip("scipy.sparse")
    n, ids, c = _grid(nx, kb, jump, weak, 3)
    held = ids[:, 1] < 0
    r, q = ids[~held, 0], ids[~held, 1]
    v, h = c[~held], ids[held, 0]
    A = sp.coo_matrix((np.concatenate([v, v, -v, -v, c[held]]),
                       (np.concatenate([r, q, r, q, h]), np.concatenate([r, q, q, r, h]))),
                      shape=(n, n)).tocsr()
    A.sort_indices()
    b = np.random.default_rng(1).normal(size=n)
    with gpu.LinearSystem(A.indptr.astype(np.int32), A.indices.astype(np.int32),
                          np.arange(0, n + 1, kb)) as s:
        for pair, w in zip(ids, c):
            s.add_a([[w, -w], [-w, w]], pair)
        s.set_b(b)
        x, it, rel = s.solve(rtol=RTOL, maxit=20000)
    M, res = A.tocoo(), b.astype(np.longdouble)
    np.subtract.at(res, M.row, M.data.astype(np.longdouble) * x[M.col].astype(np.longdouble))
    u = np.finfo(np.float64).eps / 2
    own = 14 * u * np.linalg.norm(abs(A) @ np.abs(x) + np.abs(b))
    assert rel <= RTOL
    assert np.linalg.norm(res.astype(np.float64)) <= 1.05 * RTOL * np.linalg.norm(b) + own


@pytest.mark.gpu
def test_the_iteration_limit_holds():
    n, ids, c = _grid(60, 1, 1e3, 1.0, 3)
    sp = pytest.importorskip("scipy.sparse")
    r = np.concatenate([ids[:, 0], ids[ids[:, 1] >= 0, 1], ids[ids[:, 1] >= 0, 0], ids[ids[:, 1] >= 0, 1]])
    q = np.concatenate([ids[:, 0], ids[ids[:, 1] >= 0, 1], ids[ids[:, 1] >= 0, 1], ids[ids[:, 1] >= 0, 0]])
    P = sp.coo_matrix((np.ones(len(r)), (r, q)), shape=(n, n)).tocsr()
    P.sort_indices()
    b = np.random.default_rng(1).normal(size=n)
    with gpu.LinearSystem(P.indptr.astype(np.int32), P.indices.astype(np.int32),
                          np.arange(n + 1)) as s:
        for pair, w in zip(ids, c):
            s.add_a([[w, -w], [-w, w]], pair)
        s.set_b(b)
        full = s.solve(rtol=RTOL, maxit=20000)[1]
        # cut off between the first convergence and the last: still the answer
        assert s.solve(rtol=RTOL, maxit=full - 20)[1] == full - 20
        with pytest.raises(gpu.XaraGpuError):
            s.solve(rtol=RTOL, maxit=1000)


@pytest.mark.gpu
@pytest.mark.parametrize("kb", [1, 3])
@pytest.mark.parametrize("size", [1e-148, 1e-140, 1e140, 1e150])
def test_loads_at_the_ends_of_the_range(kb, size):
    """r.z and p.q of such loads have no normal reciprocal (they are subnormal at
    the end of the smallest ones' solve, above 2^1022 at the start of the
    largest's), but their quotients are ordinary numbers.  The squares of the smallest
    residuals resolve r to 2^-537, 1e-14 of b."""
    sp = pytest.importorskip("scipy.sparse")
    n, ids, c = _grid(12, kb, 1.0, 1.0, 3)
    a = [([[w, -w], [-w, w]], p) for p, w in zip(ids, c)] + [([[0.3]], [k]) for k in range(n)]
    A = np.zeros((n, n))
    for m, p in a:
        for i, r in enumerate(p):
            for j, q in enumerate(p):
                if r >= 0 and q >= 0:
                    A[r, q] += m[i][j]
    P = sp.csr_matrix(A != 0)
    P.sort_indices()
    b = np.random.default_rng(2).normal(size=n)
    with gpu.LinearSystem(P.indptr.astype(np.int32), P.indices.astype(np.int32),
                          np.arange(0, n + 1, kb)) as s:
        for m, p in a:
            s.add_a(m, p)
        s.set_b(b * size)
        x = s.solve(rtol=RTOL, maxit=2000)[0] / size
    assert np.linalg.norm(b - A @ x) <= 2 * RTOL * np.linalg.norm(b)
