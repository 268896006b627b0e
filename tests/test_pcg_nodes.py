"""The PCG on the node-block copy over its dispatch: block orders 1, 2, 3
and 6, from one slice of 32 nodes with eight warps on it to more slices than
the device has warps (vectors in memory), ragged last slices, nodes with fewer
equations than the order, a node tied to more than 96 others (rows in chunks)
and one whose values leave the float split's range (rows in FP64).  The true
residual is taken in double precision on the host.

Tolerance: the solver stops at a recursive residual of 1e-12 |b|; the
true one differs by the products' error, 2^-46 of |A||x| an iteration, with
|A||x| below 50 |b| (diagonally dominant, condition below 50) and some 40
iterations at most: 1.4e-14 * 50 * sqrt(40) = 4.5e-12.  The bound is 1e-11."""
import numpy as np
import pytest

from xara_gb300 import gpu


def _system(kb, nnode, seed, long_node=False, tiny=False):
    sp = pytest.importorskip("scipy.sparse")
    rng = np.random.default_rng(seed)
    m = np.full(nnode, kb)
    if kb > 1:
        m[rng.random(nnode) < 0.1] = kb - 1
        m[nnode // 2] = kb
    blk = np.concatenate([[0], np.cumsum(m)]).astype(np.int32)
    pairs = [(i, i + off) for off in (1, 37) for i in range(0, nnode - off)]
    if long_node:
        pairs += [(2, j) for j in range(50, 50 + 150)]
    elems, r, c, v = [], [], [], []
    for i, j in pairs:
        ids = np.concatenate([np.arange(blk[i], blk[i + 1]), np.arange(blk[j], blk[j + 1])])
        a = rng.uniform(-0.3, 0.3, (len(ids), len(ids))) / kb
        a = a + a.T
        if tiny and i == 3:
            a[m[i]:, :m[i]] *= 1e-18
            a[:m[i], m[i]:] *= 1e-18
        a[np.diag_indices(len(ids))] = 1.0 + rng.random(len(ids))
        elems.append((np.ascontiguousarray(a), ids.astype(np.int32)))
        r.append(np.repeat(ids, len(ids)))
        c.append(np.tile(ids, len(ids)))
        v.append(a.ravel())
    n = int(blk[-1])
    r.append(np.arange(n)); c.append(np.arange(n)); v.append(np.ones(n))
    elems += [(np.eye(m[i]), np.arange(blk[i], blk[i + 1], dtype=np.int32)) for i in range(nnode)]
    A = sp.coo_matrix((np.concatenate(v), (np.concatenate(r), np.concatenate(c))),
                      shape=(n, n)).tocsr()
    A.sort_indices()
    return n, blk, elems, A


@pytest.mark.gpu
@pytest.mark.parametrize("kb,nnode,long_node,tiny", [
    (1, 5, False, False), (1, 300, True, True), (1, 40000, False, False),
    (1, 78000, False, False),
    (2, 33, False, False), (2, 9800, True, False), (2, 20000, False, False),
    (3, 2, False, False), (3, 64, False, True), (3, 1000, True, True), (3, 9800, False, False),
    (3, 20000, True, False), (3, 39000, False, False), (3, 78000, True, True),
    (6, 100, False, False), (6, 250, True, True), (6, 5000, False, False),
    (6, 10000, False, True), (6, 19500, True, False)])
def test_node_block_pcg_residual(kb, nnode, long_node, tiny):
    n, blk, elems, A = _system(kb, nnode, kb * 1000 + nnode, long_node, tiny)
    b = np.random.default_rng(n).normal(size=n)
    with gpu.LinearSystem(A.indptr.astype(np.int32), A.indices.astype(np.int32), blk) as s:
        for a, ids in elems:
            s.add_a(a, ids)
        s.set_b(b)
        x = np.array(s.solve(rtol=1e-12, maxit=2000)[0])
        again = np.array(s.solve(rtol=1e-12, maxit=2000)[0])
    assert np.linalg.norm(b - A @ x) <= 1e-11 * np.linalg.norm(b)
    assert (x == again).all()
