"""`system ProfileSPD` on models of several disconnected parts (a band each):
frames from the narrowest band to the widest the band kernels take, where the
rows held in registers and the entries per thread change, next to a tiny
part, against dense solves and against the same frame run alone."""
import numpy as np
import pytest

from xara_gb300 import configs
from xara_gb300._abi import ModelDesc

EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def gpu_mod(need_gpu):
    from xara_gb300 import gpu
    gpu.lib()
    return gpu


def _two_frames(d1, d2):
    """Both frames in one model, the second one's tags behind the first's."""
    a, b = d1.arrays, d2.arrays
    nn, ne, nu = len(a["node_tag"]), len(a["elem_tag"]), len(a["uni_type"])
    ns, nf = len(a["sec_fiber_start"]) - 1, int(a["sec_fiber_start"][-1])
    off = dict(node_tag=nn, elem_tag=ne, elem_conn=nn, elem_mat=ns, fib_mat=nu, sp_node=nn,
               load_node=nn)
    kw = {}
    for k, v in a.items():
        if v is None:
            continue
        w = b[k] + off.get(k, 0)
        kw[k] = np.concatenate([v, (b[k][1:] + nf) if k == "sec_fiber_start" else w])
    return ModelDesc(ndm=2, ndf=3, elem_type=d1.elem_type, geom_transf=d1.geom_transf,
                     fbc_num_ip=d1.fbc_num_ip, **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("bays,stories", [(1, 1), (2, 6), (5, 9), (6, 8), (7, 9), (8, 30), (10, 12),
                                          (12, 20), (13, 15), (16, 18), (18, 19), (20, 22),
                                          (23, 24)])
def test_solve_two_parts(gpu_mod, bays, stories):
    """A frame of bays x stories beside a one-bay frame: the solution of its
    yielded tangent, factored with its right-hand side and again with the
    factors kept, within 3 n u |A^-1||L||D||L'| of a refined dense one (the
    scaling by sqrt(a_ii); Higham, Accuracy and Stability, ch. 10)."""
    big, _ = configs.steel_frame_2d(bays, stories, nfib=8)
    small, _ = configs.steel_frame_2d(1, 2, nfib=8)
    with gpu_mod.DeviceModel(_two_frames(big, small)) as m:
        u = np.random.default_rng(bays).normal(size=m.nu) * 2e-3
        u.reshape(-1, 3)[:, 0] += 0.01
        m.set_trial_disp(u)
        vals, _, _ = m.update()
        rp, ci = m.pattern()
        A = np.zeros((m.neq, m.neq))
        A[np.repeat(np.arange(m.neq), np.diff(rp)), ci] = vals
        sc = np.sqrt(np.abs(np.diag(A)))
        b = np.random.default_rng(1).normal(size=m.neq) * sc
        x, _, _ = m.solve(b)
        x2, _, _ = m.solve(2.0 * b)
    As = A / sc[:, None] / sc[None, :]
    y = np.linalg.solve(As, b / sc).astype(np.longdouble)
    for _ in range(4):
        y += np.linalg.solve(As, np.asarray(b / sc - As.astype(np.longdouble) @ y, np.float64))
    n = len(A)
    L, D, T = np.eye(n), np.zeros(n), As.copy()
    for c in range(n):
        D[c] = T[c, c]
        r = np.nonzero(T[c + 1:, c])[0] + c + 1
        L[r, c] = T[r, c] / D[c]
        T[np.ix_(r, r)] -= np.outer(L[r, c], T[r, c])
    g = np.linalg.norm(np.abs(np.linalg.inv(As)) @ (np.abs(L) @ np.diag(np.abs(D)) @ np.abs(L).T), 2)
    for xx, f in ((x, 1.0), (x2, 2.0)):
        err = float(np.linalg.norm(xx * sc / f - y) / np.linalg.norm(y))
        assert err <= 3 * n * EPS * g, (err, 3 * n * EPS * g)


@pytest.mark.gpu
@pytest.mark.parametrize("bays,stories", [(2, 3), (9, 10)])
def test_pushover_beside_another_part(gpu_mod, bays, stories):
    """DisplacementControl solves two right-hand sides with one factorisation:
    the pushed frame's history equals its run alone."""
    d1, ph = configs.steel_frame_2d(bays, stories, steps=6, grav_steps=2, nfib=8)
    d2, _ = configs.steel_frame_2d(1, 1, nfib=8)
    with gpu_mod.DeviceModel(d1) as m:
        u1, l1, s1 = m.run(ph)
    with gpu_mod.DeviceModel(_two_frames(d1, d2)) as m:
        u2, l2, s2 = m.run(ph)
    n = u1.shape[1]
    assert np.linalg.norm(u2[:, :n] - u1) / np.linalg.norm(u1) < 1e-8
    assert np.linalg.norm(l2[:2] - l1[:2]) / np.linalg.norm(l1[:2]) < 1e-8
