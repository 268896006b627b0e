"""The work this framework is measured on: what its users have it do, through
the Python layer of the C ABI, from the smallest model to the largest.

Every case is one pass of a user's program:

  continuum   a whole pushover of a small plane-strain block (reset, phase,
              every load step); one element phase of a brick block
              (displacements in, resisting force and, where a host assembly
              wants it, the tangent out); one Newton iteration of a brick
              block with the block-Jacobi PCG
  frames      the next load steps of a frame under a pushover or a ground
              motion (the state moves on from pass to pass, as an analysis
              does), a whole pushover of a small frame, a batch of frames
              under their own records
  gradients   one adjoint gradient, one direct differentiation
  systems     a standalone linear system filled by a host element loop

Inputs come from the repository's seeded model builders; all arithmetic is
FP64.  ``exact`` repeats the continuum and the standalone system in plain
torch and numpy.
"""
import numpy as np
import torch

from xara_gb300 import configs, gpu
from xara_gb300._abi import PhaseDesc, XG_INT_NEWMARK


def listed():
    return [
        # the smallest call: a test-sized block's pushover, all latency
        dict(name="quad_small", kind="quad", nx=9, ny=5, steps=6),
        # the plane-strain block of the benchmark, 20 increments to 0.5 %
        dict(name="quad_block", kind="quad", nx=64, ny=16, steps=20),
        # a host assembly takes the tangent and the resisting force of a
        # small ragged brick block
        dict(name="brick_export", kind="brick_phase", nx=13, ny=11, nz=7, tangent=True),
        # the element phase of a large block, yielding almost everywhere
        dict(name="brick_phase", kind="brick_phase", nx=64, ny=64, nz=48, tangent=False),
        # a Newton iteration of a medium block: element phase and PCG solve
        dict(name="brick_newton", kind="brick_newton", nx=47, ny=33, nz=21),
        # a single steel frame under a ground motion, ten time steps a call
        dict(name="steel_quake", kind="steel_quake", bays=3, stories=5, steps=10),
        # a layered RC frame (Concrete01 / Steel01): gravity and pushover
        dict(name="rc2d_push", kind="rc2d_push", bays=2, stories=3, steps=10),
        # a ragged 3D RC frame: the next load step of a pushover
        dict(name="rc3d_medium", kind="rc3d_push", bx=5, by=3, stories=8, steps=1),
        # the benchmark's 10 x 10 x 20 RC frame: the next load step
        dict(name="rc3d_large", kind="rc3d_push", bx=10, by=10, stories=20, steps=1),
        # many uneven frames at once, each under its own record, as CUDA graphs
        dict(name="batch_quake", kind="batch_quake", frames=512, steps=2),
        # a gradient of the roof drift by the adjoint, and a directional
        # derivative by direct differentiation, over a short record
        dict(name="adjoint", kind="adjoint", frames=12, steps=20, ckpt=8),
        # a linear system filled by a host element loop, then factored
        dict(name="linsoe", kind="linsoe", nx=23, ny=9, ndf=3, spd=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["quad", "brick_phase", "brick_newton", "steel_quake", "rc2d_push",
                       "rc3d_push", "batch_quake", "adjoint", "linsoe"])
    if kind == "quad":
        return dict(kind=kind, nx=_log_int(rng, 6, 64), ny=_log_int(rng, 4, 16),
                    steps=rng.randint(3, 20))
    if kind == "brick_phase":
        nx, ny, nz = _log_int(rng, 5, 64), _log_int(rng, 5, 64), _log_int(rng, 4, 48)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, tangent=nx * ny * nz < 4000)
    if kind == "brick_newton":
        return dict(kind=kind, nx=_log_int(rng, 5, 47), ny=_log_int(rng, 5, 33),
                    nz=_log_int(rng, 4, 21))
    if kind == "steel_quake":
        return dict(kind=kind, bays=rng.randint(1, 9), stories=rng.randint(2, 15),
                    steps=rng.randint(2, 12))
    if kind == "rc2d_push":
        return dict(kind=kind, bays=rng.randint(1, 4), stories=rng.randint(2, 5),
                    steps=rng.randint(4, 12))
    if kind == "rc3d_push":
        return dict(kind=kind, bx=rng.randint(1, 10), by=rng.randint(1, 10),
                    stories=_log_int(rng, 2, 20), steps=1)
    if kind == "batch_quake":
        return dict(kind=kind, frames=_log_int(rng, 8, 512), steps=rng.randint(1, 2))
    if kind == "adjoint":
        frames = _log_int(rng, 2, 12)
        steps = rng.randint(6, 20)
        return dict(kind=kind, frames=frames, steps=steps, ckpt=rng.randint(3, steps))
    return dict(kind="linsoe", nx=_log_int(rng, 5, 23), ny=_log_int(rng, 3, 9),
                ndf=rng.choice([2, 3, 6]), spd=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------
def _quad_model(case, seed):
    """A J2 block whose yield stress and hardening come from the seed."""
    rng = np.random.default_rng(seed)
    sy = float(rng.uniform(200e6, 300e6))
    j2 = (166.7e9, 76.9e9, sy, sy, 0.0, float(rng.uniform(0.8e9, 1.2e9)), 0.0, 0.0)
    return configs.quad_block(case["nx"], case["ny"], steps=case["steps"], j2=j2,
                              strain=0.005 * case["steps"] / 20)


def _brick_model(case, seed):
    return configs.brick_block(case["nx"], case["ny"], case["nz"], steps=1, seed=seed)


def _brick_fields(case, seed, crd):
    """Two compression fields of the block, varying in space: the committed
    one and the trial one, under which most points yield."""
    rng = np.random.default_rng(seed + 17)
    n = np.array([case["nx"], case["ny"], case["nz"]], np.float64)
    x, y, z = (crd / n).T
    out = []
    for eps in (1.6e-3, 2.6e-3 * float(rng.uniform(0.9, 1.1))):
        u = np.zeros_like(crd)
        u[:, 2] = -eps * n[2] * z * (1.0 + 0.6 * np.sin(2 * np.pi * x) * np.cos(np.pi * y))
        u[:, 0] = 0.3 * eps * n[0] * (x - 0.5) * z
        u[:, 1] = 0.3 * eps * n[1] * (y - 0.5) * z
        u += rng.normal(0.0, 1e-6, size=u.shape) * (z[:, None] > 0)
        out.append(u.ravel())
    return out


def _steady_record(npts, dt, pga, seed):
    """A Kanai-Tajimi record trimmed to its strong motion: the quiet lead-in
    and the decay cut off."""
    lead = 300
    rec = configs.kanai_tajimi(npts + 2 * lead, dt, pga, seed, t_decay=lead * dt)
    return rec[lead:lead + npts]


def _batch_model(build, frames, steps, seed):
    """Uneven frames (the same shapes for every seed); yield stresses and
    ground motions from the seed, in strong motion from the first step on."""
    desc, phases = build(frames, steps=4, seed=frames)
    rng = np.random.default_rng(seed)
    q = desc.uni_param.reshape(-1, 12)
    q[:, 0] *= np.exp(rng.normal(0.0, 0.05, len(q)))
    p = phases[0]
    lead = 200
    rec = configs.kanai_tajimi_batch(frames, steps + 2 * lead, p.dt,
                                     rng.uniform(0.1, 0.8, frames) * configs.G, seed + 7)
    return desc, PhaseDesc(
        integrator=XG_INT_NEWMARK, pattern=p.pattern, num_steps=steps, dt=p.dt, gamma=p.gamma,
        beta=p.beta, gm_dof=p.gm_dof, gm_accel=np.ascontiguousarray(rec[:, lead:]), gm_dt=p.gm_dt,
        gm_node_record=p.gm_node_record, alpha_m_node=p.alpha_m_node,
        beta_k_init_elem=p.beta_k_init_elem, tol=p.tol, max_iter=p.max_iter)


def _linsoe_system(case, seed):
    """Two-node elements on an nx x ny grid: random positive definite element
    matrices, ids numbered along the short side, one corner fixed."""
    rng = np.random.default_rng(seed)
    nx, ny, ndf = case["nx"], case["ny"], case["ndf"]
    ned = 2 * ndf
    pairs = [(i * ny + j, i * ny + j + 1) for i in range(nx) for j in range(ny - 1)]
    pairs += [(i * ny + j, (i + 1) * ny + j) for i in range(nx - 1) for j in range(ny)]
    pairs = np.asarray(pairs)
    eq = np.arange(nx * ny * ndf).reshape(nx * ny, ndf) - ndf      # node 0 fixed
    ids = np.concatenate([eq[pairs[:, 0]], eq[pairs[:, 1]]], axis=1).astype(np.int32)
    g = rng.normal(size=(len(pairs), ned, ned))
    mats = np.einsum("eij,ekj->eik", g, g) + ned * np.eye(ned)
    n = (nx * ny - 1) * ndf
    return n, ids, mats, rng.normal(size=n)


def _pattern(n, ids):
    valid = (ids >= 0) & (ids < n)
    r = np.repeat(ids[:, :, None], ids.shape[1], axis=2)
    c = np.repeat(ids[:, None, :], ids.shape[1], axis=1)
    ok = valid[:, :, None] & valid[:, None, :]
    key = np.unique(r[ok].astype(np.int64) * n + c[ok])
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=n))])
    return rowptr.astype(np.int32), (key % n).astype(np.int32)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "quad":
        desc, phases = _quad_model(case, seed)
        return dict(case=case, m=gpu.DeviceModel(desc), phases=phases)
    if kind in ("brick_phase", "brick_newton"):
        desc, _ = _brick_model(case, seed)
        m = gpu.DeviceModel(desc)
        m.set_system(gpu.XG_SYSTEM_BJPCG)
        uc, ut = _brick_fields(case, seed, desc.node_crd.reshape(-1, 3))
        m.set_trial_disp(uc)
        m.update(want_vals=False, want_resid=False)
        m.commit()
        b = np.random.default_rng(seed + 29).normal(size=m.neq)
        return dict(case=case, m=m, u=ut, b=b)
    if kind == "steel_quake":
        desc, phases = configs.steel_frame_2d_eq(
            case["bays"], case["stories"], steps=8000, seed=seed % 65536 + 1, grav_steps=4,
            record=_steady_record(8000, 0.01, 0.5 * configs.G, seed))
        m = gpu.DeviceModel(desc)
        m.set_phase(phases[0])
        m.analyze(phases[0].num_steps)
        m.set_phase(phases[1])
        return dict(case=case, m=m, phases=phases)
    if kind == "rc2d_push":
        rng = np.random.default_rng(seed)
        desc, phases = configs.rc_frame_2d(
            case["bays"], case["stories"], fc=float(rng.uniform(25e6, 35e6)),
            fy=float(rng.uniform(380e6, 450e6)), steps=case["steps"], grav_steps=4,
            drift=0.0005 * case["steps"])
        return dict(case=case, m=gpu.DeviceModel(desc), phases=phases)
    if kind == "rc3d_push":
        desc, phases = configs.rc_frame_3d(case["bx"], case["by"], case["stories"],
                                           grav_steps=4, steps=400, seed=seed)
        m = gpu.DeviceModel(desc)
        m.set_phase(phases[0])
        m.analyze(phases[0].num_steps)
        m.set_phase(phases[1])
        m.analyze(2)
        return dict(case=case, m=m, phases=phases)
    if kind == "batch_quake":
        desc, p = _batch_model(configs.frame_batch, case["frames"], 1200, seed)
        m = gpu.DeviceModel(desc)
        m.set_phase(p)
        gpu.set_graph(m, True)
        m.analyze(8)
        return dict(case=case, m=m, phases=[p])
    if kind == "adjoint":
        desc, p = _batch_model(configs.adjoint_frames, case["frames"], 200, seed)
        rng = np.random.default_rng(seed)
        q = desc.uni_param.reshape(-1, 12)
        return dict(case=case, m=gpu.DeviceModel(desc), phases=[p],
                    obj=(desc.meta["obj_node"], desc.meta["obj_dof"], desc.meta["obj_weight"]),
                    dth=rng.normal(size=(1, len(q), 3)) * q[None, :, :3] * 0.1)
    n, ids, mats, b = _linsoe_system(case, seed)
    rowptr, colidx = _pattern(n, ids)
    s = gpu.LinearSystem(rowptr, colidx, blk_start=np.arange(0, n + 1, case["ndf"]),
                         system=gpu.XG_SYSTEM_PROFILE_SPD if case["spd"] else
                         gpu.XG_SYSTEM_BJPCG)
    return dict(case=case, m=s, ids=ids, mats=mats, b=b)


def run(state):
    case, m = state["case"], state["m"]
    kind = case["kind"]
    if kind in ("quad", "rc2d_push"):
        # a whole analysis from the initial state
        m.reset()
        iters = []
        for p in state["phases"]:
            m.set_phase(p)
            iters += [s[0] for s in m.analyze(p.num_steps)]
        u, lam = m.disp()
        return dict(u=u, lam=lam, iters=np.array(iters))
    if kind == "brick_phase":
        m.set_trial_disp(state["u"])
        vals, resid, _ = m.update(want_vals=case["tangent"])
        return dict(resid=resid, vals=vals) if case["tangent"] else dict(resid=resid)
    if kind == "brick_newton":
        m.set_trial_disp(state["u"])
        _, resid, _ = m.update(want_vals=False)
        x, _, _ = m.solve(state["b"])
        return dict(resid=resid, x=x)
    if kind in ("steel_quake", "rc3d_push", "batch_quake"):
        # the analysis goes on from where the last pass left it
        iters = [s[0] for s in m.analyze(case["steps"])]
        u, lam = m.disp()
        out = dict(u=u, iters=np.array(iters))
        if kind == "rc3d_push":
            out["lam"] = lam
        else:
            out["v"] = m.response(gpu.XG_REC_VEL)
        return out
    if kind == "adjoint":
        node, dof, w = state["obj"]
        p = state["phases"][0]
        m.reset()
        J = gpu.adjoint_forward(m, p, case["steps"], case["ckpt"], node, dof, w)
        grad = gpu.adjoint_backward(m)
        m.reset()
        J2, dJ = gpu.ddm_forward(m, p, case["steps"], state["dth"], node, dof, w)
        return dict(J=J, grad=grad, J2=J2, dJ=dJ)
    m.zero_a()
    for ids, mat in zip(state["ids"], state["mats"]):
        m.add_a(mat, ids)
    m.set_b(state["b"])
    x, _, _ = m.solve()
    return dict(x=x)


def _sizes(case):
    """(fibers, equations, half bandwidth) of a frame case."""
    k = case["kind"]
    if k == "rc3d_push":
        nx, ny, s = case["bx"] + 1, case["by"] + 1, case["stories"]
        beams = s * (ny * case["bx"] + nx * case["by"])
        half = 6 * 0.8 * min(nx * ny, nx * s, ny * s)
        return 5 * (120 * nx * ny * s + 64 * beams), 6 * nx * ny * s, half
    if k in ("steel_quake", "rc2d_push"):
        b, s, nf = case["bays"], case["stories"], 40 if k == "steel_quake" else 12
        return 5 * nf * (s * (2 * b + 1)), 3 * (b + 1) * s, 3 * (1 + min(b + 1, s))
    f = case["frames"]                       # 6.5 bays x 11 stories on average
    return f * 32400, f * 248, 19


def work(case):
    """Each input read and each output written once; the arithmetic of the
    state determinations (about three a step) and of the linear solves."""
    k = case["kind"]
    if k == "quad":
        pts, neq = 4 * case["nx"] * case["ny"], 2 * (case["nx"] + 1) * case["ny"]
        half = 2 * (min(case["nx"], case["ny"]) + 2)
        st = 4 * case["steps"]
        return dict(bytes=case["steps"] * (pts * 80 + neq * 16),
                    flops=st * (pts * 700.0 + neq * half * half))
    if k in ("brick_phase", "brick_newton"):
        ne = case["nx"] * case["ny"] * case["nz"]
        nn = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        nbytes = ne * 8 * 112 + nn * 48 + nn * 24
        nnz = 240.0 * nn
        if k == "brick_phase":
            return dict(bytes=nbytes + nnz * 8, flops=ne * 8 * (400.0 + 36 * 30 * 2))
        its = 18.0 * max(case["nx"], case["ny"], case["nz"])   # block-Jacobi CG at 1e-12
        return dict(bytes=nbytes + its * (nnz * 8.4 + 3 * nn * 131.0),
                    flops=ne * 8 * 2600.0 + its * nnz * 2)
    if k == "linsoe":
        n, half = case["nx"] * case["ny"] * case["ndf"], (case["ny"] + 1) * case["ndf"]
        return dict(bytes=n * half * 8.0 + n * 16.0, flops=float(n) * half * half)
    fib, neq, half = _sizes(case)
    steps = case["steps"] + (4 if k == "rc2d_push" else 0)
    passes = 6 if k == "adjoint" else 1
    per_step = 3.0 * passes
    return dict(bytes=steps * passes * (fib * 160.0 + neq * 32.0),
                flops=steps * per_step * (fib * 60.0 + neq * half * half))


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), dtype=dtype, device=_DEV)


def _j2(eps, ep, xi, p):
    """Radial return with linear hardening on [..., 3, 3] strains.  The
    material scales the plastic multiplier by 1 - 1e-8."""
    K, G, sy, H = (p[..., i] for i in (0, 1, 2, 5))
    eye = torch.eye(3, dtype=eps.dtype, device=eps.device)
    tr = eps.diagonal(dim1=-2, dim2=-1).sum(-1)
    dev = eps - tr[..., None, None] / 3 * eye
    s = 2 * G[..., None, None] * (dev - ep)
    nrm = s.square().sum((-2, -1)).sqrt()
    r23 = (2.0 / 3.0) ** 0.5
    phi = nrm - r23 * (sy + H * xi)
    gam = torch.where(phi > 0, phi / (2 * G + 2 * H / 3) * (1 - 1e-8), torch.zeros_like(phi))
    n = torch.where(nrm[..., None, None] > 1e-10 * sy[..., None, None],
                    s / nrm.clamp_min(1e-300)[..., None, None], torch.zeros_like(s))
    ep1 = ep + gam[..., None, None] * n
    sig = 2 * G[..., None, None] * (dev - ep1) + (K * tr)[..., None, None] * eye
    c1 = -4 * G * G
    c2 = torch.where(phi > 0, c1 / (2 * G + 2 * H / 3), torch.zeros_like(phi))
    c3 = torch.where(phi > 0, c1 * gam / nrm.clamp_min(1e-300), torch.zeros_like(phi))
    b = 2 * G + c3
    return sig, (K - b / 3, b, c2 - c3, n), ep1, xi + r23 * gam


class _Continuum:
    """Eight-node bricks (2 x 2 x 2 points) or four-node quads in plane strain
    (2 x 2 points), J2 plasticity."""

    def __init__(self, desc, eqn):
        self.d = d = desc.ndm
        nen = 4 if d == 2 else 8
        conn = np.searchsorted(desc.node_tag, desc.elem_conn.reshape(-1, nen))
        corners = (np.array([[-1, -1], [1, -1], [1, 1], [-1, 1]], np.float64) if d == 2 else
                   np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                             [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], np.float64))
        grid = np.stack(np.meshgrid(*[[-1, 1]] * d, indexing="ij"), -1).reshape(-1, d) / 3 ** 0.5
        dn = np.empty((len(grid), nen, d))
        for q, pt in enumerate(grid):
            f = 1 + corners * pt
            for k in range(d):
                dn[q, :, k] = corners[:, k] * np.delete(f, k, axis=1).prod(1) / 2 ** d
        # the mesh's own cells: corners in the order of the connectivity
        crd = desc.node_crd.reshape(-1, d)[conn]
        x = _t(crd)
        dn = _t(dn)
        jac = torch.einsum("qak,eai->eqik", dn, x)
        self.dvol = torch.linalg.det(jac).abs()
        self.g = torch.einsum("qak,eqki->eqai", dn, torch.linalg.inv(jac))
        self.conn = _t(conn, torch.int64)
        self.dofs = (self.conn[:, :, None] * d + torch.arange(d, device=_DEV)).reshape(len(conn), -1)
        self.eq = _t(eqn, torch.int64)[self.dofs]
        self.neq = int(eqn.max()) + 1
        self.p = _t(desc.j2_param.reshape(-1, 8))[_t(desc.elem_mat, torch.int64)][:, None, :]
        ne, nq = self.dvol.shape
        self.ep = torch.zeros(ne, nq, 3, 3, dtype=torch.float64, device=_DEV)
        self.xi = torch.zeros(ne, nq, dtype=torch.float64, device=_DEV)

    def strain(self, u):
        ue = u[self.dofs].reshape(len(self.conn), -1, self.d)
        h = torch.einsum("eqaj,eai->eqij", self.g, ue)
        eps = torch.zeros(*h.shape[:2], 3, 3, dtype=h.dtype, device=h.device)
        eps[..., :self.d, :self.d] = 0.5 * (h + h.transpose(-2, -1))
        return eps

    def state(self, u):
        return _j2(self.strain(u), self.ep, self.xi, self.p)

    def commit(self, u):
        _, _, self.ep, self.xi = self.state(u)

    def resid(self, sig):
        f = torch.einsum("eq,eqij,eqaj->eai", self.dvol, sig[..., :self.d, :self.d], self.g)
        out = torch.zeros(self.neq + 1, dtype=f.dtype, device=f.device)
        return out.index_add_(0, self.eq.reshape(-1) % (self.neq + 1), f.reshape(-1))[:-1]

    def blocks(self, tan):
        """Element tangents [ne, ned, ned]."""
        a, b, c, n = tan
        g, d = self.g, self.d
        h = torch.einsum("eqij,eqaj->eqai", n[..., :d, :d], g)
        w = self.dvol
        k = torch.einsum("eq,eqai,eqbk->eaibk", w * a, g, g)
        k += torch.einsum("eq,eqak,eqbi->eaibk", w * b / 2, g, g)
        k += torch.einsum("eq,eqai,eqbk->eaibk", w * c, h, h)
        dot = torch.einsum("eq,eqaj,eqbj->eab", w * b / 2, g, g)
        k += torch.einsum("eab,ik->eaibk", dot, torch.eye(d, dtype=g.dtype, device=_DEV))
        ned = self.dofs.shape[1]
        return k.reshape(-1, ned, ned)

    def matrix(self, tan):
        """Assembled tangent as a coalesced sparse matrix."""
        k = self.blocks(tan)
        r = self.eq[:, :, None].expand_as(k).reshape(-1)
        c = self.eq[:, None, :].expand_as(k).reshape(-1)
        ok = (r >= 0) & (c >= 0)
        # entries that cancel stay in the pattern
        return torch.sparse_coo_tensor(torch.stack([r[ok], c[ok]]), k.reshape(-1)[ok],
                                       (self.neq, self.neq)).coalesce()


def _cg(a, b, rtol=1e-14):
    a = a.to_sparse_csr()
    dia = torch.zeros_like(b)
    crow, col = a.crow_indices(), a.col_indices()
    row = torch.repeat_interleave(torch.arange(len(b), device=b.device), crow[1:] - crow[:-1])
    on = row == col
    dia[row[on]] = a.values()[on]
    x = torch.zeros_like(b)
    for _ in range(4):                       # restarted from the true residual
        r = b - a @ x
        z = r / dia
        p, rz, stop = z.clone(), r @ z, float(b.norm()) * rtol
        for it in range(6000):
            q = a @ p
            al = rz / (p @ q)
            x += al * p
            r -= al * q
            if it % 20 == 0 and float(r.norm()) <= stop:
                break
            z = r / dia
            rz, old = r @ z, rz
            p = z + rz / old * p
    return x


def _quad_path(case, seed):
    """The pushover by Newton's method with dense solves."""
    desc, phases = _quad_model(case, seed)
    p = phases[0]
    eqn, _, _ = gpu.plan(desc)
    c = _Continuum(desc, eqn)
    f = torch.zeros(c.neq, dtype=torch.float64, device=_DEV)
    node = int(np.searchsorted(desc.node_tag, p.dc_node))
    ctrl = int(eqn[node * 2 + p.dc_dof])
    f[int(eqn[int(np.searchsorted(desc.node_tag, desc.load_node[0])) * 2 + 1])] = -1.0
    eq = _t(eqn, torch.int64)
    u, lam = torch.zeros(len(eqn), dtype=torch.float64, device=_DEV), 0.0
    spread = lambda v: torch.where(eq >= 0, v[eq.clamp_min(0)], torch.zeros_like(u))  # noqa: E731
    for _ in range(p.num_steps):
        want = p.dc_incr
        for it in range(30):
            sig, tan, _, _ = c.state(u)
            k = c.matrix(tan).to_dense()
            sol = torch.linalg.solve(k, torch.stack([lam * f - c.resid(sig), f], 1))
            dl = float((want - sol[ctrl, 0]) / sol[ctrl, 1])
            du = sol[:, 0] + dl * sol[:, 1]
            u, lam, want = u + spread(du), lam + dl, 0.0
            if it > 0 and float(du.norm()) < 1e-15 * max(1.0, float(u.norm())):
                break
        c.commit(u)
    return u.cpu().numpy(), lam


def exact(case, seed):
    kind = case["kind"]
    if kind == "quad":
        u, lam = _quad_path(case, seed)
        return dict(u=u, lam=lam, iters=None)
    if kind in ("brick_phase", "brick_newton"):
        desc, _ = _brick_model(case, seed)
        eqn, rowptr, colidx = gpu.plan(desc)
        uc, ut = _brick_fields(case, seed, desc.node_crd.reshape(-1, 3))
        c = _Continuum(desc, eqn)
        c.commit(_t(uc))
        sig, tan, _, _ = c.state(_t(ut))
        resid = c.resid(sig).cpu().numpy()
        if kind == "brick_newton":
            b = np.random.default_rng(seed + 29).normal(size=c.neq)
            return dict(resid=resid, x=_cg(c.matrix(tan), _t(b)).cpu().numpy())
        if not case["tangent"]:
            return dict(resid=resid)
        k = c.matrix(tan)
        key = k.indices()[0].cpu().numpy() * c.neq + k.indices()[1].cpu().numpy()
        rows = np.repeat(np.arange(c.neq, dtype=np.int64), np.diff(rowptr))
        vals = np.zeros(len(colidx))
        vals[np.searchsorted(rows * c.neq + colidx, key)] = k.values().cpu().numpy()
        return dict(resid=resid, vals=vals)
    if kind == "linsoe":
        n, ids, mats, b = _linsoe_system(case, seed)
        a = np.zeros((n + 1, n + 1))
        idx = np.where(ids < 0, n, ids)
        for i, m in zip(idx, mats):
            a[np.ix_(i, i)] += m
        return dict(x=np.linalg.solve(a[:n, :n], b))
    return None                              # fiber frames: no short plain form
