"""The element matrices formed by several lanes per element, at element
counts around the blocks' edges (16 quads; 4 bricks; 5 2D frame elements a warp, 20 a
block; 2 3D ones a warp, 8 a block), against the oracle's element by element:
entry-wise within 1e-12 of the element's largest entry, the bound the
elements' tangents have everywhere (a few hundred roundings of 1.1e-16)."""
import numpy as np
import pytest

from xara_gb300 import configs, gpu


def _model(kind, a, b, pdelta=0):
    if kind == "quad":
        return configs.quad_block(nx=a, ny=b, steps=1)[0]
    if kind == "quad_hard":      # saturating hardening
        return configs.quad_block(nx=a, ny=b, steps=1,
                                  j2=(166.67e9, 76.92e9, 200e6, 300e6, 40.0, 1e9, 0.0, 0.0))[0]
    if kind == "brick":
        return configs.brick_block(a, b, 1, steps=1)[0]
    if kind == "frame2d":
        return configs.steel_frame_2d(bays=a, stories=b, nfib=4, pdelta=pdelta, steps=1)[0]
    return configs.rc_frame_3d(bays_x=a, bays_y=1, stories=b, col_fibers=16, beam_fibers=16,
                               steps=1)[0]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,a,b,pdelta", [
    ("quad", 1, 1, 0), ("quad", 5, 3, 0), ("quad", 4, 4, 0), ("quad", 17, 1, 0),
    ("quad", 37, 5, 0), ("quad_hard", 5, 3, 0),
    ("brick", 1, 1, 0), ("brick", 3, 1, 0), ("brick", 2, 2, 0), ("brick", 5, 1, 0),
    ("brick", 9, 3, 0),
    ("frame2d", 1, 1, 0), ("frame2d", 2, 1, 1), ("frame2d", 2, 4, 0), ("frame2d", 3, 3, 1),
    ("frame3d", 1, 1, 0), ("frame3d", 2, 1, 0), ("frame3d", 2, 2, 0)])
def test_lanes_match_the_oracle(kind, a, b, pdelta):
    from oracle import port
    desc = _model(kind, a, b, pdelta)
    rng = np.random.default_rng(100 * a + b)
    U = rng.uniform(-1.0, 1.0, (desc.num_nodes, desc.ndf)) * (2e-5 if "frame" in kind else 2e-3)
    o = port.OracleModel(desc)
    Ko, Po = o.element_matrices(U)
    o.close()
    with gpu.DeviceModel(desc) as m:
        m.set_trial_disp(U)
        m.update()
        K, P = m.element_matrices()
    kscale = np.abs(Ko).reshape(len(Ko), -1).max(axis=1)[:, None, None]
    pscale = np.maximum(np.abs(Po).max(axis=1)[:, None], 1e-300)
    assert np.max(np.abs(K - Ko) / kscale) < 1e-12
    assert np.max(np.abs(P - Po) / pscale) < 1e-12
