"""The contact phase and its reverse sweep as one launch each, at the sizes
where their shares have edges: fewer vertices than a warp's four, elements
that take a second round of a CTA's warps in the forward (two threads per tet,
256 tets per CTA and round) and in the reverse sweep (128), cloth without
tets, a broad phase and none.  Bit for bit the loop of kernels.
"""
import numpy as np
import pytest

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu

CASES = {
    "cube": (lambda: S.drop_box(nx=1, ny=1, nz=1, height=0.002, v0=-1.0), 4),
    "ragged": (lambda: S.drop_box(nx=5, ny=2, nz=3, height=0.002, v0=-1.0), 4),
    "reverse_wraps": (lambda: S.drop_box(nx=20, ny=14, nz=14, height=0.002, v0=-1.0), 2),
    "forward_wraps": (lambda: S.drop_box(nx=40, ny=14, nz=14, height=0.002, v0=-1.0), 2),
    "cloth": (lambda: S.cloth_on_ball(nv=11, radius=0.08, drop=0.004, subdiv=2), 10),
}


@pytest.mark.parametrize("cells", [None, 0])
@pytest.mark.parametrize("name", sorted(CASES))
def test_one_launch_is_the_loop_of_kernels(name, cells):
    make, n = CASES[name]
    d = make()
    if cells == 0 and name.endswith("wraps"):
        pytest.skip("covered by the small boxes")
    x = d.x0.reshape(-1).copy()
    v = np.tile([0.0, -1.0, 0.0], d.n_vertices)
    rng = np.random.default_rng(5)
    gx, gv = rng.standard_normal(x.size), rng.standard_normal(x.size)
    out = []
    for fused in (1, 0):
        g = Scene(d)
        g.set_option("fused_contact", fused)
        if cells is not None:
            g.set_limit("broad_phase_cells", cells)
        xo, vo, tr = g.forward(x, v, n_steps=n, traj=True)
        b = g.backward(gx, gv)
        out.append([tr, vo, g.contact_passes(n), g.iterations(n), b["x"], b["v"], b["E"], b["nu"]])
        g.close()
    assert out[0][2].sum() > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
