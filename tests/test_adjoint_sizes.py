"""The adjoint local steps run as two kernels, of two and three CTAs per SM, by
the number of tets: a scene's gradient is the same bit for bit alone and as a
part of a batch on either side of the line (200,000 tets)."""
import numpy as np
import pytest

from diff_fem_b200 import scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("contact", [False, True])
@pytest.mark.parametrize("parts", [2, 17])
def test_gradient_does_not_depend_on_the_batch(contact, parts):
    d = S.drop_box(nx=20, ny=13, nz=10, height=0.002) if contact else S.inverse_stiffness(nx=41, ny=8, nz=8)
    assert (parts * d.n_tets >= 200000) == (parts > 2)
    n = 2
    rng = np.random.default_rng(4)
    x = d.x0.reshape(-1) + 1e-4 * rng.standard_normal(3 * d.n_vertices)
    v = np.tile([0.0, -1.0, 0.0], d.n_vertices)
    gx, gv = rng.standard_normal(x.size), rng.standard_normal(x.size)
    one = Scene(d)
    one.solve_mode("persistent")  # the batch's arithmetic
    one.forward(x, v, n_steps=n)
    if contact:
        assert one.contact_passes(n).sum() > 0
    want = one.backward(gx, gv)
    one.close()
    b = Scene.batch([d] * parts)
    rep = lambda a: np.tile(a, parts)
    b.forward(rep(x), rep(v), n_steps=n)
    got = b.backward(rep(gx), rep(gv))
    for k in ("x", "v", "E", "nu"):
        for part in np.split(got[k], parts):
            assert np.array_equal(part, want[k]), k
    b.close()
