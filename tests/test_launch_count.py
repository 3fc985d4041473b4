"""The launch count of a call does not depend on the forms that the handle ran
before: a scene switched to the dense form counts what a fresh handle counts,
also where the adjoint replays its steps."""
import numpy as np
import pytest

from diff_fem_b200 import scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["beam", "box_on_ground"])
@pytest.mark.parametrize("replay", [False, True])
def test_launches_after_a_switch_of_forms(scene, replay):
    d = S.inverse_stiffness(nx=8, ny=4, nz=4) if scene == "beam" else S.drop_box(height=0.002)
    x = d.x0.reshape(-1).copy()
    v = np.tile([0.0, -1.0, 0.0], d.n_vertices)

    def launches(sc):
        n = []
        for _ in range(3):  # the first calls build graphs and grow stores
            a = sc.launch_count()
            sc.forward(x, v, n_steps=3)
            b = sc.launch_count()
            sc.backward(x, v)
            n = [b - a, sc.launch_count() - b]
        return n

    counts = []
    for before in ("dense", "levels"):
        sc = Scene(d)
        if replay:
            sc.set_adjoint_budget(0)
        for mode in (before, "dense"):
            sc.solve_mode(mode)
            c = launches(sc)
        counts.append(c)
        sc.close()
    assert counts[0] == counts[1]
