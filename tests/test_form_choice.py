"""The autotune's choice for a scene whose solve takes about as long in two
forms does not follow the timing's jitter: handles of one scene solve in one
form, and so give the same bits."""
import numpy as np
import pytest

from diff_fem_b200 import scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: S.drop_box(nx=1, ny=1, nz=1, height=0.002), lambda: S.inverse_stiffness(2, 2, 2),
                                  lambda: S.cloth_sheet(nv=6)], ids=["cube", "beam", "cloth"])
def test_handles_of_a_scene_choose_the_same_form(make):
    d = make()
    x = d.x0.reshape(-1).copy()
    modes, out = set(), []
    for _ in range(24):
        sc = Scene(d)
        modes.add(sc.solve_mode()["mode"])
        out.append(sc.forward(x, np.zeros_like(x), n_steps=2)[0])
        sc.close()
    assert modes == {"dense"}
    assert all(np.array_equal(out[0], o) for o in out)
