"""Grid-wide barriers that give up (their polls lowered to one through
dfem_set_limit, which the kernels meet by finishing early): the call that
launched them returns DFEM_ERR_CAP, nothing counts as built, and the same
handle then reproduces its clean results bit for bit."""
import numpy as np
import pytest

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu


def run(sc, d, n=3):
    x = d.x0.reshape(-1).copy()
    v = np.tile([0.0, -1.0, 0.0], d.n_vertices)
    xo, vo = sc.forward(x, v, n_steps=n)
    g = sc.backward(np.ones_like(x), np.zeros_like(x))
    return [xo, vo] + [g[k] for k in ("x", "v", "E", "nu")]


def gives_up(fn):
    with pytest.raises(_capi.DfemError) as ex:
        fn()
    assert ex.value.code == _capi.DFEM_ERR_CAP and "barrier" in str(ex.value), str(ex.value)


def same(a, b):
    return all(np.array_equal(u, w) for u, w in zip(a, b))


def test_block_build():
    d = S.inverse_stiffness(nx=20, ny=6, nz=6)
    sc = Scene(d)
    assert sc.solve_mode("dense")["mode"] == "dense"
    ref = run(sc, d)
    sc.set_limit("solve_wait_polls", 1)
    gives_up(lambda: sc.set_materials(2.0 * np.asarray(d.youngs), d.poisson))
    gives_up(lambda: sc.set_materials(2.0 * np.asarray(d.youngs), d.poisson))  # not a stale barrier's pass
    sc.set_limit("solve_wait_polls")
    sc.set_materials(d.youngs, d.poisson)
    assert same(run(sc, d), ref)
    sc.close()


@pytest.mark.parametrize("scene", ["beam", "box_on_ground"])
def test_steps_and_contact_phase(scene):
    """The PD steps' launch gives up, and in the level form, which waits for
    nothing, the contact phase's."""
    if scene == "beam":
        d, modes = S.inverse_stiffness(nx=20, ny=6, nz=6), ["dense"]
    else:
        d, modes = S.drop_box(nx=12, ny=8, nz=8, height=0.002), ["dense", "levels"]
    x = d.x0.reshape(-1).copy()
    v = np.tile([0.0, -1.0, 0.0], d.n_vertices)
    for mode in modes:
        sc = Scene(d)
        assert sc.solve_mode(mode)["mode"] == mode
        ref = run(sc, d)
        assert scene == "beam" or sc.contact_passes(3).sum() > 0
        for _ in range(2):
            sc.set_limit("solve_wait_polls", 1)
            gives_up(lambda: sc.forward(x, v, n_steps=3))
            with pytest.raises(_capi.DfemError) as ex:
                sc.backward(np.ones_like(x), np.zeros_like(x))
            assert ex.value.code == _capi.DFEM_ERR_STATE
            sc.set_limit("solve_wait_polls")
            assert same(run(sc, d), ref)
        sc.close()
