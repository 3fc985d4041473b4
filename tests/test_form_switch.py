"""A form of the solve whose factor cannot be built is not switched to: the
handle stays in the form it had, with a factor, and gives that form's results."""
import numpy as np
import pytest

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("old", ["levels", "persistent", "resident"])
def test_a_failed_build_keeps_the_form_in_use(old):
    d = S.inverse_stiffness(nx=20, ny=6, nz=6)
    x = d.x0.reshape(-1).copy()
    v = np.zeros_like(x)
    E = 2.0 * np.asarray(d.youngs)

    def results():
        xo, vo = sc.forward(x, v, n_steps=2)
        return [xo, vo, sc.backward(np.ones_like(x), v)["E"]]

    sc = Scene(d)
    sc.set_materials(E, d.poisson)
    sc.solve_mode("dense")
    dense = results()
    sc.solve_mode(old)
    sc.set_materials(E, d.poisson)  # the blocks are not those of the moduli any more
    ref = results()
    sc.set_limit("solve_wait_polls", 1)
    with pytest.raises(_capi.DfemError) as ex:
        sc.solve_mode("dense")
    assert ex.value.code == _capi.DFEM_ERR_CAP
    sc.set_limit("solve_wait_polls")
    assert sc.solve_mode()["mode"] == old
    assert all(np.array_equal(a, b) for a, b in zip(results(), ref))
    assert sc.solve_mode("dense")["mode"] == "dense"
    assert all(np.array_equal(a, b) for a, b in zip(results(), dense))
    sc.close()


def test_forms_share_one_regularisation():
    """Indefinite moduli: whichever form raises the regularisation, the other
    is rebuilt with it before it solves."""
    d = S.inverse_stiffness(nx=6, ny=2, nz=2)
    x = d.x0.reshape(-1).copy()
    out, regs = [], []
    sc = Scene(d)
    sc.solve_mode("persistent")
    sc.set_materials(np.full(d.n_tets, -1e6), d.poisson)
    for mode in ("persistent", "dense", "persistent", "dense"):
        sc.solve_mode(mode)
        out.append(sc.forward(x, np.zeros_like(x), n_steps=1)[0])
        regs.append(sc.info()["factor_regularisation"])
    assert regs[0] > 0 and regs[1] == regs[2] == regs[3] >= regs[0]
    assert np.array_equal(out[1], out[3])
    sc.close()
