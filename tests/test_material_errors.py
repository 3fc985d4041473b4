"""Moduli that are refused leave the scene as it was: its factor, its weights
and the forward that a backward is still to differentiate.  In every form of
the solve whose factor a material update rebuilds, and in a batch."""
import dataclasses

import numpy as np
import pytest

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu

KEYS = ("x", "v", "E", "nu", "act")


def results(sc, x, v):
    xo, vo = sc.forward(x, v, n_steps=3)
    g = sc.backward(np.ones_like(x), np.zeros_like(x))
    return [xo, vo] + [g[k] for k in KEYS]


@pytest.mark.parametrize("form", ["dense", "persistent", "levels", "mixed", "contact", "batch"])
def test_refused_moduli_change_nothing(form):
    beam = S.inverse_stiffness(nx=20, ny=6, nz=6)
    if form == "batch":
        descs = [S.inverse_stiffness(nx=6, ny=2, nz=2), beam]
        sc, x = Scene.batch(descs), np.concatenate([d.x0.reshape(-1) for d in descs])
    else:
        beam = dataclasses.replace(beam, precision=_capi.DFEM_PREC_MIXED) if form == "mixed" else beam
        if form == "contact":
            beam = S.drop_box(nx=6, ny=4, nz=4, height=0.002)
        sc, x = Scene(beam), beam.x0.reshape(-1).copy()
        sc.solve_mode({"mixed": "dense", "contact": "dense"}.get(form, form))
    v = np.tile([0.0, -1.0, 0.0], x.size // 3)
    rng = np.random.default_rng(2)
    E, nu = 10.0 ** rng.uniform(4, 6, sc.T), rng.uniform(0.2, 0.4, sc.T)
    sc.set_materials(E, nu)
    ref = results(sc, x, v)
    for bad_E, bad_nu in (((sc.T // 2, np.nan), None), (None, (0, -1.0)), ((sc.T - 1, np.inf), None)):
        e, n = 3.0 * E, 0.5 * nu
        if bad_E:
            e[bad_E[0]] = bad_E[1]
        if bad_nu:
            n[bad_nu[0]] = bad_nu[1]
        with pytest.raises(_capi.DfemError) as ex:
            sc.set_materials(e, n)
        assert ex.value.code == _capi.DFEM_ERR_INVALID
        g = sc.backward(np.ones_like(x), np.zeros_like(x))  # of the forward before
        assert all(np.array_equal(g[k], r) for k, r in zip(KEYS, ref[2:]))
        assert all(np.array_equal(a, b) for a, b in zip(results(sc, x, v), ref))
    sc.close()


@pytest.mark.parametrize("mode", ["dense", "levels"])
def test_a_failed_factorisation_leaves_no_factor(mode):
    """Finite moduli whose Hs overflows fail every regularisation."""
    d = S.inverse_stiffness(nx=6, ny=2, nz=2)
    d = dataclasses.replace(d, x0=1e3 * d.x0, attach_target=1e3 * d.attach_target)  # entries of Hs: 1e308 x 20
    sc = Scene(d)
    sc.solve_mode(mode)
    x = d.x0.reshape(-1).copy()
    v = np.zeros_like(x)
    ref = results(sc, x, v)
    with pytest.raises(_capi.DfemError) as ex:
        sc.set_materials(np.full(d.n_tets, 1e308), d.poisson)
    assert ex.value.code == _capi.DFEM_ERR_FACTOR
    for call in (lambda: sc.forward(x, v), lambda: sc.backward(x, v), lambda: sc.solve_mode("persistent")):
        with pytest.raises(_capi.DfemError) as ex:
            call()
        assert ex.value.code == _capi.DFEM_ERR_STATE
    sc.set_materials(d.youngs, d.poisson)
    assert all(np.array_equal(a, b) for a, b in zip(results(sc, x, v), ref))
    sc.close()
