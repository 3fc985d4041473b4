"""The block-inverse solve and whole steps in one launch (single FP64 scenes in
the dense form), at the sizes where their tiles, tiers and shares have edges:
one vertex tile and less, exactly one, one more, one tier and several, fewer
elements than warps; springs, bending, muscles and pneumatic springs.

Against the triangular form (kernel per phase, supernodal factor): iteration
counts equal, positions to 1e-12 and gradients to 1e-9 of their largest entry
(explicit inverses against triangular solves, as in test_solve_modes).  Within
the form everything is exact: n steps in one call are n calls of one step, a
replayed step and one regenerated from a checkpoint are the recorded one.
Mixed scenes keep X = Hs^-1 in their forward, whose steps in one launch are
the kernels launched one by one bit for bit (a batch of two runs those).
"""
import dataclasses

import numpy as np
import pytest

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu

def cube():
    """One cube, one face pinned (the beam would pin all eight vertices)."""
    d = S.inverse_stiffness(1, 1, 1)
    return dataclasses.replace(d, attach_vertex=d.attach_vertex[:4], attach_target=d.attach_target[:4],
                               attach_stiffness=d.attach_stiffness[:4])


SCENES = {
    "one_cube": cube, "27": lambda: S.inverse_stiffness(2, 2, 2),
    "64": lambda: S.inverse_stiffness(3, 3, 3), "65_up": lambda: S.inverse_stiffness(4, 3, 3),
    "625": lambda: S.inverse_stiffness(24, 4, 4), "two_tiers": lambda: S.inverse_stiffness(40, 8, 8),
    "three_tiers": lambda: S.inverse_stiffness(33, 12, 12), "cloth": lambda: S.cloth_sheet(nv=19),
    "muscles": lambda: S.muscle_beam(nx=13, ny=3, nz=3), "pneumatic": lambda: S.pneumatic_beam(),
    "star": lambda: S.muscle_star(refine=1, chains_per_arm=4, ground=False),
}


def inputs(d, n, seed):
    rng = np.random.default_rng(seed)
    x = np.asarray(d.x0, np.float64).reshape(-1) + 1e-3 * rng.standard_normal(3 * d.n_vertices)
    v = 0.1 * rng.standard_normal(x.size)
    act = rng.uniform(0, 1, (n, d.n_segments)) if d.n_segments else None
    return x, v, act, rng.standard_normal(x.size), 0.1 * rng.standard_normal(x.size)


def run(sc, n, x, v, act, gx, gv):
    xo, vo, tr = sc.forward(x, v, n_steps=n, act=act, traj=True)
    return {"x": xo, "v": vo, "traj": tr, "it": sc.iterations(n)}, sc.backward(gx, gv)


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300) if b.size else 0.0


@pytest.mark.parametrize("name", sorted(SCENES))
def test_block_form_matches_the_triangular_form(name):
    d = SCENES[name]()
    n = 3
    a = inputs(d, n, 7)
    sc = Scene(d)
    if d.n_tets:
        E = np.asarray(d.youngs) * np.random.default_rng(3).uniform(0.5, 2.0, d.n_tets)
        sc.set_materials(E, d.poisson)
    assert sc.solve_mode("dense")["mode"] == "dense"
    f, g = run(sc, n, *a)
    sc.solve_mode("persistent")
    ft, gt = run(sc, n, *a)
    assert np.array_equal(f["it"], ft["it"])
    assert rel(f["traj"], ft["traj"]) < 1e-12 and rel(f["v"], ft["v"]) < 1e-10
    for k in gt:
        assert rel(g[k], gt[k]) < 1e-9, k
    assert np.array_equal(f["traj"][-1], f["x"])
    sc.close()


@pytest.mark.parametrize("name", ["27", "625", "two_tiers", "cloth", "muscles", "pneumatic"])
def test_steps_in_one_launch_are_the_steps_one_by_one(name):
    d = SCENES[name]()
    n = 5
    x, v, act, gx, gv = inputs(d, n, 9)
    sc = Scene(d)
    sc.solve_mode("dense")
    f, g = run(sc, n, x, v, act, gx, gv)
    xs, vs = x, v
    for s in range(n):
        xs, vs = sc.forward(xs, vs, n_steps=1, act=None if act is None else act[s:s + 1])
    assert np.array_equal(xs, f["x"]) and np.array_equal(vs, f["v"])
    sc.close()
    for every, budget in ((1, 0), (3, 0), (2, None)):  # replayed, regenerated from checkpoints, stored
        sc = Scene(dataclasses.replace(d, checkpoint_every=every))
        sc.solve_mode("dense")
        if budget is not None:
            sc.set_adjoint_budget(budget)
        h, q = run(sc, n, x, v, act, gx, gv)
        assert np.array_equal(h["traj"], f["traj"]) and np.array_equal(h["it"], f["it"])
        for k in g:
            assert np.array_equal(q[k], g[k]), (every, budget, k)
        sc.close()


@pytest.mark.parametrize("name", ["one_cube", "27", "64", "625", "two_tiers", "cloth", "muscles", "pneumatic"])
def test_mixed_steps_in_one_launch_are_the_steps_one_by_one(name):
    """Bits of n steps, of single steps, and of the adjoint's replays; the
    adjoint (blocks or X) against the triangular form's on the same iterates."""
    d = dataclasses.replace(SCENES[name](), precision=_capi.DFEM_PREC_MIXED)
    n = 4
    x, v, act, gx, gv = inputs(d, n, 11)
    sc = Scene(d)
    sc.solve_mode("dense")
    f, g = run(sc, n, x, v, act, gx, gv)
    xs, vs = x, v
    for s in range(n):
        xs, vs = sc.forward(xs, vs, n_steps=1, act=None if act is None else act[s:s + 1])
    assert np.array_equal(xs, f["x"]) and np.array_equal(vs, f["v"])
    sc.set_adjoint_budget(0)
    h, q = run(sc, n, x, v, act, gx, gv)
    assert np.array_equal(h["traj"], f["traj"])
    for k in g:
        assert np.array_equal(q[k], g[k]), k
    sc.solve_mode("persistent")
    _, p = run(sc, n, x, v, act, gx, gv)  # other iterates: equal to the forces' FP32 rounding
    for k in p:
        assert rel(g[k], p[k]) < 1e-4, k
    sc.close()
