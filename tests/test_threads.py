"""Scenes of several threads, each with launches that hold every SM for a call
(block build, whole steps, contact phase) or a cluster: their barriers do not
depend on one another, and every call gives the bits it gives alone."""
import threading

import numpy as np
import pytest

from diff_fem_b200 import scene as S
from diff_fem_b200._capi import DFEM_PREC_MIXED
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu

SCENES = {
    "beam": lambda: S.inverse_stiffness(nx=20, ny=6, nz=6),
    "beam_mixed": lambda: S.inverse_stiffness(nx=12, ny=6, nz=6, precision=DFEM_PREC_MIXED),
    "box_on_ground": lambda: S.drop_box(nx=5, ny=2, nz=3, height=0.002, v0=-1.0),
    "cantilever": S.cantilever,
}


def one_pass(g, d, seed):
    rng = np.random.default_rng(seed)
    x = d.x0.reshape(-1).copy()
    v = np.tile([0.0, -1.0, 0.0], d.n_vertices)
    g.set_materials(rng.uniform(0.5, 2.0, d.n_tets) * np.asarray(d.youngs), d.poisson)
    xo, vo = g.forward(x, v, n_steps=4)
    b = g.backward(rng.standard_normal(x.size), rng.standard_normal(x.size))
    return [xo, vo, b["x"], b["v"], b["E"], b["nu"]]


@pytest.mark.parametrize("names", [("beam", "beam"), ("beam", "beam_mixed", "box_on_ground", "cantilever")])
def test_threads_get_the_bits_of_a_scene_alone(names):
    reps, work = 8, []
    for n in names:
        d = SCENES[n]()
        work.append((d, Scene(d)))
    alone = [[one_pass(g, d, k) for k in range(reps)] for d, g in work]
    start, wrong = threading.Barrier(len(work)), []

    def run(i):
        d, g = work[i]
        try:
            start.wait(60)
            for k in range(reps):
                for q, (a, b) in enumerate(zip(alone[i][k], one_pass(g, d, k))):
                    if not np.array_equal(a, b):
                        wrong.append((names[i], k, q))
        except Exception as e:  # noqa: BLE001 (reported by the test's own thread)
            wrong.append((names[i], repr(e)))

    th = [threading.Thread(target=run, args=(i,)) for i in range(len(work))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not wrong, wrong
    for _, g in work:
        g.close()
