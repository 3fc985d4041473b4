"""The corotated projection and its VJP over the element states that choose
its path: near rest, strongly stretched, inverted, close to a lower rank on
either side of the polar iteration's limit, and of extreme size.  One scene of
disjoint tets, the engine (FP64) against the oracle's SVD.

Tolerances: the polar factor's error is a few roundings of the element times
its conditioning 2 s_max / (s_mid + s_min) (Jacobian of the polar factor); 64
roundings are allowed, on values and on VJPs (one power more)."""
import numpy as np
import pytest

from diff_fem_b200 import scene as S
from diff_fem_b200.engine import Scene
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
SV = {  # singular values of F
    "near_rest": (1.02, 1.0, 0.97), "stretched": (4.0, 1.3, 0.3), "shrunk": (0.4, 0.3, 0.2), "equal": (1.0, 1.0, 1.0),
    "flat_polar": (1.0, 0.9, 0.01), "flat_svd": (1.0, 0.9, 1e-3), "needle_polar": (1.0, 0.1, 0.09),
    "needle_svd": (1.0, 0.02, 0.015), "tiny": (2e-5, 1e-5, 1e-5), "huge": (3e4, 2e4, 1e4),
}


def rotation(rng):
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else -q


def elements(kind, n, rng):
    """n disjoint rest tets and their deformed corners; every second one inverted."""
    rest = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    x0, x, inverted = [], [], []
    for k in range(n):
        r = rest @ (np.eye(3) + 0.3 * rng.uniform(-1, 1, (3, 3))).T * 0.1
        s = np.array(SV[kind]) * rng.uniform(0.95, 1.05, 3)
        if kind == "equal":
            s[:] = 1.0
        F = rotation(rng) @ np.diag(s) @ rotation(rng).T
        if k % 2:
            F = F @ np.diag([1, 1, -1.0])
        x0.append(r + 5.0 * k)
        x.append((r - r[0]) @ F.T + rng.standard_normal(3))
    return np.concatenate(x0), np.concatenate(x)


def describe(x0, n):
    return S.SceneDesc(x0=x0, mass=np.full(4 * n, 0.01), tets=np.arange(4 * n, dtype=np.int32).reshape(n, 4),
                       youngs=np.full(n, 1e5), poisson=np.full(n, 0.35), time_step=0.01, max_iterations=1)


@pytest.mark.parametrize("n", [1, 127, 128, 129])
@pytest.mark.parametrize("kind", sorted(SV))
def test_projection_and_vjp_match_the_svd(kind, n):
    rng = np.random.default_rng(len(kind) * 1000 + n)
    x0, x = elements(kind, n, rng)
    d = describe(x0, n)
    g, o = Scene(d), O.OracleScene(d)
    s = SV[kind]
    cond = 2 * 1.05 * s[0] / (0.95 * (s[1] + s[2]))
    a = g.eval_local(x.reshape(-1)).reshape(n, 12)
    b = np.asarray(o.eval_local(x.reshape(-1))).reshape(n, 12)
    err = np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)
    pos = np.abs(x).max() / (0.1 * s[2])  # the corners are differences of positions of this size
    tol = 64 * EPS * cond * max(1.0, pos)
    assert err.max() < tol, (err.max(), tol)
    # one iteration forward and back: the VJP at x and the moduli's terms
    v = np.zeros(x.size)
    g.forward(x.reshape(-1), v)
    o.forward(x.reshape(-1), v)
    gx, gv = rng.standard_normal(x.size), rng.standard_normal(x.size)
    p, q = g.backward(gx, gv), o.backward(gx, gv)
    # (near a rotation the moduli's terms cancel down to the strain: there they are held to the terms' own size,
    # vol |Y| |F| with |Y| <= 4 |G| |y| and |y| <= |cotangent| h^2 / m, times E for nu)
    G = 4 * max(np.linalg.norm(np.linalg.inv((x0[4 * t + 1:4 * t + 4] - x0[4 * t]).T)) for t in range(n))
    y = (np.abs(gx).max() + np.abs(gv).max() / d.time_step) * d.time_step ** 2 / 0.01
    term = S.tet_volumes(x0, np.asarray(d.tets)).max() * G * y * np.sqrt(3.0)
    size = {"E": term, "nu": 1e5 * term} if kind in ("equal", "near_rest") else {}
    for k in ("x", "v", "E", "nu"):
        e = np.abs(p[k] - q[k]).max() / max(np.abs(q[k]).max(), size.get(k, 0.0))
        assert e < tol * cond, (k, e, tol * cond)
    g.close()
