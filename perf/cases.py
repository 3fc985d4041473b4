"""Performance cases of the projective-dynamics engine.

A case is one call, or one short sequence of calls, that a program makes on a
`Scene` it keeps: the local step alone, forward steps, a control step with its
gradient, or a whole gradient evaluation (new moduli, forward steps, adjoint).
`listed()` names the cases, `draw(rng)` gives others of the same ranges,
`prepare` builds the scene and its inputs, `run` is one pass, `work` the least
data and arithmetic of a pass, and `exact` the same results in 64 bits from a
plain torch statement of the scheme (dense factor, no code of this package).
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

EPS = 5e-7  # early exit of the PD loop: |x^k - x^(k-1)| / 3N


def listed():
    return [
        # The local step alone on an unpinned 800-tet box: the smallest call (an energy or
        # force evaluation inside somebody else's integrator).
        dict(name="local_box", kind="box", nx=8, ny=4, nz=5, do="local", steps=0, mixed=False),
        # One time step of the cantilever, forward only: the interactive / viewer loop.
        dict(name="step_cantilever", kind="cantilever", do="forward", steps=1, mixed=False),
        # A control step of a small muscle beam from host arrays, forward and gradient: what
        # sim_act does on every step of a policy roll-out.
        dict(name="control_muscle_beam", kind="muscle_beam", nx=8, ny=3, nz=3, do="gradient", steps=1, mixed=False, host=True),
        # A hanging cloth (springs and bending), a short window with its gradient.
        dict(name="grad_cloth_31", kind="cloth_sheet", nv=31, do="gradient", steps=10, mixed=False),
        # The inverse-stiffness beam of 12,800 tets: new moduli, 60 steps, dL/dE.  The headline workload.
        dict(name="design_beam_12800", kind="beam", nx=40, ny=8, nz=8, do="design", steps=60, mixed=False),
        # The same beam in the mixed form, forward only with its trajectory: a roll-out.
        dict(name="rollout_beam_12800_mixed", kind="beam", nx=40, ny=8, nz=8, do="rollout", steps=60, mixed=True),
        # A beam of odd extents between the small scenes and the large one.
        dict(name="design_beam_5x", kind="beam", nx=23, ny=7, nz=5, do="design", steps=12, mixed=True),
        # A large single scene, 26,640 tets: new moduli, a few steps, the gradient.
        dict(name="design_beam_26640", kind="beam", nx=37, ny=12, nz=12, do="design", steps=4, mixed=False),
        # The 9,840-tet muscle star in free flight, dL/dactivation over a window.
        dict(name="grad_star", kind="star", refine=2, ground=False, do="gradient", steps=10, mixed=True),
        # The star on its ground: obstacle contact with friction, forward and gradient.
        dict(name="grad_star_ground", kind="star", refine=2, ground=True, do="gradient", steps=6, mixed=False),
        # A cloth landing on a ball (1,280-face obstacle), the first contact steps with their gradient.
        dict(name="grad_cloth_ball", kind="cloth_ball", nv=49, do="gradient", steps=6, mixed=False),
        # Uneven independent scenes as one batch: forward and all gradients.
        dict(name="grad_batch_24", kind="batch", scenes=24, t_hi=12000, ground=False, do="gradient", steps=6, mixed=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "cantilever", "muscle_beam", "cloth_sheet", "beam", "beam", "beam", "star", "cloth_ball", "batch"])
    mixed = rng.random() < 0.4
    if kind == "box":
        return dict(kind=kind, nx=_log(rng, 3, 40), ny=rng.randint(2, 12), nz=rng.randint(2, 12), do="local", steps=0, mixed=False)
    if kind == "cantilever":
        return dict(kind=kind, do=rng.choice(["forward", "gradient"]), steps=_log(rng, 1, 40), mixed=mixed)
    if kind == "muscle_beam":
        return dict(kind=kind, nx=rng.randint(4, 24), ny=rng.randint(2, 5), nz=rng.randint(2, 5), do="gradient",
                    steps=_log(rng, 1, 30), mixed=mixed, host=rng.random() < 0.5)
    if kind == "cloth_sheet":
        return dict(kind=kind, nv=_log(rng, 6, 60), do=rng.choice(["forward", "gradient"]), steps=_log(rng, 2, 30), mixed=mixed)
    if kind == "beam":
        ny, nz = rng.randint(2, 12), rng.randint(2, 12)
        nx = max(2, min(60, int(_log(rng, 200, 5000) / (ny * nz))))
        steps = max(1, min(60, int(rng.uniform(0.2, 1.0) * 100000 / (nx * ny * nz * 5))))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, do=rng.choice(["design", "design", "rollout"]), steps=steps, mixed=mixed)
    if kind == "star":
        return dict(kind=kind, refine=rng.randint(1, 2), ground=rng.random() < 0.4, do="gradient", steps=_log(rng, 2, 8), mixed=False)
    if kind == "cloth_ball":
        return dict(kind=kind, nv=_log(rng, 16, 60), do="gradient", steps=rng.randint(2, 6), mixed=False)
    return dict(kind=kind, scenes=rng.randint(3, 20), t_hi=_log(rng, 2000, 12000), ground=False, do="gradient",
                steps=rng.randint(2, 6), mixed=mixed)


# ------------------------------------------------------------------ scenes ---

@functools.lru_cache(maxsize=None)
def _geometry(kind, *p):
    if kind == "box":
        return (S.drop_box(*p),)
    if kind == "cantilever":
        return (S.cantilever(),)
    if kind == "muscle_beam":
        return (S.muscle_beam(*p),)
    if kind == "cloth_sheet":
        return (S.cloth_sheet(nv=p[0]),)
    if kind == "beam":
        return (S.inverse_stiffness(*p),)
    if kind == "star":
        return (S.muscle_star(refine=p[0], chains_per_arm=min(8, 4 * p[0]), ground=p[1]),)
    if kind == "cloth_ball":
        return (S.cloth_on_ball(nv=p[0], drop=0.004),)
    if kind == "batch":
        return tuple(S.uneven_batch(n_scenes=p[0], t_hi=float(p[1]), ground=p[2])[0])
    raise ValueError(kind)


def _descs(case):
    keys = {"box": ("nx", "ny", "nz"), "cantilever": (), "muscle_beam": ("nx", "ny", "nz"), "cloth_sheet": ("nv",), "beam": ("nx", "ny", "nz"),
            "star": ("refine", "ground"), "cloth_ball": ("nv",), "batch": ("scenes", "t_hi", "ground")}[case["kind"]]
    prec = _capi.DFEM_PREC_MIXED if case["mixed"] else _capi.DFEM_PREC_FP64
    return [dataclasses.replace(d, precision=prec) for d in _geometry(case["kind"], *[case[k] for k in keys])]


def _inputs(case, seed):
    """Host inputs of a pass: moduli, a moving start state, activations, the cotangents of a loss."""
    rng = np.random.default_rng([20, seed])
    descs = _descs(case)
    out = []
    for d in descs:
        x0 = np.asarray(d.x0, np.float64)
        span = x0.max(axis=0) - x0.min(axis=0) + 1e-12
        # smooth motion (a few waves over the body) plus a little per-vertex noise
        k = rng.uniform(0.5, 2.0, (3, 3)) * 2 * np.pi / span.max()
        ph = rng.uniform(0, 2 * np.pi, 3)
        v = 0.1 * np.sin(x0 @ k + ph) + 0.005 * rng.standard_normal(x0.shape)
        if case["kind"] == "cloth_ball":
            v = 0.02 * np.sin(x0 @ k + ph) + np.array([0.0, -2.4, 0.0])
        if case["do"] == "local":
            x0 = x0 + 0.05 * v
        act = rng.uniform(0.0, 1.0, (max(1, case["steps"]), d.n_segments)) if d.n_segments else None
        E = 10.0 ** rng.uniform(4.0, 6.0, d.n_tets) if case["do"] == "design" else np.asarray(d.youngs, np.float64).copy()
        nu = np.asarray(d.poisson, np.float64).copy()
        gx, gv = rng.standard_normal(x0.size), 0.01 * rng.standard_normal(x0.size)
        out.append(dict(desc=d, x=x0.reshape(-1).copy(), v=v.reshape(-1), act=act, E=E, nu=nu, gx=gx, gv=gv))
    return out


def prepare(case, seed):
    parts = _inputs(case, seed)
    descs = [p["desc"] for p in parts]
    sc = Scene.batch(descs) if case["kind"] == "batch" else Scene(descs[0])
    if case.get("host"):
        to = lambda a: np.ascontiguousarray(a)
    else:
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda")
    cat = lambda key: to(np.concatenate([p[key] for p in parts]))
    acts = [p["act"] for p in parts if p["act"] is not None]
    act = to(np.concatenate(acts, axis=1)) if acts else None
    if case["do"] == "local" and act is not None:
        sc.set_activations(act[0])
    return dict(case=case, sc=sc, act=act, **{k: cat(k) for k in ("x", "v", "E", "nu", "gx", "gv")})


def run(s):
    case, sc, n = s["case"], s["sc"], s["case"]["steps"]
    if case["do"] == "local":
        return {"jd": sc.eval_local(s["x"])}
    if case["do"] == "design":
        sc.set_materials(s["E"], s["nu"])
    if case["do"] == "rollout":
        x, v, traj = sc.forward(s["x"], s["v"], n_steps=n, act=s["act"], traj=True)
        return {"x": x, "v": v, "traj": traj}
    x, v = sc.forward(s["x"], s["v"], n_steps=n, act=s["act"])
    if case["do"] == "forward":
        return {"x": x, "v": v}
    g = sc.backward(s["gx"], s["gv"])
    out = {"x": x, "v": v, "gx": g["x"], "gv": g["v"]}
    if sc.T:
        out["gE"], out["gnu"] = g["E"], g["nu"]
    if sc.nseg:
        out["gact"] = g["act"]
    return out


def work(case):
    """One pass of each part at the least it can take: per time step two local-global iterations
    (and two of the adjoint), each reading the tet tables and the positions once, solving with a
    sparse factor of about 40 entries a vertex, and 800 (adjoint 1,600) flops a tet for the projection."""
    b = f = 0.0
    for d in _descs(case):
        N, T = d.n_vertices, d.n_tets
        C = T + int(np.asarray(d.muscle_segment).size) + int(np.asarray(d.spring_weight).size)
        it = 104.0 * C + 72.0 * N
        if case["do"] == "local":
            b, f = b + it, f + 800.0 * T
            continue
        n = 2 * case["steps"]
        solve_b, solve_f = 8.0 * 40 * N + 48.0 * N, 12.0 * 40 * N
        b += n * (it + solve_b)
        f += n * (800.0 * T + solve_f)
        if case["do"] in ("gradient", "design"):
            b += n * (it + 8.0 * T + solve_b)
            f += n * (1600.0 * T + solve_f)
        if case["do"] == "design":
            b += 24.0 * T + 8.0 * 40 * N
            f += 40.0 * 40 * N
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the scheme in 64 bits ---

def _gcoef(x, tets):
    """(T, 4, 3) coefficients of the deformation gradient and the volumes (positive orientation)."""
    D = (x[tets[:, 1:]] - x[tets[:, :1]]).transpose(1, 2)  # columns x_k - x_0
    inv = torch.linalg.inv(D)
    return torch.cat([-inv.sum(1, keepdim=True), inv], 1), torch.linalg.det(D).abs() / 6


def _newton(s):
    """Volume projection of singular values (5 Newton steps), its Jacobian J[i,k] = dg_i/ds_k and
    the difference quotients (g_i - g_j)/(s_i - s_j) of the pairs (01, 02, 12)."""
    D = torch.zeros_like(s)
    dD = torch.zeros(s.shape[0], 3, 3, dtype=s.dtype, device=s.device)
    q = torch.ones_like(s)
    eye = torch.eye(3, dtype=s.dtype, device=s.device)
    for _ in range(5):
        p = s + D
        g = torch.stack([p[:, 1] * p[:, 2], p[:, 0] * p[:, 2], p[:, 0] * p[:, 1]], 1)
        num = (g * D).sum(1) - (p.prod(1) - 1)
        den = (g * g).sum(1)
        c = num / den
        dp = eye + dD
        z = torch.zeros_like(p[:, 0])
        dg_dp = torch.stack([torch.stack([z, p[:, 2], p[:, 1]], 1), torch.stack([p[:, 2], z, p[:, 0]], 1),
                             torch.stack([p[:, 1], p[:, 0], z], 1)], 1)
        dg = dg_dp @ dp
        dnum = (dg * D[:, :, None]).sum(1) + (g[:, :, None] * dD).sum(1) - (g[:, :, None] * dp).sum(1)
        dden = 2 * (g[:, :, None] * dg).sum(1)
        dc = (dnum * den[:, None] - num[:, None] * dden) / (den * den)[:, None]
        q = 1 - c[:, None] * torch.stack([p[:, 2], p[:, 1], p[:, 0]], 1) * q
        dD = g[:, :, None] * dc[:, None, :] + c[:, None, None] * dg
        D = c[:, None] * g
    return s + D, eye + dD, q


class _Exact:
    """One scene without contact, links or drag."""

    def __init__(self, d, E, nu):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.t = t = lambda a, ty=torch.float64: torch.as_tensor(np.asarray(a), dtype=ty, device=dev)
        self.d, self.N, self.T = d, d.n_vertices, d.n_tets
        x0 = t(d.x0).reshape(-1, 3)
        self.h, self.K = d.time_step, d.max_iterations
        self.m = t(d.mass) / self.h ** 2
        self.mask = torch.ones(self.N, dtype=torch.float64, device=dev) if d.gravity_mask is None else t(d.gravity_mask)
        H = torch.diag(self.m)
        add = lambda idx, L: H.view(-1).index_add_(0, (idx[:, :, None] * self.N + idx[:, None, :]).reshape(-1), L.reshape(-1))
        self.tets = t(d.tets, torch.int64).reshape(-1, 4)
        if self.T:
            self.E, self.nu = t(E), t(nu)
            self.G, self.vol = _gcoef(x0, self.tets)
            add(self.tets, (self.E * self.vol)[:, None, None] * (self.G @ self.G.transpose(1, 2)))
            self.wr = self.E / (1 + self.nu) * self.vol
            self.wv = self.wr * self.nu
        self.jatt = torch.zeros_like(x0)
        if np.asarray(d.attach_vertex).size:
            av, ak = t(d.attach_vertex, torch.int64), t(d.attach_stiffness)
            H.view(-1).index_add_(0, av * (self.N + 1), ak)
            self.jatt.index_add_(0, av, ak[:, None] * t(d.attach_target).reshape(-1, 3))
        self.nseg = int(d.n_segments)
        self.M = int(np.asarray(d.muscle_segment).size)
        if self.M:
            self.mv, self.ms = t(d.muscle_tets, torch.int64).reshape(-1, 4), t(d.muscle_segment, torch.int64)
            G, vol = _gcoef(x0, self.mv)
            self.mc = (G @ t(d.muscle_fiber).reshape(-1, 3, 1))[:, :, 0]
            self.mw = vol * t(d.muscle_stiffness)
            add(self.mv, self.mw[:, None, None] * self.mc[:, :, None] * self.mc[:, None, :])
        self.S = int(np.asarray(d.spring_weight).size)
        if self.S:
            self.sv, self.sw = t(d.spring_vertices, torch.int64).reshape(-1, 2), t(d.spring_weight).sqrt()
            self.sr = (x0[self.sv[:, 0]] - x0[self.sv[:, 1]]).norm(dim=1)
            add(self.sv, self.sw[:, None, None] * t([[1.0, -1.0], [-1.0, 1.0]]))
        for b in range(int(np.asarray(d.bend_weight).size)):  # the stencils' rest Laplacian norm is 0: only H sees them
            self._bend(x0, H, b)
        self.L = torch.linalg.cholesky(H)
        self.H = H

    def _bend(self, x0, H, b):
        if b == 0:  # all stencils at once (rings of equal length)
            o = np.asarray(self.d.bend_offsets)
            n = int(o[1] - o[0])
            v = self.t(self.d.bend_vertices, torch.int64).reshape(-1, n)
            mid, ring = x0[v[:, 0]][:, None], x0[v[:, 1:]]

            def tan_half(a, m, c):
                e, f = a - m, c - m
                s = e.norm(dim=2) * f.norm(dim=2)
                num = 1 - (e * f).sum(2) / s
                return num / (torch.linalg.cross(e, f).norm(dim=2) / s)

            nxt, prv = ring.roll(-1, 1), ring.roll(1, 1)
            # the angle at the middle vertex towards the next neighbour, and the angle at the previous one
            c = (tan_half(ring, mid.expand_as(ring), nxt) + tan_half(ring, prv, mid.expand_as(ring))) / (ring - mid).norm(dim=2)
            beta = torch.cat([c.sum(1, keepdim=True), -c], 1)
            L = self.t(self.d.bend_weight)[:, None, None] ** 3 * beta[:, :, None] * beta[:, None, :]
            H.view(-1).index_add_(0, (v[:, :, None] * self.N + v[:, None, :]).reshape(-1), L.reshape(-1))

    def solve(self, r):
        return torch.cholesky_solve(r, self.L)

    def _svd(self, F):
        U, s, Vh = torch.linalg.svd(F)
        return U, s, Vh.transpose(1, 2), torch.linalg.det(F) < 0

    def _tet(self, x, y=None):
        """J d of the tets; with a cotangent y also its VJP and the moduli's terms of J d."""
        F = x[self.tets].transpose(1, 2) @ self.G
        U, s, V, flip = self._svd(F)
        g, J, q = _newton(s)
        R = U @ V.transpose(1, 2)
        R[:, :, 2] = torch.where(flip[:, None], -R[:, :, 2], R[:, :, 2])
        W = U @ (g[:, :, None] * V.transpose(1, 2))
        out = torch.zeros_like(x)
        if y is None:
            P = self.wr[:, None, None] * R + self.wv[:, None, None] * W
            return out.index_add_(0, self.tets.reshape(-1), (self.G @ P.transpose(1, 2)).reshape(-1, 3))
        Y = y[self.tets].transpose(1, 2) @ self.G
        yr, yv = (Y * R).sum((1, 2)), (Y * W).sum((1, 2))
        A = self.wr[:, None, None] * Y
        A[:, :, 2] = torch.where(flip[:, None], -A[:, :, 2], A[:, :, 2])
        MR, MG = U.transpose(1, 2) @ A @ V, U.transpose(1, 2) @ (self.wv[:, None, None] * Y) @ V
        P = torch.diag_embed((torch.diagonal(MG, dim1=1, dim2=2)[:, :, None] * J).sum(1))
        for k, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
            ss = s[:, i] + s[:, j]
            sym = q[:, k] * 0.5 * (MG[:, i, j] + MG[:, j, i])
            asy = (g[:, i] + g[:, j]) / ss * 0.5 * (MG[:, i, j] - MG[:, j, i]) + (MR[:, i, j] - MR[:, j, i]) / ss
            P[:, i, j], P[:, j, i] = sym + asy, sym - asy
        gF = U @ P @ V.transpose(1, 2)
        out.index_add_(0, self.tets.reshape(-1), (self.G @ gF.transpose(1, 2)).reshape(-1, 3))
        return out, Y, yr, yv

    def jd(self, x, act):
        """J d(x) without the constant attachments."""
        out = self._tet(x) if self.T else torch.zeros_like(x)
        if self.M:
            Ff = (self.mc[:, :, None] * x[self.mv]).sum(1)
            p = ((1 - act[self.ms]) * self.mw)[:, None] * Ff
            out.index_add_(0, self.mv.reshape(-1), (self.mc[:, :, None] * p[:, None]).reshape(-1, 3))
        if self.S:
            e = x[self.sv[:, 0]] - x[self.sv[:, 1]]
            p = (self.sw * self.sr / e.norm(dim=1))[:, None] * e
            out.index_add_(0, self.sv[:, 0], p).index_add_(0, self.sv[:, 1], -p)
        return out

    def forward(self, x, v, act, n):
        x, v = self.t(x).reshape(-1, 3), self.t(v).reshape(-1, 3)
        g = self.t(self.d.gravity)
        self.hist, self.act, traj = [], None if act is None else self.t(act), []
        for k in range(n):
            q = x + self.h * (v + self.h * self.mask[:, None] * g)
            c0 = self.m[:, None] * q - self.H @ x + self.jatt
            it, prev = [q], torch.zeros_like(q)
            while len(it) <= self.K and not float((it[-1] - prev).norm()) / (3 * self.N) < EPS:
                prev = it[-1]
                it.append(x + self.solve(c0 + self.jd(prev, None if act is None else self.act[k])))
            self.hist.append(it)
            v = self.d.damping / self.h * (it[-1] - x)
            x = it[-1]
            traj.append(x.reshape(-1))
        return x.reshape(-1), v.reshape(-1), torch.stack(traj)

    def backward(self, gx, gv):
        gx, gv = self.t(gx).reshape(-1, 3), self.t(gv).reshape(-1, 3)
        gE, gnu = torch.zeros_like(self.E) if self.T else None, torch.zeros_like(self.E) if self.T else None
        gact = torch.zeros(len(self.hist), self.nseg, dtype=torch.float64, device=gx.device)
        c = self.d.damping / self.h
        for k in range(len(self.hist) - 1, -1, -1):
            it = self.hist[k]
            xb, xt, bb = gx + c * gv, -c * gv, torch.zeros_like(gx)
            for j in range(len(it) - 2, -1, -1):
                x, x1, y = it[j], it[j + 1], self.solve(xb)
                bb, xb = bb + y, torch.zeros_like(y)
                if self.T:
                    xb, Y, yr, yv = self._tet(x, y)
                    yh = (Y * (x1[self.tets].transpose(1, 2) @ self.G)).sum((1, 2))
                    gE += self.vol / (1 + self.nu) * (yr + self.nu * yv) - self.vol * yh
                    gnu += self.E * self.vol / (1 + self.nu) ** 2 * (yv - yr)
                if self.M:
                    db = self.mw[:, None] * (self.mc[:, :, None] * y[self.mv]).sum(1)
                    Ff = (self.mc[:, :, None] * x[self.mv]).sum(1)
                    gact[k].index_add_(0, self.ms, -(db * Ff).sum(1))
                    p = (1 - self.act[k][self.ms])[:, None] * db
                    xb.index_add_(0, self.mv.reshape(-1), (self.mc[:, :, None] * p[:, None]).reshape(-1, 3))
                if self.S:
                    db = self.sw[:, None] * (y[self.sv[:, 0]] - y[self.sv[:, 1]])
                    e = x[self.sv[:, 0]] - x[self.sv[:, 1]]
                    ln = e.norm(dim=1, keepdim=True)
                    u = e / ln
                    p = self.sr[:, None] / ln * (db - (u * db).sum(1, keepdim=True) * u)
                    xb.index_add_(0, self.sv[:, 0], p).index_add_(0, self.sv[:, 1], -p)
            qb = xb + self.m[:, None] * bb
            gx, gv = xt + qb, self.h * qb
        return gx.reshape(-1), gv.reshape(-1), gE, gnu, gact


def exact(case, seed):
    if case["do"] != "local" and (case["kind"] == "cloth_ball" or case.get("ground")):
        return None  # contact: impacts and stick/slide branches of the whole phase
    parts = _inputs(case, seed)
    res = []
    for p in parts:
        e = _Exact(p["desc"], p["E"], p["nu"])
        if case["do"] == "local":
            x = e.t(p["x"]).reshape(-1, 3)
            res.append({"jd": (e.jatt + e.jd(x, None if p["act"] is None else e.t(p["act"][0]))).reshape(-1)})
            continue
        x, v, traj = e.forward(p["x"], p["v"], p["act"], case["steps"])
        r = {"x": x, "v": v}
        if case["do"] == "rollout":
            r["traj"] = traj
        if case["do"] in ("gradient", "design"):
            r["gx"], r["gv"], gE, gnu, gact = e.backward(p["gx"], p["gv"])
            if e.T:
                r["gE"], r["gnu"] = gE, gnu
            if e.nseg:
                r["gact"] = gact
        res.append(r)
        del e
    keys = {k for r in res for k in r}
    return {k: torch.cat([r[k] for r in res if k in r], 1 if k in ("gact", "traj") else 0) for k in keys}
