"""Buffers that a call cannot use are refused on the host, before anything is
launched: another kind of memory than the call's first buffer's, too few
values.  And the kernels use a device buffer in place only when the runtime
says that it is memory of the scene's GPU; other memory that a caller may pass
as device memory goes through a copy, with the same results."""
import ctypes as C
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "diff_fem_b200" / "csrc"


@pytest.fixture
def idle_scene(monkeypatch):
    """A handle without an engine behind it: 4 vertices, 1 tet, 2 activations; any library call fails the test."""
    from diff_fem_b200 import engine

    def no_call():
        raise AssertionError("a library call")

    monkeypatch.setattr(engine, "lib", no_call)
    monkeypatch.setattr(engine, "_sync_torch", lambda *a: None)
    sc = engine.Scene.__new__(engine.Scene)
    sc._h, sc.desc, sc.device, sc.nparts, sc.N, sc.T, sc.nseg, sc._last_steps = None, [], 0, 1, 4, 1, 2, 1
    return sc


def calls(sc, x, v, E, nu, act):
    return {"forward": lambda: sc.forward(x, v, act=act), "backward": lambda: sc.backward(x, v),
            "set_materials": lambda: sc.set_materials(E, nu), "eval_local": lambda: sc.eval_local(x),
            "set_activations": lambda: sc.set_activations(act)}


@pytest.mark.parametrize("call,short", [("forward", "x"), ("forward", "v"), ("forward", "act"), ("backward", "x"),
                                        ("backward", "v"), ("set_materials", "E"), ("set_materials", "nu"),
                                        ("eval_local", "x"), ("set_activations", "act")])
def test_short_buffers_are_refused(idle_scene, call, short):
    torch = pytest.importorskip("torch")
    for make in (np.zeros, lambda n: torch.zeros(n, dtype=torch.float64)):
        n = dict(x=12, v=12, E=1, nu=1, act=2)
        n[short] -= 1
        with pytest.raises(ValueError, match="values"):
            calls(idle_scene, **{k: make(q) for k, q in n.items()})[call]()


@pytest.mark.parametrize("call", ["forward", "backward", "set_materials"])
def test_two_kinds_of_memory_are_refused(idle_scene, call):
    torch = pytest.importorskip("torch")

    class OnDevice(torch.Tensor):  # as far as the handle can see
        is_cuda = True

    host = lambda n: np.zeros(n)
    cuda = lambda n: torch.zeros(n, dtype=torch.float64).as_subclass(OnDevice)
    for a, b in ((host, cuda), (cuda, host)):
        with pytest.raises(ValueError, match="same memory"):
            calls(idle_scene, a(12), b(12), a(1), b(1), None)[call]()


def test_memory_of_the_scenes_gpu_alone_is_used_in_place(tmp_path):
    src = tmp_path / "rule.cpp"
    src.write_text('#include "pointer_rule.h"\n#include <cstdlib>\nint main(int, char** a) { return dfem::used_in_place('
                   'std::atoi(a[1]), std::atoi(a[2]), std::atoi(a[3]), std::atoi(a[4])); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "rule"), str(src)], check=True)
    rule = lambda *a: subprocess.run([str(tmp_path / "rule"), *map(str, a)]).returncode
    for known in (0, 1):
        for kind in range(4):  # unregistered, host, device, managed
            for dev in (0, 1):
                assert rule(known, kind, dev, 1) == int(known == 1 and kind == 2 and dev == 1)


@pytest.mark.gpu
@pytest.mark.parametrize("contact", [False, True])
def test_registered_host_memory_as_device_memory(contact):
    """Pinned arrays passed as device pointers (the GPU can read them): the results of device tensors."""
    import torch
    from diff_fem_b200 import _capi, scene as S
    from diff_fem_b200.engine import Scene

    d = S.drop_box(height=0.002) if contact else S.muscle_beam()
    n = 2
    sc = Scene(d)
    rng = np.random.default_rng(3)
    x = torch.tensor(d.x0.reshape(-1))
    v = torch.tensor(0.1 * rng.standard_normal(x.numel()))
    act = torch.tensor(rng.uniform(0, 1, (n, d.n_segments))) if d.n_segments else None
    g = torch.tensor(rng.standard_normal(x.numel()))
    up = lambda t: None if t is None else t.cuda()
    xd, vd, td = sc.forward(up(x), up(v), n_steps=n, act=up(act), traj=True)
    bd = sc.backward(up(g), up(v))
    pin = lambda t: None if t is None else t.pin_memory()
    new = lambda *s: torch.zeros(*s, dtype=torch.float64).pin_memory()
    p = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    xi, vi, ai, gi = pin(x), pin(v), pin(act), pin(g)
    xo, vo, tr = new(x.numel()), new(x.numel()), new(n, x.numel())
    L = _capi.lib()
    _capi.check(L.dfem_step_forward(sc.handle, p(xi), p(vi), p(ai), n, p(xo), p(vo), p(tr), _capi.DFEM_MEM_DEVICE))
    gx, gv, gE, gnu, ga = new(x.numel()), new(x.numel()), new(max(1, sc.T)), new(max(1, sc.T)), new(max(1, n * sc.nseg))
    _capi.check(L.dfem_step_backward(sc.handle, p(gi), p(vi), p(gx), p(gv), p(gE), p(gnu), p(ga) if sc.nseg else None,
                                     _capi.DFEM_MEM_DEVICE))
    for a, b in ((xd, xo), (vd, vo), (td, tr), (bd["x"], gx), (bd["v"], gv), (bd["E"], gE), (bd["nu"], gnu)):
        assert torch.equal(a.cpu(), b)
    if sc.nseg:
        assert torch.equal(bd["act"].cpu().reshape(-1), ga)
    sc.close()
