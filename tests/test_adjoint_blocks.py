"""The blocks that a mixed scene's adjoint solves with are its adjoint's: a
program that only runs forward holds none, an adjoint without room for them
leaves nothing allocated and solves with Hs^-1 instead, and the next material
change tries them again."""
import dataclasses

import numpy as np
import pytest

from diff_fem_b200 import _capi, scene as S
from diff_fem_b200.engine import Scene

pytestmark = pytest.mark.gpu

MB = 1 << 20


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def beam():
    return dataclasses.replace(S.inverse_stiffness(nx=40, ny=8, nz=8), precision=_capi.DFEM_PREC_MIXED)


def backward(sc, x):
    g = sc.backward(np.ones_like(x), np.zeros_like(x))
    return [g[k] for k in ("x", "v", "E", "nu")]


def test_a_forward_alone_holds_no_blocks():
    d = beam()
    sc = Scene(d)
    assert sc.solve_mode("dense")["mode"] == "dense"
    x = d.x0.reshape(-1).copy()
    sc.forward(x, np.zeros_like(x), n_steps=2)
    before = used()
    backward(sc, x)
    assert used() - before > 10 * MB  # fronts and products of ten blocks of up to 373 columns and one of 693
    sc.close()


def test_an_adjoint_without_room_for_its_blocks():
    lib = _capi.lib()
    d = beam()
    sc = Scene(d)
    sc.solve_mode("dense")
    x = d.x0.reshape(-1).copy()
    first = None
    got = []
    try:
        for after in range(40):
            sc.set_materials(d.youngs, d.poisson)
            sc.forward(x, np.zeros_like(x), n_steps=2)
            lib.dfem_debug_fail_allocations(after)
            n = sc.launch_count()
            got.append(backward(sc, x))
            n = sc.launch_count() - n
            lib.dfem_debug_fail_allocations(-1)
            if n < 10:  # one launch (and the blocks' build): every allocation succeeded
                break
            first = used() if first is None else first
            assert used() <= first + 4 * MB, after
    finally:
        lib.dfem_debug_fail_allocations(-1)
    assert 1 < len(got) < 40
    for g in got[:-1]:  # with Hs^-1: the same bits each time, the blocks' to rounding
        assert all(np.array_equal(a, b) for a, b in zip(g, got[0]))
    assert all(np.abs(a - b).max() < 1e-9 * np.abs(b).max() for a, b in zip(got[0], got[-1]))
    sc.forward(x, np.zeros_like(x), n_steps=2)
    assert all(np.array_equal(a, b) for a, b in zip(backward(sc, x), got[-1]))
    sc.close()
