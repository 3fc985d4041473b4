"""The words in which the detections of a contact phase raise a hit.

Between two barriers of back-to-back detections the CTAs set one word, some of
them still read the last detection's, and thread 0 clears one: the three have
to differ, and a word has to be clear when a detection starts to set it.  On a
GPU: a box at rest within the contact thickness of its ground, where every
pass's iterations converge at once and every detection hits again, so the
phase ends at its cap of passes, in the one-launch form as in the loop of
kernels.
"""
import dataclasses
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "diff_fem_b200" / "csrc"


def words(tmp_path, n):
    src = tmp_path / "words.cpp"
    src.write_text('#include <cstdio>\n#include "contact_flags.h"\nint main() { for (int n = 0; n < %d; ++n) '
                   'std::printf("%%d %%d\\n", dfem::hit_word(n), dfem::cleared_word(n)); }\n' % n)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "words"), str(src)], check=True)
    out = subprocess.run([str(tmp_path / "words")], check=True, capture_output=True, text=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


def ordered(hit, cleared):
    """No word is touched by two sides between barriers n and n + 1, and none is set before it was cleared."""
    dirty = set()
    for n in range(len(hit) - 1):
        dirty.add(hit[n])  # detection n, then barrier n
        if cleared[n] in (hit[n], hit[n + 1]) or hit[n + 1] in dirty - {cleared[n]}:
            return False
        dirty.discard(cleared[n])
    return True


def test_back_to_back_detections_touch_different_words(tmp_path):
    w = words(tmp_path, 12)
    assert ordered([h for h, _ in w], [c for _, c in w])
    assert not ordered([n & 1 for n in range(12)], [1 - (n & 1) for n in range(12)])  # two words in turn


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [1, 2, 3, 7, None])
def test_converged_vertices_that_still_hit_end_at_the_cap(limit):
    from diff_fem_b200 import _capi, scene as S
    from diff_fem_b200.engine import Scene

    d = dataclasses.replace(S.drop_box(height=5e-5, v0=0.0), gravity=(0.0, 0.0, 0.0))
    x = d.x0.reshape(-1).copy()
    passes = []
    for fused in (1, 0):
        g = Scene(d)
        g.set_option("fused_contact", fused)
        if limit is not None:
            g.set_limit("contact_passes", limit)
        for _ in range(20 if fused else 1):
            with pytest.raises(_capi.DfemError) as ex:
                g.forward(x, np.zeros_like(x), n_steps=1)
            assert ex.value.code == _capi.DFEM_ERR_CAP and "pass cap" in str(ex.value)
            passes.append(int(g.contact_passes(1)[0]))
        g.close()
    assert min(passes) > 0 and len(set(passes)) == 1, passes
