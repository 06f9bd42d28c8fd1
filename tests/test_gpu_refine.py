"""The quarter-pel refinement where its warps of 16 cells end inside the frame (1, 6, 85 and 561 cells)
and where the footprint of some of a warp's cells leaves the reference's margin: texture moved by whole
and far, noise against noise. Level 0's field equals the oracle's."""
import numpy as np
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200.engine import unpack_field

pytestmark = pytest.mark.gpu


def noise(w, h, seed):
    return np.random.default_rng(seed).integers(0, 256, (h, w)).astype(np.uint8)


@pytest.mark.parametrize("w,h", [(16, 16), (24, 16), (136, 40), (264, 136)])
@pytest.mark.parametrize("content", ["still", "near", "far", "noise"])
def test_field(oracle, w, h, content):
    if content == "noise":
        src, refs = noise(w, h, 1), [noise(w, h, 2), noise(w, h, 3)]
    else:
        d = {"still": 0, "near": 3, "far": 61}[content]
        src = F.textured(w, h, 0, 0)[:h, :w]
        refs = [F.textured(w, h, d, -d)[:h, :w], F.textured(w, h, -d, d // 2)[:h, :w]]
    with E.CudaEngine(w, h) as e:
        e.decide_inter(src, refs, 120)
        for r, ref in enumerate(refs):
            got, exp = unpack_field(e.debug_field(r, 0)), oracle.me_fields(src, ref)[0]
            assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1])
