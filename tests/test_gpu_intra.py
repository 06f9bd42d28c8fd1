"""The intra stage's SATDs against the oracle's where its launch splits a superblock's work
differently (one, three or nine units, by the launch's superblock count), on content that reaches
every frame-edge rule and both z2 projections; and the plane without margin or word alignment the
allocation-free entry point may be given. Integer work: equal, no tolerance."""
import numpy as np
import pytest

import frames as F
from celv2_b200 import lam
from celv2_b200.engine import CudaEngine
from celv2_b200.records import first_difference, records_equal
from test_zz_no_alloc import noalloc

pytestmark = pytest.mark.gpu


# nine units (1, 8 and 65 superblocks), three (66 and 592), one (593); ragged right and bottom edges
@pytest.mark.parametrize("w,h", [(64, 64), (202, 122), (832, 314), (704, 378), (2048, 1180), (593 * 64 - 8, 24)])
@pytest.mark.parametrize("content", ["noise", "scene"])
def test_intra_units_match_oracle(oracle, w, h, content):
    src = F.noise(w, h, 5) if content == "noise" else F.scene_frame(w, h, 3, -2)
    with CudaEngine(w, h) as e:
        e.decide_intra(src, 120)
        got, cols, rows = e.debug_intra(), e.sb_cols, e.sb_rows
    rng = np.random.default_rng(w)
    corners = {(x, y) for x in (0, cols // 2, cols - 1) for y in (0, rows // 2, rows - 1)}
    for sx, sy in sorted(corners | {(int(rng.integers(cols)), int(rng.integers(rows))) for _ in range(3)}):
        want = oracle.intra_satd_sb(src, sx, sy)
        assert np.array_equal(got[sy * cols + sx][5:], want[5:]), f"superblock ({sx}, {sy})"


@pytest.mark.parametrize("pitch", [208, 211, 214])
def test_unaligned_plane_matches_oracle(oracle, pitch):
    w, h = 202, 122
    src = F.noise(w, h, 9)
    got = noalloc(src, w, h, 120, pitch)
    want = oracle.decide(w, h, src, [], lam.lambda_q8(120))
    assert records_equal(got, want), first_difference(got, want)
