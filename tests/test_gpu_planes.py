"""The planes kernels at the sizes where their tiles can go wrong: frames whose last tile is one
8-sample column or row wide (level 4's last sample then lies in the tile before), frames smaller than
a tile, and planes whose rows do not fill a tile of stored positions -- through decisions that reach
the margins (content moved by up to 40 pels at every level) against the oracle's, byte for byte, for
8-bit and 10-bit planes, references in one launch and one by one."""
import numpy as np
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import first_difference, records_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(16, 16), (24, 40), (72, 72), (136, 72), (72, 200), (200, 136), (64, 128), (328, 24)])
@pytest.mark.parametrize("depth", [8, 10])
def test_planes_match_oracle(oracle, w, h, depth):
    # noise around a moving scene: every sample of every level takes part in a comparison
    def frame(k):
        a = F.scene_frame(w, h, 13 * k - 40, 20 - 7 * k).astype(np.int32)
        return np.clip(a + F.noise(w, h, k) // 16 - 8, 0, 255).astype(np.uint8)

    planes = [frame(k) for k in range(5)]
    want = oracle.decide(w, h, planes[0], planes[1:], lam.lambda_q8(120))
    if depth == 10:  # rounds back to the 8-bit plane
        give = [(p.astype(np.uint16) * 4 - (p > 0) + (p == 255)).astype(np.uint16) for p in planes]
        for p, q in zip(planes, give):
            assert np.array_equal(oracle.round_to_8bit(q), p)
    else:
        give = planes
    with E.CudaEngine(w, h) as e:
        got = e.decide_inter(give[0], give[1:], 120).records
        assert records_equal(got, want), first_difference(got, want)
        for k, p in enumerate(give):
            e.upload(p, k)
        e.launch_group([0], [[1, 2, 3, 4]], 120, to_host=True)
        got = e.group_records(0)
        assert records_equal(got, want), first_difference(got, want)
