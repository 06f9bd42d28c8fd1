"""The inter stage's per-reference bests against the oracle's records where its kernel splits differently:
launches of no more units than SMs, of a few times as many, and of more (four, two, one group of threads
a unit), distinct motion vectors from one to all hundred of a superblock (one pass, several, odd counts),
windows that run past the plane's margin (sizes at which the search reaches it), byte for byte."""
import numpy as np
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import first_difference, records_equal

pytestmark = pytest.mark.gpu


def content(kind, w, h, k):
    if kind == "flat":  # one vector
        return np.full(((h + 7) & ~7, (w + 7) & ~7), 90, np.uint8)
    if kind == "noise":  # every cell its own vector
        return F.noise(w, h, 50 + k)
    return F.scene_frame(w, h, 9 * k, -5 * k)


@pytest.mark.parametrize("kind", ["flat", "noise", "scene"])
@pytest.mark.parametrize("w,h,refs", [(64, 64, 1), (328, 200, 7), (640, 328, 5), (904, 584, 7)])
def test_bests_match_oracle(oracle, kind, w, h, refs):
    planes = [content(kind, w, h, k) for k in range(refs + 1)]
    want = oracle.decide(w, h, planes[0], planes[1:], lam.lambda_q8(100))
    with E.CudaEngine(w, h) as e:
        for chunk in (64, 8):
            e.set_config(E.CFG_INTER_CHUNK, chunk)
            got = e.decide_inter(planes[0], planes[1:], 100).records
            assert records_equal(got, want), (chunk, first_difference(got, want))
