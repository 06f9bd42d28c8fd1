"""The engine's stream stands behind all of a launch: once it has run dry, the records of a frame decided
in several slices are in host memory, as those of a frame decided in one."""
import numpy as np
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import DecisionMap, records_equal

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("w,h", [(202, 122), (1272, 824)])  # one slice, two
@pytest.mark.parametrize("inter", [False, True])
def test_records_are_there_when_the_stream_is_dry(oracle, w, h, inter):
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    refs = [ref] if inter else []
    want = oracle.decide(w, h, src, refs, lam.lambda_q8(120))
    with E.CudaEngine(w, h) as e:
        stream = torch.cuda.ExternalStream(e.stream())
        for _ in range(3):
            dm = DecisionMap()
            e.launch(src, refs, 120, dm)
            stream.synchronize()
            got = dm.records.copy()
            dm.records.view(np.uint8)[:] = 0xEE  # so that the next pass of this memory shows nothing old
            e.finish()
            assert records_equal(got, want)
