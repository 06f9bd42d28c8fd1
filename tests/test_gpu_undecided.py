"""A batch one of whose kernels gave up a wait: no call hands out its records -- not the row waits, so no row
reaches a consumer, and not the second call either -- and the next batch is decided as ever. The mark that such
a kernel leaves is set from the host (debug_fail(-1)); no kernel is made to wait."""
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import DecisionMap, records_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(202, 122), (1272, 824)])  # one slice, two
def test_rows_are_not_published(oracle, w, h):
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    want = oracle.decide(w, h, src, [ref], lam.lambda_q8(120))
    with E.CudaEngine(w, h) as e:
        for _ in range(2):
            dm, gate = DecisionMap(), E.RowGate()
            e.launch(src, [ref], 120, dm)
            e.debug_fail(-1)
            with pytest.raises(RuntimeError, match="not decided"):
                e.collect(dm, gate)
            assert gate.ready_rows() == 0
            with pytest.raises(RuntimeError, match="not decided"):
                gate.wait_row(0, 1.0)
            with pytest.raises(RuntimeError, match="not decided"):
                e.finish()
            e.set_config(E.CFG_INTER_CHUNK, 64)  # reads no records
            assert records_equal(e.decide_inter(src, [ref], 120).records, want)


def test_untold_before_the_next_launch(oracle):
    w, h = 202, 122
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    with E.CudaEngine(w, h) as e:
        e.launch(src, [ref], 120, DecisionMap())
        e.debug_fail(-1)
        with pytest.raises(RuntimeError, match="not decided"):  # the caller has not heard of it yet
            e.launch(src, [ref], 120, DecisionMap())
        assert records_equal(e.decide_inter(src, [ref], 120).records, oracle.decide(w, h, src, [ref], lam.lambda_q8(120)))


def test_groups(oracle):
    w, h = 202, 122
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    want = oracle.decide(w, h, src, [ref], lam.lambda_q8(120))
    with E.CudaEngine(w, h) as a, E.CudaEngine(w, h) as b:
        for e in (a, b):
            e.upload(src, 0)
            e.upload(ref, 1)
        for _ in range(2):
            a.launch_group([0], [[1]], 120, to_host=True)
            a.debug_fail(-1)
            for _ in range(2):
                for read in (a.group_records, a.sb_costs):
                    with pytest.raises(RuntimeError, match="not decided"):
                        read(0)
            E.launch_multi([(b, 0, [1]), (a, 0, [1])], 120, to_host=True)
            assert records_equal(a.group_records(0), want) and records_equal(b.group_records(0), want)
