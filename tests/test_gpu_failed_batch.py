"""A batch that fails on the host between its slices: nothing of it runs any more when the call returns, the
records of the batch before stay readable, and the batch that follows at once -- on the same descriptors,
queues and buffers -- equals the oracle byte for byte. The failure is asked for (debug_fail), on the host alone."""
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import DecisionMap, first_difference, records_equal

pytestmark = pytest.mark.gpu
W, H = 1272, 824  # 20 x 13 superblocks: two slices a frame


@pytest.fixture(scope="module")
def want(oracle):
    p = [F.scene_frame(W, H, 3 * k, -2 * k) for k in range(2)]
    q = lam.lambda_q8(120)
    exp = {(s, tuple(r)): oracle.decide(W, H, p[s], [p[i] for i in r], q) for s, r in ((0, []), (0, [1]), (1, [0]))}
    return p, exp


def check(dms, jobs, exp):
    for dm, (s, r) in zip(dms, jobs):
        assert records_equal(dm.records, exp[s, tuple(r)]), first_difference(dm.records, exp[s, tuple(r)])


FAILS = [(0, [1]), (1, [0]), (0, [])]  # two waves, of two and four slices
NEXT = [(1, [0]), (0, []), (0, [1])]


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("slice_", [0, 1, 4])
def test_group(want, slice_, graphs):
    p, exp = want
    with E.CudaEngine(W, H) as e:
        e.set_config(E.CFG_GRAPHS, graphs)
        for k in range(2):
            e.upload(p[k], k)
        for _ in range(2):
            e.launch_group([0], [[1]], 120, to_host=True)  # into the engine's own buffer
            e.debug_fail(slice_)
            with pytest.raises(RuntimeError, match="debug_fail"):
                e.launch_group([s for s, _ in FAILS], [r for _, r in FAILS], 120, dms=[DecisionMap() for _ in FAILS])
            dms = [DecisionMap() for _ in NEXT]
            got = e.group_records(0)
            e.launch_group([s for s, _ in NEXT], [r for _, r in NEXT], 120, dms=dms)
            e.finish()
            assert records_equal(got, exp[0, (1,)])
            check(dms, NEXT, exp)


@pytest.mark.parametrize("slice_", [0, 2])
def test_two_engines(want, oracle, slice_):
    p, exp = want
    w, h = 202, 122
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    small = oracle.decide(w, h, src, [ref], lam.lambda_q8(120))
    with E.CudaEngine(W, H) as a, E.CudaEngine(w, h) as b:
        b.upload(src, 0)
        b.upload(ref, 1)
        for k in range(2):
            a.upload(p[k], k)
        for lead, other in ((a, b), (b, a), (a, b)):
            jobs = [(lead, 0, [1]), (other, 0, [1]), (a, 1, [0])]
            lead.debug_fail(slice_)
            with pytest.raises(RuntimeError, match="debug_fail"):
                E.launch_multi(jobs, 120, dms=[DecisionMap() for _ in jobs])
            dms = [DecisionMap() for _ in jobs]
            E.launch_multi(jobs, 120, dms=dms)
            a.finish()
            b.finish()
            for dm, (e, s, r) in zip(dms, jobs):
                w_ = small if e is b else exp[s, tuple(r)]
                assert records_equal(dm.records, w_), first_difference(dm.records, w_)


@pytest.mark.parametrize("inter", [False, True])
def test_frame(want, inter):
    p, exp = want
    refs = [1] if inter else []
    with E.CudaEngine(W, H) as e:
        for _ in range(2):
            e.debug_fail(1)
            with pytest.raises(RuntimeError, match="debug_fail"):
                e.launch(p[0], [p[r] for r in refs], 120, DecisionMap(), ref_keys=refs or None)
            got = [e.decide_inter(p[0], [p[r] for r in refs], 120, ref_keys=refs or None)]
            check(got, [(0, refs)], exp)
