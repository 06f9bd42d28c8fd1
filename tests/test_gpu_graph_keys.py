"""Batches replayed as graphs whose waves look alike but hold different stages: KEY frames alone in a
batch have their intra stage in the slices, outside the graph, KEY frames alone in the first wave of a
batch with references have it inside. In both orders on one engine, each batch of other content: the
records equal the oracle's byte for byte, and a batch launches the kernels that it launches without
graphs."""
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import DecisionMap, first_difference, records_equal

pytestmark = pytest.mark.gpu
W, H = 1272, 824  # 20 x 13 superblocks: a KEY frame alone is decided in two slices

ALONE = {1: [(0, [])], 2: [(0, []), (1, [])]}
MIXED = {1: [(1, []), (0, [1])], 2: [(1, []), (0, []), (0, [1]), (1, [0])]}  # two waves: the KEY frames, the others


@pytest.fixture(scope="module")
def want(oracle):
    p = [F.scene_frame(W, H, 3 * k, -2 * k) for k in range(2)]
    q = lam.lambda_q8(120)
    exp = {(s, tuple(r)): oracle.decide(W, H, p[s], [p[i] for i in r], q)
           for s, r in ((0, []), (1, []), (0, [1]), (1, [0]))}
    return p, exp


def decide(e, jobs):
    """The batch's maps and the kernels it launched."""
    before = e.kernel_launches()
    dms = [DecisionMap() for _ in jobs]
    e.launch_group([s for s, _ in jobs], [r for _, r in jobs], 120, dms=dms)
    e.finish()
    return dms, e.kernel_launches() - before


@pytest.mark.parametrize("first", ["alone", "mixed"])
@pytest.mark.parametrize("keys", [1, 2])
def test_keys_alone_and_in_a_wave(want, keys, first):
    p, exp = want
    batches = [ALONE[keys], MIXED[keys]] if first == "alone" else [MIXED[keys], ALONE[keys]]
    with E.CudaEngine(W, H) as e:
        for k in range(2):
            e.upload(p[k], k)
        for jobs in batches:  # the phase planes are there before any batch's kernels are counted
            decide(e, jobs)
        plain = [decide(e, jobs)[1] for jobs in batches]
        e.set_config(E.CFG_GRAPHS, 1)
        for _ in range(2):
            for jobs, n in zip(batches, plain):
                dms, launched = decide(e, jobs)
                for dm, (s, r) in zip(dms, jobs):
                    w = exp[s, tuple(r)]
                    assert records_equal(dm.records, w), first_difference(dm.records, w)
                assert launched == n
