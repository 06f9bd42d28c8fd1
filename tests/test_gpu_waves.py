"""Batches whose jobs are searched and decided in two waves (from 480 superblocks on, at most five
references a superblock) or just not: the records equal the oracle's byte for byte, whichever jobs the
waves fall on (KEY frames alone in one, frames of two engines), replayed as a graph, with keep words,
with sources still on their way to the GPU, and batch upon batch."""
import numpy as np
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import DecisionMap, first_difference, records_equal

pytestmark = pytest.mark.gpu
W, H = 632, 376  # 10 x 6 superblocks


@pytest.fixture(scope="module")
def clip(oracle):
    p = [F.scene_frame(W, H, 3 * k, -2 * k) for k in range(4)]
    q = lam.lambda_q8(120)
    known = {}

    def want(s, refs):
        key = (s, tuple(refs))
        if key not in known:
            known[key] = oracle.decide(W, H, p[s], [p[r] for r in refs], q)
        return known[key]

    return p, want


def check(dms, jobs, want):
    for dm, (s, refs) in zip(dms, jobs):
        exp = want(s, refs)
        assert records_equal(dm.records, exp), first_difference(dm.records, exp)


JOBS = {
    "seven": [(0, [1]), (1, [0]), (0, []), (2, [1]), (1, [2, 0]), (0, [1]), (1, [0])],  # 420 superblocks: one wave
    "eight": [(0, [1]), (1, [0]), (0, []), (2, [1]), (1, [2, 0]), (0, [1]), (1, [0]), (2, [])],
    "keys first": [(0, []), (1, []), (2, []), (0, []), (0, [1]), (1, [0]), (2, [1]), (1, [2, 0])],
    "keys last": [(0, [1]), (1, [0]), (2, [1]), (1, [2, 0]), (0, []), (1, []), (2, []), (0, []), (1, [])],
}


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("jobs", JOBS)
def test_batch(clip, jobs, graphs):
    p, want = clip
    with E.CudaEngine(W, H) as e:
        e.set_config(E.CFG_GRAPHS, graphs)
        for k in range(3):
            e.upload(p[k], k)
        for order in (JOBS[jobs], JOBS[jobs][::-1], JOBS[jobs]):
            dms = [DecisionMap() for _ in order]
            e.launch_group([s for s, _ in order], [r for _, r in order], 120, dms=dms)
            e.launch_group([0] * 8, [[1]] * 8, 120)  # at once, its records left on the device
            e.finish()
            check(dms, order, want)


@pytest.mark.parametrize("nrefs", [1, 3])
def test_fresh_sources(clip, nrefs):
    p, want = clip
    jobs = [(k % 4, [r for r in range(4) if r != k % 4][:nrefs]) for k in range(9)]
    with E.CudaEngine(W, H) as e:
        for _ in range(2):
            got = e.decide_group([p[s] for s, _ in jobs], [[p[r] for r in rs] for _, rs in jobs], 120)
            check(got, jobs, want)


@pytest.mark.parametrize("graphs", [0, 1])
def test_keep_words(clip, graphs):
    p, want = clip
    full = np.full(60, 0xFFFFFFFF, np.uint32)
    with E.CudaEngine(W, H) as e:
        e.set_config(E.CFG_GRAPHS, graphs)
        for k in range(2):
            e.upload(p[k], k)
        for j in (1, 5, 6):
            e.set_keep(j, full)
        jobs = [(j & 1, [1 - (j & 1)]) for j in range(8)]
        dms = [DecisionMap() for _ in jobs]
        e.launch_group([s for s, _ in jobs], [r for _, r in jobs], 120, dms=dms)
        e.finish()
        check(dms, jobs, want)


def test_two_engines(clip, oracle):
    p, want = clip
    w, h = 202, 122
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    small = oracle.decide(w, h, src, [ref], lam.lambda_q8(120))
    with E.CudaEngine(W, H) as a, E.CudaEngine(w, h) as b:
        b.upload(src, 0)
        b.upload(ref, 1)
        for k in range(2):
            a.upload(p[k], k)
        for lead in (a, b):
            jobs = [(lead, 0, [1])] + [(a, j & 1, [1 - (j & 1)]) for j in range(8)] + [(b, 0, [1])]
            dms = [DecisionMap() for _ in jobs]
            E.launch_multi(jobs, 120, dms=dms)
            a.finish()
            b.finish()
            for dm, (e, s, r) in zip(dms, jobs):
                exp = small if e is b else want(s, r)
                assert records_equal(dm.records, exp), first_difference(dm.records, exp)
