"""Launches large enough for their superblock stages to run in slices (from 256 superblocks on):
the records equal the oracle's byte for byte whatever the row order, for a KEY frame and an inter
frame, for a group whose slices cross its jobs (replayed as a graph too) and for frames of two sizes
in one batch."""
import pytest

import frames as F
from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.records import DecisionMap, first_difference, records_equal

pytestmark = pytest.mark.gpu
W, H = 1272, 824  # 20 x 13 superblocks: two slices, the boundary inside no row


@pytest.fixture(scope="module")
def want(oracle):
    src, ref = F.scene_frame(W, H, 3, -2), F.scene_frame(W, H)
    q = lam.lambda_q8(120)
    return {"src": src, "ref": ref, "key": oracle.decide(W, H, src, [], q), "inter": oracle.decide(W, H, src, [ref], q),
            "back": oracle.decide(W, H, ref, [src], q)}


def same(got, exp):
    assert records_equal(got, exp), first_difference(got, exp)


@pytest.mark.parametrize("streams", [1, 2, 5, 13])
def test_row_streams(want, streams):
    with E.CudaEngine(W, H) as e:
        e.set_row_streams(streams)
        for kind in ("key", "inter", "key"):
            dm, gate = DecisionMap(), E.RowGate()
            e.launch(want["src"], [] if kind == "key" else [want["ref"]], 120, dm)
            assert sorted(e.row_order()) == list(range(13))
            e.collect(dm, gate)
            same(dm.records, want[kind])


@pytest.mark.parametrize("graphs", [0, 1])
def test_group(want, graphs):
    with E.CudaEngine(W, H) as e:
        e.set_config(E.CFG_GRAPHS, graphs)
        e.upload(want["src"], 0)
        e.upload(want["ref"], 1)
        for rep in range(2):
            dms = [DecisionMap() for _ in range(3)]
            e.launch_group([0, 0, 1], [[1], [], [0]], 120, dms=dms)
            e.launch_group([0], [[1]], 120)  # the same engine again at once, records left on the device
            e.finish()
            for dm, kind in zip(dms, ("inter", "key", "back")):
                same(dm.records, want[kind])


def test_two_sizes(want, oracle):
    w, h = 202, 122
    src, ref = F.scene_frame(w, h, 3, -2), F.scene_frame(w, h)
    with E.CudaEngine(W, H) as a, E.CudaEngine(w, h) as b:
        for e, s, r in ((a, want["src"], want["ref"]), (b, src, ref)):
            e.upload(s, 0)
            e.upload(r, 1)
        dms = [DecisionMap() for _ in range(4)]
        E.launch_multi([(b, 0, [1]), (a, 0, [1]), (a, 1, [0]), (b, 0, [])], 120, dms=dms)
        a.finish()
        b.finish()
        q = lam.lambda_q8(120)
        for dm, exp in zip(dms, (oracle.decide(w, h, src, [ref], q), want["inter"], want["back"],
                                 oracle.decide(w, h, src, [], q))):
            same(dm.records, exp)
