"""The autotuner's choice of the inter stage's chunk, from stage times as a launch without keep words gives them:
32 unless 64 is faster by more than the times' own scatter (the two are one setting to such a launch, and
pruned batches run the faster with 32)."""
import pytest

from celv2_b200 import engine as E
from celv2_b200 import tune


class FakeEngine:
    def __init__(self, inter_ms):
        self.config, self.inter_ms, self.runs = {}, inter_ms, 0

    def set_config(self, key, value):
        self.config[key] = value

    def stage_timing(self, enable):
        pass

    def stage_times(self):
        self.runs += 1
        t = {name: (1.0, 1) for name in E.STAGE_NAMES}
        t["inter"] = (self.inter_ms[self.config.get(E.CFG_INTER_CHUNK, 64)] * (1 + 1e-3 * (self.runs % 3)), 1)
        return t


@pytest.mark.parametrize("ms32,ms64,chunk", [(10.0, 10.0, 32), (10.0, 9.9, 32), (10.0, 9.5, 64), (9.0, 10.0, 32)])
def test_inter_chunk(ms32, ms64, chunk):
    e = FakeEngine({32: ms32, 64: ms64})
    chosen = tune.autotune_run(e, lambda: None)
    assert chosen["inter_chunk"] == chunk and e.config[E.CFG_INTER_CHUNK] == chunk
