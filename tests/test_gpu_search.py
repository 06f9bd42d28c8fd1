"""The motion search where cells need no search and where they just do: SADs of 0 to a few around the
penalty a whole pel costs, ties everywhere, and centre SATDs around what a quarter-pel move has to save,
with CTAs of seven cells (small levels) and of thirty. The fields of every level and the records equal
the oracle's."""
import numpy as np
import pytest

from celv2_b200 import engine as E
from celv2_b200 import lam
from celv2_b200.engine import unpack_field
from celv2_b200.records import first_difference, records_equal

pytestmark = pytest.mark.gpu


def sparse(w, h, seed, share, step, shift=0):
    """Flat tiles of three levels, a share of the samples off by up to `step`."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    p = 100 + 40 * (((x - shift) // 48 + y // 40) % 3)
    p = p + np.where(rng.random((h, w)) < share, rng.integers(-step, step + 1, (h, w)), 0)
    return np.clip(p, 0, 255).astype(np.uint8)


@pytest.mark.parametrize("w,h,refs", [(136, 72, 2), (1272, 824, 3)])
@pytest.mark.parametrize("share,step", [(0.0, 1), (0.02, 1), (0.05, 3), (0.3, 1)])
def test_cells_with_little_to_search(oracle, w, h, refs, share, step):
    src = sparse(w, h, 1, share, step)
    planes = [sparse(w, h, 2 + k, share, step, shift=3 * k) for k in range(refs)]
    want = oracle.decide(w, h, src, planes, lam.lambda_q8(120))
    with E.CudaEngine(w, h) as e:
        got = e.decide_inter(src, planes, 120).records
        fields = [[unpack_field(e.debug_field(r, l)) for l in range(5)] for r in range(refs)]
    for r in range(refs):
        exp = oracle.me_fields(src, planes[r])
        for l in range(5):
            assert np.array_equal(fields[r][l][0], exp[l][0]) and np.array_equal(fields[r][l][1], exp[l][1]), (r, l)
    assert records_equal(got, want), first_difference(got, want)
