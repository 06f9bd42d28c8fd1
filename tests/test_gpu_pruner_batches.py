"""The pruner's forward and backward passes where their kernels' loops and remainders begin: one or two
samples of a pair, 32 samples a dense CTA, 64 a weight-gradient tile, more samples than resident CTAs;
and buffers that start at any float. The logits (against the restatement in test_gpu_pruner.py) equal
those of each sample alone, bit for bit. The gradients against the numpy restatement with the same BF16
operands: the products are exact in FP32, so what differs is the order of FP32 sums (relative 2^-24 a step over at
most 65,536 steps for the weight gradients, far below) and operands of the backward pass that such a
difference moves across a BF16 rounding boundary (2^-8 of the operand, a small share of them): 2e-3 of a
parameter's gradient norm, as for the other batches."""
import ctypes as C

import numpy as np
import pytest

from celv2_b200 import engine as E
from oracle import pruner_ref as R
from test_gpu_pruner import case, dev, ptr

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("batch,shift", [(1, 0), (2, 1), (31, 2), (33, 3), (297, 1), (901, 0)])
def test_forward_and_backward(batch, shift):
    p, x = case(batch, seed=batch + 100)
    dl = np.random.default_rng(batch).normal(0, 1, (batch, E.PRUNER_OUTPUTS)).astype(np.float32)
    lib, st = E.library(), C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def room(n):  # n floats, `shift` floats past a 16-byte boundary, and a guard behind them
        return torch.full((n + shift + 64,), 7.0, device="cuda")

    def at(t):
        return C.c_void_p(t.data_ptr() + 4 * shift)

    acts, work, grads = room(batch * E.PRUNER_ACTS), room(batch * E.PRUNER_WORK), room(E.PRUNER_PARAMS)
    xt, pt, dlt = room(x.size), room(p.size), room(dl.size)
    for t, v in ((xt, x), (pt, p), (dlt, dl)):
        t[shift:shift + v.size] = dev(v).reshape(-1)
    assert lib.celv2_pruner_forward(at(pt), at(xt), batch, at(acts), st) == 0
    assert lib.celv2_pruner_backward(at(pt), batch, at(acts), at(dlt), at(work), at(grads), st) == 0
    # a sample's logits do not depend on where in a batch it stands: its sums run in one order
    z = acts[shift + batch * (E.PRUNER_ACTS - E.PRUNER_OUTPUTS):shift + batch * E.PRUNER_ACTS].view(batch, -1)
    one = room(E.PRUNER_ACTS)
    for i in sorted({0, 1, batch // 2, batch - 2, batch - 1} & set(range(batch))):
        row = dev(x[i])
        assert lib.celv2_pruner_forward(at(pt), ptr(row), 1, at(one), st) == 0
        assert torch.equal(z[i], one[shift + E.PRUNER_ACTS - E.PRUNER_OUTPUTS:shift + E.PRUNER_ACTS]), i
    _, cache = R.forward(p, x, bf=True)
    got, ref = grads[shift:shift + E.PRUNER_PARAMS].cpu().numpy(), R.backward(p, cache, dl, bf=True)
    o = 0
    for name, shape in R.SHAPES:
        n = int(np.prod(shape))
        err = np.linalg.norm(got[o:o + n] - ref[o:o + n]) / max(np.linalg.norm(ref[o:o + n]), 1e-12)
        assert err < 2e-3, (name, err)
        o += n
    for t, n in ((acts, batch * E.PRUNER_ACTS), (work, batch * E.PRUNER_WORK), (grads, E.PRUNER_PARAMS)):
        assert bool((t[shift + n:] == 7).all()) and bool((t[:shift] == 7).all())  # nothing outside
