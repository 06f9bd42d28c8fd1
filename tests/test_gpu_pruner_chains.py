"""The pruner's convolution weight gradients at a batch of many samples a CTA. The tensor cores' accumulators
round towards zero, so a sum of terms of one sign loses a part of itself with every step that adds to it: no chain
of theirs may grow with the batch. Everything is positive here (parameters, features, gradients); the reference is
the sum in FP64 of the gradients of 256 samples at a time, which hold one sample a chain and are otherwise the
same numbers (a sample's values do not depend on the batch it stands in).
The bound: a chain of 32 samples has at most 128 steps (W2: 64 positions a sample, 16 a step); at a rounding of
2^-23 each they lose sum(i / 128) 2^-23 = 64.5 * 2^-23 = 7.7e-6 of the sum; the chains meet in FP32 atomics, some
4,144 of them, whose round-to-nearest errors add up as a random walk, sqrt(4144 / 3) * 2^-24 = 2.2e-6: 1e-5 of a
gradient's norm. (Chains over all of a CTA's samples, 443, lost 5.9e-5 of W1's and 1.3e-4 of W2's.)"""
import ctypes as C

import numpy as np
import pytest

from celv2_b200 import engine as E
from oracle import pruner_ref as R

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BATCH, PART = 131072, 256


def gradients(params, x, dl):
    n = x.shape[0]
    acts = torch.empty(n * E.PRUNER_ACTS, device="cuda")
    work = torch.empty(n * E.PRUNER_WORK, device="cuda")
    grads = torch.empty(E.PRUNER_PARAMS, device="cuda")
    lib, st = E.library(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = [C.c_void_p(t.data_ptr()) for t in (params, x, acts, dl, work, grads)]
    assert lib.celv2_pruner_forward(p[0], p[1], n, p[2], st) == 0
    assert lib.celv2_pruner_backward(p[0], n, p[2], p[3], p[4], p[5], st) == 0
    return grads.double()


def test_weight_gradient_chains_are_bounded():
    torch.manual_seed(5)
    params = torch.rand(E.PRUNER_PARAMS, device="cuda") * 0.04 + 0.01
    x = torch.rand(BATCH, E.PRUNER_FEATURES, device="cuda") + 0.5
    dl = torch.rand(BATCH, E.PRUNER_OUTPUTS, device="cuda") + 0.5
    want = torch.zeros(E.PRUNER_PARAMS, device="cuda", dtype=torch.float64)
    for b in range(0, BATCH, PART):
        want += gradients(params, x[b:b + PART].contiguous(), dl[b:b + PART].contiguous())
    got = gradients(params, x, dl)
    torch.cuda.empty_cache()
    o = 0
    for name, shape in R.SHAPES:
        n = int(np.prod(shape))
        g, w = got[o:o + n], want[o:o + n]
        o += n
        if name in ("W1", "W2", "W3"):
            err = ((g - w).norm() / w.norm()).item()
            print(name, err)
            assert err < 1e-5, (name, err)


def test_bias_gradients_meet_in_few_additions():
    """The last layer's biases: FP32 sums of 131,072 positive numbers, in FP64 the sum of them. At most 64 CTAs' four
    row groups are added in a row to the same number: a random walk of 256 round-to-nearest errors (0.29 of an ulp, the
    ulp at most 2^-23 of the sum so far), 0.29 * 2^-23 * sqrt(256 / 3) = 3.2e-7 of a bias; the threads' own sums before it
    (512 in a row, 256 of them side by side) add a tenth of that. 6e-7 leaves the walk its spread. (2,048 CTAs' lost
    1.0e-6.)"""
    torch.manual_seed(6)
    params = torch.rand(E.PRUNER_PARAMS, device="cuda") * 0.04 + 0.01
    x = torch.rand(BATCH, E.PRUNER_FEATURES, device="cuda") + 0.5
    dl = torch.rand(BATCH, E.PRUNER_OUTPUTS, device="cuda") + 0.5
    got = gradients(params, x, dl)[-E.PRUNER_OUTPUTS:]
    want = dl.double().sum(0)
    torch.cuda.empty_cache()
    assert ((got - want).norm() / want.norm()).item() < 6e-7
