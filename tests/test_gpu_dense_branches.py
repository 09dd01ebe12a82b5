"""Every tile shape and work split of the dense FP64 kernel, real and complex: whole
waves of tiles before cut ragged ones, all tiles cut, none cut, 128 x 32 tiles, and
exchanged operands. That the plan sends a case where it is meant to go is
asserted for 148 SMs (what the plan takes on another GPU is not).

Tolerance as in the other tests of the kernel: k * 2^-53 of the absolute values
(complex products: four times that).
"""
import numpy as np
import pytest

from tests.test_gpu_dense_kernel import check

pytestmark = pytest.mark.gpu

T128, T64, TALL = (128, 128), (64, 64), (128, 32)

# m, n, k, complex, tile, exchanged, cut, whole waves before the cut tiles
CASES = [
    (2305, 2180, 500, False, T128, False, True, True),
    (1300, 1100, 900, False, T128, False, True, False),
    (1500, 1400, 300, False, T128, False, False, None),
    (900, 800, 700, False, T64, False, True, False),
    (2000, 1300, 300, False, T64, False, False, None),
    (2500, 12, 900, False, TALL, False, True, False),
    (30000, 20, 60, False, TALL, False, False, None),
    (12, 2500, 900, False, TALL, True, True, False),
    (20, 30000, 100, False, TALL, True, False, None),
    (2000, 1301, 300, True, T128, False, True, True),
    (1301, 601, 1100, True, T128, False, True, False),
    (30000, 20, 60, True, T128, False, False, None),
    (400, 400, 300, True, T64, False, True, False),
    (1300, 1100, 48, True, T64, False, False, None),
    (2500, 12, 900, True, TALL, False, True, False),
    (12, 2500, 900, True, TALL, True, True, False),
    (5, 400, 4000, True, TALL, True, True, False),
]


@pytest.mark.parametrize("m,n,k,cplx,tile,exchanged,cut,waves", CASES)
@pytest.mark.parametrize("layout", ["mk,kn,mn", "km,nk,nm"])
def test_branch(cuda, m, n, k, cplx, tile, exchanged, cut, waves, layout):
    import torch
    import tblis_b200 as tb
    sA, sB, sC = layout.split(",")
    beta = 0.5
    p = tb.dense_plan(m, n, k, 1, cplx, beta, 148)
    assert p["tile"] == tile and p["exchanged"] == exchanged and p["cut"] == cut, p
    if waves is not None:
        assert (p["whole"] > 0) == waves, p
    if torch.cuda.get_device_properties(cuda).multi_processor_count != 148:
        pytest.skip("the plan is for 148 SMs")
    lens = {"m": m, "n": n, "k": k}
    conjs = [(False, True), (True, False)] if cplx else [(False, False)]
    for conj in conjs:
        for shift in (0, 1):
            check(cuda, lens, sA, sB, sC, cplx=cplx, alpha=0.75 - 0.5j if cplx else -1.5,
                  beta=0.25 + 1j if cplx else beta, conj=conj, shift=shift, seed=m + n)
