"""Block-sparse adds, dots and sums of tensors with more dimensions than a kernel's
index space holds, but which fold to fewer (as dense calls do).

Adds are exact; dots and sums of n terms are in double precision (n * 2^-53).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dpd(tb, torch, cuda, lens, x):
    t = tb.DpdTensor(0, len(lens[0]), lens, torch.from_numpy(x).to(cuda))
    assert t.size() == x.size
    return t


@pytest.mark.parametrize("ndim", [12, 13, 16])
@pytest.mark.parametrize("turn", [False, True])
def test_many_dimensions(cuda, ndim, turn):
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(ndim)
    lens = [[2]] * ndim
    x, y = rng.uniform(-1, 1, 2 ** ndim), rng.uniform(-1, 1, 2 ** ndim)
    X, Y = dpd(tb, torch, cuda, lens, x), dpd(tb, torch, cuda, lens, y)
    la = "abcdefghijklmnop"[:ndim]
    # the turned tensor has its halves exchanged: each half stays contiguous
    lb = la[5:] + la[:5] if turn else la
    want = x.reshape(2 ** 5, -1).T.reshape(-1) if turn else x
    tb.dpd_add(1.0, X, la, 0.0, Y, lb)
    assert np.array_equal(Y.data.cpu().numpy(), want)
    Z = dpd(tb, torch, cuda, lens, y)
    zt = y.reshape(-1, 2 ** 5).T.reshape(-1) if turn else y          # Z in X's order
    assert abs(tb.dpd_dot(X, la, Z, lb) - x @ zt) <= 2 ** ndim * 2.0 ** -53 * (abs(x) @ abs(zt))
    assert abs(tb.dpd_reduce(tb.REDUCE_NORM_2, X, la)[0] - np.linalg.norm(x)) <= 2 ** ndim * 2.0 ** -53 * np.linalg.norm(x)
    assert abs(tb.dpd_reduce(tb.REDUCE_SUM, X, la)[0] - x.sum()) <= 2 ** ndim * 2.0 ** -53 * abs(x).sum()
