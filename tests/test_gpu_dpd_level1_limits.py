"""Block-sparse adds, dots and sums of tensors with more dimensions than a kernel's
index space holds, but which fold to fewer (as dense calls do), and float sums
whose terms leave float's range.

Adds are exact; dots and sums of n terms are in double precision (n * 2^-53) and
rounded to the element type at the end.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {np.float32: 2.0 ** -24, np.complex64: 2.0 ** -24, np.float64: 2.0 ** -53}


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


@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
@pytest.mark.parametrize("size", [1e25, 1e-25, 1.0])
def test_float_sums_in_double(cuda, dtype, size):
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(3)
    lens = [[3, 5], [7, 2], [4, 6]]
    n = tb.DpdTensor(0, 2, lens, None).size()
    x = rng.uniform(0.5, 1, n) * size
    if np.dtype(dtype).kind == "c":
        x = x + 1j * rng.uniform(0.5, 1, n) * size
    x = x.astype(dtype)
    X = dpd(tb, torch, cuda, lens, x)
    w = x.astype(np.complex128)
    norm, total = np.linalg.norm(w), np.abs(w).sum()
    # nothing but the last rounding is in float
    tol = EPS[dtype] * 1.01 + n * 2.0 ** -53
    assert abs(tb.dpd_reduce(tb.REDUCE_NORM_2, X, "abc")[0] - norm) <= tol * norm
    assert abs(tb.dpd_reduce(tb.REDUCE_SUM_ABS, X, "abc")[0] - total) <= tol * total
