"""Adds, dots and sums over tensors whose fastest dimensions differ, are short or
ragged, at the edges of the tiles that serve them (extents 1 to a few hundred,
several outer indices to a tile), dense and block-sparse, against numpy.

Adds of alpha = 1 are exact. Other adds round twice; sums of n terms round n
times (block-sparse ones in double precision): n * eps * sum |terms| bounds
them.
"""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {np.float32: 2.0 ** -24, np.complex64: 2.0 ** -24, np.float64: 2.0 ** -53, np.complex128: 2.0 ** -53}


def rand(rng, shape, dtype):
    x = rng.uniform(-1, 1, shape)
    if np.dtype(dtype).kind == "c":
        x = x + 1j * rng.uniform(-1, 1, shape)
    return x.astype(dtype)


def put(torch, cuda, x, order, shift=0):
    """x on the device, stored with dimension order[0] fastest, `shift` elements into its allocation."""
    rev = list(order)[::-1]
    flat = torch.from_numpy(np.ascontiguousarray(x.transpose(rev)).reshape(-1))
    base = torch.zeros(flat.numel() + shift, dtype=flat.dtype, device=cuda)
    base[shift:] = flat.to(cuda)
    strides = [0] * x.ndim
    s = 1
    for d in order:
        strides[d] = s
        s *= x.shape[d]
    return torch.as_strided(base, x.shape, strides, shift)


SHAPES = [(1,), (7, 5), (64, 64), (65, 63), (97, 31), (3, 2, 5, 4), (31, 33, 2, 7), (2, 130, 3, 129), (17, 1, 19, 23),
          (300, 5), (4, 1030), (40, 6, 9, 11)]


@pytest.mark.parametrize("dtype", sorted(EPS, key=str))
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("shift", [0, 1])
def test_add_and_dot(cuda, dtype, shape, shift):
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(sum(shape) + shift)
    n = len(shape)
    idx = "abcd"[:n]
    cx = np.dtype(dtype).kind == "c"
    al, be = (0.75 - 0.5j, -1.25 + 0.25j) if cx else (0.75, -1.25)
    perms = list(itertools.permutations(range(n)))
    for perm in perms if n < 3 else [perms[i] for i in rng.choice(len(perms), 5, replace=False)]:
        X, Y = rand(rng, shape, dtype), rand(rng, shape, dtype)
        A = put(torch, cuda, X, range(n), shift)
        B = put(torch, cuda, Y, perm, shift)
        nan = put(torch, cuda, np.full_like(Y, np.nan), perm, shift)
        tb.add(1.0, A, idx, 0.0, nan, idx)
        assert np.array_equal(nan.cpu().numpy(), X)
        got = tb.dot(A, idx, B, idx, conj_A=cx)
        want = (X.astype(complex).conj() * Y).sum()
        size = float((np.abs(X).astype(float) * np.abs(Y)).sum())
        assert abs(got - want) <= 4 * (X.size + 4) * EPS[dtype] * size
        tb.add(al, A, idx, be, B, idx, conj_A=cx, conj_B=cx)
        want = al * X.conj() + be * Y.conj()
        assert np.abs(B.cpu().numpy() - want).max() <= 16 * EPS[dtype]


@pytest.mark.parametrize("dtype", sorted(EPS, key=str))
@pytest.mark.parametrize("n", [4, 8])
def test_block_sparse(cuda, dtype, n):
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(n)
    o, v = [3, 0, 5, 1, 2, 7, 1, 4][:n], [9, 2, 0, 17, 5, 1, 33, 6][:n]
    irrep = 1 if n == 4 else 0
    mk = lambda lens: tb.DpdTensor(irrep, n, lens, None)
    X, R, V = mk([v, v, o, o]), mk([v, v, o, o]), mk([o, o, v, v])
    host = {}
    for t in (X, R, V):
        host[id(t)] = rand(rng, t.size(), dtype)
        t.data = torch.from_numpy(host[id(t)].copy()).to(cuda)
        t.code = tb._dtype_code(t.data)[0]

    def blocks(t):
        for irr in itertools.product(range(n), repeat=4):
            if irr[0] ^ irr[1] ^ irr[2] ^ irr[3] != irrep or min(t.lens[d][irr[d]] for d in range(4)) == 0:
                continue
            off, L, S = t.block(irr)
            yield irr, np.lib.stride_tricks.as_strided(host[id(t)][off:], L, [s * host[id(t)].itemsize for s in S])
    hx, hr, hv = (dict(blocks(t)) for t in (X, R, V))
    cx = np.dtype(dtype).kind == "c"
    al, be = (0.5 + 0.25j, -1.5j) if cx else (0.5, -1.5)
    dot, size, total, square = 0.0, 0.0, 0.0, 0.0
    for (a, b, i, j), y in hr.items():
        y[...] = al * hx[b, a, j, i].transpose(1, 0, 3, 2) + be * y
        w = hv[i, j, a, b].transpose(2, 3, 0, 1)
        dot += (y.astype(complex) * w).sum()
        size += float((np.abs(y).astype(float) * np.abs(w)).sum())
        total += y.astype(complex).sum()
        square += float((np.abs(y.astype(complex)) ** 2).sum())
    tb.dpd_add(al, X, "baji", be, R, "abij")
    got = R.data.cpu().numpy()
    assert np.abs(got - host[id(R)]).max() <= 16 * EPS[dtype]
    tol = 4 * (got.size * 2.0 ** -53 + 8 * EPS[dtype])
    assert abs(tb.dpd_dot(R, "abij", V, "ijab") - dot) <= tol * size
    assert abs(tb.dpd_reduce(tb.REDUCE_NORM_2, R, "abij")[0] - np.sqrt(square)) <= tol * np.sqrt(square)
    assert abs(tb.dpd_reduce(tb.REDUCE_SUM, R, "abij")[0] - total) <= tol * np.abs(got).sum()
    off, idx = -1, tb.dpd_reduce(tb.REDUCE_MAX, R, "abij")
    assert idx[0] == (got[np.argmax(got.real)] if cx else got.max())
