"""Which method a large float contraction runs, what its report says, and what it
does without room for the residue planes.

A caller that names FP64 (method 1 or the b200_fp64 configuration) gets FP64; one
that names nothing gets verified moduli, reported as method 6 with 13 moduli and
the 2^-30 that they may differ by. Tolerance: one rounding to float with that, and
k * 2^-53 of the absolute values (FP64).
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

M, N, K = 1700, 1650, 2048


def problem(cuda):
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(11)
    A, B = (torch.empty(s, device=cuda).normal_(generator=g) for s in ((M, K), (K, N)))
    return A, B, torch.full((M, N), float("nan"), device=cuda)


def check(A, B, C, eps):
    a, b = A.double(), B.double()
    want = a @ b
    assert bool(((C.double() - want).abs() <= want.abs() * (2.0 ** -24 + eps) + (a.abs() @ b.abs()) * (K * 2.0 ** -53)).all())


def run(tb, cuda, **kw):
    import torch
    A, B, C = problem(cuda)
    tb.kernel_timer(True)
    r = tb.mult_ex(1.0, A, "ik", B, "kj", 0.0, C, "ij", **kw)
    torch.cuda.synchronize()
    launches = tb.kernel_time("oz_crt_gemm")[1]
    tb.kernel_timer(False)
    tb.synchronize()
    return (A, B, C), r, launches


def test_named_fp64_stays_fp64(cuda):
    import tblis_b200 as tb
    for kw in (dict(method=1), dict(cfg=tb.get_config("b200_fp64"))):
        ops, r, launches = run(tb, cuda, **kw)
        assert launches == 0 and r["method"] == 1 and r["slices"] == 0 and r["est_error"] < 1e-14
        check(*ops, 0.0)


def test_unnamed_reports_moduli(cuda):
    import tblis_b200 as tb
    ops, r, launches = run(tb, cuda)
    assert launches == 1 and r["method"] == 6 and r["slices"] == 13 and r["est_error"] >= 2.0 ** -30
    assert (r["m"] * r["n"], r["k"], r["l"]) == (M * N, K, 1) and r["flops"] == 2.0 * M * N * K
    check(*ops, 2.0 ** -29)


def test_without_room(cuda):
    """No room for the residue planes (13 bytes an element of A): FP64, and the
    report says so; no room for the widened operands either is an error."""
    import tblis_b200 as tb
    limit = tb.lib.tblis_b200_limit_allocations
    limit.argtypes, limit.restype = [ctypes.c_size_t], None
    limit(8 * max(M * K, K * N, M * N))
    try:
        ops, r, launches = run(tb, cuda)
        assert launches == 0 and r["method"] == 1 and r["slices"] == 0
        check(*ops, 0.0)
        limit(4 * M * N)
        with pytest.raises(tb.TblisError) as e:
            run(tb, cuda)
        assert e.value.code == 3
    finally:
        limit(0)
        tb.kernel_timer(False)
    ops, r, launches = run(tb, cuda)
    assert launches == 1 and r["method"] == 6
    check(*ops, 2.0 ** -29)


def test_dense_without_workspace(cuda):
    """A contraction whose plan cuts tiles, without room for their sums."""
    import torch
    import tblis_b200 as tb
    limit = tb.lib.tblis_b200_limit_allocations
    limit.argtypes, limit.restype = [ctypes.c_size_t], None
    for dtype in (torch.float64, torch.complex128):
        m, n, k = 97, 90, 20000
        assert tb.dense_plan(m, n, k, 1, dtype == torch.complex128)["cut"]
        A, B = torch.randn(m, k, dtype=dtype, device=cuda), torch.randn(k, n, dtype=dtype, device=cuda)
        C = torch.full((m, n), float("nan"), dtype=dtype, device=cuda)
        limit(1 << 10)
        try:
            tb.mult(1.0, A, "ik", B, "kj", 0.0, C, "ij")
        finally:
            limit(0)
        assert bool(((C - A @ B).abs() <= 4 * k * 2.0 ** -53 * (A.abs() @ B.abs())).all())
