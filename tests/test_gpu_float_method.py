"""Which method a large float contraction runs, and what its report says.

A caller that names FP64 (method 1 or the b200_fp64 configuration) gets FP64; one
that names nothing gets verified moduli, reported as method 6 with 13 moduli and
the 2^-30 that they may differ by. Tolerance: one rounding to float with that, and
k * 2^-53 of the absolute values (FP64).
"""
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
