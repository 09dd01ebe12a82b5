"""Float contractions large enough for the INT8 cores: every element must be as
good as an FP64 contraction rounded to float, also where the integers lose bits
(wide exponent ranges within a row: recomputed or done in FP64), where results
cancel to zero, and for infinities and NaN.

Bound: one rounding to float, 2^-24 |result|, with 2^-29 of it for what the
verification lets pass, plus the FP64 path's own K 2^-53 |A||B| and, with beta,
the same of the sum's terms.
"""
import pytest

pytestmark = pytest.mark.gpu

M, N, K = 1543, 1290, 2311


def inputs(torch, kind, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(7)
    A = torch.empty(K, M, device=dev).uniform_(-1, 1, generator=g).t()       # m contiguous
    B = torch.empty(N, K, device=dev).uniform_(-1, 1, generator=g).t()       # k contiguous
    if kind == "normal":
        A.normal_(generator=g)
        B.normal_(generator=g)
    elif kind == "spread":                       # 2^-20 .. 2^20 within every row
        A.mul_(torch.exp2(torch.randint(-20, 21, A.shape, generator=g, device=dev).float()))
        B.mul_(torch.exp2(torch.randint(-20, 21, B.shape, generator=g, device=dev).float()))
    elif kind == "graded":                       # a few rows whose products cancel their large entries
        A[:5, 0] = 1e25
        B[0, :] = 0
        A[7, ::2] = 0
        B[1::2, 11] = 0
    elif kind == "blocks":                       # structural zeros: half of C is exactly zero
        A[: M // 2, K // 2:] = 0
        B[: K // 2, : N // 2] = 0
    elif kind == "special":
        A[3, 17] = float("inf")
        A[9, 5] = float("nan")
        B[40, 23] = -float("inf")
        A[100] = 0
        B[:, 77] = 0
        A[200] *= 1e-38
    return A, B


@pytest.mark.parametrize("kind", ["uniform", "normal", "spread", "graded", "blocks", "special"])
@pytest.mark.parametrize("beta", [0.0, -0.75])
def test_every_element(cuda, kind, beta):
    import torch
    import tblis_b200 as tb
    A, B = inputs(torch, kind, cuda)
    C = torch.empty(N, M, device=cuda).uniform_(-1, 1).t()
    alpha = 1.5
    a, b = A.double(), B.double()
    want = alpha * (a @ b) + (beta * C.double() if beta else 0.0)
    size = alpha * (a.abs() @ b.abs()) + abs(beta) * C.double().abs()
    if not beta:
        C.fill_(float("nan"))
    tb.kernel_timer(True)
    tb.mult(alpha, A, "ik", B, "kj", beta, C, "ij")
    torch.cuda.synchronize()
    launches = tb.kernel_time("oz_crt_gemm")[1]
    tb.kernel_timer(False)
    assert launches == 1
    tb.synchronize()
    got = C.double()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    inf = torch.isinf(want)
    assert torch.equal(got[inf], want[inf])
    err = (got - want).abs()
    bound = want.abs() * (2.0 ** -24 + 2.0 ** -29) + size * (K * 2.0 ** -53) + 2.0 ** -149
    bad = finite & ~(err <= bound)
    assert not bad.any(), (int(bad.sum()), float((err / bound)[finite].max()))
    if kind == "blocks" and not beta:
        assert bool((got[: M // 2, : N // 2] == 0).all())


def test_permuted_odd(cuda):
    """A ladder with odd extents and other storage orders."""
    import torch
    import tblis_b200 as tb
    o, v = 31, 51
    g = torch.Generator(device=cuda)
    g.manual_seed(3)
    A = torch.empty(v, v, v, v, device=cuda).normal_(generator=g).permute(2, 0, 3, 1)
    B = torch.empty(o, v, o, v, device=cuda).normal_(generator=g).permute(1, 3, 0, 2)
    C = torch.zeros(v, o, v, o, device=cuda).permute(0, 2, 1, 3)
    tb.kernel_timer(True)
    tb.mult(1.0, A, "abef", B, "efij", 0.0, C, "abij")
    torch.cuda.synchronize()
    launches = tb.kernel_time("oz_crt_gemm")[1]
    tb.kernel_timer(False)
    assert launches == 1
    want = torch.einsum("abef,efij->abij", A.double(), B.double())
    size = torch.einsum("abef,efij->abij", A.double().abs(), B.double().abs())
    assert bool(((C.double() - want).abs() <= want.abs() * (2.0 ** -24 + 2.0 ** -29) + size * (v * v * 2.0 ** -53)).all())
