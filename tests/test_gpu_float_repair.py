"""The elements of a verified float contraction that are recomputed in FP64: a few to
some hundreds of them (below the list's capacity of one element in 2500, and 256),
with permuted storage, a batch label, alpha and beta; and one more than fit, where FP64
does all of C. The number that was listed is asserted, so that the branch that
wrote C is known.

Bound as in the other float tests: one rounding to float, 2^-29 of the value, and
k * 2^-53 of the absolute values.
"""
import pytest

pytestmark = pytest.mark.gpu


def listed(tb):
    import ctypes
    fn = tb.lib.tblis_b200_verified_listed
    fn.restype = ctypes.c_int64
    return fn()


def store(torch, x, order):
    """x stored with dimension order[0] fastest."""
    rev = list(order)[::-1]
    return x.permute(rev).contiguous().permute([rev.index(d) for d in range(x.dim())])


def run(tb, torch, A, B, spec, alpha, beta, orders, cap, few):
    ia, ib, ic = spec
    ein = "%s,%s->%s" % spec
    a, b = A.double(), B.double()
    want = alpha * torch.einsum(ein, a, b)
    size = abs(alpha) * torch.einsum(ein, a.abs().nan_to_num(0, 0, 0), b.abs().nan_to_num(0, 0, 0))
    C = torch.empty(want.shape, device=A.device).uniform_(-1, 1)
    if beta:
        want, size = want + beta * C.double(), size + abs(beta) * C.double().abs()
    else:
        C.fill_(float("nan"))
    A, B, C = store(torch, A, orders[0]), store(torch, B, orders[1]), store(torch, C, orders[2])
    tb.kernel_timer(True)
    tb.mult(alpha, A, ia, B, ib, beta, C, ic)
    torch.cuda.synchronize()
    launches = tb.kernel_time("oz_crt_gemm")[1]
    tb.kernel_timer(False)
    assert launches >= 1
    n = listed(tb)
    assert (0 < n <= cap) if few else n > cap, (n, cap)
    got = C.double()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    inf = torch.isinf(want)
    assert torch.equal(got[inf], want[inf])
    k = 1
    for c, x in zip(ia, a.shape):
        k *= x if c in ib and c not in ic else 1
    fin = torch.isfinite(want)
    bound = want.abs() * (2.0 ** -24 + 2.0 ** -29) + size * (k * 2.0 ** -53) + 2.0 ** -149
    assert bool((((got - want).abs() <= bound) | ~fin).all())
    return n


M, N, K = 3001, 2003, 1511
CAP = M * N // 2500


@pytest.mark.parametrize("orders", [((0, 1), (0, 1), (0, 1)), ((1, 0), (1, 0), (1, 0)), ((0, 1), (1, 0), (1, 0))])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.75, 0.5)])
@pytest.mark.parametrize("kind", ["cancel", "infinite", "nan"])
def test_matrices(cuda, orders, alpha, beta, kind):
    import torch
    import tblis_b200 as tb
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    A = torch.empty(M, K, device=cuda).normal_(generator=g)
    B = torch.empty(K, N, device=cuda).normal_(generator=g)
    if kind == "cancel":
        # row 1234 holds one entry that dwarfs the others and meets zeros in most
        # columns only: those elements lose all their bits to the row's scaling
        A[1234, 77] = 1e25
        B[77] = 1
        B[77, 100:500] = 0
    elif kind == "infinite":
        # reaches the N elements of its row of C
        A[17, 3] = float("inf")
    else:
        A[2000, 1500] = float("nan")
    n = run(tb, torch, A, B, ("ik", "kj", "ij"), alpha, beta, orders, CAP, True)
    assert n >= (400 if kind == "cancel" else N)


def test_batch_label_and_permuted(cuda):
    """Extents 3 x (40 x 37) x (35 x 41) x (31 x 47), every operand in an order of its own."""
    import torch
    import tblis_b200 as tb
    g = torch.Generator(device=cuda)
    g.manual_seed(9)
    A = torch.empty(3, 40, 37, 31, 47, device=cuda).normal_(generator=g)         # l a b e f
    B = torch.empty(3, 31, 47, 35, 41, device=cuda).normal_(generator=g)         # l e f i j
    A[2, 13, 36, 4, 40] = 1e24
    A[1, 0, 5, 30, 0] = -1e26
    B[2, 4, 40] = 0
    B[2, 4, 40, 30:] = 1
    B[1, 30, 0, :, ::2] = 0
    cap = 3 * 40 * 37 * 35 * 41 // 2500
    n = run(tb, torch, A, B, ("labef", "lefij", "laibj"), 0.5, -1.25, ((3, 1, 0, 4, 2), (2, 4, 0, 1, 3), (4, 0, 2, 1, 3)), cap, True)
    assert n >= 30 * 41 + 35 * 20


def test_one_list_too_many(cuda):
    """More elements than the list holds."""
    import torch
    import tblis_b200 as tb
    g = torch.Generator(device=cuda)
    g.manual_seed(6)
    A = torch.empty(M, K, device=cuda).normal_(generator=g)
    B = torch.empty(K, N, device=cuda).normal_(generator=g)
    A[100:104, 9] = 1e25
    B[9, :1000] = 0
    run(tb, torch, A, B, ("ik", "kj", "ij"), 2.0, 0.0, ((1, 0), (0, 1), (0, 1)), CAP, False)
