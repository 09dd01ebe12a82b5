"""The dense FP64 kernel (real and complex) at the sizes where its tiles and its
work split change: edges of the 128 x 128, 64 x 64 and 128 x 32 tiles and of the
16-wide k step, tiles cut over many SMs, batches, and every gather (along the
rows or along k, in pairs or not, rows in blocks), against numpy in the same
arithmetic type.

Tolerance: a sum of k products in any order has a normwise error below
k * 2^-53 * || |A||B| || (complex products: 2 more roundings each); the bound used
is that with the elementwise |A||B|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stored(rng, lens, order, cplx):
    """A tensor with len(lens) labels stored with order[0] fastest."""
    x = rng.uniform(-1, 1, [lens[c] for c in reversed(order)])
    if cplx:
        x = x + 1j * rng.uniform(-1, 1, x.shape)
    return x.transpose([order[::-1].index(c) for c in sorted(order)]), "".join(sorted(order))


def device(torch, cuda, x, shift=0):
    """The array's storage on the device, `shift` elements into an allocation."""
    order = np.argsort([-s for s in x.strides], kind="stable")
    flat = np.ascontiguousarray(x.transpose(order)).reshape(-1)
    base = torch.zeros(flat.size + shift, dtype=torch.complex128 if np.iscomplexobj(x) else torch.float64, device=cuda)
    base[shift:] = torch.from_numpy(flat).to(cuda)
    es = x.itemsize
    return torch.as_strided(base, x.shape, [s // es for s in x.strides], shift)


def check(cuda, lens, sA, sB, sC, cplx=False, alpha=1.0, beta=0.0, conj=(False, False), shift=0, seed=0):
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(seed)
    A, iA = stored(rng, lens, sA, cplx)
    B, iB = stored(rng, lens, sB, cplx)
    C, iC = stored(rng, lens, sC, cplx)
    a = A.conj() if conj[0] else A
    b = B.conj() if conj[1] else B
    spec = "%s,%s->%s" % (iA, iB, iC)
    want = alpha * np.einsum(spec, a, b, optimize=True)
    size = np.einsum(spec, np.abs(a), np.abs(b), optimize=True)
    if beta:
        want = want + beta * C
    k = np.prod([lens[c] for c in iA if c in iB and c not in iC], dtype=float)
    dC = device(torch, cuda, C if beta else np.full_like(C, np.nan), shift)
    dA, dB = device(torch, cuda, A, shift), device(torch, cuda, B, shift)
    kw = dict(conj_A=conj[0], conj_B=conj[1])
    tb.mult(alpha, dA, iA, dB, iB, beta, dC, iC, **kw)
    torch.cuda.synchronize()
    got = dC.cpu().numpy()
    err = np.linalg.norm(got - want)
    bound = (k + 8) * 2.0 ** -53 * (abs(alpha) * np.linalg.norm(size) + abs(beta) * np.linalg.norm(C)) * (4 if cplx else 1)
    assert err <= bound, (err, bound)


EDGES = [(1, 1, 1), (16, 8, 16), (17, 9, 15), (64, 64, 33), (65, 63, 17), (127, 129, 31), (128, 128, 16),
         (300, 32, 700), (5, 400, 90), (31, 31, 4097), (130, 260, 1000), (700, 16, 50), (1300, 1100, 48)]


@pytest.mark.parametrize("mnk", EDGES)
@pytest.mark.parametrize("layout", ["mk,kn", "mk,nk", "km,kn", "km,nk"])
@pytest.mark.parametrize("shift", [0, 1])
def test_matrices(cuda, mnk, layout, shift):
    m, n, k = mnk
    sA, sB = layout.split(",")
    check(cuda, {"m": m, "n": n, "k": k}, sA, sB, "mn", alpha=-1.5, beta=0.5, shift=shift, seed=m + n + k)


@pytest.mark.parametrize("mnk", EDGES)
@pytest.mark.parametrize("layout", ["mk,kn", "km,nk"])
@pytest.mark.parametrize("conj", [(False, False), (True, False), (False, True), (True, True)])
def test_complex_matrices(cuda, mnk, layout, conj):
    m, n, k = (min(x, 500) for x in mnk)
    sA, sB = layout.split(",")
    check(cuda, {"m": m, "n": n, "k": k}, sA, sB, "nm", True, 0.75 - 0.5j, 0.25 + 1j, conj, seed=m + n + k)
    check(cuda, {"m": m, "n": n, "k": k}, sA, sB, "mn", True, 2.0, 0.0, conj, seed=m + n + k)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("lens", [dict(a=11, b=9, e=7, i=5, j=6, m=10), dict(a=24, b=20, e=18, i=16, j=12, m=14),
                                  dict(a=33, b=3, e=40, i=2, j=31, m=1), dict(a=2, b=40, e=5, i=37, j=17, m=3)])
@pytest.mark.parametrize("orders", [("imae", "ejbm", "abij"), ("aeim", "mbej", "aibj"), ("miea", "bjem", "jbia"),
                                    ("eima", "jmbe", "ibaj")])
def test_permuted_ring(cuda, cplx, lens, orders):
    check(cuda, lens, *orders, cplx=cplx, alpha=1.0, beta=1.0, seed=sum(lens.values()))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("l,m,n,k", [(3, 40, 50, 60), (17, 130, 20, 35), (200, 5, 6, 7)])
def test_batch_label(cuda, cplx, l, m, n, k):
    check(cuda, dict(l=l, m=m, n=n, k=k), "mkl", "lkn", "nlm", cplx=cplx, seed=l)


def test_complex_not_16_byte_aligned(cuda):
    """A complex tensor at an 8-byte boundary takes the four real contractions."""
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(3)
    z = lambda *s: rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)
    A, B = z(30, 41), z(41, 23)
    dA = torch.zeros(2 * A.size + 1, dtype=torch.float64, device=cuda)
    dA[1:] = torch.from_numpy(A.reshape(-1).view(np.float64)).to(cuda)
    dB = torch.from_numpy(B).to(cuda)
    dC = torch.zeros(30, 23, dtype=torch.complex128, device=cuda)
    va = tb._View(dB, 1.0)                                  # a complex view; its pointer and shape are set by hand
    va.len[0], va.len[1], va.stride[0], va.stride[1] = 30, 41, 41, 1
    va.t.data = dA.data_ptr() + 8
    vb, vc = tb._View(dB), tb._View(dC, 0.0)
    tb.lib.tblis_tensor_mult(None, None, va.ref, b"ik", vb.ref, b"kj", vc.ref, b"ij")
    tb._check()
    torch.cuda.synchronize()
    assert np.linalg.norm(dC.cpu().numpy() - A @ B) <= 41 * 2.0 ** -50 * np.linalg.norm(np.abs(A) @ np.abs(B))
