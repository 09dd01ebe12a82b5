"""Infinities in complex contractions: a factor of zero leaves its product out,
so a real alpha or beta acts on each part by itself and an infinite (or
overflowing) part does not turn the other into NaN. Tiles done whole, cut over
several SMs and the four real contractions of unaligned elements.

The expected parts are sums and products in the same arithmetic: NaN and
infinities have to agree, finite parts to k * 2^-50 of the absolute values.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALARS = [1.0, -2.0, 0.5 - 0.25j, 1.5j]


def times(s, re, im):
    """s*(re + i im) by parts, without the products by a zero part of s."""
    s = complex(s)
    r = [t for t in ((s.real * re,) if s.real else ()) + ((-s.imag * im,) if s.imag else ())]
    i = [t for t in ((s.real * im,) if s.real else ()) + ((s.imag * re,) if s.imag else ())]
    return (sum(r[1:], r[0]), sum(i[1:], i[0])) if r else (0 * np.ones_like(re), 0 * np.ones_like(im))


@pytest.mark.parametrize("mnk", [(40, 33, 20), (64, 64, 5000), (301, 270, 90), (1200, 1100, 40)])
@pytest.mark.parametrize("where", ["A", "B", "C", "overflow"])
@pytest.mark.parametrize("shift", [0, 1])
def test_infinite_parts(cuda, mnk, where, shift):
    import torch
    import tblis_b200 as tb
    m, n, k = mnk
    rng = np.random.default_rng(m)
    A, B, C0 = (rng.uniform(0.5, 1, s) + 1j * rng.uniform(0.5, 1, s) for s in ((m, k), (k, n), (m, n)))
    if where == "A":
        A[3, 5] = complex(np.inf, 1)
        A[m - 1, k - 1] = complex(0.5, -np.inf)
    elif where == "B":
        B[2, n - 1] = complex(0.75, np.inf)
    elif where == "C":
        C0[4, 7] = complex(np.inf, 2)
        C0[m - 1, n - 2] = complex(1, -np.inf)
    else:
        # real part 0.9e308 - 0.9e308, imaginary part 1.8e308
        A[6, 3] = complex(1, 1) * 1e155
        B[3] = complex(1, 1) * 0.9e153
        A[:6, 3] = A[7:, 3] = 0.5
    with np.errstate(all="ignore"):
        re, im = A.real @ B.real - A.imag @ B.imag, A.real @ B.imag + A.imag @ B.real
        size = np.abs(A) @ np.abs(B)

    def put(x, off):
        # elements off a 16-byte boundary take the four real contractions
        base = torch.zeros(2 * x.size + 2, dtype=torch.float64, device=cuda)
        base[off:off + 2 * x.size] = torch.from_numpy(np.ascontiguousarray(x).reshape(-1).view(np.float64).copy())
        return base

    bufA, bufB = put(A, shift), put(B, 0)
    proto = torch.empty(1, 1, dtype=torch.complex128, device=cuda)

    def view(buf, off, shape, scalar):
        v = tb._View(proto, scalar)
        v.len[0], v.len[1], v.stride[0], v.stride[1] = shape[0], shape[1], shape[1], 1
        v.t.data = buf.data_ptr() + 8 * off
        return v

    over = where == "overflow"
    for alpha in [1.0] if over else SCALARS:
        for beta in [0.0, 1.0] if over else [0.0] + SCALARS:
            bufC = put(C0, 0)
            va, vb, vc = view(bufA, shift, (m, k), alpha), view(bufB, 0, (k, n), 1.0), view(bufC, 0, (m, n), beta)
            tb.lib.tblis_tensor_mult(None, None, va.ref, b"ik", vb.ref, b"kj", vc.ref, b"ij")
            tb._check()
            got = bufC.cpu().numpy()[:2 * m * n].reshape(m, n, 2)
            with np.errstate(all="ignore"):
                wr, wi = times(alpha, re, im)
                if beta:
                    br, bi = times(beta, C0.real, C0.imag)
                    wr, wi = wr + br, wi + bi
                bound = (k + 8) * 2.0 ** -50 * (abs(alpha) * size + abs(beta) * np.abs(C0))
            for g, w in ((got[..., 0], wr), (got[..., 1], wi)):
                assert np.array_equal(np.isnan(g), np.isnan(w)), (alpha, beta)
                inf = np.isinf(w)
                assert np.array_equal(g[inf], w[inf]) and not np.isinf(g[~inf]).any(), (alpha, beta)
                fin = np.isfinite(w) & np.isfinite(bound)
                assert (np.abs(g - w)[fin] <= bound[fin]).all(), (alpha, beta)
