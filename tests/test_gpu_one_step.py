"""Contractions of up to 16 k at the edges of the rule that gives them to the
kernel of small CTAs (large C, tiny or full matrices of a batch), in every storage
order of the operands, against numpy. k products of a sum: k * 2^-53 of the
absolute values, and the roundings of alpha and beta."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l,m,n", [(1, 1025, 513), (1, 33, 16000), (1, 4100, 2060), (300, 4, 4), (50, 5, 40),
                                   (40, 64, 64), (30, 70, 61), (20, 128, 67), (9, 16, 17)])
@pytest.mark.parametrize("k", [1, 15, 16, 17])
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_against_numpy(cuda, l, m, n, k, beta):
    import torch
    import tblis_b200 as tb
    rng = np.random.default_rng(l + m + n + k)
    lens = dict(l=l, m=m, n=n, k=k)
    ops = [[x for x in s if x != "l" or l > 1] for s in ("lmk", "lkn", "lmn")]
    orders = list(itertools.product(*([p for p in itertools.permutations(o)] for o in ops)))
    for pick in rng.choice(len(orders), min(3, len(orders)), replace=False):
        T, D = [], []
        for labels in orders[pick]:
            x = rng.uniform(-1, 1, [lens[c] for c in labels])
            T.append(x)
            D.append(torch.from_numpy(x).to(cuda))
        ia, ib, ic = ("".join(o) for o in orders[pick])
        if not beta:
            D[2].fill_(float("nan"))
        tb.mult(1.5, D[0], ia, D[1], ib, beta, D[2], ic)
        spec = "%s,%s->%s" % (ia, ib, ic)
        want = 1.5 * np.einsum(spec, T[0], T[1], optimize=True) + (beta * T[2] if beta else 0.0)
        size = 1.5 * np.einsum(spec, abs(T[0]), abs(T[1]), optimize=True) + abs(beta * T[2])
        assert (np.abs(D[2].cpu().numpy() - want) <= (k + 4) * 2.0 ** -52 * size).all(), (ia, ib, ic)


CAPTURED = r"""
import torch
import tblis_b200 as tb
A, B, C = (torch.rand(*s, dtype=torch.float64, device="cuda") for s in ((800, 8), (8, 800), (800, 800)))
s = torch.cuda.Stream()
tb.set_stream(s.cuda_stream)
with torch.cuda.stream(s):
    tb.mult(1.0, A, "ik", B, "kj", 0.0, C, "ij")       # small CTAs; the shape's tables are cached from here on
torch.cuda.synchronize()
C.fill_(1.0)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    tb.mult(1.0, A, "ik", B, "kj", 0.5, C, "ij")       # the process's first call of the dense kernel
g.replay()
torch.cuda.synchronize()
assert bool(((C - (A @ B + 0.5)).abs() <= 12 * 2.0 ** -52 * (A @ B + 0.5)).all())
print("captured ok")
"""


def test_first_dense_call_under_capture(cuda):
    """With the shape's tables cached a call is capturable, whichever kernel it takes."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", CAPTURED], cwd=root, env=dict(os.environ, PYTHONPATH=root),
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "captured ok" in p.stdout, p.stdout[-500:] + p.stderr[-1500:]
