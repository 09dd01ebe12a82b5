"""The dense grouped path (forced by TBLIS_B200_GEMM_VARIANT in a child process)
on batches and block-sparse contractions whose groups sit at the edges of its
tiles and whose tiles are cut over several CTAs, against numpy; the default
choice of path on the same inputs.

Tolerance: k * 2^-53 times the product of the absolute values, elementwise norms.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import itertools, random, sys
import numpy as np, torch
import tblis_b200 as tb

def check(got, want, size, k, what):
    err = np.linalg.norm(got - want)
    assert err <= (k + 8) * 2.0 ** -53 * np.linalg.norm(size), (what, err)

rnd = random.Random(5)
rng = np.random.default_rng(5)
for lo, hi, count in ((1, 6, 40), (2, 13, 60), (4, 32, 30), (30, 40, 2)):
    for beta in (0.0, -0.5):
        items, host = [], []
        for _ in range(count):
            l = {c: rnd.randint(lo, hi) for c in "abefij"}
            ia, ib, ic = ("".join(rnd.sample(s, 4)) for s in ("abef", "efij", "abij"))
            A, B, C = (rng.uniform(-1, 1, [l[c] for c in s]) for s in (ia, ib, ic))
            host.append((A, ia, B, ib, C, ic))
            items.append((1.5, torch.from_numpy(A).cuda(), ia, torch.from_numpy(B).cuda(), ib, beta,
                          torch.from_numpy(C if beta else np.full_like(C, np.nan)).cuda(), ic))
        for rep in range(2):
            if rep:
                for it, h in zip(items, host):
                    it[6].copy_(torch.from_numpy(h[4]))
            r = tb.mult_batch(items)
            for (A, ia, B, ib, C, ic), it in zip(host, items):
                s = "%s,%s->%s" % (ia, ib, ic)
                want = 1.5 * np.einsum(s, A, B, optimize=True) + (beta * C if beta else 0)
                size = 1.5 * np.einsum(s, abs(A), abs(B), optimize=True) + abs(beta * C)
                check(it[6].cpu().numpy(), want, size, A.size, (lo, hi, s))
print("batch variant", r["n"])
for n, o, v in ((4, [3, 1, 4, 2], [9, 14, 5, 11]), (8, [2, 0, 1, 3, 1, 1, 2, 1], [5, 3, 0, 7, 2, 6, 4, 9])):
    for lay in (0, 3, 5):
        for ib, lb in (("efij", [v, v, o, o]), ("jeif", [o, v, o, v])):
            mk = lambda l: tb.DpdTensor(0, n, l, None, lay)
            T = A, B, C = mk([v] * 4), mk(lb), mk([v, v, o, o])
            h = {}
            for t in T:
                h[id(t)] = rng.uniform(-1, 1, t.size())
                t.data = torch.from_numpy(h[id(t)].copy()).cuda()
            def blk(t, irr):
                off, L, S = t.block(irr)
                return np.lib.stride_tricks.as_strided(h[id(t)][off:], L, [8 * s for s in S])
            size = np.abs(h[id(C)])
            for a, b, i in itertools.product(range(n), repeat=3):
                j = a ^ b ^ i
                if min(v[a], v[b], o[i], o[j]) == 0:
                    continue
                c = blk(C, (a, b, i, j))
                c *= 0.25
                for e in range(n):
                    f = e ^ a ^ b
                    irr = {"e": e, "f": f, "i": i, "j": j}
                    if min(v[e], v[f]) == 0:
                        continue
                    c += np.einsum("abef,%s->abij" % ib, blk(A, (a, b, e, f)), blk(B, [irr[x] for x in ib]))
            r = tb.dpd_mult(1.0, A, "abef", B, ib, 0.25, C, "abij")
            err = np.linalg.norm(C.data.cpu().numpy() - h[id(C)])
            k = sum(v) ** 2
            assert err <= k * 2.0 ** -53 * k * np.sqrt(C.size()), (n, lay, ib, err)
print("dpd variant", r["n"])
"""


@pytest.mark.parametrize("variant", ["6", ""])
def test_batches_and_blocks(cuda, variant):
    env = dict(os.environ)
    env.pop("TBLIS_B200_GEMM_VARIANT", None)
    if variant:
        env["TBLIS_B200_GEMM_VARIANT"] = variant
    p = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout[-500:] + p.stderr[-1500:]
    if variant:
        assert "batch variant 6" in p.stdout and "dpd variant 6" in p.stdout
