"""The dense grouped path's workspaces, which all plans share: a dozen plans hold no
more than four, and plans on several streams and threads that meet in them give
what they give alone. In a child process with that path forced.

Tolerance: k * 2^-53 of the absolute values.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import threading
import torch
import tblis_b200 as tb

dev = torch.device("cuda:0")
g = torch.Generator(device=dev)
g.manual_seed(1)

def plan(n):
    # three GEMMs with cut tiles, extents of its own
    items, size = [], []
    for m, k in ((90 + n, 6000), (260 - n, 2500), (30, 9000 + n)):
        A, B = (torch.randn(*s, dtype=torch.float64, device=dev, generator=g) for s in ((m, k), (k, 110)))
        C = torch.zeros(m, 110, dtype=torch.float64, device=dev)
        items.append((1.0, A, "ik", B, "kj", 0.0, C, "ij"))
        size.append((A @ B, k * 2.0 ** -53 * (A.abs() @ B.abs())))
    return tb.PreparedBatch(items), items, size

def check(p):
    for it, (want, bound) in zip(p[1], p[2]):
        assert bool(((it[6] - want).abs() <= bound).all())

plans = [plan(n) for n in range(12)]
for p in plans[:1]:
    p[0].run()
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
for p in plans:
    r = p[0].run()
    assert r["n"] == 6, r
tb.synchronize()
held = free - torch.cuda.mem_get_info()[0]
for p in plans:
    check(p)
# a workspace is 39 MB; the plans' own tables are below 2 MB each
assert held < 4 * 39e6 + 12 * 2e6, held

streams = [torch.cuda.Stream() for _ in range(6)]
for rep in range(30):
    for i, p in enumerate(plans):
        for it in p[1]:
            it[6].fill_(float("nan"))
    torch.cuda.synchronize()
    for i, p in enumerate(plans):
        tb.set_stream(streams[(i * (rep + 1)) % 6].cuda_stream)
        p[0].run()
    torch.cuda.synchronize()
    for p in plans:
        check(p)
tb.set_stream(0)

errors = []
def work(t):
    try:
        s = torch.cuda.Stream()
        tb.set_stream(s.cuda_stream)
        for rep in range(40):
            for p in plans[3 * t:3 * t + 3]:
                p[0].run()
        s.synchronize()
        tb.synchronize()
    except Exception as e:
        errors.append(e)
for p in plans:
    for it in p[1]:
        it[6].fill_(float("nan"))
torch.cuda.synchronize()
threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not errors, errors
for p in plans:
    check(p)
print("workspaces ok", held)
"""


def test_plans_share_workspaces(cuda):
    env = dict(os.environ, TBLIS_B200_GEMM_VARIANT="6", PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0 and "workspaces ok" in p.stdout, p.stdout[-500:] + p.stderr[-2500:]
