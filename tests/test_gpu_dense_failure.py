"""Failure detection of the dense FP64 kernel, without any GPU fault.

Every wait of the kernel is bounded. tblis_b200_dense_inject_wait_timeout keeps one
ring stage from ever becoming full and shortens the bound, so that the wait for
it runs out: the CTAs record it, wait for the copies that they issued and return.
tblis_b200_synchronize reports it once (TB_ERR_TIMEOUT, 6), a contraction of host
data reports it itself, and the same contraction is then right on the same context.
"""
import contextlib
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def held_stage(tb, stage=3, seconds=0.05):
    fn = tb.lib.tblis_b200_dense_inject_wait_timeout
    fn.argtypes, fn.restype = [ctypes.c_int, ctypes.c_double], ctypes.c_int
    assert fn(stage, seconds) == 0
    try:
        yield
    finally:
        assert fn(-1, 0.0) == 0


# whole 64 x 64 tiles, 128 x 128 tiles, a cut tile, 128 x 32, and complex ones
CASES = [(700, 700, 300, False), (1500, 1400, 300, False), (97, 97, 20000, False), (5000, 20, 700, False),
         (400, 400, 300, True), (97, 97, 20000, True)]


@pytest.mark.parametrize("m,n,k,cplx", CASES)
def test_wait_runs_out_and_context_recovers(cuda, m, n, k, cplx):
    import torch
    import tblis_b200 as tb
    dt = torch.complex128 if cplx else torch.float64
    A, B = torch.randn(m, k, dtype=dt, device=cuda), torch.randn(k, n, dtype=dt, device=cuda)
    C = torch.zeros(m, n, dtype=dt, device=cuda)
    call = lambda: tb.mult(1.0, A, "ik", B, "kj", 0.0, C, "ij")
    call()
    tb.synchronize()
    with held_stage(tb):
        call()
        with pytest.raises(tb.TblisError) as e:
            tb.synchronize()
        assert e.value.code == 6
    tb.synchronize()                            # reported once
    C.fill_(float("nan"))
    call()
    tb.synchronize()
    assert bool(((C - A @ B).abs() <= 4 * k * 2.0 ** -53 * (A.abs() @ B.abs())).all())


@pytest.mark.parametrize("cplx", [False, True])
def test_host_data_reports_it(cuda, cplx):
    import tblis_b200 as tb
    rng = np.random.default_rng(2)
    A, B = rng.uniform(-1, 1, (300, 512)), rng.uniform(-1, 1, (512, 260))
    if cplx:
        A, B = A + 1j * A[::-1], B - 1j * B[::-1]
    C = np.zeros((300, 260), dtype=A.dtype)
    tb.synchronize()
    with held_stage(tb):
        with pytest.raises(tb.TblisError) as e:
            tb.mult(1.0, A, "ik", B, "kj", 0.0, C, "ij")
        assert e.value.code == 6
    tb.synchronize()
    tb.mult(1.0, A, "ik", B, "kj", 0.0, C, "ij")
    assert (np.abs(C - A @ B) <= 4 * 512 * 2.0 ** -53 * (np.abs(A) @ np.abs(B))).all()


GROUPED = r"""
import numpy as np, torch
import tblis_b200 as tb
from tests.test_gpu_dense_failure import held_stage
dev = torch.device("cuda:0")
rng = np.random.default_rng(9)
items = []
for m, n, k in ((96, 80, 2048), (64, 64, 1024), (300, 270, 1500)):
    A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))
    items.append((1.0, torch.from_numpy(A).to(dev), "ik", torch.from_numpy(B).to(dev), "kj", 0.0,
                  torch.zeros((m, n), dtype=torch.float64, device=dev), "ij"))
batch = tb.PreparedBatch(items)
batch.run()
tb.synchronize()
with held_stage(tb):
    batch.run()
    try:
        tb.synchronize()
        raise SystemExit("no timeout reported")
    except tb.TblisError as e:
        assert e.code == 6, e.code
tb.synchronize()
for it in items:
    it[6].fill_(float("nan"))
batch.run()
tb.synchronize()
for _, A, _, B, _, _, C, _ in items:
    assert bool(((C - A @ B).abs() <= 4 * A.shape[1] * 2.0 ** -53 * (A.abs() @ B.abs())).all())
print("grouped timeout ok")
"""


def test_grouped_wait_runs_out_and_context_recovers(cuda):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, TBLIS_B200_GEMM_VARIANT="6", PYTHONPATH=root)
    r = subprocess.run([sys.executable, "-c", GROUPED], cwd=root, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "grouped timeout ok" in r.stdout, (r.stdout[-2000:], r.stderr[-3000:])
