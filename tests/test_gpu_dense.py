"""The layers' dense products on the tensor cores against fp64, at the edges of tiles, stages, splits and
alignments, and with values that have no bf16 split."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, ta, tb, seed=0, pad=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda a, b: torch.randn(a, b + pad, generator=g, device="cuda")[:, :b]
    A, B = r(*((K, M) if ta else (M, K))), r(*((N, K) if tb else (K, N)))
    return A, B, (A.t() if ta else A).double(), (B.t() if tb else B).double()


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 15, 31), (128, 16, 32), (129, 17, 33), (300, 130, 65), (5, 257, 4),
                                   (2100, 47, 100), (2048, 256, 64), (100, 48, 20000), (256, 256, 4097), (64, 3, 9999)])
def test_dense_product_is_at_least_as_accurate_as_fp32(M, N, K, ta, tb):
    from paramspmm_ae_b200 import ops
    for pad in (0, 1, 4):  # row strides that are and are not multiples of 16 bytes
        A, B, A64, B64 = _operands(M, N, K, ta, tb, pad=pad)
        out = torch.full((M, N + pad), float("nan"), device="cuda")
        got = ops.dense_mm(A, B, ta, tb, out=out[:, :N])
        want = A64 @ B64
        bound = 1e-6 * (A64.abs() @ B64.abs())  # fp32 chains leave about sqrt(K) * 6e-8 of it
        assert bool(((got.double() - want).abs() <= bound).all())
        assert pad == 0 or bool(out[:, N:].isnan().all())
        fp32 = torch.mm(A64.float(), B64.float()).double()
        assert float((got.double() - want).norm()) <= 1.5 * float((fp32 - want).norm()) + 1e-7 * float(want.norm())


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False)])
@pytest.mark.parametrize("side", ["A", "B"])
def test_infinities_and_overflowing_values(ta, tb, side):
    from paramspmm_ae_b200 import ops
    A, B, _, _ = _operands(2600, 40, 70, ta, tb, seed=2)
    t = A if side == "A" else B
    t[3, 5], t[4, 6], t[1, 2] = float("inf"), float("nan"), 3.4e38
    got = ops.dense_mm(A, B, ta, tb)
    want = torch.mm(A.t() if ta else A, B.t() if tb else B)
    torch.testing.assert_close(got, want, rtol=1e-4, atol=1e-3, equal_nan=True)


def test_no_wait_has_run_out():
    import ctypes
    from paramspmm_ae_b200 import _lib
    v = ctypes.c_int32(-1)
    _lib.check(_lib.lib().pspmm_dense_status(ctypes.byref(v)))
    assert v.value == 0


_STALLED = """
import ctypes, sys, torch
sys.path.insert(0, %r)
from paramspmm_ae_b200 import _lib, ops
real = _lib.lib().pspmm_dense_mm
for ta, tb, M, N, K in ((0, 0, 300, 40, 200), (0, 1, 300, 130, 64), (1, 0, 200, 50, 9000), (1, 1, 129, 17, 70),
                        (0, 0, 40000, 256, 300), (1, 0, 40000, 47, 300)):
    A, B = torch.randn(*((K, M) if ta else (M, K)), device="cuda"), torch.randn(*((N, K) if tb else (K, N)), device="cuda")
    out = torch.zeros(M, N + 3, device="cuda")
    _lib.lib().pspmm_dense_mm = _lib.lib().pspmm_dense_mm_stalled
    ops.dense_mm(A, B, ta, tb, out=out[:, :N])
    torch.cuda.synchronize()
    assert ops.dense_status() == 1 and bool(out[:, :N].isnan().all()) and not bool(out[:, N:].any()), (ta, tb, M, N, K)
    _lib.lib().pspmm_dense_mm = real  # the next product finds everything as it should be
    want = (A.t() if ta else A).double() @ (B.t() if tb else B).double()
    assert float((ops.dense_mm(A, B, ta, tb).double() - want).norm()) <= 1e-6 * float(want.norm()), (ta, tb, M, N, K)
print("filled")
"""


def test_a_wait_that_runs_out_leaves_nan_and_the_status():
    """One arrival per stage is withheld, so every wait gives up after 20 ms.  In a process of its own, since the
    status stays set."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", _STALLED % root], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and "filled" in p.stdout, p.stdout[-500:] + p.stderr[-2000:]
