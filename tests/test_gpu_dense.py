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


@pytest.mark.parametrize("M,N", [(256, 256), (100, 256), (256, 47)])
def test_weight_gradients_over_millions_of_nodes(M, N):
    """The product this kernel was built for: K = the nodes of a full-size graph.  Each element is a sum of some
    hundred chains per split and as many splits, every add rounded to nearest: less than fp32 chains leave."""
    from paramspmm_ae_b200 import ops
    A, B, A64, B64 = _operands(M, N, 2_449_029, True, False, seed=5)
    got = ops.dense_mm(A, B, True, False).double()
    want = A64 @ B64
    assert bool(((got - want).abs() <= 1e-7 * (A64.abs() @ B64.abs())).all())
    fp32 = torch.mm(A.t(), B).double()
    assert float((got - want).norm()) <= 1.5 * float((fp32 - want).norm())


@pytest.mark.parametrize("kind", ["plan", "legacy"])
def test_gcn_step_gradients_match_fp64_at_the_steps_own_masks(kind):
    """Three GCN layers on half a million nodes, forward and backward, against fp64 algebra in which the ReLUs
    keep what they kept in the step: without a pre-activation that changes sides, the gradients are sums of
    fp32 products with errors of 2e-7 .. 4e-7 of their norm (six seeds, up to 2.4 M nodes)."""
    from paramspmm_ae_b200 import decider, gnn_conv, ops, pcsr, synth
    dev, n, dims = torch.device("cuda:0"), 500_003, [100, 64, 64, 47]
    g = synth.powerlaw_graph(n, 5_000_000, seed=4, device=dev)
    stats, P = decider.row_stats(g.rowPtr, g.colIdx), {}
    for d in set(dims[1:]):
        plan = decider.choose(stats, d)
        if kind == "plan":
            P[d] = pcsr.pcsr_spmm.from_plan(plan, g.rowPtr, g.colIdx, g.val)
        else:
            rp, tr = ops.split_csr_device(g.rowPtr, 32)
            P[d] = pcsr.pcsr_spmm(None, 1, True, n, g.nnz, rp, g.colIdx, g.val, tr, CF=1, blkWarpNum=8)
    torch.manual_seed(4)
    layers = [gnn_conv.GCNConv(a, b).to(dev) for a, b in zip(dims, dims[1:])]
    X = synth.dense_normal(n, dims[0], 5, dev)
    y = torch.randint(0, dims[-1], (n,), device=dev)
    h, masks = X, []
    for layer in layers:
        h = layer(h, P)
        if layer is not layers[-1]:
            masks.append(h.detach() > 0)
            h = torch.relu(h)
    torch.nn.functional.cross_entropy(h, y).backward()
    A = torch.sparse_csr_tensor(g.rowPtr.long(), g.colIdx.long(), g.val.double(), size=(n, n))
    W = [layer.weights.detach().double() for layer in layers]
    hs = [X.double()]
    for i, w in enumerate(W):
        z = torch.sparse.mm(A, hs[-1] @ w)
        if i < 2:
            hs.append(z * masks[i])
    assert float((h.detach().double() - z).norm()) <= 1e-6 * float(z.norm())
    G = torch.softmax(z, 1)
    G[torch.arange(n, device=dev), y] -= 1
    G /= n
    for i in (2, 1, 0):
        AG = torch.sparse.mm(A, G)
        want = hs[i].t() @ AG
        assert float((layers[i].weights.grad.double() - want).norm()) <= 2e-6 * float(want.norm()), i
        if i:
            G = (AG @ W[i].t()) * masks[i - 1]


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
