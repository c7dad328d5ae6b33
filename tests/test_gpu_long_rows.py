"""Rows of an unsplit layout that are longer than 64 entries: the kernels cut them over the GPU; everything
else stays with one lane group."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(lengths, n_cols, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n_cols, k, replace=False)) for k in lengths] + [[]]).astype(np.int32)
    return rp, ci, rng.random(len(ci), dtype=np.float32)


LAYOUTS = {
    "around the threshold": [63, 0, 64, 65, 3, 66, 0, 0, 129, 1],
    "long rows back to back": [600] * 9 + [0, 5] + [513] * 4,
    "one row holds all": [0, 0, 4097, 0],
    "first and last": [5000] + [2] * 700 + [5000],
    "short rows between hubs": ([1, 0, 2, 900] * 40),
}


@pytest.mark.parametrize("dim", [1, 6, 16, 47, 64, 132])
@pytest.mark.parametrize("name", sorted(LAYOUTS))
def test_long_rows_match_the_oracle(oracle, name, dim):
    from paramspmm_ae_b200 import ops
    dev = torch.device("cuda:0")
    n_cols = 6001
    rp, ci, v = _matrix(LAYOUTS[name], n_cols, 3)
    n = len(rp) - 1
    rng = np.random.default_rng(4)
    B = rng.uniform(-1, 1, (n_cols, dim)).astype(np.float32)
    t = lambda x: torch.from_numpy(x).to(dev)
    rpd, cid, vd, Bd = t(rp), t(ci), t(v), t(B)
    out = torch.full((n, dim), float("nan"), device=dev)
    ops.spmm_into(out, Bd, rpd, cid, vd)
    np.testing.assert_allclose(out.cpu().numpy(), oracle.spmm_csr(rp, ci, v, B), rtol=1e-5, atol=1e-4)
    for V in (2, 3):
        rpb, cb, vb = ops.bcsr_from_csr(torch.from_numpy(rp), torch.from_numpy(ci), torch.from_numpy(v), n_cols, V)
        nb = rpb.shape[0] - 1
        out = torch.full((nb * V, dim), float("nan"), device=dev)
        ops.spmm_into(out, Bd, rpb.to(dev), cb.to(dev), vb.to(dev), V=V)
        np.testing.assert_allclose(out[:n].cpu().numpy(), oracle.spmm_csr(rp, ci, v, B), rtol=1e-5, atol=1e-4)
    A = rng.uniform(-1, 1, (n, dim)).astype(np.float32)
    got = ops.csr_sddmm(t(A), Bd, rpd, cid, vd, 1, 4)
    np.testing.assert_allclose(got.cpu().numpy(), oracle.sddmm_csr(rp, ci, A, B), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("dim", [4, 32, 64, 132, 256])
@pytest.mark.parametrize("softmax", [True, False])
@pytest.mark.parametrize("name", sorted(LAYOUTS))
def test_long_rows_of_the_fused_aggregation(oracle, name, dim, softmax):
    from paramspmm_ae_b200 import ops
    dev = torch.device("cuda:0")
    n_cols = 6001
    rp, ci, _ = _matrix(LAYOUTS[name], n_cols, 5)
    n = len(rp) - 1
    rng = np.random.default_rng(6)
    A, B, V = ((rng.uniform(-1, 1, (k, dim)) / np.sqrt(dim)).astype(np.float32) for k in (n, n_cols, n_cols))
    t = lambda x: torch.from_numpy(x).to(dev)
    want = oracle.agnn_aggregate(rp, ci, A, B, 2.0, softmax)
    got = ops.agnn_fused(t(A), t(B), t(rp), t(ci), 2.0, softmax)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-5, atol=1e-4)
    rps, tr = ops.split_csr(torch.from_numpy(rp), 7)  # hundreds of pieces per row: the merge takes whole thread blocks
    got = ops.agnn_fused(t(A), t(B), rps.to(dev), t(ci), 2.0, softmax, target_row=tr.to(dev), n_out_rows=n)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-5, atol=1e-4)
    got = ops.agnn_fused(t(A), t(B), t(rp), t(ci), 2.0, softmax, V=t(V)).double().cpu().numpy()
    for r in range(n):
        c = ci[rp[r]:rp[r + 1]]
        s = 2.0 * B[c].astype(np.float64) @ A[r].astype(np.float64)
        w = s if not softmax else np.exp(s - s.max(initial=-np.inf)) / max(np.exp(s - s.max(initial=-np.inf)).sum(), 1e-300)
        np.testing.assert_allclose(got[r], w @ V[c].astype(np.float64), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("dim", [8, 64, 100])
def test_sums_of_long_rows_have_a_fixed_order(dim):
    """Equal columns stay bitwise equal and a second call gives the same bits, rows that span several
    shares of the entries included."""
    from paramspmm_ae_b200 import ops
    dev = torch.device("cuda:0")
    rp, ci, v = _matrix([30000, 3, 700, 20000] + [70] * 500 + [25000], 40001, 7)
    t = [torch.from_numpy(x).to(dev) for x in (rp, ci, v)]
    B = torch.rand(40001, 1, device=dev).expand(-1, dim).contiguous()
    a = torch.empty(len(rp) - 1, dim, device=dev)
    ops.spmm_into(a, B, *t)
    assert bool((a == a[:, :1]).all())
    for _ in range(5):
        b = torch.empty_like(a)
        ops.spmm_into(b, B, *t)
        assert torch.equal(a, b)


@pytest.mark.parametrize("offset, part", [(0, 1), (4, 1), (8, 1), (0, 2)])
def test_scratch_that_cannot_be_used_is_not(oracle, offset, part):
    """Partial sums are stored 16 bytes at a time: scratch off that boundary, or half of what is asked for,
    leaves the plain walk, with the same product."""
    import ctypes
    from paramspmm_ae_b200 import _lib
    dev, dim = torch.device("cuda:0"), 64
    rp, ci, v = _matrix([5000, 3, 700, 2] * 3, 6001, 8)
    n = len(rp) - 1
    B = np.random.default_rng(9).uniform(-1, 1, (6001, dim)).astype(np.float32)
    t = [torch.from_numpy(x).to(dev) for x in (rp, ci, v, B)]
    need = ctypes.c_size_t(0)
    _lib.check(_lib.lib().pspmm_spmm_scratch_bytes(n, len(ci), dim, 1, ctypes.byref(need)))
    scratch = torch.full((need.value + 64,), 255, dtype=torch.uint8, device=dev)
    out = torch.full((n, dim), float("nan"), device=dev)
    _lib.check(_lib.lib().pspmm_spmm_csr_ws(*(x.data_ptr() for x in t), out.data_ptr(), n, 6001, len(ci), dim, dim, dim, None,
                                            None, None, 0, scratch.data_ptr() + offset, need.value // part,
                                            torch.cuda.current_stream().cuda_stream))
    np.testing.assert_allclose(out.cpu().numpy(), oracle.spmm_csr(rp, ci, v, B), rtol=1e-5, atol=1e-4)
    assert bool((scratch[need.value + offset:] == 255).all())


def test_positions_beyond_32_bits():
    """Long rows of almost 2^31 entries: the positions that shares are counted in (entries plus one per row)
    pass 2^31.  Values of 0 and 1 make every share's sum exact; a hub's fewer than 200 shares are then
    added in fp32, 2^-24 each, 1.2e-5 in all.  A share that is lost or taken twice moves a row by 0.5 %."""
    from paramspmm_ae_b200 import ops
    dev = torch.device("cuda:0")
    n, n_cols, nnz, hubs = 2_000_003, 4096, 2_147_400_000, [0, 17, 400_000, 400_001, 999_999, 2_000_002]
    ln = (torch.arange(n) % 3 == 0).long()
    ln[hubs] = 0
    ln[hubs] = (nnz - int(ln.sum())) // len(hubs)
    ln[hubs[-1]] += nnz - int(ln.sum())
    rp = torch.cat([torch.zeros(1, dtype=torch.int64), ln.cumsum(0)])
    assert int(rp[-1]) == nnz and int(ln[hubs].sum()) + n > 2**31
    ci = torch.arange(nnz, dtype=torch.int32, device=dev).bitwise_and_(n_cols - 1)
    B = torch.randint(0, 2, (n_cols, 4), generator=torch.Generator().manual_seed(2)).float()
    B[:, 0] = 1.0
    upto = torch.cat([torch.zeros(1, 4, dtype=torch.float64), B.double().cumsum(0)])  # sums of the first k columns
    total = lambda e: (e // n_cols).double()[:, None] * upto[-1] + upto[e % n_cols]
    want = (total(rp[1:]) - total(rp[:-1])).numpy()
    rpd, Bd = rp.int().to(dev), B.to(dev)
    out = torch.full((n, 4), float("nan"), device=dev)
    ops.spmm_into(out, Bd, rpd, ci, None)
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=2e-5)
    A = torch.zeros(n, 4, device=dev)
    A[:, 0] = 1.0  # every score is one
    got = ops.agnn_fused(A, Bd, rpd, ci, 1.0, False)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2e-5)


@pytest.mark.parametrize("dim", [4, 64])
def test_ranges_that_end_near_the_index_limit(dim):
    """A piece of 300,000 entries beside pieces of three whose entries lie 180,000 below 2^31: their groups run
    along to the longest range of the warp, past 2^31.  (The row pointer starts high; small whole values
    make every sum exact.)"""
    from paramspmm_ae_b200 import ops
    dev, n_cols, first = torch.device("cuda:0"), 4096, 2_147_000_000
    ln = torch.tensor([300_000, 3, 3, 0, 5, 3, 1, 3, 3, 40, 3])
    rp = first + torch.cat([torch.zeros(1, dtype=torch.int64), ln.cumsum(0)])
    n, nnz = len(ln), int(rp[-1])
    assert nnz < 2**31 <= nnz + 300_000
    ci = torch.arange(nnz, dtype=torch.int32, device=dev).bitwise_and_(n_cols - 1)
    g = torch.Generator().manual_seed(3)
    B = torch.randint(0, 2, (n_cols, dim), generator=g).float()
    B[:, 0] = 1.0
    A = torch.randint(0, 4, (n, dim), generator=g).float()
    cols, row = ci[first:].cpu().long(), torch.repeat_interleave(torch.arange(n), ln)
    e0 = torch.zeros(n, dim)
    e0[:, 0] = 1.0  # every score is one
    want = torch.zeros(n, dim).index_add_(0, row, B[cols])
    target = torch.arange(n, dtype=torch.int32, device=dev)
    rpd, Ad, Bd = rp.int().to(dev), A.to(dev), B.to(dev)
    got = ops.agnn_fused(e0.to(dev), Bd, rpd, ci, 1.0, False, target_row=target, n_out_rows=n)
    assert torch.equal(got.cpu(), want)
    got = ops.agnn_fused(e0.to(dev), Bd, rpd, ci, 1.0, False)
    assert torch.equal(got.cpu(), want)
    scores = (A[row] * B[cols]).sum(1)
    val = torch.empty(nnz, device=dev)
    got = ops.csr_split_sddmm(Ad, Bd, rpd, ci, val, target, 1, 8)[first:]
    assert torch.equal(got.cpu(), scores)
    got = ops.csr_sddmm(Ad, Bd, rpd, ci, val, 1, 8)[first:]
    assert torch.equal(got.cpu(), scores)


@pytest.mark.parametrize("rows", [1, 511, 512, 513, 32768, 32769])
@pytest.mark.parametrize("dim", [16, 47, 64, 68])
def test_long_rows_beside_the_segments(rows, dim):
    """Row counts on both sides of what a share looks at by itself (64 x 512 rows): first, last and neighbouring rows long,
    repeated calls on one scratch-sized allocation, rows of the threshold's length."""
    from paramspmm_ae_b200 import ops
    dev = torch.device("cuda")
    n_cols = max(rows, 700)
    ln = torch.zeros(rows, dtype=torch.int64)
    ln[::7] = 3
    ln[rows // 2:rows // 2 + 3] = torch.tensor([64, 65, 600])[: min(3, rows - rows // 2)]
    ln[0], ln[-1] = 300, 700
    rp = torch.cat([torch.zeros(1, dtype=torch.int64), ln.cumsum(0)]).to(torch.int32).to(dev)
    gen = torch.Generator().manual_seed(rows + dim)
    ci = torch.cat([torch.randperm(n_cols, generator=gen)[:k].sort().values for k in ln.tolist() if k]).to(torch.int32).to(dev)
    val = torch.rand(ci.shape[0], generator=gen).to(dev)
    X = torch.randn(n_cols, dim, generator=gen).to(dev)
    r = torch.repeat_interleave(torch.arange(rows, device=dev), ln.to(dev))
    terms = val.double()[:, None] * X.double()[ci.long()]
    want = torch.zeros(rows, dim, dtype=torch.float64, device=dev).index_add_(0, r, terms)
    scale = torch.zeros(rows, dim, dtype=torch.float64, device=dev).index_add_(0, r, terms.abs())
    first = None
    for _ in range(5):
        got = ops.csr_spmm(X, rp, ci, val, 1, 8)[:rows]
        assert bool(((got.double() - want).abs() <= 1e-5 * scale + 1e-12).all())
        first = got if first is None else first
        assert torch.equal(got, first)


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("rows, mean", [(1536, 3), (4099, 9), (8193, 40), (8193, 80)])
def test_own_look_and_its_limits(rows, mean, offset):
    """Shares that look for long rows themselves, four row pointers at a time: row pointers off that boundary and more entries
    than that is done for; long rows at the edges of a look's 512, of its quarters and of the matrix."""
    from paramspmm_ae_b200 import ops
    dev, dim, n_cols = torch.device("cuda:0"), 32, 4000
    ln = torch.full((rows,), mean)
    for r in (0, 1, 3, 4, 127, 128, 511, 512, 1023, rows - 2, rows - 1):
        ln[r] = 65 + r % 300
    rp = torch.zeros(rows + 1, dtype=torch.int64)
    rp[1:] = ln.cumsum(0)
    buf = torch.zeros(rows + 4, dtype=torch.int32, device=dev)
    ptr = buf[offset:offset + rows + 1]
    ptr.copy_(rp)
    assert ptr.data_ptr() % 16 == 4 * offset
    gen = torch.Generator().manual_seed(rows)
    ci = torch.randint(0, n_cols, (int(rp[-1]),), generator=gen).int().to(dev)
    val, X = torch.rand(ci.shape[0], generator=gen).to(dev), torch.randn(n_cols, dim, generator=gen).to(dev)
    r = torch.repeat_interleave(torch.arange(rows, device=dev), ln.to(dev))
    terms = val.double()[:, None] * X.double()[ci.long()]
    want = torch.zeros(rows, dim, dtype=torch.float64, device=dev).index_add_(0, r, terms)
    scale = torch.zeros(rows, dim, dtype=torch.float64, device=dev).index_add_(0, r, terms.abs())
    out = torch.full((rows, dim), float("nan"), device=dev)
    for _ in range(3):
        ops.spmm_into(out, X, ptr, ci, val)
        # (sums of up to 364 terms in another order: 1e-5 of the terms' absolute sum)
        assert bool(((out.double() - want).abs() <= 1e-5 * scale + 1e-12).all())
