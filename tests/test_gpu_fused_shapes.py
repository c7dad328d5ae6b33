"""The fused aggregation at widths that leave lanes idle and rows that end inside a gather batch: a lane's registers
then hold an earlier batch's rows, which must not reach a sum even where they are infinite."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows_of_one_to_nine(n, inf_col, seed):
    """CSR of n rows with 1..9 distinct columns; about half of the rows have `inf_col` in their first batch of four."""
    g = np.random.default_rng(seed)
    cols = []
    for i in range(n):
        c = np.sort(g.choice(np.arange(inf_col + 1, n), 1 + i % 9, replace=False))
        if g.random() < 0.5:
            c[0] = inf_col
        cols.append(c)
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])])
    return torch.from_numpy(rp.astype(np.int32)), torch.from_numpy(np.concatenate(cols).astype(np.int32)), cols


def _reference(cols, A, B, V, beta, softmax):
    out = np.zeros((len(cols), V.shape[1]))
    with np.errstate(all="ignore"):
        for i, c in enumerate(cols):
            s = beta * (B[c] @ A[i])
            if softmax:
                # (a row whose scores are all -inf has no weight to give, as in the kernel: its sums are empty)
                s = np.exp(s - s.max()) if s.max() > -np.inf else np.zeros_like(s)
                s = s / max(s.sum(), 1e-300) if s.sum() == s.sum() else s
            out[i] = (s[:, None] * V[c]).sum(0)
    return out


@pytest.mark.parametrize("dim", [4, 20, 36, 52, 100, 132, 252])
@pytest.mark.parametrize("softmax", [False, True])
@pytest.mark.parametrize("sep", [False, True])
def test_infinite_rows_reach_only_the_rows_that_hold_them(dim, softmax, sep):
    from paramspmm_ae_b200 import ops
    n, inf_col = 301, 5
    g = torch.Generator().manual_seed(dim)
    A = torch.rand(n, dim, generator=g) / dim + 0.01
    B = torch.rand(n, dim, generator=g) - 0.3
    V = torch.rand(n, dim, generator=g) + 0.5 if sep else B
    rp, ci, cols = _rows_of_one_to_nine(n, inf_col, dim)
    for target, sign in ((B, 1.0), (B, -1.0)) + (((V, 1.0),) if sep else ()):
        keep = target[inf_col].clone()
        target[inf_col, dim // 2] = sign * float("inf")
        want = _reference(cols, A.double().numpy(), B.double().numpy(), V.double().numpy(), 0.9, softmax)
        args = [t.cuda() for t in (A, B, rp, ci)]
        kw = dict(V=V.cuda()) if sep else {}
        layouts = [(args[2], {})]
        rps, tr = ops.split_csr(rp, 4)
        layouts.append((rps.cuda(), dict(target_row=tr.cuda(), n_out_rows=n)))
        for ptr, extra in layouts:
            got = ops.agnn_fused(args[0], args[1], ptr, args[3], 0.9, softmax, **kw, **extra).cpu().double().numpy()
            clean = np.array([inf_col not in c for c in cols])
            # sums of up to nine terms: a few fp32 roundings of the terms' absolute sum
            np.testing.assert_allclose(got[clean], want[clean], rtol=2e-5, atol=2e-6)
            if not extra:  # (pieces of a cut row meet with weights of their own: 0 * inf there is not the plain row's)
                np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want))
        target[inf_col] = keep


@pytest.mark.parametrize("dim", [4, 16, 24, 32, 40, 64, 68, 128, 132, 256])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("pairs", [0, 40, 20000])
def test_scores_kept_between_the_layer_passes(dim, split, pairs):
    """The scores that the forward leaves and the backward that takes them, against dense fp64 algebra: empty,
    sparse and long-row patterns, every default shape of the two kernels."""
    from paramspmm_ae_b200 import ops, synth
    dev = torch.device("cuda:0")
    n = 301
    g = synth.powerlaw_graph(n, pairs, seed=4, self_loops=pairs != 0)
    rp, ci = g.rowPtr.to(dev), g.colIdx.to(dev)
    rows = torch.repeat_interleave(torch.arange(n, device=dev), (rp[1:] - rp[:-1]).long())
    cols = ci.long()
    gen = torch.Generator(device=dev).manual_seed(5)
    X, G = (torch.randn(n + (0 if split else 2), dim, device=dev, generator=gen) / dim ** 0.5 for _ in range(2))
    beta = torch.tensor([0.7], device=dev)
    tr = None
    if split:
        rp, tr = ops.split_csr_device(rp, 9)
    scores = torch.full((ci.shape[0],), float("nan"), device=dev)
    out = ops.agnn_layer_forward(X, rp, ci, beta, tr, scores)
    assert torch.equal(out, ops.agnn_layer_forward(X, rp, ci, beta, tr))
    X64, G64 = X.double(), G.double()
    # dot products of dim terms below 1: a few roundings of their absolute sum
    want = 0.7 * (X64[rows] * X64[cols]).sum(1)
    bound = 1e-6 * (X64[rows] * X64[cols]).abs().sum(1)
    assert bool(((scores.double() - want).abs() <= bound).all())
    D, d_beta = ops.agnn_layer_backward(None, G, rp, ci, None, tr, scores=scores)
    terms = scores.double()[:, None] * G64[cols]
    want = torch.zeros(n, dim, dtype=torch.float64, device=dev).index_add_(0, rows, terms)
    scale = torch.zeros(n, dim, dtype=torch.float64, device=dev).index_add_(0, rows, terms.abs())
    assert bool(((D[:n].double() - want).abs() <= 2e-6 * scale + 1e-30).all())
    assert float(D[n:].abs().sum()) == 0
    terms = (G64[rows] * G64[cols]).sum(1) * cols.double()
    assert abs(float(d_beta) - float(terms.sum())) <= 1e-6 * float(terms.abs().sum())
    assert ops.agnn_layer_backward(None, G, rp, ci, None, tr, beta_grad=False, scores=scores)[1] is None


def test_agnn_layer_trains_without_room_for_the_scores(monkeypatch):
    """Where the score array cannot be allocated the backward recomputes the scores."""
    from paramspmm_ae_b200 import gnn_conv, pcsr, synth
    dev = torch.device("cuda:0")
    g = synth.powerlaw_graph(301, 3000, seed=4)
    P = pcsr.pcsr_sddmm(None, 1, False, 301, g.nnz, g.rowPtr, g.colIdx, g.val, None, CF=1, blkWarpNum=8)
    layer = gnn_conv.AGNNConv(16, 32).to(dev)
    X, G = torch.randn(301, 16, device=dev), torch.randn(301, 32, device=dev)

    def step():
        x = X.clone().requires_grad_(True)
        layer.zero_grad()
        out = layer(x, {32: P}, P.colIdx.unsqueeze(-1))
        out.backward(G)
        return out.detach(), x.grad, layer.weights.grad.clone(), layer.attention_w.grad.clone()

    taken, backward = [], gnn_conv.ops.agnn_layer_backward

    def watched(*args, scores=None, **kw):
        taken.append(scores is not None)
        return backward(*args, scores=scores, **kw)

    monkeypatch.setattr(gnn_conv.ops, "agnn_layer_backward", watched)
    kept = step()
    empty, refused = torch.empty, []

    def refuse(*size, **kw):
        if size == (g.nnz,):
            refused.append(size)
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(gnn_conv.torch, "empty", refuse)
    for a, b in zip(kept, step()):
        assert float((a - b).norm()) <= 1e-5 * float(b.norm())
    assert len(refused) == 1 and taken == [True, False]


def _agnn_network(n, mean, dim, layers, classes):
    from paramspmm_ae_b200 import gnn_conv, pcsr
    dev = torch.device("cuda:0")
    ci = torch.randint(0, n, (n * mean,), generator=torch.Generator().manual_seed(4), dtype=torch.int32)
    P = pcsr.pcsr_sddmm(None, 1, False, n, n * mean, torch.arange(n + 1, dtype=torch.int32) * mean, ci, torch.ones(n * mean), None, CF=1,
                        blkWarpNum=8)
    torch.manual_seed(5)
    net = torch.nn.ModuleList([gnn_conv.AGNNConv(dim, dim) for _ in range(layers)]).to(dev)
    last = torch.nn.Linear(dim, classes, bias=False).to(dev)
    X = torch.nn.functional.normalize(torch.randn(n, dim, device=dev))

    def step():
        net.zero_grad(set_to_none=True)
        h = X
        for layer in net:
            h = torch.nn.functional.normalize(torch.relu(layer(h, {dim: P}, P.colIdx.unsqueeze(-1))))
        torch.relu(last(h)).sum().backward()
        return [p.grad.clone() for p in net.parameters()]

    return net, P, step


def _close(got, want):
    # (scores kept and recomputed are sums of the same products in another order)
    return all(0 < float(b.norm()) < float("inf") and float((a - b).norm()) <= 1e-4 * float(b.norm()) for a, b in zip(got, want))


@pytest.mark.parametrize("mean, dim", [(20, 16), (200, 16), (20, 256)])
def test_agnn_layers_keep_no_scores_when_told(mean, dim):
    net, P, step = _agnn_network(301, mean, dim, 2, 8)
    saved = []

    def pack(t):
        saved.append(tuple(t.shape))
        return t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        kept = step()
        assert saved.count((P.colIdx.shape[0],)) == 2
        saved.clear()
        for layer in net:
            layer.keep_scores = False
        assert _close(step(), kept) and saved.count((P.colIdx.shape[0],)) == 0


def test_agnn_network_trains_in_the_memory_it_took_without_scores(monkeypatch):
    """Scores of 80 MB per layer in a network whose last layer needs several hundred: a limit that it keeps to with recomputed scores
    is kept to by default."""
    from paramspmm_ae_b200 import gnn_conv
    torch.cuda.empty_cache()
    net, P, step = _agnn_network(20000, 1000, 8, 2, 4096)
    dev = torch.device("cuda:0")
    total = torch.cuda.get_device_properties(dev).total_memory
    empty, nnz = torch.empty, P.colIdx.shape[0]

    def refuse(*size, **kw):
        if size == (nnz,):
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    try:
        with monkeypatch.context() as m:
            m.setattr(gnn_conv.torch, "empty", refuse)
            step()
            torch.cuda.reset_peak_memory_stats(dev)
            step()
            limit = torch.cuda.max_memory_allocated(dev) + (90 << 20)  # (what the allocator may hold in parts; rows of 8 stay out of its large blocks)
            torch.cuda.empty_cache()
            torch.cuda.set_per_process_memory_fraction(limit / total, dev)
            want = step()
        torch.cuda.empty_cache()
        assert _close(step(), want)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, dev)
        torch.cuda.empty_cache()


@pytest.mark.parametrize("dim", [5, 20, 47, 68, 70, 100, 132, 200, 256, 260])
@pytest.mark.parametrize("split", [False, True])
def test_scores_of_finite_rows_stay_finite_beside_infinite_ones(dim, split):
    """Edge scores of rows that end inside a batch of gathers, and of widths that leave lanes without a column."""
    from paramspmm_ae_b200 import ops
    n, inf_col = 301, 5
    g = torch.Generator().manual_seed(dim)
    A, B = (torch.rand(n, dim, generator=g) - 0.3 for _ in range(2))
    rp, ci, cols = _rows_of_one_to_nine(n, inf_col, dim)
    B[inf_col, :: 2] = float("inf")
    rows = torch.repeat_interleave(torch.arange(n), (rp[1:] - rp[:-1]).long())
    want = (A.double()[rows] * B.double()[ci.long()]).sum(1)
    bound = 1e-6 * (A.double()[rows] * B.double()[ci.long()]).abs().sum(1)
    val = torch.ones(ci.shape[0])
    args = [t.cuda() for t in (A, B)]
    if split:
        rps, tr = ops.split_csr(rp, 4)
        got = ops.csr_split_sddmm(*args, rps.cuda(), ci.cuda(), val.cuda(), tr.cuda(), 1, 8).cpu().double()
    else:
        got = ops.csr_sddmm(*args, rp.cuda(), ci.cuda(), val.cuda(), 1, 8).cpu().double()
    clean = ci != inf_col
    assert bool(((got - want).abs() <= bound)[clean].all()) and not bool(torch.isfinite(got[~clean]).any())


def _moving_scores(n):
    """Scores of one row that rise and fall by more and by less than what moves the reference of the exponentials."""
    t = np.linspace(-20.0, 20.0, n) if n > 1 else np.array([3.0])
    spike, steps = np.zeros(n), np.full(n, 7.9)
    spike[-1] = 30.0
    steps[: min(4, n)] = 0.0  # (all weights of the later batches are e^7.9 of the first reference)
    return [t, t[::-1], 20.0 * (-1.0) ** np.arange(n), spike, spike[::-1], steps, np.repeat(np.arange(-(n // 8) - 1.0, 0.0), 8)[:n] * 8.1]


def _moving_case(dim, lengths, seed):
    """Every row has columns of its own; column 0 of B is the score, A takes it alone, so scores are exact."""
    rows = [s for k in lengths for s in _moving_scores(k)]
    rp = np.concatenate([[0], np.cumsum([len(s) for s in rows])]).astype(np.int32)
    g = torch.Generator().manual_seed(seed)
    A, B = torch.zeros(len(rows), dim), torch.rand(int(rp[-1]), dim, generator=g) - 0.3
    A[:, 0] = 1.0
    B[:, 0] = torch.from_numpy(np.concatenate(rows)).float()
    return rp, torch.arange(int(rp[-1]), dtype=torch.int32), A, B


def _softmax_rows(rp, scores, V):
    """Results in fp64, and their terms' absolute sums."""
    out, scale = np.zeros((len(rp) - 1, V.shape[1])), np.zeros((len(rp) - 1, V.shape[1]))
    for i in range(len(rp) - 1):
        s = scores[rp[i]:rp[i + 1]]
        w = np.exp(s - s.max())
        w /= w.sum()
        out[i], scale[i] = w @ V[rp[i]:rp[i + 1]], w @ np.abs(V[rp[i]:rp[i + 1]])
    return out, scale


@pytest.mark.parametrize("dim", [4, 16, 20, 64, 100, 128, 132, 256])
@pytest.mark.parametrize("sep", [False, True])
@pytest.mark.parametrize("lengths", [(1, 2, 4, 5, 9, 33, 64), (65, 300, 1500)], ids=["short", "long"])
def test_softmax_whose_scores_move_within_a_row(dim, sep, lengths):
    """Rows of several batches, long rows cut over shares, split rows whose pieces' references lie far apart."""
    from paramspmm_ae_b200 import ops
    rp, ci, A, B = _moving_case(dim, lengths, dim)
    n = len(rp) - 1
    V = torch.rand(B.shape, generator=torch.Generator().manual_seed(1)) + 0.5 if sep else B
    want, scale = _softmax_rows(rp, B[:, 0].double().numpy(), V.double().numpy())
    # an exponent of up to 50 is off by half of its last bit, 2e-6, once for the entry and once for each move of the reference that
    # still counts; then one rounding per term of two sums
    bound = (1e-5 + 2 * max(lengths) * 2.0 ** -24) * scale
    kw = dict(V=V.cuda()) if sep else {}
    rpt = torch.from_numpy(rp)
    for granularity in (None, 4, 32):
        ptr, extra = rpt, {}
        if granularity:
            ptr, tr = ops.split_csr(rpt, granularity)
            extra = dict(target_row=tr.cuda(), n_out_rows=n)
        got = ops.agnn_fused(A.cuda(), B.cuda(), ptr.cuda(), ci.cuda(), 1.0, True, **kw, **extra).cpu().double().numpy()
        assert (np.abs(got - want) <= bound).all(), (granularity, np.abs(got - want).max())
        if granularity is None and lengths[0] == 1:  # (the weight of an only entry is one)
            one = np.flatnonzero(np.diff(rp) == 1)
            np.testing.assert_array_equal(got[one], V.double().numpy()[rp[one]])


@pytest.mark.parametrize("dim", [16, 100, 128, 256])
@pytest.mark.parametrize("granularity", [None, 32])
def test_softmax_of_values_near_the_largest(dim, granularity):
    """Weighted averages of values of 4e33: weights above one would leave sums of 64 terms no room."""
    from paramspmm_ae_b200 import ops
    rp, ci, A, B = _moving_case(dim, (64, 300), dim)
    n = len(rp) - 1
    V = 4e33 * (torch.rand(B.shape, generator=torch.Generator().manual_seed(1)) + 0.5)
    want, scale = _softmax_rows(rp, B[:, 0].double().numpy(), V.double().numpy())
    ptr, extra = torch.from_numpy(rp), {}
    if granularity:
        ptr, tr = ops.split_csr(ptr, granularity)
        extra = dict(target_row=tr.cuda(), n_out_rows=n)
    got = ops.agnn_fused(A.cuda(), B.cuda(), ptr.cuda(), ci.cuda(), 1.0, True, V=V.cuda(), **extra).cpu().double().numpy()
    assert (np.abs(got - want) <= (1e-5 + 600 * 2.0 ** -24) * scale).all()
