"""SpMM shapes that the library chooses without a plan: widths where the number of lanes and slices changes,
row lengths where the number of segments per lane group changes, fewer and more rows than a wave."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [16, 36, 40, 44, 48, 64, 68, 96, 128, 132, 192, 19, 23, 33, 47, 49, 38, 74, 94])
@pytest.mark.parametrize("n, degree", [(301, 5), (40000, 3), (40000, 12), (90001, 8)])
@pytest.mark.parametrize("layout", ["csr", "split", "block"])
def test_default_shapes_match_a_dense_sum(layout, n, degree, dim):
    from paramspmm_ae_b200 import ops
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(dim * 1000 + degree)
    length = rng.integers(0, 2 * degree + 1, n)
    length[rng.integers(0, n, 5)] = 0
    rp = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    row = torch.from_numpy(np.repeat(np.arange(n), length)).to(dev)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    if layout == "block":  # (its builder wants distinct columns in a row)
        ci = ((np.arange(rp[-1]) - rp[np.repeat(np.arange(n), length)]) * 3 + np.repeat(np.arange(n), length)) % n
        ci = ci.astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    X = torch.from_numpy(rng.uniform(-1, 1, (n, dim)).astype(np.float32)).to(dev)
    t = [torch.from_numpy(x).to(dev) for x in (rp, ci, v)]
    if layout == "csr":
        got = ops.csr_spmm(X, *t, 1, 8)
    elif layout == "split":
        rps, target = ops.split_csr_device(t[0], 32)
        got = ops.csr_split_spmm(X, rps, t[1], t[2], target, 1, 8)
    else:
        got = ops.bcsr_spmm(X, *[a.to(dev) for a in ops.bcsr_from_csr(*[a.cpu() for a in t], n, 2)], 1, 8)[:n]
    terms = t[2].double()[:, None] * X.double()[t[1].long()]
    want = torch.zeros(n, dim, dtype=torch.float64, device=dev).index_add_(0, row, terms)
    bound = torch.zeros(n, dim, dtype=torch.float64, device=dev).index_add_(0, row, terms.abs())
    assert bool(((got.double() - want).abs() <= 1e-6 * bound).all())
