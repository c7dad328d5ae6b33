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
