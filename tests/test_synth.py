"""The generators give the same matrix for the same seed: what decides an endpoint must not depend on the
order in which a device adds."""
import numpy as np
import pytest
import torch

NODES = 2_449_029


def _tables(monkeypatch, device, builds):
    """The endpoint tables and the graphs of several builds from one seed."""
    from paramspmm_ae_b200 import synth
    tables, graphs = [], []
    search = torch.searchsorted
    monkeypatch.setattr(torch, "searchsorted", lambda t, u: (tables.append(t.clone()), search(t, u))[1])
    for _ in range(builds):
        graphs.append(synth.powerlaw_graph(NODES, 300_000, seed=9, device=device))
    return tables, graphs


def test_endpoint_table_is_the_exact_distribution(monkeypatch):
    """Within three units of 2**-53 of sums in extended precision: the rounding of the total's parts
    (a random walk of 2.4 M halves in 2**61 .. 2**62, below one unit), the quotient's and the conversions'
    (half a unit each).  A serial float64 scan of this many weights is a thousand units off."""
    tables, _ = _tables(monkeypatch, "cpu", 1)
    w = (torch.arange(NODES, dtype=torch.float64) + 10.0) ** (-1.0 / 1.1)
    exact = np.cumsum(w.numpy().astype(np.longdouble))
    exact /= exact[-1]
    got = tables[0].numpy()
    assert got[-1] == 1.0 and bool((np.diff(got) > 0).all())
    assert float(np.max(np.abs(got - exact))) <= 3 * 2.0 ** -53


@pytest.mark.gpu
def test_a_seed_gives_one_graph_on_the_gpu(monkeypatch):
    tables, graphs = _tables(monkeypatch, "cuda:0", 6)
    for t in tables[1:]:
        assert torch.equal(t, tables[0])
    for m in graphs[1:]:
        assert torch.equal(m.rowPtr, graphs[0].rowPtr) and torch.equal(m.colIdx, graphs[0].colIdx)
        assert torch.equal(m.val, graphs[0].val)
