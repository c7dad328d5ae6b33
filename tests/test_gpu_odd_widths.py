"""Products whose width is no multiple of 4, gathered from an operand with rows padded to 16 bytes: every layout, edges of
lane groups, slices and column tiles, outputs at any alignment, content of the added columns without effect."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _graphs():
    from paramspmm_ae_b200 import synth
    hub = synth.powerlaw_graph(1500, 30000, seed=7)                     # rows of up to several hundred entries
    gaps = synth.with_empty_rows(synth.uniform_rows(2000, 5, seed=8), 3)
    tail = synth.uniform_rows(700, 3, seed=9)
    tail.rowPtr[300:] = tail.rowPtr[300]                                # 400 rows without entries behind one another
    tail.colIdx, tail.val = tail.colIdx[: int(tail.rowPtr[-1])], tail.val[: int(tail.rowPtr[-1])]
    return {"hub": hub, "gaps": gaps, "tail": tail}


def _check(got, want, scale):
    # fp32 sums of up to a few hundred terms in another order: 1e-5 of the terms' absolute sum
    assert bool(((got.double() - want).abs() <= 1e-5 * scale + 1e-12).all())


@pytest.mark.parametrize("dim", [1, 2, 3, 5, 15, 17, 31, 47, 49, 65, 101, 127, 129, 255, 257, 515, 1031])
def test_padded_operand_matches_fp64(dim):
    from paramspmm_ae_b200 import _lib, ops
    for name, g in _graphs().items():
        m = g.to("cuda")
        n = m.n_rows
        gen = torch.Generator(device="cuda").manual_seed(dim)
        X = torch.randn(m.n_cols, dim, device="cuda", generator=gen)
        Xp = ops._pad_rows(X)
        assert Xp.shape[1] == dim + -dim % 4 and torch.equal(Xp[:, :dim], X) and not Xp[:, dim:].any()
        Xp[:, dim:] = float("nan")
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (m.rowPtr[1:] - m.rowPtr[:-1]).long())
        terms = m.val.double()[:, None] * X.double()[m.colIdx.long()]
        want = torch.zeros(n, dim, dtype=torch.float64, device="cuda").index_add_(0, rows, terms)
        scale = torch.zeros(n, dim, dtype=torch.float64, device="cuda").index_add_(0, rows, terms.abs())
        rps, tr = ops.split_csr_device(m.rowPtr, 7)
        seg, cb, vb, tb = ops.bucket_pcsr(m.rowPtr, m.colIdx, m.val, 7)
        layouts = [("csr", m.rowPtr, m.colIdx, m.val, None, 0), ("split", rps, m.colIdx, m.val, tr, 0), ("bucketed", seg, cb, vb, tb, 1)]
        cfgs = [{}, dict(lanes_per_row=2), dict(lanes_per_row=32, gather_batch=4), dict(lanes_per_row=8, gather_batch=16, rows_per_group=3, cta_threads=64),
                dict(col_tile=32), dict(no_long_rows=1)]
        for label, rp, ci, v, target, bucketed in layouts:
            for kw in cfgs if dim in (5, 47, 129, 515) else cfgs[:1]:
                cfg = _lib.make_cfg(bucketed=bucketed, **kw)
                for out in (torch.full((n, dim), float("nan"), device="cuda"), torch.full((n, dim + 3), float("nan"), device="cuda")[:, 1:dim + 1]):
                    ops.spmm_into(out, Xp, rp, ci, v, target_row=target, n_out_rows=n, cfg=cfg, dim=dim)
                    _check(out, want, scale)


def test_operands_that_do_not_fit_are_refused():
    from paramspmm_ae_b200 import _lib, ops, synth
    m = synth.uniform_rows(100, 3, seed=1).to("cuda")
    X, out = torch.randn(100, 48, device="cuda"), torch.empty(100, 47, device="cuda")
    with pytest.raises(RuntimeError):
        ops.spmm_into(out, X, m.rowPtr, m.colIdx, m.val)              # (a narrower output has to be asked for)
    with pytest.raises(RuntimeError):
        ops.spmm_into(out, torch.randn(100, 52, device="cuda"), m.rowPtr, m.colIdx, m.val, dim=47)
    for cfg in (_lib.make_cfg(accumulate=1), _lib.make_cfg(vec_width=2)):
        with pytest.raises(_lib.PspmmError):
            ops.spmm_into(out, X, m.rowPtr, m.colIdx, m.val, cfg=cfg, dim=47)
    null, one = None, ctypes.c_void_p(X.data_ptr())
    for ptr, ld in ((X.data_ptr() + 4, 48), (X.data_ptr(), 47), (X.data_ptr(), 44)):
        assert _lib.lib().pspmm_spmm_csr_padded(one, one, one, ctypes.c_void_p(ptr), one, 1, 1, 1, 47, ld, 47, null, null, null, 0,
                                                null, 0, null) == _lib.PSPMM_E_ARG


@pytest.mark.parametrize("dim", [31, 63, 101, 255])
@pytest.mark.parametrize("split", [False, True])
def test_legacy_calls_on_both_sides_of_the_rule(dim, split, monkeypatch):
    """The widths' own path and the padded one give the same sums through the legacy signatures, scores included."""
    from paramspmm_ae_b200 import ops, synth
    m = synth.powerlaw_graph(3000, 120000, seed=3).to("cuda")
    rp, tr = ops.split_csr_device(m.rowPtr, 32) if split else (m.rowPtr, None)
    X, Y = (torch.randn(3000, dim, device="cuda") for _ in range(2))

    def run():
        if split:
            return (ops.csr_split_spmm(X, rp, m.colIdx, m.val, tr, 1, 8), ops.csr_split_sddmm(X, X, rp, m.colIdx, m.val, tr, 1, 8),
                    ops.csr_split_sddmm(X, Y, rp, m.colIdx, m.val, tr, 1, 8))
        return (ops.csr_spmm(X, rp, m.colIdx, m.val, 1, 8), ops.csr_sddmm(X, X, rp, m.colIdx, m.val, 1, 8),
                ops.csr_sddmm(X, Y, rp, m.colIdx, m.val, 1, 8))

    results = []
    for pays in (False, True):
        monkeypatch.setattr(ops, "_padding_pays", lambda *a: pays)
        monkeypatch.setattr(ops, "_sddmm_padding_pays", lambda *a: pays)
        results.append(run())
    for a, b in zip(*results):
        assert a.shape == b.shape and float((a - b).norm()) <= 1e-6 * float(a.norm())


@pytest.mark.parametrize("vec_width", [0, 1, 2, 4])
def test_plans_and_tuners_with_narrower_loads_take_odd_widths(vec_width, monkeypatch):
    """Configurations of the caller that ask for narrower loads go the way they went, without the padded product."""
    from paramspmm_ae_b200 import decider, ops, pcsr, synth
    m = synth.powerlaw_graph(3000, 120000, seed=3).to("cuda")
    X = torch.randn(3000, 255, device="cuda")
    want = ops.csr_spmm(X, m.rowPtr, m.colIdx, m.val, 1, 8)
    plan = decider.Plan(vec_size=1, lanes_per_row=0, vec_width=vec_width, cta_threads=0, rows_per_group=0, gather_batch=0, col_tile=0,
                        if_split=1, granularity=32, bucketed=0)
    P = pcsr.pcsr_spmm.from_plan(plan, m.rowPtr, m.colIdx, m.val)
    H, W = torch.randn(3000, 16, device="cuda"), torch.randn(16, 47, device="cuda")
    conv = ops.csr_spmm_forward(H, W, m.rowPtr, m.colIdx, m.val, 1, 8)
    monkeypatch.setattr(ops, "tuner", lambda *a: dict(vec_width=vec_width))
    for got, ref in ((P.GIN_spmm(X), want), (ops.csr_spmm(X, m.rowPtr, m.colIdx, m.val, 1, 8), want),
                     (ops.csr_spmm_forward(H, W, m.rowPtr, m.colIdx, m.val, 1, 8), conv), (P.forward(H, W), conv)):
        assert got.shape == ref.shape and got.is_contiguous() and float((got - ref).norm()) <= 1e-5 * float(ref.norm())


@pytest.mark.parametrize("vec_width", [0, 1, 2, 4])
@pytest.mark.parametrize("split", [False, True])
def test_tuners_with_narrower_loads_take_odd_widths_into_an_output(vec_width, split, monkeypatch):
    from paramspmm_ae_b200 import ops, synth
    m = synth.powerlaw_graph(3000, 120000, seed=3).to("cuda")
    rp, tr = ops.split_csr_device(m.rowPtr, 32) if split else (m.rowPtr, None)
    X = torch.randn(3000, 255, device="cuda")
    want = ops.csr_spmm(X, m.rowPtr, m.colIdx, m.val, 1, 8)
    monkeypatch.setattr(ops, "_padding_pays", lambda *a: True)
    monkeypatch.setattr(ops, "tuner", lambda *a: dict(vec_width=vec_width))
    got = ops.spmm_into(torch.full_like(X, float("nan")), X, rp, m.colIdx, m.val, tr, n_out_rows=3000)
    assert float((got - want).norm()) <= 1e-5 * float(want.norm())
    assert ops.spmm_time_ms(X, rp, m.colIdx, m.val, tr, iters=2, n_out_rows=3000) > 0


def test_timing_of_scores_at_odd_widths_holds_nothing_beside_its_calls(monkeypatch):
    from paramspmm_ae_b200 import ops, synth
    m = synth.powerlaw_graph(3000, 120000, seed=3).to("cuda")
    X = torch.randn(3000, 63, device="cuda")
    monkeypatch.setattr(ops, "_sddmm_padding_pays", lambda *a: True)
    assert ops.csr_sddmm_profile(X, X, m.rowPtr, m.colIdx, m.val, 1, 8) > 0
    held, before = [], torch.cuda.memory_allocated()
    monkeypatch.setattr(ops, "_loop_ms", lambda *a: held.append(torch.cuda.memory_allocated()) or 1.0)
    ops.csr_sddmm_profile(X, X, m.rowPtr, m.colIdx, m.val, 1, 8)
    assert held == [before]


def test_products_run_without_room_for_the_copy(monkeypatch):
    from paramspmm_ae_b200 import ops, synth
    m = synth.powerlaw_graph(3000, 120000, seed=3).to("cuda")
    X, Y = (torch.randn(3000, 31, device="cuda") for _ in range(2))
    monkeypatch.setattr(ops, "_padding_pays", lambda *a: True)
    monkeypatch.setattr(ops, "_sddmm_padding_pays", lambda *a: True)
    call = lambda: (ops.csr_spmm(X, m.rowPtr, m.colIdx, m.val, 1, 8), ops.csr_sddmm(X, Y, m.rowPtr, m.colIdx, m.val, 1, 8))
    padded, pad, seen = call(), ops._pad_rows, []

    def refuse(t):
        seen.append(t)
        if len(seen) == 2:  # (the first operand of the scores fits, the second does not)
            return pad(t)
        raise torch.cuda.OutOfMemoryError("no room")

    monkeypatch.setattr(ops, "_pad_rows", refuse)
    for a, b in zip(padded, call()):
        assert float((a - b).norm()) <= 1e-6 * float(b.norm())
    assert len(seen) == 3
