"""CPU tests of the C-ABI library: it loads, exports what include/pspmm.h declares, its host
builders are bit-exact, and argument errors are reported as codes (no GPU call is made)."""
import ctypes
import os
import re

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    text = open(os.path.join(ROOT, "include", "pspmm.h")).read()
    return sorted(set(re.findall(r"PSPMM_API\s+[\w \*]+?\b(pspmm_\w+)\s*\(", text)))


def test_library_exports_every_declared_symbol(pspmm_lib):
    names = _declared()
    assert len(names) >= 15
    for n in names:
        assert hasattr(pspmm_lib, n), "libpspmm.so does not export %s" % n
    from paramspmm_ae_b200 import _lib
    assert sorted(_lib.EXPORTED) == sorted(n for n in names if n in _lib.EXPORTED)
    assert set(_lib.EXPORTED) <= set(names)
    assert pspmm_lib.pspmm_version() >= 100
    assert pspmm_lib.pspmm_strerror(0) == b"ok"
    assert b"CF" in pspmm_lib.pspmm_strerror(-2)


def test_split_csr_bit_exact_with_golden_and_oracle(pspmm_lib, oracle, golden_dir):
    from paramspmm_ae_b200 import ops
    z = np.load(os.path.join(golden_dir, "split_ref.npz"))
    for i in range(int(z["n_cases"])):
        rp = torch.from_numpy(z["rowPtr_%d" % i])
        gran = int(z["gran_%d" % i])
        rps, tr = ops.split_csr(rp, gran)
        assert rps.dtype == torch.int32 and tr.dtype == torch.int32
        assert np.array_equal(rps.numpy(), z["rowPtr_split_%d" % i])
        assert np.array_equal(tr.numpy(), z["target_row_%d" % i])
        pieces = oracle.row_split_counts(z["rowPtr_%d" % i], gran)
        off = torch.from_numpy(np.concatenate([[0], np.cumsum(pieces)]).astype(np.int32))
        rps2, tr2 = ops.split_csr_par(rp, off, gran)
        assert torch.equal(rps, rps2) and torch.equal(tr, tr2)


def test_split_csr_large_random_matches_oracle(pspmm_lib, oracle):
    from paramspmm_ae_b200 import ops
    rng = np.random.default_rng(8)
    ln = rng.zipf(1.8, size=300000).clip(max=50000)
    ln[rng.random(ln.shape[0]) < 0.1] = 0
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    for gran in (32, 512):
        rps, tr = ops.split_csr(torch.from_numpy(rp), gran)
        o_rps, o_tr = oracle.split_csr(rp, gran)
        assert np.array_equal(rps.numpy(), o_rps) and np.array_equal(tr.numpy(), o_tr)


def test_split_csr_edge_cases(pspmm_lib):
    from paramspmm_ae_b200 import ops
    rps, tr = ops.split_csr(torch.zeros(1, dtype=torch.int32), 32)  # no rows
    assert rps.tolist() == [0] and tr.numel() == 0
    rps, tr = ops.split_csr(torch.zeros(6, dtype=torch.int32), 32)  # only empty rows
    assert rps.tolist() == [0] and tr.numel() == 0
    rps, tr = ops.split_csr(torch.tensor([0, 64], dtype=torch.int32), 32)  # exact multiple
    assert rps.tolist() == [0, 32, 64] and tr.tolist() == [0, 0]
    with pytest.raises(RuntimeError):
        ops.split_csr(torch.tensor([0, 4], dtype=torch.int32), 0)
    with pytest.raises(RuntimeError):
        ops.split_csr(torch.tensor([0, 4], dtype=torch.int64), 2)


def test_bcsr_builder_bit_exact(pspmm_lib, oracle, golden_dir):
    from paramspmm_ae_b200 import ops
    z = np.load(os.path.join(golden_dir, "bcsr_scipy.npz"))
    for i in range(int(z["n_cases"])):
        rp, ci, v, V = z["rowPtr_%d" % i], z["colIdx_%d" % i], z["val_%d" % i], int(z["V_%d" % i])
        rpb, cb, vb = ops.bcsr_from_csr(torch.from_numpy(rp), torch.from_numpy(ci), torch.from_numpy(v),
                                        rp.shape[0] - 1, V)
        assert np.array_equal(rpb.numpy(), z["rowPtr_b_%d" % i])
        assert np.array_equal(cb.numpy(), z["colIdx_b_%d" % i])
        assert np.array_equal(vb.numpy(), z["val_b_%d" % i])


def test_bcsr_builder_matches_scipy_on_power_law(pspmm_lib):
    from paramspmm_ae_b200 import ops, synth
    m = synth.powerlaw_graph(3001, 20000, seed=5)
    rp, ci, v = m.numpy()
    import scipy.sparse as sp
    n = m.n_rows
    pad = np.concatenate([rp, [rp[-1]]])
    b = sp.csr_array((v, ci, pad), shape=(n + 1, n + 1)).tobsr(blocksize=(2, 1))
    rpb, cb, vb = ops.bcsr_from_csr(m.rowPtr, m.colIdx, m.val, n, 2)
    assert np.array_equal(rpb.numpy(), b.indptr) and np.array_equal(cb.numpy(), b.indices)
    assert np.array_equal(vb.numpy(), b.data.reshape(-1, 2))


def test_argument_errors_are_codes_not_crashes(pspmm_lib):
    from paramspmm_ae_b200 import _lib
    null = ctypes.c_void_p(0)
    one = ctypes.c_void_p(16)  # never dereferenced: validation fails first
    cfg = _lib.make_cfg()
    # dim <= 0
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 4, 0, 8, 8, ctypes.byref(cfg),
                                    null, null, 0, null) == _lib.PSPMM_E_ARG
    # leading dimension smaller than dim
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 4, 16, 8, 16, ctypes.byref(cfg),
                                    null, null, 0, null) == _lib.PSPMM_E_ARG
    # null operand
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, null, one, 4, 4, 4, 16, 16, 16, ctypes.byref(cfg),
                                    null, null, 0, null) == _lib.PSPMM_E_ARG
    # split arrays must come together
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 4, 16, 16, 16, ctypes.byref(cfg),
                                    one, null, 3, null) == _lib.PSPMM_E_ARG
    # index range
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 2 ** 31, 16, 16, 16,
                                    ctypes.byref(cfg), null, null, 0, null) == _lib.PSPMM_E_RANGE
    # legacy hints keep the reference's domain
    for bad in (_lib.make_cfg(CF=9, blkWarpNum=4), _lib.make_cfg(CF=1, blkWarpNum=5),
                _lib.make_cfg(lanes_per_row=3), _lib.make_cfg(vec_width=3), _lib.make_cfg(cta_threads=100),
                _lib.make_cfg(accumulate=2), _lib.make_cfg(accumulate=-1), _lib.make_cfg(col_tile=6)):
        assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 4, 16, 16, 16, ctypes.byref(bad),
                                        null, null, 0, null) == _lib.PSPMM_E_CONFIG
    assert pspmm_lib.pspmm_sddmm_csr(one, one, one, one, one, 4, 4, 16, 16, 16,
                                     ctypes.byref(_lib.make_cfg(CF=5, blkWarpNum=4)), null, null, 0,
                                     null) == _lib.PSPMM_E_CONFIG
    # SDDMM has nothing to add into
    assert pspmm_lib.pspmm_sddmm_csr(one, one, one, one, one, 4, 4, 16, 16, 16,
                                     ctypes.byref(_lib.make_cfg(accumulate=1)), null, null, 0,
                                     null) == _lib.PSPMM_E_CONFIG
    assert pspmm_lib.pspmm_spmm_bcsr(one, one, one, 4, one, one, 4, 4, 4, 16, 16, 16, ctypes.byref(cfg),
                                     null, null, 0, null) == _lib.PSPMM_E_UNSUPPORTED
    with pytest.raises(_lib.PspmmError):
        _lib.check(_lib.PSPMM_E_ARG)


def test_config_resolution_covers_every_dim(pspmm_lib):
    """Every dim 1..1100 and block height resolves to an instantiated kernel shape."""
    from paramspmm_ae_b200 import _lib
    for V in (1, 2, 3):
        for dim in list(range(1, 300)) + [512, 1000, 1024, 1100]:
            cfg = _lib.make_cfg()
            rc = pspmm_lib.pspmm_resolve_cfg(ctypes.byref(cfg), dim, dim, dim, V, ctypes.c_void_p(256),
                                             ctypes.c_void_p(256))
            assert rc == 0
            assert cfg.vec_width == (4 if dim % 4 == 0 else 2 if dim % 2 == 0 else 1)
            assert cfg.lanes_per_row in (1, 2, 4, 8, 16, 32)
    cfg = _lib.make_cfg()
    assert pspmm_lib.pspmm_resolve_cfg(ctypes.byref(cfg), 64, 64, 64, 1, ctypes.c_void_p(256),
                                       ctypes.c_void_p(256)) == 0
    assert (cfg.lanes_per_row, cfg.vec_width) == (16, 4)
    # a misaligned base pointer or odd leading dimension narrows the vector width
    cfg = _lib.make_cfg()
    pspmm_lib.pspmm_resolve_cfg(ctypes.byref(cfg), 64, 64, 64, 1, ctypes.c_void_p(260), ctypes.c_void_p(256))
    assert cfg.vec_width == 1
    cfg = _lib.make_cfg()
    pspmm_lib.pspmm_resolve_cfg(ctypes.byref(cfg), 64, 66, 64, 1, ctypes.c_void_p(256), ctypes.c_void_p(256))
    assert cfg.vec_width == 2


def _resolved(lib, dim, V, split, n_seg, n_entries, **kw):
    from paramspmm_ae_b200 import _lib
    cfg = _lib.make_cfg(**kw)
    rc = lib.pspmm_resolve_spmm(ctypes.byref(cfg), dim, dim, dim, V, ctypes.c_void_p(256), ctypes.c_void_p(256), int(split),
                                n_seg, n_entries)
    return rc, tuple(getattr(cfg, f) for f, _ in cfg._fields_), cfg


def test_resolved_shapes_see_the_layout_and_the_sizes(pspmm_lib):
    """pspmm_resolve_spmm goes through the launch's own rules: split or not, few and many rows, short and
    long ones.  (pspmm_resolve_cfg takes every layout for an unsplit one of unknown size.)"""
    from paramspmm_ae_b200 import _lib
    shape = lambda *a, **k: _resolved(pspmm_lib, *a, **k)[2]
    assert shape(48, 1, False, 10**6, 8 * 10**6).lanes_per_row == 4
    assert shape(46, 1, True, 10**6, 8 * 10**6).lanes_per_row == 32      # 23 vectors of 8 bytes: three slices only unsplit
    assert shape(46, 1, False, 10**6, 8 * 10**6).lanes_per_row == 8
    assert shape(96, 1, False, 10**6, 15 * 10**6).cta_threads == 128
    assert shape(96, 1, False, 10**6, 16 * 10**6).cta_threads == 256     # (long rows of neighbouring columns)
    assert shape(96, 1, True, 10**6, 16 * 10**6).cta_threads == 128
    assert shape(128, 1, False, 10**6, 8 * 10**6).rows_per_group == 8
    assert shape(128, 1, False, 10**6, 32 * 10**6).rows_per_group == 4
    assert shape(128, 1, False, 1000, 8000).rows_per_group == 1          # (a small matrix fills the chip with single rows)
    assert shape(16, 1, True, 10**6, 8 * 10**6).rows_per_group == 2
    assert shape(8, 1, True, 10**6, 8 * 10**6, accumulate=1).lanes_per_row == 4
    assert shape(240, 1, False, 10**6, 16 * 10**6, col_tile=64).lanes_per_row == 16
    assert _resolved(pspmm_lib, 47, 1, False, 100, 400, accumulate=1)[0] == _lib.PSPMM_E_UNSUPPORTED
    assert _resolved(pspmm_lib, 64, 1, False, -1, 400)[0] == _lib.PSPMM_E_ARG


def test_small_split_layouts_take_single_segments(pspmm_lib):
    """Three slices on four or eight lanes: two segments per group, one up to about seven waves of groups
    (the skewed layouts lost up to 20 % there), where 11 vectors keep one slice on sixteen lanes."""
    def shape(dim, n_seg):
        c = _resolved(pspmm_lib, dim, 1, True, n_seg, 11 * n_seg)[2]
        return c.lanes_per_row, c.rows_per_group
    waves7 = 7 * 768 * 148
    assert shape(48, waves7 // 4) == (4, 1) and shape(48, waves7 // 4 + 1) == (4, 2)
    assert shape(44, waves7 // 4)[0] == 16 and shape(44, waves7 // 4 + 1) == (4, 2)
    for dim in (68, 76, 96):
        assert shape(dim, waves7 // 8) == (8, 1) and shape(dim, waves7 // 8 + 1) == (8, 2)
    assert shape(160, 40000) == (16, 2) and shape(160, 10**6) == (16, 2)  # (below that the waves decide)
    assert shape(40, 10**5)[0] == 16


def test_a_resolved_configuration_resolves_to_itself(pspmm_lib):
    import random
    rng = random.Random(3)
    for _ in range(4000):
        V, split = rng.choice([1, 1, 1, 2, 3]), rng.random() < 0.5
        dim, n_seg = rng.randint(1, 300), int(10 ** rng.uniform(0, 7))
        n_entries = int(n_seg * 10 ** rng.uniform(-1, 3))
        kw = {}
        for field, values in (("lanes_per_row", (2, 4, 8, 16, 32)), ("vec_width", (1, 2, 4)), ("cta_threads", (64, 256)),
                              ("rows_per_group", (1, 4, 8)), ("gather_batch", (4, 16)), ("col_tile", (32, 48, 64, 128))):
            if rng.random() < 0.25:
                kw[field] = rng.choice(values)
        if V == 1 and dim % 4 == 0 and kw.get("vec_width", 4) == 4 and rng.random() < 0.2:
            kw["accumulate"] = 1
        rc, first, cfg = _resolved(pspmm_lib, dim, V, split, n_seg, n_entries, **kw)
        assert rc == 0, (dim, V, split, n_seg, n_entries, kw)
        again = {f: getattr(cfg, f) for f in ("lanes_per_row", "vec_width", "cta_threads", "rows_per_group", "gather_batch",
                                              "col_tile", "accumulate")}
        assert _resolved(pspmm_lib, dim, V, split, n_seg, n_entries, **again)[1] == first, (dim, V, split, n_seg, n_entries, kw)


def test_odd_widths_resolve_to_the_padded_product(pspmm_lib):
    """The product on padded rows has a resolution of its own: 16-byte loads, at least four lanes, at most four slices on them
    below a whole warp, and a resolved configuration resolves to itself."""
    import random
    from paramspmm_ae_b200 import _lib
    B = ctypes.c_void_p(256)

    def shape(dim, split, n_seg, n_entries, **kw):
        cfg = _lib.make_cfg(**kw)
        rc = pspmm_lib.pspmm_resolve_spmm_padded(ctypes.byref(cfg), dim, dim + -dim % 4, B, int(split), n_seg, n_entries)
        return rc, cfg, tuple(getattr(cfg, f) for f, _ in cfg._fields_)

    rng = random.Random(4)
    for _ in range(3000):
        dim, n_seg = rng.randint(1, 1100), int(10 ** rng.uniform(0, 7))
        kw = {f: rng.choice(v) for f, v in (("lanes_per_row", (2, 4, 8, 16, 32)), ("vec_width", (0, 4)), ("gather_batch", (2, 4, 16)),
                                            ("rows_per_group", (1, 8)), ("col_tile", (32, 64))) if rng.random() < 0.3}
        sizes = rng.random() < 0.5, n_seg, int(n_seg * 10 ** rng.uniform(-1, 3))
        rc, cfg, first = shape(dim, *sizes, **kw)
        wide = min(dim + 3, kw.get("col_tile", dim + 3)) // 4
        assert rc == 0 and cfg.vec_width == 4 and cfg.lanes_per_row >= 4 and cfg.gather_batch in (4, 8, 16)
        assert cfg.lanes_per_row == 32 or wide <= 4 * cfg.lanes_per_row, (dim, kw)
        again = {f: getattr(cfg, f) for f in ("lanes_per_row", "vec_width", "cta_threads", "rows_per_group", "gather_batch", "col_tile")}
        assert shape(dim, *sizes, **again)[2] == first, (dim, kw)
    assert shape(142, False, 300000, 3600000, lanes_per_row=8)[1].lanes_per_row == 16  # (five slices of 8 lanes)
    assert shape(47, False, 100, 400, accumulate=1)[0] == shape(47, False, 100, 400, vec_width=2)[0] == _lib.PSPMM_E_UNSUPPORTED
    cfg = _lib.make_cfg()
    for ld, ptr in ((47, 256), (44, 256), (48, 260)):
        assert pspmm_lib.pspmm_resolve_spmm_padded(ctypes.byref(cfg), 47, ld, ctypes.c_void_p(ptr), 0, 10, 10) == _lib.PSPMM_E_ARG


def test_ops_reject_cpu_tensors_and_bad_hints():
    """The torch-level operators never fall back: a CPU tensor or an invalid CF / blkWarpNum is
    an error, as in the reference (SpMM/SpMM.cpp:5-13, 110, 139)."""
    from paramspmm_ae_b200 import ops
    X = torch.zeros(4, 8)
    rp = torch.zeros(5, dtype=torch.int32)
    ci = torch.zeros(0, dtype=torch.int32)
    v = torch.zeros(0)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        ops.csr_spmm(X, rp, ci, v, 1, 4)
    with pytest.raises(RuntimeError, match="blkWarpNum"):
        ops.csr_spmm(X, rp, ci, v, 1, 6)
    with pytest.raises(RuntimeError, match="CF"):
        ops.csr_spmm(X, rp, ci, v, 9, 4)
    with pytest.raises(RuntimeError, match="CF"):
        ops.csr_sddmm(X, X, rp, ci, v, 5, 4)


def test_dropin_modules_expose_reference_names():
    import paramspmm_ae_b200
    paramspmm_ae_b200.install_dropin()
    import ParamSDDMM
    import ParamSpCONV
    import ParamSpMM
    spmm_names = """split_csr split_csr_par csr_spmm csr_split_spmm bcsr_spmm bcsr_split_spmm vec_spmm
        vec_split_spmm csr_spmm_profile csr_split_spmm_profile bcsr_spmm_profile bcsr_split_spmm_profile
        vec_spmm_profile vec_split_spmm_profile cusparse_compute cusparse_profile cusparse_compute_csr_alg2
        cusparse_profile_csr_alg2 cusparse_compute_coo_alg4 cusparse_profile_coo_alg4 cusparse_compute_csc
        cusparse_profile_csc gespmm_compute gespmm_profile""".split()
    sddmm_names = """csr_sddmm csr_split_sddmm bcsr_sddmm bcsr_split_sddmm vec_sddmm vec_split_sddmm
        csr_sddmm_profile csr_split_sddmm_profile bcsr_sddmm_profile bcsr_split_sddmm_profile
        vec_sddmm_profile vec_split_sddmm_profile cusparse_sddmm_compute cusparse_sddmm_profile genmask""".split()
    conv_names = """split_csr split_csr_par csr_spmm_forward csr_spmm_backward csr_split_spmm_forward
        csr_split_spmm_backward bcsr_spmm_forward bcsr_spmm_backward bcsr_split_spmm_forward
        bcsr_split_spmm_backward""".split()
    for mod, names in ((ParamSpMM, spmm_names), (ParamSDDMM, sddmm_names), (ParamSpCONV, conv_names)):
        for n in names:
            assert callable(getattr(mod, n)), "%s.%s missing" % (mod.__name__, n)


def test_table_plans_become_valid_kernel_configurations():
    """Every entry of the measured table decodes into a pspmm_cfg the library accepts (including
    the column-tile field), for every regime and every dim key."""
    import ctypes
    from paramspmm_ae_b200 import _lib, decider
    lib = _lib.lib()
    tab = decider.load_table()
    seen = 0
    for regime, per_dim in tab["entries"]["spmm"].items():
        for dim_key, e in per_dim.items():
            plan = decider.Plan(if_split=0, vec_size=1, granularity=None)
            plan.update(e)
            cfg = _lib.make_cfg(**plan.kernel_cfg())
            assert cfg.col_tile in (0, 32, 64, 128) and cfg.bucketed in (0, 1)
            dim = int(dim_key)
            rc = lib.pspmm_resolve_cfg(ctypes.byref(cfg), dim, dim, dim, 1, ctypes.c_void_p(256), ctypes.c_void_p(256))
            assert rc == _lib.PSPMM_OK, (regime, dim_key, e)
            assert cfg.lanes_per_row in (2, 4, 8, 16, 32) and cfg.cta_threads in (32, 64, 128, 256)
            seen += 1
    assert seen >= 64


def test_table_measures_every_regime_and_the_decider_reaches_them():
    """The committed table holds a measured entry for every regime the fit covers and for every
    dim key; the regime rule sends the generators' matrices where the fit put them; a regime
    without measurements borrows from its nearest measured neighbour."""
    import torch
    from paramspmm_ae_b200 import decider, sweep, synth
    tab = decider.load_table()
    regimes = tab["entries"]["spmm"]
    for r in sweep.ALL_REGIMES:
        assert r in regimes, r
        assert set(regimes[r]) == {str(d) for d in range(16, 257, 16)}, r
    cases = [(synth.uniform_rows(4000, 4, seed=1), "tiny_even"), (synth.uniform_rows(4000, 16, seed=1), "short_even"),
             (synth.banded_rows(4000, 16, 32, seed=1), "short_local"), (synth.uniform_rows(3000, 64, seed=1), "medium_even"),
             (synth.banded_rows(3000, 64, 96, seed=1), "medium_local"), (synth.rmat(12, 4 * 4096, seed=1), "tiny_skewed"),
             (synth.rmat(12, 16 * 4096, seed=1), "short_skewed"), (synth.powerlaw_graph(3000, 75000, seed=1), "medium_skewed")]
    for m, want in cases:
        st = decider.row_stats(m.rowPtr, m.colIdx)
        assert decider.regime(st) == want, (want, st)
        for dim in (16, 100, 256, 300):
            p = decider.choose(st, dim)
            assert p["regime"] == want and p["vec_size"] in (1, 2)
            assert (p["granularity"] is not None) == bool(p["if_split"])
    # without column indices a banded matrix is an even one; long_local borrows (no fit matrix for it)
    b = synth.banded_rows(4000, 16, 32, seed=1)
    assert decider.regime(decider.row_stats(b.rowPtr)) == "short_even"
    st = {"n_rows": 10, "nnz": 3000, "avg": 300.0, "cov": 0.1, "max": 310, "real_avg": 300.0, "near_diag": 1.0}
    assert decider.regime(st) == "long_local" and decider.choose(st, 64)["regime"] == "long_local"


def test_plans_fit_the_size_of_the_matrix():
    """Plans of the table stand for matrices that fill the GPU; smaller ones get shorter groups, or the launch's own rules."""
    from paramspmm_ae_b200 import decider

    def plan(n, k, dim, cov=2.0, n_cols=None):
        stats = {"n_rows": n, "nnz": n * k, "avg": float(k), "cov": cov, "max": k * (300 if cov else 1), "real_avg": float(k), "near_diag": 0.0}
        p = decider.choose(stats, dim, n_cols=n_cols)
        assert (p["granularity"] is not None) == bool(p["if_split"]) and p["no_long_rows"] == int(not cov)
        return p

    table = decider.table()["entries"]["spmm"]
    for dim in (16, 64, 128, 256):
        full = table["medium_skewed"][str(dim)]
        assert all(plan(4_000_000, 25, dim)[k] == full[k] for k in ("granularity", "rows_per_group", "bucketed", "lanes_per_row"))
        p = plan(100_000, 25, dim)
        assert p["bucketed"] and p["granularity"] * p["rows_per_group"] <= 128 and p["lanes_per_row"] == full["lanes_per_row"]
        p = plan(5_000, 8, dim)
        assert p["if_split"] and not p["bucketed"] and not p["lanes_per_row"] and p["granularity"] == 32
        p = plan(8_000, 16, dim, cov=0.0)
        assert not p["if_split"] and not p["col_tile"] and (dim > 212 or not p["lanes_per_row"])
    assert plan(1_000_000, 16, 256, cov=0.0)["col_tile"] and not plan(100_000, 16, 256, cov=0.0)["col_tile"]
    assert plan(100_000, 16, 256, cov=0.0, n_cols=1_000_000)["col_tile"]      # (a shard: the dense operand is the whole one)


def test_column_tiles_of_local_matrices_stay_from_a_third_of_the_l2_on():
    from paramspmm_ae_b200 import decider
    for n, tiled in ((20_000, False), (50_000, False), (60_000, True), (120_000, True), (1_000_000, True)):
        for k in (30, 77):
            stats = {"n_rows": n, "nnz": n * k, "avg": float(k), "cov": 0.0, "max": k, "real_avg": float(k), "near_diag": 1.0}
            assert bool(decider.choose(stats, 160)["col_tile"]) == tiled, (n, k)


def test_plans_of_even_matrices_cut_rows_that_end_late():
    """A matrix counts as even up to rows of 16 times the mean.  Where one lane group would walk such a row long after the product's
    other rows, the plan keeps its split or lets the launch cut the row, in small matrices and in large ones."""
    from paramspmm_ae_b200 import decider

    def plan(n, k, longest, dim, drop=()):
        stats = {"n_rows": n, "nnz": n * k, "avg": float(k), "cov": 0.2, "max": longest, "real_avg": float(k), "near_diag": 0.0}
        p = decider.choose({f: v for f, v in stats.items() if f not in drop}, dim)
        assert p["regime"].endswith("_even")
        assert p.kernel_cfg()["no_long_rows"] == p["no_long_rows"]
        return p

    cut = lambda p: bool(p["if_split"]) or not p["no_long_rows"]
    for n, k, longest in ((5000, 400, 5000), (20000, 50, 800), (6000, 100, 1600), (30000, 60, 900), (50000, 400, 6000)):
        assert all(cut(plan(n, k, longest, dim)) for dim in (16, 64, 128, 256) if n * dim <= 4e6)
    for n, k in ((5000, 16), (20000, 50), (100000, 16), (1000000, 16)):
        assert all(plan(n, k, 16 * k if k == 16 else 2 * k, dim)["no_long_rows"] for dim in (64, 128))
    assert cut(plan(100000, 100, 1600, 64)) and not cut(plan(100000, 100, 300, 64))
    assert plan(20000, 50, 800, 64, drop=("nnz",))["no_long_rows"]  # (statistics without sizes go by the regime)


def test_header_is_plain_c_and_declares_what_the_python_shim_binds(tmp_path):
    """include/pspmm.h must compile as C99 and as C++ on its own (it is what a foreign-language
    binding includes), and every function the ctypes shim binds must be declared in it."""
    import os
    import re
    import subprocess
    from paramspmm_ae_b200 import _lib
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    hdr = os.path.join(root, "include", "pspmm.h")
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-fsyntax-only", "-x", "c", hdr], check=True)
    subprocess.run(["g++", "-std=c++14", "-Wall", "-Werror", "-fsyntax-only", "-x", "c++", hdr], check=True)
    text = open(hdr).read()
    declared = set(re.findall(r"PSPMM_API\s+[\w\s\*]+?\b(pspmm_\w+)\s*\(", text))
    assert set(_lib.EXPORTED) <= declared, sorted(set(_lib.EXPORTED) - declared)
    # a C caller can fill the configuration struct by name
    src = tmp_path / "use.c"
    src.write_text('#include "pspmm.h"\nint main(void) { pspmm_cfg c = {0}; c.col_tile = 128; c.hint_CF = 2; '
                   'return pspmm_version() > 0 && c.col_tile == 128 ? 0 : 1; }\n')
    exe = tmp_path / "use"
    subprocess.run(["gcc", "-std=c99", "-I", os.path.join(root, "include"), str(src), "-o", str(exe),
                    _lib.LIB_PATH, "-Wl,-rpath," + os.path.dirname(_lib.LIB_PATH)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_new_entry_points_validate_before_touching_the_device(pspmm_lib):
    """pspmm_pull_rows, pspmm_agnn_fused_apply_csr, the bucketed flag and the block SDDMM's row count
    of A: bad arguments come back as codes (no CUDA call is reached with them)."""
    from paramspmm_ae_b200 import _lib
    null, one = ctypes.c_void_p(0), ctypes.c_void_p(16)
    src = _lib.RowSources()
    src.n_src = 1
    src.base[0] = 16
    src.first[0], src.first[1] = 0, 8
    call = lambda n, dim, lds, ldd, rot, s=src: pspmm_lib.pspmm_pull_rows(ctypes.byref(s), one, n, one, dim, lds, ldd, rot, 0, null)
    assert call(8, 0, 16, 16, 0) == _lib.PSPMM_E_ARG            # dim
    assert call(8, 16, 8, 16, 0) == _lib.PSPMM_E_ARG            # row stride smaller than dim
    assert call(8, 16, 16, 16, 8) == _lib.PSPMM_E_ARG           # rotate outside the list
    assert call(9, 16, 16, 16, 0) == _lib.PSPMM_E_ARG           # the sources do not cover the list
    assert call(8, 18, 20, 20, 0) == _lib.PSPMM_E_UNSUPPORTED   # not 128-bit accessible
    assert call(0, 16, 16, 16, 0) == _lib.PSPMM_OK              # nothing to copy
    bad = _lib.RowSources()
    bad.n_src = _lib.MAX_ROW_SOURCES + 1
    assert call(8, 16, 16, 16, 0, bad) == _lib.PSPMM_E_ARG
    # the bulk-copy form checks the same way; its status query wants somewhere to write
    bulk = lambda n, dim, lds, ldd, rot: pspmm_lib.pspmm_pull_rows_bulk(ctypes.byref(src), one, n, one, dim, lds, ldd, rot, 0, null)
    assert bulk(8, 0, 16, 16, 0) == _lib.PSPMM_E_ARG
    assert bulk(8, 16, 16, 16, 8) == _lib.PSPMM_E_ARG
    assert bulk(8, 18, 20, 20, 0) == _lib.PSPMM_E_UNSUPPORTED
    assert bulk(0, 16, 16, 16, 0) == _lib.PSPMM_OK
    assert pspmm_lib.pspmm_pull_rows_status(None) == _lib.PSPMM_E_ARG
    # bucketed is a 0/1 flag of the SpMM only
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 4, 16, 16, 16, ctypes.byref(_lib.make_cfg(bucketed=2)),
                                    null, null, 0, null) == _lib.PSPMM_E_CONFIG
    assert pspmm_lib.pspmm_sddmm_csr(one, one, one, one, one, 4, 4, 16, 16, 16, ctypes.byref(_lib.make_cfg(bucketed=1)),
                                     null, null, 0, null) == _lib.PSPMM_E_CONFIG
    # block SDDMM: A must reach into the last block-row
    cfg = _lib.make_cfg()
    assert pspmm_lib.pspmm_sddmm_bcsr(one, one, one, 2, one, one, one, 5, 8, 4, 16, 16, 16, ctypes.byref(cfg),
                                      null, null, 0, null) == _lib.PSPMM_E_ARG
    # fused aggregation with a separate operand: V missing, V's stride too small
    f = pspmm_lib.pspmm_agnn_fused_apply_csr
    assert f(one, one, one, one, null, one, 4, 4, 16, 16, 16, 16, 16, 1.0, 0, 0, 0, 0, null, null, 0, null, 0, null) == _lib.PSPMM_E_ARG
    assert f(one, one, one, one, one, one, 4, 4, 16, 16, 16, 8, 16, 1.0, 0, 0, 0, 0, null, null, 0, null, 0, null) == _lib.PSPMM_E_ARG


def test_block_builder_rejects_bad_columns_and_inconsistent_counts(pspmm_lib):
    """The host block builder range-checks column ids and never writes more blocks than the row
    pointer it is given allows."""
    import numpy as np
    from paramspmm_ae_b200 import _lib
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    rp = np.array([0, 2, 3, 5], dtype=np.int32)
    ci = np.array([0, 3, 1, 2, 9], dtype=np.int32)    # 9 is outside [0, 4)
    v = np.ones(5, dtype=np.float32)
    rpb = np.zeros(3, dtype=np.int32)
    nblk = ctypes.c_int64(0)
    assert pspmm_lib.pspmm_bcsr_count(p(rp), p(ci), 3, 4, 2, p(rpb), ctypes.byref(nblk)) == _lib.PSPMM_E_ARG
    ci[4] = 3
    assert pspmm_lib.pspmm_bcsr_count(p(rp), p(ci), 3, 4, 2, p(rpb), ctypes.byref(nblk)) == _lib.PSPMM_OK
    assert rpb.tolist() == [0, 3, 5] and nblk.value == 5
    # a row pointer that promises fewer blocks than the rows hold: an error, and the arrays' tails stay untouched
    lie = np.array([0, 1, 2], dtype=np.int32)
    cb = np.full(6, -7, dtype=np.int32)
    vb = np.full(12, -7.0, dtype=np.float32)
    assert pspmm_lib.pspmm_bcsr_fill(p(rp), p(ci), p(v), 3, 4, 2, p(lie), p(cb), p(vb)) == _lib.PSPMM_E_ARG
    assert (cb[2:] == -7).all() and (vb[4:] == -7).all()


def test_timing_and_tuning_launch_what_the_operator_launches(monkeypatch):
    """A plan becomes one configuration: the operator's product, the sweep's timer and the decider's command
    line hand the same one to the library, and candidates of an unsplit matrix differ in what they time."""
    from paramspmm_ae_b200 import _lib, decider, ops, sweep, synth
    fields = lambda cfg: tuple(getattr(cfg, f) for f, _ in cfg._fields_)
    seen = {"run": [], "time": []}
    monkeypatch.setattr(ops, "spmm_into", lambda out, *a, cfg=None, **k: (seen["run"].append(fields(cfg)), out.zero_())[1])
    monkeypatch.setattr(ops, "spmm_time_ms", lambda *a, cfg=None, **k: (seen["time"].append(fields(cfg)), 1.0)[1])
    flag = [f for f, _ in _lib.PspmmCfg._fields_].index("no_long_rows")
    for m, unsplit_flag in ((synth.uniform_rows(4000, 16, seed=1), 1), (synth.banded_rows(4000, 16, 32, seed=1), 1),
                            (synth.powerlaw_graph(3000, 9000, seed=1), 0)):
        stats = decider.row_stats(m.rowPtr, m.colIdx)
        for dim in (16, 64, 128):
            plan = decider.choose(stats, dim)
            if plan["if_split"]:  # the layouts without a GPU: the same plan on the unsplit rows
                plan.update(if_split=0, granularity=None, bucketed=0, no_long_rows=0)
            X, out = torch.zeros(m.n_cols, dim), torch.zeros(m.n_rows, dim)
            op = decider.PlannedSpMM(plan, m.rowPtr, m.colIdx, m.val, n_cols=m.n_cols)
            seen["run"].clear()
            op(out, X)
            timer = sweep.Timer.__new__(sweep.Timer)
            timer.m, timer.dim, timer.dev, timer.warmup, timer.iters = m, dim, torch.device("cpu"), 0, 1
            timer.lay, timer.B = sweep.Layouts(m, torch.device("cpu")), X
            timer.ref, timer.tol = torch.zeros(m.n_rows, dim), torch.ones(m.n_rows, dim)
            seen["time"].clear()
            timer.ms(dict(plan))
            assert seen["time"] and seen["time"][-1] == seen["run"][0] == fields(_lib.make_cfg(**plan.kernel_cfg()))
            assert seen["run"][0][flag] == unsplit_flag
    old = decider.Plan({k: v for k, v in plan.items() if k != "no_long_rows"}, regime="short_even")  # (saved without the key)
    assert old.kernel_cfg()["no_long_rows"] == 1 and decider.Plan(old, if_split=1).kernel_cfg()["no_long_rows"] == 0
    for regime in sweep.ALL_REGIMES:
        unsplit = [c for c in sweep.candidates(64, regime) if not c["if_split"] and c["vec_size"] == 1]
        skewed = regime.endswith("skewed")
        assert all(c["no_long_rows"] == int(not skewed) for c in unsplit)
        assert {c["gather_batch"] for c in unsplit} == ({8} if skewed else {4, 8, 16})


def test_the_long_rows_flag_is_a_flag_of_the_spmm(pspmm_lib):
    from paramspmm_ae_b200 import _lib
    one, null = ctypes.c_void_p(256), ctypes.c_void_p(0)
    assert pspmm_lib.pspmm_spmm_csr(one, one, one, one, one, 4, 4, 4, 16, 16, 16,
                                    ctypes.byref(_lib.make_cfg(no_long_rows=2)), null, null, 0, null) == _lib.PSPMM_E_CONFIG
    assert pspmm_lib.pspmm_sddmm_csr(one, one, one, one, one, 4, 4, 16, 16, 16,
                                     ctypes.byref(_lib.make_cfg(no_long_rows=1)), null, null, 0, null) == _lib.PSPMM_E_CONFIG


def test_edge_columns_are_compared_again_when_they_change():
    """The fused attention layer weights edges by the operator's own columns; the tensor a caller hands in is
    compared with them once, and again when it was written to or is another one."""
    import types
    from paramspmm_ae_b200 import gnn_conv
    P = types.SimpleNamespace(colIdx=torch.arange(7, dtype=torch.int32))
    edges = P.colIdx.clone().unsqueeze(-1)
    assert gnn_conv._is_operator_colidx(P, edges) and gnn_conv._is_operator_colidx(P, edges)
    held = P._colidx_checked
    assert gnn_conv._is_operator_colidx(P, edges[:]) and P._colidx_checked is held  # (a view of the same entries)
    edges[3] = 0
    assert not gnn_conv._is_operator_colidx(P, edges)
    edges[3] = 3
    assert gnn_conv._is_operator_colidx(P, edges)
    P.colIdx[0] = 5
    assert not gnn_conv._is_operator_colidx(P, edges)
    with torch.inference_mode():
        assert gnn_conv._is_operator_colidx(P, P.colIdx.clone())


def test_scores_are_kept_by_what_memory_they_take(monkeypatch):
    """Up to what they replace, up to a fixed size, up to a 32nd of the room; an allocator without figures is not asked."""
    from paramspmm_ae_b200 import gnn_conv
    asked = []
    monkeypatch.setattr(gnn_conv, "_room", lambda device: asked.append(device) or 32 * 4 * 5_000_000)
    few, many = torch.zeros(10, 4), torch.zeros(1).expand(1_500_000, 4)
    assert gnn_conv._keeps_scores(4_000_000, few) and gnn_conv._keeps_scores(6_000_000, many) and not asked
    assert gnn_conv._keeps_scores(5_000_000, few) and not gnn_conv._keeps_scores(5_000_001, few) and len(asked) == 2
    monkeypatch.undo()

    def no_figures(*a):
        raise RuntimeError("not supported")

    monkeypatch.setattr(torch.cuda, "get_per_process_memory_fraction", lambda d: 0.5)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: type("P", (), {"total_memory": 1000}))
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda d: {"allocated_bytes": {"all": {"current": 400}}})
    assert gnn_conv._room(None) == 100
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", no_figures)
    assert gnn_conv._room(None) == float("inf") and gnn_conv._keeps_scores(2**30, few)
