"""The work that users of this framework have it do, as cases that can be timed and compared.

``kind`` names the entry points a case goes through:

* ``spmm``       one sparse x dense product: the drop-in signatures (``csr_spmm``, ``csr_split_spmm``,
                 ``bcsr_spmm``) or an operator bound to the decider's plan (``pcsr_spmm.from_plan``)
* ``sddmm``      edge scores on a pattern (``csr_sddmm``, ``csr_split_sddmm``)
* ``attention``  ``agnn_fused``: scores, edge softmax and aggregation
* ``gcn``        one training step (forward and backward) of a network of ``GCNConv`` layers
* ``agnn``       forward and backward of one ``AGNNConv`` layer

Everything is fp32 with int32 indices, the only types the framework has.  ``graph`` is the kind of
matrix (``synth.py``): uniform random columns, a band around the diagonal, R-MAT, or a symmetric
power-law graph with self-loops and GCN weights.
"""
import math

import torch

from paramspmm_ae_b200 import decider, gnn_conv, ops, pcsr, synth


def listed():
    return [
        # A citation-size graph at the narrowest usual width: launches and host work are what counts.
        dict(name="spmm csr small", kind="spmm", layout="csr", graph="powerlaw", n=19717, nnz=197013, dim=16),
        # The row-split layout a loader hands over for a skewed graph, at a class-count width (odd: no vector loads).
        dict(name="spmm split odd width", kind="spmm", layout="split", graph="powerlaw", n=100003, nnz=2500003, dim=47),
        # The dim sweep's three million-row matrices (bench.py), through the decider's plan.
        dict(name="spmm plan uniform", kind="spmm", layout="plan", graph="uniform", n=1000000, nnz=16000000, dim=128),
        dict(name="spmm plan banded", kind="spmm", layout="plan", graph="banded", n=1000000, nnz=16000000, dim=64),
        dict(name="spmm plan rmat", kind="spmm", layout="plan", graph="rmat", n=1000000, nnz=16000000, dim=256),
        # 2 x 1 blocks on a locality-ordered matrix with an odd row count.
        dict(name="spmm block", kind="spmm", layout="block", graph="banded", n=200001, nnz=2400012, dim=96),
        # Edge scores for a host that keeps them (attention weights, link prediction) on a plain CSR graph.
        dict(name="sddmm csr", kind="sddmm", layout="csr", graph="powerlaw", n=169343, nnz=4000003, dim=100),
        # Inference of an attention layer with edge softmax.
        dict(name="attention softmax", kind="attention", layout="split", graph="powerlaw", n=120001, nnz=12000001, dim=128),
        # Training a small citation graph: many short launches per step.
        dict(name="gcn small step", kind="gcn", operators="legacy", graph="powerlaw", n=19717, nnz=197013, feats=500,
             hidden=16, classes=3, layers=2),
        # The full-size training step (workloads.gcn_forward_backward).
        dict(name="gcn large step", kind="gcn", operators="plan", graph="powerlaw", n=2449029, nnz=126249029, feats=100,
             hidden=256, classes=47, layers=3),
        # An attention layer trained on a medium graph whose rows are left unsplit ...
        dict(name="agnn layer medium", kind="agnn", layout="csr", graph="powerlaw", n=89251, nnz=900003, dim_in=128, dim=32),
        # ... and on the dense full-size graph (workloads.agnn_layer).
        dict(name="agnn layer large", kind="agnn", layout="split", graph="powerlaw", n=232965, nnz=114592965, dim_in=64,
             dim=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _graph(rng, case, nnz_max):
    """Rows and entries over the listed range; a mean row of at most 500 and at most 1/300 of the columns."""
    case["n"] = _log(rng, 5000, 2400000)
    if case["graph"] == "banded":
        deg = rng.randint(4, 32)
    elif case["graph"] == "uniform":
        deg = rng.randint(4, 48)
    else:
        deg = _log(rng, 5, min(500, max(6, case["n"] // 300)))
    deg = max(4, min(deg, nnz_max // case["n"]))
    case["nnz"] = case["n"] * deg
    if case["graph"] == "powerlaw":
        case["nnz"] = case["n"] + 2 * ((case["nnz"] - case["n"]) // 2)
    elif case["graph"] == "rmat":
        case["nnz"] -= rng.randint(0, case["n"] // 2)
    return case


def _width(rng):
    """A dense width in 16..256: mostly multiples of 16, as the decider's table has them, some of 4, some odd."""
    r = rng.random()
    return 16 * rng.randint(1, 16) if r < 0.6 else (4 * rng.randint(4, 64) if r < 0.8 else rng.randint(17, 255))


def draw(rng):
    kind = rng.choice(["spmm", "spmm", "spmm", "sddmm", "attention", "gcn", "agnn"])
    if kind == "spmm":
        layout = rng.choice(["csr", "split", "plan", "plan", "block"])
        graph = rng.choice({"csr": ["uniform", "banded", "powerlaw", "rmat"], "split": ["powerlaw", "rmat"],
                            "plan": ["uniform", "banded", "rmat", "powerlaw"], "block": ["banded"]}[layout])
        return _graph(rng, dict(kind=kind, layout=layout, graph=graph, dim=_width(rng)), 32000000)
    if kind == "sddmm":
        layout, graph = rng.choice(["csr", "split"]), rng.choice(["uniform", "banded", "powerlaw"])
        return _graph(rng, dict(kind=kind, layout=layout, graph=graph, dim=_width(rng)), 32000000)
    if kind == "gcn":
        case = dict(kind=kind, operators=rng.choice(["legacy", "plan"]), graph="powerlaw", feats=rng.randint(50, 500),
                    hidden=rng.choice([16, 32, 64, 128, 256]), classes=rng.randint(3, 64), layers=rng.choice([2, 3]))
        return _graph(rng, case, 64000000)
    case = dict(kind=kind, layout=rng.choice(["csr", "split"]), graph="powerlaw")
    if kind == "agnn":
        case.update(dim_in=16 * rng.randint(1, 16), dim=16 * rng.randint(1, 16))
    else:
        case.update(dim=4 * rng.randint(4, 64))
    return _graph(rng, case, 32000000)


def _matrix(case, seed, dev):
    n, nnz = case["n"], case["nnz"]
    if case["graph"] == "uniform":
        return synth.uniform_rows(n, nnz // n, seed=seed, device=dev)
    if case["graph"] == "banded":
        return synth.banded_rows(n, nnz // n, seed=seed, device=dev)
    if case["graph"] == "rmat":
        return synth.rmat((n - 1).bit_length(), nnz, n=n, seed=seed, device=dev)
    return synth.powerlaw_graph(n, (nnz - n) // 2, seed=seed, device=dev)


def _split(m):
    """The partition a loader builds: pieces of the mean row length rounded up to 32."""
    return ops.split_csr_device(m.rowPtr, decider.auto_granularity(decider.row_stats(m.rowPtr)["real_avg"]))


def _gradient(n, width, seed, dev):
    """What a mean cross-entropy loss sends back: (probabilities - label) / n, uneven class sizes."""
    g = torch.Generator(device=dev).manual_seed(seed)
    p = torch.softmax(torch.randn(n, width, generator=g, device=dev), 1)
    label = (torch.rand(n, generator=g, device=dev) ** 2 * width).long().clamp_(max=width - 1)
    p[torch.arange(n, device=dev), label] -= 1
    return p / n


def prepare(case, seed):
    dev = torch.device("cuda:0")
    m = _matrix(case, 5 * seed + 1, dev)
    n, s = m.n_rows, dict(kind=case["kind"], m=m)
    torch.manual_seed(5 * seed + 2)
    if case["kind"] == "gcn":
        dims = [case["hidden"]] * (case["layers"] - 1) + [case["classes"]]
        stats = decider.row_stats(m.rowPtr, m.colIdx)
        s["operators"] = {}
        for d in set(dims):
            plan = decider.choose(stats, d)
            if case["operators"] == "plan":
                s["operators"][d] = pcsr.pcsr_spmm.from_plan(plan, m.rowPtr, m.colIdx, m.val)
            else:
                rp, tr = _split(m) if plan["if_split"] else (m.rowPtr, None)
                s["operators"][d] = pcsr.pcsr_spmm(None, 1, tr is not None, n, m.nnz, rp, m.colIdx, m.val, tr, CF=1,
                                                   blkWarpNum=8)
        s["layers"] = [gnn_conv.GCNConv(a, b).to(dev) for a, b in zip([case["feats"]] + dims, dims)]
        s["X"] = synth.dense_normal(n, case["feats"], 5 * seed + 3, dev)
        s["y"] = torch.randint(0, case["classes"], (n,), device=dev)
        return s
    dim = case["dim"]
    if case["kind"] == "agnn":
        rp, tr = _split(m) if case["layout"] == "split" else (m.rowPtr, None)
        P = pcsr.pcsr_sddmm(None, 1, tr is not None, n, m.nnz, rp, m.colIdx, m.val, tr, CF=(dim + 31) // 32, blkWarpNum=8)
        s["operators"] = {dim: P}
        s["layer"] = gnn_conv.AGNNConv(case["dim_in"], dim).to(dev)
        X = synth.dense_normal(n, case["dim_in"], 5 * seed + 3, dev)
        s["X"] = (X / X.norm(dim=1, keepdim=True)).requires_grad_(True)
        s["edges"] = m.colIdx.unsqueeze(-1)
        s["G"] = _gradient(n, dim, 5 * seed + 4, dev)
        return s
    if case["kind"] == "spmm":
        s["X"] = synth.dense_uniform(n, dim, 5 * seed + 3, dev)
        if case["layout"] == "plan":
            stats = decider.row_stats(m.rowPtr, m.colIdx)
            P = pcsr.pcsr_spmm.from_plan(decider.choose(stats, dim), m.rowPtr, m.colIdx, m.val)
            s["call"], s["args"] = P.GIN_spmm, ()
            return s
        if case["layout"] == "block":
            arrays = ops.bcsr_from_csr(m.rowPtr.cpu(), m.colIdx.cpu(), m.val.cpu(), m.n_cols, 2)
            s["call"], s["args"] = ops.bcsr_spmm, tuple(t.to(dev) for t in arrays)
        elif case["layout"] == "split":
            rp, tr = _split(m)
            s["call"], s["args"] = ops.csr_split_spmm, (rp, m.colIdx, m.val, tr)
        else:
            s["call"], s["args"] = ops.csr_spmm, (m.rowPtr, m.colIdx, m.val)
        s["args"] += (min(8, (dim + 31) // 32), 8)
        return s
    X = synth.dense_normal(n, dim, 5 * seed + 3, dev)
    s["X"] = X / X.norm(dim=1, keepdim=True)
    s["rp"], s["tr"] = _split(m) if case["layout"] == "split" else (m.rowPtr, None)
    return s


def run(s):
    m, X = s["m"], s["X"]
    if s["kind"] == "spmm":
        return s["call"](X, *s["args"])
    if s["kind"] == "sddmm":
        CF = min(4, (X.shape[1] + 31) // 32)
        if s["tr"] is None:
            return ops.csr_sddmm(X, X, s["rp"], m.colIdx, m.val, CF, 8)
        return ops.csr_split_sddmm(X, X, s["rp"], m.colIdx, m.val, s["tr"], CF, 8)
    if s["kind"] == "attention":
        return ops.agnn_fused(X, X, s["rp"], m.colIdx, 1.0, True, target_row=s["tr"],
                              n_out_rows=None if s["tr"] is None else X.shape[0])
    if s["kind"] == "agnn":
        layer = s["layer"]
        X.grad = layer.weights.grad = layer.attention_w.grad = None
        out = layer(X, s["operators"], s["edges"])
        out.backward(s["G"])
        return dict(out=out, dX=X.grad, dW=layer.weights.grad, dbeta=layer.attention_w.grad)
    h, last = X, s["layers"][-1]
    for layer in s["layers"]:
        layer.weights.grad = None
        h = layer(h, s["operators"])
        if layer is not last:
            h = torch.relu(h)
    loss = torch.nn.functional.cross_entropy(h, s["y"])
    loss.backward()
    return dict(loss=loss, logits=h, grads=[layer.weights.grad for layer in s["layers"]])


def work(case):
    n, nnz, kind = case["n"], case["nnz"], case["kind"]
    pattern = 4 * (n + 1) + 4 * nnz
    if kind == "gcn":
        f, c = case["feats"], case["classes"]
        dims = [f] + [case["hidden"]] * (case["layers"] - 1) + [c]
        weights = sum(a * b for a, b in zip(dims, dims[1:]))
        # per layer: projection and aggregation, their transposes, and (but for the first) the input gradient
        flops = sum(4 * n * a * b + 4 * nnz * b for a, b in zip(dims, dims[1:]))
        flops += sum(2 * n * a * b for a, b in zip(dims[1:], dims[2:]))
        return {"bytes": pattern + 4 * nnz + 4 * n * (f + c) + 8 * n + 8 * weights, "flops": flops}
    if kind == "agnn":
        i, d = case["dim_in"], case["dim"]
        # forward: scores and aggregation; backward: the aggregation's transpose and the edge scores of the gradient
        return {"bytes": pattern + 4 * nnz + 4 * n * (2 * i + 2 * d) + 8 * i * d, "flops": 8 * nnz * d + 6 * n * i * d}
    d = case["dim"]
    if kind == "attention":
        return {"bytes": pattern + 8 * n * d, "flops": 4 * nnz * d}
    return {"bytes": pattern + 4 * nnz + 8 * n * d, "flops": 2 * nnz * d}


def tolerance(case):
    """fp32 sums in another order; the steps of several dependent products (and the attention
    weight's gradient, one sum over all edges) accumulate a little more."""
    return {"rel": 3e-5} if case["kind"] in ("gcn", "agnn") else {"rel": 1e-5}
