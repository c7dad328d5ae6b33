"""GCN / GIN / AGNN layers over the PCSR operators: mirror of the reference's ``gnn_conv.py``.

Same module and autograd-function names, constructor arguments and forward signatures
(gnn_conv.py:13-238 of the reference).  The layer semantics are the reference's:

* GCN   forward  A (H W); backward AG = A G (A itself: the normalised adjacency is symmetric),
        dH = AG W^T, dW = H^T AG.  With REORDER_NARROW_FIRST (off by default) layers that widen
        their input aggregate first instead, (A H) W.
* GIN   forward  (A X) W; backward dW = (A X)^T G, dX = A (G W^T).
* AGNN  forward  X' = X W, e = SDDMM(X', X') * beta, out = SpMM(e, X'); no edge softmax and no
        row normalisation (the reference has none); the gradient w.r.t. beta follows the
        reference's expression (gnn_conv.py:164-172).
"""
from __future__ import annotations

import math

import torch

from . import ops

n_heads = 1


# When a GCN layer widens its input (fan-in < fan-out) the aggregation is cheaper before the
# projection: A (H W) = (A H) W, and the SpMM then runs at the narrower width.  The reference always
# aggregates after the projection (SpCONV/SpCONV.h:43-72), and so does this module by default, so
# that layer outputs and gradients are the reference's up to the summation order inside the SpMM.
# Setting this to True is an opt-in: results then differ from the reference's by fp32
# re-association of the two products (both orders are tested against fp64 algebra), the backward
# keeps A H instead of H, and the operator is looked up under the input width when the caller's
# dictionary has one for it.
REORDER_NARROW_FIRST = False


def _aggregate(P, X):
    out = P.GIN_spmm(X.contiguous())
    return out[: X.shape[0]] if out.shape[0] != X.shape[0] else out  # block layouts pad the row count


class GCNFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, H, weight, ParamSpMM):
        ctx.ParamSpMM = ParamSpMM
        ctx.narrow_first = bool(REORDER_NARROW_FIRST and weight.shape[0] < weight.shape[1])
        if ctx.narrow_first:
            AH = _aggregate(ParamSpMM, H)
            ctx.save_for_backward(AH, weight)
            return torch.mm(AH, weight)
        ctx.save_for_backward(H, weight)
        return ParamSpMM.forward(H, weight)

    @staticmethod
    def backward(ctx, d_output):
        P = ctx.ParamSpMM
        d_output = d_output.contiguous()
        if ctx.narrow_first:
            # dW = (A H)^T G with A H kept from the forward; dH = A (G W^T) (A is symmetric),
            # skipped when the layer input needs no gradient (the first layer).
            AH, weight = ctx.saved_tensors
            d_weight = ops.dense_mm(AH, d_output, transA=True)
            d_input = _aggregate(P, ops.dense_mm(d_output, weight, transB=True)) if ctx.needs_input_grad[0] else None
            return d_input, d_weight, None
        H, weight = ctx.saved_tensors
        if ctx.needs_input_grad[0]:
            d_input, d_weight = P.backward(d_output, H, weight)
        else:  # the first layer: dH = AG W^T is not formed (the reference forms and drops it)
            d_input, d_weight = P.backward(d_output, H, weight, input_grad=False)
        return d_input, d_weight, None


class GINFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, X, weight, ParamSpMM):
        X_agg = ParamSpMM.GIN_spmm(X)
        ctx.save_for_backward(X_agg, weight)
        ctx.ParamSpMM = ParamSpMM
        return torch.mm(X_agg, weight)

    @staticmethod
    def backward(ctx, d_output):
        X_agg, weight = ctx.saved_tensors
        d_weight = ops.dense_mm(X_agg, d_output, transA=True)
        d_input = ctx.ParamSpMM.GIN_spmm(ops.dense_mm(d_output, weight, transB=True).contiguous())
        return d_input, d_weight, None


# Under torch.no_grad() an AGNN layer on a plain or split CSR operator runs as the fused kernel
# (SDDMM -> scale -> SpMM in one pass).  Set to False to always use the three-kernel composition.
FUSE_AGNN_INFERENCE = True

# With gradients enabled the same layers run AGNNFusedFunction: the forward is the fused kernel, which leaves
# the edge scores for the backward (4 bytes per edge; the reference's composition writes the attention values in
# the forward and the score gradient in the backward, gnn_conv.py:130-180).  Outputs and gradients are the
# reference's up to fp32 summation order.
# Set to False to train through the three-kernel composition (AGNNFunction).  ``AGNNConv.keep_scores`` chooses per layer
# whether the scores are kept.
FUSE_AGNN_TRAINING = True
_SCORES_UNASKED = 16 << 20  # bytes up to which scores are kept without a look at the free memory (12 us of host time)


def _room(device):
    """Bytes of a device that torch has not handed out, within the limit of the process.  (The driver's own figure for free memory
    takes 0.2 ms, at times several.)"""
    try:
        limit = torch.cuda.get_per_process_memory_fraction(device) * torch.cuda.get_device_properties(device).total_memory
        return limit - torch.cuda.memory_stats_as_nested_dict(device)["allocated_bytes"]["all"]["current"]
    except (RuntimeError, KeyError):  # an allocator of the host's, which keeps no figures: its allocation tells
        return float("inf")


def _keeps_scores(nnz, Xp):
    """Whether the scores of ``nnz`` edges may take memory until the backward.  They stand in for the projected features, up to
    whose size a step takes no more than without; beyond it up to a 32nd of what is free, so that the layers behind this one find
    the room they found without (a second gather per edge instead: 115 M edges, 64 columns, a step of 4.1 ms becomes 6.1)."""
    nbytes = 4 * nnz
    return nbytes <= _SCORES_UNASKED or nbytes <= Xp.numel() * Xp.element_size() or 32 * nbytes <= _room(Xp.device)


def _beta(attention_w):
    """The attention weight as the one float on the device that the fused passes read."""
    return attention_w.detach().reshape(1).to(torch.float32)


def _can_fuse(P, dim):
    return getattr(P, "vec_size", 1) == 1 and dim % 4 == 0 and dim <= 256


def _is_operator_colidx(P, colIdx):
    """The fused backward weights edges by the operator's own column ids; callers pass them as an
    [nnz, 1] column (GNN.py:224-225).  Compared once per content of a tensor, not per step: the operator holds
    the last one it compared, so that its memory is not another tensor's meanwhile, and its version."""
    own = P.colIdx
    if colIdx.is_inference() or own.is_inference():  # (these keep no version)
        return _same_entries(colIdx, own)
    seen = P.__dict__.get("_colidx_checked")
    if seen is None or own is not seen[1] or (colIdx._version, own._version) != seen[2] or (
            colIdx is not seen[0] and (colIdx.data_ptr() != seen[0].data_ptr() or colIdx.shape != seen[0].shape
                                       or colIdx.stride() != seen[0].stride() or colIdx.dtype != seen[0].dtype)):
        seen = P._colidx_checked = (colIdx, own, (colIdx._version, own._version), _same_entries(colIdx, own))
    return seen[3]


def _same_entries(colIdx, own):
    flat = colIdx.reshape(-1)
    return bool(flat.shape == own.shape and flat.dtype == own.dtype and torch.equal(flat, own))


class AGNNFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, X, weights, attention_w, ParamSpMM, colIdx):
        X_prime = ops.dense_mm(X, weights)
        edge = ParamSpMM.AGNN_sddmm(X_prime)
        # [n_edges] for CSR, [n_blocks, V] for block layouts; one attention head
        edge_attentions = (edge * attention_w.reshape(())).contiguous()
        out = ParamSpMM.AGNN_spmm(edge_attentions, X_prime)
        ctx.save_for_backward(X, weights, edge_attentions)
        ctx.colIdx, ctx.ParamSpMM = colIdx, ParamSpMM
        return out

    @staticmethod
    def backward(ctx, d_output):
        P = ctx.ParamSpMM
        X, weights, edge_attentions = ctx.saved_tensors
        d_output = d_output.contiguous()
        d_prime = P.AGNN_spmm(edge_attentions, d_output)
        d_input = ops.dense_mm(d_prime, weights, transB=True)
        d_weights = ops.dense_mm(X, d_prime, transA=True)
        d_att = P.AGNN_sddmm(d_output)
        if d_att.dim() != 1:
            d_att = d_att.reshape(-1)[P.mask]  # back to CSR entry order
        d_attention_w = torch.mm(d_att[None, :].expand(n_heads, -1), ctx.colIdx.float()).transpose(0, 1)
        return d_input, d_weights, d_attention_w, None, None


class AGNNFusedFunction(torch.autograd.Function):
    """AGNN layer on a CSR / split-CSR operator in one pass over the pattern per direction.

    forward   X' = X W,  out_i = sum_j beta <X'_i, X'_j> X'_j     (one fused pass, which leaves the scores)
    backward  D_i = sum_j beta <X'_i, X'_j> G_j           (gradient rows gathered, scores read; with ``keep_scores=False``, or
              little room for them, the rows of X' are kept and gathered again and the scores recomputed)
              dX = D W^T,  dW = X^T D                                      (gnn_conv.py:157-160)
              d_beta = sum over edges of <G_i, G_j> * colIdx[e]              (gnn_conv.py:163-172: the
              reference multiplies the score gradient by the column-index column it is handed), summed
              in the same pass while the gradient row is in registers.
    The attention weight stays on the device (reading it back made every forward wait for the GPU).
    Like the reference's backward, the edge values are treated as constants with respect to X'."""

    @staticmethod
    def forward(ctx, X, weights, attention_w, P, colIdx, keep_scores=True):
        Xp = ops.dense_mm(X, weights)
        beta, scores = _beta(attention_w), None
        if keep_scores and _keeps_scores(P.colIdx.shape[0], Xp):
            try:
                scores = torch.empty(P.colIdx.shape[0], dtype=torch.float32, device=Xp.device)
            except torch.cuda.OutOfMemoryError:
                pass
        if scores is None:
            beta = beta.clone()  # (the backward uses the value of this forward)
        out = ops.agnn_layer_forward(Xp, P.rowPtr, P.colIdx, beta, P.target_row, scores)
        ctx.save_for_backward(X, weights, *((Xp, beta) if scores is None else (scores,)))
        ctx.P = P
        return out

    @staticmethod
    def backward(ctx, d_output):
        X, weights, *rest = ctx.saved_tensors
        Xp, beta, scores = (*rest, None) if len(rest) == 2 else (None, None, *rest)
        P = ctx.P
        D, d_att = ops.agnn_layer_backward(Xp, d_output.contiguous(), P.rowPtr, P.colIdx, beta, P.target_row,
                                           beta_grad=ctx.needs_input_grad[2], scores=scores)
        d_input = ops.dense_mm(D, weights, transB=True) if ctx.needs_input_grad[0] else None
        d_weights = ops.dense_mm(X, D, transA=True) if ctx.needs_input_grad[1] else None
        return d_input, d_weights, d_att, None, None, None


class _Conv(torch.nn.Module):
    def __init__(self, input_dim, output_dim):
        super().__init__()
        self.weights = torch.nn.Parameter(torch.randn(input_dim, output_dim))
        self.reset_parameters()

    def reset_parameters(self):
        stdv = 1.0 / math.sqrt(self.weights.size(1))
        self.weights.data.uniform_(-stdv, stdv)

    def _operator(self, spmm_dict):
        dim = self.weights.size(1)
        if dim not in spmm_dict:
            raise ValueError("SpMMDecider not support dim: " + str(dim))
        return spmm_dict[dim]


class GCNConv(_Conv):
    def forward(self, H, spmm_dict):
        P = self._operator(spmm_dict)
        if REORDER_NARROW_FIRST and self.weights.size(0) < self.weights.size(1):
            P = spmm_dict.get(self.weights.size(0), P)  # the aggregation runs at the input width
        return GCNFunction.apply(H, self.weights, P)


class GINConv(_Conv):
    def forward(self, X, spmm_dict):
        return GINFunction.apply(X, self.weights, self._operator(spmm_dict))


class AGNNConv(_Conv):
    # False: a fused training step keeps the projected features and recomputes the edge scores in the backward, for a
    # network that has no room for 4 bytes per edge and layer
    keep_scores = True

    def __init__(self, input_dim, output_dim):
        super().__init__(input_dim, output_dim)
        self.attention_w = torch.nn.Parameter(torch.randn(1, n_heads))

    def forward(self, X, spmm_dict, colIdx):
        P = self._operator(spmm_dict)
        if FUSE_AGNN_INFERENCE and not torch.is_grad_enabled() and _can_fuse(P, self.weights.size(1)):
            # No gradient will be asked for: scores, scaling and aggregation in one kernel, without
            # the per-edge array the backward would need.
            Xp = ops.dense_mm(X, self.weights)
            out = ops.agnn_layer_forward(Xp, P.rowPtr, P.colIdx, _beta(self.attention_w), P.target_row)
            return out[: P.mtx_nodes if P.target_row is not None else P.rowPtr.shape[0] - 1]
        if (FUSE_AGNN_TRAINING and torch.is_grad_enabled() and _can_fuse(P, self.weights.size(1))
                and _is_operator_colidx(P, colIdx)):
            return AGNNFusedFunction.apply(X, self.weights, self.attention_w, P, colIdx, self.keep_scores)
        return AGNNFunction.apply(X, self.weights, self.attention_w, P, colIdx)
