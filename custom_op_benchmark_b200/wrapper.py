"""Autograd wiring of the graphop ops: the four `torch.autograd.Function` classes of the
reference (wrapper.py:8-55) with the same names, the same positional `apply` signatures and
the same `None` gradients for every index argument, plus `GraphAttention`, the fused chain.

`apply` of these classes runs the same Function in native code (csrc/binding/graphop_native.cpp): on small graphs the
Python forward and backward below took several times as long as the kernels.  They are what `apply` runs when `_g` is
another module with the ops of `graphop` (the compiled module of that name, say), and where torch.autograd.Function does
more than the native node: while torch.jit.trace records, under torch.func's transforms and dispatch modes, on tensors
with a forward-mode tangent; and all there is in a package built without the compiled modules.
"""
from torch.autograd import Function

from . import graphop as _g
from . import graphop as _graphop
from . import native_functions_if_built
from .part_csr import partition_csr  # noqa: F401  (the reference wrapper re-exports it, wrapper.py:4)

__all__ = ["SparseSoftmax", "MaskedMMCSR", "NodeMulEdge", "VectorSPMM", "GraphAttention", "GraphAttentionBias", "GraphAttentionPlanned",
           "graph_attention", "partition_csr", "chunk_size"]

chunk_size = 32  # wrapper.py:6


def _native():
    """The native module where `apply` goes through it."""
    return native_functions_if_built() if _g is _graphop else None


def _run(function, name, *args):
    """`function` on `args`: `name` of the native module, or, where that leaves the call to it (see above), the Function."""
    native = _native()
    out = getattr(native, name)(*args) if native is not None else None
    if out is not None:
        return out
    return super(function, function).apply(*args)


class SparseSoftmax(Function):
    """wrapper.py:8-18"""

    @staticmethod
    def apply(row, indptr, eid, x):
        return _run(SparseSoftmax, "sparse_softmax", row, indptr, eid, x)

    @staticmethod
    def forward(ctx, row, indptr, eid, x):
        y = _g.sparse_softmax_forward(row, indptr, eid, x)
        ctx.save_for_backward(row, indptr, eid, y)
        return y

    @staticmethod
    def backward(ctx, dy):
        row, indptr, eid, y = ctx.saved_tensors
        return None, None, None, _g.sparse_softmax_backward(row, indptr, eid, y, dy.contiguous())


class MaskedMMCSR(Function):
    """wrapper.py:20-30"""

    @staticmethod
    def apply(row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B):
        return _run(MaskedMMCSR, "maskedmm_csr", row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B)

    @staticmethod
    def forward(ctx, row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B):
        ctx.save_for_backward(row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B)
        return _g.maskedmm_csr_forward(row, indptr_r, eid_r, indices_r, A, B)

    @staticmethod
    def backward(ctx, grad):
        row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B = ctx.saved_tensors
        dA, dB = _g.maskedmm_csr_backward(row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B,
                                          grad)
        return None, None, None, None, None, None, None, None, dA, dB


class NodeMulEdge(Function):
    """wrapper.py:32-42"""

    @staticmethod
    def apply(row, indptr, eid, A, B):
        return _run(NodeMulEdge, "node_mul_edge", row, indptr, eid, A, B)

    @staticmethod
    def forward(ctx, row, indptr, eid, A, B):
        ctx.save_for_backward(row, indptr, eid, A, B)
        return _g.node_mul_edge_forward(row, indptr, eid, A, B)

    @staticmethod
    def backward(ctx, grad):
        row, indptr, eid, A, B = ctx.saved_tensors
        dA, dB = _g.node_mul_edge_backward(row, indptr, eid, A, B, grad)
        return None, None, None, dA, dB


class VectorSPMM(Function):
    """wrapper.py:44-55"""

    @staticmethod
    def apply(row, indptr, eid, indices, col, ptr_t, eid_t, indices_t, edata, x):
        return _run(VectorSPMM, "vector_spmm", row, indptr, eid, indices, col, ptr_t, eid_t, indices_t, edata, x)

    @staticmethod
    def forward(ctx, row, indptr, eid, indices, col, ptr_t, eid_t, indices_t, edata, x):
        y = _g.vector_spmm_forward(row, indptr, eid, indices, edata, x)
        ctx.save_for_backward(row, indptr, eid, indices, col, ptr_t, eid_t, indices_t, edata, x)
        return y

    @staticmethod
    def backward(ctx, dy):
        row, indptr, eid, indices, col, ptr_t, eid_t, indices_t, edata, x = ctx.saved_tensors
        dedata, dx = _g.vector_spmm_backward(row, indptr, eid, indices, col, ptr_t, eid_t, indices_t, edata,
                                             dy.contiguous(), x)
        return None, None, None, None, None, None, None, None, dedata, dx


class GraphAttention(Function):
    """O = VectorSPMM(SparseSoftmax(scale * MaskedMMCSR(Q, K)), V) in one kernel per direction.

    ``apply(row, indptr, indices, col, indptr_t, indices_t, Q, K, V, scale, eid_t=None)``; no edge tensor is
    materialised and only the (n, h) log-sum-exp is saved.  ``eid_t`` (the transposed CSR's edge ids, valid
    when the row CSR's edge ids are its positions) lets the backward pass each edge's probability from its
    destination-side kernel to its source-side kernel instead of recomputing it."""

    @staticmethod
    def apply(row, indptr, indices, col, indptr_t, indices_t, Q, K, V, scale, eid_t=None):
        # the same graph tensors come back every step: their plans are built once and looked up here, so this per-call
        # signature runs the planned kernels (and, on a dense band in bfloat16, the tensor-core ones)
        native = _native()
        if native is not None and _g.plan_cache_size > 0 and indices.numel() > 0:
            plans = _g.cached_plan(row, indptr, None, indices, Q.size(0)), _g.cached_plan(col, indptr_t, eid_t, indices_t,
                                                                                         K.size(0))
            out = native.attention_planned(plans[0].native(), plans[1].native(), Q, K, V, scale)
            if out is not None:
                return out
        return super(GraphAttention, GraphAttention).apply(row, indptr, indices, col, indptr_t, indices_t, Q, K, V, scale,
                                                           eid_t)

    @staticmethod
    def forward(ctx, row, indptr, indices, col, indptr_t, indices_t, Q, K, V, scale, eid_t=None):
        cached = getattr(_g, "cached_plan", None)
        if cached is not None and getattr(_g, "plan_cache_size", 0) > 0 and indices.numel() > 0:
            # the same graph tensors come back every step: their plans are built once and looked up here, so this
            # per-call signature runs the planned kernels (and, on a dense band in bfloat16, the tensor-core ones)
            ctx.plans = (cached(row, indptr, None, indices, Q.size(0)), cached(col, indptr_t, eid_t, indices_t, K.size(0)))
            o, lse = _g.attention_forward_planned(ctx.plans[0], Q, K, V, scale)
        else:
            ctx.plans = None
            o, lse = _g.attention_forward(row, indptr, indices, Q, K, V, scale)
        ctx.save_for_backward(row, indptr, indices, col, indptr_t, indices_t, Q, K, V, o, lse)
        ctx.scale = scale
        ctx.eid_t = eid_t
        return o

    @staticmethod
    def backward(ctx, d_o):
        row, indptr, indices, col, indptr_t, indices_t, Q, K, V, o, lse = ctx.saved_tensors
        if ctx.plans is not None:
            dq, dk, dv = _g.attention_backward_planned(ctx.plans[0], ctx.plans[1], Q, K, V, o, lse, d_o, ctx.scale)
        else:
            dq, dk, dv = _g.attention_backward(row, indptr, indices, col, indptr_t, indices_t, Q, K, V, o, lse, d_o,
                                               ctx.scale, eid_t=ctx.eid_t)
        return None, None, None, None, None, None, dq, dk, dv, None, None


class GraphAttentionBias(Function):
    """The attention layer with a relative-position term, fused:
    O = VectorSPMM(SparseSoftmax(scale * (MaskedMMCSR(Q, K) + NodeMulEdge(Q, rel))), V), the chain the reference's
    ops compose (wrapper.py:20-55) without the (e, h) score tensors.

    ``apply(row, indptr, indices, col, indptr_t, eid_t, indices_t, Q, K, V, rel, scale)``; ``rel`` is (e, d), one row
    per edge in row-CSR order, shared by the heads; ``eid_t`` gives for every position of the transposed CSR the
    row-CSR position of the same edge."""

    @staticmethod
    def apply(row, indptr, indices, col, indptr_t, eid_t, indices_t, Q, K, V, rel, scale):
        return _run(GraphAttentionBias, "attention_bias", row, indptr, indices, col, indptr_t,
                    eid_t, indices_t, Q, K, V, rel, scale)

    @staticmethod
    def forward(ctx, row, indptr, indices, col, indptr_t, eid_t, indices_t, Q, K, V, rel, scale):
        o, lse = _g.attention_bias_forward(row, indptr, indices, Q, K, V, rel, scale)
        ctx.save_for_backward(row, indptr, indices, col, indptr_t, eid_t, indices_t, Q, K, V, rel, o, lse)
        ctx.scale = scale
        return o

    @staticmethod
    def backward(ctx, d_o):
        row, indptr, indices, col, indptr_t, eid_t, indices_t, Q, K, V, rel, o, lse = ctx.saved_tensors
        dq, dk, dv, d_rel = _g.attention_bias_backward(row, indptr, indices, col, indptr_t, eid_t, indices_t, Q, K, V,
                                                       rel, o, lse, d_o, ctx.scale)
        return None, None, None, None, None, None, None, dq, dk, dv, d_rel, None


class GraphAttentionPlanned(Function):
    """GraphAttention on graph plans: ``apply(plan_r, plan_t, Q, K, V, scale)`` with ``graphop.GraphPlan`` objects of
    the row CSR and of the transposed CSR (the latter built with its edge ids).  Nothing that depends on the graph
    alone is recomputed per call."""

    @staticmethod
    def apply(plan_r, plan_t, Q, K, V, scale):
        native = _native()
        if native is not None:
            out = native.attention_planned(plan_r.native(), plan_t.native(), Q, K, V, scale)
            if out is not None:
                return out
        return super(GraphAttentionPlanned, GraphAttentionPlanned).apply(plan_r, plan_t, Q, K, V, scale)

    @staticmethod
    def forward(ctx, plan_r, plan_t, Q, K, V, scale):
        o, lse = _g.attention_forward_planned(plan_r, Q, K, V, scale)
        ctx.save_for_backward(Q, K, V, o, lse)
        ctx.plans, ctx.scale = (plan_r, plan_t), scale
        return o

    @staticmethod
    def backward(ctx, d_o):
        Q, K, V, o, lse = ctx.saved_tensors
        dq, dk, dv = _g.attention_backward_planned(ctx.plans[0], ctx.plans[1], Q, K, V, o, lse, d_o, ctx.scale)
        return None, None, dq, dk, dv, None


def graph_attention(row, indptr, eid, indices, col, indptr_t, eid_t, indices_t, Q, K, V, scale):
    """The attention chain with the argument list of the unfused ops: the fused kernels when the
    shape allows, otherwise MaskedMMCSR -> scale -> SparseSoftmax -> VectorSPMM."""
    if _g.attention_supported(Q):
        return GraphAttention.apply(row, indptr, indices, col, indptr_t, indices_t, Q, K, V, scale)
    s = MaskedMMCSR.apply(row, indptr, eid, indices, col, indptr_t, eid_t, indices_t, Q, K) * scale
    p = SparseSoftmax.apply(row, indptr, eid, s)
    return VectorSPMM.apply(row, indptr, eid, indices, col, indptr_t, eid_t, indices_t, p, V)
