"""The autograd Functions where torch.autograd.Function does more than run a forward and a backward: traces, forward-mode
differentiation, torch.func's transforms, dispatch modes.  What it carries gives its results, what it refuses is refused."""
import pytest
import torch as th
import torch.autograd.forward_ad as forward_ad
from torch.utils._python_dispatch import TorchDispatchMode

from helpers import chunked, random_graph
from custom_op_benchmark_b200 import graphop, wrapper

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
N, H, D = 60, 2, 16


def _calls():
    g = random_graph(N, N, [7] * N, 5)
    r = [t.to(DEV) for t in chunked(g, 32)]
    c = [t.to(DEV) for t in chunked(g, 32, transposed=True)]
    plans = graphop.GraphPlan(*r, N), graphop.GraphPlan(*c, N)
    gen = th.Generator().manual_seed(3)
    node, edge, rel = (th.randn(*s, generator=gen).to(DEV) for s in ((N, H, D), (g.n_edges, H), (g.n_edges, D)))
    return {
        "SparseSoftmax": (edge, lambda x: wrapper.SparseSoftmax.apply(*r[:3], x)),
        "MaskedMMCSR": (node, lambda x: wrapper.MaskedMMCSR.apply(*r, *c, x, node)),
        "NodeMulEdge": (node, lambda x: wrapper.NodeMulEdge.apply(*r[:3], x, rel)),
        "VectorSPMM": (edge, lambda x: wrapper.VectorSPMM.apply(*r, *c, x, node)),
        "GraphAttention": (node, lambda x: wrapper.GraphAttention.apply(r[0], r[1], r[3], c[0], c[1], c[3], x, node, node, 0.25,
                                                                       c[2])),
        "GraphAttentionBias": (node, lambda x: wrapper.GraphAttentionBias.apply(r[0], r[1], r[3], *c, x, node, node, rel, 0.25)),
        "GraphAttentionPlanned": (node, lambda x: wrapper.GraphAttentionPlanned.apply(*plans, x, node, node, 0.25)),
    }


NAMES = ["SparseSoftmax", "MaskedMMCSR", "NodeMulEdge", "VectorSPMM", "GraphAttention", "GraphAttentionBias",
         "GraphAttentionPlanned"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning", "ignore::DeprecationWarning")
def test_a_trace_computes(name):
    x, call = _calls()[name]
    traced = th.jit.trace(call, (x.clone(),), check_trace=False)   # not the tensor the call holds as a constant
    other = x.flip(0).contiguous()
    assert th.equal(traced(other), call(other))


@pytest.mark.parametrize("name", NAMES)
def test_forward_mode_is_refused(name):
    x, call = _calls()[name]
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(x, th.ones_like(x))
        with pytest.raises(NotImplementedError, match="jvp"):
            call(dual)


@pytest.mark.parametrize("name", NAMES)
def test_functional_transforms_are_refused(name):
    x, call = _calls()[name]
    with pytest.raises(RuntimeError, match="setup_context|generate_vmap_rule"):
        th.func.vmap(call)(th.stack([x, x]))
    with pytest.raises(RuntimeError, match="setup_context"):
        th.func.grad(lambda t: call(t).sum())(x)


@pytest.mark.parametrize("name", NAMES)
def test_dispatch_modes_see_the_allocations(name):
    x, call = _calls()[name]
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    want = call(x)
    leaf = x.clone().requires_grad_(True)
    with Mode():
        out = call(leaf)
    assert th.equal(out, want) and any("empty" in f for f in seen)
    assert th.autograd.grad(out, leaf, th.ones_like(out))[0].shape == x.shape
