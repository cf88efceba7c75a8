"""What the native autograd Functions keep, and for how long: device memory beyond the tensors a call was given and
returned, one graph's backward from several threads."""
import threading

import pytest
import torch as th

from helpers import chunked, random_graph
from custom_op_benchmark_b200 import wrapper

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
N, H, D = 4000, 4, 32


@pytest.fixture(scope="module")
def tables():
    deg = th.randint(0, 100, (N,), generator=th.Generator().manual_seed(1))
    g = random_graph(N, N, deg, 2)
    return ([t.to(DEV) for t in chunked(g, 32, dtype=th.int64)],
            [t.to(DEV) for t in chunked(g, 32, transposed=True, dtype=th.int64)], g.n_edges)


def _normal(*shape, seed):
    return th.randn(*shape, generator=th.Generator().manual_seed(seed)).to(DEV)


def _call(name, tables):
    """(apply on fresh leaves, the leaves) of each Function that takes chunk tables."""
    r, c, e = tables
    node, edge = [_normal(N, H, D, seed=k) for k in range(3)], _normal(e, H, seed=3)
    if name == "SparseSoftmax":
        return wrapper.SparseSoftmax, r[:3], [edge]
    if name == "MaskedMMCSR":
        return wrapper.MaskedMMCSR, [*r, *c], node[:2]
    if name == "NodeMulEdge":
        return wrapper.NodeMulEdge, r[:3], [node[0], _normal(e, D, seed=4)]
    if name == "VectorSPMM":
        return wrapper.VectorSPMM, [*r, *c], [edge, node[0]]
    return wrapper.GraphAttentionBias, [r[0], r[1], r[3], *c], [*node, _normal(e, D, seed=4), D ** -0.5]


FUNCTIONS = ["SparseSoftmax", "MaskedMMCSR", "NodeMulEdge", "VectorSPMM", "GraphAttentionBias"]


def _leaves(given):
    return [t.clone().requires_grad_(True) if isinstance(t, th.Tensor) else t for t in given]


def _tensors(given):
    return [t for t in given if isinstance(t, th.Tensor)]


@pytest.mark.parametrize("name", FUNCTIONS)
def test_one_graph_backward_from_several_threads(tables, name):
    function, tabs, given = _call(name, tables)
    leaves = _leaves(given)
    out = function.apply(*tabs, *leaves)
    grad = _normal(*out.shape, seed=9)
    want = th.autograd.grad(out, _tensors(leaves), grad, retain_graph=True)
    out = function.apply(*tabs, *leaves)   # a graph no backward has run on yet
    th.cuda.synchronize()
    got, errors, ready = [], [], threading.Barrier(4)

    def work():
        try:
            ready.wait()
            for _ in range(5):
                got.append(th.autograd.grad(out, _tensors(leaves), grad, retain_graph=True))
        except Exception as e:   # reported by the main thread
            errors.append(e)
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    th.cuda.synchronize()
    assert not errors and len(got) == 20
    assert all(th.equal(a, b) for grads in got for a, b in zip(grads, want))


@pytest.mark.parametrize("name", ["MaskedMMCSR", "VectorSPMM", "GraphAttentionBias"])
def test_index_types_of_the_two_orientations_agree(tables, name):
    function, tabs, given = _call(name, tables)
    leaves, half = _leaves(given), len(tabs) - 4
    out = function.apply(*tabs[:half], *[t.int() for t in tabs[half:]], *leaves)
    with pytest.raises(RuntimeError, match="expected all index tensors to share dtype torch.int64, got torch.int32"):
        out.sum().backward()


@pytest.mark.parametrize("name", FUNCTIONS)
def test_nothing_but_the_tensors_of_the_call_is_held(tables, name):
    """Between the directions: the output (and the attention's log-sum, 4 bytes per node and head). After the backward: the
    output alone, and not the call's own index tensors."""
    function, tabs, given = _call(name, tables)
    leaves = _leaves(given)

    def asked():   # what was asked for: blocks handed out may be larger
        return th.cuda.memory_stats()["requested_bytes.all.current"]
    before = asked()
    own = [t.clone() for t in tabs]
    indices = asked() - before
    out = function.apply(*own, *leaves)
    lse = N * H * 4 if name == "GraphAttentionBias" else 0
    assert asked() - before == indices + out.numel() * 4 + lse
    del own
    ones = th.ones_like(out)
    grads = th.autograd.grad(out, _tensors(leaves), ones)
    assert asked() - before == sum(t.numel() * 4 for t in (out, ones, *grads))
    del ones, grads, out
    assert asked() == before


@pytest.mark.parametrize("name", FUNCTIONS)
def test_saved_tensor_hooks_see_all_that_is_saved(tables, name):
    """Offloading: what the hooks move to the host leaves the device, and the backward runs on what they bring back."""
    function, tabs, given = _call(name, tables)
    leaves = _leaves(given)
    want = function.apply(*tabs, *leaves)
    grad = _normal(*want.shape, seed=9)
    want_grads = th.autograd.grad(want, _tensors(leaves), grad)
    packed = []

    def pack(t):
        packed.append(t.data_ptr())
        return t.cpu()
    with th.autograd.graph.saved_tensors_hooks(pack, lambda t: t.to(DEV)):
        out = function.apply(*[t.clone() for t in tabs], *leaves)
    extra = {"SparseSoftmax": 0, "GraphAttentionBias": 2}.get(name, 0)   # the softmax saves its output for its input
    assert len(packed) == len(tabs) + len(_tensors(given)) + extra
    th.empty(1 << 20, device=DEV).fill_(7)   # over what the clones held
    assert all(th.equal(a, b) for a, b in zip(th.autograd.grad(out, _tensors(leaves), grad), want_grads))


def test_index_tensors_are_checked_and_may_come_from_inference_mode(tables):
    function, tabs, given = _call("MaskedMMCSR", tables)
    with th.inference_mode():
        tabs = [t.clone() for t in tabs]
    leaves = _leaves(given)
    out = function.apply(*tabs, *leaves)
    th.autograd.grad(out, _tensors(leaves), th.ones_like(out))
    tabs = [t.clone() for t in tabs]
    out = function.apply(*tabs, *leaves)
    tabs[5].add_(0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


@pytest.mark.parametrize("name", ["MaskedMMCSR", "VectorSPMM", "GraphAttentionBias"])
def test_inference_without_the_column_side(tables, name):
    """Only the backward reads the column CSR: a call without a gradient may leave it out, a backward says what is missing."""
    function, tabs, given = _call(name, tables)
    half = len(tabs) - 4
    with th.no_grad():
        assert th.equal(function.apply(*tabs[:half], None, None, None, None, *given), function.apply(*tabs, *given))
    out = function.apply(*tabs[:half], None, None, None, None, *_leaves(given))
    with pytest.raises(RuntimeError, match="col must be a CUDA tensor"):
        out.sum().backward()


@pytest.mark.parametrize("name", FUNCTIONS)
def test_nodes_have_the_names_of_their_functions(tables, name):
    function, tabs, given = _call(name, tables)
    leaves = _leaves(given)
    with th.autograd.set_detect_anomaly(True):   # which reports nodes by these names
        out = function.apply(*tabs, *leaves)
        assert out.grad_fn.name() == name + "Backward"
        th.autograd.grad(out, _tensors(leaves), th.ones_like(out))


@pytest.mark.parametrize("name", FUNCTIONS)
@pytest.mark.parametrize("start", [0, 3])
def test_chunk_tables_without_chunks(name, start):
    """No chunk, seven edges: outputs and gradients are zero, whatever position the table stops at."""
    empty, stop = th.zeros(0, dtype=th.int64, device=DEV), th.full((1,), start, dtype=th.int64, device=DEV)
    ids = th.arange(7, device=DEV) % 5
    table = [empty, stop, th.arange(7, device=DEV), ids]
    node, edge, rel = _normal(5, H, D, seed=1), _normal(7, H, seed=2), _normal(7, D, seed=3)
    tabs, given = {"SparseSoftmax": (table[:3], [edge]), "MaskedMMCSR": (table * 2, [node, node]),
                   "NodeMulEdge": (table[:3], [node, rel]), "VectorSPMM": (table * 2, [edge, node]),
                   "GraphAttentionBias": ([empty, stop, ids, *table], [node, node, node, rel, 0.25])}[name]
    leaves = _leaves(given)
    out = getattr(wrapper, name).apply(*tabs, *leaves)
    assert not out.any()
    assert not any(g.any() for g in th.autograd.grad(out, _tensors(leaves), th.ones_like(out)))
