"""The kernels' tiles at their edges: rows one short of, as long as and one longer than a work tile, a softmax tile and an
expansion step, a row over many of them, empty rows between; head sizes and counts of every kind (each geometry the walker
is compiled for: test_geometries_gpu.py).  Against the float64 oracle."""
import threading

import pytest
import torch as th

from helpers import assert_close, chunked, random_graph
from custom_op_benchmark_b200 import graphop, graphs, wrapper
from oracle import edge_list_f64 as ref
from oracle import graphop_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DEGREES = [0, 1, 31, 32, 33, 0, 0, 255, 256, 257, 3, 1023, 1024, 1025, 0, 9000, 1, 7, 0, 2047, 2048, 2049, 40, 0, 0]
TOL = {th.float32: 3e-5, th.float64: 1e-12, th.bfloat16: 2e-2}


@pytest.fixture(scope="module")
def graph():
    return random_graph(len(DEGREES), len(DEGREES), DEGREES, 17)


def _inputs(graph, cs, idt):
    return chunked(graph, cs, dtype=idt), chunked(graph, cs, transposed=True, dtype=idt)


def _draw(dtype, *shape, seed=0):
    g = th.Generator().manual_seed(seed + sum(shape))
    return th.randn(*shape, generator=g, dtype=th.float64).to(dtype)


def _check(function, oracle, tables, given, grad):
    """function.apply(*tables, *given) and its gradients against oracle(*float64 copies) -> (output, gradients)."""
    dev = [t.to(DEV).requires_grad_(True) for t in given]
    out = function.apply(*[t.to(DEV) for t in tables], *dev)
    grads = th.autograd.grad(out, dev, grad.to(DEV))
    want, want_grads = oracle([t.double() for t in given], grad.double())
    tol = TOL[given[0].dtype]
    for name, a, b in [("output", out, want)] + [("gradient %d" % i, a, b) for i, (a, b) in enumerate(zip(grads, want_grads))]:
        assert_close(a, b, tol, tol * max(1.0, float(b.abs().max())), name)


# rows of one, two and several slots per lane; heads that share a block, that fill none, that are cut into pieces
@pytest.mark.parametrize("dtype,h,d", [(th.float32, 3, 20), (th.float32, 1, 25), (th.float32, 16, 8), (th.float32, 9, 16),
                                       (th.float32, 2, 256), (th.float64, 6, 20), (th.float64, 2, 32),
                                       (th.bfloat16, 4, 64), (th.bfloat16, 3, 25), (th.bfloat16, 5, 12)])
@pytest.mark.parametrize("cs,idt", [(32, th.int64), (None, th.int32)])
def test_gathering_ops(graph, dtype, h, d, cs, idt):
    r, c = _inputs(graph, cs, idt)
    n, e = graph.n_dst, graph.n_edges
    A, B = _draw(dtype, n, h, d), _draw(dtype, n, h, d, seed=1)
    es = (e,) if h == 1 else (e, h)
    _check(wrapper.MaskedMMCSR, lambda x, g: (orc.maskedmm_csr_forward(*r, *x).view(es),
                                              orc.maskedmm_csr_backward(*r, *c, *x, g)), [*r, *c], [A, B], _draw(dtype, *es))
    w = _draw(dtype, *es, seed=2)
    _check(wrapper.VectorSPMM, lambda x, g: (orc.vector_spmm_forward(*r, *x),
                                             orc.vector_spmm_backward(*r, *c, x[0], g, x[1])), [*r, *c], [w, A],
           _draw(dtype, n, h, d, seed=3))


@pytest.mark.parametrize("dtype,h,d", [(th.float32, 2, 16), (th.float32, 4, 32), (th.float32, 8, 64), (th.float32, 1, 32),
                                       (th.float32, 4, 8), (th.float32, 3, 32), (th.float32, 2, 20), (th.float32, 4, 256),
                                       (th.float64, 4, 8), (th.float64, 8, 16), (th.bfloat16, 2, 64), (th.bfloat16, 8, 32),
                                       (th.bfloat16, 5, 25)])
def test_edge_feature_op(graph, dtype, h, d):
    r, _ = _inputs(graph, 32, th.int64)
    e = graph.n_edges
    es = (e,) if h == 1 else (e, h)
    _check(wrapper.NodeMulEdge, lambda x, g: (orc.node_mul_edge_forward(*r[:3], *x).view(es),
                                              orc.node_mul_edge_backward(*r[:3], *x, g)), r[:3],
           [_draw(dtype, graph.n_dst, h, d), _draw(dtype, e, d)], _draw(dtype, *es))


@pytest.mark.parametrize("dtype", [th.float32, th.float64, th.bfloat16])
@pytest.mark.parametrize("h", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("repeat", [1, 60])   # 60: more tiles than merge their rows' statistics for themselves
def test_softmax(graph, dtype, h, repeat):
    if repeat > 1:
        if h not in (2, 3) or dtype != th.float32:
            pytest.skip("one type is enough for the second merge")
        graph = random_graph(len(DEGREES) * repeat, 10, DEGREES * (repeat - 1) + [60000] * len(DEGREES), 18)
    r, _ = _inputs(graph, 32, th.int64)
    es = (graph.n_edges,) if h == 1 else (graph.n_edges, h)

    def oracle(x, g):
        y = orc.sparse_softmax_forward(*r[:3], *x)
        return y, [orc.sparse_softmax_backward(*r[:3], y, g)]
    _check(wrapper.SparseSoftmax, oracle, r[:3], [_draw(dtype, *es) * 3], _draw(dtype, *es, seed=4))


@pytest.mark.parametrize("idt", [th.int32, th.int64])
@pytest.mark.parametrize("lo,hi", [(0, 0), (5, 0), (0, 9), (40, 700)])
def test_chunk_tables_that_cover_a_part(graph, idt, lo, hi):
    """Positions before the first and after the last chunk belong to no node: their edge outputs are zero."""
    row, ptr, eid, idx = chunked(graph, 32, dtype=idt)
    keep = (ptr[:-1] >= lo) & (ptr[1:] <= graph.n_edges - hi)
    a, b = int(keep.nonzero()[0]), int(keep.nonzero()[-1])
    row, ptr = row[a:b + 1].contiguous(), ptr[a:b + 2].contiguous()
    x = _draw(th.float32, graph.n_edges, 4)
    A = _draw(th.float32, graph.n_dst, 4, 32)
    r = [t.to(DEV) for t in (row, ptr, eid, idx)]
    got = wrapper.MaskedMMCSR.apply(*r, *r, A.to(DEV), A.to(DEV))
    assert_close(got, orc.maskedmm_csr_forward(row, ptr, eid, idx, A.double(), A.double()), 3e-5, 3e-4)
    got = wrapper.SparseSoftmax.apply(*r[:3], x.to(DEV))
    assert_close(got, orc.sparse_softmax_forward(row, ptr, eid, x.double()), 3e-5, 3e-5)
    got = wrapper.VectorSPMM.apply(*r, *r, x.to(DEV), A.to(DEV))
    assert_close(got, orc.vector_spmm_forward(row, ptr, eid, idx, x.double(), A.double()), 3e-5, 3e-3)
    plan = graphop.GraphPlan(*r, graph.n_dst)
    assert_close(graphop.vector_spmm_forward_planned(plan, x.to(DEV), A.to(DEV)), got.cpu(), 3e-5, 3e-3)


def test_functions_from_several_threads(graph):
    r, c = _inputs(graph, 32, th.int64)
    tables = [t.to(DEV) for t in (*r, *c)]
    A = _draw(th.float32, graph.n_dst, 4, 32).to(DEV)
    want = wrapper.MaskedMMCSR.apply(*tables, A, A)
    got, errors = [None] * 4, []

    def work(k):
        try:
            with th.cuda.stream(th.cuda.Stream()):
                for _ in range(5):
                    x = A.clone().requires_grad_(True)
                    y = wrapper.MaskedMMCSR.apply(*tables, x, x)
                    y.sum().backward()
                th.cuda.current_stream().synchronize()
            got[k] = y.detach()
        except Exception as e:   # reported by the main thread
            errors.append(e)
    th.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert all(th.equal(y, want) for y in got)


# one block of the band's 64 keys to six of them, tiles that end inside a sequence; scores that grow along the band, so that
# the forward's running maximum has to move its reference (and ones that fall, and a scale that turns them round)
@pytest.mark.parametrize("length,window,ramp,scale", [(1, 0, 0, 0.125), (63, 5, 0, 0.125), (128, 31, 0, 0.125),
                                                      (129, 32, 30, 0.5), (500, 64, 60, 0.5), (700, 128, 100, 1.0),
                                                      (700, 128, -100, 1.0), (300, 100, 0, -0.125), (300, 100, 0, 0.0)])
def test_dense_band(length, window, ramp, scale):
    g = graphs.banded_graph(2, length, window)
    n, h, d = g.n_dst, 3, 64
    rc, cc = [t.to(DEV) for t in chunked(g, 32)], [t.to(DEV) for t in chunked(g, 32, transposed=True)]
    plans = graphop.GraphPlan(*rc, n), graphop.GraphPlan(*cc, n)
    assert plans[0].dense_band and plans[1].dense_band
    Q, K, V, dO = (_draw(th.float32, n, h, d, seed=k).to(DEV) for k in range(4))
    at = th.linspace(0, 1, n, device=DEV).view(-1, 1, 1)
    K = 0.3 * K + ramp * (at if ramp >= 0 else 1 - at) * Q.mean(0, keepdim=True).sign() / d
    Q = 0.3 * Q + (1.0 if ramp else 0.0) * Q.mean(0, keepdim=True).sign()
    Q, K, V, dO = (t.to(th.bfloat16) for t in (Q, K, V, dO))
    leaves = [t.clone().requires_grad_(True) for t in (Q, K, V)]
    o = wrapper.GraphAttentionPlanned.apply(*plans, *leaves, scale)
    got = [o, *th.autograd.grad(o, leaves, dO)]
    want = ref.attention_f64(g.indptr.to(DEV), g.indices.to(DEV), Q, K, V, scale, dO)
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, (want[0], *want[2:])):
        assert_close(a, b, 3e-2, 3e-2 * max(1.0, float(b.abs().max())), name)
    _, lse = graphop.attention_forward_planned(plans[0], Q, K, V, scale)
    assert_close(lse, want[1], 2e-3, 2e-3, "lse")
