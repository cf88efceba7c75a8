"""Every geometry that the gathering walker is compiled for (bytes per slot, lanes per edge, slots per lane, lanes per head
known at compile time or not, heads whole or in pieces), each at the smallest row that gets it: aggregation and edge dot
product through VectorSPMM, the fused layers through GraphAttentionPlanned and GraphAttentionBias.  Rows of the graph are
shorter than, as long as and longer than the smallest tile."""
import pytest
import torch as th

from helpers import assert_close, chunked, random_graph
from custom_op_benchmark_b200 import graphop, wrapper
from oracle import edge_list_f64 as ref
from oracle import graphop_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DEGREES = [0, 1, 31, 33, 0, 257, 3, 600, 2, 0]
TOL = {th.float32: 3e-5, th.float64: 1e-12, th.bfloat16: 2e-2}   # sums of at most 600 terms, as for the tile edges
N = len(DEGREES)

ROWS = {
    th.float32: [(1, 1), (1, 2), (1, 4), (1, 5), (1, 9), (1, 10), (3, 5), (1, 18), (1, 20), (3, 10), (1, 32), (2, 16), (1, 33),
                 (1, 36), (3, 20), (1, 64), (2, 32), (4, 16), (1, 66), (1, 128), (2, 64), (4, 32), (8, 16), (1, 132), (1, 65),
                 (1, 130), (1, 512), (1, 768)],
    th.bfloat16: [(1, 2), (1, 4), (1, 8), (1, 10), (1, 18), (1, 20), (1, 34), (1, 36), (1, 40), (1, 64), (2, 32), (1, 68),
                  (1, 72), (1, 128), (2, 64), (4, 32), (1, 136), (1, 66), (1, 130), (1, 132), (1, 512), (1, 260), (1, 768),
                  (1, 1200)],
    th.float64: [(1, 1), (1, 2), (1, 5), (1, 9), (1, 10), (3, 5), (1, 18), (3, 10), (1, 33), (1, 66), (1, 65), (1, 130),
                 (1, 258)],
}
ATTENTION_ROWS = {
    th.float32: [(1, 4), (5, 4), (1, 32), (2, 16), (5, 8), (1, 64), (2, 32), (4, 16), (5, 16), (1, 128), (2, 64), (4, 32),
                 (8, 16), (1, 256), (1, 512), (1, 1024)],
    th.bfloat16: [(1, 8), (5, 8), (1, 64), (2, 32), (5, 16), (1, 128), (2, 64), (4, 32), (1, 256), (1, 512), (1, 1024),
                  (1, 2048)],
    th.float64: [(1, 2), (5, 2), (5, 4), (5, 8), (1, 128), (1, 256), (1, 512)],
}


def _cases(rows):
    return [pytest.param(dt, h, d, id="%s-%dx%d" % (str(dt)[6:], h, d)) for dt, l in rows.items() for h, d in l]


@pytest.fixture(scope="module")
def graph():
    g = random_graph(N, N, DEGREES, 21)
    return g, chunked(g, 32), chunked(g, 32, transposed=True)


def _draw(dtype, *shape, seed):
    return th.randn(*shape, generator=th.Generator().manual_seed(seed), dtype=th.float64).to(dtype)


def _compare(dtype, got, want):
    for name, a, b in zip(("output", "gradient 0", "gradient 1", "gradient 2", "gradient 3"), got, want):
        assert_close(a, b, TOL[dtype], TOL[dtype] * max(1.0, float(b.abs().max())), name)


@pytest.mark.parametrize("dtype,h,d", _cases(ROWS))
def test_aggregation_and_dot(graph, dtype, h, d):
    g, r, c = graph
    w, x = _draw(dtype, *((g.n_edges,) if h == 1 else (g.n_edges, h)), seed=1), _draw(dtype, N, h, d, seed=2)
    dy = _draw(dtype, N, h, d, seed=3)
    leaves = [t.to(DEV).requires_grad_(True) for t in (w, x)]
    y = wrapper.VectorSPMM.apply(*[t.to(DEV) for t in (*r, *c)], *leaves)
    got = [y, *th.autograd.grad(y, leaves, dy.to(DEV))]
    _compare(dtype, got, [orc.vector_spmm_forward(*r, w, x), *orc.vector_spmm_backward(*r, *c, w, dy, x)])


@pytest.mark.parametrize("dtype,h,d", _cases(ATTENTION_ROWS))
@pytest.mark.parametrize("bias", [False, True])
def test_fused_layers(graph, dtype, h, d, bias):
    g, r, c = graph
    rc, cc = [t.to(DEV) for t in r], [t.to(DEV) for t in c]
    given = [_draw(dtype, N, h, d, seed=k).to(DEV) for k in range(3)]
    if bias:
        given.append(_draw(dtype, g.n_edges, d, seed=4).to(DEV))
    do, scale = _draw(dtype, N, h, d, seed=5).to(DEV), d ** -0.5
    leaves = [t.clone().requires_grad_(True) for t in given]
    if bias:
        o = wrapper.GraphAttentionBias.apply(rc[0], rc[1], rc[3], *cc, *leaves, scale)
    else:
        o = wrapper.GraphAttentionPlanned.apply(graphop.GraphPlan(*rc, N), graphop.GraphPlan(*cc, N), *leaves, scale)
    want = ref.attention_f64(g.indptr.to(DEV), g.indices.to(DEV), *given[:3], scale, do, rel=given[3] if bias else None)
    _compare(dtype, [o, *th.autograd.grad(o, leaves, do)], [want[0], *want[2:]])
