"""The streaming edge kernels (row softmax, node-edge products with all heads in a thread) with edge ids at every alignment of
their table and every remainder of its length: ids that are the positions, ids in another order."""
import pytest
import torch as th

from helpers import assert_close, chunked, random_graph
from custom_op_benchmark_b200 import graphop
from oracle import graphop_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("extra", [0, 1, 2, 3])
@pytest.mark.parametrize("shuffled", [False, True])
def test_softmax(offset, extra, shuffled):
    g = random_graph(6, 6, [5, 0, 1500, 2, 37, 1024 - 44 + extra], 5)
    row, ptr, eid, _ = chunked(g, 32, dtype=th.int32)
    e, gen = g.n_edges, th.Generator().manual_seed(offset + 4 * extra)
    if shuffled:
        eid = th.randperm(e, generator=gen).int()
    x, dy = (th.randn(e, 2, generator=gen) for _ in range(2))
    ids = th.empty(e + offset, dtype=th.int32, device=DEV)[offset:]   # a view at 4 * offset bytes
    ids.copy_(eid)
    tables = [row.to(DEV), ptr.to(DEV), ids]
    y = graphop.sparse_softmax_forward(*tables, x.to(DEV))
    dx = graphop.sparse_softmax_backward(*tables, y, dy.to(DEV))
    want = orc.sparse_softmax_forward(row, ptr, eid, x.double())
    assert_close(y, want, 1e-5, 1e-6, "y")   # sums of 1500 exponentials in float
    assert_close(dx, orc.sparse_softmax_backward(row, ptr, eid, want, dy.double()), 1e-5, 1e-5, "dx")


@pytest.mark.parametrize("dtype,h,d", [(th.float32, 4, 32), (th.float32, 3, 20), (th.bfloat16, 8, 64)])
@pytest.mark.parametrize("offset,extra", [(0, 0), (1, 3), (2, 6), (3, 1), (0, 7)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_node_mul_edge(dtype, h, d, offset, extra, shuffled):
    g = random_graph(6, 6, [5, 0, 150, 2, 37, 30 + extra], 5)
    row, ptr, eid, _ = chunked(g, 32, dtype=th.int32)
    e, gen = g.n_edges, th.Generator().manual_seed(offset + 4 * extra)
    if shuffled:
        eid = th.randperm(e, generator=gen).int()
    a, b, dy = (th.randn(*shape, generator=gen).to(dtype) for shape in ((6, h, d), (e, d), (e, h)))
    ids = th.empty(e + offset, dtype=th.int32, device=DEV)[offset:]
    ids.copy_(eid)
    tables = [row.to(DEV), ptr.to(DEV), ids]
    y = graphop.node_mul_edge_forward(*tables, a.to(DEV), b.to(DEV))
    da, db = graphop.node_mul_edge_backward(*tables, a.to(DEV), b.to(DEV), dy.to(DEV))
    tol = 1e-5 if dtype == th.float32 else 2e-2   # sums of up to 187 products of size 1
    a, b, dy = a.double(), b.double(), dy.double()
    assert_close(y, orc.node_mul_edge_forward(row, ptr, eid, a, b), tol, tol * 10, "y")
    for name, got, want in zip(("dA", "dB"), (da, db), orc.node_mul_edge_backward(row, ptr, eid, a, b, dy)):
        assert_close(got, want, tol, tol * 10, name)
