"""Row softmax with edge ids at every alignment of their table and every remainder of its length: ids that are the positions,
ids in another order."""
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
def test_ids_at_any_address(offset, extra, shuffled):
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
