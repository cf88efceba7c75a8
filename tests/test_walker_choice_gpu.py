"""Which walker sums gathered rows on tables beyond the L2: the question how often the samples repeat, against what chance gives for
that many rows, and the lines by the size of the table and of a block of heads' share of it.  The two walkers add a row's edges
up in different groupings, so the bits of a sum tell which one ran."""
import pytest
import torch as th

from custom_op_benchmark_b200 import graphop, graphs
from custom_op_benchmark_b200.part_csr import partition_csr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _graph(n, e, seed, hub=False):
    gen = th.Generator(device=DEV).manual_seed(seed)
    dst, src = (th.randint(0, n, (e,), generator=gen, device=DEV) for _ in range(2))
    if hub:
        src[::8] = n // 3
    g = graphs.coo_to_graph(dst, src, n, index_dtype=th.int32)
    row, ptr = partition_csr(g.indptr, 32)
    return g, [row.int(), ptr.int(), g.eid, g.indices]


def _sums(plan, w, x, repeats):
    """The sums under a plan that has found so many repeats among its samples."""
    found, plan.c.gather_repeats = plan.c.gather_repeats, repeats
    try:
        return graphop.vector_spmm_forward_planned(plan, w, x)
    finally:
        plan.c.gather_repeats = found


# 156 MB in rows of 8 KB: 1024 of uniform edges name one of the 20 thousand rows again about 25 times
def test_repeats_by_chance_are_no_skew():
    n, h, d = 20_000, 16, 128
    x = th.randn(n, h, d, device=DEV)
    for seed, hub in [(s, False) for s in range(12)] + [(0, True)]:
        g, tables = _graph(n, 200_000, seed, hub)
        plan = graphop.GraphPlan(*tables, n)
        w = th.rand(g.n_edges, h, device=DEV)
        y, few, many = (_sums(plan, w, x, r) for r in (plan.c.gather_repeats, 0, 1024))
        assert not th.equal(few, many)
        assert th.equal(y, many if hub else few), (seed, plan.c.gather_repeats)
        assert th.equal(graphop.vector_spmm_forward(*tables, w, x), y)


# a block of heads is 512 bytes of every row
@pytest.mark.parametrize("n,h,d,asked", [(32_000, 8, 128, False),      # 125 MiB, blocks of 16
                                         (62_000, 8, 64, False),       # 121, blocks of 30
                                         (70_000, 2, 128, True),       # 68, blocks of 34
                                         (14_000, 32, 128, False),     # 219, blocks of 7: so few rows
                                         (18_000, 8, 256, True)])      # 141, blocks of 9
def test_lines(n, h, d, asked):
    g, tables = _graph(n, 12 * n, 3)
    plan = graphop.GraphPlan(*tables, n)
    w, x = th.rand(g.n_edges, h, device=DEV), th.randn(n, h, d, device=DEV)
    few, many = _sums(plan, w, x, 0), _sums(plan, w, x, 1024)
    assert th.equal(few, many) != asked
    assert th.equal(graphop.vector_spmm_forward(*tables, w, x), _sums(plan, w, x, plan.c.gather_repeats))
    some = th.arange(0, n, 97, device=DEV)
    dst = th.repeat_interleave(th.arange(n, device=DEV), (g.indptr[1:] - g.indptr[:-1]).long())
    want = th.zeros(n, dtype=th.bool, device=DEV).index_fill_(0, some, True)[dst].nonzero()[:, 0]
    ref = th.zeros(len(some), h, d, dtype=th.float64, device=DEV)
    at = th.searchsorted(some, dst[want])
    ref.index_add_(0, at, w[want].double().unsqueeze(-1) * x[g.indices[want].long()].double())
    for y in (few, many):   # at most some dozens of terms of size 1
        assert float((y[some].double() - ref).abs().max()) <= 3e-6 * max(1.0, float(ref.abs().max()))
