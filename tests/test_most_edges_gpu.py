"""The most edges the entry points admit, 2^31 - 1: positions at the very top of 32-bit range, where a step, tile or block
that starts below the end reaches past 2^31.  Rows of 140 million edges and, over the last positions, many short ones."""
import pytest
import torch as th

from custom_op_benchmark_b200 import graphop

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
E, BIG, SMALL, D = 2 ** 31 - 1, 15, 700, 8


@pytest.fixture(scope="module")
def graph():
    if th.cuda.get_device_properties(0).total_memory < 120e9:
        pytest.skip("needs about 50 GB")
    small = th.randint(0, 20, (SMALL,), generator=th.Generator().manual_seed(1))
    small[-1] = 1   # the last position is a row of its own
    top = E - int(small.sum())
    big = th.full((BIG,), top // BIG)
    big[-1] += top - int(big.sum())
    deg = th.cat([big, small])
    ptr = th.cat([th.zeros(1, dtype=th.int64), deg.cumsum(0)])
    assert int(ptr[-1]) == E
    row = th.arange(BIG + SMALL, dtype=th.int32, device=DEV)   # one chunk per row, empty ones included
    return row, ptr.to(DEV, th.int32), deg, top


def _tail(top):
    return th.arange(top, E, dtype=th.int64, device=DEV)


def test_softmax(graph):
    row, ptr, deg, top = graph
    eid = th.arange(E, dtype=th.int32, device=DEV)
    x = th.zeros(E, dtype=th.bfloat16, device=DEV)
    x[top:] = th.randn(E - top, generator=th.Generator().manual_seed(2)).to(DEV, th.bfloat16)
    y = graphop.sparse_softmax_forward(row, ptr, eid, x)
    owner = th.repeat_interleave(th.arange(SMALL, device=DEV), deg[BIG:].to(DEV))
    ex = x[top:].double().exp()
    want = ex / th.zeros(SMALL, dtype=th.float64, device=DEV).index_add_(0, owner, ex)[owner]
    assert bool(((y[top:].double() - want).abs() <= 2 ** -8 * want).all())   # one bfloat16 rounding
    for at in (0, top // 2, top - 1):
        assert abs(float(y[at]) * int(deg[0]) - 1) <= 2 ** -7


@pytest.mark.parametrize("planned", [False, True])
def test_aggregation(graph, planned):
    row, ptr, deg, top = graph
    src = th.zeros(E, dtype=th.int32, device=DEV)
    src[top:] = (_tail(top) % 4).int()
    w = th.full((E,), 2.0 ** -20, dtype=th.bfloat16, device=DEV)
    w[top:] = th.rand(E - top, generator=th.Generator().manual_seed(3)).to(DEV, th.bfloat16)
    x = (1.0 + th.arange(4 * D, device=DEV).view(4, 1, D) / 64).to(th.bfloat16)
    n = BIG + SMALL
    if planned:
        plan = graphop.GraphPlan(row, ptr, None, src, n)
        assert not plan.dense_band and not plan.no_carry
        y = graphop.vector_spmm_forward_planned(plan, w, x, num_dst=n)
    else:
        eid = th.arange(E, dtype=th.int32, device=DEV)
        y = graphop.vector_spmm_forward(row, ptr, eid, src, w, x, num_dst=n)
    owner = th.repeat_interleave(th.arange(SMALL, device=DEV), deg[BIG:].to(DEV))
    terms = w[top:].double().view(-1, 1) * x.double().view(4, D)[src[top:].long()]
    want = th.zeros(SMALL, D, dtype=th.float64, device=DEV).index_add_(0, owner, terms)
    assert bool(((y[BIG:, 0].double() - want).abs() <= 2 ** -8 * want).all())   # one bfloat16 rounding
    big = deg[:BIG].to(DEV).double().view(-1, 1) * 2.0 ** -20 * x.double().view(4, D)[0]
    assert bool(((y[:BIG, 0].double() - big).abs() <= 2 ** -7 * big).all())
