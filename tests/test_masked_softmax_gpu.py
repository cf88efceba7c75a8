"""Scores of minus infinity (masked edges) in the row softmax: runs of them that fill a row's part of a softmax tile (1024
positions), whichever way the row's parts are merged.  Against the float64 oracle, which knows no tiles."""
import pytest
import torch as th

from helpers import chunked, random_graph
from custom_op_benchmark_b200 import graphop, wrapper
from oracle import edge_list_f64 as ref
from oracle import graphop_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF = float("inf")


# (degrees, masked runs of positions): a two-edge row over a boundary with either edge masked; rows over several tiles with
# their first part, a whole tile of theirs, or their last part masked; the same where a second launch merges (more than 1024
# tiles) and for a row of more tiles than one warp merges
CASES = {
    "two_edges": ([1023, 2, 1022, 2, 900], [(1023, 1024), (2048, 2049)]),
    "parts": ([1000, 3000, 100, 5000, 30], [(1000, 1024), (1024, 2048), (4096, 4100), (5120, 7168), (9000, 9100)]),
    "merged": ([700] * 1600 + [300000, 2100], [(700, 1024), (1048576, 1048800), (1120000, 1120256), (1200128, 1210368),
                                               (1300000, 1419999), (1421312, 1422100)]),
}


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("h,dtype", [(1, th.float32), (3, th.float32), (4, th.float64), (2, th.bfloat16)])
def test_masked_runs(case, h, dtype):
    degrees, runs = CASES[case]
    g = random_graph(len(degrees), 50, degrees, 3)
    r = chunked(g, 32)
    gen = th.Generator().manual_seed(5)
    x = th.randn(g.n_edges, h, generator=gen, dtype=th.float64)
    for a, b in runs:
        x[r[2][a:b]] = -INF
    x[r[2][5], 0] = -INF
    x = x.squeeze(1) if h == 1 else x
    x = x.to(dtype)
    dy = th.randn(x.shape, generator=gen, dtype=th.float64).to(dtype)
    want = orc.sparse_softmax_forward(*r[:3], x.double())
    assert bool(th.isfinite(want).all())   # no row is masked as a whole
    leaf = x.to(DEV).requires_grad_(True)
    tabs = [t.to(DEV) for t in r[:3]]
    y = wrapper.SparseSoftmax.apply(*tabs, leaf)
    (dx,) = th.autograd.grad(y, leaf, dy.to(DEV))
    want_dx = orc.sparse_softmax_backward(*r[:3], want, dy.double())
    tol = {th.float32: 2e-5, th.float64: 1e-12, th.bfloat16: 2e-2}[dtype]
    for got, exp in ((y, want), (dx, want_dx)):
        err = (got.detach().double().cpu() - exp).abs()
        # relative to the row's largest value: a probability or gradient of 1 / degree is what a long row has
        assert bool((err <= tol * (exp.abs() + 1.0 / 700)).all()), float(err.max())


@pytest.mark.parametrize("what", ["row", "nan"])
def test_what_has_no_value_stays_nan(what):
    """A row masked as a whole, and a NaN among masked edges, give NaN in the whole row and nowhere else."""
    degrees = [1000, 3000, 500]
    g = random_graph(3, 50, degrees, 4)
    r = chunked(g, 32)
    x = th.randn(g.n_edges, 2, generator=th.Generator().manual_seed(6))
    owner = orc.expand_rows(r[0], r[1], g.n_edges)
    middle = r[2][owner == 1]
    if what == "row":
        x[middle] = -INF
    else:
        x[r[2][1024:2048]] = -INF
        x[r[2][1500]] = float("nan")
    y = wrapper.SparseSoftmax.apply(*[t.to(DEV) for t in r[:3]], x.to(DEV)).cpu()
    bad = th.zeros(g.n_edges, dtype=th.bool)
    bad[middle] = True
    assert bool(th.isnan(y[bad]).all()) and bool(th.isfinite(y[~bad]).all())


@pytest.mark.parametrize("h,d,dtype", [(4, 32, th.float32), (8, 64, th.float32), (1, 16, th.float32), (2, 64, th.bfloat16)])
def test_scores_that_overflow_in_the_fused_layer(h, d, dtype):
    """Finite queries and keys whose product is -inf in float: such an edge has probability 0, also where a node's first
    edges are all of that kind (half of the sources are, in runs of any length)."""
    g = random_graph(300, 200, [40] * 299 + [3000], 11)
    gen = th.Generator().manual_seed(12)
    q, k, v, do = (th.randn(n, h, d, generator=gen) for n in (300, 200, 200, 300))
    q[..., 0], k[..., 0] = 1e20, 0.0
    k[::2, :, 0] = -1e20
    q, k, v, do = (t.to(dtype).to(DEV) for t in (q, k, v, do))
    r, c = [t.to(DEV) for t in chunked(g, 32)], [t.to(DEV) for t in chunked(g, 32, transposed=True)]
    plans = graphop.GraphPlan(*r, 300), graphop.GraphPlan(*c, 200)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    scale = d ** -0.5
    o = wrapper.GraphAttentionPlanned.apply(*plans, *leaves, scale)
    got = [o, *th.autograd.grad(o, leaves, do)]
    want = ref.attention_f64(g.indptr.to(DEV), g.indices.to(DEV), q, k, v, scale, do)
    tol = 3e-5 if dtype == th.float32 else 2e-2
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, (want[0], *want[2:])):
        assert bool(th.isfinite(a).all()), name
        a, b = a.double()[..., 1:], b[..., 1:]   # feature 0 of dk is a sum of terms of 1e20 that cancel
        assert bool(((a - b).abs() <= tol * (b.abs() + max(1.0, float(b.abs().max())))).all()), name
