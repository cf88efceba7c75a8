"""Wide rows on many work tiles: a lane group then walks several of the graph's tiles as one.  Rows within a tile, rows that
cross the boundaries between the tiles of one walk, rows over several walks, empty rows; the last walk has fewer tiles than
the others.  Against float64 on the same inputs."""
import pytest
import torch as th

from helpers import random_graph
from custom_op_benchmark_b200 import graphop, wrapper
from custom_op_benchmark_b200.part_csr import partition_csr
from oracle import edge_list_f64 as ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# relative to the largest entry; sums of up to 3000 products of size 1 and their square roots' worth of rounding
TOL = {th.float32: 3e-5, th.bfloat16: 2e-2}


def _graph(nodes, most):
    gen = th.Generator().manual_seed(5)
    deg = th.randint(0, most, (nodes,), generator=gen)
    deg[th.rand(deg.numel(), generator=gen) < 0.2] = 0
    deg[[7, 3 * nodes // 10, 3 * nodes // 10 + 1, nodes - 1_000]] = th.tensor([3_000, 40, 700, 131])
    g = random_graph(deg.numel(), deg.numel(), deg, 6)
    row, ptr = partition_csr(g.indptr, 32)
    col, ptr_t = partition_csr(g.indptr_t, 32)
    tables = [[t.int().to(DEV) for t in o] for o in ((row, ptr, g.eid, g.indices), (col, ptr_t, g.eid_t, g.indices_t))]
    return g, tables


@pytest.fixture(scope="module")
def graph():
    return _graph(30_000, 12)


@pytest.fixture(scope="module")
def long_rows():
    return _graph(5_003, 240)


def _draw(dtype, *shape, seed=0):
    gen = th.Generator(device=DEV).manual_seed(seed)
    return th.randn(*shape, generator=gen, device=DEV).to(dtype).requires_grad_(True)


def _close(got, want, tol, what):
    err = float((got.detach().double() - want).abs().max())
    assert err <= tol * max(1.0, float(want.abs().max())), (what, err)


# 8 head blocks of 512 bytes or 16 of 256, K and V beyond the L2: two tiles per walk, for the forward and the destination side
@pytest.mark.parametrize("dtype,h,d", [(th.float32, 8, 128), (th.bfloat16, 16, 128)])
@pytest.mark.parametrize("planned", [False, True])
def test_attention(graph, dtype, h, d, planned):
    _attention(graph, dtype, h, d, planned)


# K and V of 41 MB together, 15697 tiles: walks of any length, of three tiles in 4-byte elements and of six in bfloat16
@pytest.mark.parametrize("dtype,h,d", [(th.float32, 8, 128), (th.bfloat16, 16, 128)])
@pytest.mark.parametrize("planned", [False, True])
def test_attention_in_long_walks(long_rows, dtype, h, d, planned):
    g = long_rows[0]
    assert ((g.n_edges + 4 * g.n_dst) // 32 + 1) % 3 != 0   # the last walk is shorter in both
    _attention(long_rows, dtype, h, d, planned)


def _attention(graph, dtype, h, d, planned):
    g, (r, c) = graph
    q, k, v = (_draw(dtype, g.n_dst, h, d, seed=i) for i in range(3))
    grad = _draw(dtype, g.n_dst, h, d, seed=3).detach()
    if planned:
        out = wrapper.GraphAttentionPlanned.apply(graphop.GraphPlan(*r, g.n_dst), graphop.GraphPlan(*c, g.n_src), q, k, v, d ** -0.5)
    else:
        out = wrapper.GraphAttention.apply(r[0], r[1], r[3], c[0], c[1], c[3], q, k, v, d ** -0.5, c[2])
    got = [out] + list(th.autograd.grad(out, (q, k, v), grad))
    want = ref.attention_f64(g.indptr.to(DEV), g.indices.to(DEV), q.detach(), k.detach(), v.detach(), d ** -0.5, grad, chunk=1 << 15)
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, [want[0]] + list(want[2:])):
        _close(a, b, TOL[dtype], name)


# one head in 64 or 128 pieces: ten tiles per walk of the 4-byte sums, two in bfloat16
@pytest.mark.parametrize("dtype,d", [(th.float32, 8192), (th.float32, 8188), (th.bfloat16, 16384)])
def test_aggregate_and_dot(graph, dtype, d):
    g, (r, c) = graph
    n, e = 2_000, int(g.indptr[2_000])   # the first rows, sources folded onto them
    row, ptr = partition_csr(g.indptr[:n + 1], 32)
    src = g.indices[:e] % n
    eid = th.arange(e)
    order = th.argsort(src, stable=True)
    ptr_t = th.zeros(n + 1, dtype=th.int64)
    ptr_t[1:] = th.cumsum(th.bincount(src, minlength=n), 0)
    dst = th.repeat_interleave(th.arange(n), g.indptr[1:n + 1] - g.indptr[:n])
    col, cptr = partition_csr(ptr_t, 32)
    tables = [t.int().to(DEV) for t in (row, ptr, eid, src, col, cptr, order, dst[order])]
    w, x = _draw(dtype, e, 1, seed=4), _draw(dtype, n, 1, d, seed=5)
    grad = _draw(dtype, n, 1, d, seed=6).detach()
    out = wrapper.VectorSPMM.apply(*tables, w, x)
    dw, dx = th.autograd.grad(out, (w, x), grad)
    adj = th.zeros(n, n, dtype=th.float64, device=DEV)
    adj.index_put_((dst.to(DEV), src.to(DEV)), w.detach().double()[:, 0], accumulate=True)
    xd, gd = x.detach().double()[:, 0], grad.double()[:, 0]
    _close(out[:, 0], adj @ xd, TOL[dtype], "y")
    _close(dx[:, 0], adj.t() @ gd, TOL[dtype], "dx")
    _close(dw.view(-1), (gd @ xd.t())[dst.to(DEV), src.to(DEV)], TOL[dtype], "dw")
