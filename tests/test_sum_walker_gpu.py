"""Sums of gathered rows on either side of the lines between the summing walker and the gathering one (the table's size, few
rows gathered by many edges), and the summing walker where its batches of four positions can go wrong: rows of 0 to 9 edges in every order, rows that end
with a batch and with a block of positions, positions that belong to no chunk, one round of warps and several.  Against
float64 on the same inputs."""
import pytest
import torch as th

from helpers import chunked, random_graph
from custom_op_benchmark_b200 import _capi, graphop, wrapper
from custom_op_benchmark_b200.part_csr import partition_csr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {th.float32: 3e-5, th.float64: 1e-12}   # of the largest entry; sums of at most a few hundred terms


def _draw(dtype, *shape, seed):
    gen = th.Generator(device=DEV).manual_seed(seed)
    return th.randn(*shape, generator=gen, device=DEV, dtype=dtype)


def _close(got, want, dtype, what):
    err = float((got.detach().double() - want).abs().max())
    assert err <= TOL[dtype] * max(1.0, float(want.abs().max())), (what, err)


def _sums(w, x, dst, src, n):
    """sum of w[e] * x[src[e]] per dst in float64, edge by edge."""
    out = th.zeros(n, *x.shape[1:], dtype=th.float64, device=DEV)
    return out.index_add_(0, dst, w.double().view(len(dst), -1, 1) * x[src].double())


# Tables beyond the L2 and beyond what the summing walker takes; edges on few nodes (skewed) and on many; a row of 32 slots of
# 16 bytes, one with lanes to spare, one of 8-byte elements.
@pytest.mark.parametrize("dtype,h,d", [(th.float32, 4, 32), (th.float32, 3, 20), (th.float64, 1, 64)])
@pytest.mark.parametrize("megabytes", [70, 1600])
@pytest.mark.parametrize("touched", [3_000, 100_000])
def test_large_tables(dtype, h, d, megabytes, touched):
    n, e = (megabytes << 20) // (h * d * th.empty((), dtype=dtype).element_size()), 40_000
    gen = th.Generator().manual_seed(3)
    used = th.sort(th.randperm(n, generator=gen)[:touched])[0]     # the nodes that have edges
    dst = used[th.randint(0, touched, (e,), generator=gen)]
    dst[:3_000] = used[7]                                          # a row over many tiles
    dst = th.sort(dst)[0]
    src = used[th.randint(0, touched, (e,), generator=gen)]
    src[-1] = n - 1
    order = th.argsort(src, stable=True)
    orientations = []
    for rows, others, eid in ((dst, src, th.arange(e)), (src[order], dst[order], order)):
        ptr = th.zeros(n + 1, dtype=th.int64)
        ptr[1:] = th.cumsum(th.bincount(rows, minlength=n), 0)
        row, chunks = partition_csr(ptr, 32)
        orientations.append([t.int().to(DEV) for t in (row, chunks, eid, others)])
    w, x = _draw(dtype, e, h, seed=1).requires_grad_(True), _draw(dtype, n, h, d, seed=2).requires_grad_(True)
    grad = _draw(dtype, n, h, d, seed=3)
    y = wrapper.VectorSPMM.apply(*orientations[0], *orientations[1], w, x)
    dw, dx = th.autograd.grad(y, (w, x), grad)
    plan = graphop.GraphPlan(*orientations[0], n)
    assert bool(plan.c.flags & _capi.PLAN_SKEWED) == (touched == 3_000)
    assert th.equal(graphop.vector_spmm_forward_planned(plan, w.detach(), x.detach()), y)   # the same bits
    dst, src = dst.to(DEV), src.to(DEV)
    for got, rows, cols, of, what in ((y, dst, src, x.detach(), "y"), (dx, src, dst, grad, "dx")):
        there, at = th.unique(rows, return_inverse=True)
        want = th.zeros(len(there), h, d, dtype=th.float64, device=DEV)
        want.index_add_(0, at, w.detach().double().view(-1, h, 1) * of[cols].double())
        _close(got[there], want, dtype, what)
        idle = th.ones(n, dtype=th.bool, device=DEV)
        idle[there] = False
        assert not got.detach()[idle].any(), what
    _close(dw.view(-1, h), (grad[dst].double() * x.detach()[src].double()).sum(-1), dtype, "dw")


@pytest.mark.parametrize("dtype,h,d", [(th.float32, 8, 64), (th.float32, 1, 32), (th.float32, 1, 4), (th.float64, 2, 16)])
@pytest.mark.parametrize("nodes", [40, 3_000, 60_000])
def test_short_rows(dtype, h, d, nodes):
    gen = th.Generator().manual_seed(nodes + d)
    deg = th.randint(0, 10, (nodes,), generator=gen)
    deg[::7] = th.tensor([4, 8, 32, 28, 0, 1, 36])[th.arange(len(deg[::7])) % 7]
    g = random_graph(nodes, nodes, deg, 9)
    r, c = chunked(g, 32, dtype=th.int32), chunked(g, 5, transposed=True, dtype=th.int32)
    tables = [t.to(DEV) for t in (*r, *c)]
    w, x = _draw(dtype, g.n_edges, h, seed=4).requires_grad_(True), _draw(dtype, nodes, h, d, seed=5).requires_grad_(True)
    grad = _draw(dtype, nodes, h, d, seed=6)
    y = wrapper.VectorSPMM.apply(*tables, w, x)
    dw, dx = th.autograd.grad(y, (w, x), grad)
    dst = th.repeat_interleave(th.arange(nodes), deg).to(DEV)
    src = g.indices.long().to(DEV)
    _close(y, _sums(w.detach(), x.detach(), dst, src, nodes), dtype, "y")
    _close(dx, _sums(w.detach(), grad, src, dst, nodes), dtype, "dx")


# the first and the last positions belong to no chunk: nothing of theirs may reach a node, not even an infinite row
@pytest.mark.parametrize("lead,tail", [(3, 0), (0, 5), (37, 70)])
def test_uncovered_positions(lead, tail):
    g = random_graph(50, 50, [5, 0, 9, 1, 40] * 10, 11)
    e = g.n_edges
    ptr = g.indptr + lead
    row, chunks = partition_csr(ptr, 32)
    src = th.cat([th.full((lead,), 49), g.indices % 49, th.full((tail,), 49)])
    eid = th.arange(lead + e + tail)
    x = _draw(th.float32, 50, 4, 32, seed=7)
    x[49] = float("inf")
    w = _draw(th.float32, lead + e + tail, 4, seed=8)
    tables = [t.int().to(DEV) for t in (row, chunks, eid, src)]
    y = graphop.vector_spmm_forward(*tables, w, x)
    dst = th.repeat_interleave(th.arange(50), g.indptr[1:] - g.indptr[:-1]).to(DEV)
    keep = slice(lead, lead + e)
    _close(y, _sums(w[keep], x[:49], dst, src[keep].to(DEV), 50), th.float32, "y")


# A caller of the C interface may pass edges that no chunk covers and a gathered table without rows.  Nothing of the table may be
# read then; the pointers here lie in live allocations, and the kernels' names tell who ran.
@pytest.mark.parametrize("op", ["vector_spmm_forward", "attention_backward"])
def test_gathered_table_without_rows(op):
    lib, e, n, h, d = _capi.lib(), 40, 5, 4, 32
    none = th.zeros(2, dtype=th.int32, device=DEV)   # one chunk, of node 0, from position 0 to position 0
    ids, w = th.arange(e, dtype=th.int32, device=DEV), _draw(th.float32, e, h, seed=1)
    table = th.full((n, h, d), float("nan"), device=DEV)
    out = th.full((3, n, h, d), float("nan"), device=DEV)
    query = _capi.OP_SPMM_FWD if op == "vector_spmm_forward" else _capi.OP_ATTENTION_BWD_PAIRS
    ws = th.empty(lib.graphop_workspace_bytes(query, e, n, h, d, 4, 4), dtype=th.uint8, device=DEV)
    tail = [h, d, ws.data_ptr(), ws.numel(), th.cuda.current_stream().cuda_stream]
    p = [t.data_ptr() for t in (none, none, ids, ids, w, table)]
    if op == "vector_spmm_forward":
        args, written = p + [out[0].data_ptr(), 1, e, n, 0] + tail, out[:1]
    else:
        rows = [table.data_ptr()] * 4 + [w.data_ptr(), table.data_ptr()]   # q, k, v, o, lse, d_o
        args = p[:2] + [p[2], 1] + p[:4] + [1] + rows + [1.0] + [t.data_ptr() for t in out] + [e, 0, n] + tail
        written = out[1:]
    with th.profiler.profile(activities=[th.profiler.ProfilerActivity.CUDA]) as seen:
        assert getattr(lib, "graphop_%s_f32_i32" % op)(*args) == _capi.OK
        th.cuda.synchronize()
    ran = [x.name for x in seen.events()]
    assert any("group_walk_kernel" in x for x in ran) and not any("sum_walk_kernel" in x for x in ran), ran
    assert bool((written == 0).all())
