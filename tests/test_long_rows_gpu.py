"""Rows longer than a work tile, on rows so wide that a lane group walks several tiles as one.  The gathering walker sums such a row
in the pieces that the tiles make of it, so the error against float64 is that of a walk of one tile: head by head the rows are
narrow enough for that, and everything else is the same; what may differ is the order in which a row's few pieces are added up
(the tenth).  The summing walker has its two levels instead, and walks short enough for them."""
import pytest
import torch as th

from custom_op_benchmark_b200 import graphop, graphs
from custom_op_benchmark_b200.part_csr import partition_csr
from oracle import edge_list_f64 as ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NODES, DEGREE = 4096, 500   # 2M edges: tiles of 64, a row is cut into eight pieces; 32 K tiles
# A walk of n edges of one row adds up n / 32 blocks one after the other, squared roundings n 32^2 / 3 + n^3 / 96; a tile per walk,
# two blocks each, and its records n 32^2 / 3 + n^3 / 192.  For the at most 8 tiles of 64 in a walk that is 1.33 times the error.
SUMS = 1.33 * 1.1


@pytest.fixture(scope="module")
def graph():
    gen = th.Generator(device=DEV).manual_seed(1)
    dst = th.arange(NODES, device=DEV).repeat_interleave(DEGREE)
    g = graphs.coo_to_graph(dst, th.randint(0, NODES, dst.shape, generator=gen, device=DEV), NODES, index_dtype=th.int32)
    row, ptr = partition_csr(g.indptr, 32)
    col, ptr_t = partition_csr(g.indptr_t, 32)
    return g, [row.int(), ptr.int(), g.eid, g.indices], [col.int(), ptr_t.int(), g.eid_t, g.indices_t]


def _draw(*shape, seed):
    gen = th.Generator(device=DEV).manual_seed(seed)
    return th.rand(*shape, generator=gen, device=DEV)   # terms of one sign: a chain's roundings show


def _check(run, inputs, want, names, sums=()):
    """run(inputs of some heads) -> outputs; want: float64, (n, heads, ...) each; sums: names of the summing walker's."""
    whole = run(*inputs)
    apart = [th.cat(parts, 1) for parts in zip(*(run(*(t[:, h:h + 1].contiguous() for t in inputs)) for h in range(inputs[0].size(1))))]
    for name, a, b, w in zip(names, whole, apart, want):
        error = [float((x.view(w.shape).double() - w).norm() / w.norm()) for x in (a, b)]
        assert error[0] <= (SUMS if name in sums else 1.1) * error[1], (name, error)


@pytest.mark.parametrize("planned", [False, True])
def test_attention(graph, planned):
    g, r, c = graph
    h, d = 8, 128
    q, k, v, grad = (_draw(NODES, h, d, seed=i) for i in range(4))
    scale = d ** -0.5
    plans = (graphop.GraphPlan(*r, NODES), graphop.GraphPlan(*c, NODES))

    def run(q, k, v, grad):
        if planned:
            o, lse = graphop.attention_forward_planned(plans[0], q, k, v, scale)
            back = graphop.attention_backward_planned(*plans, q, k, v, o, lse, grad, scale)
        else:   # without the transposed edge ids: the source side forms the probabilities again
            o, lse = graphop.attention_forward(r[0], r[1], r[3], q, k, v, scale)
            back = graphop.attention_backward(r[0], r[1], r[3], c[0], c[1], c[3], q, k, v, o, lse, grad, scale)
        return (o, lse.view(NODES, -1), *back)
    want = ref.attention_f64(g.indptr, g.indices, q, k, v, scale, grad, chunk=1 << 17)
    _check(run, (q, k, v, grad), want, ("o", "lse", "dq", "dk", "dv"), sums=("dk", "dv") if planned else ())


@pytest.mark.parametrize("h", [6, 8])   # the rows of the edges copied once per head, and once for all heads
def test_sums_of_edge_rows(graph, h):
    g, r, _ = graph
    d = 128
    x, a, grad = _draw(g.n_edges, d, seed=5), _draw(NODES, h, d, seed=6), _draw(g.n_edges, h, seed=7)
    want = th.zeros(NODES, h, d, dtype=th.float64, device=DEV)
    for part in th.arange(NODES, device=DEV).split(256):   # the graph's rows are runs of DEGREE edges, edge ids in order
        e = slice(int(part[0]) * DEGREE, (int(part[-1]) + 1) * DEGREE)
        want[part] = th.einsum("nkh,nkd->nhd", grad[e].double().view(len(part), DEGREE, h), x[e].double().view(len(part), DEGREE, d))

    def run(a, grad):
        return graphop.node_mul_edge_backward(*r[:3], a, x, grad)[:1]
    _check(run, (a, grad), [want], ("dA",))


def test_aggregation():
    """One head of 8192 features is 64 blocks of 128, and would be a hundred tiles of 128 per walk; alone, a block has two.  As above:
    a row's 2.6 walks of 6 tiles, 24 blocks one after the other each, are no more than 1.6 times the error of its 8 walks of 8
    blocks; with the row in one chain of 63 blocks it is 2.1 times."""
    n, degree, d = 2000, 2000, 8192
    gen = th.Generator(device=DEV).manual_seed(2)
    dst = th.arange(n, device=DEV).repeat_interleave(degree)
    g = graphs.coo_to_graph(dst, th.randint(0, n, dst.shape, generator=gen, device=DEV), n, index_dtype=th.int32)
    row, ptr = partition_csr(g.indptr, 32)
    r = [row.int(), ptr.int(), g.eid, g.indices]
    w, x = _draw(g.n_edges, seed=8), _draw(n, 1, d, seed=9)
    whole = graphop.vector_spmm_forward(*r, w, x)
    assert th.equal(whole, graphop.vector_spmm_forward_planned(graphop.GraphPlan(*r, n), w, x))   # the same pieces
    rows = th.arange(3, n, 61, device=DEV)
    for block in (slice(0, 128), slice(4096, 4224)):
        alone = graphop.vector_spmm_forward(*r, w, x[:, :, block].contiguous())
        at = rows.view(-1, 1) * degree + th.arange(degree, device=DEV)
        want = th.einsum("nk,nkd->nd", w[at].double(), x[g.indices[at].long(), 0, block].double())
        error = [float((t.view(n, -1)[rows].double() - want).norm() / want.norm()) for t in (whole[..., block], alone)]
        assert error[0] <= 1.6 * error[1], error
