"""Performance cases of the graph-attention ops: what a user's program has them do, at the sizes it does it.

A case is a dict of plain values:
    work     "attention"      GraphAttentionPlanned (entry "plans") or GraphAttention on chunk tables (entry "chunks")
             "attention_bias" GraphAttentionBias
             "chain"          the same layer as the reference's script composes it:
                              MaskedMMCSR -> scale -> SparseSoftmax -> VectorSPMM
             "gat"            NodeMulEdge and VectorSPMM on one graph, softmax-normalised edge weights
             "sddmm_softmax"  MaskedMMCSR -> SparseSoftmax, inputs scaled by 3
             "spmm"           VectorSPMM
             "new_graph"      a graph met for the first time: partition_csr of both orientations, transpose_csr, both
                              graph plans, then one GraphAttentionPlanned step on them
    graph    "blocks" (batch x length, fully connected blocks), "band" (batch x length, +-window), "regular" (nodes,
             degree: random in-neighbours and a self-loop each), "uniform" (nodes, edges: both ends random), "rmat"
             (scale, edge_factor), "zipf" (nodes, edges: rank-size in-degrees, s = 1.1)
    heads, dim, dtype ("float32", "float64", "bfloat16"), index ("int32", "int64"), train (forward + backward, or
    forward alone)
"""
import math

import torch as th

from custom_op_benchmark_b200 import graphop, graphs, wrapper
from custom_op_benchmark_b200.part_csr import partition_csr

DEV = "cuda"
DTYPES = {"float32": th.float32, "float64": th.float64, "bfloat16": th.bfloat16}
INDEX = {"int32": th.int32, "int64": th.int64}
ITEM = {"float32": 4, "float64": 8, "bfloat16": 2, "int32": 4, "int64": 8}
MAX_GATHER = 17.7e9  # edges * heads * dim * bytes per element of the largest fused case: drawn cases stay below


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def _case(name, work, graph, heads=1, dim=1, dtype="float32", index="int32", train=True, entry="chunks", **sizes):
    c = dict(work=work, graph=graph, heads=heads, dim=dim, dtype=dtype, index=index, train=train, entry=entry)
    if name:
        c["name"] = name
    c.update(sizes)
    return c


def listed():
    return [
        # a few short sentences through the reference's own three Functions: launches and host work are all there is
        _case("blocks_small_chain", "chain", "blocks", 8, 64, index="int64", batch=8, length=30),
        # the reference's own script: 512 fully connected blocks of 30 nodes, 8 heads of 64, int64 chunk tables
        _case("blocks_script_chain", "chain", "blocks", 8, 64, index="int64", batch=512, length=30),
        # the small attention layer of the benchmark (Erdos-Renyi, 15 in-neighbours and a self-loop), through plans
        _case("er_small_attention", "attention", "regular", 8, 64, entry="plans", nodes=4096, degree=16),
        # a sampled neighbourhood with head sizes that fit no vector width
        _case("sampled_ragged_chain", "chain", "uniform", 3, 20, index="int64", nodes=20011, edges=150001),
        # the benchmark's banded local attention: four sequences of 8192 positions, +-128, training step
        _case("banded_train", "attention", "band", 8, 64, "bfloat16", entry="plans", batch=4, length=8192, window=128),
        # one ragged sequence, inference
        _case("banded_infer_ragged", "attention", "band", 4, 64, "bfloat16", train=False, entry="plans", batch=1,
              length=3001, window=64),
        # the benchmark's headline: fused attention on R-MAT scale 21, 4 heads of 32
        _case("rmat21_attention", "attention", "rmat", 4, 32, entry="plans", scale=21, edge_factor=16),
        # the edge-term layer in bfloat16 on a graph of a quarter of a million nodes, chunk tables
        _case("rmat18_attention_bias", "attention_bias", "rmat", 4, 64, "bfloat16", scale=18, edge_factor=16),
        # the benchmark's node-edge multiply and aggregation, one scale below the headline graph
        _case("rmat20_gat", "gat", "rmat", 4, 32, scale=20, edge_factor=16),
        # the benchmark's skewed-degree stress of scores and softmax
        _case("zipf_sddmm_softmax", "sddmm_softmax", "zipf", 2, 64, nodes=1_000_000, edges=50_000_000),
        # the benchmark's large aggregation (one head of 128 features) at the scale one GPU's share has
        _case("rmat22_spmm", "spmm", "rmat", 1, 128, scale=22, edge_factor=16),
        # mini-batch training: every step a newly sampled graph, prepared and used once
        _case("new_graph_step", "new_graph", "uniform", 4, 32, nodes=60_013, edges=600_007),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, kinds, max_edges, max_nodes):
    """A graph kind and its sizes: nodes and average degree spread over their logarithms."""
    kind = rng.choice(kinds)
    nodes = _log(rng, 500, max_nodes)
    degree = math.exp(rng.uniform(math.log(4), math.log(50)))
    nodes = max(100, int(min(nodes, max_edges / degree)))
    if kind == "rmat":
        ef = rng.randint(6, 24)
        return kind, dict(scale=max(9, int(math.log2(min(nodes, max_edges / (ef + 1))))), edge_factor=ef)
    if kind == "blocks":
        length = rng.randint(5, 60)
        return kind, dict(batch=max(1, int(min(nodes, max_edges / length) / length)), length=length)
    if kind == "regular":
        degree = max(2, int(degree))
        return kind, dict(nodes=nodes, degree=degree)
    return kind, dict(nodes=nodes, edges=int(nodes * degree))


def draw(rng):
    work = rng.choice(["attention", "attention", "band", "chain", "gat", "sddmm_softmax", "spmm", "attention_bias",
                       "new_graph"])
    index = rng.choice(["int32", "int32", "int64"])
    if work == "band":
        heads, dim = rng.choice([1, 2, 4, 8, 12]), rng.choice([32, 64, 64, 64, 128])
        dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
        window = _log(rng, 8, 256)
        cap = 0.5 * MAX_GATHER / (heads * dim * ITEM[dtype] * (2 * window + 1))
        total = min(_log(rng, 300, 64_000), int(cap))
        batch = min(rng.choice([1, 1, 2, 4, 7]), max(1, total // 200))
        return _case(None, "attention", "band", heads, dim, dtype, train=rng.random() < 0.7,
                     entry=rng.choice(["plans", "chunks"]), batch=batch, length=max(50, total // batch), window=window)
    if work == "chain":
        heads, dim = rng.choice([1, 2, 3, 4, 6, 8]), rng.choice([8, 16, 20, 25, 32, 48, 50, 64, 100, 128])
        dtype = rng.choice(["float32", "float32", "float64", "bfloat16"])
        kind, sizes = _draw_graph(rng, ["blocks", "uniform", "regular", "zipf"],
                                  min(4e6, 0.1 * MAX_GATHER / (heads * dim * ITEM[dtype])), 200_000)
        return _case(None, work, kind, heads, dim, dtype, rng.choice(["int64", "int64", "int32"]), **sizes)
    if work == "spmm":
        heads, dim = rng.choice([(1, 32), (1, 64), (1, 128), (1, 256), (2, 64), (4, 32), (8, 16)])
        kinds, nodes, share = ["rmat", "uniform", "zipf"], 4_000_000, 1.0
    elif work == "sddmm_softmax":
        heads, dim = rng.choice([(1, 64), (1, 128), (2, 32), (2, 64), (4, 32), (8, 16), (8, 64)])
        kinds, nodes, share = ["zipf", "uniform", "rmat"], 1_000_000, 1.0
    elif work == "gat":
        heads, dim = rng.choice([(1, 64), (2, 32), (4, 16), (4, 32), (8, 16), (8, 32)])
        kinds, nodes, share = ["rmat", "uniform", "zipf"], 1_500_000, 0.5
    else:
        heads, dim = rng.choice([(1, 32), (1, 64), (1, 128), (2, 32), (2, 64), (4, 16), (4, 32), (4, 64), (8, 16),
                                 (8, 32), (8, 64)])
        kinds, nodes, share = ["rmat", "uniform", "zipf", "regular", "blocks"], 2_000_000, 0.9
    if work in ("attention_bias", "new_graph"):
        nodes, share = 300_000, 0.2
    dtype = rng.choice(["float32", "float32", "bfloat16"])
    kind, sizes = _draw_graph(rng, kinds, min(4.5e7, share * MAX_GATHER / (heads * dim * ITEM[dtype])), nodes)
    train = rng.random() < 0.75 if work == "attention" else True
    return _case(None, work, kind, heads, dim, dtype, index, train, rng.choice(["plans", "chunks"]), **sizes)


# ------------------------------------------------------------------------------------------
# graphs
# ------------------------------------------------------------------------------------------
def _zipf_degrees(n, total, s=1.1):
    """Rank-size in-degrees clip(floor(c r**-s), 1, total), c bisected so that they sum to about `total`."""
    r = th.arange(1, n + 1, dtype=th.float64, device=DEV) ** (-s)
    lo, hi = 1.0, 4.0 * total
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        if int((mid * r).floor_().clamp_(1, total).sum()) < total:
            lo = mid
        else:
            hi = mid
    return (hi * r).floor_().clamp_(1, total).long()


def _rmat_graph(scale, edge_factor, gen, index, a=0.57, b=0.19, c=0.19):
    """The benchmark's R-MAT recipe with an edge count that does not depend on the seed: a quarter more edges are drawn,
    duplicates and self-loops leave, edge_factor * 2**scale of the rest stay (a graph too small to have that many
    repeats some) and every node gets its self-loop."""
    n = 1 << scale
    want = edge_factor * n
    dst, src = (th.zeros(want + want // 4, dtype=th.int64, device=DEV) for _ in range(2))
    for _ in range(scale):
        u = th.rand(dst.numel(), generator=gen, device=DEV)
        dst = (dst << 1) | (u >= a + b)
        src = (src << 1) | ((u >= a) & (u < a + b) | (u >= a + b + c))
    keys = th.unique((dst * n + src)[dst != src])
    keys = keys[th.randperm(keys.numel(), generator=gen, device=DEV)]
    keys = keys[:want] if keys.numel() >= want else keys.repeat(-(-want // keys.numel()))[:want]
    keys = th.cat([keys, th.arange(n, device=DEV) * (n + 1)])
    return graphs.coo_to_graph(keys // n, keys % n, n, index_dtype=index)


def _graph(case, seed):
    kind, index = case["graph"], INDEX[case["index"]]
    gen = th.Generator(device=DEV).manual_seed(seed)

    def ids(count, n):
        return th.randint(0, n, (count,), generator=gen, device=DEV)
    if kind == "blocks":
        return graphs.block_diagonal_graph(case["batch"], case["length"], index, DEV)
    if kind == "band":
        return graphs.banded_graph(case["batch"], case["length"], case["window"], index, DEV)
    if kind == "rmat":
        return _rmat_graph(case["scale"], case["edge_factor"], gen, index)
    n = case["nodes"]
    nodes = th.arange(n, device=DEV)
    if kind == "regular":
        dst = nodes.repeat_interleave(case["degree"])
        src = ids(dst.numel(), n)
        src[:: case["degree"]] = nodes
        return graphs.coo_to_graph(dst, src, n, index_dtype=index)
    if kind == "uniform":
        return graphs.coo_to_graph(ids(case["edges"], n), ids(case["edges"], n), n, index_dtype=index)
    deg = _zipf_degrees(n, case["edges"])[th.randperm(n, generator=gen, device=DEV)]
    dst = nodes.repeat_interleave(deg)
    return graphs.coo_to_graph(dst, ids(dst.numel(), n), n, index_dtype=index)


# ------------------------------------------------------------------------------------------
# what a program has in hand, and one pass
# ------------------------------------------------------------------------------------------
def prepare(case, seed):
    g = _graph(case, seed)
    index, work = INDEX[case["index"]], case["work"]
    st = {"case": case, "graph": g}
    h, d, e, n, dt = case["heads"], case["dim"], g.n_edges, g.n_dst, DTYPES[case["dtype"]]
    row, ptr = partition_csr(g.indptr, 32)
    col, ptr_t = partition_csr(g.indptr_t, 32)
    st["R"] = [row.to(index), ptr.to(index), g.eid, g.indices]
    st["C"] = [col.to(index), ptr_t.to(index), g.eid_t, g.indices_t]
    if work == "attention" and case["entry"] == "plans":
        st["plans"] = (graphop.GraphPlan(*st["R"], g.n_dst), graphop.GraphPlan(*st["C"], g.n_src))
    gen = th.Generator(device=DEV).manual_seed(seed + 7919)
    edge_shape = (e,) if h == 1 else (e, h)     # what the ops return for one head
    make = th.float64 if dt == th.float64 else th.float32

    def normal(*shape, mag=1.0):
        return (th.randn(*shape, generator=gen, device=DEV, dtype=make) * mag).to(dt)

    def weights():
        return th.rand(e, h, generator=gen, device=DEV, dtype=make).to(dt)
    if work == "gat":
        w = graphop.sparse_softmax_forward(*st["R"][:3], weights(), num_nodes=n)
        st["in"] = [normal(n, h, d), normal(e, d), w]
        st["grad"] = [normal(*edge_shape), normal(n, h, d)]
    elif work == "sddmm_softmax":
        st["in"] = [normal(n, h, d, mag=3.0), normal(n, h, d, mag=3.0)]
        st["grad"] = [normal(*edge_shape)]
    elif work == "spmm":
        st["in"] = [weights(), normal(n, h, d)]
        st["grad"] = [normal(n, h, d)]
    else:
        st["in"] = [normal(n, h, d) for _ in range(3)]
        if work == "attention_bias":
            st["in"].append(normal(e, d, mag=0.5))
        st["grad"] = [normal(n, h, d)]
    if case["train"]:
        for t in st["in"]:
            t.requires_grad_(True)
    return st


def _new_graph(g, index):
    """The transposed CSR and the plans of both orientations, from the row CSR alone."""
    row, ptr = partition_csr(g.indptr, 32)
    ptr_t, indices_t, eid_t = graphop.transpose_csr(g.indptr, g.indices, g.n_src)
    col, cptr = partition_csr(ptr_t, 32)
    plans = (graphop.GraphPlan(row.to(index), ptr.to(index), None, g.indices, g.n_dst),
             graphop.GraphPlan(col.to(index), cptr.to(index), eid_t, indices_t, g.n_src))
    return plans, [ptr_t, indices_t, eid_t]


def run(st):
    case = st["case"]
    work, scale = case["work"], case["dim"] ** -0.5
    R, C, x, built = st["R"], st["C"], st["in"], []
    if work == "new_graph":
        plans, built = _new_graph(st["graph"], INDEX[case["index"]])
        out = [wrapper.GraphAttentionPlanned.apply(*plans, *x, scale)]
    elif work == "attention":
        if case["entry"] == "plans":
            out = [wrapper.GraphAttentionPlanned.apply(*st["plans"], *x, scale)]
        else:
            out = [wrapper.GraphAttention.apply(R[0], R[1], R[3], C[0], C[1], C[3], *x, scale, C[2])]
    elif work == "attention_bias":
        out = [wrapper.GraphAttentionBias.apply(R[0], R[1], R[3], *C, *x, scale)]
    elif work == "chain":
        s = wrapper.MaskedMMCSR.apply(*R, *C, x[0], x[1]) * scale
        out = [wrapper.VectorSPMM.apply(*R, *C, wrapper.SparseSoftmax.apply(*R[:3], s), x[2])]
    elif work == "gat":
        out = [wrapper.NodeMulEdge.apply(*R[:3], x[0], x[1]), wrapper.VectorSPMM.apply(*R, *C, x[2], x[0])]
    elif work == "sddmm_softmax":
        out = [wrapper.SparseSoftmax.apply(*R[:3], wrapper.MaskedMMCSR.apply(*R, *C, x[0], x[1]))]
    else:
        out = [wrapper.VectorSPMM.apply(*R, *C, x[0], x[1])]
    if not case["train"]:
        return out
    return built + [t.detach() for t in out] + list(th.autograd.grad(out, x, st["grad"]))


# ------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct passes may differ
# ------------------------------------------------------------------------------------------
def _counts(case):
    """Nodes and edges."""
    k = case["graph"]
    if k in ("blocks", "band"):
        n = case["batch"] * case["length"]
        if k == "blocks":
            return n, n * case["length"]
        w = min(case["window"], case["length"] - 1)
        return n, case["batch"] * (case["length"] * (2 * w + 1) - w * (w + 1))
    if k == "rmat":
        return 1 << case["scale"], (1 << case["scale"]) * (case["edge_factor"] + 1)
    return case["nodes"], case["nodes"] * case["degree"] if k == "regular" else case["edges"]


def work(case):
    n, e = _counts(case)
    h, d, s, i = case["heads"], case["dim"], ITEM[case["dtype"]], ITEM[case["index"]]
    F, S, B = n * h * d * s, e * h * s, e * d * s        # a node tensor, an edge tensor, an edge-feature tensor
    I, P = (e + n + 1) * i, e * i                        # a CSR, its edge ids
    kind, train, one = case["work"], case["train"], 2 * e * h * d   # one multiply-add per edge and feature
    if case["graph"] == "band" and kind == "attention":
        I, P = 8 * n, 0                                  # first neighbour and count say it all
    if kind in ("attention", "attention_bias", "new_graph"):
        b, f = 4 * F + I + 4 * n * h, 2 * one
        if train:
            b, f = b + 8 * F + 2 * I + P + 4 * n * h, f + 5 * one
        if kind == "new_graph":     # CSR in; transposed CSR with edge ids, chunk tables and owner tables out
            b += 2 * I + P + 2 * 16 * max(n, e // 32) + 2 * 4 * e
        if kind == "attention_bias":
            b, f = b + 3 * B, f + 3 * one
        return {"bytes": b, "flops": f}
    sddmm, softmax, spmm = 2 * F + S + I, 2 * S + (n + 1) * i, 2 * F + S + I
    sddmm_b, softmax_b, spmm_b = 4 * F + S + 2 * I + P, 3 * S + (n + 1) * i, 3 * F + 2 * S + 2 * I + P
    if kind == "chain":
        return {"bytes": sddmm + softmax + spmm + sddmm_b + softmax_b + spmm_b, "flops": 6 * one}
    if kind == "sddmm_softmax":
        return {"bytes": sddmm + softmax + sddmm_b + softmax_b, "flops": 3 * one}
    if kind == "spmm":
        return {"bytes": spmm + spmm_b, "flops": 3 * one}
    return {"bytes": spmm + spmm_b + 3 * F + 3 * B + 2 * S, "flops": 6 * one}


def tolerance(case):
    return {"rel": {"float32": 1e-5, "float64": 1e-12, "bfloat16": 1e-2}[case["dtype"]]}
