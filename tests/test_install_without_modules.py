"""A package built with ``build.py --no-module`` (no compiler, no torch headers at install time): every call goes to the
library through ctypes, with the same results."""
import pytest
import torch as th

from helpers import chunked, graph_zoo
import custom_op_benchmark_b200 as pkg
from custom_op_benchmark_b200 import build, graphop, wrapper
from custom_op_benchmark_b200.part_csr import partition_csr

DEV = "cuda:0"
ZOO = graph_zoo()


@pytest.fixture
def without_modules(monkeypatch, tmp_path):
    monkeypatch.setattr(pkg, "_NATIVE", None)
    monkeypatch.setattr(build, "module_path", lambda name="graphop": str(tmp_path / (name + ".so")))


def test_the_functions_answer(without_modules):
    with pytest.raises(ImportError):
        pkg.native_functions()
    t = th.zeros(2, dtype=th.int64)
    with pytest.raises(RuntimeError, match="row must be a CUDA tensor"):
        wrapper.SparseSoftmax.apply(t, t, t, th.zeros(2))


def test_a_module_that_does_not_load_is_an_error(without_modules, tmp_path):
    (tmp_path / "graphop_native.so").write_bytes(b"not a module")
    with pytest.raises(ImportError):
        pkg.native_functions_if_built()


def _all_calls(g, idt):
    r = [t.to(DEV) for t in chunked(g, 32, dtype=idt)]
    c = [t.to(DEV) for t in chunked(g, 32, transposed=True, dtype=idt)]
    gen = th.Generator().manual_seed(8)
    x, y, w, rel = (th.randn(*s, generator=gen).to(DEV) for s in
                    ((g.n_dst, 2, 16), (g.n_src, 2, 16), (g.n_edges, 2), (g.n_edges, 16)))
    plans = graphop.GraphPlan(*r, g.n_dst), graphop.GraphPlan(*c, g.n_src)
    calls = [(wrapper.MaskedMMCSR, [*r, *c], [x, y]), (wrapper.SparseSoftmax, r[:3], [w]), (wrapper.NodeMulEdge, r[:3], [x, rel]),
             (wrapper.GraphAttentionBias, [r[0], r[1], r[3], *c], [x, y, y, rel, 0.25]),
             (wrapper.GraphAttention, [r[0], r[1], r[3], c[0], c[1], c[3]], [x, y, y, 0.25, c[2]]),
             (wrapper.GraphAttentionPlanned, plans, [x, y, y, 0.25])]
    if g.n_dst == g.n_src:
        calls.append((wrapper.VectorSPMM, [*r, *c], [w, y]))
    out = [*partition_csr(g.indptr.to(DEV), 7), *graphop.transpose_csr(g.indptr.to(DEV), g.indices.to(DEV), g.n_src)]
    for p in plans:
        out.append(th.tensor([p.c.flags, p.c.band_span, p.c.tile, p.c.n_edges, p.c.n_nodes, p.c.n_chunks]))
    for function, tables, given in calls:
        given = [t.clone().requires_grad_(True) if isinstance(t, th.Tensor) and t.is_floating_point() else t
                 for t in given]
        y_ = function.apply(*tables, *given)
        out += [y_, *th.autograd.grad(y_, [t for t in given if isinstance(t, th.Tensor) and t.is_floating_point()],
                                      th.ones_like(y_))]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name,g", ZOO, ids=[z[0] for z in ZOO])
@pytest.mark.parametrize("idt", [th.int32, th.int64])
def test_same_results(name, g, idt, request):
    want = _all_calls(g, idt)
    request.getfixturevalue("without_modules")
    got = _all_calls(g, idt)
    assert len(got) == len(want) and all(th.equal(a, b) for a, b in zip(got, want))
