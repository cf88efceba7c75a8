// The autograd Functions of wrapper.py in native code: what `apply` of each class runs.
//
// A graph-attention layer on a small graph is a handful of kernels of a few microseconds; the same Functions written in
// Python (argument checks, ctypes calls, torch.autograd.Function's Python forward and backward) cost 40 to 60 us of
// host time per op and direction, several times the kernels.  Here an op is one pybind call, a C++ autograd node and the
// C ABI's planned entry point; the backward runs on autograd's thread without taking the interpreter lock.
//
// The chunk-table signatures (row, indptr, eid, indices) of the reference carry the graph on every call.  The owner
// table, 32-bit index copies and work tiles that the forward makes from them (a "view": a plan without the shape
// analysis) are saved for the backward of the same call, beside its tensors.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <limits>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../graphop_internal.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------
// checks: the texts and exception types of graphop.py
// ------------------------------------------------------------------------------------------
[[noreturn]] void fail(const std::string& text) { throw std::runtime_error(text); }

void check_input(const Tensor& t, const char* name) {
  if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor");
  if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
}
std::string dtype_text(const Tensor& t) {
  const auto names = c10::getDtypeNames(t.scalar_type());
  return "torch." + names.first;
}
int index_bytes_of(at::ArrayRef<const Tensor*> ts) {
  const Tensor* first = nullptr;
  for (const Tensor* t : ts) {
    if (!t || !t->defined()) continue;
    if (!first) first = t;
    if (first->scalar_type() != at::kInt && first->scalar_type() != at::kLong)
      fail("index tensors must be int32 or int64, got " + dtype_text(*first));
    if (t->scalar_type() != first->scalar_type())
      fail("expected all index tensors to share dtype " + dtype_text(*first) + ", got " + dtype_text(*t));
  }
  return first && first->scalar_type() == at::kLong ? 8 : 4;
}
int elem_of(std::initializer_list<const Tensor*> ts) {
  const at::ScalarType dt = (*ts.begin())->scalar_type();
  if (dt != at::kFloat && dt != at::kDouble && dt != at::kBFloat16)
    fail("\"graphop\" not implemented for '" + std::string(toString(dt)) + "'");
  for (const Tensor* t : ts)
    if (t->scalar_type() != dt)
      fail("expected all floating tensors to share dtype " + dtype_text(**ts.begin()) + ", got " + dtype_text(*t));
  return dt == at::kFloat ? 0 : dt == at::kDouble ? 1 : 2;
}
struct NodeShape { int64_t n; int H, D; };
NodeShape node_shape(const Tensor& t) {
  if (t.dim() != 2 && t.dim() != 3) fail("node tensors must be (n, d) or (n, h, d)");
  return {t.size(0), t.dim() == 2 ? 1 : (int)t.size(1), (int)t.size(-1)};
}
int edge_heads(const Tensor& t) {
  if (t.dim() != 1 && t.dim() != 2) fail("edge tensors must be (e,) or (e, h)");
  return t.dim() == 1 ? 1 : (int)t.size(1);
}
void check_status(int rc, const char* what) {
  if (rc == GRAPHOP_OK) return;
  std::string msg = std::string("graphop_") + what + ": " + graphop_error_string(rc);
  if (rc == GRAPHOP_ERR_CUDA) msg += " (cudaError " + std::to_string(graphop_last_cuda_error()) + ")";
  fail(msg);
}

// ------------------------------------------------------------------------------------------
// graphs: plans made by Python, views made here
// ------------------------------------------------------------------------------------------
struct Graph {
  graphop_plan_t plan{};
  std::vector<Tensor> keep;   // device memory the plan refers to
};
using GraphPtr = std::shared_ptr<Graph>;

void check_chunks(const Tensor& row, const Tensor& indptr) {
  if (indptr.size(0) != row.size(0) + 1) fail("indptr must hold row.size(0) + 1 entries");
}

// The view of a chunk table; eid and indices may be undefined.  n_nodes < 0: for an op that walks no node rows.  clear: an
// edge output that is zero where no chunk covers it, done on the way.
GraphPtr view_of(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& indices, int64_t n_edges,
                 int64_t n_nodes, cudaStream_t stream, const Tensor& clear = Tensor()) {
  const int ib = index_bytes_of({&row, &indptr, &eid, &indices});
  const auto data = [](const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
  auto g = std::make_shared<Graph>();
  const size_t bytes = graphop_internal_view_bytes(n_edges, n_nodes, ib);
  const Tensor memory = at::empty({(int64_t)bytes}, row.options().dtype(at::kByte));
  check_status(graphop_internal_view_build(data(row), data(indptr), data(eid), data(indices), ib, row.size(0), n_edges,
                                           n_nodes, data(clear), clear.defined() ? clear.nbytes() : 0, memory.data_ptr(), bytes,
                                           &g->plan, (graphop_stream_t)stream),
               "view_build");
  g->keep = {memory};
  // 32-bit index arrays are used where they are
  for (const Tensor* t : {&eid, &indices})
    if (ib == 4 && t->defined()) g->keep.push_back(*t);
  return g;
}

// What one op call needs besides its tensors: device guard, stream, workspace.
struct Call {
  c10::cuda::CUDAGuard guard;
  cudaStream_t stream;
  Tensor scratch;
  void* ws = nullptr;
  size_t bytes = 0;
  explicit Call(const Tensor& on) : guard(on.device()), stream(at::cuda::getCurrentCUDAStream(on.get_device())) {}
  void workspace(int op, int64_t n_edges, int64_t n_nodes, int H, int D, const Tensor& like) {
    bytes = graphop_workspace_bytes(op, n_edges, n_nodes, H, D, (int)like.element_size(), 4);
    scratch = at::empty({(int64_t)bytes + 256}, like.options().dtype(at::kByte));
    ws = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(scratch.data_ptr()) + 255) / 256 * 256);
  }
};

// a tensor's storage as the element type the entry point wants
template <typename E> E* ptr(const Tensor& t) { return reinterpret_cast<E*>(t.data_ptr()); }

// f is called with a null pointer of the element type
template <class F> auto by_elem(int elem, F&& f) {
  if (elem == 0) return f((float*)nullptr);
  if (elem == 1) return f((double*)nullptr);
  return f((uint16_t*)nullptr);
}

// one overload set per op over the three element types
#define GRAPHOP_OVERLOADS(op)                                                                                        \
  template <class... X> int op(float*, X... x) { return graphop_##op##_f32(x...); }                                  \
  template <class... X> int op(double*, X... x) { return graphop_##op##_f64(x...); }                                 \
  template <class... X> int op(uint16_t*, X... x) { return graphop_##op##_bf16(x...); }
GRAPHOP_OVERLOADS(maskedmm_csr_forward_planned)
GRAPHOP_OVERLOADS(maskedmm_csr_backward_planned)
GRAPHOP_OVERLOADS(node_mul_edge_forward_planned)
GRAPHOP_OVERLOADS(node_mul_edge_backward_planned)
GRAPHOP_OVERLOADS(sparse_softmax_forward_planned)
GRAPHOP_OVERLOADS(sparse_softmax_backward_planned)
GRAPHOP_OVERLOADS(vector_spmm_forward_planned)
GRAPHOP_OVERLOADS(vector_spmm_backward_planned)
GRAPHOP_OVERLOADS(attention_forward_planned)
GRAPHOP_OVERLOADS(attention_backward_planned)
GRAPHOP_OVERLOADS(internal_attention_bias_forward)
GRAPHOP_OVERLOADS(internal_attention_bias_backward)
#undef GRAPHOP_OVERLOADS

// ------------------------------------------------------------------------------------------
// the chunk-table arguments of one Function: views made when needed, versions checked in the backward
// ------------------------------------------------------------------------------------------
struct Tables {
  std::vector<Tensor> t;
  std::vector<uint32_t> versions;
  GraphPtr rows;
  Tables(std::initializer_list<Tensor> list) : t(list) {
    versions.reserve(t.size());
    for (const Tensor& x : t) versions.push_back(x.defined() && !x.is_inference() ? x._version() : 0);
  }
  void check_unmodified() const {
    for (size_t i = 0; i < t.size(); ++i)
      if (t[i].defined() && !t[i].is_inference() && t[i]._version() != versions[i])
        fail("one of the variables needed for gradient computation has been modified by an inplace operation: an index "
             "tensor of a graphop function");
  }
};
using TablesPtr = std::shared_ptr<Tables>;

// Links `outputs` to a backward node of type N made from `inputs` (the differentiable ones, in the order of the
// gradients the node returns) when any of them needs a gradient; `save` stores what the backward reads.
template <class N, class Save>
void record(std::initializer_list<Tensor> inputs, Tensor& output, Save&& save) {
  if (!c10::GradMode::is_enabled()) return;
  bool any = false;
  for (const Tensor& t : inputs) any = any || t.requires_grad();
  if (!any) return;
  std::shared_ptr<N> node(new N(), torch::autograd::deleteNode);
  torch::autograd::edge_list edges;
  edges.reserve(inputs.size());
  for (const Tensor& t : inputs) edges.push_back(torch::autograd::impl::gradient_edge(t));
  for (auto& e : edges)
    if (!e.function) e = torch::autograd::Edge();
  node->set_next_edges(std::move(edges));
  torch::autograd::set_history(output, node);
  save(*node);   // an output is saved after it has its history, so that it does not hold the node that holds it
}

Tensor upstream(variable_list& grads, const char* name) {
  Tensor g = grads[0].contiguous();
  check_input(g, name);
  return g;
}
Tensor edge_out(const Tensor& node, int64_t n_edges, int H) {
  return H == 1 ? at::empty({n_edges}, node.options()) : at::empty({n_edges, H}, node.options());
}
graphop_stream_t raw(cudaStream_t s) { return (graphop_stream_t)s; }

// What a node of these ops keeps: written when the call is recorded and read-only from then on, but for `saved`, which a
// backward that does not retain the graph releases.  Two threads may run the backward of one graph: `saved` is touched
// under the node's mutex, everything else a backward makes is its own.
struct GraphNode : Node {
  TablesPtr tables;             // chunk-table forms
  std::vector<SavedVariable> saved;
  std::string name() const override { return "GraphopBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    for (SavedVariable& s : saved) s.reset_data();
  }
  std::vector<Tensor> unpack_saved() {
    const std::shared_ptr<Node> self = shared_from_this();   // for a saved output
    std::lock_guard<std::mutex> hold(mutex_);
    std::vector<Tensor> t;
    t.reserve(saved.size());
    for (const SavedVariable& s : saved) t.push_back(s.unpack(self));
    return t;
  }
};

// ---- SparseSoftmax (wrapper.py:8-18) ------------------------------------------------------
struct SparseSoftmaxBackward : GraphNode {
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor()};
    tables->check_unmodified();
    const std::vector<Tensor> kept = unpack_saved();
    const Tensor y = kept[0], dy = upstream(grads, "dy");
    const int elem = elem_of({&y, &dy}), H = edge_heads(dy);
    Call c(y);
    Tensor dx = at::empty_like(dy);
    const int64_t e = tables->t[2].size(0);
    if (e == 0) return {dx};
    c.workspace(GRAPHOP_OP_SOFTMAX_BWD, e, 0, H, 1, y);
    const graphop_plan_t* p = &tables->rows->plan;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return sparse_softmax_backward_planned(k, p, (const E*)ptr<E>(y), (const E*)ptr<E>(dy), ptr<E>(dx), H, c.ws, c.bytes,
                                             raw(c.stream));
    }), "sparse_softmax_backward");
    return {dx};
  }
};
Tensor sparse_softmax(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& x) {
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(eid, "eid"); check_input(x, "x");
  const int elem = elem_of({&x}), H = edge_heads(x);
  index_bytes_of({&row, &indptr, &eid});
  check_chunks(row, indptr);
  auto tb = std::make_shared<Tables>(std::initializer_list<Tensor>{row, indptr, eid});
  Call c(x);
  const int64_t e = eid.size(0);
  Tensor y = at::empty_like(x.detach());
  if (e > 0) {
    tb->rows = view_of(row, indptr, eid, Tensor(), e, -1, c.stream, y);
    c.workspace(GRAPHOP_OP_SOFTMAX_FWD, e, 0, H, 1, x);
    graphop_plan_t cleared = tb->rows->plan;   // by the view, for this call's output
    cleared.flags |= GRAPHOP_PLAN_COVERED;
    const graphop_plan_t* p = &cleared;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return sparse_softmax_forward_planned(k, p, (const E*)ptr<E>(x), ptr<E>(y), H, c.ws, c.bytes, raw(c.stream));
    }), "sparse_softmax_forward");
  }
  record<SparseSoftmaxBackward>({x}, y, [&](SparseSoftmaxBackward& n) {
    n.tables = tb;
    n.saved.emplace_back(y, true);
  });
  return y;
}

// ---- MaskedMMCSR (wrapper.py:20-30) -------------------------------------------------------
// the view of the other orientation, whose tables start at t[at]
GraphPtr column_view(const Tables& tb, int at, int64_t e, int64_t n_src, cudaStream_t stream) {
  const char* names[] = {"col", "indptr", "eid", "indices"};
  for (int i = 0; i < 4; ++i) check_input(tb.t[at + i], names[i]);
  check_chunks(tb.t[at], tb.t[at + 1]);
  std::vector<const Tensor*> all;   // both orientations: one call has one index type
  for (const Tensor& t : tb.t) all.push_back(&t);
  index_bytes_of(all);
  return view_of(tb.t[at], tb.t[at + 1], tb.t[at + 2], tb.t[at + 3], e, n_src, stream);
}
struct MaskedMMBackward : GraphNode {
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    tables->check_unmodified();
    const std::vector<Tensor> kept = unpack_saved();
    const Tensor A = kept[0], B = kept[1], dy = upstream(grads, "dy");
    const int elem = elem_of({&A, &B, &dy});
    const NodeShape s = node_shape(A);
    Call c(A);
    const int64_t e = tables->t[2].size(0), nb = B.size(0);
    Tensor dA = at::empty_like(A.detach()), dB = at::empty_like(B.detach());
    if (e == 0) return {dA.zero_(), dB.zero_()};
    const GraphPtr cols = column_view(*tables, 4, e, nb, c.stream);
    c.workspace(GRAPHOP_OP_MASKEDMM_BWD, e, std::max(s.n, nb), s.H, s.D, A);
    const graphop_plan_t *pr = &tables->rows->plan, *pc = &cols->plan;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return maskedmm_csr_backward_planned(k, pr, pc, (const E*)ptr<E>(A), (const E*)ptr<E>(B), (const E*)ptr<E>(dy),
                                           ptr<E>(dA), ptr<E>(dB), s.n, nb, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "maskedmm_csr_backward");
    return {dA, dB};
  }
};
Tensor maskedmm_csr(const Tensor& row, const Tensor& indptr_r, const Tensor& eid_r, const Tensor& indices_r,
                    const Tensor& col, const Tensor& indptr_c, const Tensor& eid_c, const Tensor& indices_c,
                    const Tensor& A, const Tensor& B) {
  check_input(row, "row"); check_input(indptr_r, "indptr"); check_input(eid_r, "eid"); check_input(indices_r, "indices");
  check_input(A, "A"); check_input(B, "B");
  const int elem = elem_of({&A, &B});
  index_bytes_of({&row, &indptr_r, &eid_r, &indices_r});
  const NodeShape s = node_shape(A);
  check_chunks(row, indptr_r);
  auto tb = std::make_shared<Tables>(
      std::initializer_list<Tensor>{row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c});
  Call c(A);
  const int64_t e = eid_r.size(0), nb = B.size(0);
  Tensor y = edge_out(A, e, s.H);
  if (e > 0) {
    tb->rows = view_of(row, indptr_r, eid_r, indices_r, e, s.n, c.stream, y);
    c.workspace(GRAPHOP_OP_MASKEDMM_FWD, e, std::max(s.n, nb), s.H, s.D, A);
    graphop_plan_t cleared = tb->rows->plan;   // by the view, for this call's output
    cleared.flags |= GRAPHOP_PLAN_COVERED;
    const graphop_plan_t* p = &cleared;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return maskedmm_csr_forward_planned(k, p, (const E*)ptr<E>(A), (const E*)ptr<E>(B), ptr<E>(y), s.n, nb, s.H, s.D, c.ws,
                                          c.bytes, raw(c.stream));
    }), "maskedmm_csr_forward");
  }
  record<MaskedMMBackward>({A, B}, y, [&](MaskedMMBackward& n) {
    // the backward reads the column side; wrong tensors are reported there, as its arguments always were
    n.tables = tb;
    n.saved.emplace_back(A, false);
    n.saved.emplace_back(B, false);
  });
  return y;
}

// ---- NodeMulEdge (wrapper.py:32-42) -------------------------------------------------------
struct NodeMulEdgeBackward : GraphNode {
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    tables->check_unmodified();
    const std::vector<Tensor> kept = unpack_saved();
    const Tensor A = kept[0], B = kept[1], dy = upstream(grads, "dy");
    const int elem = elem_of({&A, &B, &dy});
    const NodeShape s = node_shape(A);
    Call c(A);
    const int64_t e = tables->t[2].size(0);
    Tensor dA = at::empty_like(A.detach()), dB = at::empty_like(B.detach());
    if (e == 0) return {dA.zero_(), dB};
    c.workspace(GRAPHOP_OP_NODE_MUL_EDGE_BWD, e, s.n, s.H, s.D, A);
    const graphop_plan_t* p = &tables->rows->plan;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return node_mul_edge_backward_planned(k, p, (const E*)ptr<E>(A), (const E*)ptr<E>(B), (const E*)ptr<E>(dy), ptr<E>(dA),
                                            ptr<E>(dB), s.n, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "node_mul_edge_backward");
    return {dA, dB};
  }
};
Tensor node_mul_edge(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& A, const Tensor& B) {
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(eid, "eid"); check_input(A, "A"); check_input(B, "B");
  const int elem = elem_of({&A, &B});
  index_bytes_of({&row, &indptr, &eid});
  const NodeShape s = node_shape(A);
  check_chunks(row, indptr);
  auto tb = std::make_shared<Tables>(std::initializer_list<Tensor>{row, indptr, eid});
  Call c(A);
  const int64_t e = eid.size(0);
  Tensor y = edge_out(A, e, s.H);
  if (e > 0) {
    tb->rows = view_of(row, indptr, eid, Tensor(), e, s.n, c.stream, y);
    c.workspace(GRAPHOP_OP_NODE_MUL_EDGE_FWD, e, s.n, s.H, s.D, A);
    graphop_plan_t cleared = tb->rows->plan;   // by the view, for this call's output
    cleared.flags |= GRAPHOP_PLAN_COVERED;
    const graphop_plan_t* p = &cleared;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return node_mul_edge_forward_planned(k, p, (const E*)ptr<E>(A), (const E*)ptr<E>(B), ptr<E>(y), s.n, s.H, s.D, c.ws,
                                           c.bytes, raw(c.stream));
    }), "node_mul_edge_forward");
  }
  record<NodeMulEdgeBackward>({A, B}, y, [&](NodeMulEdgeBackward& n) {
    n.tables = tb;
    n.saved.emplace_back(A, false);
    n.saved.emplace_back(B, false);
  });
  return y;
}

// ---- VectorSPMM (wrapper.py:44-55) --------------------------------------------------------
struct VectorSPMMBackward : GraphNode {
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    tables->check_unmodified();
    const std::vector<Tensor> kept = unpack_saved();
    const Tensor w = kept[0], x = kept[1], dy = upstream(grads, "dy");
    const int elem = elem_of({&w, &dy, &x});
    const NodeShape s = node_shape(x);
    Call c(x);
    const int64_t e = tables->t[2].size(0), n_dst = dy.size(0);
    Tensor dw = at::empty_like(w.detach()), dx = at::empty_like(x.detach());
    if (e == 0) return {dw, dx.zero_()};
    const GraphPtr cols = column_view(*tables, 4, e, s.n, c.stream);
    c.workspace(GRAPHOP_OP_SPMM_BWD, e, std::max(n_dst, s.n), s.H, s.D, x);
    const graphop_plan_t *pr = &tables->rows->plan, *pt = &cols->plan;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return vector_spmm_backward_planned(k, pr, pt, (const E*)ptr<E>(w), (const E*)ptr<E>(dy), (const E*)ptr<E>(x),
                                          ptr<E>(dw), ptr<E>(dx), n_dst, s.n, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "vector_spmm_backward");
    return {dw, dx};
  }
};
Tensor vector_spmm(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& indices, const Tensor& col,
                   const Tensor& indptr_t, const Tensor& eid_t, const Tensor& indices_t, const Tensor& w, const Tensor& x) {
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(eid, "eid"); check_input(indices, "indices");
  check_input(w, "edata"); check_input(x, "x");
  const int elem = elem_of({&w, &x});
  index_bytes_of({&row, &indptr, &eid, &indices});
  const NodeShape s = node_shape(x);
  if (edge_heads(w) != s.H) fail("edata and x disagree on the number of heads");
  check_chunks(row, indptr);
  auto tb = std::make_shared<Tables>(std::initializer_list<Tensor>{row, indptr, eid, indices, col, indptr_t, eid_t, indices_t});
  Call c(x);
  const int64_t e = eid.size(0);
  Tensor y = at::empty(x.sizes(), x.options());
  if (e == 0) {
    y.zero_();
  } else {
    tb->rows = view_of(row, indptr, eid, indices, e, s.n, c.stream);
    c.workspace(GRAPHOP_OP_SPMM_FWD, e, s.n, s.H, s.D, x);
    const graphop_plan_t* p = &tb->rows->plan;
    check_status(by_elem(elem, [&](auto* k) {
      using E = std::remove_pointer_t<decltype(k)>;
      return vector_spmm_forward_planned(k, p, (const E*)ptr<E>(w), (const E*)ptr<E>(x), ptr<E>(y), s.n, s.n, s.H, s.D, c.ws,
                                         c.bytes, raw(c.stream));
    }), "vector_spmm_forward");
  }
  record<VectorSPMMBackward>({w, x}, y, [&](VectorSPMMBackward& n) {
    n.tables = tb;
    n.saved.emplace_back(w, false);
    n.saved.emplace_back(x, false);
  });
  return y;
}

// ---- fused attention on plans, with and without the edge term ------------------------------
struct AttentionBackward : GraphNode {
  GraphPtr rows, cols;   // cols: null for chunk tables
  double scale = 1.0;
  bool bias = false;
  variable_list apply(variable_list&& grads) override {
    const size_t n_out = bias ? 4 : 3;
    if (!grads[0].defined()) return variable_list(n_out);
    if (tables) tables->check_unmodified();
    const std::vector<Tensor> kept = unpack_saved();
    const Tensor q = kept[0], k = kept[1], v = kept[2], o = kept[3], lse = kept[4], rel = bias ? kept[5] : Tensor(),
                 g = upstream(grads, "d_o");
    const int elem = elem_of({&q, &k, &v, &o, &g});
    const NodeShape s = node_shape(q);
    Call c(q);
    Tensor dq = at::empty_like(q.detach()), dk = at::empty_like(k.detach()), dv = at::empty_like(v.detach());
    Tensor drel = bias ? at::empty_like(rel.detach()) : Tensor();
    const int64_t nk = k.size(0);
    if (rows->plan.n_edges == 0) {
      variable_list out{dq.zero_(), dk.zero_(), dv.zero_()};
      if (bias) out.push_back(drel);
      return out;
    }
    const GraphPtr other = cols ? cols : column_view(*tables, 3, rows->plan.n_edges, nk, c.stream);
    const graphop_plan_t *pr = &rows->plan, *pt = &other->plan;
    c.workspace(pt->eid ? GRAPHOP_OP_ATTENTION_BWD_PAIRS : GRAPHOP_OP_ATTENTION_BWD, rows->plan.n_edges, std::max(s.n, nk), s.H,
                s.D, q);
    check_status(by_elem(elem, [&](auto* e) {
      using E = std::remove_pointer_t<decltype(e)>;
      if (bias)
        return internal_attention_bias_backward(
            e, pr, pt, (const void*)ptr<E>(q), (const void*)ptr<E>(k), (const void*)ptr<E>(v), (const void*)ptr<E>(rel),
            (const void*)ptr<E>(o), (const void*)lse.data_ptr(), (const void*)ptr<E>(g), scale, (void*)ptr<E>(dq),
            (void*)ptr<E>(dk), (void*)ptr<E>(dv), (void*)ptr<E>(drel), s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
      return attention_backward_planned(e, pr, pt, (const E*)ptr<E>(q), (const E*)ptr<E>(k), (const E*)ptr<E>(v),
                                        (const E*)ptr<E>(o), (const void*)lse.data_ptr(), (const E*)ptr<E>(g), scale,
                                        ptr<E>(dq), ptr<E>(dk), ptr<E>(dv), s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), bias ? "attention_bias_backward" : "attention_backward");
    variable_list out{dq, dk, dv};
    if (bias) out.push_back(drel);
    return out;
  }
};

Tensor attention_common(const GraphPtr& rows, const GraphPtr& cols, const TablesPtr& tables, Call& c, const Tensor& q,
                        const Tensor& k, const Tensor& v, const Tensor& rel, double scale) {
  const bool bias = rel.defined();
  const int elem = elem_of({&q, &k, &v});
  const NodeShape s = node_shape(q);
  const int64_t nk = k.size(0);
  Tensor o = at::empty_like(q.detach());
  Tensor lse = at::empty({s.n, s.H}, q.options().dtype(elem == 1 ? at::kDouble : at::kFloat));
  if (rows->plan.n_edges == 0) {
    o.zero_();
    lse.fill_(-std::numeric_limits<double>::infinity());
  } else {
    c.workspace(GRAPHOP_OP_ATTENTION_FWD, rows->plan.n_edges, std::max(s.n, nk), s.H, s.D, q);
    const graphop_plan_t* p = &rows->plan;
    check_status(by_elem(elem, [&](auto* e) {
      using E = std::remove_pointer_t<decltype(e)>;
      if (bias)
        return internal_attention_bias_forward(e, p, (const void*)ptr<E>(q), (const void*)ptr<E>(k), (const void*)ptr<E>(v),
                                               (const void*)ptr<E>(rel), scale, (void*)ptr<E>(o), (void*)lse.data_ptr(),
                                               s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
      return attention_forward_planned(e, p, (const E*)ptr<E>(q), (const E*)ptr<E>(k), (const E*)ptr<E>(v), scale, ptr<E>(o),
                                       (void*)lse.data_ptr(), s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), bias ? "attention_bias_forward" : "attention_forward");
  }
  auto save = [&](AttentionBackward& n) {
    n.tables = tables;
    n.rows = rows;
    n.cols = cols;
    n.scale = scale;
    n.bias = bias;
    for (const Tensor* t : {&q, &k, &v}) n.saved.emplace_back(*t, false);
    n.saved.emplace_back(o, true);
    n.saved.emplace_back(lse, false);
    if (bias) n.saved.emplace_back(rel, false);
  };
  if (bias) record<AttentionBackward>({q, k, v, rel}, o, save);
  else record<AttentionBackward>({q, k, v}, o, save);
  return o;
}

// A plan built by graphop.GraphPlan: the struct is copied, the memory it refers to kept alive.
struct PlanHandle {
  GraphPtr graph;
  PlanHandle(uintptr_t address, std::vector<Tensor> keep) : graph(std::make_shared<Graph>()) {
    graph->plan = *reinterpret_cast<const graphop_plan_t*>(address);
    graph->keep = std::move(keep);
      }
};
Tensor attention_planned(const PlanHandle& plan_r, const PlanHandle& plan_t, const Tensor& q, const Tensor& k,
                         const Tensor& v, double scale) {
  check_input(q, "q"); check_input(k, "k"); check_input(v, "v");
  Call c(q);
  return attention_common(plan_r.graph, plan_t.graph, nullptr, c, q, k, v, Tensor(), scale);
}
Tensor attention_bias(const Tensor& row, const Tensor& indptr, const Tensor& indices, const Tensor& col,
                      const Tensor& indptr_t, const Tensor& eid_t, const Tensor& indices_t, const Tensor& q,
                      const Tensor& k, const Tensor& v, const Tensor& rel, double scale) {
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(indices, "indices");
  check_input(q, "q"); check_input(k, "k"); check_input(v, "v"); check_input(rel, "rel");
  elem_of({&q, &k, &v, &rel});
  index_bytes_of({&row, &indptr, &indices});
  const NodeShape s = node_shape(q);
  check_chunks(row, indptr);
  const int64_t e = indices.size(0);
  if (rel.dim() != 2 || rel.size(0) != e || rel.size(1) != s.D) fail("rel must be (e, d)");
  auto tb = std::make_shared<Tables>(std::initializer_list<Tensor>{row, indptr, indices, col, indptr_t, eid_t, indices_t});
  Call c(q);
  GraphPtr rows = e > 0 ? view_of(row, indptr, Tensor(), indices, e, s.n, c.stream) : std::make_shared<Graph>();
  return attention_common(rows, nullptr, tb, c, q, k, v, rel, scale);
}

// ---- graph preparation: graphop.py's functions of the same names ---------------------------
Tensor scratch_of(size_t bytes, const Tensor& like, void** base) {
  Tensor t = at::empty({(int64_t)bytes + 256}, like.options().dtype(at::kByte));
  *base = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(t.data_ptr()) + 255) / 256 * 256);
  return t;
}
template <class I> I* as(const Tensor& t) { return t.defined() ? reinterpret_cast<I*>(t.data_ptr()) : nullptr; }

std::tuple<Tensor, Tensor> partition_csr(const Tensor& indptr, int64_t chunk_size) {
  const Tensor ip = indptr.contiguous();
  Call c(ip);
  const int64_t n = ip.numel() - 1;
  const bool wide = ip.scalar_type() == at::kLong;
  const size_t bytes = graphop_partition_csr_workspace_bytes(n);
  void* ws = nullptr;
  const Tensor scratch = scratch_of(bytes, ip, &ws);
  int64_t count = 0;
  check_status(wide ? graphop_partition_csr_count_i64(as<int64_t>(ip), n, chunk_size, ws, bytes, &count, raw(c.stream))
                    : graphop_partition_csr_count_i32(as<int32_t>(ip), n, chunk_size, ws, bytes, &count, raw(c.stream)),
               "partition_csr_count");
  Tensor row = at::empty({count}, ip.options().dtype(at::kLong)), ptr = at::empty({count + 1}, ip.options().dtype(at::kLong));
  check_status(wide ? graphop_partition_csr_fill_i64(as<int64_t>(ip), n, chunk_size, ws, count, as<int64_t>(row),
                                                     as<int64_t>(ptr), raw(c.stream))
                    : graphop_partition_csr_fill_i32(as<int32_t>(ip), n, chunk_size, ws, count, as<int64_t>(row),
                                                     as<int64_t>(ptr), raw(c.stream)),
               "partition_csr_fill");
  return {row, ptr};
}

std::tuple<Tensor, Tensor, Tensor> transpose_csr(const Tensor& indptr, const Tensor& indices, int64_t n_src) {
  const Tensor ip = indptr.contiguous(), idx = indices.contiguous();
  Call c(ip);
  const int64_t n_dst = ip.numel() - 1, e = idx.numel();
  const bool wide = ip.scalar_type() == at::kLong;
  const size_t bytes = graphop_transpose_csr_workspace_bytes(e, wide ? 8 : 4);
  void* ws = nullptr;
  const Tensor scratch = scratch_of(bytes, ip, &ws);
  Tensor ptr_t = at::empty({n_src + 1}, ip.options()), idx_t = at::empty_like(idx), eid_t = at::empty_like(idx);
  check_status(wide ? graphop_transpose_csr_i64(as<int64_t>(ip), as<int64_t>(idx), n_dst, n_src, e, as<int64_t>(ptr_t),
                                                as<int64_t>(idx_t), as<int64_t>(eid_t), ws, bytes, raw(c.stream))
                    : graphop_transpose_csr_i32(as<int32_t>(ip), as<int32_t>(idx), n_dst, n_src, e, as<int32_t>(ptr_t),
                                                as<int32_t>(idx_t), as<int32_t>(eid_t), ws, bytes, raw(c.stream)),
               "transpose_csr");
  return {ptr_t, idx_t, eid_t};
}

// Fills the graphop_plan_t at `address`; returns the memory it refers to.
Tensor plan_build(const Tensor& row, const Tensor& indptr, const c10::optional<Tensor>& eid_in,
                  const c10::optional<Tensor>& indices_in, int64_t n_edges, int64_t n_nodes, uintptr_t address) {
  const Tensor eid = eid_in.value_or(Tensor()), indices = indices_in.value_or(Tensor());
  const int ib = index_bytes_of({&row, &indptr, &eid, &indices});
  Call c(row);
  const size_t bytes = graphop_plan_bytes(row.size(0), n_edges, n_nodes, ib);
  void* base = nullptr;
  Tensor memory = scratch_of(bytes, row, &base);
  auto* plan = reinterpret_cast<graphop_plan_t*>(address);
  check_status(ib == 8 ? graphop_plan_build_i64(as<int64_t>(row), as<int64_t>(indptr), as<int64_t>(eid),
                                                as<int64_t>(indices), row.size(0), n_edges, n_nodes, base, bytes, plan,
                                                raw(c.stream))
                       : graphop_plan_build_i32(as<int32_t>(row), as<int32_t>(indptr), as<int32_t>(eid),
                                                as<int32_t>(indices), row.size(0), n_edges, n_nodes, base, bytes, plan,
                                                raw(c.stream)),
               "plan_build");
  return memory;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "the autograd Functions of custom_op_benchmark_b200.wrapper and the graph preparation in native code";
  using free_gil = py::call_guard<py::gil_scoped_release>;
  py::class_<PlanHandle>(m, "PlanHandle").def(py::init<uintptr_t, std::vector<Tensor>>());
  m.def("sparse_softmax", &sparse_softmax, free_gil());
  m.def("maskedmm_csr", &maskedmm_csr, free_gil());
  m.def("node_mul_edge", &node_mul_edge, free_gil());
  m.def("vector_spmm", &vector_spmm, free_gil());
  m.def("attention_planned", &attention_planned, free_gil());
  m.def("attention_bias", &attention_bias, free_gil());
  m.def("partition_csr", &partition_csr, free_gil());
  m.def("transpose_csr", &transpose_csr, free_gil());
  m.def("plan_build", &plan_build, free_gil());
}
