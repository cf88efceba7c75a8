// The autograd Functions of wrapper.py in native code: what `apply` of each class runs.
//
// A graph-attention layer on a small graph is a handful of kernels of a few microseconds; the same Functions written in
// Python (argument checks, ctypes calls, torch.autograd.Function's Python forward and backward) cost 40 to 60 us of
// host time per op and direction, several times the kernels.  Here an op is one pybind call, a C++ autograd node and the
// C ABI's planned entry point; the backward runs on autograd's thread without taking the interpreter lock.
//
// The chunk-table signatures (row, indptr, eid, indices) of the reference carry the graph on every call.  The owner
// table, 32-bit index copies and work tiles that the kernels make from them are workspace of each direction: kept from
// the forward to the backward (one launch less for MaskedMMCSR and GraphAttentionBias) they held 12 to 18 bytes per edge,
// and as much again afterwards, as long as the output lived.
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

#include "../../../include/graphop_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// Calls that the code below does not carry are left to torch.autograd.Function (an empty result; wrapper.py goes on there):
// a trace being recorded, a transform of torch.func or a dispatch mode at work, a tangent of forward-mode differentiation,
// tensors that wrap others.
using Result = c10::optional<Tensor>;
bool left_to_python(std::initializer_list<const Tensor*> ts) {
  using c10::DispatchKey;
  constexpr c10::DispatchKeySet modes({DispatchKey::Tracer, DispatchKey::Python, DispatchKey::FuncTorchDynamicLayerFrontMode,
                                       DispatchKey::FuncTorchDynamicLayerBackMode});
  if (c10::impl::tls_local_dispatch_key_set().included_.has_any(modes)) return true;
  for (const Tensor* t : ts)
    if (t->defined() && (t->key_set().has(DispatchKey::Python) || !t->has_storage() || t->_fw_grad(0).defined())) return true;
  return false;
}

// ------------------------------------------------------------------------------------------
// checks: the texts and exception types of graphop.py
// ------------------------------------------------------------------------------------------
[[noreturn]] void fail(const std::string& text) { throw std::runtime_error(text); }

void check_input(const Tensor& t, const char* name) {
  if (!t.defined() || !t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor");
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
// calling the C ABI
// ------------------------------------------------------------------------------------------
void check_chunks(const Tensor& row, const Tensor& indptr) {
  if (indptr.size(0) != row.size(0) + 1) fail("indptr must hold row.size(0) + 1 entries");
}

// What one op call needs besides its tensors: device guard, stream, workspace.
struct Call {
  c10::cuda::CUDAGuard guard;
  cudaStream_t stream;
  Tensor scratch;
  void* ws = nullptr;
  size_t bytes = 0;
  explicit Call(const Tensor& on) : guard(on.device()), stream(at::cuda::getCurrentCUDAStream(on.get_device())) {}
  void workspace(int op, int64_t n_edges, int64_t n_nodes, int H, int D, const Tensor& like, int index_bytes = 4) {
    bytes = graphop_workspace_bytes(op, n_edges, n_nodes, H, D, (int)like.element_size(), index_bytes);
    scratch = at::empty({(int64_t)bytes + 256}, like.options().dtype(at::kByte));
    ws = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(scratch.data_ptr()) + 255) / 256 * 256);
  }
};

// a tensor's storage as the element type the entry point wants; null for an undefined one
template <typename E> E* ptr(const Tensor& t) { return t.defined() ? reinterpret_cast<E*>(t.data_ptr()) : nullptr; }

// The owner nodes of a chunk table.  One without chunks is a table like any other (every edge output is zero), but has no
// memory, and the entry points refuse a null pointer: nothing is read through this one.
template <typename I> const I* owners(const Tensor& row, const Tensor& indptr) {
  return row.size(0) ? ptr<I>(row) : ptr<I>(indptr);
}

// An argument that only the backward reads: a call without one may leave it out.
using Later = c10::optional<Tensor>;
Tensor given(const Later& t) { return t.value_or(Tensor()); }

// f is called with a null pointer of the element type
template <class F> auto by_elem(int elem, F&& f) {
  if (elem == 0) return f((float*)nullptr);
  if (elem == 1) return f((double*)nullptr);
  return f((uint16_t*)nullptr);
}
// and of the index type
template <class F> auto by_types(int elem, int index_bytes, F&& f) {
  return by_elem(elem, [&](auto* e) { return index_bytes == 8 ? f(e, (int64_t*)nullptr) : f(e, (int32_t*)nullptr); });
}

// one overload set per op over the three element types (and the two index types)
#define GRAPHOP_OVERLOADS(op)                                                                                        \
  template <class... X> int op(float*, int32_t*, X... x) { return graphop_##op##_f32_i32(x...); }                    \
  template <class... X> int op(float*, int64_t*, X... x) { return graphop_##op##_f32_i64(x...); }                    \
  template <class... X> int op(double*, int32_t*, X... x) { return graphop_##op##_f64_i32(x...); }                   \
  template <class... X> int op(double*, int64_t*, X... x) { return graphop_##op##_f64_i64(x...); }                   \
  template <class... X> int op(uint16_t*, int32_t*, X... x) { return graphop_##op##_bf16_i32(x...); }                \
  template <class... X> int op(uint16_t*, int64_t*, X... x) { return graphop_##op##_bf16_i64(x...); }
GRAPHOP_OVERLOADS(maskedmm_csr_forward)
GRAPHOP_OVERLOADS(maskedmm_csr_backward)
GRAPHOP_OVERLOADS(node_mul_edge_forward)
GRAPHOP_OVERLOADS(node_mul_edge_backward)
GRAPHOP_OVERLOADS(sparse_softmax_forward)
GRAPHOP_OVERLOADS(sparse_softmax_backward)
GRAPHOP_OVERLOADS(vector_spmm_forward)
GRAPHOP_OVERLOADS(vector_spmm_backward)
GRAPHOP_OVERLOADS(attention_bias_forward)
GRAPHOP_OVERLOADS(attention_bias_backward)
#undef GRAPHOP_OVERLOADS
#define GRAPHOP_OVERLOADS(op)                                                                                        \
  template <class... X> int op(float*, X... x) { return graphop_##op##_f32(x...); }                                  \
  template <class... X> int op(double*, X... x) { return graphop_##op##_f64(x...); }                                 \
  template <class... X> int op(uint16_t*, X... x) { return graphop_##op##_bf16(x...); }
GRAPHOP_OVERLOADS(attention_forward_planned)
GRAPHOP_OVERLOADS(attention_backward_planned)
#undef GRAPHOP_OVERLOADS

// ------------------------------------------------------------------------------------------
// autograd nodes
// ------------------------------------------------------------------------------------------
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

// What a node of these ops keeps from its forward: the tensors of the call, index tensors included, as saved variables
// (so that hooks see them, in-place changes are found and a backward that does not retain the graph lets go of them), and
// nothing else: the tables that the kernels make of a chunk table are workspace of either direction.  Two threads may run
// the backward of one graph: the saved tensors are read and released under the node's mutex.
struct GraphNode : Node {
  void save(const Tensor& t, bool is_output = false) {
    // an index tensor made in inference mode has no version to check: kept as it is
    const bool plain = t.defined() && t.is_inference() && !at::isFloatingType(t.scalar_type());
    saved.emplace_back(plain ? Tensor() : t, is_output);
    unversioned.push_back(plain ? t : Tensor());
  }
  void save_all(std::initializer_list<Tensor> ts) {
    saved.reserve(ts.size() + 2);
    unversioned.reserve(ts.size() + 2);
    for (const Tensor& t : ts) save(t);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    for (SavedVariable& s : saved) s.reset_data();
    for (Tensor& t : unversioned) t = Tensor();
  }
  std::vector<Tensor> unpack_saved() {
    const std::shared_ptr<Node> self = shared_from_this();   // for a saved output
    std::lock_guard<std::mutex> hold(mutex_);
    std::vector<Tensor> t;
    t.reserve(saved.size());
    for (size_t i = 0; i < saved.size(); ++i) t.push_back(unversioned[i].defined() ? unversioned[i] : saved[i].unpack(self));
    return t;
  }

 private:
  std::vector<SavedVariable> saved;
  std::vector<Tensor> unversioned;
};

// The column side's arguments, which only the backward reads: wrong ones are reported there, as they always were.  t: the
// call's index tensors, the four of the column side from t[at]; n: how many there are.
int check_columns(const std::vector<Tensor>& t, size_t at, size_t n, const char* const (&names)[4]) {
  for (int i = 0; i < 4; ++i) check_input(t[at + i], names[i]);
  std::vector<const Tensor*> all;   // both orientations: one call has one index type
  for (size_t i = 0; i < n; ++i) all.push_back(&t[i]);
  const int ib = index_bytes_of(all);
  check_chunks(t[at], t[at + 1]);
  return ib;
}

// ---- SparseSoftmax (wrapper.py:8-18) ------------------------------------------------------
struct SparseSoftmaxBackward : GraphNode {
  std::string name() const override { return "SparseSoftmaxBackward"; }
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor()};
    const std::vector<Tensor> t = unpack_saved();   // row, indptr, eid, y
    const Tensor &y = t[3], dy = upstream(grads, "dy");
    const int elem = elem_of({&y, &dy}), ib = index_bytes_of({&t[0], &t[1], &t[2]}), H = edge_heads(dy);
    Call c(y);
    Tensor dx = at::empty_like(dy);
    const int64_t e = t[2].size(0), chunks = t[0].size(0);
    if (e == 0) return {dx};
    c.workspace(GRAPHOP_OP_SOFTMAX_BWD, e, 0, H, 1, y, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return sparse_softmax_backward(k, i, owners<I>(t[0], t[1]), (const I*)ptr<I>(t[1]), (const I*)ptr<I>(t[2]),
                                     (const E*)ptr<E>(y), (const E*)ptr<E>(dy), ptr<E>(dx), chunks, e, (int64_t)0, H, c.ws,
                                     c.bytes, raw(c.stream));
    }), "sparse_softmax_backward");
    return {dx};
  }
};
Result sparse_softmax(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& x) {
  if (left_to_python({&row, &indptr, &eid, &x})) return c10::nullopt;
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(eid, "eid"); check_input(x, "x");
  const int elem = elem_of({&x}), H = edge_heads(x), ib = index_bytes_of({&row, &indptr, &eid});
  check_chunks(row, indptr);
  Call c(x);
  const int64_t e = eid.size(0), chunks = row.size(0);
  Tensor y = at::empty_like(x.detach());
  if (e > 0) {
    c.workspace(GRAPHOP_OP_SOFTMAX_FWD, e, 0, H, 1, x, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return sparse_softmax_forward(k, i, owners<I>(row, indptr), (const I*)ptr<I>(indptr), (const I*)ptr<I>(eid),
                                    (const E*)ptr<E>(x), ptr<E>(y), chunks, e, (int64_t)0, H, c.ws, c.bytes, raw(c.stream));
    }), "sparse_softmax_forward");
  }
  record<SparseSoftmaxBackward>({x}, y, [&](SparseSoftmaxBackward& n) {
    n.save_all({row, indptr, eid});
    n.save(y, true);
  });
  return y;
}

// ---- MaskedMMCSR (wrapper.py:20-30) -------------------------------------------------------
struct MaskedMMBackward : GraphNode {
  std::string name() const override { return "MaskedMMCSRBackward"; }
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const std::vector<Tensor> t = unpack_saved();   // row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B
    const Tensor &A = t[8], &B = t[9], dy = upstream(grads, "dy");
    const int elem = elem_of({&A, &B, &dy});
    const int ib = check_columns(t, 4, 8, {"col", "indptr_c", "eid_c", "indices_c"});
    const NodeShape s = node_shape(A);
    Call c(A);
    const int64_t e = t[2].size(0), nb = B.size(0), chunks = t[0].size(0), chunks_c = t[4].size(0);
    Tensor dA = at::empty_like(A.detach()), dB = at::empty_like(B.detach());
    if (e == 0) return {dA.zero_(), dB.zero_()};
    c.workspace(GRAPHOP_OP_MASKEDMM_BWD, e, std::max(s.n, nb), s.H, s.D, A, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      const auto in = [&](int at) { return (const I*)ptr<I>(t[at]); };
      return maskedmm_csr_backward(k, i, owners<I>(t[0], t[1]), in(1), in(2), in(3), chunks, owners<I>(t[4], t[5]), in(5), in(6), in(7), chunks_c,
                                   (const E*)ptr<E>(A), (const E*)ptr<E>(B), (const E*)ptr<E>(dy), ptr<E>(dA), ptr<E>(dB), e,
                                   s.n, nb, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "maskedmm_csr_backward");
    return {dA, dB};
  }
};
Result maskedmm_csr(const Tensor& row, const Tensor& indptr_r, const Tensor& eid_r, const Tensor& indices_r,
                    const Later& col_in, const Later& indptr_c_in, const Later& eid_c_in, const Later& indices_c_in,
                    const Tensor& A, const Tensor& B) {
  const Tensor col = given(col_in), indptr_c = given(indptr_c_in), eid_c = given(eid_c_in), indices_c = given(indices_c_in);
  if (left_to_python({&row, &indptr_r, &eid_r, &indices_r, &col, &indptr_c, &eid_c, &indices_c, &A, &B})) return c10::nullopt;
  check_input(row, "row"); check_input(indptr_r, "indptr"); check_input(eid_r, "eid"); check_input(indices_r, "indices");
  check_input(A, "A"); check_input(B, "B");
  const int elem = elem_of({&A, &B}), ib = index_bytes_of({&row, &indptr_r, &eid_r, &indices_r});
  const NodeShape s = node_shape(A);
  check_chunks(row, indptr_r);
  Call c(A);
  const int64_t e = eid_r.size(0), nb = B.size(0), chunks = row.size(0);
  Tensor y = edge_out(A, e, s.H);
  if (e > 0) {
    c.workspace(GRAPHOP_OP_MASKEDMM_FWD, e, std::max(s.n, nb), s.H, s.D, A, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return maskedmm_csr_forward(k, i, owners<I>(row, indptr_r), (const I*)ptr<I>(indptr_r), (const I*)ptr<I>(eid_r),
                                  (const I*)ptr<I>(indices_r), (const E*)ptr<E>(A), (const E*)ptr<E>(B), ptr<E>(y), chunks, e,
                                  s.n, nb, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "maskedmm_csr_forward");
  }
  record<MaskedMMBackward>({A, B}, y, [&](MaskedMMBackward& n) {
    n.save_all({row, indptr_r, eid_r, indices_r, col, indptr_c, eid_c, indices_c, A, B});
  });
  return y;
}

// ---- NodeMulEdge (wrapper.py:32-42) -------------------------------------------------------
struct NodeMulEdgeBackward : GraphNode {
  std::string name() const override { return "NodeMulEdgeBackward"; }
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const std::vector<Tensor> t = unpack_saved();   // row, indptr, eid, A, B
    const Tensor &A = t[3], &B = t[4], dy = upstream(grads, "dy");
    const int elem = elem_of({&A, &B, &dy}), ib = index_bytes_of({&t[0], &t[1], &t[2]});
    const NodeShape s = node_shape(A);
    Call c(A);
    const int64_t e = t[2].size(0), chunks = t[0].size(0);
    Tensor dA = at::empty_like(A.detach()), dB = at::empty_like(B.detach());
    if (e == 0) return {dA.zero_(), dB};
    c.workspace(GRAPHOP_OP_NODE_MUL_EDGE_BWD, e, s.n, s.H, s.D, A, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return node_mul_edge_backward(k, i, owners<I>(t[0], t[1]), (const I*)ptr<I>(t[1]), (const I*)ptr<I>(t[2]),
                                    (const E*)ptr<E>(A), (const E*)ptr<E>(B), (const E*)ptr<E>(dy), ptr<E>(dA), ptr<E>(dB),
                                    chunks, e, s.n, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "node_mul_edge_backward");
    return {dA, dB};
  }
};
Result node_mul_edge(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& A, const Tensor& B) {
  if (left_to_python({&row, &indptr, &eid, &A, &B})) return c10::nullopt;
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(eid, "eid"); check_input(A, "A"); check_input(B, "B");
  const int elem = elem_of({&A, &B}), ib = index_bytes_of({&row, &indptr, &eid});
  const NodeShape s = node_shape(A);
  check_chunks(row, indptr);
  Call c(A);
  const int64_t e = eid.size(0), chunks = row.size(0);
  Tensor y = edge_out(A, e, s.H);
  if (e > 0) {
    c.workspace(GRAPHOP_OP_NODE_MUL_EDGE_FWD, e, s.n, s.H, s.D, A, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return node_mul_edge_forward(k, i, owners<I>(row, indptr), (const I*)ptr<I>(indptr), (const I*)ptr<I>(eid),
                                   (const E*)ptr<E>(A), (const E*)ptr<E>(B), ptr<E>(y), chunks, e, s.n, s.H, s.D, c.ws, c.bytes,
                                   raw(c.stream));
    }), "node_mul_edge_forward");
  }
  record<NodeMulEdgeBackward>({A, B}, y, [&](NodeMulEdgeBackward& n) { n.save_all({row, indptr, eid, A, B}); });
  return y;
}

// ---- VectorSPMM (wrapper.py:44-55) --------------------------------------------------------
struct VectorSPMMBackward : GraphNode {
  std::string name() const override { return "VectorSPMMBackward"; }
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const std::vector<Tensor> t = unpack_saved();   // row, indptr, eid, indices, col, indptr_t, eid_t, indices_t, w, x
    const Tensor &w = t[8], &x = t[9], dy = upstream(grads, "dy");
    const int elem = elem_of({&w, &dy, &x});
    const int ib = check_columns(t, 4, 8, {"col", "indptr_t", "eid_t", "indices_t"});
    const NodeShape s = node_shape(x);
    Call c(x);
    const int64_t e = t[2].size(0), n_dst = dy.size(0), chunks = t[0].size(0), chunks_t = t[4].size(0);
    Tensor dw = at::empty_like(w.detach()), dx = at::empty_like(x.detach());
    if (e == 0) return {dw, dx.zero_()};
    c.workspace(GRAPHOP_OP_SPMM_BWD, e, std::max(n_dst, s.n), s.H, s.D, x, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      const auto in = [&](int at) { return (const I*)ptr<I>(t[at]); };
      return vector_spmm_backward(k, i, owners<I>(t[0], t[1]), in(1), in(2), in(3), chunks, owners<I>(t[4], t[5]), in(5), in(6), in(7), chunks_t,
                                  (const E*)ptr<E>(w), (const E*)ptr<E>(dy), (const E*)ptr<E>(x), ptr<E>(dw), ptr<E>(dx), e,
                                  n_dst, s.n, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "vector_spmm_backward");
    return {dw, dx};
  }
};
Result vector_spmm(const Tensor& row, const Tensor& indptr, const Tensor& eid, const Tensor& indices, const Later& col_in,
                   const Later& indptr_t_in, const Later& eid_t_in, const Later& indices_t_in, const Tensor& w,
                   const Tensor& x) {
  const Tensor col = given(col_in), indptr_t = given(indptr_t_in), eid_t = given(eid_t_in), indices_t = given(indices_t_in);
  if (left_to_python({&row, &indptr, &eid, &indices, &col, &indptr_t, &eid_t, &indices_t, &w, &x})) return c10::nullopt;
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(eid, "eid"); check_input(indices, "indices");
  check_input(w, "edata"); check_input(x, "x");
  const int elem = elem_of({&w, &x}), ib = index_bytes_of({&row, &indptr, &eid, &indices});
  const NodeShape s = node_shape(x);
  if (edge_heads(w) != s.H) fail("edata and x disagree on the number of heads");
  check_chunks(row, indptr);
  Call c(x);
  const int64_t e = eid.size(0), chunks = row.size(0);
  Tensor y = at::empty(x.sizes(), x.options());
  if (e == 0) {
    y.zero_();
  } else {
    c.workspace(GRAPHOP_OP_SPMM_FWD, e, s.n, s.H, s.D, x, ib);
    check_status(by_types(elem, ib, [&](auto* k, auto* i) {
      using E = std::remove_pointer_t<decltype(k)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return vector_spmm_forward(k, i, owners<I>(row, indptr), (const I*)ptr<I>(indptr), (const I*)ptr<I>(eid),
                                 (const I*)ptr<I>(indices), (const E*)ptr<E>(w), (const E*)ptr<E>(x), ptr<E>(y), chunks, e, s.n,
                                 s.n, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "vector_spmm_forward");
  }
  record<VectorSPMMBackward>({w, x}, y, [&](VectorSPMMBackward& n) {
    n.save_all({row, indptr, eid, indices, col, indptr_t, eid_t, indices_t, w, x});
  });
  return y;
}

// ---- fused attention on plans --------------------------------------------------------------
// A plan built by graphop.GraphPlan: the struct is copied, the memory it refers to kept alive.
struct Graph {
  graphop_plan_t plan{};
  std::vector<Tensor> keep;
};
using GraphPtr = std::shared_ptr<Graph>;
struct PlanHandle {
  GraphPtr graph;
  PlanHandle(uintptr_t address, std::vector<Tensor> keep) : graph(std::make_shared<Graph>()) {
    graph->plan = *reinterpret_cast<const graphop_plan_t*>(address);
    graph->keep = std::move(keep);
  }
};
Tensor lse_like(const Tensor& q, const NodeShape& s, int elem) {
  return at::empty({s.n, s.H}, q.options().dtype(elem == 1 ? at::kDouble : at::kFloat));
}
void no_edges(Tensor& o, Tensor& lse) {
  o.zero_();
  lse.fill_(-std::numeric_limits<double>::infinity());
}

struct AttentionBackward : GraphNode {
  std::string name() const override { return "GraphAttentionPlannedBackward"; }
  GraphPtr rows, cols;
  double scale = 1.0;
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return variable_list(3);
    const std::vector<Tensor> t = unpack_saved();   // q, k, v, lse, o
    const Tensor &q = t[0], &k = t[1], &v = t[2], &lse = t[3], &o = t[4], g = upstream(grads, "d_o");
    const int elem = elem_of({&q, &k, &v, &o, &g});
    const NodeShape s = node_shape(q);
    Call c(q);
    Tensor dq = at::empty_like(q.detach()), dk = at::empty_like(k.detach()), dv = at::empty_like(v.detach());
    const int64_t nk = k.size(0);
    const graphop_plan_t *pr = &rows->plan, *pt = &cols->plan;
    if (pr->n_edges == 0) return {dq.zero_(), dk.zero_(), dv.zero_()};
    c.workspace(pt->eid ? GRAPHOP_OP_ATTENTION_BWD_PAIRS : GRAPHOP_OP_ATTENTION_BWD, pr->n_edges, std::max(s.n, nk), s.H, s.D, q);
    check_status(by_elem(elem, [&](auto* e) {
      using E = std::remove_pointer_t<decltype(e)>;
      return attention_backward_planned(e, pr, pt, (const E*)ptr<E>(q), (const E*)ptr<E>(k), (const E*)ptr<E>(v),
                                        (const E*)ptr<E>(o), (const void*)lse.data_ptr(), (const E*)ptr<E>(g), scale,
                                        ptr<E>(dq), ptr<E>(dk), ptr<E>(dv), s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "attention_backward");
    return {dq, dk, dv};
  }
};
Result attention_planned(const PlanHandle& plan_r, const PlanHandle& plan_t, const Tensor& q, const Tensor& k,
                         const Tensor& v, double scale) {
  if (left_to_python({&q, &k, &v})) return c10::nullopt;
  check_input(q, "q"); check_input(k, "k"); check_input(v, "v");
  const int elem = elem_of({&q, &k, &v});
  const NodeShape s = node_shape(q);
  const int64_t nk = k.size(0);
  Call c(q);
  Tensor o = at::empty_like(q.detach()), lse = lse_like(q, s, elem);
  const graphop_plan_t* p = &plan_r.graph->plan;
  if (p->n_edges == 0) {
    no_edges(o, lse);
  } else {
    c.workspace(GRAPHOP_OP_ATTENTION_FWD, p->n_edges, std::max(s.n, nk), s.H, s.D, q);
    check_status(by_elem(elem, [&](auto* e) {
      using E = std::remove_pointer_t<decltype(e)>;
      return attention_forward_planned(e, p, (const E*)ptr<E>(q), (const E*)ptr<E>(k), (const E*)ptr<E>(v), scale, ptr<E>(o),
                                       (void*)lse.data_ptr(), s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "attention_forward");
  }
  record<AttentionBackward>({q, k, v}, o, [&](AttentionBackward& n) {
    n.rows = plan_r.graph;
    n.cols = plan_t.graph;
    n.scale = scale;
    n.save_all({q, k, v, lse});
    n.save(o, true);
  });
  return o;
}

// ---- fused attention with an edge term on chunk tables --------------------------------------
struct AttentionBiasBackward : GraphNode {
  std::string name() const override { return "GraphAttentionBiasBackward"; }
  double scale = 1.0;
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return variable_list(4);
    // row, indptr, indices, col, indptr_t, eid_t, indices_t, q, k, v, rel, lse, o
    const std::vector<Tensor> t = unpack_saved();
    const Tensor &q = t[7], &k = t[8], &v = t[9], &rel = t[10], &lse = t[11], &o = t[12], g = upstream(grads, "d_o");
    const int ib = check_columns(t, 3, 7, {"col", "indptr_t", "eid_t", "indices_t"});
    const int elem = elem_of({&q, &k, &v, &rel, &o, &g});
    const NodeShape s = node_shape(q);
    Call c(q);
    const int64_t e = t[2].size(0), nk = k.size(0), chunks = t[0].size(0), chunks_t = t[3].size(0);
    Tensor dq = at::empty_like(q.detach()), dk = at::empty_like(k.detach()), dv = at::empty_like(v.detach()),
           drel = at::empty_like(rel.detach());
    if (e == 0) return {dq.zero_(), dk.zero_(), dv.zero_(), drel};
    c.workspace(GRAPHOP_OP_ATTENTION_BWD_PAIRS, e, std::max(s.n, nk), s.H, s.D, q, ib);
    check_status(by_types(elem, ib, [&](auto* x, auto* i) {
      using E = std::remove_pointer_t<decltype(x)>;
      using I = std::remove_pointer_t<decltype(i)>;
      const auto in = [&](int at) { return (const I*)ptr<I>(t[at]); };
      return attention_bias_backward(x, i, owners<I>(t[0], t[1]), in(1), in(2), chunks, owners<I>(t[3], t[4]), in(4), in(5), in(6), chunks_t,
                                     (const E*)ptr<E>(q), (const E*)ptr<E>(k), (const E*)ptr<E>(v), (const E*)ptr<E>(rel),
                                     (const E*)ptr<E>(o), (const void*)lse.data_ptr(), (const E*)ptr<E>(g), scale, ptr<E>(dq),
                                     ptr<E>(dk), ptr<E>(dv), ptr<E>(drel), e, s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "attention_bias_backward");
    return {dq, dk, dv, drel};
  }
};
Result attention_bias(const Tensor& row, const Tensor& indptr, const Tensor& indices, const Later& col_in,
                      const Later& indptr_t_in, const Later& eid_t_in, const Later& indices_t_in, const Tensor& q,
                      const Tensor& k, const Tensor& v, const Tensor& rel, double scale) {
  const Tensor col = given(col_in), indptr_t = given(indptr_t_in), eid_t = given(eid_t_in), indices_t = given(indices_t_in);
  if (left_to_python({&row, &indptr, &indices, &col, &indptr_t, &eid_t, &indices_t, &q, &k, &v, &rel})) return c10::nullopt;
  check_input(row, "row"); check_input(indptr, "indptr"); check_input(indices, "indices");
  check_input(q, "q"); check_input(k, "k"); check_input(v, "v"); check_input(rel, "rel");
  const int elem = elem_of({&q, &k, &v, &rel}), ib = index_bytes_of({&row, &indptr, &indices});
  const NodeShape s = node_shape(q);
  check_chunks(row, indptr);
  const int64_t e = indices.size(0), nk = k.size(0), chunks = row.size(0);
  if (rel.dim() != 2 || rel.size(0) != e || rel.size(1) != s.D) fail("rel must be (e, d)");
  Call c(q);
  Tensor o = at::empty_like(q.detach()), lse = lse_like(q, s, elem);
  if (e == 0) {
    no_edges(o, lse);
  } else {
    c.workspace(GRAPHOP_OP_ATTENTION_FWD, e, std::max(s.n, nk), s.H, s.D, q, ib);
    check_status(by_types(elem, ib, [&](auto* x, auto* i) {
      using E = std::remove_pointer_t<decltype(x)>;
      using I = std::remove_pointer_t<decltype(i)>;
      return attention_bias_forward(x, i, owners<I>(row, indptr), (const I*)ptr<I>(indptr), (const I*)ptr<I>(indices), chunks,
                                    (const E*)ptr<E>(q), (const E*)ptr<E>(k), (const E*)ptr<E>(v), (const E*)ptr<E>(rel), scale,
                                    ptr<E>(o), (void*)lse.data_ptr(), e, s.n, nk, s.H, s.D, c.ws, c.bytes, raw(c.stream));
    }), "attention_bias_forward");
  }
  record<AttentionBiasBackward>({q, k, v, rel}, o, [&](AttentionBiasBackward& n) {
    n.scale = scale;
    n.save_all({row, indptr, indices, col, indptr_t, eid_t, indices_t, q, k, v, rel, lse});
    n.save(o, true);
  });
  return o;
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
