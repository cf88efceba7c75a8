/* Entry points of the library for its own torch binding (binding/graphop_native.cpp); not part of the C ABI. */
#ifndef GRAPHOP_INTERNAL_H
#define GRAPHOP_INTERNAL_H
#include "../../include/graphop_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* A view is a plan without the shape analysis: owner table, 32-bit index copies and work tiles of a chunk table, built
 * without waiting for the device.  n_nodes < 0: no work tiles (the softmax has no use for them).  `clear` (may be null):
 * an edge output set to zero if some position belongs to no chunk. */
size_t graphop_internal_view_bytes(int64_t n_edges, int64_t n_nodes, int index_bytes);
int graphop_internal_view_build(const void* row, const void* indptr, const void* eid, const void* indices,
                                int index_bytes, int64_t n_chunks, int64_t n_edges, int64_t n_nodes, void* clear,
                                size_t clear_bytes, void* memory, size_t memory_bytes, graphop_plan_t* plan, graphop_stream_t stream);

#define GRAPHOP_DECLARE_INTERNAL(SUF)                                                                                \
  int graphop_internal_attention_bias_forward_##SUF(                                                                 \
      const graphop_plan_t* plan, const void* q, const void* k, const void* v, const void* rel, double scale,        \
      void* o, void* lse, int64_t n_dst, int64_t n_src, int H, int D, void* ws, size_t wsb,                          \
      graphop_stream_t stream);                                                                                      \
  int graphop_internal_attention_bias_backward_##SUF(                                                                \
      const graphop_plan_t* plan_r, const graphop_plan_t* plan_t, const void* q, const void* k, const void* v,       \
      const void* rel, const void* o, const void* lse, const void* d_o, double scale, void* dq, void* dk, void* dv,  \
      void* d_rel, int64_t n_dst, int64_t n_src, int H, int D, void* ws, size_t wsb, graphop_stream_t stream);
GRAPHOP_DECLARE_INTERNAL(f32)
GRAPHOP_DECLARE_INTERNAL(f64)
GRAPHOP_DECLARE_INTERNAL(bf16)

#ifdef __cplusplus
}
#endif
#endif
