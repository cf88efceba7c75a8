// Host side of the C ABI: argument checks, workspace carving, kernel selection and the
// launch sequences.  Everything here enqueues on the caller's stream and never synchronises.
#pragma once
#include <atomic>
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/graphop_b200.h"
#include "gk_common.cuh"
#include "gk_group.cuh"
#include "gk_ops.cuh"
#include "gk_softmax.cuh"

namespace gk {

inline thread_local int g_last_cuda_error = 0;

#define GK_CUDA(expr)                                   \
  do {                                                  \
    cudaError_t err__ = (expr);                         \
    if (err__ != cudaSuccess) {                         \
      gk::g_last_cuda_error = (int)err__;                 \
      return GRAPHOP_ERR_CUDA;                          \
    }                                                   \
  } while (0)
#define GK_LAUNCH_CHECK() GK_CUDA(cudaGetLastError())

// Every kernel launch of the library goes through GK_LAUNCHED(name), which checks the launch.  The benchmark's
// instrumented twin of the library (compiled with -DGK_BENCH_HOOKS, see csrc/bench/) also counts the launch and,
// while a profile is open, records a CUDA event behind the kernel on the caller's stream, so that the time
// between two consecutive events is the device time of the later kernel.  The product library has none of it.
#ifdef GK_BENCH_HOOKS
struct Profiler {
  std::mutex lock;   // autograd runs the backward ops on another host thread
  bool enabled = false;
  long long launches = 0;
  std::vector<std::pair<const char*, cudaEvent_t>> marks;
};
inline Profiler& profiler() {
  static Profiler p;
  return p;
}
inline void mark(const char* name, cudaStream_t st) {
  Profiler& p = profiler();
  std::lock_guard<std::mutex> hold(p.lock);
  ++p.launches;
  if (p.enabled) {
    cudaEvent_t e;
    if (cudaEventCreate(&e) == cudaSuccess) {
      cudaEventRecord(e, st);
      p.marks.emplace_back(name, e);
    }
  }
}
#define GK_LAUNCHED(name)  \
  do {                     \
    GK_LAUNCH_CHECK();     \
    gk::mark(name, st);    \
  } while (0)
#else
#define GK_LAUNCHED(name) GK_LAUNCH_CHECK()
#endif
#define GK_TRY(expr)                    \
  do {                                  \
    int rc__ = (expr);                  \
    if (rc__ != GRAPHOP_OK) return rc__; \
  } while (0)

constexpr size_t kAlign = 256;
inline size_t align_up(size_t v) { return (v + kAlign - 1) / kAlign * kAlign; }

// Bump allocator over the caller's workspace.  With base == nullptr it only measures.
struct Arena {
  char* base;
  size_t cap, used = 0;
  bool overflow = false;
  Arena(void* b, size_t c) : base((char*)b), cap(c) {}
  void* take(size_t bytes) {
    const size_t at = used;
    used += align_up(bytes ? bytes : 1);
    if (!base) return nullptr;
    if (used > cap) { overflow = true; return nullptr; }
    return base + at;
  }
};

// ---------------------------------------------------------------------------------------
// tiling
// ---------------------------------------------------------------------------------------
constexpr int kMaxLevels = 12;
// Tile of walk_kernel's carry levels: wider ones save a launch but run slower, a warp walks its slots one after the other
// (attention on 4096 nodes of 16 edges, when these levels were its: 0.27 -> 0.40 ms with 256).
constexpr int kCarryTile = 32;

// Positions per warp at level 0 of the register-fetch walker.
inline int pick_tile(long long n_edges) {
  long long t = 32;
  while (t < 256 && n_edges / t > 16384) t <<= 1;
  return (int)t;
}

// Cost of a work tile of the gathering walker (see cut_tiles: positions and nodes) and the number of tiles.  Large
// graphs get tiles of 256, which keeps carries and the fixed part of a tile a fraction of the work; smaller ones get the
// smallest tile, down to 32, that makes no more than kTilesWanted: enough for every SM to have several rounds of warps
// (attention step, 4 heads x 32 fp32: R-MAT 15 with tiles of 256 / 128 / 64 / 32 355 / 274 / 265 / 256 us, R-MAT 18
// 1480 / 1437 / 1462 / 1545 us, R-MAT 21 12.97 / 12.95 / 13.00 / 14.06 ms).
constexpr long long kTilesWanted = 49152;
constexpr int kSmallestTile = 32;
inline int tile_cost(long long E, long long n_nodes) {
  const long long total = E + kRowCost * n_nodes;
  int t = kSmallestTile;
  while (t < 256 && total / t > kTilesWanted) t <<= 1;
  return t;
}
inline long long tile_count(long long E, long long n_nodes, int tile) { return (E + kRowCost * n_nodes) / tile + 1; }
// the most tiles any graph of E positions and up to n_nodes nodes gets
inline long long tile_bound(long long E, long long n_nodes) {
  const int t = tile_cost(E, n_nodes);
  const long long n = tile_count(E, n_nodes, t);
  return t > kSmallestTile && n < kTilesWanted + 2 ? kTilesWanted + 2 : n;
}

struct Levels {
  int n = 0;
  long long len[kMaxLevels];
  int tile[kMaxLevels];
  long long ntiles[kMaxLevels];
};
inline Levels make_levels(long long n_edges, int tile0) {
  Levels lv;
  long long len = n_edges;
  int tile = tile0;
  for (;;) {
    const long long nt = (len + tile - 1) / tile;
    lv.len[lv.n] = len; lv.tile[lv.n] = tile; lv.ntiles[lv.n] = nt;
    ++lv.n;
    if (nt <= 1 || lv.n == kMaxLevels) break;
    len = 2 * nt;
    tile = kCarryTile;
  }
  return lv;
}

inline unsigned grid_for_warps(long long warps, int warps_per_cta) {
  long long g = (warps + warps_per_cta - 1) / warps_per_cta;
  return (unsigned)(g < 1 ? 1 : g);
}

// ---------------------------------------------------------------------------------------
// graph preparation: erow[] and 32-bit index arrays
// ---------------------------------------------------------------------------------------
struct GraphView {
  const PlanHeader* hdr;
  const int32_t* erow;
  const int32_t* other;  // may be null (ops without a second endpoint)
  const int32_t* eid;    // may be null: identity
  long long E;
  // work tiles: their boundaries (null: the op has no use for them), number and cost; whether the boundaries were moved
  // to row starts already (a plan's), and whether no row crosses one (then there is nothing to merge)
  const int32_t* tile_start = nullptr;
  long long n_tiles = 0;
  int tile = 0;
  bool aligned = false, no_carry = false;
  int repeats = -1;   // gather_repeats, a plan's finding; -1: skew_kernel counts them
};

// an edge output that starts from zero when some position belongs to no chunk
struct Clear { void* out = nullptr; size_t bytes = 0; };
// arrays of 32-bit words set on the way
struct Fill { int32_t* out[3]; long long n[3]; int32_t with[3]; };

template <typename I>
inline int prepare_graph(Arena& ar, const I* row, const I* indptr, const I* eid, const I* indices, long long C,
                         long long E, long long n_nodes, cudaStream_t st, GraphView* g, Clear clear = {},
                         PlanHeader* hdr = nullptr, const Fill& fill = {}) {
  if (!hdr) hdr = (PlanHeader*)ar.take(sizeof(PlanHeader));
  auto* erow = (int32_t*)ar.take((size_t)E * 4);
  // n_nodes < 0: an op that cuts no tiles
  TileCut cut{nullptr, 0, 0};
  if (n_nodes >= 0) {
    g->tile = tile_cost(E, n_nodes);
    while ((1 << cut.shift) < g->tile) ++cut.shift;
    cut.n = tile_count(E, n_nodes, g->tile);
    cut.start = (int32_t*)ar.take((size_t)(cut.n + 1) * 4);
    g->tile_start = cut.start; g->n_tiles = cut.n;
  }
  int32_t* other32 = nullptr;
  int32_t* eid32 = nullptr;
  if (sizeof(I) == 8) {
    if (indices) other32 = (int32_t*)ar.take((size_t)E * 4);
    if (eid) eid32 = (int32_t*)ar.take((size_t)E * 4);
  }
  if (!ar.base) return GRAPHOP_OK;
  if (ar.overflow) return GRAPHOP_ERR_WORKSPACE;
  const ExpandExtra<I> extra{{other32 ? indices : nullptr, eid32 ? eid : nullptr}, {other32, eid32}, (uint16_t*)clear.out,
                             (long long)(clear.bytes / 2), {fill.out[0], fill.out[1], fill.out[2]},
                             {fill.n[0], fill.n[1], fill.n[2]}, {fill.with[0], fill.with[1], fill.with[2]}};
  // About one step of positions per block, fewer where that would leave most of the chip idle: below kExpandBlocks blocks
  // the time is one block's chain of loads, and a shorter block has a shorter one.
  constexpr long long kExpandBlocks = 3 * 148;
  long long per_block = C > 0 ? kExpandTile * C / E : 1;
  if (C / kExpandBlocks < per_block) per_block = C / kExpandBlocks;
  per_block = per_block < 1 ? 1 : per_block > kExpandThreads ? kExpandThreads : per_block;
  long long blocks = C > 0 ? (C + per_block - 1) / per_block : 1;
  const long long copies = (other32 || eid32 || clear.out || fill.out[0]) ? (E + kExpandTile - 1) / kExpandTile : 1;
  if (blocks < copies && blocks < 1024) blocks = copies < 1024 ? copies : 1024;   // long chunks: blocks for the copies
  expand_rows_kernel<I><<<(unsigned)blocks, kExpandThreads, 0, st>>>(row, indptr, C, (int)E, (int)per_block, erow, hdr, cut,
                                                                  extra);
  GK_LAUNCHED("expand_rows");
  g->hdr = hdr;
  g->erow = erow;
  g->E = E;
  if (sizeof(I) == 8) {
    g->other = other32;
    g->eid = eid32;
  } else {
    g->other = (const int32_t*)indices;
    g->eid = (const int32_t*)eid;
  }
  return GRAPHOP_OK;
}

// Where an op's GraphView comes from: expanded on the spot from the caller's chunk table (into the workspace), or
// taken from a plan that graphop_plan_build_* made once for the graph.
template <typename I>
struct FromChunks {
  const I* row; const I* indptr; const I* eid; const I* indices; long long C, E;
  bool valid(bool need_indices) const { return row && indptr && (!need_indices || indices); }
  int operator()(Arena& ar, long long n_nodes, cudaStream_t st, GraphView* g, Clear clear = {}) const {
    return prepare_graph<I>(ar, row, indptr, eid, indices, C, E, n_nodes, st, g, clear);
  }
};
struct FromPlan {
  const graphop_plan_t* p;
  bool valid(bool need_indices) const { return p && p->erow && p->header && (!need_indices || p->other); }
  int operator()(Arena&, long long, cudaStream_t st, GraphView* g, Clear clear = {}) const {
    g->hdr = (const PlanHeader*)p->header;
    g->erow = p->erow;
    g->other = p->other;
    g->eid = p->eid;
    g->E = p->n_edges;
    g->tile_start = p->tile_start;
    g->tile = p->tile;
    g->n_tiles = p->tile ? tile_count(p->n_edges, p->n_nodes, p->tile) : 0;
    g->aligned = (p->flags & GRAPHOP_PLAN_ROW_TILES) != 0;
    g->no_carry = (p->flags & GRAPHOP_PLAN_NO_CARRY) != 0;
    g->repeats = p->gather_repeats;
    const long long words = (long long)(clear.bytes / 2);
    if (words && !(p->flags & GRAPHOP_PLAN_COVERED)) {
      zero_uncovered_kernel<uint16_t><<<(unsigned)((words + 1023) / 1024 < 2048 ? (words + 1023) / 1024 : 2048), 256, 0, st>>>(
          g->hdr, g->E, (uint16_t*)clear.out, words);
      GK_LAUNCHED("zero_uncovered");
    }
    return GRAPHOP_OK;
  }
};

// ---------------------------------------------------------------------------------------
// vector shape selection
// ---------------------------------------------------------------------------------------
template <typename T> struct VecMax { static constexpr int value = 16 / (int)sizeof(T); };

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
inline bool is_pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

}  // namespace gk
#include "gk_launch.cuh"
namespace gk {

// ---------------------------------------------------------------------------------------
// level-0 + carry-level launch sequence of a row-producing op of the register-fetch walker (gk_common.cuh): the shapes
// the gathering walker has no slot width for
// ---------------------------------------------------------------------------------------
template <class MakeOp>
inline int run_row_levels(Arena& ar, const GraphView& g, int tile0, long long n_rows, size_t carry_elem_bytes,
                          long long carry_stride, cudaStream_t st, MakeOp&& make_op) {
  Levels lv = make_levels(g.E, tile0);
  void* carry[kMaxLevels];
  int32_t* rows[kMaxLevels + 1];
  rows[0] = nullptr;
  for (int k = 0; k < lv.n; ++k) {
    const bool last = k == lv.n - 1;
    carry[k] = last ? nullptr : ar.take((size_t)(2 * lv.ntiles[k]) * carry_stride * carry_elem_bytes);
    rows[k + 1] = last ? nullptr : (int32_t*)ar.take((size_t)(2 * lv.ntiles[k]) * 4);
  }
  if (!ar.base) return GRAPHOP_OK;
  if (ar.overflow) return GRAPHOP_ERR_WORKSPACE;
  {
    auto op = make_op(carry[0], nullptr);
    using Op = decltype(op);
    walk_kernel<Op, false><<<grid_for_warps(lv.ntiles[0], kWarpsPerCta), kWarpsPerCta * 32, 0, st>>>(
        op, g.hdr, g.erow, g.other, g.eid, g.E, lv.tile[0], n_rows, rows[1]);
    GK_LAUNCHED(Op::kName);
  }
  for (int k = 1; k < lv.n; ++k) {
    auto op = make_op(carry[k], carry[k - 1]);
    using Op = decltype(op);
    walk_kernel<Op, true><<<grid_for_warps(lv.ntiles[k], kWarpsPerCta), kWarpsPerCta * 32, 0, st>>>(
        op, g.hdr, rows[k], nullptr, nullptr, lv.len[k], lv.tile[k], n_rows, rows[k + 1]);
    GK_LAUNCHED("carry_level");
  }
  return GRAPHOP_OK;
}

// Whether an op with an edge feature row shared by the heads can take all heads in a lane: slots of 16 bytes, a power of
// two of them per row, 4 to 32, and 2, 4 or 8 heads (8 heads of 8-byte accumulators would not fit the registers; one head
// gains nothing: 1 x 64 fp32 1.43 against 1.40 ms).  Returns the slots per row or 0.  R-MAT 18, NodeMulEdge and VectorSPMM
// forward and backward, against the walker with a copy of the row per head: 2 x 32 fp32 1.28 -> 1.19, 4 x 32 1.78 -> 1.60,
// 8 x 32 3.21 -> 2.74 ms, bf16 1.04 -> 0.97, 1.44 -> 1.31, 2.63 -> 2.37 ms.
template <typename T>
inline int feat_slots(int H, int D, std::initializer_list<const void*> rows16) {
  constexpr int VM = VecMax<T>::value;
  for (const void* p : rows16) if (!aligned16(p)) return 0;
  if (D % VM || !(H == 2 || H == 4 || (H == 8 && sizeof(T) <= 4))) return 0;
  const int ds = D / VM;
  return ds == 4 || ds == 8 || ds == 16 || ds == 32 ? ds : 0;
}
// f(TypeTag<integral_constant heads>, TypeTag<integral_constant slots>)
template <typename T, class F>
inline int dispatch_feat(int H, int ds, F&& f) {
  const auto heads = [&](auto slots) -> int {
    if (H == 2) return f(std::integral_constant<int, 2>{}, slots);
    if (H == 4) return f(std::integral_constant<int, 4>{}, slots);
    if constexpr (sizeof(T) <= 4) return f(std::integral_constant<int, 8>{}, slots);
    else return GRAPHOP_ERR_UNSUPPORTED;
  };
  if (ds == 4) return heads(std::integral_constant<int, 4>{});
  if (ds == 8) return heads(std::integral_constant<int, 8>{});
  if (ds == 16) return heads(std::integral_constant<int, 16>{});
  return heads(std::integral_constant<int, 32>{});
}

// The most repeats among the samples (gather_repeats) that chance explains where E positions gather n rows uniformly: their mean
// and four standard deviations, at least 16 (24 for many rows, 36 for 49 thousand, 88 for 10 thousand; seen on 200 uniform draws
// each: 16, 23, 69 at most).
inline int skew_allowed(long long n, long long E) {
  const double s = E < kSkewSamples ? (double)E : kSkewSamples, bits = kSkewBits, rows = n > 1 ? (double)n : 1;
  const double distinct = n > 1 ? -rows * std::expm1(s * std::log1p(-1 / rows)) : 1;
  const double chance = s + bits * std::expm1(distinct * std::log1p(-1 / bits)), spread = 4 * std::sqrt(chance > 0 ? chance : 0);
  return (int)std::ceil(chance + (spread > 16 ? spread : 16));
}

// Which sums of gathered rows go to the summing walker (gk_sum.cuh has what either side of the lines measures): elements of 4
// and 8 bytes.  Tables that fit the L2, which for `nhb` blocks of heads, walked one after the other, is up to twice as much if
// a block's share is not large: 33 thousand nodes of 30 edges, 16 x 64 fp32 (129 MB, blocks of 16), 320 against 405 us; 60
// thousand of 16, 8 x 64 (117 MB, blocks of 29), 177 to 207 against 202 to 214; 80 thousand (156 MB, blocks of 39) 266 against 248.
// Any larger one of so few rows that several blocks' shares fit, as long as the walks stay short enough for the blocks to follow
// one another: 4000 nodes of 30 edges, 128 x 128 (250 MB, blocks of 2), 632 against 726 us, but 926 in walks of any length; 20
// thousand of 16, 16 x 128 (156 MB, blocks of 10), 234 against 246.  Other larger ones, up to kSumTableBytes each and
// kSumAllBytes together, where few of their rows are gathered by many edges (two tables, 2.1 GB, R-MAT 21: 4.40 -> 4.09 ms; 3.0 GB,
// 6.2M skewed edges on 1.47M nodes, 4 x 64: 1.41 against 1.64 ms).  f(sums, only, most) launches the summing or the gathering walker: where the graph's skew
// is known to the device alone both are, and the one that it does not ask for returns at once (14 us a call, with the question:
// 98 -> 112 us on 1.4M uniform edges, 358 -> 379 on 6M; hubs 284 -> 112 and 541 -> 193).
template <typename T> constexpr bool kSumsByRegister = sizeof(T) >= 4;
constexpr long long kSumTableBytes = 3ll << 29, kSumAllBytes = 5ll << 29, kSumShare = 32ll << 20, kSumFewRows = 8ll << 20;
template <class F>
inline int choose_walker(Arena& ar, const GraphView& g, int tables, long long table, int nhb, long long n_gathered, cudaStream_t st,
                         F&& f) {
  const long long all = tables * table, share = all / nhb;
  // No row to gather, so no position has an edge: the summing walker loads row 0 in the place of one that is not there.
  if (all == 0) return f(false, -1, 0);
  if (all <= kL2Table || (all <= 2 * kL2Table && share <= kSumShare)) return f(true, -1, 0);
  if (table > kSumTableBytes || all > kSumAllBytes) return f(false, -1, tiles_near(table));
  if (share <= kSumFewRows) return f(true, -1, tiles_near(table));
  const int allowed = skew_allowed(n_gathered, g.E);
  if (g.repeats >= 0) return g.repeats > allowed ? f(true, -1, 0) : f(false, -1, tiles_near(table));
  if (ar.base && !ar.overflow) {
    skew_kernel<1024><<<1, 1024, 0, st>>>(g.other, g.E, allowed, const_cast<PlanHeader*>(g.hdr));
    GK_LAUNCHED("skew");
  }
  const size_t mark = ar.used;
  GK_TRY(f(true, 1, 0));
  ar.used = mark;   // one of the two does the work: the same scratch
  return f(false, 0, tiles_near(table));
}

// out[node] = sum_k w[eid[k]] * feat(k)
template <typename T, bool kEdgeFeat>
inline int run_aggregate(Arena& ar, const GraphView& g, const T* w, const T* x, T* y, long long n_rows, long long n_gathered,
                         int H, int D, cudaStream_t st) {
  using A = typename AccOf<T>::type;
  const long long table = n_gathered * H * D * (long long)sizeof(T);   // 0: the edges' own rows
  if constexpr (kEdgeFeat) {
    if (const int ds = feat_slots<T>(H, D, {x, y}))
      return dispatch_feat<T>(H, ds, [&](auto heads, auto slots) -> int {
        GeoPick p;
        p.SB = 16; p.G = p.L = decltype(slots)::value; p.W = decltype(heads)::value; p.nhb = 1;
        GroupFeatAggregate<FeatGeo<T, decltype(slots)::value, decltype(heads)::value>> op;
        fill_geo(op, p, H, D);
        op.w = w; op.x = x; op.y = y;
        return launch_walk(ar, g, p, op, n_rows, tiles_near(table), st);
      });
  }
  if constexpr (!kEdgeFeat && kSumsByRegister<T>) {
    const GeoPick p = pick_sum_geo(H, D, sizeof(T), slot_align_of({x, y})), ring = pick_geo(H, D, sizeof(T), slot_align_of({x, y}), true);
    if (p.SB && p.nhb <= kMaxHeadBlocks)
      return choose_walker(ar, g, 1, table, p.nhb, n_gathered, st, [&](bool sums, int only, int most) -> int {
        if (sums)
          return dispatch_sum_geo<T, true>(p, [&](auto tag) -> int {
            SumAggregate<typename decltype(tag)::type> op;
            fill_geo(op, p, H, D);
            op.w = w; op.x = x; op.y = y;
            op.wide_scalars = wide_scalars(p, w, H, sizeof(T));
            return launch_walk(ar, g, p, op, n_rows, most, st, only);
          });
        return dispatch_geo<T, true, false>(ring, [&](auto tag) -> int {
          GroupAggregate<typename decltype(tag)::type, false> op;
          fill_geo(op, ring, H, D);
          op.w = w; op.x = x; op.y = y;
          return launch_walk(ar, g, ring, op, n_rows, most, st, only);
        });
      });
  }
  const GeoPick p = pick_geo(H, D, sizeof(T), slot_align_of({x, y}), true);
  if (p.SB && p.nhb <= kMaxHeadBlocks)
    return dispatch_geo<T, true, false>(p, [&](auto tag) -> int {
      GroupAggregate<typename decltype(tag)::type, kEdgeFeat> op;
      fill_geo(op, p, H, D);
      op.w = w; op.x = x; op.y = y;
      return launch_walk(ar, g, p, op, n_rows, tiles_near(table), st);
    });
  // 2-byte elements with an odd D: one element per slot, feature blocks of 256
  const int HD = H * D, tile0 = pick_tile(g.E);
  constexpr int kBlock = 256;
  for (int feat0 = 0; feat0 < HD; feat0 += kBlock) {
    const size_t mark = ar.used;
    GK_TRY(run_row_levels(ar, g, tile0, n_rows, sizeof(A), HD, st, [&](void* cout, void* cin) {
      AggregateOp<T, 1, 8, kEdgeFeat> op;
      op.w = w; op.x = x; op.y = y; op.carry = (A*)cout; op.carry_in = (const A*)cin;
      op.H = H; op.D = D; op.HD = HD; op.S = HD - feat0 < kBlock ? HD - feat0 : kBlock; op.feat0 = feat0;
      return op;
    }));
    if (feat0 + kBlock < HD) ar.used = mark;  // blocks run back to back on one stream: reuse the scratch
  }
  return GRAPHOP_OK;
}

// y[eid[k], h] = a[node(k), h, :] . feat(k)[h, :]
template <typename T, bool kEdgeFeat>
inline int run_edge_dot(Arena& ar, const GraphView& g, const T* a, const T* b, T* y, long long n_gathered, int H, int D,
                        cudaStream_t st) {
  if constexpr (kEdgeFeat) {
    const size_t row = (size_t)H * sizeof(T);
    const int ds = (uintptr_t)y % (row < 16 ? row : 16) == 0 ? feat_slots<T>(H, D, {a, b}) : 0;
    if (ds) {
      if (!ar.base) return GRAPHOP_OK;
      return dispatch_feat<T>(H, ds, [&](auto heads, auto slots) -> int {
        const long long blocks = ((g.E + kMixPer - 1) / kMixPer * ds + 255) / 256;
        edge_feat_dot_kernel<T, VecMax<T>::value, decltype(heads)::value, decltype(slots)::value>
            <<<(unsigned)blocks, 256, 0, st>>>(g.erow, g.eid, a, b, y, g.E, D);
        GK_LAUNCHED("edge_dot");
        return GRAPHOP_OK;
      });
    }
  }
  const GeoPick p = narrow_fix(pick_geo(H, D, sizeof(T), slot_align_of({a, b}), false));
  if (p.SB && p.nhb <= kMaxHeadBlocks)
    return dispatch_geo<T, true, true>(p, [&](auto tag) -> int {
      GroupEdgeDot<typename decltype(tag)::type, kEdgeFeat> op;
      fill_geo(op, p, H, D);
      op.a = a; op.b = b; op.y = y;
      return launch_walk(ar, g, p, op, 0, tiles_near(n_gathered * H * D * (long long)sizeof(T)), st);
    });
  const int tile0 = pick_tile(g.E);
  EdgeDotAnyOp<T, kEdgeFeat> op;
  op.a = a; op.b = b; op.y = y; op.H = H; op.D = D; op.HD = H * D;
  walk_kernel<decltype(op), false><<<grid_for_warps((g.E + tile0 - 1) / tile0, kWarpsPerCta), kWarpsPerCta * 32, 0, st>>>(
      op, g.hdr, g.erow, g.other, g.eid, g.E, tile0, 0, nullptr);
  GK_LAUNCHED("edge_dot_any");
  return GRAPHOP_OK;
}

// db[edge, :] = sum_h g[edge, h] * a[node, h, :]; g = dy by edge id or, kPairs, the score gradients by position.
template <typename T, bool kPairs>
inline int run_edge_mix(const GraphView& g, const T* dy, const EdgePair<typename AccOf<T>::type>* pairs, int Hp, const T* a,
                        T* db, int H, int D, cudaStream_t st) {
  constexpr int VM = VecMax<T>::value;
  const bool vec = aligned16(a) && aligned16(db) && D % VM == 0;
  const size_t row = (size_t)H * sizeof(T);
  // the head counts whose row of g is whole aligned moves
  const int hh = vec && (H == 1 || H == 2 || H == 4 || H == 8) && (kPairs || (uintptr_t)dy % (row < 16 ? row : 16) == 0) ? H : 0;
  const int ds = vec ? D / VM : D;
  int shift = -1;
  if (is_pow2(ds)) for (shift = 0; (1 << shift) < ds; ++shift) {}
  const long long blocks = ((g.E + kMixPer - 1) / kMixPer * ds + 255) / 256;
#define GK_MIX(VV, HH)                                                                                                \
  edge_mix_kernel<T, VV, HH, kPairs><<<(unsigned)blocks, 256, 0, st>>>(g.erow, g.eid, dy, pairs, a, db, g.E, H, Hp, D, shift)
  if (!vec) GK_MIX(1, 0);
  else if (hh == 1) GK_MIX(VM, 1);
  else if (hh == 2) GK_MIX(VM, 2);
  else if (hh == 4) GK_MIX(VM, 4);
  else if (hh == 8) GK_MIX(VM, 8);
  else GK_MIX(VM, 0);
#undef GK_MIX
  GK_LAUNCHED(kPairs ? "attention_bias_grad" : "edge_mix_heads");
  return GRAPHOP_OK;
}

// ---------------------------------------------------------------------------------------
// softmax
// ---------------------------------------------------------------------------------------
// Columns h0 .. h0 + H - 1 of (E, hs) tensors.
template <typename T, int H, bool kBackward, bool kVec>
inline int run_softmax_heads(Arena& ar, const GraphView& g, const T* in0, const T* in1, T* out, int hs, int h0,
                             cudaStream_t st) {
  using A = typename AccOf<T>::type;
  const long long nt = (g.E + kSoftmaxTile - 1) / kSoftmaxTile;
  const size_t slot_bytes = (size_t)(2 * nt) * (kBackward ? H : 2 * H) * sizeof(A);
  A* slots = (A*)ar.take(slot_bytes);
  int32_t* rows = (int32_t*)ar.take((size_t)(2 * nt) * 4);
  A* merged = nt > kSoftmaxSelfMerge ? (A*)ar.take(slot_bytes) : nullptr;
  if (!ar.base) return GRAPHOP_OK;
  if (ar.overflow) return GRAPHOP_ERR_WORKSPACE;
  softmax_tile_kernel<T, H, kBackward, kVec><<<(unsigned)nt, kSoftmaxThreads, 0, st>>>(g.erow, g.eid, in0, in1, out, slots,
                                                                                      rows, g.E, hs, h0);
  GK_LAUNCHED(kBackward ? "softmax_bwd_tile" : "softmax_fwd_tile");
  if (nt == 1) return GRAPHOP_OK;   // nothing crosses
  if (merged) {
    softmax_merge_kernel<A, H, kBackward><<<grid_for_warps(nt, kSoftmaxWarps), kSoftmaxThreads, 0, st>>>(slots, rows, merged,
                                                                                                         nt);
    GK_LAUNCHED("softmax_merge");
  }
  softmax_finish_kernel<T, H, kBackward, kVec><<<(unsigned)nt, kSoftmaxThreads, 0, st>>>(g.erow, g.eid, in0, in1, out, slots,
                                                                                        rows, merged, g.E, nt, hs, h0);
  GK_LAUNCHED(kBackward ? "softmax_bwd_finish" : "softmax_fwd_finish");
  return GRAPHOP_OK;
}

// Head counts whose edge rows are whole vector moves go in one pass; any other count, and rows at an address that the
// moves cannot take, in passes of up to four heads read one by one.
template <typename T, bool kBackward>
inline int run_softmax(Arena& ar, const GraphView& g, const T* in0, const T* in1, T* out, int H, cudaStream_t st) {
  const size_t hb = (size_t)H * sizeof(T), want = hb < 16 ? hb : 16;
  const bool vec_ok = (uintptr_t)in0 % want == 0 && (uintptr_t)out % want == 0 && (!kBackward || (uintptr_t)in1 % want == 0);
  if (vec_ok && H == 1) return run_softmax_heads<T, 1, kBackward, true>(ar, g, in0, in1, out, 1, 0, st);
  if (vec_ok && H == 2) return run_softmax_heads<T, 2, kBackward, true>(ar, g, in0, in1, out, 2, 0, st);
  if (vec_ok && H == 4) return run_softmax_heads<T, 4, kBackward, true>(ar, g, in0, in1, out, 4, 0, st);
  if (vec_ok && H == 8) return run_softmax_heads<T, 8, kBackward, true>(ar, g, in0, in1, out, 8, 0, st);
  const int passes = (H + 3) / 4, step = (H + passes - 1) / passes;
  const size_t mark = ar.used;
  for (int h = 0; h < H; h += step) {
    ar.used = mark;   // the passes run back to back on one stream: scratch reused
    const int n = H - h < step ? H - h : step;
    if (n == 1) GK_TRY((run_softmax_heads<T, 1, kBackward, false>(ar, g, in0, in1, out, H, h, st)));
    if (n == 2) GK_TRY((run_softmax_heads<T, 2, kBackward, false>(ar, g, in0, in1, out, H, h, st)));
    if (n == 3) GK_TRY((run_softmax_heads<T, 3, kBackward, false>(ar, g, in0, in1, out, H, h, st)));
    if (n == 4) GK_TRY((run_softmax_heads<T, 4, kBackward, false>(ar, g, in0, in1, out, H, h, st)));
    if (!ar.base) break;
  }
  return GRAPHOP_OK;
}

// ---------------------------------------------------------------------------------------
// argument checks shared by the entry points
// ---------------------------------------------------------------------------------------
inline int check_sizes(long long C, long long E, long long n0, long long n1, int H, int D) {
  if (C < 0 || E < 0 || n0 < 0 || n1 < 0 || H < 1 || D < 1) return GRAPHOP_ERR_INVALID_ARGUMENT;
  if (E >= (1LL << 31) || n0 >= (1LL << 31) || n1 >= (1LL << 31)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  if ((long long)H * D >= (1LL << 24)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  return GRAPHOP_OK;
}
inline int check_ws(const void* ws) {
  if (!ws || ((uintptr_t)ws & (kAlign - 1))) return GRAPHOP_ERR_WORKSPACE;
  return GRAPHOP_OK;
}

// ---------------------------------------------------------------------------------------
// the ten operations
// ---------------------------------------------------------------------------------------
template <typename T, class GS>
inline int maskedmm_forward(const GS& gs, const T* A_, const T* B_, T* y, long long C, long long E, long long n_dst,
                            long long n_src, int H, int D, void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  if (E == 0) return GRAPHOP_OK;
  if (!gs.valid(true) || !A_ || !B_ || !y) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  GK_TRY(gs(ar, n_dst, st, &g, Clear{y, (size_t)E * H * sizeof(T)}));
  return run_edge_dot<T, false>(ar, g, A_, B_, y, n_src, H, D, st);
}

template <typename T, class GS>
inline int maskedmm_backward(const GS& gs_r, const GS& gs_c, long long Cr, long long Cc, const T* A_, const T* B_,
                             const T* dy, T* dA, T* dB, long long E, long long n_dst, long long n_src, int H, int D,
                             void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(Cr, E, n_dst, n_src, H, D));
  if (Cc < 0) return GRAPHOP_ERR_INVALID_ARGUMENT;
  const size_t HD = (size_t)H * D;
  if (E == 0) {
    if (n_dst) GK_CUDA(cudaMemsetAsync(dA, 0, (size_t)n_dst * HD * sizeof(T), st));
    if (n_src) GK_CUDA(cudaMemsetAsync(dB, 0, (size_t)n_src * HD * sizeof(T), st));
    return GRAPHOP_OK;
  }
  if (!gs_r.valid(true) || !gs_c.valid(true) || !A_ || !B_ || !dy || !dA || !dB) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  {
    GraphView g;
    GK_TRY(gs_r(ar, n_dst, st, &g));
    GK_TRY((run_aggregate<T, false>(ar, g, dy, B_, dA, n_dst, n_src, H, D, st)));
  }
  ar.used = 0;  // the second pass runs after the first on the same stream: reuse the scratch
  GraphView g;
  GK_TRY(gs_c(ar, n_src, st, &g));
  return run_aggregate<T, false>(ar, g, dy, A_, dB, n_src, n_dst, H, D, st);
}

template <typename T, class GS>
inline int node_mul_edge_forward(const GS& gs, const T* A_, const T* B_, T* y, long long C, long long E,
                                 long long n_dst, int H, int D, void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(C, E, n_dst, 0, H, D));
  if (E == 0) return GRAPHOP_OK;
  if (!gs.valid(false) || !A_ || !B_ || !y) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  GK_TRY(gs(ar, n_dst, st, &g, Clear{y, (size_t)E * H * sizeof(T)}));
  return run_edge_dot<T, true>(ar, g, A_, B_, y, 0, H, D, st);
}

template <typename T, class GS>
inline int node_mul_edge_backward(const GS& gs, const T* A_, const T* B_, const T* dy, T* dA, T* dB, long long C,
                                  long long E, long long n_dst, int H, int D, void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(C, E, n_dst, 0, H, D));
  if (E == 0) {
    if (n_dst) GK_CUDA(cudaMemsetAsync(dA, 0, (size_t)n_dst * H * D * sizeof(T), st));
    return GRAPHOP_OK;
  }
  if (!gs.valid(false) || !A_ || !B_ || !dy || !dA || !dB) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  GK_TRY(gs(ar, n_dst, st, &g, Clear{dB, (size_t)E * D * sizeof(T)}));
  GK_TRY((run_aggregate<T, true>(ar, g, dy, B_, dA, n_dst, 0, H, D, st)));
  if (!ar.base) return GRAPHOP_OK;
  return run_edge_mix<T, false>(g, dy, nullptr, 0, A_, dB, H, D, st);
}

template <typename T, bool kBackward, class GS>
inline int sparse_softmax(const GS& gs, const T* in0, const T* in1, T* out, long long C, long long E,
                          long long n_nodes, int H, void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(C, E, n_nodes, 0, H, 1));
  if (E == 0) return GRAPHOP_OK;
  if (!gs.valid(false) || !in0 || !out || (kBackward && !in1)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  GK_TRY(gs(ar, -1, st, &g, Clear{out, (size_t)E * H * sizeof(T)}));
  return run_softmax<T, kBackward>(ar, g, in0, in1, out, H, st);
}

template <typename T, class GS>
inline int spmm_forward(const GS& gs, const T* edata, const T* x, T* y, long long C, long long E, long long n_dst,
                        long long n_src, int H, int D, void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  if (n_dst == 0) return GRAPHOP_OK;
  if (E == 0) {
    GK_CUDA(cudaMemsetAsync(y, 0, (size_t)n_dst * H * D * sizeof(T), st));
    return GRAPHOP_OK;
  }
  if (!gs.valid(true) || !edata || !x || !y) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  GK_TRY(gs(ar, n_dst, st, &g));
  return run_aggregate<T, false>(ar, g, edata, x, y, n_dst, n_src, H, D, st);
}

template <typename T, class GS>
inline int spmm_backward(const GS& gs_r, const GS& gs_c, long long C, long long Ct, const T* edata, const T* dy,
                         const T* x, T* dedata, T* dx, long long E, long long n_dst, long long n_src, int H, int D,
                         void* ws, size_t wsb, cudaStream_t st) {
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  if (Ct < 0) return GRAPHOP_ERR_INVALID_ARGUMENT;
  if (E == 0) {
    if (n_src) GK_CUDA(cudaMemsetAsync(dx, 0, (size_t)n_src * H * D * sizeof(T), st));
    return GRAPHOP_OK;
  }
  if (!gs_r.valid(true) || !gs_c.valid(true) || !edata || !dy || !x || !dedata || !dx) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  {
    GraphView g;
    GK_TRY(gs_r(ar, n_dst, st, &g, Clear{dedata, (size_t)E * H * sizeof(T)}));
    if (ar.base) GK_TRY((run_edge_dot<T, false>(ar, g, dy, x, dedata, n_src, H, D, st)));
  }
  ar.used = 0;
  GraphView g;
  GK_TRY(gs_c(ar, n_src, st, &g));
  return run_aggregate<T, false>(ar, g, edata, dy, dx, n_src, n_dst, H, D, st);
}

template <typename A>
__global__ void fill_kernel(A* __restrict__ out, A value, long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = value;
}
template <typename A> inline A neg_inf_host();
template <> inline float neg_inf_host<float>() { return -INFINITY; }
template <> inline double neg_inf_host<double>() { return -(double)INFINITY; }

// The fused kernels take heads of a power-of-two number of 16-byte slots and node rows of at most 4 KB.
template <typename T>
inline bool attention_shape_ok(int H, int D, bool al, GeoPick* p) {
  constexpr int VM = VecMax<T>::value;
  if (!al || D % VM || !is_pow2(D / VM) || (long long)H * D / VM > 256) return false;
  *p = pick_geo(H, D, sizeof(T), 16, false);
  return p->SB == 16;
}

template <typename T, bool kBias>
inline int run_attn_forward(Arena& ar, const GraphView& g, const GeoPick& s, const T* q, const T* k, const T* v,
                            const T* rel, double scale, T* o, void* lse, long long n_dst, long long n_src, int H,
                            int D, cudaStream_t st) {
  return dispatch_geo<T, false, true>(s, [&](auto tag) -> int {
    GroupAttnFwd<typename decltype(tag)::type, kBias> op;
    using A = typename decltype(op)::A;
    fill_geo(op, s, H, D);
    op.q = q; op.k = k; op.v = v; op.rel = rel; op.o = o; op.lse = (A*)lse; op.scale = (A)scale;
    return launch_walk(ar, g, s, op, n_dst, tiles_near(2 * n_src * H * D * (long long)sizeof(T)), st);
  });
}
template <typename T, bool kBias, class A>
inline int run_attn_bwd_dst(Arena& ar, const GraphView& g, const GeoPick& s, const T* q, const T* k, const T* v,
                            const T* rel, const T* o, const T* dout, const void* lse, StatPair<A>* stat,
                            EdgePair<A>* pd, double scale, T* dq, long long n_dst, long long n_src, int H, int D,
                            cudaStream_t st) {
  return dispatch_geo<T, false, true>(s, [&](auto tag) -> int {
    GroupAttnBwdDst<typename decltype(tag)::type, kBias> op;
    fill_geo(op, s, H, D);
    op.q = q; op.k = k; op.v = v; op.rel = rel; op.o = o; op.dout = dout; op.lse = (const A*)lse; op.stat = stat;
    op.pd = pd; op.dq = dq; op.scale = (A)scale; op.Hp = stat_heads(H, (int)sizeof(A));
    return launch_walk(ar, g, s, op, n_dst, tiles_near(2 * n_src * H * D * (long long)sizeof(T)), st);
  });
}
template <typename T, bool kPairs, class A>
inline int run_attn_bwd_src(Arena& ar, const GraphView& g, const GeoPick& s, const T* q, const T* k, const T* v,
                            const T* dout, const StatPair<A>* stat, const EdgePair<A>* pd, double scale, T* dk, T* dv,
                            long long n_src, int H, int D, cudaStream_t st, int most, int only = -1) {
  return dispatch_geo<T, false, true>(s, [&](auto tag) -> int {
    GroupAttnBwdSrc<typename decltype(tag)::type, kPairs> op;
    fill_geo(op, s, H, D);
    op.q = q; op.k = k; op.v = v; op.dout = dout; op.stat = stat; op.pd = pd; op.dk = dk; op.dv = dv;
    op.scale = (A)scale; op.Hp = stat_heads(H, (int)sizeof(A));
    return launch_walk(ar, g, s, op, n_src, most, st, only);
  });
}

// from the pairs that the destination side left
template <typename T, class A>
inline int run_attn_bwd_pairs(Arena& ar, const GraphView& g, const GeoPick& s, const T* q, const T* k, const T* v,
                              const T* dout, const StatPair<A>* stat, const EdgePair<A>* pd, double scale, T* dk, T* dv,
                              long long n_dst, long long n_src, int H, int D, cudaStream_t st) {
  if constexpr (kSumsByRegister<T>) {
    const long long table = n_dst * H * D * (long long)sizeof(T);
    const GeoPick p = pick_sum_geo(H, D, sizeof(T), 16);
    return choose_walker(ar, g, 2, table, p.nhb, n_dst, st, [&](bool sums, int only, int most) -> int {
      if (!sums) return run_attn_bwd_src<T, true>(ar, g, s, q, k, v, dout, stat, pd, scale, dk, dv, n_src, H, D, st, most, only);
      return dispatch_sum_geo<T, false>(p, [&](auto tag) -> int {
        SumAttnPairs<typename decltype(tag)::type> op;
        fill_geo(op, p, H, D);
        op.q = q; op.dout = dout; op.pd = pd; op.dk = dk; op.dv = dv;
        op.Hp = stat_heads(H, (int)sizeof(A));
        op.wide_scalars = wide_scalars(p, pd, op.Hp, 2 * (int)sizeof(A));
        return launch_walk(ar, g, p, op, n_src, most, st, only);
      });
    });
  } else {
    return run_attn_bwd_src<T, true>(ar, g, s, q, k, v, dout, stat, pd, scale, dk, dv, n_src, H, D, st,
                                     tiles_near(2 * n_dst * H * D * (long long)sizeof(T)));
  }
}

template <typename T, class GS>
inline int attention_forward(const GS& gs, long long C, const T* q, const T* k, const T* v, double scale, T* o,
                             void* lse, long long E, long long n_dst, long long n_src, int H, int D, void* ws,
                             size_t wsb, cudaStream_t st) {
  using A = typename AccOf<T>::type;
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  GeoPick s;
  if (!attention_shape_ok<T>(H, D, aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o), &s))
    return GRAPHOP_ERR_UNSUPPORTED;
  if (n_dst == 0) return GRAPHOP_OK;
  if (!q || !k || !v || !o || !lse) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  const int HD = H * D;
  if (E == 0) {
    // no edge anywhere: o = 0 and lse = -inf for every node
    GK_CUDA(cudaMemsetAsync(o, 0, (size_t)n_dst * HD * sizeof(T), st));
    const long long cells = n_dst * H;
    const unsigned grid = (unsigned)((cells + 255) / 256 < 4096 ? (cells + 255) / 256 : 4096);
    fill_kernel<A><<<grid ? grid : 1, 256, 0, st>>>((A*)lse, neg_inf_host<A>(), cells);
    GK_LAUNCHED("fill");
    return GRAPHOP_OK;
  }
  if (!gs.valid(true)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(gs(ar, n_dst, st, &g));
  return run_attn_forward<T, false>(ar, g, s, q, k, v, (const T*)nullptr, scale, o, lse, n_dst, n_src, H, D, st);
}

// Defined in gk_banded.cuh for bfloat16: the tensor-core kernel for dense-band graphs.  Returns
// GRAPHOP_ERR_UNSUPPORTED when the shape is not one it takes (the caller then runs the walker).
template <typename T>
int banded_attention_forward(const graphop_plan_t* plan, const T* q, const T* k, const T* v, double scale, T* o,
                             void* lse, long long n_dst, long long n_src, int H, int D, cudaStream_t st);
template <typename T>
inline int banded_attention_forward(const graphop_plan_t*, const T*, const T*, const T*, double, T*, void*, long long,
                                    long long, int, int, cudaStream_t) {
  return GRAPHOP_ERR_UNSUPPORTED;
}

template <typename T>
int banded_attention_backward(const graphop_plan_t* plan_r, const graphop_plan_t* plan_t, const T* q, const T* k,
                              const T* v, const T* o, const void* lse, const T* d_o, double scale, T* dq, T* dk, T* dv,
                              long long n_dst, long long n_src, int H, int D, void* ws, size_t wsb, cudaStream_t st);
template <typename T>
inline int banded_attention_backward(const graphop_plan_t*, const graphop_plan_t*, const T*, const T*, const T*,
                                     const T*, const void*, const T*, double, T*, T*, T*, long long, long long, int, int,
                                     void*, size_t, cudaStream_t) {
  return GRAPHOP_ERR_UNSUPPORTED;
}

template <typename T>
inline int attention_forward_planned(const graphop_plan_t* plan, const T* q, const T* k, const T* v, double scale,
                                     T* o, void* lse, long long n_dst, long long n_src, int H, int D, void* ws,
                                     size_t wsb, cudaStream_t st) {
  if (!plan) return GRAPHOP_ERR_INVALID_ARGUMENT;
  if ((plan->flags & GRAPHOP_PLAN_DENSE_BAND) && q && k && v && o && lse) {
    const int rc = banded_attention_forward<T>(plan, q, k, v, scale, o, lse, n_dst, n_src, H, D, st);
    if (rc != GRAPHOP_ERR_UNSUPPORTED) return rc;
  }
  return attention_forward<T>(FromPlan{plan}, plan->n_chunks, q, k, v, scale, o, lse, plan->n_edges, n_dst, n_src, H,
                              D, ws, wsb, st);
}

// has_eid_t: the transposed source carries edge ids (the positions of its edges in the row CSR)
template <typename T, class GS>
inline int attention_backward(const GS& gs_r, const GS& gs_c, bool has_eid_t, long long C, long long Ct, const T* q,
                              const T* k, const T* v, const T* o, const void* lse, const T* dout, double scale, T* dq,
                              T* dk, T* dv, long long E, long long n_dst, long long n_src, int H, int D, void* ws,
                              size_t wsb, cudaStream_t st) {
  using A = typename AccOf<T>::type;
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  if (Ct < 0) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GeoPick s;
  const bool al = aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o) && aligned16(dout) && aligned16(dq) &&
                  aligned16(dk) && aligned16(dv);
  if (!attention_shape_ok<T>(H, D, al, &s)) return GRAPHOP_ERR_UNSUPPORTED;
  if (E == 0) {  // no edge: every gradient is zero
    if ((n_dst && !dq) || (n_src && (!dk || !dv))) return GRAPHOP_ERR_INVALID_ARGUMENT;
    const size_t rowb = (size_t)H * D * sizeof(T);
    if (n_dst) GK_CUDA(cudaMemsetAsync(dq, 0, (size_t)n_dst * rowb, st));
    if (n_src) GK_CUDA(cudaMemsetAsync(dk, 0, (size_t)n_src * rowb, st));
    if (n_src) GK_CUDA(cudaMemsetAsync(dv, 0, (size_t)n_src * rowb, st));
    return GRAPHOP_OK;
  }
  if (!gs_r.valid(true) || !gs_c.valid(true) || !q || !k || !v || !o || !lse || !dout || !dq || !dk || !dv)
    return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  const int Hp = stat_heads(H, (int)sizeof(A));
  StatPair<A>* stat = (StatPair<A>*)ar.take((size_t)n_dst * Hp * sizeof(StatPair<A>));  // survives both passes
  // with the transposed CSR's edge ids the destination pass leaves (p, ds) of every edge for the source pass
  EdgePair<A>* pd = has_eid_t ? (EdgePair<A>*)ar.take((size_t)E * Hp * sizeof(EdgePair<A>)) : nullptr;
  const size_t mark = ar.used;
  {
    GraphView g;
    GK_TRY(gs_r(ar, n_dst, st, &g));
    GK_TRY((run_attn_bwd_dst<T, false>(ar, g, s, q, k, v, (const T*)nullptr, o, dout, lse, stat, pd, scale, dq, n_dst,
                                       n_src, H, D, st)));
  }
  ar.used = mark;
  GraphView g;
  GK_TRY(gs_c(ar, n_src, st, &g));
  if (pd) return run_attn_bwd_pairs<T>(ar, g, s, q, k, v, dout, stat, pd, scale, dk, dv, n_dst, n_src, H, D, st);
  return run_attn_bwd_src<T, false>(ar, g, s, q, k, v, dout, stat, pd, scale, dk, dv, n_src, H, D, st,
                                    tiles_near(2 * n_dst * H * D * (long long)sizeof(T)));
}

// ---------------------------------------------------------------------------------------
// Attention with an edge term in the scores: s_k = scale * q[n] . (k[other[k]] + rel[k]), rel an (n_edges, D)
// tensor indexed by row-CSR position and shared by the heads.  It is the reference's node_mul_edge
// (graphop_kernel.cu:16-34, "designed for relative positional encoding") added to maskedmm's scores before
// the softmax, computed in the fused pass instead of as two more (n_edges, H) tensors.
// ---------------------------------------------------------------------------------------
template <typename T, class GS>
inline int attention_bias_forward(const GS& gs, long long C, const T* q, const T* k, const T* v, const T* rel,
                                  double scale, T* o, void* lse, long long E, long long n_dst, long long n_src, int H,
                                  int D, void* ws, size_t wsb, cudaStream_t st) {
  using A = typename AccOf<T>::type;
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  GeoPick s;
  if (!attention_shape_ok<T>(H, D, aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o) && aligned16(rel), &s))
    return GRAPHOP_ERR_UNSUPPORTED;
  if (E == 0 || n_dst == 0)   // no edge: the edge term has nothing to add
    return attention_forward<T>(gs, C, q, k, v, scale, o, lse, E, n_dst, n_src, H, D, ws, wsb, st);
  if (!q || !k || !v || !rel || !o || !lse || !gs.valid(true)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  GraphView g;
  GK_TRY(gs(ar, n_dst, st, &g));
  return run_attn_forward<T, true>(ar, g, s, q, k, v, rel, scale, o, lse, n_dst, n_src, H, D, st);
}

// Gradients of the above.  The transposed CSR must carry eid_t (for each of its positions the row-CSR position of
// the same edge): the destination pass leaves (p, ds) of every edge in the workspace, the source pass aggregates
// them into dk and dv, and d_rel[j] = sum_h ds[j, h] q[node(j), h] comes from the same pairs.
template <typename T, class GS>
inline int attention_bias_backward(const GS& gs_r, const GS& gs_c, bool has_eid_t, long long C, long long Ct,
                                   const T* q, const T* k, const T* v, const T* rel, const T* o, const void* lse,
                                   const T* dout, double scale, T* dq, T* dk, T* dv, T* d_rel, long long E,
                                   long long n_dst, long long n_src, int H, int D, void* ws, size_t wsb,
                                   cudaStream_t st) {
  using A = typename AccOf<T>::type;
  GK_TRY(check_sizes(C, E, n_dst, n_src, H, D));
  if (Ct < 0) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GeoPick s;
  const bool al = aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o) && aligned16(dout) && aligned16(dq) &&
                  aligned16(dk) && aligned16(dv) && aligned16(rel);
  if (!attention_shape_ok<T>(H, D, al, &s)) return GRAPHOP_ERR_UNSUPPORTED;
  if (E == 0)
    return attention_backward<T>(gs_r, gs_c, has_eid_t, C, Ct, q, k, v, o, lse, dout, scale, dq, dk, dv, E, n_dst,
                                 n_src, H, D, ws, wsb, st);
  if (!has_eid_t || !gs_r.valid(true) || !gs_c.valid(true) || !q || !k || !v || !rel || !o || !lse || !dout || !dq ||
      !dk || !dv || !d_rel)
    return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(ws));
  Arena ar(ws, wsb);
  const int Hp = stat_heads(H, (int)sizeof(A));
  StatPair<A>* stat = (StatPair<A>*)ar.take((size_t)n_dst * Hp * sizeof(StatPair<A>));
  EdgePair<A>* pd = (EdgePair<A>*)ar.take((size_t)E * Hp * sizeof(EdgePair<A>));
  const size_t mark = ar.used;
  {
    GraphView g;
    GK_TRY(gs_r(ar, n_dst, st, &g));
    GK_TRY((run_attn_bwd_dst<T, true>(ar, g, s, q, k, v, rel, o, dout, lse, stat, pd, scale, dq, n_dst, n_src, H,
                                      D, st)));
    GK_TRY((run_edge_mix<T, true>(g, nullptr, pd, Hp, q, d_rel, H, D, st)));
  }
  ar.used = mark;
  GraphView g;
  GK_TRY(gs_c(ar, n_src, st, &g));
  return run_attn_bwd_pairs<T>(ar, g, s, q, k, v, dout, stat, pd, scale, dk, dv, n_dst, n_src, H, D, st);
}

template <typename T>
inline int attention_backward_planned(const graphop_plan_t* plan_r, const graphop_plan_t* plan_t, const T* q,
                                      const T* k, const T* v, const T* o, const void* lse, const T* dout, double scale,
                                      T* dq, T* dk, T* dv, long long n_dst, long long n_src, int H, int D, void* ws,
                                      size_t wsb, cudaStream_t st) {
  if (!plan_r || !plan_t) return GRAPHOP_ERR_INVALID_ARGUMENT;
  if ((plan_r->flags & plan_t->flags & GRAPHOP_PLAN_DENSE_BAND) && q && k && v && o && lse && dout && dq && dk && dv) {
    const int rc = banded_attention_backward<T>(plan_r, plan_t, q, k, v, o, lse, dout, scale, dq, dk, dv, n_dst, n_src,
                                                H, D, ws, wsb, st);
    if (rc != GRAPHOP_ERR_UNSUPPORTED) return rc;
  }
  return attention_backward<T>(FromPlan{plan_r}, FromPlan{plan_t}, plan_t->eid != nullptr, plan_r->n_chunks,
                               plan_t->n_chunks, q, k, v, o, lse, dout, scale, dq, dk, dv, plan_r->n_edges, n_dst,
                               n_src, H, D, ws, wsb, st);
}

}  // namespace gk
