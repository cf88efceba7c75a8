// Launching the gathering walker (gk_group.cuh): which geometry a row shape gets, the carry records, the launch.
#pragma once
#include "gk_group.cuh"
#include "gk_sum.cuh"

namespace gk {

// ---------------------------------------------------------------------------------------
// geometry of an (H, D) row
// ---------------------------------------------------------------------------------------
struct GeoPick {
  int SB = 0;      // 0: no slot width fits (2-byte elements with an odd D), or the head is too wide
  int G = 0, W = 0, LT = 0, L = 0, parts = 1, nhb = 0;
  int accs(int elem) const { return SB ? W * (SB / elem) * G : 0; }
};

// slot_align: the largest of 16, 8, 4 that divides every operand's address.  split: a head wider than a block may be
// walked piece by piece (aggregations; a dot product needs the whole head in one step).
//
// Blocks of heads of about 32 slots (512 bytes with 16-byte slots) as 16 lanes x 2 slots, narrower rows 8 x 2, 8 x 1,
// 4 x 1: two slots per lane halve the shuffles and the address arithmetic per byte.  Narrower blocks of a wide row were
// measured slower although a head's share of the tensor fits the L2 better (4 x 32 fp32 on R-MAT 21, forward: blocks of
// 512 / 256 / 128 bytes 3.5 / 3.7 / 5.3 ms): every block walks the nodes again.  Four slots per lane touch 32 bytes of
// four heads per copy instruction: 6.3 ms.  2-byte elements have twice the accumulators per slot: one slot per lane and
// blocks of 16 slots (16 lanes x 2 slots spilled and ran half as fast).
inline GeoPick pick_geo(int H, int D, int elem, int slot_align, bool split, bool one_slot = false) {
  GeoPick g;
  const int target = elem == 2 ? 16 : 32;
  const long long db = (long long)D * elem;
  int sb = 16;
  while (sb >= 4 && (db % sb || slot_align % sb)) sb >>= 1;
  if (sb < 4 || sb < elem) return g;
  int ds = (int)(db / sb);   // slots per head
  const auto pow2 = [](int v) { int p = 1; while (p < v) p <<= 1; return p; };
  bool exact = (ds & (ds - 1)) == 0;
  const bool two_byte = elem == 2 || one_slot;
  if (split && ds > target) {
    g.parts = (ds + target - 1) / target;
    exact = exact && ds % target == 0;
    ds = target;
  }
  if (ds > 32) {
    const int w = pow2((ds + 31) / 32);
    if (w > 8) return g;
    g.G = 32; g.W = w; g.L = 32;
  } else {
    const int dp = pow2(ds);
    int heads = pow2(H * g.parts);
    if (heads * dp > target) heads = target / dp > 0 ? target / dp : 1;
    if (heads > kMaxBlockHeads) heads = kMaxBlockHeads;
    const int ns = heads * dp;
    if (ns == 32) { g.G = two_byte ? 32 : 16; g.W = two_byte ? 1 : 2; }
    else if (ns == 16) { g.G = two_byte ? 16 : 8; g.W = two_byte ? 1 : 2; }
    else if (ns == 8) { g.G = 8; g.W = 1; }   // (heads of one slot: at most 8 of them, so never wider)
    else { g.G = 4; g.W = 1; }
    g.L = dp / g.W;
  }
  g.SB = sb;
  const int per = g.G / g.L;
  g.nhb = (H * g.parts + per - 1) / per;
  if (exact && ds == g.L * g.W && H * g.parts % per == 0 && sb == 16) g.LT = g.L;
  return g;
}

inline int slot_align_of(std::initializer_list<const void*> ptrs) {
  uintptr_t bits = 16;
  for (const void* p : ptrs) bits |= (uintptr_t)p;
  return (bits & 3) ? 1 : (bits & 7) ? 4 : (bits & 15) ? 8 : 16;
}

// The summing walker's: one slot per lane, and no head is too wide, it is walked piece by piece.  With rows of 512 bytes as
// 16 lanes x 2 slots a load instruction touches 64 bytes of every head: 15360 nodes of 30 edges, 8 x 64 fp32, 61 us for a
// table's rows alone against 44.
inline GeoPick pick_sum_geo(int H, int D, int elem, int slot_align) { return pick_geo(H, D, elem, slot_align, true, true); }

// Whether an edge's scalars (per_edge of them, elem bytes each) are whole 16-byte pieces for every block of heads
inline bool wide_scalars(const GeoPick& p, const void* base, int per_edge, int elem) {
  return p.LT > 0 && p.parts == 1 && ((uintptr_t)base & 15) == 0 && (long long)per_edge * elem % 16 == 0;
}

constexpr int kMaxHeadBlocks = 65535;   // grid.y

template <class X> struct TypeTag { using type = X; };

// Calls f(TypeTag<Geo<...>>) for the geometry.  kNarrowSlots: slots of 8 and 4 bytes are instantiated too; kWide: heads of more
// than 32 slots (an op that may split them never has one).  A whole warp with one slot per lane is for 2-byte elements.  The
// compile-time lane counts cover the heads of 16 to 128 features of the common shapes; every other one reads L.
template <typename T, bool kNarrowSlots, bool kWide, class F>
inline int dispatch_geo(const GeoPick& p, F&& f) {
#define GK_GEO(SB_, G_, W_, LT_) \
  if (p.SB == SB_ && p.G == G_ && p.W == W_ && (LT_ == 0 || p.LT == LT_)) return f(TypeTag<Geo<T, SB_, G_, W_, LT_>>{});
  if constexpr (sizeof(T) <= 4) {
    if constexpr (sizeof(T) == 4) {
      GK_GEO(16, 16, 2, 2)
      GK_GEO(16, 16, 2, 4)
      GK_GEO(16, 16, 2, 8)
      GK_GEO(16, 16, 2, 16)
      GK_GEO(16, 8, 2, 2)
      GK_GEO(16, 8, 2, 4)
      GK_GEO(16, 8, 2, 8)
    }
    GK_GEO(16, 8, 1, 4)
    GK_GEO(16, 8, 1, 8)
    if constexpr (sizeof(T) == 2) {
      GK_GEO(16, 16, 1, 4)
      GK_GEO(16, 16, 1, 8)
      GK_GEO(16, 16, 1, 16)
    }
  }
  if constexpr (sizeof(T) == 2) {
    GK_GEO(16, 32, 1, 0)
    GK_GEO(16, 16, 1, 0)
  } else {
    GK_GEO(16, 16, 2, 0)
    GK_GEO(16, 8, 2, 0)
  }
  GK_GEO(16, 8, 1, 0)
  GK_GEO(16, 4, 1, 0)
  if constexpr (kWide) {
    GK_GEO(16, 32, 2, 0)
    GK_GEO(16, 32, 4, 0)
    GK_GEO(16, 32, 8, 0)
  }
  if constexpr (kNarrowSlots) {
    if constexpr (sizeof(T) == 2) {
      GK_GEO(8, 32, 1, 0)
      GK_GEO(8, 16, 1, 0)
    } else {
      GK_GEO(8, 16, 2, 0)
      GK_GEO(8, 8, 2, 0)
    }
    GK_GEO(8, 8, 1, 0)
    GK_GEO(8, 4, 1, 0)
    if constexpr (kWide) {
      GK_GEO(8, 32, 2, 0)
      GK_GEO(8, 32, 8, 0)
    }
    if constexpr (sizeof(T) <= 4) {
      if constexpr (sizeof(T) == 2) {
        GK_GEO(4, 32, 1, 0)
        GK_GEO(4, 16, 1, 0)
      } else {
        GK_GEO(4, 16, 2, 0)
        GK_GEO(4, 8, 2, 0)
      }
      GK_GEO(4, 8, 1, 0)
      GK_GEO(4, 4, 1, 0)
      if constexpr (kWide) {
        GK_GEO(4, 32, 2, 0)
        GK_GEO(4, 32, 8, 0)
      }
    }
  }
#undef GK_GEO
  return GRAPHOP_ERR_UNSUPPORTED;
}
// The same for the summing walker.
template <typename T, bool kNarrowSlots, class F>
inline int dispatch_sum_geo(const GeoPick& p, F&& f) {
#define GK_GEO(SB_, G_, LT_) \
  if (p.SB == SB_ && p.G == G_ && p.W == 1 && (LT_ == 0 || p.LT == LT_)) return f(TypeTag<Geo<T, SB_, G_, 1, LT_>>{});
  if constexpr (sizeof(T) == 4) {
    GK_GEO(16, 32, 4)
    GK_GEO(16, 32, 8)
    GK_GEO(16, 32, 16)
    GK_GEO(16, 32, 32)
    GK_GEO(16, 16, 4)
    GK_GEO(16, 16, 8)
    GK_GEO(16, 16, 16)
    GK_GEO(16, 8, 4)
    GK_GEO(16, 8, 8)
  }
  GK_GEO(16, 32, 0)
  GK_GEO(16, 16, 0)
  GK_GEO(16, 8, 0)
  GK_GEO(16, 4, 0)
  if constexpr (kNarrowSlots) {
    GK_GEO(8, 32, 0)
    GK_GEO(8, 16, 0)
    GK_GEO(8, 8, 0)
    GK_GEO(8, 4, 0)
    if constexpr (sizeof(T) == 4) {
      GK_GEO(4, 32, 0)
      GK_GEO(4, 16, 0)
      GK_GEO(4, 8, 0)
      GK_GEO(4, 4, 0)
    }
  }
#undef GK_GEO
  return GRAPHOP_ERR_UNSUPPORTED;
}
// the narrow-slot set has no 32 x 4: such rows take 32 x 8
inline GeoPick narrow_fix(GeoPick p) {
  if (p.SB && p.SB < 16 && p.G == 32 && p.W == 4) p.W = 8;
  return p;
}

// workspace of the carry slots: records of `carry_elems` accumulators and their ids, two per tile and head block
inline size_t carry_bytes(long long tiles, int nhb, long long carry_elems, size_t acc) {
  const size_t slots = (size_t)nhb * 2 * tiles;
  return align_up(slots * (size_t)carry_elems * acc) + align_up(slots * 4);
}

template <class GEO>
inline void fill_geo(GEO& op, const GeoPick& p, int H, int D) {
  op.H = H; op.D = D; op.HD = H * D; op.L = p.L; op.parts = p.parts;
  op.drowb = (unsigned)(D * (int)sizeof(typename GEO::T));
  op.rowb = (unsigned)H * op.drowb;
}

// Dynamic shared memory above 48 KB is asked for once per device and kernel; several host threads may get here at once
// (autograd's backward thread): setting the attribute twice is harmless, the flag only saves the call.
template <class Kernel>
inline int allow_smem(Kernel kernel, int bytes, std::atomic<bool> (&configured)[64]) {
  if (bytes <= 48 * 1024) return GRAPHOP_OK;
  int dev = 0;
  GK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    GK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  return GRAPHOP_OK;
}

// How many of the graph's tiles a lane group walks as one.  A tile begins with a chain of dependent loads (boundaries, nodes
// and endpoints, the first rows) and ends in carry records; with the head blocks of a wide row the smallest tiles make far
// more warps than it takes to fill the chip.  About kWarpsWanted warps leave every SM six rounds or more of them.  Step times
// with a tile each and with about 16 K, 20 K and 40 K warps: 15360 nodes of 30 edges, 8 x 64 fp32, three Functions 811 / 747 /
// - / 811 us; R-MAT 18 with an edge term, 4 x 64 bf16, 2.79 / 2.58 / 2.59 / 2.79 ms; R-MAT 20, 4 x 32, multiply and aggregate
// 5.84 / - / 5.70 / 5.84; R-MAT 22, 1 x 128, aggregate 13.5 / - / 12.7 / 12.5; with 4 K the chip is not filled evenly (R-MAT
// 18: 3.0 ms).
//
// The summing walker's warps run in step on a small graph, and what counts is how many rounds of the resident ones (`slots`: what
// the launch bounds of its kernels allow, which use their registers up) they are.  Whole rounds are best, and a part of one just
// above a whole one is worst: kernel times by rounds, 15360 nodes of 30 edges, 8 x 64 fp32, 15.8 / 3.9 / 3.2 / 2.6 / 2.0 / 1.6 / 1.3 /
// 0.98 / 0.66 108 / 69 / 73 / 69 / 63 / 69 / 77 / 62 / 75 us.  So the warps are cut to one round, and to two where one round would
// make them long (a warp inside hubs then ends last).  441 graphs of 1.1 to 25 rounds (blocks of 30, 16 and 50 random sources per
// node, uniform, skewed; 1 to 8 blocks of heads), time over the best of the spans tried, mean and worst: a tile each 1.28, 1.90;
// one round up to 4 and else two 1.03, 1.19 (at 4.1 rounds: 1.4 are left); up to 8 1.015, 1.12; up to 12 1.008, 1.12; always one
// 1.006, 1.19 (skewed, 15 rounds).  The source side alone, 100 graphs: the same order.  Larger graphs get tiles of more than
// kSmallestTile.
//
// The nodes of neighbouring tiles often gather the same rows (blocks, bands).  Where the tables do not fit the L2 as they are,
// the warps at work had better lie close together: `most` (0: any number) is two.  That goes by the tables' size alone for the
// gathering walker, skewed or not; the summing walker has no limit on skewed graphs and two on tables of few rows
// (choose_walker).  Where a plan says that no row is cut there are no records to save, and the gathering walker stays with a tile
// each: 900 thousand nodes in blocks of 50, 1 x 64 fp32, backward 1.84 + 1.66 ms, with two 1.93 + 2.17; 9.6M uniform edges on 2M
// nodes, 2 x 64, 1.71 + 2.07 + 1.98 ms against 1.75 + 2.09 + 2.01.  331
// thousand nodes in blocks of 47, 4 x 64 fp32, backward: 2.36 + 1.95 ms with a tile each, 2.83 + 2.37 with three; a row of 7M
// edges on 1M nodes, 2 x 64: its records take 326 us to merge with a tile each, 168 with two.
constexpr long long kWarpsWanted = 20480;
constexpr int kOneRound = 12;
constexpr long long kL2Table = 64ll << 20;
inline int tiles_near(long long table) { return table > kL2Table ? 2 : 0; }
inline unsigned tile_span(long long n_tiles, int nhb, int per_warp, int tile, long long slots, int most) {
  const long long warps = (n_tiles * nhb + per_warp - 1) / per_warp;
  long long span = (warps + kWarpsWanted / 2) / kWarpsWanted;
  if (most) {
    span = span < most ? span : most;
  } else if (slots && tile == kSmallestTile) {
    const long long round = warps <= kOneRound * slots ? slots : 2 * slots;
    span = (warps + round - 1) / round;
  }
  return span < 1 ? 1 : span < n_tiles ? (unsigned)span : (unsigned)n_tiles;
}

// The most tiles that a lane group of the summing walker takes as one.  A run of n edges there is a second level of n / G blocks
// of G positions one after the other: squared rounding errors that add up to n G^2 / 3 + n^3 / 3G of a single one's.  In pieces
// of a tile of t positions, one after the other too, they are n t^2 / 3 + n^3 / 3t: the walk is not the worse of the two up to
// n = t sqrt(t G / (t - G)).  (6 tiles of 256 for rows of 512 bytes.  2000 nodes of 2000 edges, 1 x 8192 fp32: 1.02e-7 off float64
// with 98 tiles in a walk.)
inline unsigned sum_span(int t, int G) {
  unsigned span = 1;
  while (t > G && (long long)(span + 1) * (span + 1) * (t - G) <= (long long)t * G) ++span;
  return t > G ? span : ~0u;
}

// The op over every position and head block, and the merge of the rows that tiles had to cut.  most: see tile_span; only: see
// WalkArgs.
template <class Op>
inline int launch_walk(Arena& ar, const GraphView& g, const GeoPick& p, const Op& op, long long n_rows, int most,
                       cudaStream_t st, int only = -1) {
  WalkArgs a{};
  a.hdr = g.hdr; a.erow = g.erow; a.other = g.other; a.eid = g.eid;
  a.tile_start = g.tile_start;
  a.E = g.E; a.n_rows = n_rows; a.tile = g.tile; a.aligned = g.aligned; a.only = only;
  a.cut_tiles = (unsigned)g.n_tiles;
  a.span = tile_span(g.n_tiles, p.nhb, Op::NE, g.tile, Op::kSums ? 148ll * Op::kMinCtas * Op::kWarps : 0,
                     most && g.no_carry && !Op::kSums ? 1 : most);
  if (Op::kSums) a.span = a.span < sum_span(g.tile, Op::G) ? a.span : sum_span(g.tile, Op::G);
  a.n_tiles = (a.cut_tiles + a.span - 1) / a.span;
  const bool cuts = Op::kRowOut && !g.no_carry;
  if (cuts) {
    const size_t slots = (size_t)p.nhb * 2 * a.n_tiles;
    a.carry = ar.take(slots * Op::kCarryElems * sizeof(typename Op::A));
    a.rows = (uint32_t*)ar.take(slots * 4);
  }
  if (!ar.base) return GRAPHOP_OK;
  if (ar.overflow) return GRAPHOP_ERR_WORKSPACE;
  {
    constexpr int smem = Op::kWarps * Op::kWarpBytes, per_block = Op::kWarps * Op::NE;   // one tile per lane group
    const dim3 grid((a.n_tiles + per_block - 1) / per_block, (unsigned)p.nhb);
    const auto launch = [&](void (*kernel)(const Op, const WalkArgs), std::atomic<bool> (&configured)[64]) -> int {
      GK_TRY(allow_smem(kernel, smem, configured));
      kernel<<<grid, Op::kWarps * 32, smem, st>>>(op, a);
      GK_LAUNCHED(Op::kName);
      return GRAPHOP_OK;
    };
    static std::atomic<bool> configured[64];
    if constexpr (Op::kSums) {
      GK_TRY(launch(sum_walk_kernel<Op>, configured));
    } else {
      bool pieces = false;
      if constexpr (Op::kRowOut) {
        static std::atomic<bool> configured_pieces[64];
        pieces = cuts && a.span > 1;
        if (pieces) GK_TRY(launch(group_walk_kernel<Op, true>, configured_pieces));
      }
      if (!pieces) GK_TRY(launch(group_walk_kernel<Op, false>, configured));
    }
  }
  if constexpr (Op::kRowOut) {
    if (cuts) {
      static std::atomic<bool> configured[64];
      constexpr int threads = kCarryThreads<Op>, smem = threads / Op::G * Op::kCarryElems * (int)sizeof(typename Op::A);
      GK_TRY(allow_smem(carry_rows_kernel<Op>, smem, configured));
      const dim3 grid((2 * a.n_tiles + threads - 1) / threads, (unsigned)p.nhb);
      carry_rows_kernel<Op><<<grid, threads, smem, st>>>(op, a);
      GK_LAUNCHED("carry_rows");
    }
  }
  return GRAPHOP_OK;
}

}  // namespace gk
