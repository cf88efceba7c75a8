// The gathering walker: row-owned reductions and per-edge products over a CSR position stream.
//
// Decomposition (as in gk_common.cuh): the positions 0..E-1 are cut into tiles of equal cost (cut_tiles), so the work of a
// tile does not depend on the degrees.  A warp is NE = 32 / G groups of G lanes and every group walks a tile of its own:
//   * A step folds one position per group.  A lane owns W slots (16, 8 or 4 bytes each) of one head of the row, a row of
//     128 bytes is 8 lanes: four edges per step share the address arithmetic, shuffles, exponentials and loop work that one
//     edge spread over 32 lanes would need alone.  Groups never exchange partial results: a node's edges are folded by the
//     group whose tile they lie in, one after the other.
//   * Where a node ends and the next begins, the groups concerned store and begin inside one branch that the warp takes
//     when any of its groups needs it; short rows therefore cost one pass through that branch for several groups, not one each.
//   * Only as many heads as a group is wide are walked at a time; blockIdx.y counts these head blocks.  Rows of several KB
//     run the same narrow code at full occupancy, and one head block's share of the gathered tensor is what competes for
//     the L2 at a time.
//   * The gathered rows come through a ring of kDepth steps per warp in shared memory (cp.async; each lane reads back the
//     bytes it copied itself, so no barriers), and so do the rows of the node that begins at a position: a node's start
//     waits for nothing.  Per-edge scalars (weights, probabilities, statistics) come through a table,
//     copied for a block of G positions at a time, one position per lane; node, other endpoint and edge id of the next
//     positions sit in registers, one per lane.
//   * Tiles have equal cost (cut_tiles) and begin at row starts wherever a row is no longer than a tile.  A longer row is
//     cut: every tile leaves the partials of its open first / last segment in two carry slots, and a second launch
//     merges each such row's partials in tile order.  Every sum is a function of the graph and the tile cost alone:
//     results are bit-reproducible, and no warp waits for another.
//   * A group may walk several tiles as one (`span`).  A row that the tiles cut is summed in the pieces they make of it all the
//     same (kPieces): where one ends, the sum so far goes to the walk's carry slot and the next starts from zero, so that no
//     chain of adds is longer than a tile whatever the span.  o of 16384 nodes of 1000 edges, 8 x 64 fp32, is 6.8e-7 off
//     float64 with six tiles in one chain and 3.8e-7 in pieces, as with a tile per walk.
#pragma once
#include <type_traits>

#include "gk_frag.cuh"
#include "gk_ops.cuh"

namespace gk {

// BYTES from global to shared memory; live = false: nothing is read, the destination becomes zeros
template <int BYTES>
__device__ __forceinline__ void cp_async_slot(unsigned s, const void* g, bool live) {
  const int n = live ? BYTES : 0;
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(g), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr uint32_t kNoRow = 0xffffffffu;
constexpr int kMaxBlockHeads = 8;   // heads per block at most

// What a launch of the walker sees of the graph and of the carry records.
struct WalkArgs {
  const PlanHeader* hdr;
  const int32_t* erow;
  const int32_t* other;
  const int32_t* eid;          // null: an edge's id is its position
  const int32_t* tile_start;   // (cut_tiles + 1) boundaries
  long long E, n_rows;
  int tile;                    // nominal cost of a tile; rows at least this long may be cut
  int aligned;                 // the boundaries are row starts already wherever a row can be kept whole
  unsigned cut_tiles, span;    // tiles the graph was cut into; `span` consecutive ones are one tile of this launch
  unsigned n_tiles;            // tiles of this launch
  void* carry;                 // (head blocks, 2 * n_tiles) partial records; null: no row crosses a tile boundary
  int only;                    // 0 / 1: nothing is done unless hdr->skewed is that; -1: always
  uint32_t* rows;              // what each record stands for: 2 * node + 1, 2 * node where the slot holds nothing (its tile
                               // lies inside one node that goes on), kNoRow: unused
};

// ---------------------------------------------------------------------------------------
// geometry: which part of a row a lane owns
// ---------------------------------------------------------------------------------------
// SB bytes per slot, G lanes per edge, W slots per lane.  LT > 0: lanes per head known at compile time, and every slot
// of every lane exists (D is exactly LT * W slots and the heads fill the blocks); LT = 0: read at run time, with tests.
template <typename T_, int SB_, int G_, int W_, int LT_>
struct Geo {
  using T = T_;
  using A = typename AccOf<T>::type;
  static constexpr int SB = SB_, G = G_, W = W_, LT = LT_, V = SB / (int)sizeof(T), NE = 32 / G;
  using F = Frag<A, V>;
  using Word = typename SlotWord<SB>::type;
  static constexpr int kAccs = W * V * G;   // accumulators of one row of a head block
  static constexpr int kRow = W * 32 * SB;  // ring bytes of one operand row per group
  static constexpr int kHeads = LT > 0 ? G / LT : (G < kMaxBlockHeads ? G : kMaxBlockHeads);   // heads (or pieces) per block at most
  static constexpr bool kAllHeads = false;
  int H, D, HD;
  unsigned rowb, drowb;   // bytes of a node row and of a D-vector
  int L;        // lanes per head, a power of two, at most G
  int parts;    // pieces a head is cut into when it is wider than a block (aggregations only), else 1
  struct Lane {
    int head, part;
    unsigned ok;         // bit i: slot i exists
    unsigned off, eoff;  // element offsets of slot 0 inside the node row / inside a D-vector; slot i: + i * L * V
    bool first;          // the head's first lane
  };
  __device__ __forceinline__ int lanes_per_head() const { return LT > 0 ? LT : L; }
  __device__ __forceinline__ int slot_step() const { return lanes_per_head() * V; }   // elements
  __device__ __forceinline__ int block_heads() const { return G / lanes_per_head(); }   // heads (or pieces) per block
  __device__ __forceinline__ int scalar_at(int gl) const { return gl / lanes_per_head(); }   // this lane's first head
  __device__ __forceinline__ Lane lane_of(int gl, int hb) const {
    Lane ln;
    const int l = lanes_per_head();
    const int hl = gl / l, sub = gl - hl * l;   // powers of two
    const int ph = hb * (G / l) + hl;
    ln.head = parts == 1 ? ph : ph / parts;
    ln.part = parts == 1 ? 0 : ph - ln.head * parts;
    const int e0 = (ln.part * l * W + sub) * V;
    ln.ok = 0;
#pragma unroll
    for (int i = 0; i < W; ++i)
      if (LT > 0 || (ln.head < H && e0 + i * l * V < D)) ln.ok |= 1u << i;
    if (LT == 0 && ln.ok == 0) ln.head = 0;   // a lane without a slot still forms addresses of scalars
    ln.eoff = (LT > 0 || ln.ok) ? e0 : 0;
    ln.off = (unsigned)ln.head * D + ln.eoff;
    ln.first = sub == 0 && ln.part == 0 && ln.ok != 0;
    return ln;
  }
  __device__ __forceinline__ bool has(const Lane& ln, int i) const { return LT > 0 || ((ln.ok >> i) & 1u); }
  __device__ __forceinline__ A head_sum(A v) const {
    if constexpr (LT > 0) {
#pragma unroll
      for (int o = 1; o < LT; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
    } else {
      for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
    }
    return v;
  }
  // The dot product of two rows with the sum formed slot by slot: the elements of a slot in order, then a butterfly over
  // the slots of the head, neighbours first.  The result does not depend on how many slots a lane owns (1 or 2), so a
  // score is the same number whatever geometry its row shape gets.  Two slots per lane: the lanes of a pair first hand
  // each other one of their two partial sums (one shuffle instead of two), the even lanes carry the lower half of the
  // head on, the odd lanes the upper half, and the halves meet in the last step.
  __device__ __forceinline__ A ordered_dot(const F (&a)[W], const F (&b)[W]) const {
    A p[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
      A x[V], y[V];
      a[i].get(x);
      b[i].get(y);
      p[i] = x[0] * y[0];
#pragma unroll
      for (int j = 1; j < V; ++j) p[i] = fma(x[j], y[j], p[i]);
    }
    if constexpr (W == 2) {
      const int l = lanes_per_head();
      if (l == 1) return p[0] + p[1];
      const bool odd = (threadIdx.x & 1) != 0;
      A keep = odd ? p[1] : p[0];
      keep += __shfl_xor_sync(kFull, odd ? p[0] : p[1], 1);
      if constexpr (LT > 0) {
#pragma unroll
        for (int o = 2; o < LT; o <<= 1) keep += __shfl_xor_sync(kFull, keep, o);
      } else {
        for (int o = 2; o < l; o <<= 1) keep += __shfl_xor_sync(kFull, keep, o);
      }
      return keep + __shfl_xor_sync(kFull, keep, 1);
    } else {
      A s = p[0];
#pragma unroll
      for (int i = 1; i < W; ++i) s += p[i];
      return head_sum(s);
    }
  }
  // copy a row's slots of this lane: base = the tensor at the lane's slot 0, id = row, rowb = bytes per row.  Nothing is
  // read where live is false or the slot does not exist: those ring bytes become zeros, so that whatever is multiplied
  // with them adds nothing
  __device__ __forceinline__ void stage_row(const Lane& ln, unsigned dst, const unsigned char* base, int id, unsigned rowb,
                                            bool live) const {
    const unsigned char* p = base + (unsigned long long)(unsigned)id * rowb;
#pragma unroll
    for (int i = 0; i < W; ++i)
      cp_async_slot<SB>(dst + i * 32 * SB, p + (size_t)(i * slot_step()) * sizeof(T), live && has(ln, i));
  }
  // the lane's first slot of a row, as it lies in memory; zeros where it does not exist
  __device__ __forceinline__ void fetch_slot(const Lane& ln, Word& w, const unsigned char* base, int id, unsigned rowb) const {
    if (LT == 0 && !has(ln, 0)) w = Word{};
    else ldg_word(w, base + (unsigned long long)(unsigned)id * rowb);
  }
  __device__ __forceinline__ void load_staged(F (&f)[W], unsigned src) const {
#pragma unroll
    for (int i = 0; i < W; ++i) frag_lds<T, SB>(f[i], src + i * 32 * SB);
  }
  __device__ __forceinline__ void store_row_slots(const Lane& ln, T* row, const F (&f)[W]) const {
#pragma unroll
    for (int i = 0; i < W; ++i)
      if (has(ln, i)) frag_stg<T, SB>(row + i * slot_step(), f[i]);
  }
  __device__ __forceinline__ void zero_slots(const Lane& ln, T* base, long long n) const {
    F z;
    z.zero();
#pragma unroll
    for (int i = 0; i < W; ++i)
      if (has(ln, i)) frag_stg<T, SB>(base + n * HD + ln.off + i * slot_step(), z);
  }
  __device__ __forceinline__ void save_acc(A* rec, int gl, const F (&f)[W]) const {
#pragma unroll
    for (int i = 0; i < W; ++i) frag_save<A, V>(rec + (i * G + gl) * V, f[i]);
  }
  __device__ __forceinline__ void load_acc_raw(F (&f)[W], const A* rec, int gl) const {
#pragma unroll
    for (int i = 0; i < W; ++i) frag_load_raw<A, V>(f[i], rec + (i * G + gl) * V);
  }
};

// Rows that all heads of a node share (one D-vector per edge): G lanes, one slot each, with the accumulators of all W heads
// in a lane.  A row is copied once instead of once per head.
template <typename T_, int G_, int W_>
struct FeatGeo : Geo<T_, 16, G_, W_, G_> {
  using Base = Geo<T_, 16, G_, W_, G_>;
  using T = T_;
  using A = typename Base::A;
  using F = typename Base::F;
  using Lane = typename Base::Lane;
  static constexpr int G = G_, W = W_, V = Base::V;
  static constexpr int kRow = 32 * 16, kHeads = W_;
  static constexpr bool kAllHeads = true;
  __device__ __forceinline__ int block_heads() const { return W; }
  __device__ __forceinline__ int scalar_at(int) const { return 0; }
  __device__ __forceinline__ Lane lane_of(int gl, int) const {
    Lane ln;
    ln.head = ln.part = 0;
    ln.ok = 1;
    ln.off = ln.eoff = (unsigned)(gl * V);
    ln.first = gl == 0;
    return ln;
  }
  __device__ __forceinline__ void stage_row(unsigned dst, const unsigned char* base, int id, unsigned rowb, bool live) const {
    cp_async_slot<16>(dst, base + (unsigned long long)(unsigned)id * rowb, live);
  }
  __device__ __forceinline__ void store_row_slots(T* row, const F (&f)[W]) const {
#pragma unroll
    for (int i = 0; i < W; ++i) frag_stg<T, 16>(row + i * this->D, f[i]);
  }
};

// Launch shape of an op with kRows operand rows per ring step.  One warp per block: warps are independent and their tiles
// take different times, a block of several would hold its slot until the slowest is done.
// A ring step holds kRows operand rows of a position's edge and, should a node begin there, kNode rows and kNodeScalar bytes
// per lane of it.  kShare: the kUnroll steps of an iteration have room for one node together (a second one, after a node of
// one edge, is fetched when its turn comes), where a room per step would leave too few warps.  kScalar bytes per edge and head wait in a table; kState fragments of W slots live in a lane's registers.
template <class GEO, int kRows, int kScalar, int kState, int kNode, int kNodeScalar, int kU, bool kShare = false>
struct Shape {
  static constexpr bool kSums = false;
  static constexpr bool kOptional = false;   // may be one of two walkers launched for the same sums
  static constexpr int kWarps = 1;
  static constexpr int kStepBytes = kRows * GEO::kRow;
  static constexpr int kNodeScalarAt = kNode * GEO::kRow;                  // from the node's room
  // Positions folded per iteration: two share the loop, the waits and the checks and give the scheduler two independent
  // chains; one where the step's rows or the registers would leave too few warps.  Two iterations are in flight.
  static constexpr int kUnroll = GEO::W <= 2 || GEO::kAllHeads ? kU : 1;
  static constexpr int kDepth = 2 * kUnroll;
  static constexpr int kNodeAt = kUnroll * kStepBytes;                     // from the iteration's first step
  static constexpr int kNodeBytes = kNodeScalarAt + 32 * kNodeScalar;
  static constexpr bool kShareNode = kShare && kUnroll > 1;
  static constexpr int kIterBytes = kNodeAt + (kShareNode ? 1 : kUnroll) * kNodeBytes;
  // where the node that begins at step v waits
  __device__ __forceinline__ static constexpr unsigned node_at(int v) { return kNodeAt + (kShareNode ? 0 : v * kNodeBytes); }
  static constexpr int kScalarBytes = kScalar;
  static constexpr int kTable = 32 * GEO::kHeads * kScalar;                // one block of positions
  static constexpr int kWarpBytes = 2 * kIterBytes + 2 * kTable;
  static constexpr bool kNodeRows = kNode > 0;
  static constexpr int kFit = 226 * 1024 / (kWarps * kWarpBytes + 1024);   // blocks the shared memory allows
  static constexpr int kWords = GEO::W * GEO::V * (int)sizeof(typename GEO::A) / 4;
  static constexpr int kRegs = 50 + kWords * (GEO::kAllHeads ? kState + 1 : kState + 2);
  static constexpr int kRegFit = 65536 / 32 / (kRegs < 64 ? 64 : kRegs > 255 ? 255 : kRegs);
  static constexpr int kMinCtas = kFit < kRegFit ? kFit : kRegFit;
};

// Two walkers are launched where the better one is known on the device alone: one of them has nothing to do.  Ops that are never
// one of two do not ask (in their merge kernel the question alone took the loads of records apart: 17804 nodes, 82 thousand skewed
// edges, 8 x 64 bf16, destination side, 8.9 -> 15.6 us).
template <class Op>
__device__ __forceinline__ bool not_asked(const WalkArgs& a) { return Op::kOptional && a.only >= 0 && a.hdr->skewed != a.only; }

// The positions of tile t of a launch, for the lane group that walks it (called by the whole warp; here: the tile exists).  A
// nominal boundary moves up to the first row start within the following `tile` positions, so that only rows longer than a
// tile are ever cut (in a plan's boundaries that is done; else every group looks for its own).
template <int G>
__device__ __forceinline__ void tile_of(const WalkArgs& a, unsigned t, bool here, int& begin, int& n) {
  const int lane = threadIdx.x & 31, g = lane / G, gl = lane & (G - 1);
  const unsigned cut0 = here ? t * a.span : 0u, cut1 = here ? min(cut0 + a.span, a.cut_tiles) : 0u;
  begin = __ldg(a.tile_start + cut0);
  int end = __ldg(a.tile_start + cut1);
  if (!a.aligned) {
    const int E = (int)a.E;
    const auto move_up = [&](int x) {
      int found = x <= 0 ? 0 : x >= E ? E : -1;
      for (int s = 0; s < a.tile; s += G) {
        if (__all_sync(kFull, found >= 0)) break;
        const bool in = found < 0 && s + gl < a.tile && s + gl < E - x;
        const bool starts = in && __ldg(a.erow + x + s + gl) != __ldg(a.erow + x + s + gl - 1);
        const unsigned m = (__ballot_sync(kFull, starts) >> (g * G)) & (kFull >> (32 - G));
        if (found < 0 && m) found = x + s + __ffs(m) - 1;
      }
      return found >= 0 ? found : x;
    };
    begin = move_up(begin);
    end = move_up(end);
  }
  n = here ? end - begin : 0;
}

// Whether the graph's tiles cut the row of position j there (r: its node, also that of the position before): a boundary lies
// where the cost reaches it (cut_tiles), and it has stayed there if no row starts within the following tile (tile_of).
__device__ __forceinline__ bool cut_inside(const WalkArgs& a, unsigned j, int r) {
  if (r < 0 || ((j + (unsigned)kRowCost * (unsigned)r) & (unsigned)(a.tile - 1))) return false;
  const unsigned last = j + (unsigned)a.tile - 1, E = (unsigned)a.E;
  return __ldg(a.erow + (last < E ? last : E - 1)) == r;
}

// Op interface (all members __device__), on top of its Geo and Shape; `slot` is the ring step's memory at this lane:
//   kRowOut, kUsesOther, kUsesEid, kFoldsEid; State, Carry
//   setup(st, gl, hb)
//   stage(st, slot, id, edge, live)               copy the rows of (other endpoint, edge) into the ring
//   scalar_of(h, id, edge)                        where the edge's scalars of head h are
//   fold<N>(st, slot, tab, active, pos, edge)     fold N = 1 or 2 positions per group (called by the whole warp); tab: the
//                                                 table's entry of the first position and this lane's head
//   stage_node(st, buf, lane, node)               copy what begin(node) will read into the node buffer
//   begin(st, buf, lane)                          a node begins (called by the groups concerned)
//   began(st, node, mine)                         the part of begin that needs the whole warp
//   store_row(st, node), zero_row(st, node)
//   begin_merge(st), merge(st, Carry), load_carry, save_carry, kCarryElems
//
// kPieces: walks of several tiles on a graph whose rows the tiles may cut.  A kernel of its own, because the few instructions
// per block and per node that it has more cost 2 to 5 % where there is nothing to cut (the loop is bound by issue and its code
// by the instruction cache; the same tests behind a flag cost as much).
template <class Op, bool kPieces>
__global__ void __launch_bounds__(Op::kWarps * 32, Op::kMinCtas)
group_walk_kernel(const __grid_constant__ Op op, const __grid_constant__ WalkArgs a) {
  constexpr int NE = Op::NE, G = Op::G, DS = Op::kDepth, CH = G / DS, STEP = Op::kStepBytes, ITER = Op::kIterBytes, U = Op::kUnroll;   // CH ring turns per G positions
  static_assert(CH * DS == G, "whole ring turns per block of positions");
  constexpr unsigned kOneLane = NE == 1 ? 1u : NE == 2 ? 0x00010001u : NE == 4 ? 0x01010101u : 0x11111111u;
  constexpr bool kOut = Op::kRowOut;
  extern __shared__ uint4 gk_ring[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane / G, gl = lane & (G - 1);
  const int hb = blockIdx.y;
  const unsigned t0 = (blockIdx.x * Op::kWarps + w) * NE;   // the warp's first tile
  if (t0 >= a.n_tiles || not_asked<Op>(a)) return;
  const unsigned t = t0 + g;
  const bool here = t < a.n_tiles;
  int begin, n;   // the group's first position and their number
  tile_of<G>(a, t, here, begin, n);
  const long long j0 = begin, j1 = j0 + n;
  int longest = n;
#pragma unroll
  for (int o = G; o < 32; o <<= 1) {
    const int x = __shfl_xor_sync(kFull, longest, o);
    longest = x > longest ? x : longest;
  }

  typename Op::State st;
  op.setup(st, gl, hb);
  if constexpr (kOut) {
    if (t0 == 0 && a.hdr->cover_hi <= a.hdr->cover_lo)   // no covered position at all
      for (long long r = g; r < a.n_rows; r += NE) op.zero_row(st, r);
  }

  // a block of G positions per group in registers: node (-1: none, -2: past the tile), staging key (-1: nothing to
  // copy), edge id
  auto load_block = [&](int b, int& r, int& o, int& e) {
    const int i = b * G + gl;
    const bool in = i < n;
    r = in ? __ldg(a.erow + j0 + i) : -2;
    e = Op::kUsesEid ? (in ? (a.eid ? __ldg(a.eid + j0 + i) : (int)(j0 + i)) : 0) : 0;
    o = Op::kUsesOther ? (in ? __ldg(a.other + j0 + i) : 0) : 0;
    if (r < 0) { o = -1; e = 0; }
  };
  // bit of every lane whose position (of block b) starts another row than the position before it, or another piece of its row
  auto starts_of = [&](int b, int r, int before_block) {
    int up = __shfl_up_sync(kFull, r, 1, G);
    if (gl == 0) up = before_block;
    bool starts = r != up;
    if constexpr (kPieces)
      if (!starts) starts = cut_inside(a, (unsigned)begin + b * G + gl, r);
    return __ballot_sync(kFull, starts);
  };
  int r0, o0, e0, r1, o1, e1;
  load_block(0, r0, o0, e0);
  load_block(1, r1, o1, e1);
  const int before = here && j0 > 0 ? __ldg(a.erow + j0 - 1) : -1;
  unsigned starts0 = starts_of(0, r0, -3);

  const unsigned ring = (unsigned)__cvta_generic_to_shared(gk_ring) + w * Op::kWarpBytes + lane * Op::SB;
  // start the copies of positions i .. i + U - 1 of a block (its registers r, o, e and start bits) into U ring steps
  auto stage_some = [&](unsigned slot, int i, int r, int o, int e, unsigned starts) {
#pragma unroll
    for (int v = 0; v < U; ++v) {
      const int oo = __shfl_sync(kFull, o, i + v, G);
      const int ee = Op::kUsesEid ? __shfl_sync(kFull, e, i + v, G) : 0;
      op.stage(st, slot + v * STEP, oo < 0 ? 0 : oo, ee, oo >= 0);
    }
    if constexpr (Op::kNodeRows) {
      const unsigned m = starts >> i;
      if (m & (((1u << U) - 1u) * kOneLane)) {
        bool taken = false;
#pragma unroll
        for (int v = 0; v < U; ++v) {
          const int rr = __shfl_sync(kFull, r, i + v, G);
          const bool begins = ((m >> (g * G + v)) & 1u) && rr >= 0;
          if (begins && !(Op::kShareNode && taken)) op.stage_node(st, slot + Op::node_at(v), lane, rr);
          taken = taken || begins;
        }
      }
    }
    cp_async_commit();
  };
  // The scalars of a block of positions, one position per lane: asked for while the block before it is folded, read
  // by all lanes of the group afterwards.  cp.async moves 4 bytes at least: 2-byte scalars wait in registers meanwhile.
  constexpr int SC = Op::kScalarBytes, TB = Op::kTable, ENTRY = Op::kHeads * SC;
  const unsigned table = ring - lane * Op::SB + 2 * ITER;
  uint16_t held[SC == 2 ? Op::kHeads : 1];
  auto fetch_scalars = [&](unsigned tab, int o, int e) {
    if constexpr (SC > 0) {
      const int per = op.block_heads(), pieces = op.parts * op.H - hb * per;   // heads in this block
#pragma unroll
      for (int k = 0; k < Op::kHeads; ++k) {
        const bool live = o >= 0 && k < per && k < pieces;
        const int ph = live ? hb * per + k : 0;
        const void* src = op.scalar_of(op.parts == 1 ? ph : ph / op.parts, live ? o : 0, live ? e : 0);
        if constexpr (SC == 2) held[k] = live ? __ldg(reinterpret_cast<const uint16_t*>(src)) : (uint16_t)0;
        else cp_async_slot<SC>(tab + lane * ENTRY + k * SC, src, live);
      }
    }
  };
  auto publish_scalars = [&](unsigned tab) {
    if constexpr (SC == 2) {
#pragma unroll
      for (int k = 0; k < Op::kHeads; ++k)
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(tab + lane * ENTRY + k * SC), "h"(held[k]) : "memory");
    }
  };
  fetch_scalars(table, o0, e0);
  publish_scalars(table);
  const unsigned my_scalar = table + g * G * ENTRY + (SC > 0 ? op.scalar_at(gl) * SC : 0);
  static_assert(DS == 2 * U, "two iterations in flight");
  stage_some(ring, 0, r0, o0, e0, starts0);
  stage_some(ring + ITER, U, r0, o0, e0, starts0);

  const int first = __shfl_sync(kFull, r0, 0, G);
  const bool head_open = before >= 0 && before == first;
  bool first_seg = true;
  int cur = -1, last_valid = before;
  int lim = 0;   // positions below lim are folded: the tile's length while a node is open, else 0
  typename Op::A* rec = nullptr;
  if constexpr (kOut)
    rec = reinterpret_cast<typename Op::A*>(a.carry) + ((size_t)hb * 2 * a.n_tiles + 2 * (size_t)t) * Op::kCarryElems;
  uint32_t head_id = kNoRow, tail_id = kNoRow;
  // The open node's earlier pieces wait in the slot that the whole of it goes to if it stays open: the head slot for one that
  // began in an earlier tile, else the tail slot, which nothing else needs before the walk's end.
  [[maybe_unused]] bool kept = false;
  [[maybe_unused]] const auto piece_slot = [&] { return first_seg && head_open ? rec : rec + Op::kCarryElems; };
  [[maybe_unused]] const auto join_pieces = [&] {
    if (kept) {
      typename Op::Carry c;
      op.load_carry(c, piece_slot(), gl);
      op.merge(st, c);
      kept = false;
    }
  };

  for (int b = 0; b * G < longest; ++b) {
    int r2, o2, e2;
    load_block(b + 2, r2, o2, e2);
    if constexpr (SC > 0) {
      cp_async_wait<DS / U - 1>();
      __syncwarp();   // every lane's part of this block's table has landed, and nobody reads the other table any more
      fetch_scalars(table + ((b + 1) & 1) * TB, o1, e1);
    }
    const unsigned tab0 = my_scalar + (b & 1) * TB;
    const unsigned starts1 = starts_of(b + 1, r1, __shfl_sync(kFull, r0, G - 1, G));
#pragma unroll 1
    for (int c = 0; c < CH; ++c) {
      if (b * G + c * DS >= longest) break;
      const bool turn = c == CH - 1;
      const int rs = turn ? r1 : r0, os = turn ? o1 : o0, es = turn ? e1 : e0;
      const unsigned ss = turn ? starts1 : starts0;
      const int ahead = turn ? -c * DS : DS;   // from a position of this turn to the one staged in its place
      // one copy of the code for every two steps: with the ring unrolled the loop missed the instruction cache
      unsigned slot = ring;
#pragma unroll 1
      for (int i = c * DS; i < c * DS + DS; i += U, slot += ITER) {
        const int p = b * G + i;
        cp_async_wait<DS / U - 1>();
        const unsigned m = (starts0 >> i) & (((1u << U) - 1u) * kOneLane);
        if (m == 0) {
          bool act[U];
          int ed[U];
#pragma unroll
          for (int v = 0; v < U; ++v) {
            act[v] = p + v < lim;
            ed[v] = Op::kFoldsEid ? __shfl_sync(kFull, e0, i + v, G) : 0;
          }
          op.template fold<U>(st, slot, tab0 + i * ENTRY, act, (unsigned)j0 + p, ed);
        } else {
          [[maybe_unused]] bool taken = false;   // the iteration's room for a node held an earlier one
#pragma unroll 1
          for (int v = 0; v < U; ++v) {
            const unsigned mv = m >> v;
            if (mv & kOneLane) {   // some group's node ends here and another begins
              const int r = __shfl_sync(kFull, r0, i + v, G);
              const bool mine = ((mv >> (g * G)) & 1u) && r > -2;
              if constexpr (Op::kShareNode) {
                const bool late = mine && r >= 0 && taken;
                if (__any_sync(kFull, late)) {
                  if (late) op.stage_node(st, slot + Op::node_at(v), lane, r);
                  cp_async_commit();
                  cp_async_wait<0>();
                }
                taken = taken || (mine && r >= 0);
              }
              if (mine) {
                if constexpr (kOut) {
                  if (kPieces && cur >= 0) join_pieces();
                  if (kPieces && cur >= 0 && r == cur) {   // another piece of the same node
                    op.save_carry(st, piece_slot(), gl);
                    kept = true;
                  } else if (cur >= 0) {
                    if (first_seg && head_open) {
                      op.save_carry(st, rec, gl);
                      head_id = 2u * (unsigned)cur + 1u;
                    } else {
                      op.store_row(st, cur);
                    }
                    first_seg = false;
                    if (r < 0)   // coverage ended
                      for (long long z = (long long)cur + 1; z < a.n_rows; ++z) op.zero_row(st, z);
                  }
                  if (r >= 0) {
                    if (!(first_seg && head_open))
                      for (int z = last_valid + 1; z < r; ++z) op.zero_row(st, z);
                    last_valid = r;
                  }
                }
                if (r >= 0) op.begin(st, slot + Op::node_at(v), lane);
                cur = r;
                lim = r >= 0 ? n : 0;
              }
              __syncwarp();
              op.began(st, cur, mine && r >= 0);
            }
            const bool act[1] = {p + v < lim};
            const int ed[1] = {Op::kFoldsEid ? __shfl_sync(kFull, e0, i + v, G) : 0};
            op.template fold<1>(st, slot + v * STEP, tab0 + (i + v) * ENTRY, act, (unsigned)j0 + p + v, ed);
          }
        }
        stage_some(slot, i + ahead, rs, os, es, ss);
      }
    }
    publish_scalars(table + ((b + 1) & 1) * TB);
    r0 = r1; o0 = o1; e0 = e1;
    r1 = r2; o1 = o2; e1 = e2;
    starts0 = starts1;
  }
  cp_async_wait<0>();

  if constexpr (kOut) {
    if (cur >= 0) {
      if constexpr (kPieces) join_pieces();
      const int next = j1 < a.E ? __ldg(a.erow + j1) : -1;
      const bool tail_open = next == cur;
      if (first_seg && head_open) {   // the whole tile lies inside one node that started earlier
        op.save_carry(st, rec, gl);
        head_id = 2u * (unsigned)cur + 1u;
        if (tail_open) tail_id = 2u * (unsigned)cur;
      } else if (tail_open) {
        op.save_carry(st, rec + Op::kCarryElems, gl);
        tail_id = 2u * (unsigned)cur + 1u;
      } else {
        op.store_row(st, cur);
      }
      if (next < 0)   // last covered position
        for (long long z = (long long)cur + 1; z < a.n_rows; ++z) op.zero_row(st, z);
    }
    if (a.carry && here && gl == 0)
      *reinterpret_cast<uint2*>(a.rows + (size_t)hb * 2 * a.n_tiles + 2 * (size_t)t) = make_uint2(head_id, tail_id);
  }
}

// Second launch, where rows may cross tile boundaries: every such row's records are merged in tile order and stored.  A
// row starts in a tail slot and goes on in the head slots of the following tiles, up to the first one whose tail slot
// is not its own.  Rows over a few tiles are merged by one lane group each; a row over more than kLongRow tiles by the
// whole block, a contiguous share of its records per lane group, the shares' sums meeting in shared memory in order.
template <class Op> constexpr int kCarryThreads = Op::W <= 2 ? 256 : 128;
constexpr int kLongRow = 24;
template <class Op>
__global__ void __launch_bounds__(kCarryThreads<Op>)
carry_rows_kernel(const __grid_constant__ Op op, const __grid_constant__ WalkArgs a) {
  using A = typename Op::A;
  constexpr int G = Op::G, THREADS = kCarryThreads<Op>, UNITS = THREADS / G, CE = Op::kCarryElems;
  constexpr int B = Op::W <= 2 ? 4 : 2;   // records in flight
  extern __shared__ uint4 gk_ring[];
  A* part = reinterpret_cast<A*>(gk_ring);   // UNITS records
  __shared__ unsigned s_start[THREADS / 2], s_long[THREADS / 2];
  __shared__ int s_n, s_nlong, s_end;
  if (not_asked<Op>(a)) return;
  const int tid = threadIdx.x, u = tid / G, gl = tid & (G - 1), hb = blockIdx.y;
  const uint32_t* ids = a.rows + (size_t)hb * 2 * a.n_tiles;
  const A* rec = reinterpret_cast<const A*>(a.carry) + (size_t)hb * 2 * a.n_tiles * CE;
  if (tid == 0) { s_n = 0; s_nlong = 0; }
  __syncthreads();
  // thread i looks at the tail slot of tile blockIdx.x * THREADS / 2 + i / 2 (odd slots start rows)
  const unsigned slot = blockIdx.x * THREADS + tid;
  if ((slot & 1u) && slot < 2 * a.n_tiles) {
    const uint32_t id = ids[slot];
    if (id != kNoRow && (id & 1u)) s_start[atomicAdd(&s_n, 1)] = slot >> 1;
  }
  __syncthreads();
  const int n = s_n;
  if (n == 0) return;
  typename Op::State st;
  op.setup(st, gl, hb);
  const unsigned group = (G == 32 ? kFull : ((1u << G) - 1u) << ((tid & 31) & ~(G - 1)));
  // record r of a row that starts in tile t: its tail slot, then the head slots of the tiles after it
  auto record = [&](unsigned t, int r) { return rec + (2 * (size_t)t + 1 + (r > 0 ? 2 * (size_t)r - 1 : 0)) * CE; };
  auto merge_range = [&](unsigned t, int r0, int r1) {
    op.begin_merge(st);
    for (int r = r0; r < r1; r += B) {
      typename Op::Carry in[B];
#pragma unroll
      for (int i = 0; i < B; ++i)
        if (r + i < r1) op.load_carry(in[i], record(t, r + i), gl);
#pragma unroll
      for (int i = 0; i < B; ++i)
        if (r + i < r1) op.merge(st, in[i]);
    }
  };
  for (int k = u; k < n; k += UNITS) {
    const unsigned t = s_start[k];
    const uint32_t inside = ids[2 * (size_t)t + 1] & ~1u;
    int more = 0;   // tiles after t that hold a record of the row
    for (bool open = true; open && more <= kLongRow; more += G) {
      const unsigned x = t + 1 + more + gl;
      const bool ends = x >= a.n_tiles || ids[2 * (size_t)x + 1] != inside;
      const unsigned m = __ballot_sync(group, ends) >> ((tid & 31) & ~(G - 1)) & (kFull >> (32 - G));
      if (m) { more += __ffs(m) - G; open = false; }
    }
    if (more > kLongRow) {
      if (gl == 0) s_long[atomicAdd(&s_nlong, 1)] = t;
      continue;
    }
    merge_range(t, 0, 1 + more);
    op.store_row(st, (int)(inside >> 1));
  }
  __syncthreads();
  for (int k = 0; k < s_nlong; ++k) {
    const unsigned t = s_long[k];
    const uint32_t inside = ids[2 * (size_t)t + 1] & ~1u;
    if (tid == 0) s_end = 0x7fffffff;
    __syncthreads();
    int more = 0;
    for (;; more += THREADS) {
      const unsigned x = t + 1 + more + tid;
      if (x >= a.n_tiles || ids[2 * (size_t)x + 1] != inside) atomicMin(&s_end, more + tid + 1);
      __syncthreads();
      if (s_end != 0x7fffffff) break;
      __syncthreads();
    }
    const int total = 1 + s_end;
    merge_range(t, (int)((long long)total * u / UNITS), (int)((long long)total * (u + 1) / UNITS));
    op.save_carry(st, part + (size_t)u * CE, gl);
    __syncthreads();
    if (u == 0) {
      op.begin_merge(st);
      for (int i = 0; i < UNITS; ++i) {
        typename Op::Carry in;
        op.load_carry(in, part + (size_t)i * CE, gl);
        op.merge(st, in);
      }
      op.store_row(st, (int)(inside >> 1));
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// the ops
// ---------------------------------------------------------------------------------------
// y[node, h, :] = sum over the node's positions of w[edge, h] * feat: feat = x[other] or, kEdgeFeat, one D-vector per
// edge shared by the heads (the kernels of graphop_kernel.cu this stands for: see AggregateOp)
template <class GEO, bool kEdgeFeat>
struct GroupAggregate : GEO, Shape<GEO, 1, (int)sizeof(typename GEO::T), 1, 0, 0, 2> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr const char* kName = kEdgeFeat ? "aggregate_edge_feat" : "aggregate";
  static constexpr bool kRowOut = true, kUsesOther = !kEdgeFeat, kUsesEid = true,
                        kFoldsEid = false, kOptional = !kEdgeFeat && sizeof(T) >= 4;
  static constexpr int W = GEO::W;
  const T* __restrict__ w;
  const T* __restrict__ x;
  T* __restrict__ y;
  struct State { typename GEO::Lane ln; const unsigned char* xb; F acc[W]; };
  struct Carry { F x[W]; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.xb = reinterpret_cast<const unsigned char*>(x + (kEdgeFeat ? st.ln.eoff : st.ln.off));
    begin_merge(st);
  }
  __device__ __forceinline__ void stage(const State& st, unsigned slot, int id, int e, bool live) const {
    this->stage_row(st.ln, slot, st.xb, kEdgeFeat ? e : id, kEdgeFeat ? this->drowb : this->rowb, live);
  }
  __device__ __forceinline__ const void* scalar_of(int h, int, int e) const {
    return w + ((unsigned long long)(unsigned)e * (unsigned)this->H + h);
  }
  template <int N>
  __device__ __forceinline__ void fold(State& st, unsigned slot, unsigned tab, const bool (&)[N], unsigned,
                                       const int (&)[N]) const {
    // positions without an edge have rows and weights of zeros
#pragma unroll
    for (int v = 0; v < N; ++v) {
      F f[W];
      this->load_staged(f, slot + v * this->kStepBytes);
      T wt;
      lds(wt, tab + v * GEO::kHeads * (int)sizeof(T));
      const A wv = to_acc<T>(wt);
#pragma unroll
      for (int i = 0; i < W; ++i) st.acc[i].axpy(wv, f[i]);
    }
  }
  __device__ __forceinline__ void stage_node(const State&, unsigned, int, int) const {}
  __device__ __forceinline__ void begin(State& st, unsigned, int) const { begin_merge(st); }
  __device__ __forceinline__ void began(State&, int, bool) const {}
  __device__ __forceinline__ void store_row(const State& st, int node) const {
    this->store_row_slots(st.ln, y + (long long)node * this->HD + st.ln.off, st.acc);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const { this->zero_slots(st.ln, y, n); }
  static constexpr int kCarryElems = GEO::kAccs;
  __device__ __forceinline__ void begin_merge(State& st) const {
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].zero();
  }
  __device__ __forceinline__ void save_carry(const State& st, A* rec, int gl) const { this->save_acc(rec, gl, st.acc); }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const { this->load_acc_raw(c.x, rec, gl); }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const {
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].add(c.x[i]);
  }
};

// The edge-feature aggregate with all heads in a lane: y[node, h, :] = sum over the node's positions of w[edge, h] * x[edge].
// Bound by reading x; with a copy of the row per head (GroupAggregate) 17.8M edges, 4 x 32 fp32, took 0.97 ms.
template <class GEO>
struct GroupFeatAggregate : GEO, Shape<GEO, 1, (int)sizeof(typename GEO::T), 1, 0, 0, 2> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr const char* kName = "aggregate_edge_feat";
  static constexpr bool kRowOut = true, kUsesOther = false, kUsesEid = true, kFoldsEid = false;
  static constexpr int W = GEO::W;
  const T* __restrict__ w;
  const T* __restrict__ x;
  T* __restrict__ y;
  struct State { typename GEO::Lane ln; const unsigned char* xb; F acc[W]; };
  struct Carry { F x[W]; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.xb = reinterpret_cast<const unsigned char*>(x + st.ln.eoff);
    begin_merge(st);
  }
  __device__ __forceinline__ void stage(const State& st, unsigned slot, int, int e, bool live) const {
    this->stage_row(slot, st.xb, e, this->drowb, live);
  }
  __device__ __forceinline__ const void* scalar_of(int h, int, int e) const {
    return w + ((unsigned long long)(unsigned)e * (unsigned)W + h);
  }
  template <int N>
  __device__ __forceinline__ void fold(State& st, unsigned slot, unsigned tab, const bool (&)[N], unsigned,
                                       const int (&)[N]) const {
#pragma unroll
    for (int v = 0; v < N; ++v) {
      F f;
      frag_lds<T, 16>(f, slot + v * this->kStepBytes);
      T wt[W];
#pragma unroll
      for (int h = 0; h < W; ++h) lds(wt[h], tab + (v * W + h) * (int)sizeof(T));
#pragma unroll
      for (int h = 0; h < W; ++h) st.acc[h].axpy(to_acc<T>(wt[h]), f);
    }
  }
  __device__ __forceinline__ void stage_node(const State&, unsigned, int, int) const {}
  __device__ __forceinline__ void begin(State& st, unsigned, int) const { begin_merge(st); }
  __device__ __forceinline__ void began(State&, int, bool) const {}
  __device__ __forceinline__ void store_row(const State& st, int node) const {
    this->store_row_slots(y + (long long)node * this->HD + st.ln.off, st.acc);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const {
    F z[W];
#pragma unroll
    for (int i = 0; i < W; ++i) z[i].zero();
    this->store_row_slots(y + n * this->HD + st.ln.off, z);
  }
  static constexpr int kCarryElems = GEO::kAccs;
  __device__ __forceinline__ void begin_merge(State& st) const {
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].zero();
  }
  __device__ __forceinline__ void save_carry(const State& st, A* rec, int gl) const { this->save_acc(rec, gl, st.acc); }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const { this->load_acc_raw(c.x, rec, gl); }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const {
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].add(c.x[i]);
  }
};

// y[edge, h] = a[node, h, :] . feat (EdgeDotOp's kernels)
template <class GEO, bool kEdgeFeat>
struct GroupEdgeDot : GEO, Shape<GEO, 1, 0, 1, 1, 0, 2> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr const char* kName = "edge_dot";
  static constexpr bool kRowOut = false, kUsesOther = !kEdgeFeat, kUsesEid = true,
                        kFoldsEid = true;
  static constexpr int W = GEO::W;
  const T* __restrict__ a;
  const T* __restrict__ b;
  T* __restrict__ y;
  struct State { typename GEO::Lane ln; const unsigned char* bb; F a[W]; };
  struct Carry {};
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.bb = reinterpret_cast<const unsigned char*>(b + (kEdgeFeat ? st.ln.eoff : st.ln.off));
#pragma unroll
    for (int i = 0; i < W; ++i) st.a[i].zero();
  }
  __device__ __forceinline__ void stage(const State& st, unsigned slot, int id, int e, bool live) const {
    this->stage_row(st.ln, slot, st.bb, kEdgeFeat ? e : id, kEdgeFeat ? this->drowb : this->rowb, live);
  }
  __device__ __forceinline__ const void* scalar_of(int, int, int) const { return nullptr; }
  template <int N>
  __device__ __forceinline__ void fold(State& st, unsigned slot, unsigned, const bool (&active)[N], unsigned,
                                       const int (&e)[N]) const {
    A s[N];
#pragma unroll
    for (int v = 0; v < N; ++v) {
      F f[W];
      this->load_staged(f, slot + v * this->kStepBytes);
      s[v] = this->ordered_dot(st.a, f);
    }
#pragma unroll
    for (int v = 0; v < N; ++v)
      if (active[v] && st.ln.first)
        y[(unsigned long long)(unsigned)e[v] * (unsigned)this->H + st.ln.head] = from_acc<T>(s[v]);
  }
  __device__ __forceinline__ void stage_node(const State& st, unsigned buf, int, int node) const {
    this->stage_row(st.ln, buf, reinterpret_cast<const unsigned char*>(a + st.ln.off), node, this->rowb, true);
  }
  __device__ __forceinline__ void begin(State& st, unsigned buf, int) const { this->load_staged(st.a, buf); }
  __device__ __forceinline__ void began(State&, int, bool) const {}
  __device__ __forceinline__ void store_row(const State&, int) const {}
  __device__ __forceinline__ void zero_row(const State&, long long) const {}
  static constexpr int kCarryElems = 0;
  __device__ __forceinline__ void begin_merge(State&) const {}
  __device__ __forceinline__ void save_carry(const State&, A*, int) const {}
  __device__ __forceinline__ void load_carry(Carry&, const A*, int) const {}
  __device__ __forceinline__ void merge(State&, const Carry&) const {}
};

// Fused attention forward: o[node] = sum_k softmax_k(scale q.k) v.  Scores in base-2 units (q is multiplied by
// scale * log2 e when a node starts).  The accumulators are rescaled in every step: with several groups per warp some group's
// running maximum grows in most of them.
// kBias: the score's key row gets the edge's row of rel added (one D-vector per edge, shared by the heads).
template <class GEO, bool kBias>
struct GroupAttnFwd : GEO, Shape<GEO, kBias ? 3 : 2, 0, 2, 1, 0, 2> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr int W = GEO::W, V = GEO::V, kRow = GEO::kRow;   // rows of a ring step: k, v (, rel)
  static constexpr const char* kName = kBias ? "attention_bias_fwd" : "attention_fwd";
  static constexpr bool kRowOut = true, kUsesOther = true, kUsesEid = kBias,
                        kFoldsEid = false;
  const T* __restrict__ q;
  const T* __restrict__ k;
  const T* __restrict__ v;
  const T* __restrict__ rel;
  T* __restrict__ o;
  A* __restrict__ lse;
  A scale;
  struct State {
    typename GEO::Lane ln;
    const unsigned char *kb, *vb, *rb;
    F q[W], acc[W];
    A m, l;
  };
  struct Carry { F x[W]; A m, l; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.kb = reinterpret_cast<const unsigned char*>(k + st.ln.off);
    st.vb = reinterpret_cast<const unsigned char*>(v + st.ln.off);
    st.rb = kBias ? reinterpret_cast<const unsigned char*>(rel + st.ln.eoff) : nullptr;
    begin_merge(st);
#pragma unroll
    for (int i = 0; i < W; ++i) st.q[i].zero();
  }
  __device__ __forceinline__ void stage(const State& st, unsigned slot, int id, int e, bool live) const {
    this->stage_row(st.ln, slot, st.kb, id, this->rowb, live);
    this->stage_row(st.ln, slot + kRow, st.vb, id, this->rowb, live);
    if constexpr (kBias) this->stage_row(st.ln, slot + 2 * kRow, st.rb, e, this->drowb, live);
  }
  __device__ __forceinline__ const void* scalar_of(int, int, int) const { return nullptr; }
  template <int N>
  __device__ __forceinline__ void fold(State& st, unsigned slot, unsigned, const bool (&active)[N], unsigned,
                                       const int (&)[N]) const {
    A s[N], p[N];
    A mn = st.m;
#pragma unroll
    for (int v = 0; v < N; ++v) {
      F f[W];
      this->load_staged(f, slot + v * this->kStepBytes);
      if constexpr (kBias) {
        F r[W];
        this->load_staged(r, slot + v * this->kStepBytes + 2 * kRow);
#pragma unroll
        for (int i = 0; i < W; ++i) f[i].add(r[i]);
      }
      s[v] = frag_dot<V, W>(st.q, f);
    }
#pragma unroll
    for (int v = 0; v < N; ++v) {
      s[v] = this->head_sum(s[v]);
      if (!active[v]) s[v] = neg_inf<A>();
      mn = s[v] > mn ? s[v] : mn;
    }
    const A corr = st.m == mn ? A(1) : gk_exp2(st.m - mn);   // m = -inf before a node's first edge: 2^-inf = 0
    const A ref = mn == neg_inf<A>() ? A(0) : mn;            // nothing but masked scores (-inf) so far: they add 2^-inf
    st.m = mn;
    st.l *= corr;
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].scale(corr);
#pragma unroll
    for (int v = 0; v < N; ++v) {
      p[v] = active[v] ? gk_exp2(s[v] - ref) : A(0);
      st.l += p[v];
      F f[W];
      this->load_staged(f, slot + v * this->kStepBytes + kRow);
#pragma unroll
      for (int i = 0; i < W; ++i) st.acc[i].axpy(p[v], f[i]);
    }
  }
  __device__ __forceinline__ void stage_node(const State& st, unsigned buf, int, int node) const {
    this->stage_row(st.ln, buf, reinterpret_cast<const unsigned char*>(q + st.ln.off), node, this->rowb, true);
  }
  __device__ __forceinline__ void begin(State& st, unsigned buf, int) const {
    this->load_staged(st.q, buf);
    begin_merge(st);
    const A c = scale * A(kLog2e);
#pragma unroll
    for (int i = 0; i < W; ++i) st.q[i].scale(c);
  }
  __device__ __forceinline__ void began(State&, int, bool) const {}
  // m is a base-2 exponent: lse = (m + log2 l) * ln 2
  __device__ __forceinline__ void store_row(const State& st, int node) const {
    const A inv = A(1) / st.l;
    F out[W];
#pragma unroll
    for (int i = 0; i < W; ++i) { out[i] = st.acc[i]; out[i].scale(inv); }
    this->store_row_slots(st.ln, o + (long long)node * this->HD + st.ln.off, out);
    if (st.ln.first) lse[(long long)node * this->H + st.ln.head] = (st.m + gk_log2(st.l)) * A(kLn2);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const {
    this->zero_slots(st.ln, o, n);
    if (st.ln.first) lse[n * this->H + st.ln.head] = neg_inf<A>();
  }
  static constexpr int kCarryElems = GEO::kAccs + 2 * GEO::G;
  __device__ __forceinline__ void begin_merge(State& st) const {
    st.m = neg_inf<A>();
    st.l = A(0);
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].zero();
  }
  __device__ __forceinline__ void save_carry(const State& st, A* rec, int gl) const {
    this->save_acc(rec, gl, st.acc);
    rec[GEO::kAccs + gl] = st.m;
    rec[GEO::kAccs + GEO::G + gl] = st.l;
  }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const {
    this->load_acc_raw(c.x, rec, gl);
    c.m = rec[GEO::kAccs + gl];
    c.l = rec[GEO::kAccs + GEO::G + gl];
  }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const {
    const A mn = c.m > st.m ? c.m : st.m;
    // a neutral partial has m = -inf: its weight is zero, never 2^(-inf - -inf)
    const A wa = st.m == neg_inf<A>() ? A(0) : gk_exp2(st.m - mn);
    const A wb = c.m == neg_inf<A>() ? A(0) : gk_exp2(c.m - mn);
    st.l = st.l * wa + c.l * wb;
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].blend(wa, c.x[i], wb);
    st.m = mn;
  }
};

// Fused attention backward, destination side: dq[node] = sum ds (k + rel), ds = p (dO.v - delta) scale; writes
// (lse, delta) per node and, pd != null, (p, ds) per position and head for the source side.
// Two positions per iteration pay for 2-byte elements (R-MAT 18, 4 x 64 bf16 with the edge term: 1.19 -> 1.02 ms); for
// wider ones they leave fewer warps (R-MAT 21, 4 x 32 fp32: 4.64 -> 4.49 ms, but 4096 nodes, 8 x 64: 35 -> 39 us).
template <class GEO, bool kBias>
struct GroupAttnBwdDst : GEO, Shape<GEO, kBias ? 3 : 2, 0, 4, 3, (int)sizeof(typename GEO::A),
                                (sizeof(typename GEO::T) == 2 ? 2 : 1), true> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr int W = GEO::W, V = GEO::V, kRow = GEO::kRow;   // rows of a ring step: k, v (, rel)
  static constexpr const char* kName = kBias ? "attention_bias_bwd_dst" : "attention_bwd_dst";
  static constexpr bool kRowOut = true, kUsesOther = true, kUsesEid = kBias,
                        kFoldsEid = false;
  const T* __restrict__ q;
  const T* __restrict__ k;
  const T* __restrict__ v;
  const T* __restrict__ rel;
  const T* __restrict__ o;
  const T* __restrict__ dout;
  const A* __restrict__ lse;
  StatPair<A>* __restrict__ stat;
  EdgePair<A>* __restrict__ pd;
  T* __restrict__ dq;
  A scale;
  int Hp;
  struct State {
    typename GEO::Lane ln;
    const unsigned char *kb, *vb, *rb;
    F q[W], gr[W], acc[W];
    A lse2, delta;
  };
  struct Carry { F x[W]; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.kb = reinterpret_cast<const unsigned char*>(k + st.ln.off);
    st.vb = reinterpret_cast<const unsigned char*>(v + st.ln.off);
    st.rb = kBias ? reinterpret_cast<const unsigned char*>(rel + st.ln.eoff) : nullptr;
    begin_merge(st);
    st.lse2 = st.delta = A(0);
#pragma unroll
    for (int i = 0; i < W; ++i) { st.q[i].zero(); st.gr[i].zero(); }
  }
  __device__ __forceinline__ void stage(const State& st, unsigned slot, int id, int e, bool live) const {
    this->stage_row(st.ln, slot, st.kb, id, this->rowb, live);
    this->stage_row(st.ln, slot + kRow, st.vb, id, this->rowb, live);
    if constexpr (kBias) this->stage_row(st.ln, slot + 2 * kRow, st.rb, e, this->drowb, live);
  }
  __device__ __forceinline__ const void* scalar_of(int, int, int) const { return nullptr; }
  template <int N>
  __device__ __forceinline__ void fold(State& st, unsigned slot, unsigned, const bool (&active)[N], unsigned pos,
                                       const int (&)[N]) const {
    A s[N], dp[N];
    F f[N][W];
#pragma unroll
    for (int v = 0; v < N; ++v) {
      this->load_staged(f[v], slot + v * this->kStepBytes + kRow);
      dp[v] = frag_dot<V, W>(st.gr, f[v]);
      this->load_staged(f[v], slot + v * this->kStepBytes);
      if constexpr (kBias) {
        F r[W];
        this->load_staged(r, slot + v * this->kStepBytes + 2 * kRow);
#pragma unroll
        for (int i = 0; i < W; ++i) f[v][i].add(r[i]);
      }
      s[v] = frag_dot<V, W>(st.q, f[v]);
    }
#pragma unroll
    for (int v = 0; v < N; ++v) {
      s[v] = this->head_sum(s[v]);
      dp[v] = this->head_sum(dp[v]);
    }
#pragma unroll
    for (int v = 0; v < N; ++v) {
      const A p = gk_exp2(s[v] - st.lse2);
      A ds = p * (dp[v] - st.delta) * scale;
      if (!active[v]) ds = A(0);
      if (active[v] && pd && st.ln.first)
        pd[(unsigned long long)(pos + v) * (unsigned)Hp + st.ln.head] = EdgePair<A>{p, ds};
#pragma unroll
      for (int i = 0; i < W; ++i) st.acc[i].axpy(ds, f[v][i]);
    }
  }
  __device__ __forceinline__ int lse_at(int lane) const { return this->kNodeScalarAt + lane * ((int)sizeof(A) - GEO::SB); }
  __device__ __forceinline__ void stage_node(const State& st, unsigned buf, int lane, int node) const {
    this->stage_row(st.ln, buf, reinterpret_cast<const unsigned char*>(q + st.ln.off), node, this->rowb, true);
    this->stage_row(st.ln, buf + kRow, reinterpret_cast<const unsigned char*>(dout + st.ln.off), node, this->rowb, true);
    this->stage_row(st.ln, buf + 2 * kRow, reinterpret_cast<const unsigned char*>(o + st.ln.off), node, this->rowb, true);
    cp_async_slot<sizeof(A)>(buf + lse_at(lane), lse + (long long)node * this->H + st.ln.head, true);
  }
  __device__ __forceinline__ void begin(State& st, unsigned buf, int lane) const {
    F ov[W];
    this->load_staged(st.q, buf);
    this->load_staged(st.gr, buf + kRow);
    this->load_staged(ov, buf + 2 * kRow);
    lds(st.lse2, buf + lse_at(lane));
    begin_merge(st);
    st.delta = frag_dot<V, W>(st.gr, ov);   // this lane's part: summed in began()
    const A c = scale * A(kLog2e);
#pragma unroll
    for (int i = 0; i < W; ++i) st.q[i].scale(c);
  }
  // delta = dO . o in the order dO . v is formed: a node with one edge gets dp - delta = 0 exactly
  __device__ __forceinline__ void began(State& st, int node, bool mine) const {
    const A d = this->head_sum(st.delta);
    if (mine) {
      st.delta = d;
      if (st.ln.first) stat[(long long)node * Hp + st.ln.head] = StatPair<A>{st.lse2, d};
      st.lse2 *= A(kLog2e);
    }
  }
  __device__ __forceinline__ void store_row(const State& st, int node) const {
    this->store_row_slots(st.ln, dq + (long long)node * this->HD + st.ln.off, st.acc);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const {
    this->zero_slots(st.ln, dq, n);
    if (st.ln.first) stat[n * Hp + st.ln.head] = StatPair<A>{A(0), A(0)};
  }
  static constexpr int kCarryElems = GEO::kAccs;
  __device__ __forceinline__ void begin_merge(State& st) const {
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].zero();
  }
  __device__ __forceinline__ void save_carry(const State& st, A* rec, int gl) const { this->save_acc(rec, gl, st.acc); }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const { this->load_acc_raw(c.x, rec, gl); }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const {
#pragma unroll
    for (int i = 0; i < W; ++i) st.acc[i].add(c.x[i]);
  }
};

// Fused attention backward, source side, over the transposed CSR: dv[c] = sum p dO[dst], dk[c] = sum ds q[dst].
// kPairs: (p, ds) of every edge come from the destination side (by edge id); else they are recomputed from k, v and the
// destination's (lse, delta).
template <class GEO, bool kPairs>
struct GroupAttnBwdSrc : GEO, Shape<GEO, 2, 2 * (int)sizeof(typename GEO::A), kPairs ? 2 : 4, kPairs ? 0 : 2, 0, kPairs ? 2 : 1> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr int W = GEO::W, V = GEO::V, kRow = GEO::kRow;   // rows of a ring step: q, dO
  static constexpr const char* kName = "attention_bwd_src";
  static constexpr bool kRowOut = true, kUsesOther = true, kUsesEid = kPairs,
                        kFoldsEid = false, kOptional = kPairs && sizeof(T) >= 4;
  const T* __restrict__ q;
  const T* __restrict__ k;
  const T* __restrict__ v;
  const T* __restrict__ dout;
  const StatPair<A>* __restrict__ stat;
  const EdgePair<A>* __restrict__ pd;
  T* __restrict__ dk;
  T* __restrict__ dv;
  A scale;
  int Hp;
  struct State {
    typename GEO::Lane ln;
    const unsigned char *qb, *gb;
    F k[kPairs ? 1 : W], v[kPairs ? 1 : W], ak[W], av[W];
  };
  struct Carry { F k[W], v[W]; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.qb = reinterpret_cast<const unsigned char*>(q + st.ln.off);
    st.gb = reinterpret_cast<const unsigned char*>(dout + st.ln.off);
    begin_merge(st);
#pragma unroll
    for (int i = 0; i < (kPairs ? 1 : W); ++i) { st.k[i].zero(); st.v[i].zero(); }
  }
  __device__ __forceinline__ void stage(const State& st, unsigned slot, int id, int, bool live) const {
    this->stage_row(st.ln, slot, st.qb, id, this->rowb, live);
    this->stage_row(st.ln, slot + kRow, st.gb, id, this->rowb, live);
  }
  // (p, ds) of the edge or (lse, delta) of its destination
  __device__ __forceinline__ const void* scalar_of(int h, int id, int e) const {
    if constexpr (kPairs) return pd + ((unsigned long long)(unsigned)e * (unsigned)Hp + h);
    else return stat + ((unsigned long long)(unsigned)id * (unsigned)Hp + h);
  }
  template <int N>
  __device__ __forceinline__ void fold(State& st, unsigned slot, unsigned tab, const bool (&active)[N], unsigned,
                                       const int (&)[N]) const {
    // positions without an edge have rows and pairs of zeros
#pragma unroll
    for (int v = 0; v < N; ++v) {
      F fq[W], fg[W];
      this->load_staged(fq, slot + v * this->kStepBytes);
      this->load_staged(fg, slot + v * this->kStepBytes + kRow);
      A x, y;
      lds2(x, y, tab + v * GEO::kHeads * 2 * (int)sizeof(A));
      A p = x, ds = y;
      if constexpr (!kPairs) {
        const A s = this->head_sum(frag_dot<V, W>(fq, st.k));
        const A dp = this->head_sum(frag_dot<V, W>(fg, st.v));
        p = active[v] ? gk_exp2(s - x * A(kLog2e)) : A(0);
        ds = active[v] ? p * (dp - y) * scale : A(0);
      }
#pragma unroll
      for (int i = 0; i < W; ++i) { st.av[i].axpy(p, fg[i]); st.ak[i].axpy(ds, fq[i]); }
    }
  }
  __device__ __forceinline__ void stage_node(const State& st, unsigned buf, int, int node) const {
    this->stage_row(st.ln, buf, reinterpret_cast<const unsigned char*>(k + st.ln.off), node, this->rowb, true);
    this->stage_row(st.ln, buf + kRow, reinterpret_cast<const unsigned char*>(v + st.ln.off), node, this->rowb, true);
  }
  __device__ __forceinline__ void begin(State& st, unsigned buf, int) const {
    begin_merge(st);
    if constexpr (!kPairs) {
      this->load_staged(st.k, buf);
      this->load_staged(st.v, buf + kRow);
      const A c = scale * A(kLog2e);
#pragma unroll
      for (int i = 0; i < W; ++i) st.k[i].scale(c);
    }
  }
  __device__ __forceinline__ void began(State&, int, bool) const {}
  __device__ __forceinline__ void store_row(const State& st, int node) const {
    const long long at = (long long)node * this->HD + st.ln.off;
    this->store_row_slots(st.ln, dk + at, st.ak);
    this->store_row_slots(st.ln, dv + at, st.av);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const {
    this->zero_slots(st.ln, dk, n);
    this->zero_slots(st.ln, dv, n);
  }
  static constexpr int kCarryElems = 2 * GEO::kAccs;
  __device__ __forceinline__ void begin_merge(State& st) const {
#pragma unroll
    for (int i = 0; i < W; ++i) { st.ak[i].zero(); st.av[i].zero(); }
  }
  __device__ __forceinline__ void save_carry(const State& st, A* rec, int gl) const {
    this->save_acc(rec, gl, st.ak);
    this->save_acc(rec + GEO::kAccs, gl, st.av);
  }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const {
    this->load_acc_raw(c.k, rec, gl);
    this->load_acc_raw(c.v, rec + GEO::kAccs, gl);
  }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const {
#pragma unroll
    for (int i = 0; i < W; ++i) { st.ak[i].add(c.k[i]); st.av[i].add(c.v[i]); }
  }
};

}  // namespace gk
