// Shared device machinery of the graphop kernels for sm_100a.
//
// Work decomposition.  Every op sees the graph as a flat stream of CSR positions 0..E-1.  A one-pass "expansion" turns the
// caller's chunk table (row[c], indptr[c]), in which several consecutive chunks may belong to one node, into erow[j] =
// owner node of position j (-1 where no chunk covers j), and cuts the stream into work tiles of equal cost.  The walker
// of gk_group.cuh does the work of all row-reducing and per-edge ops; walk_kernel below is the plain form of it that
// takes any shape (one element per lane and slot, tiles of equal length).
//
// Row-owned reductions without atomics.  A run of equal erow[] values is one segment.  A segment that lies wholly inside
// a tile is reduced in registers and stored once.  The first segment of a tile whose node already started in an earlier
// tile ("open head") and the last segment of a tile whose node continues in the next one ("open tail") are stored as
// partials in two carry slots per tile, and later launches fold the slots of a node in ascending tile order.  The sum
// order is a function of the graph and the tile size only: results are bit-reproducible.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace gk {

constexpr int kWarpsPerCta = 8;
constexpr unsigned kFull = 0xffffffffu;

struct PlanHeader {
  long long cover_lo;  // first CSR position any chunk covers  (= indptr[0])
  long long cover_hi;  // one past the last covered position   (= indptr[C])
  int skewed;          // few rows are gathered by many edges; set by skew_kernel where an op asks for it
  int repeats;         // gather_repeats, set where a plan is built
};

// ---------------------------------------------------------------------------------------
// element types: storage type T, accumulation type AccOf<T>
// ---------------------------------------------------------------------------------------
template <typename T> struct AccOf { using type = float; };
template <> struct AccOf<double> { using type = double; };

template <typename T> __device__ __forceinline__ typename AccOf<T>::type to_acc(T v) { return v; }
template <> __device__ __forceinline__ float to_acc<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_acc(typename AccOf<T>::type v) { return (T)v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_acc<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float gk_exp(float x) { return expf(x); }
__device__ __forceinline__ double gk_exp(double x) { return exp(x); }
template <typename A> __device__ __forceinline__ A neg_inf();
template <> __device__ __forceinline__ float neg_inf<float>() { return -INFINITY; }
template <> __device__ __forceinline__ double neg_inf<double>() { return -(double)INFINITY; }

// V consecutive elements of T moved with one load/store of V*sizeof(T) bytes (4, 8 or 16).
template <typename T, int V> struct alignas(sizeof(T) * V) Pack { T v[V]; };

template <int BYTES> struct Mover;
template <> struct Mover<16> { using type = uint4; };
template <> struct Mover<8> { using type = uint2; };
template <> struct Mover<4> { using type = uint32_t; };
template <> struct Mover<2> { using type = uint16_t; };

template <typename T, int V>
__device__ __forceinline__ void load_acc(typename AccOf<T>::type (&dst)[V], const T* __restrict__ p) {
  using M = typename Mover<sizeof(T) * V>::type;
  union { M m; T t[V]; } u;
  u.m = __ldg(reinterpret_cast<const M*>(p));
#pragma unroll
  for (int i = 0; i < V; ++i) dst[i] = to_acc<T>(u.t[i]);
}

template <typename T, int V>
__device__ __forceinline__ void store_acc(T* __restrict__ p, const typename AccOf<T>::type (&src)[V]) {
  using M = typename Mover<sizeof(T) * V>::type;
  union { M m; T t[V]; } u;
#pragma unroll
  for (int i = 0; i < V; ++i) u.t[i] = from_acc<T>(src[i]);
  *reinterpret_cast<M*>(p) = u.m;
}

// plain (non-converting) vector moves for the accumulation type itself: carries
template <typename A, int V>
__device__ __forceinline__ void load_raw(A (&dst)[V], const A* p) {
#pragma unroll
  for (int i = 0; i < V; ++i) dst[i] = p[i];
}
template <typename A, int V>
__device__ __forceinline__ void store_raw(A* p, const A (&src)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) p[i] = src[i];
}

// Every cross-lane sum in these kernels is a butterfly over lane distances 1, 2, 4, ... in that order, whichever
// routine forms it: two kernels that reduce the same per-lane partials (delta in the destination pass, dO . v in
// the source pass) then agree bit for bit.
template <typename A> __device__ __forceinline__ A warp_sum(A v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Per-lane view of a node's feature row: lane owns slots lane, lane+32, ..., each V elements.
template <int R> struct SlotMap {
  int head[R];  // head index of the slot
  int feat[R];  // element offset of the slot inside the H*D row
  int efeat[R]; // element offset inside one head's D-vector (edge-feature operands)
  bool ok[R];   // slot exists (slot < S)
  __device__ __forceinline__ void init(int lane, int S, int V, int D, int feat0) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int s = lane + 32 * i;
      ok[i] = s < S;
      const int el = feat0 + (ok[i] ? s : 0) * V;
      feat[i] = el;
      head[i] = el / D;
      efeat[i] = el - head[i] * D;
    }
  }
};

// ---------------------------------------------------------------------------------------
// expansion: chunk table -> erow[], optional int64 -> int32 copies of indices / eid
// ---------------------------------------------------------------------------------------
// Work tiles of equal cost.  A position costs 1 and a node kRowCost (its begin and end cost the walker about as much as
// that many edges), so that neither a tile of one-edge nodes nor one inside a hub takes much longer than the others.
// With cost(p) = p + kRowCost * (node of p) the boundary of tile t is the first position whose cost reaches t * tile:
// every position knows which boundaries fall between its predecessor and itself, and writes them.  Positions before the
// covered ones count for node 0, those after for the last node.  Boundaries past the last position are E.
constexpr int kRowCost = 4;
struct TileCut {
  int32_t* start;      // (n + 1) boundaries, or null
  long long n;         // tiles
  int shift;           // log2 of the cost per tile
};
__device__ __forceinline__ long long tile_at(const TileCut& cut, long long p, long long node) {
  return p >= 0 ? (p + kRowCost * node) >> cut.shift : -1;
}
// position p: lo = tile_at of the position before it, hi = its own
__device__ __forceinline__ void cut_tiles(const TileCut& cut, long long p, long long E, long long lo, long long hi) {
  for (long long t = lo + 1; t <= hi && t <= cut.n; ++t) cut.start[t] = (int32_t)p;
  if (p == E - 1)
    for (long long t = hi + 1; t <= cut.n; ++t) cut.start[t] = (int32_t)E;
}

// How many of kSkewSamples evenly spaced positions gather a row that another one of them gathers, as far as a table of kSkewBits
// bits tells.  Many where few rows are gathered by many edges (R-MAT 20: 37 to 48, R-MAT 16: 141 to 166, a hub that has a tenth of
// the edges: 100), none where the neighbours follow the nodes, and as many as chance has it where the sources are uniform: 8 of
// different rows that share a bit, and more of the same row the fewer rows there are (skew_allowed).  For one block of THREADS;
// the answer is every thread's.  seen: the table, in shared or device memory, nobody else's meanwhile.
constexpr int kSkewSamples = 1024, kSkewBits = 65536;
template <int THREADS>
__device__ __forceinline__ int gather_repeats(const int32_t* __restrict__ other, long long E, unsigned* seen) {
  __shared__ int s_repeats;
  const int tid = threadIdx.x, n = E < kSkewSamples ? (int)E : kSkewSamples;
  int key[kSkewSamples / THREADS], repeats = 0;   // all asked for before any is looked at
#pragma unroll
  for (int i = 0; i < kSkewSamples / THREADS; ++i) {
    const int k = tid + i * THREADS;
    key[i] = k < n ? __ldg(other + E * k / n) : -1;
  }
  for (int i = tid; i < kSkewBits / 128; i += THREADS) reinterpret_cast<uint4*>(seen)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) s_repeats = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSkewSamples / THREADS; ++i) {
    const unsigned at = (unsigned)key[i] * 2654435761u >> 16, bit = 1u << (at & 31);
    if (key[i] >= 0 && (atomicOr(seen + (at >> 5), bit) & bit)) ++repeats;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) repeats += __shfl_xor_sync(kFull, repeats, o);
  if ((tid & 31) == 0) atomicAdd(&s_repeats, repeats);
  __syncthreads();
  return s_repeats;
}
template <int THREADS>
__global__ void __launch_bounds__(THREADS) skew_kernel(const int32_t* __restrict__ other, long long E, int allowed, PlanHeader* __restrict__ hdr) {
  __shared__ __align__(16) unsigned s_seen[kSkewBits / 32];
  const int repeats = gather_repeats<THREADS>(other, E, s_seen);
  if (threadIdx.x == 0) hdr->skewed = repeats > allowed;
}

// What an op wants done on the way: 32-bit copies of up to two 64-bit index arrays (a null source is skipped), and an
// edge output that starts from zero in the reference (at::zeros) cleared when some position belongs to no chunk.
template <typename I>
struct ExpandExtra {
  const I* src[2];
  int32_t* dst[2];
  uint16_t* clear;
  long long clear_n;   // 2-byte words
  int32_t* fill[3];    // arrays a plan's next kernels count on (null: none), with their lengths and values
  long long fill_n[3];
  int32_t fill_with[3];
};

// A block expands a run of `per_block` chunks (at most one per thread; the launch picks it for about one step of
// kExpandTile positions), so nothing has to be searched for: its positions are known as soon as its chunks are loaded.
// Every chunk that is not empty leaves its node at its first position in shared memory, and each thread fills its
// kExpandPer positions from the last one left at or before them; a chunk of many steps is written straight.  The positions
// before the first chunk fall to the first block, those after the last to the last one.  Bound by the written table
// and by how many blocks wait for their chunks at once: with a search per 256 positions 67M positions in chunks of up to
// 32 took 426 us.
constexpr int kExpandThreads = 256;
constexpr int kExpandPer = 8;
constexpr int kExpandTile = kExpandThreads * kExpandPer;

template <typename I>
__global__ void __launch_bounds__(kExpandThreads)
expand_rows_kernel(const I* __restrict__ row, const I* __restrict__ indptr, long long C, int E, int per_block,
                   int32_t* __restrict__ erow, PlanHeader* __restrict__ hdr, TileCut cut, ExpandExtra<I> extra) {
  constexpr int kNone = INT_MIN;
  __shared__ __align__(16) int s_row[kExpandTile];
  __shared__ int s_last[kExpandThreads / 32];
  __shared__ int s_long_end, s_long_row;   // a chunk of many steps: its end and node
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const long long c0 = (long long)blockIdx.x * per_block, c1 = c0 + per_block < C ? c0 + per_block : C;
  const int base = (int)indptr[0], last = (int)indptr[C], end = last < base ? base : last;
  const bool first_block = blockIdx.x == 0, last_block = first_block ? c1 >= C : c0 < C && c1 >= C;
  int s = 0, e = 0, r0 = 0;   // this thread's chunk
  if (c0 + tid < c1) {
    s = (int)indptr[c0 + tid];
    e = (int)indptr[c0 + tid + 1];
    r0 = (int)row[c0 + tid];
  }
  const bool idle = !first_block && c0 >= C;   // here for the copies alone
  const int begin = first_block || idle ? 0 : (int)indptr[c0];
  // the chunk before the block's, loaded with it
  const int ahead = first_block || idle ? 0 : (int)indptr[c0 - 1], ahead_row = first_block || idle ? 0 : (int)row[c0 - 1];
  const int finish = last_block ? E : idle ? 0 : (int)indptr[c1];
  if (first_block && tid == 0) {
    hdr->cover_lo = base;
    hdr->cover_hi = end;
  }
  if (extra.src[0] || extra.src[1]) {
    // the index copies are dealt out by position
    const long long share = ((long long)E + gridDim.x - 1) / gridDim.x, n0 = blockIdx.x * share;
    const long long n1 = n0 + share < E ? n0 + share : E;
#pragma unroll
    for (int a = 0; a < 2; ++a)
      if (extra.src[a])
#pragma unroll 8
        for (long long p = n0 + tid; p < n1; p += kExpandThreads) extra.dst[a][p] = (int32_t)extra.src[a][p];
  }
  if (extra.clear && end - base < E)
    for (long long i = (long long)blockIdx.x * kExpandThreads + tid; i < extra.clear_n;
         i += (long long)gridDim.x * kExpandThreads)
      extra.clear[i] = 0;

#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (extra.fill[a])
      for (long long i = (long long)blockIdx.x * kExpandThreads + tid; i < extra.fill_n[a];
           i += (long long)gridDim.x * kExpandThreads)
        extra.fill[a][i] = extra.fill_with[a];

  // nodes that positions without a chunk count for in the cut: 0 before the covered ones, the last node after them
  const auto node_before = [&](long long c) {   // of the last chunk before c that is not empty
    while (c > 0 && indptr[c - 1] == indptr[c]) --c;
    return c > 0 ? (int)row[c - 1] : 0;
  };
  int prev = 0, tail = 0;   // node of the position before the step; of the last covered position
  if (cut.start) {
    prev = ahead_row;
    if (tid == 0 && !first_block && ahead == begin) prev = node_before(c0 - 1);   // that chunk is empty
    if (last_block && end < E) tail = node_before(C);
  }
  int q0 = begin & ~(kExpandPer - 1);   // stores are 16 bytes wide
  for (int at = begin; at < finish;) {
    const int stop = finish - q0 > kExpandTile ? q0 + kExpandTile : finish;   // of this step
#pragma unroll
    for (int i = 0; i < kExpandPer; i += 4)
      *reinterpret_cast<int4*>(s_row + (i * kExpandThreads + tid * 4)) = make_int4(kNone, kNone, kNone, kNone);
    const bool covers = s <= at && e - at >= 4 * kExpandTile;
    if (covers) { s_long_end = e; s_long_row = r0; }
    if (__syncthreads_or(covers)) {
      // one chunk for many steps
      const int to = s_long_end;
      const int r = s_long_row;
      const int a0 = (at + 3) & ~3, a1 = to & ~3;
      if (tid < a0 - at) erow[at + tid] = r;
      if (tid < to - a1) erow[a1 + tid] = r;
      for (long long p = a0 + tid * 4; p < a1; p += kExpandThreads * 4)
        *reinterpret_cast<int4*>(erow + p) = make_int4(r, r, r, r);
      if (cut.start) {
        if (tid == 0) cut_tiles(cut, at, E, tile_at(cut, at - 1, prev), tile_at(cut, at, r));
        // inside the chunk boundary t lies where the cost reaches it
        const long long t1 = tile_at(cut, to - 1, r);
        for (long long t = tile_at(cut, at, r) + 1 + tid; t <= t1 && t <= cut.n; t += kExpandThreads)
          cut.start[t] = (int32_t)((t << cut.shift) - (long long)kRowCost * r);
        if (to == E)
          for (long long t = t1 + 1 + tid; t <= cut.n; t += kExpandThreads) cut.start[t] = (int32_t)E;
        prev = r;
      }
      at = to;
      q0 = at & ~(kExpandPer - 1);
      __syncthreads();
      continue;
    }
    if (e > s && s < stop && e > at) s_row[(s > at ? s : at) - q0] = r0;
    const bool bare = at < base || end < stop;   // some positions of the step belong to no chunk
    if (bare && tid == 0) {
      if (at < base) s_row[at - q0] = -1;
      if (end < stop) s_row[(end > at ? end : at) - q0] = -1;
    }
    __syncthreads();
    alignas(16) int r[kExpandPer];
#pragma unroll
    for (int i = 0; i < kExpandPer; i += 4)
      *reinterpret_cast<int4*>(r + i) = *reinterpret_cast<const int4*>(s_row + tid * kExpandPer + i);
#pragma unroll
    for (int i = 1; i < kExpandPer; ++i) r[i] = r[i] == kNone ? r[i - 1] : r[i];
    // the node in force before this thread's first position: of the nearest thread before it that met one
    const unsigned met = __ballot_sync(kFull, r[kExpandPer - 1] != kNone);
    const unsigned under = met & ((1u << lane) - 1);
    const int from = __shfl_sync(kFull, r[kExpandPer - 1], under ? 31 - __clz(under) : 0);
    const int top = __shfl_sync(kFull, r[kExpandPer - 1], met ? 31 - __clz(met) : 0);
    if (lane == 0) s_last[w] = met ? top : kNone;
    __syncthreads();
    int before = under ? from : kNone;
    for (int k = w - 1; k >= 0 && before == kNone; --k) before = s_last[k];
#pragma unroll
    for (int i = 0; i < kExpandPer; ++i) r[i] = r[i] == kNone ? before : r[i];
    // relative to the step: E may be 2^31 - 1, and positions of threads past the last one do not fit 32 bits then
    const int o = tid * kExpandPer, from_o = at - q0, to_o = stop - q0;
    const bool whole = o >= from_o && o + kExpandPer <= to_o;
    int32_t* const out = erow + q0;
    if (whole) {
#pragma unroll
      for (int i = 0; i < kExpandPer; i += 4) *reinterpret_cast<int4*>(out + o + i) = *reinterpret_cast<int4*>(r + i);
    } else {
#pragma unroll
      for (int i = 0; i < kExpandPer; ++i)
        if (o + i >= from_o && o + i < to_o) out[o + i] = r[i];
    }
    if (cut.start) {
      const auto node = [&](int rr, int pp) { return rr >= 0 ? rr : pp < base ? 0 : tail; };
      if (o < to_o) {
        const int p = q0 + o;
        // the first thread's predecessor lies in the step before
        const int was_node = p <= at ? prev : node(before, p - 1);
        long long was = tile_at(cut, (p > at ? p : at) - 1, was_node);
        const bool quick = whole && !bare && o + kExpandPer < E - q0;
        const long long mine = quick ? tile_at(cut, p + kExpandPer - 1, r[kExpandPer - 1]) : -1;
        if (quick && was <= mine) {
          // nodes do not decrease: boundary t lies at the first of these positions whose cost reaches it
          for (long long t = was + 1; t <= mine && t <= cut.n; ++t) {
            const long long reach = t << cut.shift;
            int below = 0;
#pragma unroll
            for (int i = 0; i < kExpandPer; ++i) below += p + i + (long long)kRowCost * r[i] < reach;
            cut.start[t] = p + (below < kExpandPer ? below : kExpandPer - 1);
          }
        } else {
#pragma unroll 1
          for (int i = 0; i < kExpandPer && o + i < to_o; ++i) {
            const int q = p + i;
            int rr = r[0];   // selected, not indexed: r stays in registers
#pragma unroll
            for (int k = 1; k < kExpandPer; ++k) rr = k == i ? r[k] : rr;
            if (q >= at) {
              const long long mine = tile_at(cut, q, node(rr, q));
              if (mine != was || q == E - 1) cut_tiles(cut, q, E, was, mine);
              was = mine;
            }
          }
        }
      }
      // the step's last node, for the next one
      if (stop < finish) {
        int x = kNone;
        for (int k = kExpandThreads / 32 - 1; k >= 0 && x == kNone; --k) x = s_last[k];
        prev = node(x, stop - 1);
      }
    }
    at = stop;
    q0 = at;
    __syncthreads();
  }
}

// Edge outputs start from zero in the reference (at::zeros); only edge ids that some chunk
// covers are written by the kernels here, so when the chunk table does not cover all E
// positions the output is cleared first: by expand_rows_kernel, or, on a plan not known to cover them all, by this
// kernel.  With full coverage it returns at once.
template <typename W>
__global__ void zero_uncovered_kernel(const PlanHeader* __restrict__ hdr, long long E, W* __restrict__ out,
                                      long long n) {
  if (hdr->cover_hi - hdr->cover_lo >= E) return;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = W(0);
}

// ---------------------------------------------------------------------------------------
// the tile walker
// ---------------------------------------------------------------------------------------
// Op interface (all members __device__):
//   static constexpr bool kRowOut;   // produces one output row per node (needs carries, gap fill)
//   static constexpr int  kUnroll;   // edges fetched ahead of the consuming loop
//   struct State; struct Fetched;
//   void setup(State&, int lane)                       once per warp
//   void begin(State&, int node, int lane)             a segment of `node` starts
//   void fetch(const State&, Fetched&, int other, int edge, int lane)   issue the edge's loads
//   void consume(State&, const Fetched&, int lane)     fold the edge into the state
//   -- kRowOut only --
//   struct CarryIn;
//   void store_row(const State&, int node, int lane)   the state is the node's final value
//   void store_carry(const State&, long long slot, int lane)    partial of an open segment
//   void store_identity(const State&, long long slot, int lane) neutral partial
//   void begin_merge(State&, int node, int lane)       neutral state, nothing loaded
//   void fetch_carry(const State&, CarryIn&, long long slot, int lane)   issue the loads of a stored partial
//   void merge_carry(State&, const CarryIn&, int lane)          fold it into the state
//   void zero_rows(long long lo, long long hi, int lane)        nodes [lo, hi) have no edge
//
// Level 0 (kCarryLevel = false) walks CSR positions.  A node whose positions cross a tile
// boundary is never stored at level 0: every tile writes the partial of its open first
// segment to carry slot 2t and of its open last segment to slot 2t+1, and rows_next[2t],
// rows_next[2t+1] name the node each slot belongs to (-1: slot unused).  A tile that lies
// wholly inside one node writes its partial to slot 2t and a neutral partial to 2t+1, so
// the slots of one node are always consecutive.  Level k+1 (kCarryLevel = true) walks that
// slot stream with the same code, merging partials instead of edges, stores the nodes whose
// slots end inside one of its tiles and emits the next stream, of two slots per tile, until a
// level fits one tile.  Every merge order is a function of (E, tile sizes) only.
template <class Op, bool kCarryLevel>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
walk_kernel(Op op, const PlanHeader* __restrict__ hdr, const int32_t* __restrict__ erow,
            const int32_t* __restrict__ other, const int32_t* __restrict__ eid, long long E, int tile,
            long long n_rows, int32_t* __restrict__ rows_next) {
  constexpr int U = Op::kUnroll;
  constexpr bool kOut = Op::kRowOut;
  constexpr bool kFill = Op::kRowOut && !kCarryLevel;
  const int lane = threadIdx.x & 31;
  const long long t = (long long)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  if (t * tile >= E) return;
  const long long j0 = t * tile, j1 = j0 + tile < E ? j0 + tile : E;

  if constexpr (kFill) {
    if (t == 0 && hdr->cover_hi <= hdr->cover_lo) {  // no covered position at all
      op.zero_rows(0, n_rows, lane);
      if (rows_next && lane == 0) { rows_next[0] = -1; rows_next[1] = -1; }
      return;
    }
  }

  typename Op::State st;
  op.setup(st, lane);
  const int before = j0 > 0 ? __ldg(erow + j0 - 1) : -1;
  const int first = __ldg(erow + j0);
  const bool head_open = before >= 0 && before == first;
  bool first_seg = true;    // the segment being built is the tile's first one
  int cur = -1;             // node of the segment being built, -1: none
  int last_valid = before;  // last node seen so far in position order (-1: none yet)
  int head_row = -1;        // node whose partial went to slot 2t

  for (long long jb = j0; jb < j1; jb += 32) {
    const long long j = jb + lane;
    const bool inb = j < j1;
    const int my_row = inb ? __ldg(erow + j) : -1;
    const int my_other = (!kCarryLevel && inb && other) ? __ldg(other + j) : 0;
    const int my_eid = (!kCarryLevel && inb && eid) ? __ldg(eid + j) : (int)j;
    const int n = (int)(j1 - jb < 32 ? j1 - jb : 32);
    // 32 positions without a node and no segment open: nothing to do (most slots of a carry level)
    if (cur < 0 && __ballot_sync(kFull, my_row >= 0) == 0u) continue;
    for (int k = 0; k < n; k += U) {
      typename Op::Fetched f[U];
      typename Op::CarryIn ci[U];
      int rr[U];
      (void)f; (void)ci;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kk = (k + u) & 31;
        const int r = __shfl_sync(kFull, my_row, kk);
        rr[u] = (k + u < n) ? r : -2;  // -2: beyond the tile, ignore
        if constexpr (kCarryLevel) {
          if (rr[u] >= 0) op.fetch_carry(st, ci[u], jb + k + u, lane);
        } else {
          const int c = __shfl_sync(kFull, my_other, kk);
          const int e = __shfl_sync(kFull, my_eid, kk);
          if (rr[u] >= 0) op.fetch(st, f[u], c, e, lane);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = rr[u];
        if (r == -2) continue;
        if (r != cur) {
          if (cur >= 0) {
            if constexpr (kOut) {
              if (first_seg && head_open) { op.store_carry(st, 2 * t, lane); head_row = cur; }
              else op.store_row(st, cur, lane);
            }
            first_seg = false;
            if constexpr (kFill) {
              if (r < 0) op.zero_rows((long long)cur + 1, n_rows, lane);  // coverage ended
            }
          }
          if (r >= 0) {
            if constexpr (kFill) {
              if (!(first_seg && head_open)) op.zero_rows((long long)last_valid + 1, r, lane);
            }
            if constexpr (kCarryLevel) op.begin_merge(st, r, lane); else op.begin(st, r, lane);
            last_valid = r;
          }
          cur = r;
        }
        if (r >= 0) {
          if constexpr (kCarryLevel) op.merge_carry(st, ci[u], lane); else op.consume(st, f[u], lane);
        }
      }
    }
  }
  int tail_row = -1;
  if constexpr (kOut) {
   if (cur >= 0) {
    const int next = j1 < E ? __ldg(erow + j1) : -1;
    const bool tail_open = next == cur;
    if (first_seg && head_open) {  // the whole tile lies inside one node that started earlier
      op.store_carry(st, 2 * t, lane);
      head_row = cur;
      if (tail_open) { op.store_identity(st, 2 * t + 1, lane); tail_row = cur; }
    } else if (tail_open) {
      op.store_carry(st, 2 * t + 1, lane);
      tail_row = cur;
    } else {
      op.store_row(st, cur, lane);
    }
    if constexpr (kFill) {
      if (next < 0) op.zero_rows((long long)cur + 1, n_rows, lane);  // last covered position
    }
   }
   if (rows_next && lane == 0) { rows_next[2 * t] = head_row; rows_next[2 * t + 1] = tail_row; }
  }
}

}  // namespace gk
