// The summing walker: sums of gathered rows with per-edge weights that are known beforehand (aggregation, the source side of
// the attention backward from stored pairs), for elements of 4 and 8 bytes.  The decomposition and the carry records are the
// gathering walker's (gk_group.cuh); what differs is how rows arrive and in which groups a row's edges are added up: blocks of
// G positions (the lanes of a group, 4 to 32), then their totals (flush).  Nothing but multiply-adds is
// done with a row, so a lane holds its slot of kUnroll positions' rows in registers and loads the slot of the position kUnroll
// on where it was used: kUnroll rows per lane group are on their way whatever the lengths of the nodes.  The loads go through
// the L1, which serves the nodes that many edges share (the ring's copies pass it by), and shared memory holds the indices
// and weights of two blocks of positions alone, so that most of the 256 KB are L1.  Bound by the L2's answers to what misses
// there, and by issue slots on short rows.
//
// Against the gathering walker, B200.  Tables that fit the L2: 15360 nodes of 30 edges, 8 x 64 fp32, 94 -> 70 us (13.5 TB/s
// of rows); 800 thousand skewed edges, 4 x 50, 180 -> 126 us; the source side of 4096 nodes of 16 edges, 8 x 64, 34 -> 23 us.
// Larger ones with hubs: 50M edges to hubs, 2 x 64, 2.85 -> 1.85 ms; R-MAT 20, 4 x 32, 0.96 + 1.12 -> 0.90 + 1.06 ms; the
// source side of R-MAT 21, 4 x 32, 4.40 -> 4.09 ms.  Wide rows of few nodes: choose_walker.  It loses, and the gathering walker
// stays, on larger tables without hubs (321 thousand nodes, 6.3M edges, 2 x 64: 347 + 438 against 410 + 474 us; blocks of 47,
// 4 x 64: 1.95 against 3.6 ms: fewer rows are on their way, and the L1 has nothing to add), on tables of 2 GB, which the DRAM
// bounds whatever the L1 holds (R-MAT 22, 1 x 128: 3.46 + 4.28 against 4.00 + 4.75 ms), and for 2-byte elements, whose
// accumulators are twice as many registers per slot (R-MAT 18, 2 x 64 bf16: 215 against 236 us; pairs, 4 x 64: 541 against 595 us).
#pragma once
#include "gk_group.cuh"

namespace gk {

__device__ __forceinline__ void lds_ints(int (&v)[4], unsigned at) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at));
}
__device__ __forceinline__ void sts_int(unsigned at, int v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }

// Launch shape of an op that gathers kRows rows per position; kScalar bytes per edge and head wait in a table.  Two warps per
// block: with one, the 32 blocks an SM takes are too few warps; with more, a block holds its place until the slowest is done.
template <class GEO, int kRows, int kScalar>
struct SumShape {
  static constexpr bool kSums = true, kOptional = true;
  static constexpr int kWarps = 2;
  static constexpr int kUnroll = 4;
  static constexpr int kIdsBytes = 32 * 4;                                 // the gathered rows' ids of a block of positions
  static constexpr int kScalarBytes = kScalar;
  static constexpr int kTableAt = 2 * kIdsBytes;
  static constexpr int kTable = 32 * GEO::kHeads * kScalar;
  static constexpr int kWarpBytes = kTableAt + 2 * kTable;
  static constexpr int kWords = GEO::V * (int)sizeof(typename GEO::A) / 4;
  static constexpr int kRegs = 44 + kRows * (kUnroll * GEO::SB / 4 + 2 * kWords);   // fewer spill in the loop
  static constexpr int kRegsRounded = (kRegs + 7) / 8 * 8;
  static constexpr int kMinCtas = 65536 / (32 * kWarps * kRegsRounded);
  static_assert(kMinCtas * (kWarps * kWarpBytes + 1024) <= 226 * 1024, "the registers say how many blocks are resident");
};

// Op interface (all members __device__), on top of its Geo and SumShape:
//   State, Carry, Rows (a position's slots)
//   setup(st, gl, hb)
//   fetch(st, rows, id)                load the slots of row id
//   scalar_of(h, edge)                 where the edge's scalars of head h are
//   fold(st, rows, tab)                add a position's rows; tab: the table's entry of the position and this lane's head
//   flush(st)                          a block of positions is done: its sums join those of the node's blocks before it, so that
//                                      a long run is summed in two levels (in one, a tile's hundreds of edges one after the
//                                      other, R-MAT 18's dv is 1.16e-7 off float64 instead of 0.83e-7); sum_span bounds the second
//   store_row(st, node), zero_row(st, node), begin_merge(st), merge(st, Carry), load_carry, save_carry, kCarryElems
template <class Op>
__global__ void __launch_bounds__(Op::kWarps * 32, Op::kMinCtas)
sum_walk_kernel(const __grid_constant__ Op op, const __grid_constant__ WalkArgs a) {
  constexpr int NE = Op::NE, G = Op::G, U = Op::kUnroll;
  constexpr unsigned kOneLane = NE == 1 ? 1u : NE == 2 ? 0x00010001u : NE == 4 ? 0x01010101u : 0x11111111u;
  constexpr unsigned kBatch = ((1u << U) - 1u) * kOneLane;
  extern __shared__ uint4 gk_ring[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane / G, gl = lane & (G - 1);
  const int hb = blockIdx.y;
  const unsigned t0 = (blockIdx.x * Op::kWarps + w) * NE;   // the warp's first tile
  if (t0 >= a.n_tiles || not_asked<Op>(a)) return;
  const unsigned t = t0 + g;
  const bool here = t < a.n_tiles;
  int j0, n;   // the group's first position and their number
  tile_of<G>(a, t, here, j0, n);
  int longest = n;
#pragma unroll
  for (int o = G; o < 32; o <<= 1) {
    const int x = __shfl_xor_sync(kFull, longest, o);
    longest = x > longest ? x : longest;
  }

  typename Op::State st;
  op.setup(st, gl, hb);
  if (t0 == 0 && a.hdr->cover_hi <= a.hdr->cover_lo)   // no covered position at all
    for (long long r = g; r < a.n_rows; r += NE) op.zero_row(st, r);

  // a block of G positions per group, one per lane: node (-1: none, -2: past the tile), row to gather, edge id
  const auto load_block = [&](int b, int& r, int& o, int& e) {
    const int i = b * G + gl;
    const unsigned j = (unsigned)j0 + i;
    r = -2;
    o = e = 0;
    if (i < n) {
      r = __ldg(a.erow + j);
      e = a.eid ? __ldg(a.eid + j) : (int)j;
      o = __ldg(a.other + j);
    }
    if (r < 0) o = e = 0;   // row 0 is loaded in its place and not used
  };
  constexpr bool kFar = G <= 8;   // short blocks: the indices of the block after the next are asked for, too
  int r0, r1, o1, e1;
  [[maybe_unused]] int r2, o2, e2;
  load_block(0, r1, o1, e1);
  if constexpr (kFar) load_block(1, r2, o2, e2);
  const int before = here && j0 > 0 ? __ldg(a.erow + j0 - 1) : -1;

  const unsigned mem = (unsigned)__cvta_generic_to_shared(gk_ring) + w * Op::kWarpBytes;
  const unsigned ids = mem + g * G * 4;   // this group's part of a block's ids
  // The scalars of a block of positions, one position per lane: asked for half a block ahead, read by all lanes of the group
  // afterwards.
  constexpr int SC = Op::kScalarBytes, TB = Op::kTable, ENTRY = Op::kHeads * SC;
  const unsigned table = mem + Op::kTableAt;
  const auto fetch_scalars = [&](unsigned tab) {
    const bool live = r1 >= 0;
    if constexpr (ENTRY % 16 == 0 && Op::LT > 0) {
      if (op.wide_scalars) {
        const unsigned char* src = reinterpret_cast<const unsigned char*>(op.scalar_of(hb * Op::kHeads, e1));
#pragma unroll
        for (int k = 0; k < ENTRY; k += 16) cp_async_slot<16>(tab + lane * ENTRY + k, src + k, live);
        return;
      }
    }
    const int per = op.block_heads(), pieces = op.parts * op.H - hb * per;   // heads in this block
#pragma unroll
    for (int k = 0; k < Op::kHeads; ++k) {
      const bool some = live && k < per && k < pieces;
      int h = hb * per + k;
      if (op.parts != 1) h /= op.parts;
      cp_async_slot<SC>(tab + lane * ENTRY + k * SC, op.scalar_of(some ? h : 0, e1), some);
    }
  };
  const unsigned my_scalar = table + g * G * ENTRY + op.scalar_at(gl) * SC;

  // Block b, in r1, o1 and e1: its ids to shared memory, its scalars asked for.  starts: bit of every lane whose position
  // starts another node than the one before it, the last of which is `up`; gaps: whose position has no edge
  unsigned starts0, gaps0, starts1, gaps1;
  const auto publish = [&](int b, int up, unsigned& starts, unsigned& gaps) {
    sts_int(mem + (b & 1) * Op::kIdsBytes + lane * 4, o1);
    fetch_scalars(table + (b & 1) * TB);
    gaps = __ballot_sync(kFull, r1 < 0);
    int prev = __shfl_up_sync(kFull, r1, 1, G);
    if (gl == 0) prev = up;
    starts = __ballot_sync(kFull, r1 != prev && r1 != -2);
    __syncwarp();
  };
  publish(0, -3, starts0, gaps0);
  r0 = r1;
  const int first = __shfl_sync(kFull, r0, 0, G);
  const bool head_open = before >= 0 && before == first;
  bool first_seg = true;
  int cur = -1, last_valid = before;
  // the tile's record `which` (0: open first run, 1: open last run) and what it stands for
  const auto record = [&](int which) { return (size_t)hb * 2 * a.n_tiles + 2 * (size_t)t + which; };
  const auto save = [&](int which, uint32_t id) {
    op.save_carry(st, reinterpret_cast<typename Op::A*>(a.carry) + record(which) * Op::kCarryElems, gl);
    if (gl == 0) a.rows[record(which)] = id;
  };
  const auto end_node = [&](int r) {   // the open node ends where r begins (below zero: where coverage ends)
    if (cur >= 0) {
      if (first_seg && head_open) save(0, 2u * (unsigned)cur + 1u);
      else op.store_row(st, cur);
      first_seg = false;
      if (r < 0)
        for (long long z = (long long)cur + 1; z < a.n_rows; ++z) op.zero_row(st, z);
    }
    if (r >= 0) {
      if (!(first_seg && head_open))
        for (int z = last_valid + 1; z < r; ++z) op.zero_row(st, z);
      last_valid = r;
    }
    op.begin_merge(st);
    cur = r;
  };

  typename Op::Rows rows[U];
  int next[U];   // the rows of the batch after this one
  lds_ints(next, ids);
#pragma unroll
  for (int v = 0; v < U; ++v) op.fetch(st, rows[v], next[v]);

#pragma unroll 1
  for (int b = 0; b * G < longest; ++b) {
    if constexpr (kFar) {
      r1 = r2; o1 = o2; e1 = e2;
      load_block(b + 2, r2, o2, e2);
    } else {
      load_block(b + 1, r1, o1, e1);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();   // every lane's part of this block's table has landed
    const unsigned odd = b & 1, tab0 = my_scalar + odd * TB;
    const unsigned special = starts0 | gaps0;
#pragma unroll 1
    for (int i = 0; i < G; i += U) {
      if (b * G + i >= longest) break;
      if (i == G / 2 / U * U) publish(b + 1, __shfl_sync(kFull, r0, G - 1, G), starts1, gaps1);
      lds_ints(next, i + U == G ? ids + (odd ^ 1) * Op::kIdsBytes : ids + odd * Op::kIdsBytes + (i + U) * 4);
      const unsigned tab = tab0 + i * ENTRY;
      if (((special >> i) & kBatch) == 0) {
#pragma unroll
        for (int v = 0; v < U; ++v) {
          op.fold(st, rows[v], tab + v * ENTRY);
          op.fetch(st, rows[v], next[v]);
        }
      } else {
#pragma unroll
        for (int v = 0; v < U; ++v) {
          if ((starts0 >> (i + v)) & kOneLane) {
            const int r = __shfl_sync(kFull, r0, i + v, G);
            if ((starts0 >> (g * G + i + v)) & 1u) end_node(r);
          }
          if (!((gaps0 >> (g * G + i + v)) & 1u)) op.fold(st, rows[v], tab + v * ENTRY);
          op.fetch(st, rows[v], next[v]);
        }
      }
    }
    op.flush(st);
    r0 = r1;
    starts0 = starts1; gaps0 = gaps1;
  }
  cp_async_commit();   // what the last block published past the end, too: no copy is under way when the warp leaves
  cp_async_wait<0>();

  uint32_t tail_id = kNoRow;
  if (cur >= 0) {
    const int after = n < (int)a.E - j0 ? __ldg(a.erow + j0 + n) : -1;
    const bool tail_open = after == cur;
    if (first_seg && head_open) {   // the whole tile lies inside one node that started earlier
      save(0, 2u * (unsigned)cur + 1u);
      first_seg = false;
      if (tail_open) tail_id = 2u * (unsigned)cur;
    } else if (tail_open) {
      save(1, 2u * (unsigned)cur + 1u);
      tail_id = 2u * (unsigned)cur + 1u;
    } else {
      op.store_row(st, cur);
    }
    if (after < 0)   // last covered position
      for (long long z = (long long)cur + 1; z < a.n_rows; ++z) op.zero_row(st, z);
  }
  if (a.carry && here && gl == 0) {
    if (first_seg || !head_open) a.rows[record(0)] = kNoRow;
    a.rows[record(1)] = tail_id;
  }
}

// y[node, h, :] = sum over the node's positions of w[edge, h] * x[other] (the kernels of graphop_kernel.cu this stands for:
// see AggregateOp)
template <class GEO>
struct SumAggregate : GEO, SumShape<GEO, 1, (int)sizeof(typename GEO::T)> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr const char* kName = "aggregate";
  static constexpr bool kRowOut = true;
  const T* __restrict__ w;
  const T* __restrict__ x;
  T* __restrict__ y;
  bool wide_scalars;   // an edge's weights are whole 16-byte pieces for every block of heads
  struct State { typename GEO::Lane ln; const unsigned char* xb; F acc[1], sum[1]; };
  struct Carry { F x[1]; };
  struct Rows { typename GEO::Word x; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.xb = reinterpret_cast<const unsigned char*>(x + st.ln.off);
    begin_merge(st);
  }
  __device__ __forceinline__ void fetch(const State& st, Rows& r, int id) const {
    this->fetch_slot(st.ln, r.x, st.xb, id, this->rowb);
  }
  __device__ __forceinline__ const void* scalar_of(int h, int e) const {
    return w + ((unsigned long long)(unsigned)e * (unsigned)this->H + h);
  }
  __device__ __forceinline__ void fold(State& st, const Rows& r, unsigned tab) const {
    F f;
    frag_unpack<T, GEO::SB>(f, r.x);
    T wt;
    lds(wt, tab);
    st.acc[0].axpy(to_acc<T>(wt), f);
  }
  __device__ __forceinline__ void flush(State& st) const {
    st.sum[0].add(st.acc[0]);
    st.acc[0].zero();
  }
  __device__ __forceinline__ void store_row(State& st, int node) const {
    flush(st);
    this->store_row_slots(st.ln, y + (long long)node * this->HD + st.ln.off, st.sum);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const { this->zero_slots(st.ln, y, n); }
  static constexpr int kCarryElems = GEO::kAccs;
  __device__ __forceinline__ void begin_merge(State& st) const { st.acc[0].zero(); st.sum[0].zero(); }
  __device__ __forceinline__ void save_carry(State& st, A* rec, int gl) const {
    flush(st);
    this->save_acc(rec, gl, st.sum);
  }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const { this->load_acc_raw(c.x, rec, gl); }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const { st.sum[0].add(c.x[0]); }
};

// The attention backward's source side over the transposed CSR from the pairs that the destination side left by edge id:
// dv[c] = sum p dO[dst], dk[c] = sum ds q[dst]
template <class GEO>
struct SumAttnPairs : GEO, SumShape<GEO, 2, 2 * (int)sizeof(typename GEO::A)> {
  using T = typename GEO::T;
  using A = typename GEO::A;
  using F = typename GEO::F;
  static constexpr const char* kName = "attention_bwd_src";
  static constexpr bool kRowOut = true;
  const T* __restrict__ q;
  const T* __restrict__ dout;
  const EdgePair<A>* __restrict__ pd;
  T* __restrict__ dk;
  T* __restrict__ dv;
  int Hp;
  bool wide_scalars;
  struct State { typename GEO::Lane ln; const unsigned char *qb, *gb; F ak[1], av[1], sk[1], sv[1]; };
  struct Carry { F k[1], v[1]; };
  struct Rows { typename GEO::Word q, g; };
  __device__ __forceinline__ void setup(State& st, int gl, int hb) const {
    st.ln = this->lane_of(gl, hb);
    st.qb = reinterpret_cast<const unsigned char*>(q + st.ln.off);
    st.gb = reinterpret_cast<const unsigned char*>(dout + st.ln.off);
    begin_merge(st);
  }
  __device__ __forceinline__ void fetch(const State& st, Rows& r, int id) const {
    this->fetch_slot(st.ln, r.q, st.qb, id, this->rowb);
    this->fetch_slot(st.ln, r.g, st.gb, id, this->rowb);
  }
  __device__ __forceinline__ const void* scalar_of(int h, int e) const {
    return pd + ((unsigned long long)(unsigned)e * (unsigned)Hp + h);
  }
  __device__ __forceinline__ void fold(State& st, const Rows& r, unsigned tab) const {
    F fq, fg;
    frag_unpack<T, GEO::SB>(fq, r.q);
    frag_unpack<T, GEO::SB>(fg, r.g);
    A p, ds;
    lds2(p, ds, tab);
    st.av[0].axpy(p, fg);
    st.ak[0].axpy(ds, fq);
  }
  __device__ __forceinline__ void flush(State& st) const {
    st.sk[0].add(st.ak[0]);
    st.sv[0].add(st.av[0]);
    st.ak[0].zero();
    st.av[0].zero();
  }
  __device__ __forceinline__ void store_row(State& st, int node) const {
    flush(st);
    const long long at = (long long)node * this->HD + st.ln.off;
    this->store_row_slots(st.ln, dk + at, st.sk);
    this->store_row_slots(st.ln, dv + at, st.sv);
  }
  __device__ __forceinline__ void zero_row(const State& st, long long n) const {
    this->zero_slots(st.ln, dk, n);
    this->zero_slots(st.ln, dv, n);
  }
  static constexpr int kCarryElems = 2 * GEO::kAccs;
  __device__ __forceinline__ void begin_merge(State& st) const {
    st.ak[0].zero(); st.av[0].zero();
    st.sk[0].zero(); st.sv[0].zero();
  }
  __device__ __forceinline__ void save_carry(State& st, A* rec, int gl) const {
    flush(st);
    this->save_acc(rec, gl, st.sk);
    this->save_acc(rec + GEO::kAccs, gl, st.sv);
  }
  __device__ __forceinline__ void load_carry(Carry& c, const A* rec, int gl) const {
    this->load_acc_raw(c.k, rec, gl);
    this->load_acc_raw(c.v, rec + GEO::kAccs, gl);
  }
  __device__ __forceinline__ void merge(State& st, const Carry& c) const { st.sk[0].add(c.k[0]); st.sv[0].add(c.v[0]); }
};

}  // namespace gk
