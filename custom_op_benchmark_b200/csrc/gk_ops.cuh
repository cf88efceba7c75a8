// The ops of walk_kernel (gk_common.cuh), for the row shapes that the gathering walker (gk_group.cuh) has no slot width
// for, and the kernels over edge feature rows that all heads of a node share.  Each cites the reference kernel whose
// arithmetic it computes (graphop/graphop_kernel.cu); none of them shares its scheduling: no transposed copies of the node
// tensors, no atomics.
#pragma once
#include "gk_common.cuh"

namespace gk {

// ---------------------------------------------------------------------------------------
// Edge-weighted aggregation of gathered feature rows:
//     out[node, h, :] = sum over the node's positions k of  w[eid[k], h] * feat(k)[h, :]
// feat(k) = x[other[k]]            (kEdgeFeat = false)  -> vector_spmm forward
//                                   (graphop_kernel.cu:123-128), vector_spmm backward dx over
//                                   the transposed CSR (:156-161), maskedmm backward dA / dB
//                                   (:105-110, w = dy, x = B or A)
// feat(k) = xe[eid[k]] (one D-vector shared by all heads, kEdgeFeat = true)
//                                   -> node_mul_edge backward dA (graphop_kernel.cu:66-71)
// ---------------------------------------------------------------------------------------
template <typename T, int V, int R, bool kEdgeFeat>
struct AggregateOp {
  using A = typename AccOf<T>::type;
  static constexpr const char* kName = kEdgeFeat ? "aggregate_edge_feat" : "aggregate";
  static constexpr bool kRowOut = true;
  static constexpr int kUnroll = (R * V * (int)sizeof(A) <= 16) ? 8 : (R * V * (int)sizeof(A) <= 32 ? 4 : 2);
  const T* __restrict__ w;    // (E, H)
  const T* __restrict__ x;    // (n_src, H, D) or (E, D)
  T* __restrict__ y;          // (n_dst, H, D)
  A* __restrict__ carry;      // (2 * n_tiles, HD) partial rows written by this level
  const A* carry_in;          // partial rows of the level below (carry levels only)
  int H, D, HD, S, feat0;

  struct State { SlotMap<R> sm; A acc[R][V]; };
  struct Fetched { A w[R]; A x[R][V]; };
  struct CarryIn { A x[R][V]; };

  __device__ __forceinline__ void setup(State& st, int lane) const { st.sm.init(lane, S, V, D, feat0); }
  __device__ __forceinline__ void begin(State& st, int, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int v = 0; v < V; ++v) st.acc[i][v] = A(0);
  }
  __device__ __forceinline__ void fetch(const State& st, Fetched& f, int c, int e, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (st.sm.ok[i]) {
        f.w[i] = to_acc<T>(__ldg(w + (long long)e * H + st.sm.head[i]));
        const T* src = kEdgeFeat ? x + (long long)e * D + st.sm.efeat[i] : x + (long long)c * HD + st.sm.feat[i];
        load_acc<T, V>(f.x[i], src);
      }
    }
  }
  __device__ __forceinline__ void consume(State& st, const Fetched& f, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int v = 0; v < V; ++v) st.acc[i][v] += f.w[i] * f.x[i][v];
  }
  __device__ __forceinline__ void store_row(const State& st, int node, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (st.sm.ok[i]) store_acc<T, V>(y + (long long)node * HD + st.sm.feat[i], st.acc[i]);
  }
  __device__ __forceinline__ void store_carry(const State& st, long long slot, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (st.sm.ok[i]) store_raw<A, V>(carry + slot * HD + st.sm.feat[i], st.acc[i]);
  }
  __device__ __forceinline__ void store_identity(const State& st, long long slot, int) const {
    A z[V];
#pragma unroll
    for (int v = 0; v < V; ++v) z[v] = A(0);
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (st.sm.ok[i]) store_raw<A, V>(carry + slot * HD + st.sm.feat[i], z);
  }
  __device__ __forceinline__ void begin_merge(State& st, int node, int lane) const { begin(st, node, lane); }
  __device__ __forceinline__ void fetch_carry(const State& st, CarryIn& c, long long slot, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (st.sm.ok[i]) load_raw<A, V>(c.x[i], carry_in + slot * HD + st.sm.feat[i]);
  }
  __device__ __forceinline__ void merge_carry(State& st, const CarryIn& c, int) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (st.sm.ok[i]) {
#pragma unroll
        for (int v = 0; v < V; ++v) st.acc[i][v] += c.x[i][v];
      }
  }
  __device__ __forceinline__ void zero_rows(long long lo, long long hi, int lane) const {
    if (hi <= lo) return;
    A z[V];
#pragma unroll
    for (int v = 0; v < V; ++v) z[v] = A(0);
    const long long n = (hi - lo) * S;
    for (long long k = lane; k < n; k += 32) {
      const long long node = lo + k / S;
      const int s = (int)(k % S);
      store_acc<T, V>(y + node * HD + feat0 + s * V, z);
    }
  }
};

// ---------------------------------------------------------------------------------------
// Sampled dot products on the edges:
//     y[eid[k], h] = sum_d a[node(k), h, d] * feat(k)[h, d]
// feat(k) = b[other[k]]  -> maskedmm forward (graphop_kernel.cu:45-53) and the dedata half of
//                           vector_spmm backward (:140-147, a = dy, b = x)
// feat(k) = be[eid[k]]   -> node_mul_edge forward (graphop_kernel.cu:24-32)
// GroupEdgeDot (gk_group.cuh) computes them; this is the form for any shape: scalar loads, a full-warp reduction per
// head.  Used where no slot width fits (2-byte elements with an odd D, heads wider than 4 KB).
// ---------------------------------------------------------------------------------------
template <typename T, bool kEdgeFeat>
struct EdgeDotAnyOp {
  using A = typename AccOf<T>::type;
  static constexpr bool kRowOut = false;
  static constexpr int kUnroll = 1;
  const T* __restrict__ a;
  const T* __restrict__ b;
  T* __restrict__ y;
  int H, D, HD;
  struct State { int node; };
  struct Fetched { int c, e; };
  struct CarryIn {};
  __device__ __forceinline__ void setup(State&, int) const {}
  __device__ __forceinline__ void begin(State& st, int node, int) const { st.node = node; }
  __device__ __forceinline__ void fetch(const State&, Fetched& f, int c, int e, int) const { f.c = c; f.e = e; }
  __device__ __forceinline__ void consume(State& st, const Fetched& f, int lane) const {
    const T* ar = a + (long long)st.node * HD;
    for (int h = 0; h < H; ++h) {
      const T* br = kEdgeFeat ? b + (long long)f.e * D : b + (long long)f.c * HD + h * D;
      A p = A(0);
      for (int d = lane; d < D; d += 32) p += to_acc<T>(__ldg(ar + h * D + d)) * to_acc<T>(__ldg(br + d));
      p = warp_sum(p);
      if (lane == 0) y[(long long)f.e * H + h] = from_acc<T>(p);
    }
  }
};

// (lse, delta) of one (destination node, head), written side by side by the destination pass so that the
// source pass fetches both with one load.  Rows hold `stat_heads(H)` pairs: H rounded up so that a row is
// a whole number of 16-byte pieces.
template <typename A> struct alignas(2 * sizeof(A)) StatPair { A lse, delta; };
// (p, ds) of one (edge, head): the probability and the score gradient the destination pass computed, kept
// for the source pass when the caller gives the transposed CSR's edge ids.  Rows hold stat_heads(H) pairs.
template <typename A> struct alignas(2 * sizeof(A)) EdgePair { A p, ds; };
__host__ __device__ constexpr int stat_heads(int H, int acc_bytes) { return acc_bytes >= 8 ? H : ((H + 1) & ~1); }

// ---------------------------------------------------------------------------------------
// node_mul_edge backward, edge half:  db[eid[k], :] = sum_h g[eid[k], h] * a[node(k), h, :]
// (graphop_kernel.cu:84-92), and the gradient of the edge term of the biased attention, the same sum with the score
// gradients ds that the destination pass left in the (p, ds) pairs, by position.  No reduction across edges.
//
// A thread owns one slot of V features of kMixPer consecutive positions: the positions' nodes, ids and g are loaded
// together, the node's slots of all heads stay in registers while the node lasts.  Consecutive threads own the slots of a
// position, so that a store covers whole rows.  Bound by the written tensor; with a thread per position and slot, which
// reads the H slots of its node again for every edge, 17.8M edges, 4 x 32 fp32, took 1.07 ms.
// kH: the head count when it is 1, 2, 4 or 8, 0: read it from H, one head at a time.  ds_shift >= 0: D / V is that power
// of two.
// ---------------------------------------------------------------------------------------
constexpr int kMixPer = 8;
// The edge ids of kMixPer positions from j0 (their own numbers where there are none), in two loads where the table allows it: as
// eight they are as many accesses to the L1 as the rows.  17.8M edges, 4 x 32 fp32: edge_mix 705 -> 652 us, edge_feat_dot 646
// -> 601 us.
__device__ __forceinline__ void mix_ids(int (&edge)[kMixPer], const int32_t* __restrict__ eid, long long j0, long long E) {
  if (eid && ((uintptr_t)eid & 15) == 0 && j0 + kMixPer <= E) {
#pragma unroll
    for (int i = 0; i < kMixPer; i += 4) *reinterpret_cast<int4*>(edge + i) = __ldg(reinterpret_cast<const int4*>(eid + j0 + i));
    return;
  }
#pragma unroll
  for (int i = 0; i < kMixPer; ++i) edge[i] = eid && j0 + i < E ? __ldg(eid + j0 + i) : (int)(j0 + i);
}
template <typename T, int V, int kH, bool kPairs>
__global__ void __launch_bounds__(256)
edge_mix_kernel(const int32_t* __restrict__ erow, const int32_t* __restrict__ eid, const T* __restrict__ dy,
                const EdgePair<typename AccOf<T>::type>* __restrict__ pairs, const T* __restrict__ a, T* __restrict__ db,
                long long E, int H, int Hp, int D, int ds_shift) {
  using A = typename AccOf<T>::type;
  constexpr int P = kMixPer, N = kH ? kH : 1;
  const unsigned ds = (unsigned)(D / V);
  const int nh = kH ? kH : H;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long chunk = ds_shift >= 0 ? idx >> ds_shift : idx <= 0xffffffffLL ? (unsigned)idx / ds : idx / ds;
  const int s = (int)(idx - chunk * ds);
  const long long j0 = chunk * P;
  if (j0 >= E) return;
  alignas(16) int node[P], edge[P];
  const bool whole = j0 + P <= E;
  if (whole) {
#pragma unroll
    for (int i = 0; i < P; i += 4) *reinterpret_cast<int4*>(node + i) = __ldg(reinterpret_cast<const int4*>(erow + j0 + i));
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) node[i] = j0 + i < E ? __ldg(erow + j0 + i) : -2;   // -2: nothing to do
  }
  mix_ids(edge, kPairs ? nullptr : eid, j0, E);
  const T* base = a + s * V;
  const auto slot_of = [&](int r, int h) { return base + ((long long)r * nh + h) * D; };
  const auto g_of = [&](int i, int h) -> A {
    if constexpr (kPairs) return pairs[(long long)edge[i] * Hp + h].ds;
    else return to_acc<T>(__ldg(dy + (long long)edge[i] * nh + h));
  };
  if constexpr (kH != 0) {
    A g[P][N];
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (node[i] >= 0) {
        if constexpr (!kPairs && N * sizeof(T) <= 16 && N > 1) {
          // rows of g start at multiples of their size wherever the tensor does (checked by the launch)
          load_acc<T, N>(g[i], dy + (long long)edge[i] * N);
        } else if constexpr (!kPairs && N > 1) {
          constexpr int per = 16 / (int)sizeof(T);
#pragma unroll
          for (int h = 0; h < N; h += per) load_acc<T, per>(*reinterpret_cast<A(*)[per]>(&g[i][h]), dy + (long long)edge[i] * N + h);
        } else {
#pragma unroll
          for (int h = 0; h < N; ++h) g[i][h] = g_of(i, h);
        }
      }
    A av[N][V];
    int cur = -1;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      if (node[i] < 0) {
        if (kPairs && node[i] == -1) {   // a position of no chunk has no gradient
          A zero[V];
#pragma unroll
          for (int v = 0; v < V; ++v) zero[v] = A(0);
          store_acc<T, V>(db + (long long)edge[i] * D + s * V, zero);
        }
        continue;
      }
      if (node[i] != cur) {
        cur = node[i];
#pragma unroll
        for (int h = 0; h < N; ++h) load_acc<T, V>(av[h], slot_of(cur, h));
      }
      A acc[V];
#pragma unroll
      for (int v = 0; v < V; ++v) acc[v] = A(0);
#pragma unroll
      for (int h = 0; h < N; ++h)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += g[i][h] * av[h][v];
      store_acc<T, V>(db + (long long)edge[i] * D + s * V, acc);
    }
  } else {
    A acc[P][V];
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int v = 0; v < V; ++v) acc[i][v] = A(0);
    for (int h = 0; h < nh; ++h) {
      A av[V], g[P];
      int cur = -1;
#pragma unroll
      for (int i = 0; i < P; ++i) g[i] = node[i] >= 0 ? g_of(i, h) : A(0);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        if (node[i] < 0) continue;
        if (node[i] != cur) {
          cur = node[i];
          load_acc<T, V>(av, slot_of(cur, h));
        }
#pragma unroll
        for (int v = 0; v < V; ++v) acc[i][v] += g[i] * av[v];
      }
    }
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (node[i] >= 0 || (kPairs && node[i] == -1)) store_acc<T, V>(db + (long long)edge[i] * D + s * V, acc[i]);
  }
}

// y[edge, h] = a[node, h, :] . b[edge, :], b an edge tensor shared by the heads (graphop_kernel.cu:16-34): edge_mix_kernel
// the other way round.  A thread owns one slot of kMixPer consecutive positions and the node's slots of all kH heads, so
// that an edge's row is read once, whatever the number of heads; the partial sums of DS lanes meet by halves: a lane gives
// away half of its positions at every step and ends with one position's scores, written together.  The sums are formed in
// the order of Geo::ordered_dot.  Bound by reading b; on the gathering walker, which copies the row once per head, 17.8M
// edges, 4 x 32 fp32, took 1.05 ms.
template <typename T, int V, int kH, int DS>
__global__ void __launch_bounds__(256)
edge_feat_dot_kernel(const int32_t* __restrict__ erow, const int32_t* __restrict__ eid, const T* __restrict__ a,
                     const T* __restrict__ b, T* __restrict__ y, long long E, int D) {
  using A = typename AccOf<T>::type;
  constexpr int P = kMixPer, B = DS < P ? DS : P;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
  const int s = threadIdx.x & (DS - 1);
  const long long j0 = idx / DS * P;
  alignas(16) int node[P], edge[P];
  if (j0 + P <= E) {
#pragma unroll
    for (int i = 0; i < P; i += 4) *reinterpret_cast<int4*>(node + i) = __ldg(reinterpret_cast<const int4*>(erow + j0 + i));
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) node[i] = j0 + i < E ? __ldg(erow + j0 + i) : -1;
  }
  mix_ids(edge, eid, j0, E);
  using M = typename Mover<sizeof(T) * V>::type;
  union { M m; T t[V]; } feat[P];
#pragma unroll
  for (int i = 0; i < P; ++i)
    if (node[i] >= 0) feat[i].m = __ldg(reinterpret_cast<const M*>(b + (long long)edge[i] * D + s * V));
  A av[kH][V], part[P][kH];
  int cur = -1;
#pragma unroll
  for (int i = 0; i < P; ++i) {
#pragma unroll
    for (int h = 0; h < kH; ++h) part[i][h] = A(0);
    if (node[i] < 0) continue;
    if (node[i] != cur) {
      cur = node[i];
#pragma unroll
      for (int h = 0; h < kH; ++h) load_acc<T, V>(av[h], a + ((long long)cur * kH + h) * D + s * V);
    }
#pragma unroll
    for (int h = 0; h < kH; ++h) {
      part[i][h] = av[h][0] * to_acc<T>(feat[i].t[0]);
#pragma unroll
      for (int v = 1; v < V; ++v) part[i][h] = fma(av[h][v], to_acc<T>(feat[i].t[v]), part[i][h]);
    }
  }
#pragma unroll
  for (int k = 0; k < P; k += B) {
#pragma unroll
    for (int d = 1; d < B; d <<= 1) {
      const bool up = (s & d) != 0;
#pragma unroll
      for (int j = 0; j < B / 2 / d; ++j)
#pragma unroll
        for (int h = 0; h < kH; ++h) {
          const A keep = up ? part[k + 2 * j + 1][h] : part[k + 2 * j][h];
          const A give = up ? part[k + 2 * j][h] : part[k + 2 * j + 1][h];
          part[k + j][h] = keep + __shfl_xor_sync(kFull, give, d);
        }
    }
#pragma unroll
    for (int d = B; d < DS; d <<= 1)
#pragma unroll
      for (int h = 0; h < kH; ++h) part[k][h] += __shfl_xor_sync(kFull, part[k][h], d);
    const long long j = j0 + k + (s & (B - 1));   // the position whose sums ended here
    if (s < B && j < E && __ldg(erow + j) >= 0) {
      const long long e = eid ? (long long)__ldg(eid + j) : j;
      constexpr int per = kH * (int)sizeof(T) <= 16 ? kH : 16 / (int)sizeof(T);
#pragma unroll
      for (int h = 0; h < kH; h += per) store_acc<T, per>(y + e * kH + h, *reinterpret_cast<const A(*)[per]>(&part[k][h]));
    }
  }
}

}  // namespace gk
