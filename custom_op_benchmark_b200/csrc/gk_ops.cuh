// The per-edge bodies ("ops") that the tile walker of gk_common.cuh drives, one per
// reference kernel family.  Each op cites the reference kernel whose arithmetic it computes
// (graphop/graphop_kernel.cu); none of them shares its scheduling: no transposed copies of
// the node tensors, no atomics, 128-bit loads of whole feature rows.
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

// ---------------------------------------------------------------------------------------
// node_mul_edge backward, edge half:  dB[eid[k], :] = sum_h dy[eid[k], h] * A[node(k), h, :]
// (graphop_kernel.cu:84-92).  One thread per (position, D-slot); no reduction across edges.
// ---------------------------------------------------------------------------------------
// kH: the head count when it is 1, 2, 4 or 8 (all of an edge's loads are then issued before the first use),
// 0: read it from H.  ds_shift >= 0: D / V is that power of two (no 64-bit division per element).
template <typename T, int V, int kH>
__global__ void __launch_bounds__(256)
edge_mix_heads_kernel(const int32_t* __restrict__ erow, const int32_t* __restrict__ eid, const T* __restrict__ dy,
                      const T* __restrict__ a, T* __restrict__ db, long long E, int H, int D, int ds_shift) {
  using A = typename AccOf<T>::type;
  const int ds = D / V;
  const int nh = kH ? kH : H;
  const long long total = E * ds;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    const long long j = ds_shift >= 0 ? (idx >> ds_shift) : idx / ds;
    const int s = (int)(idx - j * ds);
    const int node = __ldg(erow + j);
    if (node < 0) continue;
    const long long e = eid ? (long long)__ldg(eid + j) : j;
    const T* arow = a + (long long)node * nh * D + s * V;
    const T* grow = dy + e * nh;
    A acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = A(0);
    if constexpr (kH != 0) {
      A g[kH], av[kH][V];
#pragma unroll
      for (int h = 0; h < kH; ++h) {
        g[h] = to_acc<T>(__ldg(grow + h));
        load_acc<T, V>(av[h], arow + (long long)h * D);
      }
#pragma unroll
      for (int h = 0; h < kH; ++h)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += g[h] * av[h][v];
    } else {
      for (int h = 0; h < nh; ++h) {
        const A g = to_acc<T>(__ldg(grow + h));
        A av[V];
        load_acc<T, V>(av, arow + (long long)h * D);
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += g * av[v];
      }
    }
    store_acc<T, V>(db + e * D + s * V, acc);
  }
}

// (lse, delta) of one (destination node, head), written side by side by the destination pass so that the
// source pass fetches both with one load.  Rows hold `stat_heads(H)` pairs: H rounded up so that a row is
// a whole number of 16-byte pieces.
template <typename A> struct alignas(2 * sizeof(A)) StatPair { A lse, delta; };
// (p, ds) of one (edge, head): the probability and the score gradient the destination pass computed, kept
// for the source pass when the caller gives the transposed CSR's edge ids.  Rows hold stat_heads(H) pairs.
template <typename A> struct alignas(2 * sizeof(A)) EdgePair { A p, ds; };
__host__ __device__ constexpr int stat_heads(int H, int acc_bytes) { return acc_bytes >= 8 ? H : ((H + 1) & ~1); }

// Gradient of the edge term of the biased attention:  d_rel[j, :] = sum_h ds[j, h] * q[node(j), h, :]
// (the dB half of node_mul_edge backward, graphop_kernel.cu:79-93, with the score gradients the destination
// pass left in `pairs`).  One thread per (position, slot of V features); consecutive threads cover a position's
// features, consecutive positions of a node re-read its q row from L1 / L2; positions no chunk covers get 0.
// shift = log2(D / V) when that is a power of two, else -1.
template <typename T, int V>
__global__ void __launch_bounds__(256)
bias_grad_kernel(const int32_t* __restrict__ erow, const EdgePair<typename AccOf<T>::type>* __restrict__ pairs,
                 const T* __restrict__ q, T* __restrict__ d_rel, long long E, int H, int Hp, int D, int shift) {
  using A = typename AccOf<T>::type;
  const int slots = D / V;
  const long long stride = (long long)gridDim.x * blockDim.x, total = E * slots;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const long long j = shift >= 0 ? (i >> shift) : i / slots;
    const int d = (int)(i - j * slots) * V;
    const int r = __ldg(erow + j);
    A sum[V];
#pragma unroll
    for (int e = 0; e < V; ++e) sum[e] = A(0);
    if (r >= 0) {
      const T* qrow = q + (long long)r * H * D + d;
      const EdgePair<A>* pr = pairs + j * Hp;
      for (int h = 0; h < H; ++h) {
        const A ds = pr[h].ds;
        A qv[V];
        load_acc<T, V>(qv, qrow + (long long)h * D);
#pragma unroll
        for (int e = 0; e < V; ++e) sum[e] += ds * qv[e];
      }
    }
    store_acc<T, V>(d_rel + j * D + d, sum);
  }
}

}  // namespace gk
