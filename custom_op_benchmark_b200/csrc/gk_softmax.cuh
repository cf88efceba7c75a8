// Sparse row softmax over each node's edges, forward and backward
// (reference: graphop_kernel.cu:170-202 and :208-230, three and two launches of h-thread
// blocks with one atomic per edge; here one streaming pass with segmented scans).
//
// Mapping: a block takes a tile of 1024 CSR positions, each thread four consecutive ones with H heads.  Runs of equal
// erow[] inside the tile are segments.  A segment's total (its maximum, then its sum) is folded inside the thread first,
// then over the lanes of the warp by one segmented scan, then over the warps through shared memory, so the shuffles are a
// quarter of those of a scan per 32 positions, and a total reaches back to the positions before it by one indexed shuffle.
// The order of every sum is fixed by (E, H).  Bound by the edge tensors' traffic.
//
// Nodes whose positions cross a tile boundary: the tile leaves the partial statistics of its open first / last segment
// in slots 2t / 2t+1 and the node each belongs to in slot_rows (-1: unused); a tile that lies inside one node uses the
// first slot alone.  The slots of a node are then one odd slot, of the tile it starts in, and the even ones of the tiles
// after it.  softmax_finish_kernel merges them and revisits the positions of open segments.
#pragma once
#include "gk_common.cuh"

namespace gk {

constexpr int kSoftmaxThreads = 256;
constexpr int kSoftmaxWarps = kSoftmaxThreads / 32;
constexpr int kSoftmaxPer = 4;
constexpr int kSoftmaxTile = kSoftmaxThreads * kSoftmaxPer;

template <typename T, int N>
__device__ __forceinline__ void load_vec(typename AccOf<T>::type (&dst)[N], const T* __restrict__ p) {
  constexpr int kPer = (N * (int)sizeof(T) <= 16) ? N : 16 / (int)sizeof(T);
#pragma unroll
  for (int c = 0; c < N / kPer; ++c) {
    typename AccOf<T>::type tmp[kPer];
    load_acc<T, kPer>(tmp, p + c * kPer);
#pragma unroll
    for (int i = 0; i < kPer; ++i) dst[c * kPer + i] = tmp[i];
  }
}
template <typename T, int N>
__device__ __forceinline__ void store_vec(T* __restrict__ p, const typename AccOf<T>::type (&src)[N]) {
  constexpr int kPer = (N * (int)sizeof(T) <= 16) ? N : 16 / (int)sizeof(T);
#pragma unroll
  for (int c = 0; c < N / kPer; ++c) {
    typename AccOf<T>::type tmp[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) tmp[i] = src[c * kPer + i];
    store_acc<T, kPer>(p + c * kPer, tmp);
  }
}

// The heads of one edge: columns h0 .. h0 + H - 1 of an (E, hs) tensor.  kVec: hs == H and H * sizeof(T) is a width of
// one or several aligned moves.
template <typename T, int H, bool kVec>
__device__ __forceinline__ void load_heads(typename AccOf<T>::type (&dst)[H], const T* __restrict__ p) {
  if constexpr (kVec) {
    load_vec<T, H>(dst, p);
  } else {
#pragma unroll
    for (int h = 0; h < H; ++h) dst[h] = to_acc<T>(__ldg(p + h));
  }
}
template <typename T, int H, bool kVec>
__device__ __forceinline__ void store_heads(T* __restrict__ p, const typename AccOf<T>::type (&src)[H]) {
  if constexpr (kVec) {
    store_vec<T, H>(p, src);
  } else {
#pragma unroll
    for (int h = 0; h < H; ++h) p[h] = from_acc<T>(src[h]);
  }
}

template <bool kMax, typename A> __device__ __forceinline__ A seg_op(A a, A b) {
  return kMax ? (b > a ? b : a) : a + b;
}
// What the exponents of a part of a row are relative to: its maximum, or 0 where all of the part is masked (scores of -inf,
// maximum -inf).  Such a part's sum is 0 and has no weight in the row's; -inf - -inf would make it, and with it the row, NaN.
template <typename A> __device__ __forceinline__ A exp_ref(A m) { return m == neg_inf<A>() ? A(0) : m; }
template <bool kMax, typename A> __device__ __forceinline__ A seg_identity() { return kMax ? neg_inf<A>() : A(0); }

// The edge ids of four consecutive positions from p, where keep has their bit (elsewhere, and where there are no ids, the
// positions), in one load where the table allows it: as four they are as many accesses to the L1 as two heads of values.  50M
// skewed edges, 2 heads fp32: forward 438 + 300 -> 414 + 284 us, backward 257 + 248 -> 252 + 208.
__device__ __forceinline__ void load_ids(int (&e)[kSoftmaxPer], const int32_t* __restrict__ eid, long long p, long long E,
                                         unsigned keep) {
  if (eid && ((uintptr_t)eid & 15) == 0 && p + kSoftmaxPer <= E) {
    const int4 v = __ldg(reinterpret_cast<const int4*>(eid + p));
    e[0] = v.x; e[1] = v.y; e[2] = v.z; e[3] = v.w;
    return;
  }
#pragma unroll
  for (int i = 0; i < kSoftmaxPer; ++i) e[i] = eid && p + i < E && ((keep >> i) & 1u) ? __ldg(eid + p + i) : (int)(p + i);
}

// Where the segments of a thread's positions begin.
struct Starts {
  unsigned f;        // bit i: position i starts a segment
  unsigned lanes;    // lanes of the warp with a start
  unsigned warps;    // warps of the block with a start
  int lane, w;
  __device__ __forceinline__ bool none_before() const {   // no start in earlier lanes of the warp
    return (lanes & ((1u << lane) - 1)) == 0;
  }
  __device__ __forceinline__ bool none_after() const { return lane == 31 || (lanes >> (lane + 1)) == 0; }
  __device__ __forceinline__ bool first_at(int i) const { return (f & ((2u << i) - 1)) == 0; }   // no start at or before i
  __device__ __forceinline__ bool last_at(int i) const { return (f >> (i + 1)) == 0; }           // none after i
  // position i lies in the tile's first / last segment
  __device__ __forceinline__ bool in_head(int i) const {
    return first_at(i) && none_before() && (warps & ((1u << w) - 1)) == 0;
  }
  __device__ __forceinline__ bool in_tail(int i) const { return last_at(i) && none_after() && (warps >> (w + 1)) == 0; }
};

// v[i] := fold of v over the part of position i's segment that lies in the tile.  s_head / s_tail: per warp the fold
// of its positions before its first start (all, if none) and since its last one.
template <typename A, int H, bool kMax>
__device__ __forceinline__ void segment_totals(A (&v)[kSoftmaxPer][H], const Starts& st, A (*s_head)[H], A (*s_tail)[H]) {
  constexpr int P = kSoftmaxPer;
  // inside the thread: running folds forward, then each segment's last one carried back
#pragma unroll
  for (int i = 1; i < P; ++i)
    if (!((st.f >> i) & 1))
#pragma unroll
      for (int h = 0; h < H; ++h) v[i][h] = seg_op<kMax>(v[i - 1][h], v[i][h]);
  A run[H];   // fold over the lanes up to this one, since the last start
#pragma unroll
  for (int h = 0; h < H; ++h) run[h] = v[P - 1][h];
#pragma unroll
  for (int i = P - 2; i >= 0; --i)
    if (!((st.f >> (i + 1)) & 1))
#pragma unroll
      for (int h = 0; h < H; ++h) v[i][h] = v[i + 1][h];
  const unsigned upto = st.lanes & (0xffffffffu >> (31 - st.lane));
  const int lo = upto ? 31 - __clz(upto) : 0;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const A t = __shfl_up_sync(kFull, run[h], d);
      if (st.lane - d >= lo) run[h] = seg_op<kMax>(t, run[h]);
    }
  // the fold of the segment that this thread's first positions continue (start: nothing before them)
  const unsigned beyond = st.lane == 31 ? 0u : st.lanes & ~(0xffffffffu >> (31 - st.lane));
  const int next = beyond ? __ffs(beyond) - 1 : 31;
  const bool head = (st.f & 1) == 0;
  A in[H], done[H];
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const A t = __shfl_up_sync(kFull, run[h], 1);
    in[h] = st.lane ? t : seg_identity<kMax, A>();
    // complete as far as the warp goes: what the first positions' segment comes to here
    done[h] = head ? seg_op<kMax>(in[h], v[0][h]) : in[h];
    const A at_next = __shfl_sync(kFull, st.f ? done[h] : run[h], next);
    const A at_end = __shfl_sync(kFull, run[h], 31);
    const A out = beyond ? at_next : at_end;   // what the last position's segment comes to, within the warp
#pragma unroll
    for (int i = 0; i < P; ++i) {
      if (st.last_at(i)) v[i][h] = out;
      else if (st.first_at(i)) v[i][h] = done[h];
    }
    if (st.lane == 31) s_tail[st.w][h] = run[h];
    if (st.lane == (st.lanes ? __ffs(st.lanes) - 1 : 31)) s_head[st.w][h] = st.lanes ? done[h] : run[h];
  }
  __syncthreads();
  A left[H], right[H];
#pragma unroll
  for (int h = 0; h < H; ++h) left[h] = right[h] = seg_identity<kMax, A>();
  for (int k = st.w - 1; k >= 0; --k) {
#pragma unroll
    for (int h = 0; h < H; ++h) left[h] = seg_op<kMax>(s_tail[k][h], left[h]);
    if ((st.warps >> k) & 1) break;
  }
  for (int k = st.w + 1; k < kSoftmaxWarps; ++k) {
#pragma unroll
    for (int h = 0; h < H; ++h) right[h] = seg_op<kMax>(right[h], s_head[k][h]);
    if ((st.warps >> k) & 1) break;
  }
  const bool nb = st.none_before(), na = st.none_after();
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const bool l = nb && st.first_at(i), r = na && st.last_at(i);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      if (l) v[i][h] = seg_op<kMax>(left[h], v[i][h]);
      if (r) v[i][h] = seg_op<kMax>(v[i][h], right[h]);
    }
  }
}

// Forward (kBackward = false):  y = exp(x - max) / sum exp(x - max) per (node, head).
//   in0 = x, in1 unused; slot = [H max][H sum]
// Backward (kBackward = true):  dx = y * (dy - sum_node dy * y).
//   in0 = y, in1 = dy;   slot = [H sum]
template <typename T, int H, bool kBackward, bool kVec>
__global__ void __launch_bounds__(kSoftmaxThreads)
softmax_tile_kernel(const int32_t* __restrict__ erow, const int32_t* __restrict__ eid, const T* __restrict__ in0,
                    const T* __restrict__ in1, T* __restrict__ out, typename AccOf<T>::type* __restrict__ slots,
                    int32_t* __restrict__ slot_rows, long long E, int hs, int h0) {
  using A = typename AccOf<T>::type;
  constexpr int P = kSoftmaxPer;
  constexpr int kSlot = kBackward ? H : 2 * H;
  __shared__ A s_head[2][kSoftmaxWarps][H], s_tail[2][kSoftmaxWarps][H];   // maxima and sums (backward: [0] alone)
  __shared__ unsigned s_warps;
  const int tid = threadIdx.x;
  const long long t = blockIdx.x, j0 = t * kSoftmaxTile, p = j0 + tid * P;
  if (tid == 0) s_warps = 0;
  __syncthreads();
  alignas(16) int r[P];
  int e[P];
  if (p + P <= E) {
    *reinterpret_cast<int4*>(r) = __ldg(reinterpret_cast<const int4*>(erow + p));
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) r[i] = p + i < E ? __ldg(erow + p + i) : -1;
  }
  load_ids(e, eid, p, E, ~0u);
  Starts st;
  st.lane = tid & 31;
  st.w = tid >> 5;
  int up = __shfl_up_sync(kFull, r[P - 1], 1);
  if (st.lane == 0) up = p > 0 && p <= E ? __ldg(erow + p - 1) : -1;
  const int next = j0 + kSoftmaxTile < E ? __ldg(erow + j0 + kSoftmaxTile) : -1;
  // four consecutive edges are one piece of memory (always so where the edge ids are the positions)
  bool run = kVec && e[1] == e[0] + 1 && e[2] == e[0] + 2 && e[3] == e[0] + 3 && r[0] >= 0 && r[1] >= 0 && r[2] >= 0 &&
             r[3] >= 0;
  if constexpr (kVec) {
    constexpr int kWide = P * H * (int)sizeof(T) < 16 ? P * H * (int)sizeof(T) : 16;
    run = run && ((uintptr_t)(in0 + (long long)e[0] * H) % kWide) == 0 && ((uintptr_t)(out + (long long)e[0] * H) % kWide) == 0 &&
          (!kBackward || ((uintptr_t)(in1 + (long long)e[0] * H) % kWide) == 0);
    run = __all_sync(kFull, run);
  }
  A a[P][H];                   // x / y
  A b[kBackward ? P : 1][H];   // dy
  if (run) {
    load_vec<T, P * H>(reinterpret_cast<A(&)[P * H]>(a), in0 + (long long)e[0] * H);
    if constexpr (kBackward) load_vec<T, P * H>(reinterpret_cast<A(&)[P * H]>(b), in1 + (long long)e[0] * H);
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      if (r[i] >= 0) {
        load_heads<T, H, kVec>(a[i], in0 + (long long)e[i] * hs + h0);
        if constexpr (kBackward) load_heads<T, H, kVec>(b[i], in1 + (long long)e[i] * hs + h0);
      } else {
#pragma unroll
        for (int h = 0; h < H; ++h) {
          a[i][h] = kBackward ? A(0) : neg_inf<A>();
          if constexpr (kBackward) b[i][h] = A(0);
        }
      }
    }
  }
  st.f = 0;
#pragma unroll
  for (int i = 0; i < P; ++i) st.f |= (unsigned)(r[i] != (i ? r[i - 1] : up)) << i;
  st.lanes = __ballot_sync(kFull, st.f != 0);
  if (st.lane == 0 && st.lanes) atomicOr(&s_warps, 1u << st.w);
  __syncthreads();
  st.warps = s_warps;

  if (st.warps == 0) {
    // The tile lies inside one node that began before it (most tiles of a skewed graph): two block reductions, no scans, and
    // nothing to write yet.
    const int row = r[0];
    if (row >= 0) {
      A m[H], l[H];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        m[h] = kBackward ? A(0) : neg_inf<A>();
#pragma unroll
        for (int i = 0; i < P; ++i) {
          if constexpr (kBackward) m[h] += a[i][h] * b[i][h];
          else m[h] = seg_op<true>(m[h], a[i][h]);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) m[h] = seg_op<!kBackward>(m[h], __shfl_xor_sync(kFull, m[h], o));
        if (st.lane == 0) s_head[0][st.w][h] = m[h];
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < H; ++h) {
        m[h] = s_head[0][0][h];
#pragma unroll
        for (int k = 1; k < kSoftmaxWarps; ++k) m[h] = seg_op<!kBackward>(m[h], s_head[0][k][h]);
      }
      if constexpr (!kBackward) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
          l[h] = A(0);
#pragma unroll
          for (int i = 0; i < P; ++i) l[h] += gk_exp(a[i][h] - exp_ref(m[h]));
          l[h] = warp_sum(l[h]);
          if (st.lane == 0) s_head[1][st.w][h] = l[h];
        }
        __syncthreads();
      }
      if (tid == 0)
#pragma unroll
        for (int h = 0; h < H; ++h) {
          slots[2 * t * kSlot + h] = m[h];
          if constexpr (!kBackward) {
#pragma unroll
            for (int k = 1; k < kSoftmaxWarps; ++k) l[h] += s_head[1][k][h];
            slots[2 * t * kSlot + H + h] = l[h];
          }
        }
    }
    if (tid == 0) {
      slot_rows[2 * t] = row;
      slot_rows[2 * t + 1] = -1;
    }
    return;
  }

  A m[P][H];    // maxima (backward: sums)
  A l[kBackward ? 1 : P][H];
  if constexpr (kBackward) {
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int h = 0; h < H; ++h) m[i][h] = a[i][h] * b[i][h];
    segment_totals<A, H, false>(m, st, s_head[0], s_tail[0]);
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int h = 0; h < H; ++h) m[i][h] = a[i][h];
    segment_totals<A, H, true>(m, st, s_head[0], s_tail[0]);
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int h = 0; h < H; ++h) l[i][h] = a[i][h] = r[i] >= 0 ? gk_exp(a[i][h] - exp_ref(m[i][h])) : A(0);
    segment_totals<A, H, false>(l, st, s_head[1], s_tail[1]);
  }

  // closed segments are final
  // whether the tile's first segment began before it; whether the last one goes on (a thread can tell for its own)
  const auto head_open = [&](int i) { return j0 > 0 && st.in_head(i); };
  A y[P][H];
  bool open[P], any_open = false;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    open[i] = head_open(i) || (st.in_tail(i) && r[i] == next);
    any_open = any_open || open[i];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      if constexpr (kBackward) y[i][h] = a[i][h] * (b[i][h] - m[i][h]);
      else y[i][h] = a[i][h] / l[i][h];
    }
  }
  if (run && !any_open) {
    store_vec<T, P * H>(out + (long long)e[0] * H, reinterpret_cast<A(&)[P * H]>(y));
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (r[i] >= 0 && !open[i]) store_heads<T, H, kVec>(out + (long long)e[i] * hs + h0, y[i]);
  }

  if (tid == 0) {
    const bool is = r[0] >= 0 && head_open(0);
    slot_rows[2 * t] = is ? r[0] : -1;
    if (is)
#pragma unroll
      for (int h = 0; h < H; ++h) {
        slots[2 * t * kSlot + h] = m[0][h];
        if constexpr (!kBackward) slots[2 * t * kSlot + H + h] = l[0][h];
      }
  }
  if (tid == kSoftmaxThreads - 1) {   // a segment that goes on holds the tile's last position
    const bool is = r[P - 1] >= 0 && r[P - 1] == next && !head_open(P - 1);
    slot_rows[2 * t + 1] = is ? r[P - 1] : -1;
    if (is)
#pragma unroll
      for (int h = 0; h < H; ++h) {
        slots[(2 * t + 1) * kSlot + h] = m[P - 1][h];
        if constexpr (!kBackward) slots[(2 * t + 1) * kSlot + H + h] = l[P - 1][h];
      }
  }
}

// How many tiles t+dir, t+2*dir, ... in a row have their first slot in use for `row` (whole warp).
__device__ __forceinline__ long long same_row_tiles(const int32_t* __restrict__ slot_rows, long long t, int dir, int row,
                                                    long long nt, int lane) {
  const auto same = [&](long long d) {
    const long long u = t + dir * d;
    return u >= 0 && u < nt && __ldg(slot_rows + 2 * u) == row;
  };
  const int c = __popc(__ballot_sync(kFull, lane < 31 && same(1LL << lane)));
  if (c == 0) return 0;
  long long lo = 1LL << (c - 1), hi = 1LL << c;   // same(lo), not same(hi)
  while (hi - lo > 1) {
    const long long span = hi - lo;
    const auto pivot = [&](int k) {
      const long long m = lo + span * (k + 1) / 33;
      return m <= lo ? lo + 1 : (m >= hi ? hi - 1 : m);
    };
    const int cnt = __popc(__ballot_sync(kFull, same(pivot(lane))));
    const long long below = cnt ? pivot(cnt - 1) : lo;
    hi = cnt < 32 ? pivot(cnt) : hi;
    lo = below;
  }
  return lo;
}

template <typename A, bool kBackward>
__device__ __forceinline__ void merge_stat(A& m, A& l, A m2, A l2) {
  if (kBackward) {
    m += m2;
  } else {
    const A mn = m2 > m ? m2 : m;
    const A wa = m == neg_inf<A>() ? A(0) : gk_exp(m - mn);
    const A wb = m2 == neg_inf<A>() ? A(0) : gk_exp(m2 - mn);
    l = l * wa + l2 * wb;
    m = mn;
  }
}

// Statistics of a node from its slots: the odd one of tile first - 1, the even ones of tiles first .. first + n - 1.
// `size` threads (a warp or the block) take the slots in turn; every lane of a warp ends with its warp's fold.
template <typename A, int H, bool kBackward>
__device__ __forceinline__ void fold_slots(A (&m)[H], A (&l)[H], const A* __restrict__ slots, long long first, long long n,
                                           int rank, int size) {
  constexpr int kSlot = kBackward ? H : 2 * H;
#pragma unroll
  for (int h = 0; h < H; ++h) {
    m[h] = kBackward ? A(0) : neg_inf<A>();
    l[h] = A(0);
  }
#pragma unroll 4
  for (long long q = rank; q <= n; q += size) {
    const A* s = slots + (q ? 2 * (first + q - 1) : 2 * first - 1) * kSlot;
#pragma unroll
    for (int h = 0; h < H; ++h) merge_stat<A, kBackward>(m[h], l[h], s[h], kBackward ? A(0) : s[H + h]);
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const A m2 = __shfl_xor_sync(kFull, m[h], o);
      const A l2 = kBackward ? A(0) : __shfl_xor_sync(kFull, l[h], o);
      merge_stat<A, kBackward>(m[h], l[h], m2, l2);
    }
}

// More tiles than this: softmax_merge_kernel merges every node's slots once; up to it each tile that has a part of the
// node merges them again for itself (at most as many reads a tile), which saves a launch.
constexpr long long kSoftmaxSelfMerge = 1024;
// Slots of a node that one warp merges; more are spread over the block.
constexpr long long kSoftmaxWarpSlots = 256;

// merged[slot] := the statistics of the node, for every slot in use.  A warp per tile: it acts for the node whose
// positions start in the tile and go on.
template <typename A, int H, bool kBackward>
__global__ void __launch_bounds__(kSoftmaxThreads)
softmax_merge_kernel(const A* __restrict__ slots, const int32_t* __restrict__ slot_rows, A* __restrict__ merged,
                     long long nt) {
  constexpr int kSlot = kBackward ? H : 2 * H;
  __shared__ long long s_count[kSoftmaxWarps];
  __shared__ A s_m[kSoftmaxWarps][H], s_l[kSoftmaxWarps][H];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const long long t = (long long)blockIdx.x * kSoftmaxWarps + w;
  const int row = t < nt ? __ldg(slot_rows + 2 * t + 1) : -1;
  const long long n = row >= 0 ? same_row_tiles(slot_rows, t, 1, row, nt, lane) : 0;
  const auto write = [&](const A (&m)[H], const A (&l)[H], long long first, long long count, int rank, int size) {
    for (long long q = rank; q <= count; q += size) {
      A* s = merged + (q ? 2 * (first + q - 1) : 2 * first - 1) * kSlot;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        s[h] = m[h];
        if (!kBackward) s[H + h] = l[h];
      }
    }
  };
  if (lane == 0) s_count[w] = n;
  A m[H], l[H];
  if (row >= 0 && n <= kSoftmaxWarpSlots) {
    fold_slots<A, H, kBackward>(m, l, slots, t + 1, n, lane, 32);
    write(m, l, t + 1, n, lane, 32);
  }
  __syncthreads();
  for (int k = 0; k < kSoftmaxWarps; ++k) {
    const long long count = s_count[k], first = (long long)blockIdx.x * kSoftmaxWarps + k + 1;
    if (count <= kSoftmaxWarpSlots) continue;
    fold_slots<A, H, kBackward>(m, l, slots, first, count, tid, kSoftmaxThreads);
    if (lane == 0)
#pragma unroll
      for (int h = 0; h < H; ++h) { s_m[w][h] = m[h]; s_l[w][h] = l[h]; }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < H; ++h) { m[h] = s_m[0][h]; l[h] = s_l[0][h]; }
    for (int v = 1; v < kSoftmaxWarps; ++v)
#pragma unroll
      for (int h = 0; h < H; ++h) merge_stat<A, kBackward>(m[h], l[h], s_m[v][h], s_l[v][h]);
    write(m, l, first, count, tid, kSoftmaxThreads);
    __syncthreads();
  }
}

// Revisits the positions of the tile's open segments with their node's statistics: from `merged`, or (null) merged here,
// the first segment's by warp 0 and the last one's by warp 1.
template <typename T, int H, bool kBackward, bool kVec>
__global__ void __launch_bounds__(kSoftmaxThreads)
softmax_finish_kernel(const int32_t* __restrict__ erow, const int32_t* __restrict__ eid, const T* __restrict__ in0,
                      const T* __restrict__ in1, T* __restrict__ out,
                      const typename AccOf<T>::type* __restrict__ slots, const int32_t* __restrict__ slot_rows,
                      const typename AccOf<T>::type* __restrict__ merged, long long E, long long nt, int hs, int h0) {
  using A = typename AccOf<T>::type;
  constexpr int kSlot = kBackward ? H : 2 * H;
  __shared__ A s_stat[2][kSlot];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const long long t = blockIdx.x;
  const int head_row = __ldg(slot_rows + 2 * t), tail_row = __ldg(slot_rows + 2 * t + 1);
  if (head_row < 0 && tail_row < 0) return;
  const int mine = w == 0 ? head_row : tail_row;
  if (w < 2 && mine >= 0) {
    if (merged) {
      if (lane < kSlot) s_stat[w][lane] = __ldg(merged + (2 * t + w) * kSlot + lane);
    } else {
      const long long back = w == 0 ? same_row_tiles(slot_rows, t, -1, mine, nt, lane) : 0;
      const long long ahead = same_row_tiles(slot_rows, t, 1, mine, nt, lane);
      A m[H], l[H];
      // w == 0: tiles t - back .. t + ahead hold even slots; w == 1: tiles t + 1 .. t + ahead
      fold_slots<A, H, kBackward>(m, l, slots, w == 0 ? t - back : t + 1, w == 0 ? back + 1 + ahead : ahead, lane, 32);
      if (lane == 0)
#pragma unroll
        for (int h = 0; h < H; ++h) {
          s_stat[w][h] = m[h];
          if (!kBackward) s_stat[w][H + h] = l[h];
        }
    }
  }
  __syncthreads();
  constexpr int P = kSoftmaxPer;
  const long long p = t * kSoftmaxTile + tid * P;
  alignas(16) int r[P];
  int e[P];
  if (p + P <= E) {
    *reinterpret_cast<int4*>(r) = __ldg(reinterpret_cast<const int4*>(erow + p));
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) r[i] = p + i < E ? __ldg(erow + p + i) : -1;
  }
  bool todo[P], all = true, any = false;
  unsigned keep = 0;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    todo[i] = r[i] >= 0 && (r[i] == head_row || r[i] == tail_row);
    all = all && todo[i];
    any = any || todo[i];
    keep |= (unsigned)todo[i] << i;
  }
  if (!any) return;
  load_ids(e, eid, p, E, keep);
  // four consecutive edges are one piece of memory (the tile kernel's case)
  bool run = kVec && all && e[1] == e[0] + 1 && e[2] == e[0] + 2 && e[3] == e[0] + 3;
  if constexpr (kVec) {
    constexpr int kWide = P * H * (int)sizeof(T) < 16 ? P * H * (int)sizeof(T) : 16;
    run = run && ((uintptr_t)(in0 + (long long)e[0] * H) % kWide) == 0 && ((uintptr_t)(out + (long long)e[0] * H) % kWide) == 0 &&
          (!kBackward || ((uintptr_t)(in1 + (long long)e[0] * H) % kWide) == 0);
  }
  A a[P][H];
  A b[kBackward ? P : 1][H];
  if (run) {
    load_vec<T, P * H>(reinterpret_cast<A(&)[P * H]>(a), in0 + (long long)e[0] * H);
    if constexpr (kBackward) load_vec<T, P * H>(reinterpret_cast<A(&)[P * H]>(b), in1 + (long long)e[0] * H);
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (todo[i]) {
        load_heads<T, H, kVec>(a[i], in0 + (long long)e[i] * hs + h0);
        if constexpr (kBackward) load_heads<T, H, kVec>(b[i], in1 + (long long)e[i] * hs + h0);
      }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (!todo[i]) continue;
    const A* st = s_stat[r[i] == head_row ? 0 : 1];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      if constexpr (kBackward) a[i][h] = a[i][h] * (b[i][h] - st[h]);
      else a[i][h] = gk_exp(a[i][h] - st[h]) / st[H + h];
    }
  }
  if (run) {
    store_vec<T, P * H>(out + (long long)e[0] * H, reinterpret_cast<A(&)[P * H]>(a));
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (todo[i]) store_heads<T, H, kVec>(out + (long long)e[i] * hs + h0, a[i]);
  }
}

}  // namespace gk
