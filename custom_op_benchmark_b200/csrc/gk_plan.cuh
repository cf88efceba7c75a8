// Graph plans: what the ops need from the graph alone, built once per graph in caller-provided memory
// (include/graphop_b200.h, "Graph plans").  The reference prepares its graphs on the host in Python loops
// (part_csr.py:18-21, wrapper.py:93-112); here the expansion of the chunk table, the 32-bit index copies, the
// per-node ranges and the shape analysis are kernels.
#pragma once
#include <climits>

#include "gk_host.cuh"

namespace gk {

struct BandVerdict {
  int not_contiguous;  // some node's neighbours are not one run of consecutive ids
  int max_span;        // most different neighbours any 128 consecutive nodes reach
  int row_crosses;     // some node's positions cross a row-aligned tile boundary
  int unused;
};
// what a plan finds out on the device, in one piece for one copy back
struct PlanFacts {
  PlanHeader cover;
  BandVerdict verdict;
};

constexpr int kBandTileRows = 128;

// first position and number of positions of every node, from the chunk table (integer atomics: the result does
// not depend on their order)
template <typename I>
__device__ __forceinline__ void node_ranges(const I* __restrict__ row, const I* __restrict__ indptr, long long C,
                                            long long n_nodes, int32_t* __restrict__ first, int32_t* __restrict__ deg, unsigned block,
                                            unsigned blocks) {
  const long long stride = (long long)blocks * blockDim.x;
  for (long long c = (long long)block * blockDim.x + threadIdx.x; c < C; c += stride) {
    const long long r = (long long)row[c];
    const long long s = (long long)indptr[c], e = (long long)indptr[c + 1];
    if (r < 0 || r >= n_nodes || e <= s) continue;
    atomicMin(first + r, (int)s);
    atomicAdd(deg + r, (int)(e - s));
  }
}

// every covered position must hold (first neighbour of its node) + (its offset inside the node).  On most graphs the first
// positions already say no: blocks stay few enough to go round several times and stop at the first round after the verdict.
__device__ __forceinline__ void band_positions(const int32_t* __restrict__ erow, const int32_t* __restrict__ other,
                                               long long E, const int32_t* __restrict__ first,
                                               BandVerdict* __restrict__ verdict, unsigned block, unsigned blocks) {
  const long long stride = (long long)blocks * blockDim.x;
  int bad = 0;
  for (long long j = (long long)block * blockDim.x + threadIdx.x; j < E; j += stride) {
    if (bad || *(volatile const int*)&verdict->not_contiguous) break;
    const int r = erow[j];
    if (r < 0) continue;
    const int f = first[r];
    if (other[j] != other[f] + (j - f)) bad = 1;   // in 64 bits: on any other graph the sum may pass 2^31
  }
  // one atomic per block, none once the verdict is known (one per thread serialised: 14 us on 0.6M edges)
  if (__syncthreads_or(bad) && threadIdx.x == 0 && !*(volatile const int*)&verdict->not_contiguous)
    atomicOr(&verdict->not_contiguous, 1);
}

// first neighbour per node, and the widest range of neighbours any tile of 128 consecutive nodes reaches
__device__ __forceinline__ void band_tiles(const int32_t* __restrict__ other, const int32_t* __restrict__ first,
                                           const int32_t* __restrict__ deg, long long n_nodes,
                                           int32_t* __restrict__ node_lo, BandVerdict* __restrict__ verdict,
                                           unsigned block) {
  __shared__ int s_lo[kBandTileRows / 32], s_hi[kBandTileRows / 32];
  const long long r = (long long)block * kBandTileRows + threadIdx.x;
  int lo = INT_MAX, hi = INT_MIN;
  if (r < n_nodes) {
    const int d = deg[r];
    const int l = d > 0 ? other[first[r]] : 0;
    node_lo[r] = l;
    // (the end of a run of d neighbours from l; where they are no run the graph is no band, and the clamp says nothing)
    if (d > 0) { lo = l; hi = (int)min((long long)l + d - 1, (long long)INT_MAX - 1); }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(kFull, lo, o));
    hi = max(hi, __shfl_xor_sync(kFull, hi, o));
  }
  if ((threadIdx.x & 31) == 0) { s_lo[threadIdx.x >> 5] = lo; s_hi[threadIdx.x >> 5] = hi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kBandTileRows / 32; ++w) { lo = min(lo, s_lo[w]); hi = max(hi, s_hi[w]); }
    const int span = hi >= lo ? hi - lo + 1 : 0;
    if (span > *(volatile const int*)&verdict->max_span) atomicMax(&verdict->max_span, span);
  }
}

// The boundaries of the work tiles (cut_tiles) moved up to row starts: a boundary inside a node goes to the first position
// within the next `tile` ones at which another node starts.  A boundary that finds none cuts a node in two: reported.
__device__ __forceinline__ void align_tiles(const int32_t* __restrict__ erow, long long E, int tile, long long n_tiles,
                                            int32_t* __restrict__ tile_start, BandVerdict* __restrict__ verdict,
                                            unsigned block, unsigned blocks) {
  const long long stride = (long long)blocks * blockDim.x;
  int crosses = 0;
  for (long long t = (long long)block * blockDim.x + threadIdx.x; t <= n_tiles; t += stride) {
    long long b = tile_start[t];
    if (b > 0 && b < E) {
      const long long limit = b + tile < E ? b + tile : E;
      int prev = erow[b - 1];
      long long q = b;
      for (; q < limit; ++q) {
        const int r = erow[q];
        if (r != prev) break;
        prev = r;
      }
      if (q < limit) b = q;
      else if (prev >= 0) crosses = 1;
    }
    tile_start[t] = (int32_t)b;
  }
  if (crosses) atomicOr(&verdict->row_crosses, 1);
}

// What follows the expansion: the first block looks for rows gathered repeatedly, the next `aligning` ones move the tile
// boundaries, the others find the nodes' ranges.  The first one's table lies in device memory: as shared memory every block has
// its 8 KB, which the L1 lacks (R-MAT 21: 147 us, where the kernel without the question takes 123; as it is 135 and 132).
template <typename I>
__global__ void __launch_bounds__(256)
plan_nodes_kernel(const I* __restrict__ row, const I* __restrict__ indptr, long long C, long long n_nodes,
                  int32_t* __restrict__ first, int32_t* __restrict__ deg, const int32_t* __restrict__ erow, long long E, int tile,
                  long long n_tiles, int32_t* __restrict__ tile_start, BandVerdict* __restrict__ verdict, unsigned aligning,
                  const int32_t* __restrict__ other, unsigned* __restrict__ seen, PlanHeader* __restrict__ hdr) {
  if (blockIdx.x == 0) {
    const int repeats = other ? gather_repeats<256>(other, E, seen) : 0;
    if (threadIdx.x == 0) hdr->repeats = repeats;
    return;
  }
  const unsigned block = blockIdx.x - 1;
  if (block < aligning) align_tiles(erow, E, tile, n_tiles, tile_start, verdict, block, aligning);
  else node_ranges<I>(row, indptr, C, n_nodes, first, deg, block - aligning, gridDim.x - 1 - aligning);
}
// The shape analysis, on the nodes' ranges: a block per 128 nodes, the others go over the positions.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
plan_shape_kernel(const int32_t* __restrict__ erow, const int32_t* __restrict__ other, long long E,
                  const int32_t* __restrict__ first, const int32_t* __restrict__ deg, long long n_nodes,
                  int32_t* __restrict__ node_lo, BandVerdict* __restrict__ verdict, unsigned tiles) {
  if (blockIdx.x < tiles) band_tiles(other, first, deg, n_nodes, node_lo, verdict, blockIdx.x);
  else band_positions(erow, other, E, first, verdict, blockIdx.x - tiles, gridDim.x - tiles);
}

inline size_t plan_bytes(long long C, long long E, long long n_nodes, int index_bytes) {
  (void)C;
  size_t b = align_up((size_t)E * 4) + align_up(sizeof(PlanFacts));
  b += align_up((size_t)(tile_count(E, n_nodes, tile_cost(E, n_nodes)) + 1) * 4);   // tile boundaries
  if (index_bytes == 8) b += 2 * align_up((size_t)E * 4);
  b += 3 * align_up((size_t)(n_nodes > 0 ? n_nodes : 1) * 4) + align_up(kSkewBits / 8);
  return b + kAlign;
}

template <typename I>
inline int plan_build(const I* row, const I* indptr, const I* eid, const I* indices, long long C, long long E,
                      long long n_nodes, void* memory, size_t bytes, graphop_plan_t* plan, cudaStream_t st) {
  if (!plan) return GRAPHOP_ERR_INVALID_ARGUMENT;
  *plan = graphop_plan_t{};
  if (C < 0 || E < 0 || n_nodes < 0 || E >= (1LL << 31) || n_nodes >= (1LL << 31)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  if (!indptr || (C > 0 && !row)) return GRAPHOP_ERR_INVALID_ARGUMENT;
  GK_TRY(check_ws(memory));
  Arena ar(memory, bytes);
  auto* facts = (PlanFacts*)ar.take(sizeof(PlanFacts));
  BandVerdict* verdict = &facts->verdict;
  GraphView g{};
  int32_t* first = (int32_t*)ar.take((size_t)(n_nodes > 0 ? n_nodes : 1) * 4);
  int32_t* deg = (int32_t*)ar.take((size_t)(n_nodes > 0 ? n_nodes : 1) * 4);
  int32_t* node_lo = (int32_t*)ar.take((size_t)(n_nodes > 0 ? n_nodes : 1) * 4);
  unsigned* seen = (unsigned*)ar.take(kSkewBits / 8);
  if (ar.overflow) return GRAPHOP_ERR_WORKSPACE;
  plan->n_chunks = C;
  plan->n_edges = E;
  plan->n_nodes = n_nodes;
  if (E == 0) {  // nothing to expand: the ops return before they look at a plan's arrays
    GK_CUDA(cudaMemsetAsync(deg, 0, (size_t)(n_nodes > 0 ? n_nodes : 1) * 4, st));
    plan->node_deg = deg;
    plan->node_lo = node_lo;
    return GRAPHOP_OK;
  }
  const Fill fill{{(int32_t*)verdict, deg, first},
                  {(long long)(sizeof(BandVerdict) / 4), n_nodes, n_nodes},
                  {0, 0, INT_MAX}};
  GK_TRY(prepare_graph<I>(ar, row, indptr, eid, indices, C, E, n_nodes, st, &g, Clear{}, &facts->cover, fill));
  plan->header = g.hdr;
  plan->erow = g.erow;
  plan->other = g.other;
  plan->eid = g.eid;
  plan->node_lo = node_lo;
  plan->node_deg = deg;
  {
    const unsigned aligning = (unsigned)((g.n_tiles + 256) / 256 < 4096 ? (g.n_tiles + 256) / 256 : 4096);
    const unsigned ranging = n_nodes > 0 && C > 0 ? (unsigned)((C + 255) / 256 < 8192 ? (C + 255) / 256 : 8192) : 0;
    plan_nodes_kernel<I><<<1 + aligning + ranging, 256, 0, st>>>(row, indptr, C, n_nodes, first, deg, g.erow, E, g.tile, g.n_tiles,
                                                             const_cast<int32_t*>(g.tile_start), verdict, aligning, g.other,
                                                             seen, &facts->cover);
    GK_LAUNCHED("plan_nodes");
  }
  if (g.other && n_nodes > 0) {
    const unsigned tiles = (unsigned)((n_nodes + kBandTileRows - 1) / kBandTileRows);
    const long long rounds = (E + kBandTileRows - 1) / kBandTileRows;
    plan_shape_kernel<kBandTileRows><<<tiles + (unsigned)(rounds < 592 ? rounds : 592), kBandTileRows, 0, st>>>(
        g.erow, g.other, E, first, deg, n_nodes, node_lo, verdict, tiles);
    GK_LAUNCHED("plan_shape");
  }
  const bool analysed = g.other && n_nodes > 0;
  PlanFacts back{};
  GK_CUDA(cudaMemcpyAsync(&back, facts, sizeof(back), cudaMemcpyDeviceToHost, st));
  GK_CUDA(cudaStreamSynchronize(st));
  const BandVerdict& host = back.verdict;
  plan->band_span = analysed ? host.max_span : 0;
  if (analysed && !host.not_contiguous && host.max_span > 0 && host.max_span <= GRAPHOP_BAND_MAX_SPAN)
    plan->flags |= GRAPHOP_PLAN_DENSE_BAND;
  plan->tile = g.tile;
  plan->tile_start = g.tile_start;
  plan->flags |= GRAPHOP_PLAN_ROW_TILES;
  if (!host.row_crosses) plan->flags |= GRAPHOP_PLAN_NO_CARRY;
  plan->gather_repeats = back.cover.repeats;
  if (back.cover.repeats > skew_allowed(LLONG_MAX, E)) plan->flags |= GRAPHOP_PLAN_SKEWED;
  if (back.cover.cover_hi - back.cover.cover_lo >= E) plan->flags |= GRAPHOP_PLAN_COVERED;
  return GRAPHOP_OK;
}

}  // namespace gk
