// Fused attention, forward and backward, for dense-band graphs on the sm_100a tensor cores.
//
// The reference expresses batched dense attention as a graph (512 fully connected blocks, wrapper.py:79-112) and
// runs it through the same one-thread-per-edge kernels as any other graph (graphop_kernel.cu:40-55, 170-202,
// 118-130).  When a plan says that every node's neighbours are one run of consecutive ids (GRAPHOP_PLAN_DENSE_BAND:
// sliding-window attention, block-diagonal attention), the edge list carries no information beyond a (first, count)
// pair per node, and the chain
//     scores = Q K^T on the band,  P = softmax(scale * scores),  O = P V
// is two small dense matrix products per tile of 128 query nodes and head:
//   * TMA (cp.async.bulk.tensor, 128-byte swizzle, no multicast) brings the tile's 128 q rows and, block by block of 64,
//     the k and v rows its band reaches into shared memory;
//   * tcgen05.mma (kind::f16, bf16 in, fp32 out) forms the block's 128 x 64 scores in tensor memory;
//   * two threads share a query row: each reads 32 of the block's columns from tensor memory (tcgen05.ld), masks those
//     outside its node's range and writes the probabilities, relative to a running maximum, as bf16 into shared memory;
//   * a second tcgen05.mma adds their product with v to the tile's output in tensor memory, which is rescaled where a
//     row's maximum has grown by more than 2^8; at the end each thread scales 32 of the row's 64 outputs by 1 / sum.
// Several tiles share an SM, so that one's loads and products run under the others' element-wise stages.
// Every wait on an mbarrier is bounded; a tile whose wait runs out writes NaN to its rows of O instead of hanging.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <limits.h>

#include <type_traits>

#include "gk_host.cuh"

namespace gk {
namespace banded {

constexpr int kTileM = 128;                 // nodes per block = tensor-memory lanes
constexpr int kThreads = 256;               // two threads per node row: warp w works on lanes 32 (w % 4) .. + 31 and
constexpr int kColGroups = kThreads / kTileM;   // columns 32 (w / 4) .. + 31 of a block
constexpr int kD = 64;                      // features per head: one 128-byte swizzle row of bf16
constexpr int kSpan = GRAPHOP_BAND_MAX_SPAN;  // key rows a tile reaches at most
constexpr int kRowBytes = kD * 2;           // 128
constexpr int kKeys = 64;                   // rows of the band per block
constexpr int kBandBytes = kKeys * kRowBytes;               // 8 KB
constexpr int kSlots = 2;                   // blocks of the band in shared memory
constexpr int kBlockBytes = kTileM * kRowBytes;             // 16 KB: a tile's 128 rows, or a 128 x 64 staging tile
constexpr int kOffQ = 0;
constexpr int kOffK = kOffQ + kBlockBytes;                  // per slot: k, v
constexpr int kOffP = kOffK + kSlots * 2 * kBandBytes;
constexpr int kOffBar = kOffP + kBlockBytes;
constexpr int kOffRed = kOffBar + 128;                      // maxima (and at the end sums) of the two column groups
constexpr int kSmemBytes = kOffRed + kColGroups * kTileM * 4 + 1024;   // + alignment slack: 66 KB, three tiles per SM
constexpr int kTmemCols = 128;              // scores, output
constexpr int kColO = kKeys;
constexpr unsigned kWaitLimit = 400000u;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// bounded: false when the phase did not complete within kWaitLimit polls
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (unsigned it = 0; it < kWaitLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Shared-memory matrix descriptor, 128-byte swizzle: start address, leading / stride byte offsets in 16-byte units,
// descriptor version 1 (sm_100), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, A K-major, B K-major or MN-major, M x N.
__host__ __device__ constexpr uint32_t umma_idesc(int m, int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 consecutive fp32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Two 32-column loads (two regions of the same lane) in flight together, one wait for both.  The wait names every
// destination register as an operand, so that no use of the values can be scheduled ahead of it.
__device__ __forceinline__ void tmem_ld32_pair(uint32_t taddr_a, uint32_t taddr_b, float (&a)[32], float (&b)[32]) {
  uint32_t r[32], q[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr_a));
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]),
        "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15]), "=r"(q[16]),
        "=r"(q[17]), "=r"(q[18]), "=r"(q[19]), "=r"(q[20]), "=r"(q[21]), "=r"(q[22]), "=r"(q[23]), "=r"(q[24]),
        "=r"(q[25]), "=r"(q[26]), "=r"(q[27]), "=r"(q[28]), "=r"(q[29]), "=r"(q[30]), "=r"(q[31])
      : "r"(taddr_b));
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
        "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
        "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
        "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]), "+r"(q[0]),
        "+r"(q[1]), "+r"(q[2]), "+r"(q[3]), "+r"(q[4]), "+r"(q[5]), "+r"(q[6]), "+r"(q[7]), "+r"(q[8]), "+r"(q[9]),
        "+r"(q[10]), "+r"(q[11]), "+r"(q[12]), "+r"(q[13]), "+r"(q[14]), "+r"(q[15]), "+r"(q[16]), "+r"(q[17]),
        "+r"(q[18]), "+r"(q[19]), "+r"(q[20]), "+r"(q[21]), "+r"(q[22]), "+r"(q[23]), "+r"(q[24]), "+r"(q[25]),
        "+r"(q[26]), "+r"(q[27]), "+r"(q[28]), "+r"(q[29]), "+r"(q[30]), "+r"(q[31])
      :
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) { a[i] = __uint_as_float(r[i]); b[i] = __uint_as_float(q[i]); }
}

// 16 consecutive fp32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  uint32_t r[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(v[i]);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h2);
}
// 16 fp32 values -> bf16 -> 32 bytes of global memory (NaN when the tile's waits ran out)
__device__ __forceinline__ void store_out16(__nv_bfloat16* dst, const float (&v)[16], float mul, bool ok) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = pack_bf16(ok ? v[8 * q + 2 * e] * mul : NAN, ok ? v[8 * q + 2 * e + 1] * mul : NAN);
    *reinterpret_cast<uint4*>(dst + q * 8) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// 2^x for x <= 0 (a score minus its row maximum, or minus the row's log-sum): one MUFU instruction; results below
// the normal range flush to zero
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct Params {
  __nv_bfloat16* o;          // (n_dst, H, 64)
  float* lse;                // (n_dst, H)
  const int32_t* node_lo;    // first neighbour of every destination node
  const int32_t* node_deg;   // neighbours of every destination node
  long long n_dst;
  int H;
  float scale;
};

// 32 columns of one 128 x 64 staging tile row: 4 chunks of 16 bytes at chunk c * 4 + q
__device__ __forceinline__ void store_stage_row(unsigned char* row_at, int c, int row, const uint32_t (&packed)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int chunk = (c * 4 + q) ^ (row & 7);
    *reinterpret_cast<uint4*>(row_at + chunk * 16) =
        make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
  }
}
// One block per (tile of 128 nodes, head).  Bound by the chain load - scores - softmax - output of a block of the band; three
// tiles per SM overlap theirs.  With one tile of 512 threads per SM and the whole band in shared memory, four sequences of
// 8192, 8 heads, window 128, took 121 us instead of 86.
__global__ void __launch_bounds__(kThreads, 3)
attention_forward_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const Params p) {
  extern __shared__ unsigned char raw_smem[];
  // the swizzled tiles want a 1024-byte aligned base
  unsigned char* smem = raw_smem + ((1024u - (smem_u32(raw_smem) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  // bar_load: the tile's q; bar_s: scores (and the output before them); bar_full + 8 (b % 2): the band's block b
  const uint32_t bar_load = s_base + kOffBar, bar_s = bar_load + 8, bar_full = bar_load + 64;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffBar + 32);
  int* s_red = reinterpret_cast<int*>(smem + kOffBar + 40);   // 4 ints: per-quarter minima of the first neighbour
  int* s_top = reinterpret_cast<int*>(smem + kOffBar + 96);   // 4 ints: and maxima of the last one
  float* s_row = reinterpret_cast<float*>(smem + kOffRed);    // [column group][row]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, cg = warp >> 2;
  const int row = quarter * 32 + lane;                        // row of the tile = tensor-memory lane
  const int head = blockIdx.y;
  const long long r0 = (long long)blockIdx.x * kTileM, r = r0 + row;
  int lo = INT_MAX, deg = 0;
  if (r < p.n_dst) {
    deg = p.node_deg[r];
    if (deg > 0) lo = p.node_lo[r];
  }
  int wmin = lo, wtop = deg > 0 ? lo + deg - 1 : -1;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    wmin = min(wmin, __shfl_xor_sync(kFull, wmin, o));
    wtop = max(wtop, __shfl_xor_sync(kFull, wtop, o));
  }
  if (lane == 0 && cg == 0) { s_red[quarter] = wmin; s_top[quarter] = wtop; }
  if (tid == 0) {
    mbar_init(bar_load, 1);
    mbar_init(bar_s, 1);
#pragma unroll
    for (int b = 0; b < kSlots; ++b) mbar_init(bar_full + 8 * b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const int kmin = min(min(s_red[0], s_red[1]), min(s_red[2], s_red[3]));

  if (kmin != INT_MAX) {
    const int ktop = max(max(s_top[0], s_top[1]), max(s_top[2], s_top[3]));
    int nb = (ktop - kmin) / kKeys + 1;   // blocks the tile's band reaches
    nb = nb < kSpan / kKeys ? nb : kSpan / kKeys;
    auto issue_band = [&](int b) {   // one thread
      const uint32_t bar = bar_full + 8 * (b & 1), at = s_base + kOffK + (b & 1) * 2 * kBandBytes;
      mbar_expect_tx(bar, (uint32_t)(2 * kBandBytes));
      tma_load_3d(at, &map_k, bar, 0, head, kmin + b * kKeys);
      tma_load_3d(at + kBandBytes, &map_v, bar, 0, head, kmin + b * kKeys);
    };
    auto issue_scores = [&](int b) {   // one thread: 4 steps of 16 features
      constexpr uint32_t idesc = umma_idesc(kTileM, kKeys, false);
      const uint32_t at = s_base + kOffK + (b & 1) * 2 * kBandBytes;
#pragma unroll
      for (int kk = 0; kk < kD / 16; ++kk)
        umma_f16(tmem, umma_desc(s_base + kOffQ + kk * 32, 16, 1024), umma_desc(at + kk * 32, 16, 1024), idesc, kk > 0);
    };
    if (tid == 0) {
      mbar_expect_tx(bar_load, (uint32_t)kBlockBytes);
      tma_load_3d(s_base + kOffQ, &map_q, bar_load, 0, head, (int)r0);
      tma_load_3d(s_base + kOffQ + kBandBytes, &map_q, bar_load, 0, head, (int)r0 + kKeys);
      issue_band(0);
      if (nb > 1) issue_band(1);
    }
    int issued = nb < kSlots ? nb : kSlots;
    bool ok = __syncthreads_and(mbar_wait(bar_load, 0) && mbar_wait(bar_full, 0));

    const int jlo = deg > 0 ? lo - kmin : 1, jhi = deg > 0 ? lo - kmin + deg - 1 : 0;   // this row's columns of the band
    int wlo = deg > 0 ? jlo : INT_MAX, whi = deg > 0 ? jhi : -1;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      wlo = min(wlo, __shfl_xor_sync(kFull, wlo, o));
      whi = max(whi, __shfl_xor_sync(kFull, whi, o));
    }
    const uint32_t row_taddr = tmem + ((uint32_t)(quarter * 32) << 16);
    const float sl2 = p.scale * 1.4426950408889634f;
    unsigned char* prow = smem + kOffP + row * kRowBytes;
    float m = -INFINITY, l = 0.f;   // the row's reference maximum, in both of its threads; this thread's part of the sum

    if (ok && tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      issue_scores(0);
      umma_commit(bar_s);
    }
    // Per block one wait: block b's output product and block b + 1's scores are issued back to back behind one commit, so
    // when the scores are there the staging tile is free and the output is complete as well.
    for (int b = 0; b < nb; ++b) {
      ok = __syncthreads_and(ok && mbar_wait(bar_s, b & 1));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (ok && b > 0 && b + 1 < nb) {   // block b - 1's slot is free
        if (tid == 0) issue_band(b + 1);
        issued = b + 2;
      }
      const int col0 = b * kKeys + cg * 32;
      const bool live = ok && col0 <= whi && col0 + 31 >= wlo;   // warp-uniform
      const bool whole = col0 >= jlo && col0 + 31 <= jhi;        // the whole chunk belongs to the row: no column tests
      float v[32], top = -INFINITY;
      if (live) {
        tmem_ld32(row_taddr + cg * 32, v);
        if (whole) {
#pragma unroll
          for (int j = 0; j < 32; ++j) top = fmaxf(top, v[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (col0 + j >= jlo && col0 + j <= jhi) top = fmaxf(top, v[j]);
        }
      }
      s_row[cg * kTileM + row] = top;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");   // the two warps of these rows
      top = fmaxf(top, s_row[(cg ^ 1) * kTileM + row]);
      // A reference that lags behind the maximum by up to 2^8 serves as well: the rounding is relative.
      const bool grows = top * sl2 > m * sl2 + 8.f || (m == -INFINITY && top > -INFINITY);
      const float corr = !grows ? 1.f : m == -INFINITY ? 0.f : exp2_fast((m - top) * sl2);
      if (grows) {
        m = top;
        l *= corr;
      }
      if (b > 0 && __any_sync(kFull, grows)) {
        float o[32];
        tmem_ld32(row_taddr + kColO + cg * 32, o);
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] *= corr;
        tmem_st32(row_taddr + kColO + cg * 32, o);
      }
      const float msl2 = m == -INFINITY ? 0.f : m * sl2;
      uint32_t packed[16];
      if (live && whole) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float p0 = exp2_fast(fmaf(v[j], sl2, -msl2)), p1 = exp2_fast(fmaf(v[j + 1], sl2, -msl2));
          l += p0 + p1;
          packed[j / 2] = pack_bf16(p0, p1);
        }
      } else if (live) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const int col = col0 + j;
          float p0 = 0.f, p1 = 0.f;
          if (col >= jlo && col <= jhi) p0 = exp2_fast(fmaf(v[j], sl2, -msl2));
          if (col + 1 >= jlo && col + 1 <= jhi) p1 = exp2_fast(fmaf(v[j + 1], sl2, -msl2));
          l += p0 + p1;
          packed[j / 2] = pack_bf16(p0, p1);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) packed[j] = 0u;
      }
      store_stage_row(prow, cg, row, packed);
      // the probabilities were written through the generic proxy; the tensor core reads through the async proxy
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      ok = __syncthreads_and(ok && (b + 1 >= nb || mbar_wait(bar_full + 8 * ((b + 1) & 1), ((b + 1) >> 1) & 1)));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (ok && tid == 0) {
        constexpr uint32_t idesc = umma_idesc(kTileM, kD, true);
        const uint32_t at = s_base + kOffK + (b & 1) * 2 * kBandBytes + kBandBytes;
#pragma unroll
        for (int ks = 0; ks < kKeys / 16; ++ks)
          umma_f16(tmem + kColO, umma_desc(s_base + kOffP + ks * 32, 16, 1024), umma_desc(at + ks * 16 * kRowBytes, 16, 1024),
                   idesc, (b | ks) != 0);
        if (b + 1 < nb) issue_scores(b + 1);
        umma_commit(bar_s);
      }
    }
    s_row[cg * kTileM + row] = l;
    ok = __syncthreads_and(ok && mbar_wait(bar_s, nb & 1));   // the last block's output product
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    l = s_row[row] + s_row[kTileM + row];
#pragma unroll
    for (int half = 0; half < 2; ++half) {   // this thread's 32 of the row's 64 output features
      const int f0 = cg * 32 + half * 16;
      float o[16];
      if (ok) tmem_ld16(row_taddr + kColO + f0, o);   // warp-wide, whether or not the lane's row exists
      if (r < p.n_dst) {
        if (ok && deg == 0) {
#pragma unroll
          for (int j = 0; j < 16; ++j) o[j] = 0.f;
        }
        store_out16(p.o + ((long long)r * p.H + head) * kD + f0, o, deg > 0 ? 1.f / l : 0.f, ok);
      }
    }
    if (r < p.n_dst && cg == 0)
      p.lse[(long long)r * p.H + head] = !ok ? NAN : (deg > 0 ? m * p.scale + logf(l) : -INFINITY);
    if (!ok) {   // a wait ran out: loads asked for are given (bounded) time to land before the shared memory is handed back
      mbar_wait(bar_load, 0);
      for (int b = issued > kSlots ? issued - kSlots : 0; b < issued; ++b) mbar_wait(bar_full + 8 * (b & 1), (b >> 1) & 1);
    }
  } else if (r < p.n_dst && cg == 0) {   // no node of the tile has a neighbour
    __nv_bfloat16* orow = p.o + ((long long)r * p.H + head) * kD;
#pragma unroll
    for (int q = 0; q < kD / 8; ++q) *reinterpret_cast<uint4*>(orow + q * 8) = make_uint4(0, 0, 0, 0);
    p.lse[(long long)r * p.H + head] = -INFINITY;
  }

  // every thread is done with tensor memory: hand it back
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------
// Backward.  Two kernels with the forward's structure, one per side, so that every gradient row has one owner
// (no atomics, as everywhere else):
//   destination side, a tile of 128 query nodes:  S = Q K^T and dP = dO V^T per block of 64 keys,
//       p = exp(scale S - lse), dS = p (dP - delta) scale,  dQ += dS K;   delta = dO . O is formed per row first
//       and left, with lse, in `stat` for the other side;
//   source side, a tile of 128 key nodes:  S^T = K Q^T and dP^T = V dO^T per block of 64 queries,
//       the same p and dS (transposed: a thread is a key, a column a query),  dV += P^T dO,  dK += dS^T Q.
// A tile takes the blocks its band reaches, two of them in shared memory at a time: the next but one is asked for when the
// gradient products that read its slot are done.  85 KB (destination side) or 101 KB (source side) of shared memory and
// 256 tensor-memory columns, so that two tiles share an SM and one's products and loads run under the other's
// element-wise stage: with the whole band and 128 x 128 staging tiles (one tile per SM) the tensor pipe was busy 11 to 14 %
// of the time and every wait was exposed; now 16 to 17 %.
// ---------------------------------------------------------------------------------------------------------
struct BwdParams {
  const __nv_bfloat16* o;     // (n_dst, H, 64): destination side only
  const __nv_bfloat16* d_o;   // (n_dst, H, 64): destination side only (delta)
  const float* lse;           // (n_dst, H): destination side only
  float2* stat;               // (n_dst, H) (lse, delta): written by the destination side, read by the source side
  __nv_bfloat16* out0;        // dq (destination side) / dk (source side)
  __nv_bfloat16* out1;        // dv (source side)
  const int32_t* node_lo;     // first neighbour of every owned node
  const int32_t* node_deg;
  long long n_own;            // nodes on the owning side
  long long n_other;          // nodes on the other side
  int H;
  float scale;
};

constexpr int kBOffA = 0;                          // owned tile, first operand (q | k)
constexpr int kBOffB = kBOffA + kBlockBytes;       // owned tile, second operand (dO | v)
constexpr int kBOffC = kBOffB + kBlockBytes;       // band, per slot: first operand (k | q), second operand (v | dO)
constexpr int kBOffS0 = kBOffC + kSlots * 2 * kBandBytes;   // staging tile 0 (dS | P^T)
constexpr int kBOffS1 = kBOffS0 + kBlockBytes;           // staging tile 1 (dS^T, source side)
constexpr int kBOffBar = 0, kBOffStat = 128;             // behind the staging tiles: barriers, then the (lse, delta) of the
                                                         // band's queries (source side) or the parts of delta
__host__ __device__ constexpr int bwd_tail(bool src) { return kBOffS0 + (src ? 2 : 1) * kBlockBytes; }
__host__ __device__ constexpr int bwd_smem(bool src) { return bwd_tail(src) + kBOffStat + (src ? kSpan * 8 : kColGroups * kTileM * 4) + 1024; }

constexpr int kBTmemCols = 256;   // 64 columns each: scores, dP, two gradients

// kSrc = false: destination side (owned = queries); true: source side (owned = keys)
template <bool kSrc>
__global__ void __launch_bounds__(kThreads, 2)
attention_backward_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                          const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_d,
                          const BwdParams p) {
  extern __shared__ unsigned char raw_smem[];
  unsigned char* smem = raw_smem + ((1024u - (smem_u32(raw_smem) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  constexpr int kTail = bwd_tail(kSrc);
  // bar_load: the owned tiles; bar_full + 8 (b % 2): the band's block b
  const uint32_t bar_load = s_base + kTail + kBOffBar, bar_s = bar_load + 8, bar_g = bar_load + 16, bar_full = bar_load + 64;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kTail + kBOffBar + 32);
  int* s_red = reinterpret_cast<int*>(smem + kTail + kBOffBar + 40);    // 4 ints: per-quarter minima of the first neighbour
  int* s_top = reinterpret_cast<int*>(smem + kTail + kBOffBar + 96);    // 4 ints: and maxima of the last one
  float2* s_stat = reinterpret_cast<float2*>(smem + kTail + kBOffStat);
  float* s_part = reinterpret_cast<float*>(smem + kTail + kBOffStat);   // destination side: [column group][row] parts of delta

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, cg = warp >> 2;   // tensor-memory lane quarter; which 32 of a block's 64 columns
  const int row = quarter * 32 + lane;
  const int head = blockIdx.y;
  const long long r0 = (long long)blockIdx.x * kTileM;
  const long long r = r0 + row;
  int lo = INT_MAX, deg = 0;
  if (r < p.n_own) {
    deg = p.node_deg[r];
    if (deg > 0) lo = p.node_lo[r];
  }
  int wmin = lo, wtop = deg > 0 ? lo + deg - 1 : -1;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    wmin = min(wmin, __shfl_xor_sync(kFull, wmin, o));
    wtop = max(wtop, __shfl_xor_sync(kFull, wtop, o));
  }
  if (lane == 0 && cg == 0) { s_red[quarter] = wmin; s_top[quarter] = wtop; }
  if (tid == 0) {
    mbar_init(bar_load, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_g, 1);
#pragma unroll
    for (int b = 0; b < kSlots; ++b) mbar_init(bar_full + 8 * b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kBTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const int bmin = min(min(s_red[0], s_red[1]), min(s_red[2], s_red[3]));   // first node of the band
  bool ok = true;
  constexpr int kColS = 0, kColP = kKeys, kColG0 = 2 * kKeys, kColG1 = 2 * kKeys + kD;

  if (bmin != INT_MAX) {
    const int btop = max(max(s_top[0], s_top[1]), max(s_top[2], s_top[3]));
    int nb = (btop - bmin) / kKeys + 1;                    // blocks the tile's band reaches
    nb = nb < kSpan / kKeys ? nb : kSpan / kKeys;
    auto issue_band = [&](int b) {   // one thread
      const uint32_t bar = bar_full + 8 * (b & 1), at = s_base + kBOffC + (b & 1) * 2 * kBandBytes;
      mbar_expect_tx(bar, (uint32_t)(2 * kBandBytes));
      tma_load_3d(at, &map_c, bar, 0, head, bmin + b * kKeys);
      tma_load_3d(at + kBandBytes, &map_d, bar, 0, head, bmin + b * kKeys);
    };
    if (tid == 0) {
      mbar_expect_tx(bar_load, (uint32_t)(kBlockBytes * 2));
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        tma_load_3d(s_base + kBOffA + half * kBandBytes, &map_a, bar_load, 0, head, (int)r0 + half * kKeys);
        tma_load_3d(s_base + kBOffB + half * kBandBytes, &map_b, bar_load, 0, head, (int)r0 + half * kKeys);
      }
      issue_band(0);
      if (nb > 1) issue_band(1);
    }
    int issued = nb < kSlots ? nb : kSlots;
    // per-row scalars while the tiles travel
    float lse2 = 0.f, delta = 0.f, lrow = 0.f;
    const float kL2e = 1.4426950408889634f;
    if constexpr (!kSrc) {
      // delta = <o, dO> of the row: each of its two threads takes 32 of the 64 features
      float part = 0.f;
      if (r < p.n_own) {
        const uint4* orow = reinterpret_cast<const uint4*>(p.o + ((long long)r * p.H + head) * kD) + cg * 4;
        const uint4* grow = reinterpret_cast<const uint4*>(p.d_o + ((long long)r * p.H + head) * kD) + cg * 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 ov = __ldg(orow + q), gv = __ldg(grow + q);
          const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&ov);
          const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 of = __bfloat1622float2(o2[e]), gf = __bfloat1622float2(g2[e]);
            part += of.x * gf.x + of.y * gf.y;
          }
        }
        lrow = p.lse[(long long)r * p.H + head];
        lse2 = lrow * kL2e;
      }
      s_part[cg * kTileM + row] = part;
    } else {
      // (lse, delta) of the band's queries: column j of the scores is query bmin + j
      for (int i = tid; i < nb * kKeys; i += kThreads) {
        const long long qn = (long long)bmin + i;
        s_stat[i] = qn < p.n_other ? p.stat[qn * p.H + head] : make_float2(0.f, 0.f);
      }
    }
    ok = __syncthreads_and(mbar_wait(bar_load, 0) && mbar_wait(bar_full, 0));
    if constexpr (!kSrc) {
#pragma unroll
      for (int g = 0; g < kColGroups; ++g) delta += s_part[g * kTileM + row];   // the same order in both threads
      if (cg == 0 && r < p.n_own) p.stat[(long long)r * p.H + head] = make_float2(lrow, delta);
    }

    const int jlo = deg > 0 ? lo - bmin : 1, jhi = deg > 0 ? lo - bmin + deg - 1 : 0;
    int wlo = deg > 0 ? jlo : INT_MAX, whi = deg > 0 ? jhi : -1;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      wlo = min(wlo, __shfl_xor_sync(kFull, wlo, o));
      whi = max(whi, __shfl_xor_sync(kFull, whi, o));
    }
    const uint32_t row_taddr = tmem + ((uint32_t)(quarter * 32) << 16);
    const float sl2 = p.scale * kL2e;
    unsigned char* stage0 = smem + kBOffS0 + row * kRowBytes;
    unsigned char* stage1 = smem + kBOffS1 + row * kRowBytes;

    // scores and dP of one block of the band: owned operands x the band's block (issued by one thread)
    auto issue_scores = [&](int b) {
      constexpr uint32_t idesc = umma_idesc(kTileM, kKeys, false);
      const uint32_t at = s_base + kBOffC + (b & 1) * 2 * kBandBytes;
#pragma unroll
      for (int kk = 0; kk < kD / 16; ++kk)   // scores: owned first operand x band first operand
        umma_f16(tmem + kColS, umma_desc(s_base + kBOffA + kk * 32, 16, 1024), umma_desc(at + kk * 32, 16, 1024), idesc, kk > 0);
#pragma unroll
      for (int kk = 0; kk < kD / 16; ++kk)   // dP: owned second operand x band second operand
        umma_f16(tmem + kColP, umma_desc(s_base + kBOffB + kk * 32, 16, 1024), umma_desc(at + kBandBytes + kk * 32, 16, 1024),
                 idesc, kk > 0);
    };
    if (ok && tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      issue_scores(0);
      umma_commit(bar_s);
    }
    // Per block one wait: the gradient products of block b and the score products of block b + 1 are issued back to
    // back behind one commit (every thread has read block b's scores by then, and the tensor core runs them in
    // order), so when block b + 1's scores are there the staging tiles are free as well.
    for (int b = 0; b < nb; ++b) {
      ok = __syncthreads_and(ok && mbar_wait(bar_s, b & 1));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (ok && b > 0 && b + 1 < nb) {   // block b - 1's slot is free: its gradient products were before block b's scores
        if (tid == 0) issue_band(b + 1);
        issued = b + 2;
      }

      {
        const int c = cg;   // this thread's 32 of the block's 64 columns
        const int col0 = b * kKeys + c * 32;
        const bool live = ok && col0 <= whi && col0 + 31 >= wlo;   // warp-uniform
        uint32_t pk0[16], pk1[16];
        if (live) {
          float sv[32], dv[32];
          tmem_ld32_pair(row_taddr + kColS + c * 32, row_taddr + kColP + c * 32, sv, dv);
          // kTest = false: the whole chunk belongs to the row, no column tests
          auto elements = [&](auto tested) {
            constexpr bool kTest = decltype(tested)::value;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float pa = 0.f, pb = 0.f, da = 0.f, db = 0.f;
              const int col = col0 + j;
              if (!kTest || (col >= jlo && col <= jhi)) {
                const float l2 = kSrc ? s_stat[col].x * kL2e : lse2, dl = kSrc ? s_stat[col].y : delta;
                pa = exp2_fast(fmaf(sv[j], sl2, -l2));
                da = pa * (dv[j] - dl) * p.scale;
              }
              if (!kTest || (col + 1 >= jlo && col + 1 <= jhi)) {
                const float l2 = kSrc ? s_stat[col + 1].x * kL2e : lse2, dl = kSrc ? s_stat[col + 1].y : delta;
                pb = exp2_fast(fmaf(sv[j + 1], sl2, -l2));
                db = pb * (dv[j + 1] - dl) * p.scale;
              }
              pk0[j / 2] = kSrc ? pack_bf16(pa, pb) : pack_bf16(da, db);
              pk1[j / 2] = pack_bf16(da, db);
            }
          };
          if (col0 >= jlo && col0 + 31 <= jhi) elements(std::false_type{});
          else elements(std::true_type{});
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) { pk0[j] = 0u; pk1[j] = 0u; }
        }
        store_stage_row(stage0, c, row, pk0);
        if constexpr (kSrc) store_stage_row(stage1, c, row, pk1);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      // the staging tiles are written by all, and the next block of the band has landed
      ok = __syncthreads_and(ok && (b + 1 >= nb || mbar_wait(bar_full + 8 * ((b + 1) & 1), ((b + 1) >> 1) & 1)));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (ok && tid == 0) {
        constexpr uint32_t idesc = umma_idesc(kTileM, kD, true);
        const uint32_t at = s_base + kBOffC + (b & 1) * 2 * kBandBytes;
#pragma unroll
        for (int ks = 0; ks < kKeys / 16; ++ks) {
          const uint64_t a0 = umma_desc(s_base + kBOffS0 + ks * 32, 16, 1024), c0 = umma_desc(at + ks * 16 * kRowBytes, 16, 1024);
          if constexpr (!kSrc) {   // dQ += dS K_b
            umma_f16(tmem + kColG0, a0, c0, idesc, (b | ks) != 0);
          } else {                 // dV += P^T dO_b,  dK += dS^T Q_b
            umma_f16(tmem + kColG1, a0, umma_desc(at + kBandBytes + ks * 16 * kRowBytes, 16, 1024), idesc, (b | ks) != 0);
            umma_f16(tmem + kColG0, umma_desc(s_base + kBOffS1 + ks * 32, 16, 1024), c0, idesc, (b | ks) != 0);
          }
        }
        if (b + 1 < nb) {
          issue_scores(b + 1);
          umma_commit(bar_s);
        } else {
          umma_commit(bar_g);
        }
      }
    }
    ok = __syncthreads_and(ok && mbar_wait(bar_g, 0));   // the last block's gradient products
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // gradients of the owned rows: this thread's 32 of the 64 features
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int f0 = cg * 32 + half * 16;
      float g0[16], g1[16];
      if (ok) {
        tmem_ld16(row_taddr + kColG0 + f0, g0);
        if constexpr (kSrc) tmem_ld16(row_taddr + kColG1 + f0, g1);
      }
      if (r < p.n_own) {
        const long long at = ((long long)r * p.H + head) * kD + f0;
        const float keep = deg > 0 ? 1.f : 0.f;
        if (ok && deg == 0) {
#pragma unroll
          for (int j = 0; j < 16; ++j) { g0[j] = 0.f; g1[j] = 0.f; }
        }
        store_out16(p.out0 + at, g0, keep, ok);
        if constexpr (kSrc) store_out16(p.out1 + at, g1, keep, ok);
      }
    }
    if (!ok) {   // a wait ran out: loads asked for are given (bounded) time to land before the shared memory is handed back
      mbar_wait(bar_load, 0);
      for (int b = issued > kSlots ? issued - kSlots : 0; b < issued; ++b) mbar_wait(bar_full + 8 * (b & 1), (b >> 1) & 1);
    }
  } else if (r < p.n_own && cg == 0) {  // no owned node of the tile has a neighbour: zero gradients
    const long long at = ((long long)r * p.H + head) * kD;
#pragma unroll
    for (int q = 0; q < kD / 8; ++q) {
      *reinterpret_cast<uint4*>(p.out0 + at + q * 8) = make_uint4(0, 0, 0, 0);
      if constexpr (kSrc) *reinterpret_cast<uint4*>(p.out1 + at + q * 8) = make_uint4(0, 0, 0, 0);
    }
    if constexpr (!kSrc) p.stat[(long long)r * p.H + head] = make_float2(p.lse[(long long)r * p.H + head], 0.f);
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kBTmemCols) : "memory");
  }
}

// cuTensorMapEncodeTiled, fetched from the driver at run time (no link dependency on libcuda)
inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)ptr;
  }();
  return fn;
}

// (n, H, 64) bf16 node tensor as a 3-D map (feature, head, node), boxes of 64 nodes of one head, 128-byte swizzle
inline bool make_map(CUtensorMap* map, const void* base, long long n, int H) {
  auto fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)kD, (cuuint64_t)H, (cuuint64_t)n};
  const cuuint64_t strides[2] = {(cuuint64_t)kRowBytes, (cuuint64_t)H * kRowBytes};
  const cuuint32_t box[3] = {(cuuint32_t)kD, 1u, (cuuint32_t)kKeys};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace banded

template <>
inline int banded_attention_forward<__nv_bfloat16>(const graphop_plan_t* plan, const __nv_bfloat16* q,
                                                   const __nv_bfloat16* k, const __nv_bfloat16* v, double scale,
                                                   __nv_bfloat16* o, void* lse, long long n_dst, long long n_src, int H,
                                                   int D, cudaStream_t st) {
  using namespace banded;
  if (D != kD || H < 1 || H > 65535 || n_dst < 1 || n_src < 1 || n_dst > plan->n_nodes) return GRAPHOP_ERR_UNSUPPORTED;
  if (!(plan->flags & GRAPHOP_PLAN_DENSE_BAND) || plan->band_span > kSpan || !plan->node_lo || !plan->node_deg)
    return GRAPHOP_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o) & 15) return GRAPHOP_ERR_UNSUPPORTED;
  CUtensorMap mq, mk, mv;
  if (!make_map(&mq, q, n_dst, H) || !make_map(&mk, k, n_src, H) || !make_map(&mv, v, n_src, H))
    return GRAPHOP_ERR_UNSUPPORTED;
  static std::atomic<bool> configured[64];
  int dev = 0;
  GK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    GK_CUDA(cudaFuncSetAttribute(attention_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  Params p;
  p.o = o; p.lse = (float*)lse; p.node_lo = plan->node_lo; p.node_deg = plan->node_deg; p.n_dst = n_dst; p.H = H;
  p.scale = (float)scale;
  attention_forward_kernel<<<dim3((unsigned)((n_dst + kTileM - 1) / kTileM), (unsigned)H), kThreads, kSmemBytes, st>>>(mq, mk,
                                                                                                                mv, p);
  GK_LAUNCHED("attention_fwd_banded");
  return GRAPHOP_OK;
}

// Both gradients' kernels for a dense-band graph; `stat` needs n_dst * H * 8 bytes of workspace.
template <>
inline int banded_attention_backward<__nv_bfloat16>(const graphop_plan_t* plan_r, const graphop_plan_t* plan_t,
                                                    const __nv_bfloat16* q, const __nv_bfloat16* k,
                                                    const __nv_bfloat16* v, const __nv_bfloat16* o, const void* lse,
                                                    const __nv_bfloat16* d_o, double scale, __nv_bfloat16* dq,
                                                    __nv_bfloat16* dk, __nv_bfloat16* dv, long long n_dst,
                                                    long long n_src, int H, int D, void* ws, size_t wsb,
                                                    cudaStream_t st) {
  using namespace banded;
  if (D != kD || H < 1 || H > 65535 || n_dst < 1 || n_src < 1) return GRAPHOP_ERR_UNSUPPORTED;
  for (const graphop_plan_t* pl : {plan_r, plan_t})
    if (!(pl->flags & GRAPHOP_PLAN_DENSE_BAND) || pl->band_span > kSpan || !pl->node_lo || !pl->node_deg)
      return GRAPHOP_ERR_UNSUPPORTED;
  if (n_dst > plan_r->n_nodes || n_src > plan_t->n_nodes) return GRAPHOP_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o | (uintptr_t)d_o | (uintptr_t)dq | (uintptr_t)dk |
       (uintptr_t)dv) & 15)
    return GRAPHOP_ERR_UNSUPPORTED;
  GK_TRY(check_ws(ws));
  if (wsb < (size_t)n_dst * H * sizeof(float2)) return GRAPHOP_ERR_WORKSPACE;
  CUtensorMap mq, mk, mv, mg;
  if (!make_map(&mq, q, n_dst, H) || !make_map(&mk, k, n_src, H) || !make_map(&mv, v, n_src, H) ||
      !make_map(&mg, d_o, n_dst, H))
    return GRAPHOP_ERR_UNSUPPORTED;
  static std::atomic<bool> configured[64];
  int dev = 0;
  GK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    GK_CUDA(cudaFuncSetAttribute(attention_backward_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem(false)));
    GK_CUDA(cudaFuncSetAttribute(attention_backward_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem(true)));
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  BwdParams p;
  p.o = o; p.d_o = d_o; p.lse = (const float*)lse; p.stat = (float2*)ws; p.H = H; p.scale = (float)scale;
  p.out0 = dq; p.out1 = nullptr; p.node_lo = plan_r->node_lo; p.node_deg = plan_r->node_deg; p.n_own = n_dst;
  p.n_other = n_src;
  attention_backward_kernel<false><<<dim3((unsigned)((n_dst + kTileM - 1) / kTileM), (unsigned)H), kThreads, bwd_smem(false),
                                     st>>>(mq, mg, mk, mv, p);
  GK_LAUNCHED("attention_bwd_dst_banded");
  p.out0 = dk; p.out1 = dv; p.node_lo = plan_t->node_lo; p.node_deg = plan_t->node_deg; p.n_own = n_src;
  p.n_other = n_dst;
  attention_backward_kernel<true><<<dim3((unsigned)((n_src + kTileM - 1) / kTileM), (unsigned)H), kThreads, bwd_smem(true),
                                    st>>>(mk, mv, mq, mg, p);
  GK_LAUNCHED("attention_bwd_src_banded");
  return GRAPHOP_OK;
}

}  // namespace gk
