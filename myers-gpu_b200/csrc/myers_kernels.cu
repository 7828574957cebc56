// Myers bit-parallel candidate verification kernels for sm_100a.
//
// One candidate = one query (m bases, as PEQ bitmaps) against one window of
// the 4-bit packed reference; the result is the first column of minimum
// semi-global edit distance and that distance (the reference computes the
// same in src-api/coreMyersGPU-CC50.cu:110-240 and, on the CPU,
// src-integration/myers-reorderBuffer-padding.c:97-176).
//
// Layout of the work:
//  * A candidate's query is a vector of 32*L*W rows held by L lanes, W
//    32-bit words per lane. The query occupies the TOP m rows; the bottom
//    p = 32*L*W - m rows are padding rows that match no base. Padding rows
//    add exactly p to every score of the last row (row p of the DP is the
//    constant p), so the score bit is always bit 31 of the top word and the
//    argmin is unchanged; p is subtracted at the end.
//  * Single-lane shapes (L = 1, W = 1..32): one candidate per lane, no lane
//    exchange at all; the W-word add is one add.cc/addc chain.
//  * Multi-lane shapes (L = 2..32): lane l holds rows [32*W*l, 32*W*(l+1)).
//    Lanes run as a systolic pipeline: at step t lane l processes column
//    t - l, taking the horizontal delta of its bottom row from lane l-1
//    (that lane's top-row Ph/Mh bits of the same column, produced one step
//    earlier) through __shfl_up_sync, with Myers' block rule (Eq |= hin<0,
//    hin shifted into Ph/Mh). One shuffle pair per step; no carry ripple.
//  * The PEQ of each candidate is staged once in shared memory, re-laid so
//    that the W words a lane needs for one base are contiguous 16-byte
//    groups (one LDS.128 per 4 words per column), already shifted to the
//    top-aligned row layout.
//  * The text is streamed per lane with one 32-bit load per 8 columns,
//    prefetched one block ahead; a funnel shift realigns it for the exact
//    window mode and for the per-lane skew of the systolic pipeline.
//  * min(score, column) is tracked as one 32-bit key (score << 16 | column):
//    an unsigned min keeps the smallest score and, among equal scores, the
//    first column -- the reference's strict-< tie-break.
#include <cstdint>
#include <cuda_runtime.h>
#include <utility>

#include "myers_internal.h"
#include "myers_device.cuh"
#include "myers_tile.cuh"

namespace myers {

// Plain launch: one shape over a contiguous range of (sorted) candidates.
// Warps take warp tiles from a device counter (`next`, zero at launch), so
// SMs that run ahead take more tiles and the launch ends evenly.
template <int W, bool MULTI>
__global__ void __launch_bounds__(128) k_plain(DevInputs in, const uint32_t* __restrict__ ids,
                                               const BucketState* __restrict__ st, int cfg, uint32_t first,
                                               uint32_t count, int L, uint32_t* __restrict__ next) {
  extern __shared__ __align__(16) uint32_t smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (st != nullptr) {
    first = st->first[cfg];
    count = st->count[cfg];
  }
  const int nseg = MULTI ? 32 / L : 32;
  uint32_t* wsmem = smem + wib * warp_words<W, MULTI>();
  const uint32_t tiles = (count + nseg - 1) / nseg;
  while (true) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(next, 1u);
    t = __shfl_sync(FULL_MASK, t, 0);
    if (t >= tiles) break;
    const uint32_t f = t * nseg;
    const uint32_t cnt = min((uint32_t)nseg, count - f);
    process_tile<W, MULTI, 8, fma_shift<W, MULTI, false>()>(in, ids, first + f, cnt, L, wsmem, lane);
  }
}

// ---- length bucketing on the device ----

// With TWO (the cut-off's first pass) a candidate is classified by its
// prefix's word count under `plan`, and, when the prefix covers only part of
// its query, by its full word count under `plan2` into in.esc_cfg, counted in
// in.esc_state->cursor (the second pass's layout).
template <bool TWO>
struct Lookups {
  PlanLookup plan, second;
};
template <>
struct Lookups<false> {
  PlanLookup plan;
};

template <bool TWO>
__global__ void k_classify(DevInputs in, const __grid_constant__ Lookups<TWO> plans, BucketState* st,
                           uint8_t* __restrict__ cfg_of_cand) {
  const int lane = threadIdx.x & 31;
  const uint32_t n = in.num_cands;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < n; base += stride) {
    const uint32_t i = base + lane;
    uint32_t cfg = kNoCfg;
    if (i < n) {
      const Cand cd = in.cands[i];
      uint2 q = make_uint2(0u, 0u);
      if (cd.query < in.num_queries) q = __ldg(in.qinfo + cd.query);
      const uint32_t bad = check_query(in, cd.query, q);
      const uint32_t mf = q.y;
      const uint32_t m = TWO ? d_prefix_rows(mf, in.cutoff, in.prefix_mult) : mf;
      const uint32_t wb = d_window_bases(mf, in.distance);
      const bool valid = bad == 0u && cd.position < in.ref_size &&
                         (in.ref_size - cd.position) > (unsigned long long)wb;
      const uint32_t ncol = in.exact ? wb : 8u * d_window_words(wb);
      if (bad) {
        in.results[i] = make_uint2(0u, kNoResult);
        atomicOr(in.flags, bad);
      } else if (!valid) {
        in.results[i] = make_uint2(0u, kNoResult);
      } else if (m == 0) {
        in.results[i] = make_uint2(0u, 0u);
      } else {
        const bool sized = mf <= kMaxWords * 32 && ncol <= kMaxColumns;
        uint32_t second = 0;
        if (sized) {
          cfg = plan_cfg(plans.plan, m);
          if constexpr (TWO)
            if (m < mf) second = plan_cfg(plans.second, mf);
        }
        if (cfg == kNoCfg || second == kNoCfg) {
          cfg = kNoCfg;
          in.results[i] = make_uint2(0u, kNoResult);
          atomicOr(in.flags, kFlagUnsupported);
        } else if (TWO && m < mf) {
          in.esc_cfg[i] = (uint8_t)second;
          atomicAdd(&in.esc_state->cursor[second], 1u);
        }
      }
      cfg_of_cand[i] = (uint8_t)cfg;
    }
    const unsigned peers = __match_any_sync(FULL_MASK, cfg);
    if (cfg != kNoCfg && lane == __ffs(peers) - 1) atomicAdd(&st->count[cfg], (uint32_t)__popc(peers));
  }
}

// The second pass's layout: each full-length shape's list starts where the
// candidates counted for it in the classification end up at most; the lists
// fill as the first pass appends to them.
__global__ void k_plan_escalation(const __grid_constant__ PlanShapes plan2, BucketState* esc) {
  if (threadIdx.x != 0) return;
  uint32_t acc = 0;
  for (uint32_t c = 0; c < plan2.num_cfg; ++c) {
    esc->first[c] = acc;
    acc += esc->cursor[c];
    esc->count[c] = 0;
    esc->next[c] = 0;
  }
}

// The second pass's tiles on the persistent path, once the first pass has
// filled the lists: each shape's tiles from its list length, the persistent
// kernel's tile count and a fresh work counter.
__global__ void k_plan_tiles(const __grid_constant__ PlanShapes plan2, BucketState* esc) {
  if (threadIdx.x != 0) return;
  uint32_t tiles = 0;
  for (uint32_t c = 0; c < plan2.num_cfg; ++c) {
    const Shape s = plan2.shape[c];
    const uint32_t nseg = (s.variant >= kNumSingle) ? 32u / s.L : 32u;
    if (c == plan2.num_batched) esc->total_tiles = tiles;
    esc->tile_start[c] = tiles;
    tiles += (esc->count[c] + nseg - 1) / nseg;
  }
  esc->tile_start[plan2.num_cfg] = tiles;
  if (plan2.num_batched >= plan2.num_cfg) esc->total_tiles = tiles;
  esc->queue = 0;
}

__global__ void k_plan(const __grid_constant__ PlanShapes plan, BucketState* st) {
  if (threadIdx.x != 0) return;
  uint32_t acc = 0, tiles = 0;
  for (uint32_t c = 0; c < plan.num_cfg; ++c) {
    const Shape s = plan.shape[c];
    const uint32_t nseg = (s.variant >= kNumSingle) ? 32u / s.L : 32u;
    if (c == plan.num_batched) st->total_tiles = tiles;
    st->first[c] = acc;
    st->cursor[c] = 0;
    st->tile_start[c] = tiles;
    tiles += (st->count[c] + nseg - 1) / nseg;
    acc += st->count[c];
  }
  st->tile_start[plan.num_cfg] = tiles;
  if (plan.num_batched >= plan.num_cfg) st->total_tiles = tiles;
  st->queue = 0;
}

// Stable within each warp's 32 consecutive candidates, so the candidates of
// one read (adjacent in the input) mostly stay adjacent.
__global__ void k_scatter(uint32_t n, const uint8_t* __restrict__ cfg_of_cand, BucketState* st,
                          uint32_t* __restrict__ ids) {
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < n; base += stride) {
    const uint32_t i = base + lane;
    const uint32_t cfg = i < n ? cfg_of_cand[i] : kNoCfg;
    const unsigned peers = __match_any_sync(FULL_MASK, cfg);
    const int leader = __ffs(peers) - 1;
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    uint32_t b = 0;
    if (cfg != kNoCfg && lane == leader) b = atomicAdd(&st->cursor[cfg], (uint32_t)__popc(peers));
    b = __shfl_sync(FULL_MASK, b, leader);
    if (cfg != kNoCfg) ids[st->first[cfg] + b + rank] = i;
  }
}

// ---- the persistent batched kernel ----

constexpr uint32_t cmax(uint32_t a, uint32_t b) { return a > b ? a : b; }
// the largest batched shape's footprint
constexpr uint32_t kBatchedWarpWords =
    cmax(cmax(warp_words<32, false>(), warp_words<16, false>()), warp_words<kBatchedMaxMultiW, true>());

#ifndef MYERS_BATCHED_UNROLL
#define MYERS_BATCHED_UNROLL 2
#endif

template <int V>
__device__ __forceinline__ void dispatch_one(const DevInputs& in, const uint32_t* ids, uint32_t f, uint32_t cnt,
                                             int L, uint32_t* wsmem, int lane) {
  if constexpr (V < kNumSingle) {
    process_tile<V + 1, false, MYERS_BATCHED_UNROLL, fma_shift<V + 1, false, true>()>(in, ids, f, cnt, L, wsmem,
                                                                                       lane);
  } else {
    if constexpr (kMultiW[V - kNumSingle] <= kBatchedMaxMultiW)
      process_tile<kMultiW[V - kNumSingle], true, MYERS_BATCHED_UNROLL,
                   fma_shift<kMultiW[V - kNumSingle], true, true>()>(in, ids, f, cnt, L, wsmem, lane);
  }
}

template <int... Vs>
__device__ __forceinline__ void dispatch(int v, const DevInputs& in, const uint32_t* ids, uint32_t f, uint32_t cnt,
                                         int L, uint32_t* wsmem, int lane, std::integer_sequence<int, Vs...>) {
  ((v == Vs ? (dispatch_one<Vs>(in, ids, f, cnt, L, wsmem, lane), 0) : 0), ...);
}

// Each warp pulls the next tile index from the device queue; tiles are
// ordered by shape, most expensive shape first, so the long candidates start
// early and the short ones fill the tail.
// At least three blocks of four warps per SM. ptxas then takes 159
// registers (three blocks fit); a bound of four holds it at 115 without a
// spill, and measured 0.2-0.4% slower on long and mixed reads.
#ifndef MYERS_BATCHED_MIN_BLOCKS
#define MYERS_BATCHED_MIN_BLOCKS 3
#endif
__global__ void __launch_bounds__(128, MYERS_BATCHED_MIN_BLOCKS) k_batched(DevInputs in, const uint32_t* __restrict__ ids,
                                                 const __grid_constant__ PlanShapes plan, BucketState* st) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint32_t s_tile_start[kMaxCfg + 1];
  __shared__ uint32_t s_first[kMaxCfg];
  __shared__ uint32_t s_count[kMaxCfg];
  __shared__ Shape s_shape[kMaxCfg];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t ncfg = plan.num_batched;
  for (uint32_t c = threadIdx.x; c < ncfg; c += blockDim.x) {
    s_tile_start[c] = st->tile_start[c];
    s_first[c] = st->first[c];
    s_count[c] = st->count[c];
    s_shape[c] = plan.shape[c];
  }
  __syncthreads();
  const uint32_t total = st->total_tiles;
  uint32_t* wsmem = smem + wib * kBatchedWarpWords;
  while (true) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(&st->queue, 1u);
    t = __shfl_sync(FULL_MASK, t, 0);
    if (t >= total) break;
    // last shape whose first tile is <= t
    uint32_t lo = 0, hi = ncfg - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (s_tile_start[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    const Shape s = s_shape[lo];
    const int L = s.L;
    const uint32_t nseg = (s.variant >= kNumSingle) ? 32u / (uint32_t)L : 32u;
    const uint32_t f = (t - s_tile_start[lo]) * nseg;
    const uint32_t cnt = min(nseg, s_count[lo] - f);
    dispatch(s.variant, in, ids, s_first[lo] + f, cnt, L, wsmem, lane,
             std::make_integer_sequence<int, kNumVariants>{});
  }
}

// Integer-ALU peak probe: eight independent chains of 3-input logic ops per
// thread (the instruction class of the Myers column), written out so the
// work cannot be removed.
__global__ void k_lop3_probe(uint32_t* out, int iters) {
  uint32_t a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = threadIdx.x * (k + 3) + blockIdx.x;
  uint32_t b = threadIdx.x ^ 0x5A5A5A5Au;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int r = 0; r < 16; ++r) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(a[k]) : "r"(a[(k + 1) & 7]), "r"(b));
    }
  }
  uint32_t x = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) x ^= a[k];
  out[blockIdx.x * blockDim.x + threadIdx.x] = x;
}

// ---- host-side launchers ----

using PlainFn = void (*)(DevInputs, const uint32_t*, const BucketState*, int, uint32_t, uint32_t, int, uint32_t*);

template <int V>
constexpr PlainFn plain_fn() {
  if constexpr (V < kNumSingle) return &k_plain<V + 1, false>;
  else return &k_plain<kMultiW[V - kNumSingle], true>;
}

template <int... Vs>
constexpr auto make_plain_table(std::integer_sequence<int, Vs...>) {
  struct T { PlainFn f[sizeof...(Vs)]; };
  return T{{plain_fn<Vs>()...}};
}

static const auto kPlainTable = make_plain_table(std::make_integer_sequence<int, kNumVariants>{});

uint32_t warp_smem_bytes(int v, int) {
  const int W = variant_W(v);
  const int slots = variant_multi(v) ? 32 : (W > 16 ? 16 : 32);
  const int ncol = ((slots + 7) / 8) * 8 + 1;
  return (uint32_t)(((W + 3) / 4) * 5 * ncol * 4 * 4);
}

static int blocks_per_sm(const void* fn, int threads, size_t smem) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem) != cudaSuccess || nb < 1) nb = 1;
  return nb;
}

cudaError_t launch_plain(int v, int L, const DevInputs& in, const uint32_t* d_ids, const BucketState* d_state,
                         int cfg, uint32_t first, uint32_t count, uint32_t* d_next, cudaStream_t s, int num_sms) {
  const PlainFn fn = kPlainTable.f[v];
  const int threads = 128;
  const int Lr = variant_multi(v) ? L : 1;
  const size_t smem = (size_t)warp_smem_bytes(v, Lr) * (threads / 32);
  cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int nb = blocks_per_sm((const void*)fn, threads, smem);
  uint32_t grid = (uint32_t)(num_sms * nb);
  if (d_state == nullptr) {
    const uint32_t nseg = variant_multi(v) ? 32u / (uint32_t)L : 32u;
    const uint32_t tiles = (count + nseg - 1) / nseg;
    const uint32_t need = (tiles + threads / 32 - 1) / (threads / 32);
    if (need < grid) grid = need;
    if (grid == 0) return cudaSuccess;
  }
  fn<<<grid, threads, smem, s>>>(in, d_ids, d_state, cfg, first, count, Lr, d_next);
  return cudaGetLastError();
}

int launch_bucketing(const DevInputs& in, const PlanTable& plan, BucketState* d_state, uint8_t* d_cfg_of_cand,
                     uint32_t* d_ids, cudaStream_t s, int num_sms, cudaError_t* err) {
  const int threads = 256;
  const uint32_t need = (in.num_cands + threads - 1) / threads;
  uint32_t grid = (uint32_t)num_sms * 8;
  if (need < grid) grid = need > 0 ? need : 1;
  k_classify<false><<<grid, threads, 0, s>>>(in, Lookups<false>{plan}, d_state, d_cfg_of_cand);
  k_plan<<<1, 32, 0, s>>>(plan, d_state);
  k_scatter<<<grid, threads, 0, s>>>(in.num_cands, d_cfg_of_cand, d_state, d_ids);
  *err = cudaGetLastError();
  return 3;
}

int launch_bucketing_cutoff(const DevInputs& in, const PlanTable& plan, const PlanTable& plan2,
                            BucketState* d_state, uint8_t* d_cfg_of_cand, uint32_t* d_ids, cudaStream_t s,
                            int num_sms, cudaError_t* err) {
  const int threads = 256;
  const uint32_t need = (in.num_cands + threads - 1) / threads;
  uint32_t grid = (uint32_t)num_sms * 8;
  if (need < grid) grid = need > 0 ? need : 1;
  k_classify<true><<<grid, threads, 0, s>>>(in, Lookups<true>{plan, plan2}, d_state, d_cfg_of_cand);
  k_plan<<<1, 32, 0, s>>>(plan, d_state);
  k_plan_escalation<<<1, 32, 0, s>>>(plan2, in.esc_state);
  k_scatter<<<grid, threads, 0, s>>>(in.num_cands, d_cfg_of_cand, d_state, d_ids);
  *err = cudaGetLastError();
  return 4;
}

cudaError_t launch_plan_tiles(const PlanTable& plan2, BucketState* d_esc_state, cudaStream_t s) {
  k_plan_tiles<<<1, 32, 0, s>>>(plan2, d_esc_state);
  return cudaGetLastError();
}

cudaError_t launch_batched(const DevInputs& in, const uint32_t* d_ids, const PlanTable& plan,
                           BucketState* d_state, cudaStream_t s, int num_sms, uint32_t max_tiles) {
  const int threads = 128;
  const size_t smem = (size_t)kBatchedWarpWords * 4 * (threads / 32);
  cudaError_t e = cudaFuncSetAttribute((const void*)k_batched, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  const int nb = blocks_per_sm((const void*)k_batched, threads, smem);
  uint32_t grid = (uint32_t)(num_sms * nb);
  const uint32_t need = (max_tiles + threads / 32 - 1) / (threads / 32);
  if (need < grid) grid = need > 0 ? need : 1;
  k_batched<<<grid, threads, smem, s>>>(in, d_ids, plan, d_state);
  return cudaGetLastError();
}

cudaError_t load_batched_path_kernels() {
  cudaFuncAttributes a;
  const void* fns[] = {(const void*)k_classify<false>, (const void*)k_plan, (const void*)k_scatter,
                       (const void*)k_batched, sliced_class_kernel<0>(), sliced_class_kernel<1>(),
                       sliced_class_kernel<2>(), sliced_class_kernel<3>()};
  for (const void* f : fns) {
    const cudaError_t e = cudaFuncGetAttributes(&a, f);
    if (e != cudaSuccess) return e;
  }
  for (int v = 0; v < kNumVariants; ++v) {
    if (batched_supports(v)) continue;  // shapes the persistent kernel does not carry get plain launches
    const cudaError_t e = cudaFuncGetAttributes(&a, (const void*)kPlainTable.f[v]);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_lop3_probe(uint32_t* d_out, int blocks, int threads, int iters, cudaStream_t s) {
  k_lop3_probe<<<blocks, threads, 0, s>>>(d_out, iters);
  return cudaGetLastError();
}

}  // namespace myers

// ---- packers on the device ----

namespace myers {

// ASCII base -> code: A0 C1 G2 T3 (either case), anything else 4
// (src-api/genReference-4bits.c:21-40, genCandidate-reorder.c:237-256).
__device__ __forceinline__ uint32_t ascii_code(uint32_t b) {
  const uint32_t u = b & 0xDFu;  // upper case
  return u == 'A' ? 0u : u == 'C' ? 1u : u == 'G' ? 2u : u == 'T' ? 3u : 4u;
}

// Four bases at a time. In ASCII, bits 1 and 2 tell the letters apart (A 00, C
// 01, T 10, G 11); the byte is that letter, of either case, iff bits 7, 6 and 3
// are 010, bit 4 is set for T alone and bit 0 for the other three alone.
// Non-zero bits of the result: bytes that are none of the four.
__device__ __forceinline__ uint32_t not_acgt(uint32_t w) {
  const uint32_t t = w & 0x04040404u & ~(w * 2u);  // T: bit 2 without bit 1
  const uint32_t x = w ^ (t * 4u + (t >> 2)) ^ 0x41414141u;
  return x & 0xD9D9D9D9u;
}
// Bits 0, 8, 16 and 24 of x, times 2^p, as bits 28 .. 31.
template <int P>
__device__ __forceinline__ uint32_t gather4(uint32_t x) {
  return x * (0x10204080u >> P);
}

// One lane per 32-base word, over the words of `per` consecutive reads at a
// time: the five 32-bit bitmaps of that word. Bits past the read's end are 0
// (src-api/genCandidate-reorder.c:258-317).
//
// Bound by the ALU pipe and by memory (one byte in, 0.625 out per base): the
// bytes' two letter bits are gathered four at a time by a multiplication, and
// the planes follow from the two gathered words; bytes that are no letter of
// the four take a second look. 100K reads of 1,000 bases (164 MB, 25 us of
// copying) took 176 us with a byte load and a table update per base, and take
// 43; 1M of 100 bases 1,470 (a warp per read) and 47.
__global__ void k_pack_peq(const uint8_t* __restrict__ ascii, unsigned long long ascii_bytes,
                           const unsigned long long* __restrict__ offsets, const uint2* __restrict__ qinfo,
                           uint32_t num_reads, uint32_t* __restrict__ peq, uint32_t num_entries,
                           uint32_t* __restrict__ flags, uint32_t per) {
  const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
  const int lane = threadIdx.x & 31;
  const uint32_t batches = (num_reads + per - 1) / per;
  for (uint32_t batch = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); batch < batches; batch += nwarps) {
    // lane r holds read r of the batch: its words (whole entries) before and
    // after those of the reads up to it
    const uint32_t r = batch * per + (uint32_t)lane;
    uint2 q = make_uint2(0u, 0u);
    unsigned long long o = 0;
    uint32_t words = 0;
    if ((uint32_t)lane < per && r < num_reads) {
      q = qinfo[r];
      o = offsets[r];
      const unsigned long long o1 = offsets[r + 1];
      words = (q.y + 127) / 128 * 4;
      if ((unsigned long long)q.x + words / 4 > num_entries || o1 < o || o1 - o < q.y || o1 > ascii_bytes) {
        atomicOr(flags, kFlagBadEntry);
        words = 0;
      }
    }
    uint32_t end = words;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t x = __shfl_up_sync(FULL_MASK, end, s);
      if (lane >= s) end += x;
    }
    const uint32_t total = __shfl_sync(FULL_MASK, end, 31);
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
      const uint32_t i = i0 + (uint32_t)lane;
      // the first read whose words end after i
      int at = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const uint32_t e = __shfl_sync(FULL_MASK, end, at + s - 1);
        if (e <= i) at += s;
      }
      at = min(at, 31);
      const uint32_t m = __shfl_sync(FULL_MASK, q.y, at), entry = __shfl_sync(FULL_MASK, q.x, at);
      const unsigned long long base = __shfl_sync(FULL_MASK, o, at);
      const uint32_t first = __shfl_sync(FULL_MASK, end - words, at);
      if (i >= total) continue;
      const uint32_t w = i - first;
      const uint32_t left = m > 32 * w ? m - 32 * w : 0u;
      uint32_t bm[5] = {0u, 0u, 0u, 0u, 0u};
      if (left > 0) {
        const uint8_t* p = ascii + base + 32ull * w;
        const uint32_t sh = 8u * (uint32_t)((uintptr_t)p & 3u);
        const uint8_t* a = p - (sh >> 3);
        uint32_t v[9];
        if (a >= ascii && a + 36 <= ascii + ascii_bytes) {
          const uint32_t* x = reinterpret_cast<const uint32_t*>(a);
#pragma unroll
          for (int k = 0; k < 9; ++k) v[k] = __ldg(x + k);
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = __funnelshift_r(v[k], v[k + 1], sh);
        } else {  // at an edge of the buffer: the read's bytes alone
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            v[k] = 0u;
            for (uint32_t b = 0; b < 4; ++b)
              if (4u * k + b < left) v[k] |= (uint32_t)p[4 * k + b] << (8 * b);
          }
        }
        uint32_t b1 = 0u, b2 = 0u, odd = 0u;
#pragma unroll
        for (int k = 7; k >= 0; --k) {  // in from below
          b1 = __funnelshift_l(gather4<1>(v[k] & 0x02020202u), b1, 4);
          b2 = __funnelshift_l(gather4<2>(v[k] & 0x04040404u), b2, 4);
          odd |= not_acgt(v[k]);
        }
        const uint32_t inside = left >= 32u ? FULL_MASK : (1u << left) - 1u;
        uint32_t n = 0u;
        if (odd) {
#pragma unroll
          for (int k = 7; k >= 0; --k) {
            const uint32_t z = not_acgt(v[k]);
            const uint32_t other = ((((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) >> 7) & 0x01010101u;  // byte not zero
            n = __funnelshift_l(gather4<0>(other), n, 4);
          }
        }
        const uint32_t letter = inside & ~n;
        bm[0] = letter & ~b1 & ~b2;
        bm[1] = letter & b1 & ~b2;
        bm[2] = letter & b1 & b2;
        bm[3] = letter & ~b1 & b2;
        bm[4] = inside & n;
      }
      uint32_t* e = peq + (size_t)(entry + w / 4) * 20 + (w & 3);
#pragma unroll
      for (int c = 0; c < 5; ++c) e[c * 4] = bm[c];
    }
  }
}

// One thread per packed word: eight bases, base i in bits 4*(i%8); bases at
// or past n are N (src-api/genReference-4bits.c:43-72).
__global__ void k_pack_reference(const uint8_t* __restrict__ ascii, unsigned long long n, uint32_t* __restrict__ words,
                                 unsigned long long nwords) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long w = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += stride) {
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const unsigned long long i = w * 8 + k;
      v |= (i < n ? ascii_code(ascii[i]) : 4u) << (4 * k);
    }
    words[w] = v;
  }
}

cudaError_t launch_pack_peq(const uint8_t* ascii, unsigned long long ascii_bytes, const unsigned long long* offsets,
                            const uint2* qinfo, uint32_t num_reads, uint32_t* peq, uint32_t num_entries,
                            uint32_t* flags, cudaStream_t s, int num_sms) {
  if (num_reads == 0) return cudaSuccess;
  // as many reads per warp as leave the device a few rounds of warps
  uint32_t per = 32;
  while (per > 1 && num_reads / per < (uint32_t)num_sms * 192) per /= 2;
  const uint32_t warps = (num_reads + per - 1) / per;
  const uint32_t grid = (warps + 7) / 8;
  k_pack_peq<<<grid, 256, 0, s>>>(ascii, ascii_bytes, offsets, qinfo, num_reads, peq, num_entries, flags, per);
  return cudaGetLastError();
}

cudaError_t launch_pack_reference(const uint8_t* ascii, unsigned long long n, uint32_t* words,
                                  unsigned long long nwords, cudaStream_t s, int num_sms) {
  if (nwords == 0) return cudaSuccess;
  unsigned long long grid = (nwords + 255) / 256;
  if (grid > (unsigned long long)num_sms * 32) grid = (unsigned long long)num_sms * 32;
  k_pack_reference<<<(unsigned)grid, 256, 0, s>>>(ascii, n, words, nwords);
  return cudaGetLastError();
}

}  // namespace myers
