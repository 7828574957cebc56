// Bit-sliced candidate verification for sm_100a: 32 candidates per register.
//
// The word-parallel kernels hold 32 rows of one candidate in a register, so a
// column costs a carry chain and two one-bit shifts per word: ten ALU
// instructions per 32 cells. Here bit c of a register belongs to candidate c
// of a group of 32, and a register is one row: the carries and the shifts are
// gone, because a row's horizontal delta is simply the next row's input. With
// Pv/Mv (vertical deltas) and Ph/Mh (horizontal deltas) of a cell and the
// diagonal step N = mismatch & ~Mv & ~Mh, the outputs are h' = N - v and
// v' = N - h, that is
//     Mh' = Pv & ~N    Ph' = Mh' + (N - (Pv - Mv))
//     Mv' = Ph & ~N    Pv' = Mv' + (N - (Ph - Mh))
// where no sum or difference carries from bit to bit in the end (each result
// is a bit set again). Five ALU instructions per row and column (three for N,
// see below, and Mh', Mv') and five multiply-adds by an opaque 1 or -1 on the
// FMA pipe, against ten ALU instructions before.
//
// Layout of the work:
//  * A tile is 32 / L groups of 32 candidates in one warp (L = 8, 16 or 32
//    lanes per group), or one group over NW = 2, 4 or 8 warps (LL = 32 NW
//    lanes). Lane l of a group holds R rows, R = ceil(m / LL). Reads of
//    65..10,240 bases.
//  * Lanes run as a systolic pipeline: at step t lane l takes column t - l,
//    with the horizontal delta of lane l-1's top row through two shuffles
//    (through a ring in shared memory from the warp below). Steps before a
//    lane's first column see a column that matches nothing, which leaves the
//    initial state (every v = +1, h = 0) as it is, so fill needs no test.
//  * Base codes are two bit planes (A 00, C 01, G 10, T 11) per row and per
//    column; a third plane marks text columns that match nothing (N, fill).
//    mismatch = (q0 ^ t0) | (q1 ^ t1) | t2 takes two 3-input logic ops, and
//    the third forms N. Reads with an N, and rows without any base, need the
//    query's third plane too (GEN, one more op per row); tiles whose PEQ has
//    a row with several bases run in the word-parallel tile instead.
//  * Within a group the lengths may differ by less than LL: a candidate that is
//    p rows short of LL * R skips row 0 of lanes 0..p-1 (a masked copy of the
//    horizontal delta), so every lane still runs R rows.
//  * Query rows, text columns and the last row's deltas change between "one
//    candidate per lane" and "one candidate per bit" by 32 x 32 bit
//    transpositions over the warp (five shuffles).
//  * The last row's deltas go to a ring in shared memory; per 32 columns they
//    are transposed back, and each lane scans its candidate's 32 columns four
//    at a time through a table of (change, smallest prefix, its column).
//
// What bounds it: a row and column takes 10.4 instructions, 5.1 on the ALU
// pipe (two cycles each), 5.1 multiply-adds; the loop alone measures 12.5 to
// 14.5 cycles per scheduler, near what reading 23 register operands allows
// (pairs of a 3-input logic op and a multiply-add issue every 3 cycles, not
// 2). The form with logic ops alone (7 per row) measures 15.1, the
// word-parallel kernels 21 per 32 cells. With slicing, scanning, fill and the
// last round, 330K candidates of 1,000-base reads take 6.6 ms (8.8
// word-parallel), 1.1M of 100 bases 0.38 (0.44), 100K of 1,000..10,000 bases
// 44.5 (63.2).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "myers_device.cuh"
#include "myers_internal.h"
#include "myers_tile.cuh"

namespace myers {

// A kernel per class of shapes: warps per block, blocks per SM, rows per lane.
// A row's state takes four registers, so the fewer rows, the more warps an SM
// holds; more than one warp per scheduler hides what is not the recurrence
// (slicing, scanning, the step from lane to lane).
template <int WARPS, int BLOCKS, int RLO, int RHI, bool CHAIN>
struct SlicedClass {
  static constexpr int kWarps = WARPS, kThreads = WARPS * 32, kBlocks = BLOCKS, kLo = RLO, kHi = RHI;
  static constexpr bool kChain = CHAIN;                        // groups of several warps
  static constexpr int kGroups = CHAIN ? 1 : 4;                // groups of 32 candidates per warp, at most
  static constexpr int kStride = RHI | 1;                      // plane words per lane: odd, so no bank conflicts
  static constexpr uint32_t kRing = CHAIN ? 128 : 64;          // columns of the last row's ring
  // Shared memory of a warp: the candidates' table, then the query planes,
  // which the text ring (64 columns) and the last row's ring replace.
  static constexpr uint32_t kTable = kGroups * 32 * 28;
  static constexpr uint32_t kPlanes = 3 * 32 * kStride * 4;
  static constexpr uint32_t kRings = kGroups * (64 * 16 + kRing * 8);
  static constexpr uint32_t kWords = Layout<CHAIN ? 16 : 4, true>::WORDS * 4;
  static constexpr uint32_t kMost = kPlanes > kRings ? (kPlanes > kWords ? kPlanes : kWords) : (kRings > kWords ? kRings : kWords);
  static constexpr uint32_t kWarpBytes = kTable + (kMost + 15) / 16 * 16;
  static constexpr uint32_t kSmemBytes = 256 * 8 + kWarpBytes * WARPS;
  static_assert(BLOCKS * (kSmemBytes + 1024 + 128) <= 228 * 1024, "shared memory of an SM");
  __device__ static bool has(const Shape& s) { return (s.L > 5) == CHAIN && s.W >= RLO && s.W <= RHI; }
};

// The classes; sliced_class (myers_internal.h) says which one a shape is in.
using Sliced16 = SlicedClass<4, 4, 8, 16, false>;
using Sliced24 = SlicedClass<4, 3, 17, 24, false>;
using Sliced32 = SlicedClass<4, 2, 25, 32, false>;
using SlicedChain = SlicedClass<8, 1, 17, 40, true>;

// Whether every length has a shape with a kernel for its rows per lane.
constexpr bool shapes_have_kernels() {
  for (uint32_t spread = 0; spread < 3; ++spread)
    for (uint32_t m = kSlicedMinRows; m <= kSlicedMaxRows; ++m) {
      int lg = 0, R = 0;
      sliced_shape(m, spread, &lg, &R);
      const int lo = lg > 5 ? SlicedChain::kLo : Sliced16::kLo, hi = lg > 5 ? SlicedChain::kHi : Sliced32::kHi;
      if (R < lo || R > hi || (R > 32 && R % 2 != 0)) return false;
    }
  return true;
}
static_assert(shapes_have_kernels(), "rows per lane without a kernel");

// 3-input logic op by truth table (A 0xF0, B 0xCC, C 0xAA).
constexpr int kA = 0xF0, kB = 0xCC, kC = 0xAA;
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT & 0xFF));
  return d;
}

// Multipliers the compiler cannot fold (constant memory is the host's to
// write), read as an operand of the multiply-add itself.
static __constant__ uint32_t c_one = 1u, c_mone = 0xFFFFFFFFu;

// a * b + c with such a multiplier: runs on the FMA pipe.
__device__ __forceinline__ uint32_t mad(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// 32 x 32 bit transpositions over the warp: bit c of lane i becomes bit i of
// lane c. N words at a time, so that their shuffles overlap. Halves and bytes
// change places by one byte permutation, nibbles and less by a rotation and a
// select.
template <int N>
__device__ __forceinline__ void transpose32(uint32_t (&x)[N], int lane) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const bool up = lane & s;
    const uint32_t low = s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t pick = s == 16 ? (up ? 0x3276u : 0x5410u) : (up ? 0x3715u : 0x6240u);
    const uint32_t keep = up ? ~low : low;
    const int by = up ? 32 - s : s;
    uint32_t y[N];
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = __shfl_xor_sync(FULL_MASK, x[k], s);
#pragma unroll
    for (int k = 0; k < N; ++k)
      x[k] = s >= 8 ? __byte_perm(x[k], y[k], pick)
                    : lop3<(kA & kB) | (kC & ~kB)>(x[k], keep, __funnelshift_l(y[k], y[k], by));
  }
}

// One warp's tile.
struct Tile {
  const uint32_t* ids;
  uint32_t first;      // first candidate (an index into ids, or the candidate's id)
  uint32_t cnt;        // candidates, at most 32 * nseg
  uint32_t row_min, row_limit;  // queries the plan admits
  int R;               // rows per lane
  int lg;              // log2 of the lanes per group over all its warps (LL)
  int nw, wg;          // warps of the group, this warp's place among them
  int group;           // the group's named barrier (nw > 1)
};

extern __shared__ __align__(16) unsigned char sl_smem[];

struct WarpMem {
  unsigned long long* b0;  // first text word
  uint32_t* id;
  uint32_t* mm;            // rows m | query length mf << 16
  uint32_t* nsh;           // columns n (0: nothing to do) | text shift << 16
  uint32_t* kmin;          // smallest (score << 16 | column); the first PEQ entry while rows are staged
  uint32_t* sk;            // running (score << 16 | column)
  uint32_t* buf;           // planes, then rings
};

// The share of warp `warp`. Derived from the block's shared array wherever it is
// needed, so that accesses are known to be shared-memory accesses.
template <class K>
__device__ __forceinline__ WarpMem warp_mem(int warp) {
  constexpr int n = 32 * K::kGroups;
  WarpMem w;
  w.b0 = reinterpret_cast<unsigned long long*>(sl_smem + 256 * sizeof(int2) + warp * K::kWarpBytes);
  w.id = reinterpret_cast<uint32_t*>(w.b0 + n);
  w.mm = w.id + n;
  w.nsh = w.mm + n;
  w.kmin = w.nsh + n;
  w.sk = w.kmin + n;
  w.buf = w.sk + n;
  return w;
}

__device__ __forceinline__ void group_barrier(const Tile& t) {
  if (t.nw > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + t.group), "r"(t.nw * 32) : "memory");
  else __syncwarp();
}

// Whether v is non-zero on any lane of the group's warps; also a barrier.
__device__ __forceinline__ bool group_any(const Tile& t, uint32_t v) {
  if (t.nw == 1) return __any_sync(FULL_MASK, v != 0);
  uint32_t r;
  asm volatile(
      "{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.or.pred q, %2, %3, p; selp.u32 %0, 1, 0, q; }"
      : "=r"(r)
      : "r"(v), "r"(1 + t.group), "r"(t.nw * 32)
      : "memory");
  return r != 0;
}

// Eight columns' bits of plane k from four text words; bit 4 i + w of the
// result is column 8 w + i.
__device__ __forceinline__ uint32_t gather_plane(const uint32_t (&w)[4], int k) {
  uint32_t r = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t m = 0x11111111u << j;
    const uint32_t v = k >= j ? w[j] >> (k - j) : w[j] << (j - k);
    r |= v & m;
  }
  return r;
}

// The five text words of columns 32 k .. 32 k + 31 of this lane's candidate in
// group s (the fifth for windows that start inside a word).
__device__ __forceinline__ void load_text(const DevInputs& in, const WarpMem& w, int s, uint32_t k, int lane,
                                          uint32_t (&v)[5]) {
  const uint32_t nsh = w.nsh[32 * s + lane];
  const long long b = (long long)w.b0[32 * s + lane] + 4 * (long long)k;
#pragma unroll
  for (int j = 0; j < 5; ++j) v[j] = 0u;
  if (32 * k < (nsh & 0xFFFFu)) {
    if (b + 5 <= (long long)in.ref_words) {
      const uint32_t* p = in.ref + b;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = __ldg(p + j);
      if (nsh >> 16) v[4] = __ldg(p + 4);
    } else {
#pragma unroll
      for (int j = 0; j < 5; ++j) v[j] = ref_load(in.ref, b + j, in.ref_words);
    }
  }
}

// Those words of groups s0 .. s0 + N - 1 into the text ring, transposed from a
// candidate per lane to a column per lane.
template <int N>
__device__ __forceinline__ void slice_text(const WarpMem& w, int s0, uint32_t k, int lane, const uint32_t (&v)[N][5],
                                           uint4* __restrict__ ring) {
  uint32_t t01[2 * N], t2[N], some = 0;
#pragma unroll
  for (int b = 0; b < N; ++b) {
    const uint32_t sh = w.nsh[32 * (s0 + b) + lane] >> 16;
    uint32_t x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = __funnelshift_r(v[b][j], v[b][j + 1], sh);
    const uint32_t a0 = gather_plane(x, 0), a1 = gather_plane(x, 1), a2 = gather_plane(x, 2);
    // codes 5..7 act as A, code 4 (N) matches no base
    t01[2 * b] = a0 & ~a2;
    t01[2 * b + 1] = a1 & ~a2;
    t2[b] = a2 & ~(a1 | a0);
    some |= t2[b];
  }
  transpose32(t01, lane);
  if (__any_sync(FULL_MASK, some != 0)) transpose32(t2, lane);
  const uint32_t col = 32 * k + 8 * (lane & 3) + (lane >> 2);
#pragma unroll
  for (int b = 0; b < N; ++b) ring[64 * (s0 + b) + (col & 63)] = make_uint4(t01[2 * b], t01[2 * b + 1], t2[b], 0u);
}

// Columns 32 g .. 32 g + 31 of the last row in groups s0 .. s0 + N - 1: each
// lane scans its candidate's.
template <int N>
__device__ __forceinline__ void scan_columns(const WarpMem& w, int s0, uint32_t g, int lane,
                                             const uint2* __restrict__ out, uint32_t omask,
                                             const int2* __restrict__ lut) {
  uint32_t d[2 * N], sk[N], kmin[N];
#pragma unroll
  for (int b = 0; b < N; ++b) {
    const uint2 o = out[(omask + 1) * (s0 + b) + ((32 * g + lane) & omask)];
    d[2 * b] = o.x;
    d[2 * b + 1] = o.y;
  }
  transpose32(d, lane);
#pragma unroll
  for (int b = 0; b < N; ++b) {
    const int ci = 32 * (s0 + b) + lane;
    const uint32_t n = w.nsh[ci] & 0xFFFFu;
    // columns past the candidate's window only raise the score
    const uint32_t left = n > 32 * g ? n - 32 * g : 0u;
    const uint32_t in_window = left >= 32u ? FULL_MASK : (1u << left) - 1u;
    d[2 * b] |= ~in_window;
    d[2 * b + 1] &= in_window;
    sk[b] = w.sk[ci];
    kmin[b] = w.kmin[ci];
  }
  // four columns per table entry: their +1 bits in its low nibble, their -1
  // bits in the high one; a byte of `even` / `odd` per even / odd nibble
#pragma unroll
  for (int b = 0; b < N; ++b) {
    const uint32_t p = d[2 * b], q = d[2 * b + 1];
    d[2 * b] = (p & 0x0F0F0F0Fu) | ((q << 4) & 0xF0F0F0F0u);
    d[2 * b + 1] = ((p >> 4) & 0x0F0F0F0Fu) | (q & 0xF0F0F0F0u);
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
#pragma unroll
    for (int b = 0; b < N; ++b) {
      const int2 e = lut[__byte_perm(d[2 * b + (q & 1)], 0u, 0x4440 + (q >> 1))];
      kmin[b] = min(kmin[b], sk[b] + (uint32_t)e.x);
      sk[b] += (uint32_t)e.y;
    }
  }
#pragma unroll
  for (int b = 0; b < N; ++b) {
    w.sk[32 * (s0 + b) + lane] = sk[b];
    w.kmin[32 * (s0 + b) + lane] = kmin[b];
  }
}

// The columns of a tile whose candidates and rows are staged.
template <class K, int R, bool GEN>
__device__ __forceinline__ void run_columns(const DevInputs& in, const Tile& t, uint32_t n_max, uint32_t pm) {
  const int lane = threadIdx.x & 31;
  const int2* lut = reinterpret_cast<const int2*>(sl_smem);
  const int lg = K::kChain ? 5 : t.lg, lanes = 1 << lg;  // of the group, in this warp
  const int nseg = 32 >> lg;
  const int seg = lane >> lg, l = lane & (lanes - 1);
  const WarpMem w = warp_mem<K>(threadIdx.x >> 5);
  const uint32_t one = c_one, mone = c_mone;

  // With many rows Pv - Mv is kept instead of formed anew: 1,000-base reads 12.8
  // -> 12.5 ms per 660K candidates, 950 bases 12.0 -> 11.3 (no gain on fewer
  // rows, a loss on chains of warps).
  constexpr bool kKeepV = !K::kChain && R > 24;
  uint32_t q0[R], q1[R], q2[GEN ? R : 1], Pv[R], Mv[R], V[kKeepV ? R : 1];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int at = lane * K::kStride + i;
    q0[i] = w.buf[at];
    q1[i] = w.buf[32 * K::kStride + at];
    if (GEN) q2[i] = w.buf[64 * K::kStride + at];
    Pv[i] = 0xFFFFFFFFu;
    Mv[i] = 0u;
    if (kKeepV) V[i] = 0xFFFFFFFFu;
  }
  __syncwarp();
  // Rings: 64 text columns per group; 64 columns of the last row per group,
  // or 128 where the next warp reads them two blocks later.
  uint4* ring = reinterpret_cast<uint4*>(w.buf);
  uint2* out = reinterpret_cast<uint2*>(ring + 64 * K::kGroups);
  constexpr uint32_t omask = K::kRing - 1u;
  const uint2* below = nullptr;  // the last row of the warp below
  if (K::kChain && t.wg > 0) below = reinterpret_cast<const uint2*>(warp_mem<K>((threadIdx.x >> 5) - 1).buf) + 2 * 64 * K::kGroups;
  for (int s = 0; s < nseg; ++s) ring[64 * s + 32 + lane] = make_uint4(0u, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u);

  const uint32_t lmask = l == 0 ? 0u : 0xFFFFFFFFu;
  const bool last = l == lanes - 1, top = !K::kChain || t.wg == t.nw - 1;
  const uint32_t steps = n_max + (uint32_t)lanes - 1u;
  const uint32_t blocks = (steps + 31u) >> 5, groups = (n_max + 31u) >> 5;
  const uint4* text = ring + 64 * seg;
  uint2* mine = out + K::kRing * seg;
  uint32_t oP = 0u, oM = 0u;
  // Warp wg runs its block of columns two rounds after the warp below ran it.
  const uint32_t lag = K::kChain ? 2u * (uint32_t)t.wg : 0u;
  const uint32_t rounds = blocks + (K::kChain ? 2u * (uint32_t)(t.nw - 1) : 0u);
  auto scan = [&](uint32_t g) {
    if (K::kGroups == 1 || nseg == 1) {
      scan_columns<1>(w, 0, g, lane, out, omask, lut);
    } else {
      for (int s0 = 0; s0 < nseg; s0 += 2) scan_columns<2>(w, s0, g, lane, out, omask, lut);
    }
  };
  for (uint32_t r = 0; r < rounds; ++r) {
    const uint32_t k = r - lag;
    if (k < blocks) {
      if (K::kGroups == 1 || nseg == 1) {
        uint32_t v[1][5];
        load_text(in, w, 0, k, lane, v[0]);
        slice_text<1>(w, 0, k, lane, v, ring);
      } else {
        for (int s0 = 0; s0 < nseg; s0 += 2) {
          uint32_t v[2][5];
#pragma unroll
          for (int b = 0; b < 2; ++b) load_text(in, w, s0 + b, k, lane, v[b]);
          slice_text<2>(w, s0, k, lane, v, ring);
        }
      }
      __syncwarp();
      const uint32_t end = K::kChain ? 32u : min(32u, steps - 32u * k);
#pragma unroll 1
      for (uint32_t u = 0; u < end; ++u) {
        const uint32_t at = 32u * k + u;
        const uint4 tx = text[(at - (uint32_t)l) & 63u];
        uint32_t P = __shfl_up_sync(FULL_MASK, oP, 1) & lmask;
        uint32_t M = __shfl_up_sync(FULL_MASK, oM, 1) & lmask;
        if (K::kChain && below != nullptr) {
          const uint2 d = below[at & omask];
          P |= d.x & ~lmask;
          M |= d.y & ~lmask;
        }
        const uint32_t Pin = P, Min = M;
        uint32_t H = mad(M, mone, P);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          uint32_t x;
          if (GEN) {
            x = lop3<kA ^ kB>(q0[i], tx.x, tx.x);
            x = lop3<kA | (kB ^ kC)>(x, q2[i], tx.z);
          } else {
            x = lop3<(kA ^ kB) | kC>(q0[i], tx.x, tx.z);
          }
          x = lop3<kA | (kB ^ kC)>(x, q1[i], tx.y);
          const uint32_t N = lop3<kA & ~kB & ~kC>(x, Mv[i], M);
          const uint32_t m2 = lop3<kA & ~kB>(Pv[i], N, N);
          const uint32_t h2 = mad(kKeepV ? V[i] : mad(Mv[i], mone, Pv[i]), mone, N);
          const uint32_t p2 = mad(m2, one, h2);
          const uint32_t mv = lop3<kA & ~kB>(P, N, N);
          const uint32_t v2 = mad(H, mone, N), pv = mad(mv, one, v2);
          P = p2;
          M = m2;
          H = h2;
          Pv[i] = pv;
          Mv[i] = mv;
          if (kKeepV) V[i] = v2;
          if (i == 0) {  // candidates that skip this row pass the delta on
            P = lop3<(kA & kC) | (kB & ~kC)>(Pin, P, pm);
            M = lop3<(kA & kC) | (kB & ~kC)>(Min, M, pm);
            H = mad(M, mone, P);
          }
        }
        oP = P;
        oM = M;
        if (last) mine[(at - (uint32_t)(lanes - 1)) & omask] = make_uint2(P, M);
      }
      __syncwarp();
      if (top && k > 0 && k - 1 < groups) scan(k - 1);
    }
    group_barrier(t);
  }
  if (top) {
    for (uint32_t g = blocks - 1; g < groups; ++g) scan(g);
    for (int s = 0; s < nseg; ++s) {
      const int ci = 32 * s + lane;
      if (w.nsh[ci] & 0xFFFFu) finish(in, w.id[ci], w.kmin[ci], 0u, w.mm[ci] & 0xFFFFu, w.mm[ci] >> 16);
    }
  }
}

// run_columns of the tile's rows per lane, one of R, R + 1, .. (in steps of two
// above 32).
template <class K, bool GEN, int R>
__device__ __forceinline__ void run_rows(const DevInputs& in, const Tile& t, uint32_t n_max, uint32_t pm) {
  if (t.R == R) run_columns<K, R, GEN>(in, t, n_max, pm);
  else if constexpr (R < K::kHi) run_rows<K, GEN, (R < 32 ? R + 1 : R + 2)>(in, t, n_max, pm);
}

// A tile the bit planes cannot hold (a row with several bases, a query longer
// than the shape's rows): the word-parallel tile over its candidates, shared
// out among the group's warps.
template <class K>
__device__ __forceinline__ void run_words(const DevInputs& in, const Tile& t, const WarpMem& w, uint32_t m_max, int lane) {
  const uint32_t W = !K::kChain || m_max <= 4096u ? 4u : 16u;
  const uint32_t L = max(1u, (m_max + 32u * W - 1u) / (32u * W));
  const uint32_t per = 32u / L;
  for (uint32_t f = (uint32_t)t.wg * per; f < t.cnt; f += (uint32_t)t.nw * per) {
    const uint32_t cnt = min(per, t.cnt - f);
    if (W == 4u) process_tile<4, true, 1>(in, t.ids, t.first + f, cnt, (int)L, w.buf, lane);
    else if constexpr (K::kChain) process_tile<16, true, 1>(in, t.ids, t.first + f, cnt, (int)L, w.buf, lane);
  }
}

// Apart from the kernel in the chain class, whose column loops need every register:
// with the word-parallel tile in line, the loops of single row counts ran up to 13%
// slower (4,864 bases 4.62 -> 5.31 ms). Which row counts gain changes with whatever the
// kernel holds: against a kernel with loops for 8..16 rows and the tile in line, 130
// lengths take from 6% less (32 rows) to 6% more (19 rows), one 14%, 0.2% more in all;
// with the loops for 17 rows and more and the tile in line 1.2% more in all.
template <class K>
__device__ __noinline__ void run_words_apart(const DevInputs& in, const Tile& t, const WarpMem& w, uint32_t m_max,
                                             int lane) {
  run_words<K>(in, t, w, m_max, lane);
}

template <class K>
__device__ __forceinline__ void run_tile(const DevInputs& in, const Tile& t, int lane) {
  const int LL = 1 << t.lg;
  const int lw = K::kChain ? 5 : t.lg, lanes = 1 << lw, nseg = 32 >> lw;
  const int rows = LL * t.R;
  const WarpMem w = warp_mem<K>(threadIdx.x >> 5);

  // the tile's candidates, one per lane and group; all groups' loads at once
  uint32_t n_max = 0, m_max = 0;
  {
    constexpr int G = K::kGroups;
    uint32_t ids[G];
    Cand cd[G];
    uint2 q[G];
#pragma unroll
    for (int b = 0; b < G; ++b) {
      const uint32_t i = 32u * (uint32_t)b + (uint32_t)lane;
      ids[b] = t.ids && i < t.cnt ? __ldg(t.ids + t.first + i) : t.first + i;
    }
#pragma unroll
    for (int b = 0; b < G; ++b)
      if (32u * (uint32_t)b + (uint32_t)lane < t.cnt) cd[b] = in.cands[ids[b]];
      else cd[b].query = 0xFFFFFFFFu;
#pragma unroll
    for (int b = 0; b < G; ++b) q[b] = cd[b].query < in.num_queries ? __ldg(in.qinfo + cd[b].query) : make_uint2(0u, 0u);
#pragma unroll
    for (int b = 0; b < G; ++b) {
      if (b >= nseg) break;
      const uint32_t i = 32u * (uint32_t)b + (uint32_t)lane;
      uint32_t m = 0, mf = 0, n = 0, sh = 0, entry = 0;
      unsigned long long b0 = 0;
      if (i < t.cnt) {
        const uint32_t bad = check_query(in, cd[b].query, q[b]);
        const unsigned long long pos = cd[b].position;
        mf = q[b].y;
        m = in.prefix ? d_prefix_rows(mf, in.cutoff, in.prefix_mult) : mf;
        const uint32_t wb = d_window_bases(mf, in.distance);
        const bool valid = bad == 0u && pos < in.ref_size && (in.ref_size - pos) > (unsigned long long)wb;
        n = in.exact ? wb : 8u * d_window_words(wb);
        const bool fits = m >= t.row_min && m <= t.row_limit && n <= kMaxColumns;
        if (valid && m > 0 && fits) {
          b0 = pos >> 3;
          sh = in.exact ? 4u * (uint32_t)(pos & 7u) : 0u;
          entry = q[b].x;
          // the window's first 256 columns on their way to L2
          if (b0 + 31 < in.ref_words) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(in.ref + b0));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(in.ref + b0 + 31));
          }
        } else {
          if (t.wg == 0) {
            in.results[ids[b]] = (valid && m == 0) ? make_uint2(0u, 0u) : make_uint2(0u, kNoResult);
            if (bad) atomicOr(in.flags, bad);
            else if (valid && m > 0) atomicOr(in.flags, kFlagUnsupported);
          }
          n = 0;
          m = mf = 0;
        }
      }
      w.b0[i] = b0;
      w.id[i] = ids[b];
      w.mm[i] = m | (mf << 16);
      w.nsh[i] = n | (sh << 16);
      w.kmin[i] = entry;
      w.sk[i] = m << 16;
      n_max = max(n_max, n);
      m_max = max(m_max, m);
    }
  }
  n_max = __reduce_max_sync(FULL_MASK, n_max);
  m_max = __reduce_max_sync(FULL_MASK, m_max);
  __syncwarp();

  // The rows of lane gl of a group, as a word per candidate (bit i = row i of
  // the lane), then transposed to a word per row (bit c = candidate c).
  uint32_t pm = 0, gen = 0, several = m_max > (uint32_t)rows ? 1u : 0u;
  if (!several) {
#pragma unroll 2
    for (int blk = 0; blk < 32; ++blk) {
      const int ci = 32 * (blk >> lw) + lane;
      const int gl = 32 * t.wg + (blk & (lanes - 1));
      const uint32_t m = w.mm[ci] & 0xFFFFu, entry = w.kmin[ci];
      const int nw = (int)((m + 31u) >> 5);
      const int p = rows - (int)m;
      // p < LL: lanes 0..p-1 skip their row 0; longer paddings fill the bottom
      // rows with rows that match nothing (GEN)
      const bool spread = p < LL;
      const bool skip0 = spread && gl < p;
      const int off = gl * t.R - (spread ? min(gl + 1, p) : p);
      const uint32_t skips = __ballot_sync(FULL_MASK, skip0);
      if (lane == blk) pm = skips;
      for (int h = 0; 32 * h < (K::kHi > 32 ? t.R : 1); ++h) {
        // bits o .. o + 31 of the read, from words a and a + 1 (0 outside it)
        const int o = off + 32 * h, a = o >> 5;
        const uint32_t* lo = in.peq + (((long long)entry + (a >> 2)) * 20 + (a & 3));
        const uint32_t* hi = (a & 3) == 3 ? lo + 17 : lo + 1;
        const bool has_lo = a >= 0 && a < nw, has_hi = a >= -1 && a + 1 < nw;
        uint32_t v[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          const uint32_t x = has_lo ? __ldg(lo + 4 * c) : 0u, y = has_hi ? __ldg(hi + 4 * c) : 0u;
          v[c] = __funnelshift_r(x, y, o & 31);
        }
        const int count = t.R - 32 * h;
        uint32_t rows_in = count >= 32 ? FULL_MASK : (1u << count) - 1u;
        if (skip0 && h == 0) rows_in &= ~1u;
        if (m == 0) rows_in = 0u;
        const uint32_t gt = v[2] | v[3], any = v[0] | v[1] | gt | v[4];
        several |= ((v[0] & (v[1] | gt | v[4])) | (v[1] & (gt | v[4])) | (v[2] & v[3]) | (gt & v[4])) & rows_in;
        const uint32_t none = rows_in & ~any;
        const uint32_t odd = (v[4] & rows_in) | none;
        gen |= odd;
        uint32_t planes[2] = {v[1] | v[3] | none, gt}, third[1] = {odd};
        transpose32(planes, lane);
        if (__any_sync(FULL_MASK, odd != 0)) transpose32(third, lane);
        if (lane < count) {
          uint32_t* dst = w.buf + blk * K::kStride + 32 * h + lane;
          dst[0] = planes[0];
          dst[32 * K::kStride] = planes[1];
          dst[64 * K::kStride] = third[0];
        }
      }
    }
  }
  if (group_any(t, several)) {
    __syncwarp();
    if constexpr (K::kChain) run_words_apart<K>(in, t, w, m_max, lane);
    else run_words<K>(in, t, w, m_max, lane);
    group_barrier(t);
    return;
  }
  for (int s = 0; s < nseg; ++s) w.kmin[32 * s + lane] = w.sk[32 * s + lane];  // (m, column 0) before any column
  __syncwarp();
  if (n_max == 0) return;  // nothing to do: the same on every warp of the group
  if (__any_sync(FULL_MASK, gen != 0)) run_rows<K, true, K::kLo>(in, t, n_max, pm);
  else run_rows<K, false, K::kLo>(in, t, n_max, pm);
  __syncwarp();
}

// A block's warps (groups of nw warps in a chain class) take tiles from the
// counters of the class's shapes, in the plan's order: the longest tiles
// first. The first tile of every group of the first shape is its place in the
// grid. With st == nullptr there is one shape, candidates 0..count-1.
template <class K>
__global__ void __launch_bounds__(K::kThreads, K::kBlocks)
    k_sliced(const __grid_constant__ DevInputs in, const uint32_t* __restrict__ ids, BucketState* st,
             const __grid_constant__ PlanShapes plan, uint32_t c0, uint32_t c1, uint32_t count,
             uint32_t* __restrict__ next) {
  __shared__ uint32_t s_tile[K::kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int2* lut = reinterpret_cast<int2*>(sl_smem);
  for (int x = threadIdx.x; x < 256; x += K::kThreads) {
    // four columns' +1 bits (low nibble) and -1 bits (high nibble)
    int sum = 0, least = 127, at = 0;
    for (int b = 0; b < 4; ++b) {
      sum += ((x >> b) & 1) - ((x >> (4 + b)) & 1);
      if (sum < least) {
        least = sum;
        at = b;
      }
    }
    lut[x] = make_int2((int)((uint32_t)least << 16) + at, (int)((uint32_t)sum << 16) + 4);
  }
  __syncthreads();
  uint32_t blocks = gridDim.x;
  if constexpr (!K::kChain) {
    // Only as many blocks as the class has tiles for stay, so that those of the
    // other classes find room beside them (300K reads of 35..301 bases, three
    // classes of one round or less: 0.49 -> 0.43 ms).
    __shared__ uint32_t s_tiles;
    if (threadIdx.x == 0) s_tiles = 0u;
    __syncthreads();
    uint32_t tiles = 0;
    for (uint32_t c = c0 + threadIdx.x; c < c1; c += K::kThreads) {
      const Shape s = plan.shape[c];
      const uint32_t per = 32u << (5 - s.L);
      if (K::has(s)) tiles += ((st != nullptr ? st->count[c] : count) + per - 1u) / per;
    }
    if (tiles) atomicAdd(&s_tiles, tiles);
    __syncthreads();
    blocks = min(blocks, (s_tiles + K::kWarps - 1u) / K::kWarps);
    if (blockIdx.x >= blocks) return;
  }
  int nw_before = 0;
  bool placed = false;
  Tile t;
  t.ids = ids;
  for (uint32_t c = c0; c < c1; ++c) {
    const Shape s = plan.shape[c];
    if (!K::has(s)) continue;
    uint32_t f0 = 0;
    if (st != nullptr) {
      count = st->count[c];
      f0 = st->first[c];
      next = &st->next[c];
    }
    if (count == 0) continue;
    t.R = s.W;
    t.lg = s.L;
    t.row_min = plan.row_min;
    t.row_limit = min(plan.row_limit ? plan.row_limit : (uint32_t)s.W << s.L,
                      K::kChain ? kSlicedChainWordRows : kSlicedWordRows);  // run_words' tile
    t.nw = K::kChain ? 1 << (s.L - 5) : 1;
    t.wg = warp & (t.nw - 1);
    t.group = warp / t.nw;
    const uint32_t per = s.L < 5 ? 32u << (5 - s.L) : 32u;
    const uint32_t tiles = (count + per - 1u) / per;
    const uint32_t ngroups = (uint32_t)(K::kWarps / t.nw);
    if (K::kChain) {
      if (t.nw != nw_before && nw_before != 0) __syncthreads();  // the groups' shares of shared memory change hands
      nw_before = t.nw;
    }
    const uint32_t placed_tiles = placed ? 0u : blocks * ngroups;
    bool place = !placed;
    placed = true;
    while (true) {
      uint32_t i = 0;
      if (place) {
        i = blockIdx.x * ngroups + (uint32_t)t.group;
        place = false;
      } else {
        if (lane == 0 && t.wg == 0) i = placed_tiles + atomicAdd(next, 1u);
        if (!K::kChain) {
          i = __shfl_sync(FULL_MASK, i, 0);
        } else {
          if (lane == 0 && t.wg == 0) s_tile[t.group] = i;
          group_barrier(t);
          i = s_tile[t.group];
        }
      }
      if (i >= tiles) {
        if (K::kChain) group_barrier(t);  // every warp has read s_tile
        break;
      }
      t.first = f0 + i * per;
      t.cnt = min(per, count - i * per);
      run_tile<K>(in, t, lane);
      if (K::kChain) group_barrier(t);
    }
  }
}

template <class K>
cudaError_t launch_class(const DevInputs& in, const uint32_t* d_ids, const PlanShapes& plan, BucketState* d_state,
                         uint32_t c0, uint32_t c1, uint32_t count, uint32_t* d_next, cudaStream_t s, int num_sms) {
  cudaError_t e = cudaFuncSetAttribute((const void*)k_sliced<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)K::kSmemBytes);
  if (e != cudaSuccess) return e;
  // at most a block per group of 32 candidates
  const uint32_t most = (in.num_cands + 31u) / 32u, full = (uint32_t)(num_sms * K::kBlocks);
  const uint32_t grid = most < full ? (most > 0 ? most : 1u) : full;
  k_sliced<K><<<grid, K::kThreads, K::kSmemBytes, s>>>(in, d_ids, d_state, plan, c0, c1, count, d_next);
  return cudaGetLastError();
}

// Defines the entry of a class (declared in myers_internal.h). Each class is
// compiled in a file of its own: together they take minutes.
#define MYERS_SLICED_CLASS(K, INDEX)                                                                                 \
  template <>                                                                                                        \
  cudaError_t launch_sliced_class<INDEX>(const DevInputs& in, const uint32_t* d_ids, const PlanShapes& plan,          \
                                         BucketState* d_state, uint32_t c0, uint32_t c1, uint32_t count,             \
                                         uint32_t* d_next, cudaStream_t s, int num_sms) {                            \
    return launch_class<K>(in, d_ids, plan, d_state, c0, c1, count, d_next, s, num_sms);                             \
  }                                                                                                                  \
  template <>                                                                                                        \
  const void* sliced_class_kernel<INDEX>() {                                                                         \
    return (const void*)k_sliced<K>;                                                                                 \
  }

}  // namespace myers
