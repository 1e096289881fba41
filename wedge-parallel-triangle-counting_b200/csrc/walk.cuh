// walk.cuh -- the default count of whole graphs: every edge (v, w) of the
// oriented CSR closes its wedges (v; w, u) -- u in the tail of row v behind w
// -- by one of three ways, chosen by w's row and v's place:
//
//   v in the dense core  row ANDs (k_core_count, count_kernels.cuh)
//   d+(w) <= 48          the edge's own thread intersects the tail with the
//                        short row of w, four columns of each at a time, or
//                        a warp streams the short rows through a set of its
//                        rows (k_edge_merge)
//   longer rows          the column walk: the edges are sorted by w, a block
//                        builds N+(w) once in shared memory and the tails of
//                        all rows v stream through it (k_walk_count)
//
// The wedge-check kernel (count_kernels.cuh), which serves the other calls,
// looks every u up in a set of N+(w): one random 32-byte sector of L2 or DRAM
// for each wedge. Here a wedge costs the four bytes of its u, read with the
// rest of the tail, and a compare or a shared-memory lookup.
//
// In the walk, columns of the last 65,536 vertices (the window: most columns
// of a graph with hubs) and the others are kept apart, so that the window's
// set is a plain bit row: the i-th long row stands for two middle vertices,
// 2i + 1 with its window columns and 2i with the rest, and a tail that has
// both is two entries.
//
//   k_edge_vertices  row checks, W, the longest row, core sizing, and the
//                    numbers of the long rows
//   k_walk_split     where a row's window columns start, and the wedges of
//                    rows with several hash sets
//   k_edge_merge     the short rows' edges counted, the others' entries:
//                    middle vertex, the tail's first column index and its
//                    length in 64 bits
//   radix sort       by middle vertex (primitives.cuh)
//   k_walk_starts    the first entry of every middle vertex
//   k_walk_plan      work items: a vertex, a piece of its entries and, with
//                    several hash sets, a group of them
//   k_walk_count     a block per item: the bit row, or a hash set
//   k_small_count    a small graph's whole count
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "count_kernels.cuh"
#include "primitives.cuh"
#include "readback.cuh"

namespace wetric {
namespace {

constexpr uint32_t kWalkWindow = 65536;

// Fields of an entry, low to high: tail length, first column index, middle
// vertex.
struct WalkBits {
  uint32_t w, start, len;
  __host__ __device__ uint32_t shift() const { return start + len; }
};

constexpr uint32_t kWalkBlock = 256;
constexpr uint32_t kWalkEmpty = 0xFFFFFFFFu;
constexpr uint32_t kWalkShort = 0xFFFFFFFFu;  // number of a row that is not long
constexpr uint32_t kWalkShortCols = 48;       // columns of a short row at most
constexpr uint32_t kMergeBlock = 128;
constexpr uint32_t kMergeTile = 512;          // edges per warp at most
constexpr uint32_t kRowSetCols = 64;          // columns in a warp's set at most
constexpr uint32_t kRowSetSlots = 1024;
constexpr uint32_t kRowSetFill = 24;          // edges of whole rows that fill a warp
constexpr uint32_t kRowSetRows = 4;
constexpr uint32_t kRowSetTries = 8;
constexpr uint32_t kRowSetMin = 8;            // edges that are worth a set
constexpr uint32_t kRowSetLong = 64;          // columns of a row w streamed at most
constexpr uint32_t kSearchOver = 2048;        // columns that are searched for few others
constexpr uint32_t kSearchRatio = 16;
constexpr uint32_t kMergeStage = 128;         // entries a warp gathers (64 or more)
constexpr uint32_t kWalkBig = 64;             // entries from which a block takes a vertex
constexpr uint32_t kWalkBigCols = 128;        // or columns
constexpr uint32_t kWalkPiece = 2048;         // entries per item of a block
constexpr uint32_t kWalkPer = 4;              // entries per thread streamed at once
constexpr uint32_t kWalkBigBlock = 128, kWalkSmallBlock = 32;
constexpr int kWalkBigBlocks = 10, kWalkSmallBlocks = 28;  // per SM
constexpr uint32_t kWalkSmallSlots = 512;
constexpr uint32_t kWalkSetCols = 1024;  // columns per hash set
constexpr uint32_t kWalkSetGroups = 32;  // items that share the sets of a row at most (2^k)
constexpr uint32_t kWalkSetPiece = 512;  // entries per item of a row of several sets
constexpr uint32_t kWalkSetSlots = 2048;
constexpr int kWalkCarveout = 70;  // percent of an SM's memory that is shared

// Inclusive scan over the warp.
__device__ __forceinline__ uint32_t walk_scan(uint32_t x, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  return x;
}

// The warp's hits added to *to, in 64 bits: a block that stays with one dense
// graph of a batch can pass 2^32 (a clique of 60,000: 6e9 a warp).
__device__ __forceinline__ void walk_add_hits(unsigned long long *to, unsigned long long hits,
                                              uint32_t lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
  if (lane == 0 && hits) atomicAdd(to, hits);
}

// Core lengths to size up, at most n each.
struct EdgeCores {
  uint32_t len[kCoreNumCandidates];
  uint32_t count;
};

// The graphs of a batch: graph g owns rows [base[g], base[g + 1]) of the
// disjoint union and counts into counts[g].
struct WalkGroups {
  const uint64_t *base = nullptr;
  uint32_t G = 0;
  unsigned long long *counts = nullptr;
};
__device__ __forceinline__ uint32_t walk_group(const WalkGroups &gr, uint64_t row) {
  uint32_t lo = 0, len = gr.G;
  while (len > 1) {
    const uint32_t h = len >> 1;
    if (__ldg(gr.base + lo + h) <= row) lo += h;
    len -= h;
  }
  return lo;
}
// First window column of graph g's rows.
__device__ __forceinline__ uint32_t walk_window(const WalkGroups &gr, uint32_t g) {
  const uint64_t b = __ldg(gr.base + g), e = __ldg(gr.base + g + 1);
  return (uint32_t)(e - b > kWalkWindow ? e - kWalkWindow : b);
}

// Totals of the rows: [0] W, [1] longest row, [2] rows with wedges, [3] long
// rows, [4] their wedges, then per core candidate its wedges, AND words
// (k_core_plan) and rows with wedges.
constexpr uint32_t kEdgeCand = 5;
constexpr uint32_t kEdgeTotals = kEdgeCand + 3 * kCoreNumCandidates;
// Rows of more than kWalkShortCols columns among m columns at most, when the
// offsets are monotone: the room for long_rows. The kernels that number the
// long rows are also the ones that check the offsets, and rows that overlap
// (0, m, 0, m, ...) can be long in any number, so ids past the room are
// dropped and raise kDevRowPtrRange.
__host__ __device__ inline uint64_t long_rows_room(uint64_t m) {
  return m / (kWalkShortCols + 1) + 1;
}
template <typename Off>
__global__ void __launch_bounds__(kWalkBlock)
    k_edge_vertices(const Off *__restrict__ rp, uint64_t n, uint64_t m,
                    const __grid_constant__ EdgeCores cores, unsigned long long *__restrict__ totals, uint32_t *__restrict__ number,
                    uint32_t *__restrict__ long_rows, uint32_t *err) {
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long W = 0, rows = 0, longest = 0, long_w = 0;
  unsigned long long plan[3 * kCoreNumCandidates] = {};
  const uint64_t top = cores.count ? cores.len[0] : 0u;  // the longest
  bool in_top = false;
  for (uint64_t v0 = (uint64_t)blockIdx.x * kWalkBlock + threadIdx.x - lane; v0 < n;
       v0 += (uint64_t)gridDim.x * kWalkBlock) {
    const uint64_t v = v0 + lane;
    uint64_t d = 0;
    if (v < n) {
      const uint64_t b = ld_off(rp, v), e = ld_off(rp, v + 1);
      if (e < b || e > m)
        atomicCAS(err, 0u, (uint32_t)kDevRowPtrRange);
      else
        d = e - b;
    }
    const unsigned long long w = d >= 2 ? d * (d - 1) / 2 : 0;
    W += w;
    rows += d >= 2;
    longest = longest > d ? longest : d;
    if (v < n && v >= n - top) {
      in_top = true;
#pragma unroll
      for (uint32_t c = 0; c < kCoreNumCandidates; ++c) {
        const uint64_t hc = c < cores.count ? cores.len[c] : 0u;
        if (v >= n - hc) {
          plan[3 * c] += w;
          plan[3 * c + 1] += d * (hc - (v - (n - hc))) / 64 + d;
          plan[3 * c + 2] += d >= 2;
        }
      }
    }
    if (number) {
      const bool is_long = d > kWalkShortCols;
      const uint32_t mask = __ballot_sync(0xffffffffu, is_long);
      uint32_t id = 0;
      if (mask && lane == 0) id = (uint32_t)atomicAdd(totals + 3, (unsigned long long)__popc(mask));
      id = __shfl_sync(0xffffffffu, id, 0) + __popc(mask & ((1u << lane) - 1u));
      if (v < n) number[v] = is_long ? id : kWalkShort;
      if (is_long) {
        if (id < long_rows_room(m))
          long_rows[id] = (uint32_t)v;
        else
          atomicCAS(err, 0u, (uint32_t)kDevRowPtrRange);
        long_w += w;
      }
    }
  }
  __shared__ unsigned long long s_sum[4], s_plan[3 * kCoreNumCandidates];
  if (threadIdx.x < 4) s_sum[threadIdx.x] = 0;
  if (threadIdx.x < 3 * kCoreNumCandidates) s_plan[threadIdx.x] = 0;
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) {
    W += __shfl_down_sync(0xffffffffu, W, o);
    rows += __shfl_down_sync(0xffffffffu, rows, o);
    long_w += __shfl_down_sync(0xffffffffu, long_w, o);
    const unsigned long long x = __shfl_down_sync(0xffffffffu, longest, o);
    longest = longest > x ? longest : x;
  }
  if (lane == 0) {
    atomicAdd(&s_sum[3], long_w);
    atomicAdd(&s_sum[0], W);
    atomicMax(&s_sum[1], longest);
    atomicAdd(&s_sum[2], rows);
  }
  if (__any_sync(0xffffffffu, in_top)) {
#pragma unroll
    for (uint32_t c = 0; c < 3 * kCoreNumCandidates; ++c) {
      unsigned long long x = plan[c];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0 && x) atomicAdd(&s_plan[c], x);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_sum[0]) atomicAdd(totals, s_sum[0]);
    atomicMax(totals + 1, s_sum[1]);
    if (s_sum[2]) atomicAdd(totals + 2, s_sum[2]);
    if (s_sum[3]) atomicAdd(totals + 4, s_sum[3]);
  }
  if (threadIdx.x < 3 * kCoreNumCandidates && s_plan[threadIdx.x])
    atomicAdd(totals + kEdgeCand + threadIdx.x, s_plan[threadIdx.x]);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    if (ld_off(rp, 0) != 0 || ld_off(rp, n) != m) atomicCAS(err, 0u, (uint32_t)kDevRowPtrRange);
}

// The rows with more than kWalkSetCols columns outside the window, which take
// several hash sets: their wedges there, columns there and number, and the
// blocks that are through with them. At most min(wedges, columns * rows) of a
// graph's wedges have their tail on one such row and their middle vertex on
// another, and such a wedge is looked up once for each set of that vertex, at
// most columns^2 / kWalkSetCols times in all; with more than a tenth (`most`) of
// those below the core, or a third as many lookups, it is not walked. Half full sets cost several tries a column and the tails stream
// once for each set, where a bit row costs one lookup. In an order by degree
// the columns of long rows lie in the window, and a batch, always in that
// order, does without this; in another order they need not. Walk / wedge checks
// in ms and that share: R-MAT scale 20 in id order 73 / 57 (0.71), in random
// order 31 / 27 (0.53), Chung-Lu 300,000 vertices, mean degree 20, exponent
// 2.2 5.9 / 4.3 (0.13), in random order 2.2 / 1.9 (0.02), 1,000,000, 40, 2.8
// 5.8 / 7.6 (0.25), 3.8 / 5.0 (0.06); dense parts of 3,000 vertices 9 / 6
// (0.82); skewed draws in id order 4.5 / 13 (0.01); Erdos-Renyi 150,000, 1300
// 36 / 127 (0); four hubs of 200,000 columns, all wedges theirs, 1.2 / 180 (0).
// With the lookups per wedge: 300 hubs in front of 300,000 vertices with 12
// columns to them 28 / 12 (0.36), of 1,000,000 354 / 130 (0.51); in random
// order 48 / 157 (0.33); Chung-Lu 2,000,000, 8, 2.1 13 / 14 (0.27).
struct WalkFar {
  unsigned long long wedges, columns, rows, blocks;
  __host__ __device__ bool past(unsigned long long most) const {
    return (wedges > most && columns * rows > most) ||
           columns / kWalkSetCols * columns > most / 3 * 10;
  }
};
inline uint64_t walk_most_far(uint64_t wedges) { return wedges / 10; }

// split[v] = index of row v's first window column (rows are sorted), rows
// [lo, hi), and their part of *far; *stop is set when it is past `most`.
// kBatch: of the row's own graph, and no *far.
template <bool kBatch>
__global__ void __launch_bounds__(kWalkBlock)
    k_walk_split(const uint32_t *__restrict__ rp, const uint32_t *__restrict__ ci, uint64_t n,
                 uint64_t lo_row, uint64_t hi_row, uint32_t *__restrict__ split,
                 const WalkGroups groups, WalkFar *far, unsigned long long most,
                 uint32_t *__restrict__ stop) {
  unsigned long long wedges = 0, columns = 0;
  uint32_t rows = 0;
  uint32_t t0 = n > kWalkWindow ? (uint32_t)(n - kWalkWindow) : 0u;
  for (uint64_t v = lo_row + (uint64_t)blockIdx.x * kWalkBlock + threadIdx.x; v < hi_row;
       v += (uint64_t)gridDim.x * kWalkBlock) {
    if (kBatch) t0 = walk_window(groups, walk_group(groups, v));
    const uint32_t begin = rp[v];
    uint32_t lo = begin, hi = rp[v + 1];
    if (v >= t0) hi = lo;  // every column is above its row
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (__ldg(ci + mid) >= t0) hi = mid;
      else lo = mid + 1;
    }
    split[v] = lo;
    const unsigned long long d = lo - begin;
    if (!kBatch && d > kWalkSetCols) {
      wedges += d * (d - 1) / 2;
      columns += d;
      ++rows;
    }
  }
  if (kBatch) return;
  if (rows) {  // few threads have any
    atomicAdd(&far->wedges, wedges);
    atomicAdd(&far->columns, columns);
    atomicAdd(&far->rows, (unsigned long long)rows);
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // the last block has all of them
    __threadfence();
    uint32_t *blocks = reinterpret_cast<uint32_t *>(&far->blocks);
    if (atomicInc(blocks, gridDim.x - 1) == gridDim.x - 1) {
      __threadfence();
      const volatile WalkFar *all = far;
      if (WalkFar{all->wedges, all->columns, all->rows, 0}.past(most)) *stop = 1;
    }
  }
}

// start[x] = the first of the sorted entries of middle vertex x or more, x in
// [0, n].
// A lane fills a gap of up to 8 vertices, the warp a longer one.
__global__ void __launch_bounds__(kWalkBlock)
    k_walk_starts(const uint64_t *__restrict__ keys, uint32_t m, uint32_t n, uint32_t shift,
                  uint32_t *__restrict__ start, const uint32_t *__restrict__ err) {
  if (*err != kDevOk) return;  // the sort may have run out
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * kWalkBlock;
  const uint64_t gid = (uint64_t)blockIdx.x * kWalkBlock + threadIdx.x;
  const uint64_t first = keys[0] >> shift, end = keys[m - 1] >> shift;
  for (uint64_t w = gid; w <= first && w <= n; w += stride) start[w] = 0;
  for (uint64_t w = end + 1 + gid; w <= n; w += stride) start[w] = m;
  for (uint64_t i0 = gid - lane; i0 < m; i0 += stride) {
    const uint64_t i = i0 + lane;
    uint32_t w = 0, prev = 0;
    if (i < m) {
      w = (uint32_t)(keys[i] >> shift);
      prev = i ? (uint32_t)(keys[i - 1] >> shift) : w;
      if (w > n) w = n;
      if (prev > n) prev = n;
    }
    const bool wide = w - prev > 8u;
    if (!wide)
      for (uint32_t r = prev; r < w; ++r) start[r + 1] = (uint32_t)i;
    for (uint32_t mask = __ballot_sync(0xffffffffu, wide); mask; mask &= mask - 1) {
      const int l = __ffs(mask) - 1;
      const uint32_t from = __shfl_sync(0xffffffffu, prev, l), to = __shfl_sync(0xffffffffu, w, l);
      for (uint32_t r = from + 1 + lane; r <= to; r += 32) start[r] = (uint32_t)(i0 + l);
    }
  }
}

// The set columns of middle vertex x: its row's window columns or the rest.
__device__ __forceinline__ uint2 walk_set(const uint32_t *__restrict__ rp,
                                          const uint32_t *__restrict__ split,
                                          const uint32_t *__restrict__ long_rows, uint32_t x) {
  const uint32_t w = __ldg(long_rows + (x >> 1)), s = __ldg(split + w);
  return x & 1 ? make_uint2(s, __ldg(rp + w + 1)) : make_uint2(__ldg(rp + w), s);
}

// A row of several hash sets is shared out by entries and by sets: a hub's, with
// a set for each 1,024 of its columns outside the window, was one block's
// for 2,048 long tails at a time, and the rest of the device waited for it
// (Chung-Lu in random order, as above, 5.0 ms; 1,000,000, 20, 2.4 11.2, now
// 4.3; R-MAT scale 20 in id order 271). The kernel has a form without it (R-MAT
// scale 22 5.88 ms, 5.97 with it), taken when no row has several sets.
// An item's word: its piece of the entries (of kWalkSetPiece when the top bit
// is set), its group of sets.
constexpr uint32_t kWalkSeveral = 1u << 31, kWalkGroupShift = 24;
__device__ __forceinline__ bool walk_several(uint32_t x, uint32_t d) {
  return !(x & 1) && d > kWalkSetCols;
}
// Columns of a group: a multiple of kWalkSetCols, kWalkSetGroups of them or
// fewer make d.
__device__ __forceinline__ uint32_t walk_group_cols(uint32_t d) {
  return (d + kWalkSetGroups * kWalkSetCols - 1) / (kWalkSetGroups * kWalkSetCols) * kWalkSetCols;
}
// Items of the big blocks at most, with `cap` entries and m columns.
inline uint64_t walk_most_items(uint64_t cap, uint64_t m, bool share_sets) {
  return cap / kWalkPiece + cap / kWalkBig + m / kWalkBigCols + 1 +
         (share_sets ? kWalkSetGroups * (cap / kWalkSetPiece + m / kWalkSetCols + 1) : 0);
}

// The work items over the x_end middle vertices: counts[0] shares of those
// with more than kWalkBig entries or kWalkBigCols columns, counts[1] of the
// others (whole).
__global__ void __launch_bounds__(kWalkBlock)
    k_walk_plan(const uint32_t *__restrict__ rp, const uint32_t *__restrict__ split,
                const uint32_t *__restrict__ long_rows, const uint32_t *__restrict__ start,
                uint32_t x_end, uint2 *__restrict__ big, uint2 *__restrict__ small,
                uint32_t *__restrict__ counts, bool share_sets,
                const uint32_t *__restrict__ err) {
  if (*err != kDevOk) return;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * kWalkBlock;
  for (uint64_t x0 = (uint64_t)blockIdx.x * kWalkBlock + threadIdx.x - lane; x0 < x_end;
       x0 += stride) {
    const uint64_t x = x0 + lane;
    const uint32_t E = x < x_end ? start[x + 1] - start[x] : 0u;
    bool few = false;
    uint32_t groups = 1, piece = kWalkPiece;
    if (E && (E <= kWalkBig || (share_sets && !(x & 1)))) {
      const uint2 set = walk_set(rp, split, long_rows, (uint32_t)x);
      const uint32_t d = set.y - set.x;
      few = E <= kWalkBig && d <= kWalkBigCols;
      if (share_sets && walk_several((uint32_t)x, d)) {
        groups = (d + walk_group_cols(d) - 1) / walk_group_cols(d);
        piece = kWalkSetPiece;
      }
    }
    const uint32_t each = E && !few ? (E + piece - 1) / piece : 0u, pieces = groups * each;
    const uint32_t incl = walk_scan(pieces, lane);
    const uint32_t sm = __ballot_sync(0xffffffffu, few);
    const uint32_t sum = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t add = lane == 0 ? sum : __popc(sm);
    uint32_t got = 0;
    if (lane < 2 && add) got = atomicAdd(counts + lane, add);
    const uint32_t base = __shfl_sync(0xffffffffu, got, 0) + incl - pieces;
    const uint32_t at = __shfl_sync(0xffffffffu, got, 1) + __popc(sm & ((1u << lane) - 1u));
    for (uint32_t p = 0, g = 0; g < groups; ++g)
      for (uint32_t q = 0; q < each; ++q, ++p)
        big[base + p] = make_uint2(
            (uint32_t)x, piece == kWalkPiece ? q : q | g << kWalkGroupShift | kWalkSeveral);
    if (few) small[at] = make_uint2((uint32_t)x, 0u);
  }
}

// The columns as the streams read them: in 32-byte sectors, whole ones by
// one load, those that stick out of the array by single loads. `mis` is the
// column array's offset in its first sector; indices carry it.
struct WalkColumns {
  const uint32_t *base;  // 32-byte aligned, mis columns before the array
  uint32_t mis, end;     // columns [mis, end) exist (end <= 2^32 - 8)
};
inline WalkColumns walk_columns(const uint32_t *ci, uint64_t m) {
  WalkColumns c;
  c.mis = (uint32_t)((reinterpret_cast<uintptr_t>(ci) & 31) / 4);
  c.base = ci - c.mis;
  c.end = (uint32_t)(m + c.mis);
  return c;
}

// The sector at (mis-carrying) index a; where it sticks out of the array,
// only the columns of [lo, hi).
__device__ __forceinline__ void walk_sector(const WalkColumns &cols, uint32_t a, uint32_t lo,
                                            uint32_t hi, uint32_t (&x)[8]) {
  if (a >= cols.mis && a + 8 <= cols.end) {
    const Bucket b = ld_bucket(cols.base + a);
    x[0] = b.s0, x[1] = b.s1, x[2] = b.s2, x[3] = b.s3;
    x[4] = b.s4, x[5] = b.s5, x[6] = b.s6, x[7] = b.s7;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = a + j >= lo && a + j < hi ? __ldg(cols.base + a + j) : 0u;
  }
}

// Half a sector, likewise.
__device__ __forceinline__ void walk_half(const WalkColumns &cols, uint32_t a, uint32_t lo,
                                          uint32_t hi, uint32_t (&x)[4]) {
  if (a >= cols.mis && a + 4 <= cols.end) {
    const uint4 b = __ldg(reinterpret_cast<const uint4 *>(cols.base + a));
    x[0] = b.x, x[1] = b.y, x[2] = b.z, x[3] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = a + j >= lo && a + j < hi ? __ldg(cols.base + a + j) : 0u;
  }
}

// |[t0, t1) & [s0, s1)| where the second is much shorter: each of its columns
// by bisection of what the ones before it left of the first.
__device__ __forceinline__ uint32_t search_rows(const WalkColumns &cols, uint32_t t0, uint32_t t1,
                                                uint32_t s0, uint32_t s1) {
  uint32_t hits = 0;
  for (; s0 < s1 && t0 < t1; ++s0) {
    const uint32_t x = __ldg(cols.base + s0);
    uint32_t len = t1 - t0;
    while (len > 0) {
      const uint32_t half = len >> 1;
      const bool below = __ldg(cols.base + t0 + half) < x;
      t0 = below ? t0 + half + 1 : t0;
      len = below ? len - half - 1 : half;
    }
    hits += t0 < t1 && __ldg(cols.base + t0) == x;
  }
  return hits;
}

// |[t0, t1) & [s0, s1)| of the column array (both sorted, indices with mis,
// neither empty), four columns of each at a time: all pairs of them, then
// the four with the smaller last column move on. (Eight at a time: fewer
// loads, four times the pairs; Erdos-Renyi, 13.3M edges: 670 us against
// 551.) kSearch: more than kSearchOver columns against less than a sixteenth
// of them are searched instead, which only rows of a hub have that comes
// early in the order (a graph's own order by degree keeps rows short). One
// thread merged such a row with each of its short ones: 262,144 vertices in
// id order, skewed, 53.8 ms a count, by search 7.5 (wedge checks 13.2); four
// hubs of 200,000 columns 134 and 1.2 (180). Limits of 240 to 2,048 differ by
// 2%. The kernels have a form without it, 1% faster on short rows (a batch of
// 96 graphs 7.71 ms, 7.79 with it).
struct MergeTask {
  uint32_t t0, t1, s0, s1;
};
template <bool kSearch>
__device__ __forceinline__ uint32_t merge_rows(const WalkColumns &cols, const MergeTask &task) {
  const uint32_t t0 = task.t0, t1 = task.t1, s0 = task.s0, s1 = task.s1;
  if (kSearch && max(t1 - t0, s1 - s0) > kSearchOver) {
    if (t1 - t0 > kSearchRatio * (s1 - s0)) return search_rows(cols, t0, t1, s0, s1);
    if (s1 - s0 > kSearchRatio * (t1 - t0)) return search_rows(cols, s0, s1, t0, t1);
  }
  const uint32_t t_last = __ldg(cols.base + t1 - 1), s_last = __ldg(cols.base + s1 - 1);
  uint32_t a = t0 & ~3u, b = s0 & ~3u, hits = 0;
  uint32_t x[4], y[4];
  walk_half(cols, a, t0, t1, x);
  walk_half(cols, b, s0, s1, y);
  uint32_t xm = a + 4 < t1 ? x[3] : t_last, ym = b + 4 < s1 ? y[3] : s_last;
#pragma unroll
  for (int j = 0; j < 4; ++j) {  // columns that are not the rows' match nothing
    if (a + j < t0 || a + j >= t1) x[j] = 0xFFFFFFFFu;
    if (b + j < s0 || b + j >= s1) y[j] = 0xFFFFFFFEu;
  }
  for (;;) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      hits += x[i] == y[0] || x[i] == y[1] || x[i] == y[2] || x[i] == y[3];
    const bool tail = xm <= ym;
    const uint32_t p = (tail ? a : b) + 4, end = tail ? t1 : s1;
    if (p >= end) break;
    uint32_t z[4];
    walk_half(cols, p, p, end, z);
    const uint32_t zm = p + 4 < end ? z[3] : tail ? t_last : s_last;
    const uint32_t none = tail ? 0xFFFFFFFFu : 0xFFFFFFFEu;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t c = p + j < end ? z[j] : none;
      x[j] = tail ? c : x[j];
      y[j] = tail ? y[j] : c;
    }
    if (tail) a = p, xm = zm;
    else b = p, ym = zm;
  }
  return hits;
}

// A set of (row, column) pairs in a warp's table: the pair lies at
// (column * seed) / 2^22 ^ row * 32, so that no two rows share a slot for
// the same column and a slot that holds the column answers exactly; the
// warp looks for a seed under which no two pairs share a slot.
__device__ __forceinline__ uint32_t row_set_at(uint32_t c, uint32_t seed, uint32_t key) {
  return (((c * seed) >> 20) & (4 * kRowSetSlots - 4)) ^ key;  // bytes from the tables' start
}

// Row of edge j: the last row r in [lo, hi) with rp[r] <= j (a warp together,
// 32 probes a step).
template <typename Off>
__device__ __forceinline__ uint64_t row_of_edge(const Off *__restrict__ rp, uint64_t lo,
                                                uint64_t hi, uint64_t j, uint32_t lane) {
  uint64_t count = hi - lo;
  while (count > 1) {
    const uint64_t step = (count + 31) / 32, at = (lane + 1) * step;
    const bool below = at < count && ld_off(rp, lo + at) <= j;
    const uint64_t k = __popc(__ballot_sync(0xffffffffu, below));
    lo += k * step;
    count = min(step, count - k * step);
  }
  return lo;
}

// The edges [rp[row_lo], rp[row_hi]), T per warp, one thread each: edges to
// short rows are counted here (their wedges added to out[1], triangles to
// out[0]); with kEmit, edges to long rows become entries for the walk,
// appended in any order (*made of them, those past cap are only counted) --
// but for the tail's part outside the window, which is intersected here when
// the long row has few columns there -- and without it they are counted here
// too. Nothing is done when *err is set (the row offsets cannot be trusted),
// or with kEmit when the word behind it is (the graph is not walked after all).
// An edge intersects its tail with its short row (merge_rows: 4 by 4 columns
// in about 50 instructions, with 57% of the lanes busy), or, with kSets, the
// columns of the chunk's rows become an exact set in shared memory and the
// short rows stream through it, a 32-byte sector per lane (8 columns in
// about 85 instructions, nearly all lanes busy). Bound by instruction issue
// and the shared-memory pipe (65% each). Erdos-Renyi with 700,001 vertices
// and 13.3M edges: 427 us by sets, 533 by intersections (pair streams: 584
// after a plan of 131 us and 152 us of hash sets); R-MAT scale 22: 0.76 ms
// by intersections (1.27 ms before the few edges that intersect rows there
// were gathered to fill the warp). A chunk ends with a row when that leaves
// fewer than 8 lanes idle (a batch of 96 graphs: 6.63 ms; always 32 edges:
// 6.94; whole rows only: 7.5); chunks of more than 4 rows, 64 columns or
// fewer than 8 edges to short rows intersect.
// kBatch: the rows are a batch's, the triangles go to their graphs' counts;
// with kEmit, `what` says whether it is the count (the long rows' entries
// were made before) or the making of the entries.
enum MergeWhat : uint32_t { kMergeCount = 1, kMergeEmit = 2 };
template <typename Off, bool kEmit, bool kBatch, bool kSets, bool kSearch>
__global__ void __launch_bounds__(kMergeBlock, kSets ? 7 : 8)
    k_edge_merge(const Off *__restrict__ rp, const __grid_constant__ WalkColumns cols, uint64_t n,
                 uint64_t row_lo, uint64_t row_hi, uint32_t T,
                 const uint32_t *__restrict__ number, const uint32_t *__restrict__ split,
                 const WalkBits bits, uint64_t *__restrict__ entries, uint32_t cap,
                 uint32_t *__restrict__ made, unsigned long long *__restrict__ out,
                 const uint32_t *__restrict__ err,
                 const __grid_constant__ WalkGroups groups = WalkGroups{},
                 uint32_t what = kMergeCount | kMergeEmit) {
  __shared__ uint32_t s_start[kMergeBlock / 32][32], s_row[kMergeBlock / 32][32];
  __shared__ uint64_t s_entry[kEmit ? kMergeBlock / 32 : 1][kEmit ? kMergeStage : 1];
  constexpr bool kGather = kEmit || kSets;
  __shared__ MergeTask s_task[kGather ? kMergeBlock / 32 : 1][64];
  __shared__ __align__(16) uint32_t s_set[kSets ? kMergeBlock / 32 * kRowSetSlots : 4];
  __shared__ uint4 s_unit[kSets ? kMergeBlock / 32 : 1][32];
  const uint2 stop =
      kEmit && !kBatch ? *reinterpret_cast<const uint2 *>(err) : make_uint2(*err, 0u);
  if (stop.x | stop.y) return;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, le = 0xFFFFFFFFu >> (31 - lane);
  const uint32_t *ci = cols.base + cols.mis;
  const uint32_t j_end = (uint32_t)ld_off(rp, row_hi);
  const uint64_t t = (uint64_t)blockIdx.x * (kMergeBlock / 32) + wid;
  const uint64_t from = ld_off(rp, row_lo) + t * T;
  if (from >= j_end) return;
  const uint32_t j1 = j_end - from < T ? j_end : (uint32_t)from + T;
  auto slot = [&](uint32_t at) -> uint32_t & {
    return *reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(s_set) + at);
  };
  if (kSets)
    for (uint32_t i = lane; i < kRowSetSlots; i += 32) s_set[wid * kRowSetSlots + i] = kWalkEmpty;
  __syncwarp();
  uint32_t seed = 0x9E3779B1u;
  unsigned long long wedges = 0;
  uint32_t hits = 0;
  // A warp's entries gather in shared memory and go out together: one atomic
  // on the common counter for up to 128 of them (one per round of 32 edges
  // took longer than the rest of the kernel).
  uint32_t staged = 0, tasks = 0;
  uint64_t *stage = s_entry[kEmit ? wid : 0];
  auto flush = [&]() {
    __syncwarp();
    uint32_t x = 0;
    if (lane == 0) x = atomicAdd(made, staged);
    x = __shfl_sync(0xffffffffu, x, 0);
    for (uint32_t i = lane; i < staged; i += 32)
      if (x + i < cap) entries[x + i] = stage[i];
    staged = 0;
    __syncwarp();
  };
  uint32_t g = 0;
  auto drain = [&]() {  // kBatch: the graph's hits so far
    if (kGather && lane < tasks) hits += merge_rows<kSearch>(cols, s_task[kGather ? wid : 0][lane]);
    tasks = 0;
    const uint32_t c = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0 && c) atomicAdd(groups.counts + g, (unsigned long long)c);
    hits = 0;
    __syncwarp();
  };
  for (uint32_t j = (uint32_t)from; j < j1;) {
    const uint64_t r = row_of_edge(rp, row_lo, row_hi, j, lane);
    uint64_t rows_end = row_hi;
    if (kBatch) {  // the rows at hand are one graph's
      const uint32_t now = (uint32_t)row_of_edge(groups.base, 0, groups.G, r, lane);
      if (now != g) {
        drain();
        g = now;
      }
      rows_end = __ldg(groups.base + g + 1);
    }
    const uint64_t v = r + lane < rows_end ? r + lane : rows_end;
    const uint32_t b = (uint32_t)ld_off(rp, v);
    const uint32_t e = v < rows_end ? (uint32_t)ld_off(rp, v + 1) : b;
    const uint32_t mid = kEmit && v < rows_end ? split[v] : b;
    const uint32_t stop = min(j1, __shfl_sync(0xffffffffu, e, 31));
    const uint32_t rows = __ballot_sync(0xffffffffu, e > b);
    __syncwarp();
    if (e > b) {
      s_start[wid][__popc(rows & lt)] = max(b, j) - j;
      s_row[wid][__popc(rows & lt)] = lane;
    }
    __syncwarp();
    const uint32_t c = lane < __popc(rows) ? s_start[wid][lane] : 0xFFFFFFFFu;
    uint32_t before = 0;
    uint32_t w_next = j + lane < stop ? __ldg(ci + j + lane) : 0u, s0_next = 0, s1_next = 0;
    auto next_row = [&](bool in) {
      s0_next = in && w_next < n ? (uint32_t)ld_off(rp, w_next) : 0u;
      s1_next = in && w_next < n ? (uint32_t)ld_off(rp, w_next + 1) : 0u;
    };
    if (!kEmit) next_row(j + lane < stop);
    for (uint32_t q0 = 0, len; q0 < stop - j; q0 += len) {
      const uint32_t p = j + q0;
      len = min(32u, stop - p);
      if (kSets) {  // a set of whole rows when that leaves few lanes idle
        const uint32_t whole = __reduce_max_sync(0xffffffffu, e <= p + 32 ? e : 0u);
        if (whole >= p + kRowSetFill) len = min(len, whole - p);
      }
      const uint32_t starts =
          __reduce_or_sync(0xffffffffu, c - q0 < len ? 1u << (c - q0) : 0u);
      const uint32_t at = before + __popc(starts & le) - 1;
      before += __popc(starts);
      const uint32_t edge = p + lane;
      const uint32_t row = s_row[wid][at & 31];
      const uint32_t end = __shfl_sync(0xffffffffu, e, row);
      const uint32_t first = edge + 1;
      const bool on = lane < len && first < end;
      // the next edges' columns and the offsets of their rows are under way
      // while these are counted
      const uint32_t w = w_next, r0 = s0_next, r1 = s1_next;
      w_next = edge + len < stop ? __ldg(ci + edge + len) : 0u;
      const bool ok = on && w < n;
      uint32_t id = kWalkShort, t1 = end;
      uint32_t s0 = 0, s1 = 0;
      if (kEmit) {
        const uint32_t cut = __shfl_sync(0xffffffffu, mid, row);
        if (ok) id = __ldg(number + w);
        const bool is_long = id != kWalkShort;
        const bool win = is_long && cut < end;
        bool rest = is_long && first < cut;
        if (rest) {
          s0 = (uint32_t)ld_off(rp, w);
          s1 = split[w];
          if (s1 - s0 <= kWalkShortCols) {
            rest = false;
            t1 = cut;
            wedges += cut - first;
          } else {
            s1 = s0;
          }
        }
        const uint32_t rm = __ballot_sync(0xffffffffu, rest);
        const uint32_t wm = __ballot_sync(0xffffffffu, win);
        if ((rm | wm) && (!kBatch || (what & kMergeEmit))) {
          const uint32_t add = __popc(rm) + __popc(wm);
          if (staged + add > kMergeStage) flush();
          const uint32_t xr = staged + __popc(rm & lt);
          const uint32_t xw = staged + __popc(rm) + __popc(wm & lt);
          const uint64_t key = (uint64_t)id << (bits.shift() + 1);
          const uint32_t wf = max(first, cut);
          if (rest) stage[xr] = key | ((uint64_t)first << bits.len) | (cut - first);
          if (win)
            stage[xw] = key | (1ull << bits.shift()) | ((uint64_t)wf << bits.len) | (end - wf);
          staged += add;
        }
      }
      bool task_on = s0 < s1;  // the rest of a tail
      if (ok && id == kWalkShort) {
        wedges += end - first;
        s0 = kEmit ? (uint32_t)ld_off(rp, w) : r0;
        s1 = kEmit ? (uint32_t)ld_off(rp, w + 1) : r1;
      }
      if (kBatch && !(what & kMergeCount)) continue;
      const MergeTask task{first + cols.mis, t1 + cols.mis, s0 + cols.mis, s1 + cols.mis};
      if (!kGather) {
        if (s0 < s1) hits += merge_rows<kSearch>(cols, task);
        if (!kEmit) next_row(edge + len < stop);
        continue;
      }
      const uint32_t set_end = __shfl_sync(0xffffffffu, end, len - 1);
      bool unit = !task_on && s0 < s1 && s1 - s0 <= kRowSetLong;
      task_on = s0 < s1;
      bool fetched = false;
      const uint32_t um = __ballot_sync(0xffffffffu, unit);
      if (kSets && __popc(starts) <= kRowSetRows && set_end - p <= kRowSetCols && __popc(um) >= kRowSetMin) {
        // the chunk's rows as a set, two columns a lane: those of its edges,
        // and the last row's behind them
        const uint32_t x4 =
            ((__popc(starts & le) - (starts & 1u)) * 32 | wid * kRowSetSlots) * 4;
        const uint32_t x2 = __shfl_sync(0xffffffffu, x4, len - 1);
        const bool in1 = edge < set_end, in2 = edge + 32 < set_end;
        const uint32_t x1 = lane < len ? x4 : x2;
        const uint32_t w1 = lane < len ? w : in1 ? __ldg(ci + edge) : 0u;
        const uint32_t w2 = in2 ? __ldg(ci + edge + 32) : 0u;
        bool found = false;
        for (uint32_t tries = 0; tries < kRowSetTries; ++tries) {
          const uint32_t a1 = row_set_at(w1, seed, x1), a2 = row_set_at(w2, seed, x2);
          if (in1) slot(a1) = w1;
          if (in2) slot(a2) = w2;
          __syncwarp();
          const bool lost = (in1 && slot(a1) != w1) || (in2 && slot(a2) != w2);
          found = !__any_sync(0xffffffffu, lost);
          if (found) break;
          if (in1) slot(a1) = kWalkEmpty;
          if (in2) slot(a2) = kWalkEmpty;
          __syncwarp();
          seed = seed * 0x2C9277B5u + 2u;  // odd stays odd
        }
        if (found) {
          // the sectors of the rows of w, one per lane and round
          const uint32_t f = (s0 + cols.mis) >> 3;
          const uint32_t sectors = unit ? ((s1 + cols.mis + 7) >> 3) - f : 0u;
          const uint32_t incl = walk_scan(sectors, lane), pre = incl - sectors;
          const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
          if (unit)
            s_unit[kSets ? wid : 0][__popc(um & lt)] =
                make_uint4(f - pre, s0 + cols.mis, s1 + cols.mis, x4);
          __syncwarp();
          uint32_t units = 0, key = wid * kRowSetSlots * 4, valid = 0, x[8] = {};
          auto fetch = [&](uint32_t u0) {
            const uint32_t heads = __reduce_or_sync(
                0xffffffffu, unit && pre - u0 < 32u ? 1u << (pre - u0) : 0u);
            const uint4 u = s_unit[kSets ? wid : 0][(units + __popc(heads & le) - 1) & 31];
            units += __popc(heads);
            valid = 0;
            if (u0 + lane < total) {
              const uint32_t sa = (u.x + u0 + lane) << 3;
              walk_sector(cols, sa, u.y, u.z, x);
              const uint32_t lo = u.y > sa ? u.y - sa : 0u;
              const uint32_t hi = sa + 8 > u.z ? sa + 8 - u.z : 0u;
              valid = (0xFFu << lo) & (0xFFu >> hi);
              key = u.w;
            }
          };
          fetch(0);
          if (!kEmit) next_row(edge + len < stop);
          fetched = true;
          for (uint32_t u0 = 0; u0 < total; u0 += 32) {
            uint32_t y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = x[i];
            const uint32_t in = valid, k = key;
            if (u0 + 32 < total) fetch(u0 + 32);
            uint32_t got = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (slot(row_set_at(y[i], seed, k)) == y[i]) got |= 1u << i;
            hits += __popc(got & in);
          }
          task_on = task_on && !unit;
          __syncwarp();
          if (in1) slot(row_set_at(w1, seed, x1)) = kWalkEmpty;
          if (in2) slot(row_set_at(w2, seed, x2)) = kWalkEmpty;
          __syncwarp();
        }
      }
      // the others gather until there is one for every lane
      if (!kEmit && !fetched) next_row(edge + len < stop);
      const uint32_t mm = __ballot_sync(0xffffffffu, task_on);
      if (!mm) continue;
      if (task_on) s_task[wid][tasks + __popc(mm & lt)] = task;
      tasks += __popc(mm);
      __syncwarp();
      if (tasks >= 32) {
        hits += merge_rows<kSearch>(cols, s_task[wid][lane]);
        tasks -= 32;
        const MergeTask moved = s_task[wid][32 + lane];
        __syncwarp();
        if (lane < tasks) s_task[wid][lane] = moved;
        __syncwarp();
      }
    }
    j = stop;
  }
  if (kBatch) drain();
  if (kGather && lane < tasks) hits += merge_rows<kSearch>(cols, s_task[kGather ? wid : 0][lane]);
  if (kEmit && staged) flush();
  unsigned long long h = hits;
  for (int o = 16; o > 0; o >>= 1) {
    h += __shfl_down_sync(0xffffffffu, h, o);
    wedges += __shfl_down_sync(0xffffffffu, wedges, o);
  }
  if (lane == 0) {
    if (h) atomicAdd(out, h);
    if (wedges) atomicAdd(out + 1, wedges);
  }
}

// A small graph's whole count in one launch: the row checks and totals of
// k_edge_vertices and the intersections of k_edge_merge, T edges per warp,
// block b's results in out[4b, 4b + 4) -- triangles, W, rows with wedges (and
// bit 40: bad offsets), longest row -- which may be host memory, so nothing is
// cleared before or copied after. Offsets are not trusted: each row's are
// checked before it is read. Bound by the call around it (launch, events,
// wait): 2,000 vertices, 57 -> 33 us against the two kernels, a memset and a
// copy.
constexpr uint32_t kSmallBlocks = 256;
constexpr uint32_t kSmallWords = 4;
template <typename Off>
__global__ void __launch_bounds__(kWalkBlock)
    k_small_count(const Off *__restrict__ rp, const __grid_constant__ WalkColumns cols, uint32_t n,
                  uint32_t m, uint32_t T, unsigned long long *__restrict__ out) {
  __shared__ uint32_t s_start[kWalkBlock / 32][32], s_row[kWalkBlock / 32][32];
  __shared__ unsigned long long s_sum[kSmallWords];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, le = 0xFFFFFFFFu >> (31 - lane);
  if (threadIdx.x < kSmallWords) s_sum[threadIdx.x] = 0;
  __syncthreads();
  bool bad = blockIdx.x == 0 && threadIdx.x == 0 &&
             (ld_off(rp, 0) != 0 || ld_off(rp, (uint64_t)n) != m);
  unsigned long long W = 0;
  uint32_t rows = 0, longest = 0, hits = 0;
  for (uint32_t v = blockIdx.x * kWalkBlock + threadIdx.x; v < n; v += gridDim.x * kWalkBlock) {
    const uint64_t b = ld_off(rp, (uint64_t)v), e = ld_off(rp, (uint64_t)v + 1);
    if (e < b || e > m) {
      bad = true;
    } else {
      const uint32_t d = (uint32_t)(e - b);
      W += d >= 2 ? (unsigned long long)d * (d - 1) / 2 : 0;
      rows += d >= 2;
      longest = max(longest, d);
    }
  }
  const uint32_t *ci = cols.base + cols.mis;
  const uint64_t from = (uint64_t)(blockIdx.x * (kWalkBlock / 32) + wid) * T;
  const uint32_t j1 = (uint32_t)min((uint64_t)m, from + T);
  for (uint32_t j = (uint32_t)min(from, (uint64_t)m); j < j1;) {
    const uint64_t v = row_of_edge(rp, 0, n, j, lane) + lane;
    uint64_t b64 = m, e64 = m;
    if (v < n) b64 = ld_off(rp, v), e64 = ld_off(rp, v + 1);
    if (e64 < b64 || e64 > m) b64 = e64 = 0;  // counted as bad above
    const uint32_t b = (uint32_t)b64, e = (uint32_t)e64;
    const uint32_t stop = min(j1, __shfl_sync(0xffffffffu, e, 31));
    if (stop <= j) break;  // not with good offsets
    const uint32_t some = __ballot_sync(0xffffffffu, e > b);
    __syncwarp();
    if (e > b) {
      s_start[wid][__popc(some & lt)] = max(b, j) - j;
      s_row[wid][__popc(some & lt)] = lane;
    }
    __syncwarp();
    const uint32_t c = lane < __popc(some) ? s_start[wid][lane] : 0xFFFFFFFFu;
    uint32_t before = 0;
    for (uint32_t q0 = 0; q0 < stop - j; q0 += 32) {
      const uint32_t starts = __reduce_or_sync(0xffffffffu, c - q0 < 32u ? 1u << (c - q0) : 0u);
      const uint32_t at = before + __popc(starts & le) - 1;
      before += __popc(starts);
      const uint32_t edge = j + q0 + lane;
      const uint32_t end = __shfl_sync(0xffffffffu, e, s_row[wid][at & 31]);
      if (edge < stop && edge + 1 < end) {
        const uint32_t w = __ldg(ci + edge);
        if (w < n) {
          const uint64_t s0 = ld_off(rp, (uint64_t)w), s1 = ld_off(rp, (uint64_t)w + 1);
          if (s0 < s1 && s1 <= m)
            hits += merge_rows<true>(cols, MergeTask{edge + 1 + cols.mis, end + cols.mis,
                                               (uint32_t)s0 + cols.mis, (uint32_t)s1 + cols.mis});
        }
      }
    }
    j = stop;
  }
  for (int o = 16; o > 0; o >>= 1) W += __shfl_down_sync(0xffffffffu, W, o);
  hits = __reduce_add_sync(0xffffffffu, hits);
  rows = __reduce_add_sync(0xffffffffu, rows);
  longest = __reduce_max_sync(0xffffffffu, longest);
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
    if (hits) atomicAdd(&s_sum[0], (unsigned long long)hits);
    if (W) atomicAdd(&s_sum[1], W);
    if (rows) atomicAdd(&s_sum[2], (unsigned long long)rows);
    if (bad) atomicOr(&s_sum[2], 1ull << 40);
    if (longest) atomicMax(&s_sum[3], (unsigned long long)longest);
  }
  __syncthreads();
  if (threadIdx.x < kSmallWords) out[blockIdx.x * kSmallWords + threadIdx.x] = s_sum[threadIdx.x];
}

// Whether the edges to long rows (more than 48 columns) are worth sorting for
// the walk, against intersecting every row where its edge is: intersections
// with rows of up to 128 columns waste at most 32 steps, and below 2^25
// wedges of long rows the sort's launches and passes cost more than they save
// (Chung-Lu, 100,000 vertices, mean degree 40, longest row 97: 0.24 ms
// without, 0.31 with; 300,000 and 60, longest 218: 1.42 against 0.87; with
// 1,000,000 and 40, exponent 2.8, longest 51: 0.86 against 1.04).
constexpr uint64_t kWalkMinEdges = 1ull << 19;
inline bool walk_wanted(uint64_t long_rows, uint64_t longest, uint64_t long_wedges,
                        uint64_t edges) {
  return long_rows > 0 && edges >= kWalkMinEdges && (longest > 128 || long_wedges >= (1ull << 25));
}

// How an entry's fields lie when m columns, long_rows rows of up to `longest`
// columns have to fit them; 64 bits or fewer in all, or there is no walk.
inline WalkBits walk_bits(uint64_t m, uint64_t long_rows, uint64_t longest) {
  return WalkBits{1 + (long_rows > 1 ? bits_for(long_rows - 1) : 1), bits_for(m),
                  bits_for(longest)};
}

// What counts a graph (or batch) below its core: intersections alone, with
// the walk, or neither -- the walk is wanted, so intersecting the long rows
// edge by edge is the slower way by far, but its entries do not fit, as from
// about 2^30 columns on in graphs with hubs: the wedge checks take it (R-MAT
// scale 26, 1.05e9 columns, one bit too many: 584 ms a count, 2,917 when its
// long rows were intersected).
enum class WalkForm { kMerge, kWalk, kNone };
inline WalkForm walk_form(uint64_t n, uint64_t m, uint64_t edges, uint64_t long_rows,
                          uint64_t longest, uint64_t long_wedges) {
  if (!walk_wanted(long_rows, longest, long_wedges, edges)) return WalkForm::kMerge;
  const WalkBits b = walk_bits(m, long_rows, longest);
  return n < (1ull << 31) && m < (1ull << 31) && b.w + b.start + b.len <= 64 ? WalkForm::kWalk
                                                                             : WalkForm::kNone;
}

// Whether k_edge_merge counts by sets: a set pays when many wedges share it,
// that is from some mean tail (wedges per edge) on. Measured, sets /
// intersections in us: Erdos-Renyi, 6M edges, tail 4.2 207 / 192, 5.4 200 /
// 198, 6.6 195 / 208; 13.3M, 9.2 427 / 533; 2M, 6.6 86 / 82, 8.5 79 / 80, 16
// 105 / 128. Rows of uneven lengths leave more lanes of the intersections
// idle: Chung-Lu, 6M edges, longest row 47, 3.4 184 / 196, 6.7 231 / 273.
// Fewer than 2^20 edges take 20-32 either way. Not where the walk takes most
// wedges (R-MAT scale 22: 906 / 759).
inline bool row_sets_wanted(uint64_t edges, uint64_t wedges, uint64_t longest, uint64_t walked) {
  const uint64_t tail = edges < (1ull << 22) ? 8 : longest > 40 ? 3 : 6;
  return edges >= (1ull << 20) && wedges >= tail * edges && walked < wedges / 2;
}

// Edges per warp: kMergeTile, or fewer (whole rounds) when that leaves the
// device's warps less than two tiles each.
inline uint32_t merge_tile(uint64_t edges, int sms) {
  const uint64_t per = ceil_div(ceil_div(edges, 2ull * sms * 32), 32) * 32;
  return per < kMergeTile ? (uint32_t)(per ? per : 32) : kMergeTile;
}

// The 32-byte sectors that a tail [first, first + len) touches.
__device__ __forceinline__ uint32_t walk_sectors(uint32_t first, uint32_t len) {
  return len ? ((first + len + 7) >> 3) - (first >> 3) : 0u;
}

// Streams the tails of k <= kGroup entries through test(columns, entry,
// mask), which returns how many of the masked 8 columns it finds. The
// tails' sectors lie one after another in s_pre's numbering (exclusive
// prefix of their counts, S in all), and thread `id` of kLanes takes sectors
// id, id + kLanes, ...: every thread does the same number of rounds, a round
// is 8 columns for one load, and neighbouring threads read neighbouring
// sectors. A sector's entry is the number of tails that start at or before
// it: s_head marks the starts, s_cnt counts those before each of its words.
// Steps on the way, R-MAT scale 22: a warp's 32 lanes packed over the
// columns (a reduction, popcounts and shuffles a round: 61 instructions per
// 32 columns) 4.0 ms; spans of consecutive sectors per thread (no lookup,
// but 32 lines a load) 2.3 ms; this with blocks of two sizes 2.1 ms. The next sector's load is
// out while one is tested. sync() is the threads' barrier.
template <uint32_t kGroup, uint32_t kLanes, uint32_t kWords, class Entry, class Sync, class Test>
__device__ __forceinline__ uint32_t walk_tails(const WalkColumns &cols, const Entry *s_e,
                                               const uint32_t *s_pre, uint32_t *s_head,
                                               uint32_t *s_cnt, uint32_t k, uint32_t S,
                                               uint32_t id, const Sync &sync, const Test &test) {
  static_assert(kLanes >= kWords, "a thread per word of s_head");
  const uint32_t le = 0xFFFFFFFFu >> (31 - (id & 31));
  uint32_t hits = 0;
  for (uint32_t s0 = 0; s0 < S; s0 += 32 * kWords) {
    const uint32_t s1 = min(S, s0 + 32 * kWords);
    if (s0) sync();
    if (id < kWords && 32 * id < s1 - s0) {
      s_head[id] = 0;
      uint32_t c = 0;  // entries that start before word id: the first at or past it
#pragma unroll
      for (uint32_t o = kGroup / 2; o; o >>= 1)
        if (c + o <= k && s_pre[c + o - 1] < s0 + 32 * id) c += o;
      if (c < k && s_pre[c] < s0 + 32 * id) ++c;
      s_cnt[id] = c;
    }
    sync();
    for (uint32_t i = id; i < k; i += kLanes) {
      const uint32_t at = s_pre[i] - s0;
      if (at < s1 - s0) atomicOr(&s_head[at >> 5], 1u << (at & 31));
    }
    sync();
    auto fetch = [&](uint32_t s, uint32_t(&x)[8], Entry &en) {
      uint32_t mask = 0;
      if (s < s1) {
        const uint32_t word = (s - s0) >> 5;
        const uint32_t e = s_cnt[word] + __popc(s_head[word] & le) - 1;
        en = s_e[e];
        const uint32_t a = (en.first & ~7u) + 8 * (s - s_pre[e]);
        const uint32_t end = en.first + en.len;
        mask = (0xFFu >> (en.first > a ? en.first - a : 0u)) &
               (0xFFu << (end < a + 8 ? a + 8 - end : 0u));
        walk_sector(cols, a, en.first, end, x);
      }
      return mask;
    };
    uint32_t x[8] = {}, y[8] = {};
    Entry ex{}, ey{};
    uint32_t mx = fetch(s0 + id, x, ex);
    for (uint32_t s = s0 + id; s - id < s1; s += 2 * kLanes) {
      const uint32_t my = fetch(s + kLanes, y, ey);
      hits += test(x, ex, mx);
      mx = fetch(s + 2 * kLanes, x, ex);
      hits += test(y, ey, my);
    }
  }
  return hits;
}

__device__ __forceinline__ void walk_insert(uint32_t *set, uint32_t slots, uint32_t x,
                                            uint32_t shift) {
  uint32_t h = (x * kHashMul) >> shift;
  for (;;) {
    const uint32_t old = atomicCAS(set + h, kWalkEmpty, x);
    if (old == kWalkEmpty || old == x) return;
    h = (h + 1) & (slots - 1);
  }
}
// How many of the masked columns are in the set: every column's home slot
// first, then the few that it does not decide.
__device__ __forceinline__ uint32_t walk_find8(const uint32_t *set, uint32_t slots, uint32_t shift,
                                               const uint32_t (&x)[8], uint32_t mask) {
  uint32_t found = 0, open = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t key = set[(x[j] * kHashMul) >> shift];
    found |= key == x[j] ? 128u >> j : 0u;
    open |= key != x[j] && key != kWalkEmpty ? 128u >> j : 0u;
  }
  uint32_t hits = __popc(found & mask);
  open &= mask;
  if (open) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (!((open >> (7 - j)) & 1u)) continue;
      uint32_t h = (x[j] * kHashMul) >> shift;
      for (;;) {
        h = (h + 1) & (slots - 1);
        const uint32_t key = set[h];
        if (key == x[j]) ++hits;
        if (key == x[j] || key == kWalkEmpty) break;
      }
    }
  }
  return hits;
}

// One block per item: taken from a counter (per_block == 0), or per_block
// consecutive ones per block. Window columns are bits of a 65,536 bit row,
// cleared column by column when the item is done; others a hash set at most
// half full (longer rows: 1,024 columns at a time, the tails streamed again
// for each part). The block's threads share the sectors of up to four tails
// each equally, so they meet at the barriers together: with tails handed to
// warps in groups of 64 the kernel spent half its time there. Vertices of up
// to kWalkBig entries and kWalkBigCols columns have blocks of one warp: most of
// the vertices of R-MAT scale 22, whose set-up by four warps took two thirds of
// the instructions.
// R-MAT scale 22: 1.87 ms for the blocks' vertices (shared-memory pipe 86%
// busy, DRAM 5.4 GB) and 0.38 ms for the others, where the wedge checks of
// the same edges took 7.6 ms and 0.58 for the hash sets.
template <uint32_t kThreads, int kBlocks, bool kBatch, bool kShare = false>
__global__ void __launch_bounds__(kThreads, kBlocks)
    k_walk_count(const uint32_t *__restrict__ rp, const uint32_t *__restrict__ split,
                 const uint32_t *__restrict__ long_rows, const __grid_constant__ WalkColumns cols,
                 uint32_t t0, const uint64_t *__restrict__ keys,
                 const uint32_t *__restrict__ start, const WalkBits bits,
                 const uint2 *__restrict__ items, const uint32_t *__restrict__ count,
                 uint32_t *__restrict__ ticket, uint32_t per_block,
                 unsigned long long *__restrict__ out, const __grid_constant__ WalkGroups groups,
                 const uint32_t *__restrict__ long_graph, const uint32_t *__restrict__ err) {
  if (*err != kDevOk) return;
  struct Entry {
    uint32_t first, len;
  };
  static_assert(kWalkSetSlots * 32 == kWalkWindow, "the bit row and the set share memory");
  constexpr bool kBits = kThreads > 32;  // small vertices have hash sets only
  constexpr uint32_t kSlots = kBits ? kWalkSetSlots : kWalkSmallSlots;
  constexpr uint32_t kWarps = kThreads / 32, kGroup = kWalkPer * kThreads;
  __shared__ __align__(16) uint32_t s_set[kSlots];
  __shared__ Entry s_e[kGroup];
  __shared__ uint32_t s_pre[kGroup];
  __shared__ uint32_t s_head[kThreads], s_cnt[kThreads];
  __shared__ uint32_t s_warp[kWarps], s_item;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t *ci = cols.base + cols.mis;
  const uint32_t n_items = *count;
  uint32_t not_t0 = t0 - 1, g = 0;
  const char *row = reinterpret_cast<const char *>(s_set);
  constexpr uint32_t word_mask = (kWalkSetSlots - 1) * 4;
  const uint64_t start_mask = (1ull << bits.start) - 1, len_mask = (1ull << bits.len) - 1;
  auto fill = [&](uint32_t slots, uint32_t with) {
    for (uint32_t i = tid; i < slots / 4; i += kThreads)
      reinterpret_cast<uint4 *>(s_set)[i] = make_uint4(with, with, with, with);
  };
  if (kBits) fill(kWalkSetSlots, 0u);
  unsigned long long hits = 0;
  uint32_t turn = 0, next = 0;
  if (tid == 0) next = per_block ? blockIdx.x * per_block : atomicAdd(ticket, 1u);
  for (;;) {
    if (tid == 0) s_item = next;
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= n_items) break;
    ++turn;
    if (tid == 0)  // the next item, ahead of its use
      next = per_block ? (turn < per_block ? it + 1 : n_items) : atomicAdd(ticket, 1u);
    const uint2 item = items[it];
    const uint32_t x = item.x;
    const bool several = kShare && (item.y & kWalkSeveral);
    const uint32_t piece = several ? kWalkSetPiece : kWalkPiece;
    const uint32_t e0 = start[x] + (several ? item.y & ((1u << kWalkGroupShift) - 1) : item.y) * piece;
    const uint32_t e1 = min(start[x + 1], e0 + piece);
    const uint2 set = walk_set(rp, split, long_rows, x);
    const uint32_t d = set.y - set.x;
    const uint32_t group_cols = several ? walk_group_cols(d) : d;
    const uint32_t part0 =
        several ? (item.y >> kWalkGroupShift & (kWalkSetGroups - 1)) * group_cols : 0u;
    const uint32_t part1 = min(d, part0 + group_cols);
    if (kBatch) {
      const uint32_t now = __ldg(long_graph + (x >> 1));
      if (now != g) {
        walk_add_hits(groups.counts + g, hits, lane);
        hits = 0;
        g = now;
      }
      t0 = walk_window(groups, g);
      not_t0 = t0 - 1;
    }
    const bool window = kBits && (x & 1);
    for (uint32_t part = part0; part < part1; part += window || !kBits ? d : kWalkSetCols) {
      const uint32_t ncols = window || !kBits ? d : min(d - part, kWalkSetCols);
      const uint32_t slots = min(1u << (32 - __clz(max(ncols * 4u, 256u) - 1u)), kSlots);
      const uint32_t shift = __clz(slots - 1);
      for (uint32_t at = e0; at < e1; at += kGroup) {
        if (part > part0 || at > e0) __syncthreads();  // the last group is done with
        const bool fresh = at == e0;           // the set is built with the first group
        if (fresh && !window) fill(slots, kWalkEmpty);
        Entry en[kWalkPer];
        uint32_t sec[kWalkPer], mine = 0;
#pragma unroll
        for (uint32_t j = 0; j < kWalkPer; ++j) {
          const uint32_t i = at + tid * kWalkPer + j;
          const uint64_t k = i < e1 ? __ldg(keys + i) : 0;
          en[j] = Entry{(uint32_t)((k >> bits.len) & start_mask) + cols.mis,
                        (uint32_t)(k & len_mask)};
          sec[j] = mine;
          mine += walk_sectors(en[j].first, en[j].len);
        }
        const uint32_t incl = walk_scan(mine, lane);
        uint32_t before = incl - mine, S = 0;
        if (kWarps > 1) {
          if (lane == 31) s_warp[warp] = incl;
          __syncthreads();
#pragma unroll
          for (uint32_t q = 0; q < kWarps; ++q) {
            if (q < warp) before += s_warp[q];
            S += s_warp[q];
          }
        } else {
          S = __shfl_sync(0xffffffffu, incl, 31);
          __syncwarp();
        }
        const uint32_t k = min(e1 - at, kGroup);
        if (tid * kWalkPer < k) {
#pragma unroll
          for (uint32_t j = 0; j < kWalkPer; ++j) {
            s_e[tid * kWalkPer + j] = en[j];
            s_pre[tid * kWalkPer + j] = before + sec[j];
          }
        }
        if (fresh)
          for (uint32_t i = tid; i < ncols; i += kThreads) {
            const uint32_t u = __ldg(ci + set.x + part + i), c = u - t0;
            if (!window)
              walk_insert(s_set, slots, u, shift);
            else if (c < kWalkWindow)
              atomicOr(&s_set[c >> 5], 1u << (c & 31));
          }
        __syncthreads();
        if (window)
          hits += walk_tails<kGroup, kThreads, kThreads>(
              cols, s_e, s_pre, s_head, s_cnt, k, S, tid, [] { __syncthreads(); },
              [&](const uint32_t(&x)[8], const Entry &, uint32_t mask) {
                // bit c of the row, c = x - t0, at the top of its word
                // shifted left by ~c (the byte offset wraps, for columns
                // that are not the tail's)
                uint32_t b = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const uint32_t nc = not_t0 - x[j];
                  const uint32_t word =
                      *reinterpret_cast<const uint32_t *>(row + (~(nc >> 3) & word_mask));
                  b = __funnelshift_l(word << (nc & 31), b, 1);
                }
                return (uint32_t)__popc(b & mask);
              });
        else
          hits += walk_tails<kGroup, kThreads, kThreads>(
              cols, s_e, s_pre, s_head, s_cnt, k, S, tid, [] { __syncthreads(); },
              [&](const uint32_t(&x)[8], const Entry &, uint32_t mask) {
                return walk_find8(s_set, slots, shift, x, mask);
              });
      }
    }
    __syncthreads();
    if (window) {
      for (uint32_t i = tid; i < d; i += kThreads) {
        const uint32_t c = __ldg(ci + set.x + i) - t0;
        if (c < kWalkWindow) s_set[c >> 5] = 0;
      }
    } else if (kBits) {
      fill(kWalkSetSlots, 0u);
    }
  }
  walk_add_hits(kBatch ? groups.counts + g : out, hits, lane);
}

// Room for at least x elements, in eighths of a power of two: graphs of one
// kind then ask the pool for the same sizes and find the blocks that the last
// count freed (with exact sizes the pool went to the driver now and then:
// 33-51 ms a count on R-MAT scale 24 for 32).
inline uint64_t walk_room(uint64_t x) {
  if (x < 4096) return 4096;
  const uint64_t step = 1ull << (bits_for(x) - 4);
  return ceil_div(x, step) * step;
}

// The walk of one count: its buffers and launches.
struct WalkRun {
  WalkBits bits{};
  uint64_t n = 0, m = 0, rows = 0, cap = 0, entries = 0, big_cap = 0;
  bool share_sets = false;  // there are rows of several sets (WalkFar), shared out
  Scratch<uint64_t> keys, alt;
  // [0] entries made, [1] big, [2] small items, [3, 4] tickets, [6...] WalkFar
  Scratch<uint32_t> split, start, counts;
  Scratch<uint2> big, small;
  prim::SortSpace ws;
  const uint64_t *sorted = nullptr;

  static constexpr uint32_t kFar = 6, kCounts = kFar + sizeof(WalkFar) / 4;
  WalkFar *far() const { return reinterpret_cast<WalkFar *>(counts.ptr + kFar); }
  static unsigned grid(DeviceContext *ctx, uint64_t threads) {
    const uint64_t most = (uint64_t)ctx->sm_count * 32, g = ceil_div(threads, kWalkBlock);
    return (unsigned)(g == 0 ? 1 : g < most ? g : most);
  }
  // Room for `most` entries of a graph that walk_form has walked.
  int alloc(DeviceContext *ctx, cudaStream_t st, uint64_t n_, uint64_t m_, uint64_t long_rows,
            uint64_t longest, uint64_t most) {
    n = n_;
    m = m_;
    rows = long_rows;
    bits = walk_bits(m, rows, longest);
    cap = walk_room(most);
    const uint64_t room = walk_room(2 * rows);
    WETRIC_TRY(split.alloc(ctx, st, n));
    WETRIC_TRY(keys.alloc(ctx, st, cap));
    WETRIC_TRY(alt.alloc(ctx, st, cap));
    WETRIC_TRY(counts.alloc(ctx, st, kCounts));
    WETRIC_CUDA_TRY(cudaMemsetAsync(counts.ptr, 0, kCounts * sizeof(uint32_t), st));
    big_cap = walk_most_items(cap, m, false);
    WETRIC_TRY(start.alloc(ctx, st, room + 1));
    WETRIC_TRY(small.alloc(ctx, st, room));
    WETRIC_TRY(ws.alloc(ctx, st, cap));
    return big.alloc(ctx, st, big_cap);
  }
  // Rows of several sets will be shared out (before sort); not without room
  // for their items.
  void share(DeviceContext *ctx, cudaStream_t st) {
    Scratch<uint2> more;
    if (more.alloc(ctx, st, walk_most_items(cap, m, true)) != WETRIC_OK) {
      clear_error();
      return;
    }
    big.release();
    big.ctx = more.ctx;
    big.stream = more.stream;
    big.bytes = more.bytes;
    big.ptr = more.detach();
    share_sets = true;
    big_cap = walk_most_items(cap, m, true);
  }
  // The entries made, sorted by middle vertex, and the work items.
  int sort(DeviceContext *ctx, cudaStream_t st, const uint32_t *rp, const uint32_t *long_rows,
           uint64_t made, uint32_t *err, uint32_t *launches) {
    entries = made;
    const prim::KeysFrom from{keys.ptr};
    uint64_t *to = prim::sorted_buffer(alt.ptr, keys.ptr, bits.shift(), bits.w);
    WETRIC_TRY((prim::radix_sort_into(ctx, st, from, from, alt.ptr, keys.ptr, prim::KeysTo{to},
                                      entries, bits.shift(), bits.w, err, &ws)));
    sorted = to;
    k_walk_starts<<<grid(ctx, entries), kWalkBlock, 0, st>>>(
        sorted, (uint32_t)entries, (uint32_t)(2 * rows), bits.shift(), start.ptr, err);
    WETRIC_LAUNCH_CHECK();
    k_walk_plan<<<grid(ctx, 2 * rows), kWalkBlock, 0, st>>>(
        rp, split.ptr, long_rows, start.ptr, (uint32_t)(2 * rows), big.ptr, small.ptr,
        counts.ptr + 1, share_sets, err);
    WETRIC_LAUNCH_CHECK();
    *launches += 3 + prim::digit_plan(bits.shift(), bits.w).passes;
    return WETRIC_OK;
  }
  // The count. Persistent: one wave of blocks, items from a counter; otherwise
  // short blocks, so other streams' blocks get SMs in between. The counters
  // start at zero (alloc) and are the caller's to clear for another count.
  template <bool kBatch = false>
  int count(DeviceContext *ctx, cudaStream_t st, const uint32_t *rp, const uint32_t *ci,
            const uint32_t *long_rows, bool persistent, unsigned long long *out, const uint32_t *err,
            uint64_t *most, uint32_t *launches, const WalkGroups &groups = WalkGroups{},
            const uint32_t *long_graph = nullptr) {
    // Items per block when blocks are to be short (one pass): the last block is
    // the one with most work, so few, but not a block each (1.5e6 at scale 22).
    // R-MAT scale 18 / 20 / 22 in us: 16 items 793 / 1890 / 6455, 4 574 / 1636 /
    // 6101, 1 561 / 1739 / 6925; from a counter 540 / 1548 / 5900.
    constexpr uint32_t kPerBlock = 4;
    const auto big_fn = !kBatch && share_sets
                            ? k_walk_count<kWalkBigBlock, kWalkBigBlocks, kBatch, !kBatch>
                            : k_walk_count<kWalkBigBlock, kWalkBigBlocks, kBatch>;
    const auto small_fn = k_walk_count<kWalkSmallBlock, kWalkSmallBlocks, kBatch>;
    const uint64_t g = persistent ? (uint64_t)ctx->sm_count * kWalkBigBlocks
                                  : ceil_div(big_cap, kPerBlock);
    const uint64_t gs = persistent ? (uint64_t)ctx->sm_count * kWalkSmallBlocks
                                   : ceil_div(2 * rows, kPerBlock);
    const WalkColumns cols = walk_columns(ci, m);
    const uint32_t t0 = n > kWalkWindow ? (uint32_t)(n - kWalkWindow) : 0u;
    // The sector loads need L1 lines for the data in flight: with the shared
    // memory of as many blocks as fit (218 KB) about 80 lines were left and
    // the kernel ran at 1.2 TB/s of sectors.
    WETRIC_CUDA_TRY(cudaFuncSetAttribute(
        big_fn, cudaFuncAttributePreferredSharedMemoryCarveout, kWalkCarveout));
    WETRIC_CUDA_TRY(cudaFuncSetAttribute(
        small_fn, cudaFuncAttributePreferredSharedMemoryCarveout, kWalkCarveout));
    big_fn<<<(unsigned)g, kWalkBigBlock, 0, st>>>(
        rp, split.ptr, long_rows, cols, t0, sorted, start.ptr, bits, big.ptr, counts.ptr + 1,
        counts.ptr + 3, persistent ? 0 : kPerBlock, out, groups, long_graph, err);
    WETRIC_LAUNCH_CHECK();
    small_fn<<<(unsigned)gs, kWalkSmallBlock, 0, st>>>(
        rp, split.ptr, long_rows, cols, t0, sorted, start.ptr, bits, small.ptr, counts.ptr + 2,
        counts.ptr + 4, persistent ? 0 : kPerBlock, out, groups, long_graph, err);
    WETRIC_LAUNCH_CHECK();
    *launches += 2;
    if (g > *most) *most = g;
    return WETRIC_OK;
  }
};

}  // namespace
}  // namespace wetric
