// primitives.cuh -- device-wide exclusive scan and stable LSD radix sort,
// written for this library in place of the CUB calls of the reference
// (DeviceRadixSort / DeviceSegmentedSort, tc.cu:500-558).
//
// Both are single pass over the data per step: a block takes its tile from a
// ticket counter, publishes its totals and looks back over its
// predecessors' published totals for its offset ("decoupled look-back",
// Merrill and Garland, "Single-pass parallel prefix scan with decoupled
// look-back", 2016; for the sort, Adinets and Merrill, "Onesweep", 2022).
// Tickets are handed out in order to running blocks, so a block only ever
// waits on blocks that are already running. Every wait is bounded all the
// same: on running out it records kDevLookbackTimeout, publishes a poison
// word that ends its successors' waits, and the block leaves. What such a
// pass leaves is not complete, and kernels behind it may be queued already:
// those that index with it look at the error word first and leave. In a pass
// with a look-back the first tile looks: every other one waits for a word
// that follows from the first's, so its poison keeps all of them from writing
// (orientation of R-MAT scale 22: without any look 7.03-7.07 ms, this way
// 7.08, by every block 7.12).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace wetric {
namespace prim {

// Published words: value in the low 48 bits, (epoch << 2 | flag) above it.
// A word of another epoch reads as "not published yet", so one clearing of
// the words serves every pass of a sort. 48 bits hold any number of keys,
// rows or columns; the wedge prefixes are 64 bits wide (one row of 2^25
// columns has 2^49 wedges) and take two words, each with its flag, when they
// pass 48: the low 48 bits with epoch kTileMore, and the rest (tile_rest). Every
// word is written once per flag, so two words with the same flag are of one
// value. (Two words for every value: a count of a wedge range of 10,000,000
// vertices 635 us, this way 620.)
constexpr uint32_t kTileAgg = 1, kTileIncl = 2, kTilePoison = 3;
constexpr uint64_t kTileValueMask = (1ull << 48) - 1;
constexpr uint32_t kTileMore = 1;  // an epoch of wide scans
constexpr uint32_t kLookbackSpins = 1u << 22;

__host__ __device__ __forceinline__ uint64_t tile_word(uint32_t epoch, uint32_t flag,
                                                       uint64_t value) {
  return ((uint64_t)(epoch << 2 | flag) << 48) | (value & kTileValueMask);
}
__host__ __device__ __forceinline__ uint32_t tile_flag(uint64_t w, uint32_t epoch) {
  const uint32_t tag = (uint32_t)(w >> 48);
  return (tag >> 2) == epoch ? (tag & 3u) : 0u;
}
// The second word of a 64-bit value, and the flag and value of a pair: no
// flag while the two differ, poison as soon as one has it.
__host__ __device__ __forceinline__ uint64_t tile_rest(uint32_t flag, uint64_t value) {
  return tile_word(0, flag, value >> 48);
}
__host__ __device__ __forceinline__ uint32_t tile_pair_flag(uint64_t w, uint64_t rest) {
  const uint32_t a = tile_flag(w, 0), b = tile_flag(rest, 0);
  return a == kTilePoison || b == kTilePoison ? kTilePoison : a == b ? a : 0u;
}
__host__ __device__ __forceinline__ uint64_t tile_pair_value(uint64_t w, uint64_t rest) {
  return (w & kTileValueMask) | (rest << 48);
}
__device__ __forceinline__ uint64_t ld_tile(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_tile(uint64_t *p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Exclusive prefix of `agg` over the tiles before `tile` (a whole warp
// calls it; one word per tile, with kWide another in rest for a value past 48
// bits). A step looks at 128 predecessors, four per lane: all tiles of a short
// scan start together, so the last one walks back over all of them. Returns false when a wait ran out.
constexpr int kLookWide = 4;
template <bool kWide>
__device__ __forceinline__ bool tile_prefix(uint64_t *state, uint64_t *rest, uint64_t tile,
                                            uint64_t agg, uint32_t *err, uint64_t *excl) {
  const uint32_t lane = threadIdx.x & 31;
  auto publish = [&](uint32_t flag, uint64_t value) {
    if (lane != 0) return;
    const bool more = kWide && value > kTileValueMask;
    if (more) st_tile(rest + tile, tile_rest(flag, value));
    st_tile(state + tile, tile_word(more ? kTileMore : 0, flag, value));
  };
  *excl = 0;
  if (tile == 0) {
    uint32_t on = 1;
    if (lane == 0) on = *err == kDevOk;
    on = __shfl_sync(0xffffffffu, on, 0);
    publish(on ? kTileIncl : kTilePoison, agg);
    return on;
  }
  publish(kTileAgg, agg);
  uint64_t sum = 0;
  for (int64_t hi = (int64_t)tile - 1;; hi -= 32 * kLookWide) {
    // word j of the lane: predecessor j * 32 + lane of the window
    uint64_t w[kLookWide];
    uint32_t flag[kLookWide], spins = 0;
    bool bad = false;
    for (;;) {
      bool ready = true;
#pragma unroll
      for (int j = 0; j < kLookWide; ++j) {
        const int64_t at = hi - j * 32 - lane;
        w[j] = at >= 0 ? ld_tile(state + at) : tile_word(0, kTileIncl, 0);
      }
#pragma unroll
      for (int j = 0; j < kLookWide; ++j) {
        flag[j] = tile_flag(w[j], 0);
        if (!kWide) continue;
        uint64_t r = 0;
        if (tile_flag(w[j], kTileMore)) {
          r = ld_tile(rest + hi - j * 32 - lane);
          flag[j] = tile_pair_flag(w[j] ^ tile_word(kTileMore, 0, 0), r);
        }
        w[j] = tile_pair_value(w[j], r);
      }
#pragma unroll
      for (int j = 0; j < kLookWide; ++j) {
        ready = ready && flag[j] != 0;
        bad = bad || flag[j] == kTilePoison;
      }
      if (__any_sync(0xffffffffu, bad) || __all_sync(0xffffffffu, ready)) break;
      if (++spins > kLookbackSpins) {
        bad = true;
        break;
      }
    }
    if (__any_sync(0xffffffffu, bad)) {
      if (lane == 0) {
        atomicCAS(err, 0u, (uint32_t)kDevLookbackTimeout);
        publish(kTilePoison, 0);
      }
      return false;
    }
    // up to the nearest inclusive word
    bool found = false;
    uint64_t v = 0;
#pragma unroll
    for (int j = 0; j < kLookWide; ++j) {
      const uint32_t incl = __ballot_sync(0xffffffffu, flag[j] == kTileIncl);
      const uint32_t last = incl ? __ffs(incl) - 1 : 31;
      if (!found && lane <= last) v += kWide ? w[j] : w[j] & kTileValueMask;
      found = found || incl;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    sum += v;
    if (found) break;
  }
  publish(kTileIncl, sum + agg);
  *excl = sum;
  return true;
}

// Inclusive scan of one value per thread across a block of kThreads.
// Returns the inclusive prefix; *total receives the block total. smem_warp
// holds kThreads / 32 values.
template <int kThreads, typename T>
__device__ __forceinline__ T block_inclusive_scan(T v, T *smem_warp, T *total) {
  constexpr int kWarps = kThreads / 32;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) smem_warp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    T w = lane < kWarps ? smem_warp[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kWarps) smem_warp[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v += smem_warp[warp - 1];
  *total = smem_warp[kWarps - 1];
  return v;
}

// ------------------------------------------------------------------- scan

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanChunk = kScanThreads * kScanItems;
// A 64-bit input is summed in 64 bits (wedges); 32-bit ones are flags,
// buckets or columns, whose sums stay below 2^48.
template <typename InT>
constexpr bool kScanWide = sizeof(InT) == 8;

// out[i] = exclusive prefix of in, out[n] = total, in one pass, the tile's
// offset by look-back (state null: a single tile). Item j of lane l is
// element j * 32 + l of the warp's 512, so loads and stores are whole lines
// and each item is a warp scan on top of the last one's total. Bound
// by the latency of the look-back (4.2M u32 -> u64: 27 us): on the device
// it takes as long as the reduce, scan and apply launches it replaces, and
// saves the host two launches of three. Four blocks per SM: the 64-bit form
// took 128 registers, and a wedge range of 10,000,000 vertices 620 us with two
// blocks, 530 with four.
template <typename InT, typename OutT>
__global__ void __launch_bounds__(kScanThreads, 4)
    k_scan(const InT *in, uint64_t n, OutT *out, uint64_t *state, uint64_t *rest,
           uint32_t *ticket, uint32_t *err) {
  __shared__ OutT s_warp[kScanThreads / 32];
  __shared__ uint64_t s_excl;
  __shared__ uint32_t s_tile, s_ok;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t tile = 0;
  if (state) {
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    tile = s_tile;
  }
  const uint64_t base = tile * kScanChunk + (uint64_t)warp * 32 * kScanItems + lane;
  OutT vals[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = base + (uint64_t)j * 32;
    vals[j] = i < n ? (OutT)in[i] : OutT(0);
  }
  OutT run = 0;  // of the warp's items so far
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    OutT x = vals[j];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const OutT y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    vals[j] = run + x - vals[j];
    run += __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) s_warp[warp] = run;
  __syncthreads();
  OutT off = 0, total = 0;
#pragma unroll
  for (uint32_t w = 0; w < kScanThreads / 32; ++w) {
    if (w < warp) off += s_warp[w];
    total += s_warp[w];
  }
  uint64_t before = 0;
  if (state) {
    if (warp == 0) {
      uint64_t excl = 0;
      const bool ok = tile_prefix<kScanWide<InT>>(state, rest, tile, (uint64_t)total, err, &excl);
      if (lane == 0) {
        s_excl = excl;
        s_ok = ok;
      }
    }
    __syncthreads();
    if (!s_ok) return;
    before = s_excl;
  }
  off += (OutT)before;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = base + (uint64_t)j * 32;
    if (i < n) out[i] = off + vals[j];
  }
  if (threadIdx.x == 0 && (tile + 1) * kScanChunk >= n) out[n] = (OutT)before + total;
}

// out[0..n] = exclusive prefix of in[0..n-1]; out[n] = total. out may alias
// in when InT == OutT (a tile reads its items before it writes them). A
// look-back that runs out is recorded in *err (device).
template <typename InT, typename OutT>
int exclusive_scan(DeviceContext *ctx, cudaStream_t st, const InT *in,
                   OutT *out, uint64_t n, uint32_t *err) {
  const uint64_t tiles = n == 0 ? 1 : ceil_div(n, kScanChunk);
  if (tiles == 1) {
    k_scan<InT, OutT><<<1, kScanThreads, 0, st>>>(in, n, out, nullptr, nullptr, nullptr, err);
    WETRIC_LAUNCH_CHECK();
    return WETRIC_OK;
  }
  Scratch<uint64_t> state;  // [0] the ticket, then one or two words per tile
  const uint64_t words = 1 + (kScanWide<InT> ? 2 : 1) * tiles;
  WETRIC_TRY(state.alloc(ctx, st, words));
  WETRIC_CUDA_TRY(cudaMemsetAsync(state.ptr, 0, words * sizeof(uint64_t), st));
  k_scan<InT, OutT><<<(unsigned)tiles, kScanThreads, 0, st>>>(
      in, n, out, state.ptr + 1, state.ptr + 1 + tiles, reinterpret_cast<uint32_t *>(state.ptr),
      err);
  WETRIC_LAUNCH_CHECK();
  return WETRIC_OK;
}

// ------------------------------------------------------------ radix sort

constexpr int kSortThreads = 384;
constexpr int kSortBlocks = 3;  // per SM
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;  // per thread
// Few keys: a pass is one block's latency, and a tile of a quarter shortens
// it while every tile still has an SM and the look-back stays short
// (orientation of 2,000 pairs 162 -> 149 us, of 200,000 221 -> 197 us; with
// 4 tiles per SM 400,000 pairs took 247 us against 243). Its 27 KB of shared memory
// also fit beside the resident serving kernel, whose SMs keep the
// shared-memory split they were started with: a large tile could wait there
// until that kernel ended.
constexpr int kSortFewItems = 4;
constexpr uint64_t kSortFewTiles = 148;  // the B200's SMs
constexpr uint64_t kSortFewKeys = kSortFewTiles * kSortThreads * kSortFewItems;
// Most tiles of a sort of up to n keys.
inline uint64_t sort_tiles(uint64_t n) {
  if (n <= kSortFewKeys) return ceil_div(n, kSortThreads * kSortFewItems);
  const uint64_t tiles = ceil_div(n, kSortThreads * kSortItems);
  return tiles > kSortFewTiles ? tiles : kSortFewTiles;
}
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kMaxPasses = 8;

// The passes of a sort over `bits` key bits from bit `lo`: as few as
// 8-bit digits allow, of even widths (narrow digits make longer runs).
struct DigitPlan {
  uint32_t passes;
  uint32_t shift[kMaxPasses], bits[kMaxPasses];
};
inline DigitPlan digit_plan(uint32_t lo, uint32_t bits) {
  DigitPlan p{};
  p.passes = (bits + kRadixBits - 1) / kRadixBits;
  uint32_t at = lo;
  for (uint32_t i = 0; i < p.passes; ++i) {
    p.bits[i] = (lo + bits - at + (p.passes - i) - 1) / (p.passes - i);
    p.shift[i] = at;
    at += p.bits[i];
  }
  return p;
}

// Where a pass takes its keys from and what it does with each at its sorted
// position.
struct KeysFrom {
  const uint64_t *__restrict__ keys;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const { return keys[i]; }
};
struct KeysTo {
  uint64_t *__restrict__ keys;
  __device__ __forceinline__ void operator()(uint64_t i, uint64_t k) const { keys[i] = k; }
};

// Histograms of every digit in one read of the keys (bound by the
// shared-memory atomics: 0.26 ms for 67M keys of six digits). Four copies per block
// in shared memory (lane & 3 picks one), since the digits of graph keys are
// skewed and a warp's equal digits serialise on one counter.
constexpr int kHistCopies = 4;
constexpr int kHistAhead = 4;
template <class Load>
__global__ void __launch_bounds__(256)
    k_radix_hist(Load load, uint64_t n, const __grid_constant__ DigitPlan plan,
                 unsigned long long *__restrict__ hist, const uint32_t *err) {
  extern __shared__ uint32_t s_hist[];  // [pass][digit][copy]
  const uint32_t total = plan.passes * kRadix * kHistCopies;
  for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) s_hist[i] = 0;
  // (load itself may set the word, hence one verdict per block)
  if (__syncthreads_or(*err != kDevOk)) return;
  const uint32_t copy = threadIdx.x & (kHistCopies - 1);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto add = [&](uint64_t k) {
#pragma unroll
    for (int p = 0; p < kMaxPasses; ++p)
      if (p < plan.passes) {
        const uint32_t d = (uint32_t)(k >> plan.shift[p]) & ((1u << plan.bits[p]) - 1u);
        atomicAdd(&s_hist[(p * kRadix + d) * kHistCopies + copy], 1u);
      }
  };
  // several keys' loads in flight per thread
  for (; i + (kHistAhead - 1) * stride < n; i += kHistAhead * stride) {
    uint64_t k[kHistAhead];
#pragma unroll
    for (int j = 0; j < kHistAhead; ++j) k[j] = load(i + j * stride);
#pragma unroll
    for (int j = 0; j < kHistAhead; ++j) add(k[j]);
  }
  for (; i < n; i += stride) add(load(i));
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < plan.passes * kRadix; i += blockDim.x) {
    uint32_t c = 0;
#pragma unroll
    for (int j = 0; j < kHistCopies; ++j) c += s_hist[i * kHistCopies + j];
    if (c) atomicAdd(&hist[i], (unsigned long long)c);
  }
}

// The digit of a key: bits [shift, shift + kBits) of its 64, masked to the
// pass's width. kHigh: shift >= 32.
template <bool kHigh>
__device__ __forceinline__ uint32_t key_digit(uint64_t k, uint32_t shift, uint32_t mask) {
  const uint32_t lo = (uint32_t)k, hi = (uint32_t)(k >> 32);
  return (kHigh ? hi >> (shift - 32) : __funnelshift_r(lo, hi, shift)) & mask;
}

// Lanes of `valid` with the same digit, by one ballot per digit bit: the
// cost does not depend on the digits (match.any took two to three times as
// long on digits with many values as on skewed ones).
template <int kBits>
__device__ __forceinline__ uint32_t match_digit(uint32_t d, uint32_t valid) {
  uint32_t m = valid;
#pragma unroll
  for (int b = 0; b < kBits; ++b) {
    const bool bit = (d >> b) & 1u;
    const uint32_t bal = __ballot_sync(0xffffffffu, bit);
    m &= bit ? bal : ~bal;
  }
  return m;
}

// One pass: a block ranks its tile's keys by digit (warp w owns the
// contiguous keys [w*32*Items, +32*Items) of the tile, item j of lane l is
// key j*32 + l of them, so (warp, item, lane) is the input order and the
// sort is stable), publishes the tile's digit counts, orders the keys in
// shared memory, finds each digit's global offset by look-back (thread d
// walks digit d, four predecessors at a time) and writes whole runs. Bound
// by instruction issue (about 100 warp instructions per 32 keys, a third of
// them the ballots): 0.36 ms per pass of 64M keys, 8-bit digits, where the
// histogram, scan and scatter it replaces took 0.6-0.8 ms with scattered
// 8-byte stores. Tile shape from a sweep at 64M 44-bit keys, whole sort: 384
// threads x 16 keys x 3 blocks 2.46 ms, 512 x 16 x 2 2.48, 256 x 16 x 4 2.84,
// 1024 x 12 x 1 2.97, 512 x 8 x 3 2.92; five 9-bit passes 2.61 (512 x 16).
constexpr size_t sort_smem(int items) {
  return kSortThreads * items * sizeof(uint64_t) + kSortWarps * kRadix * sizeof(uint32_t) +
         kRadix * (sizeof(uint64_t) + sizeof(uint32_t));
}
constexpr int kLookAhead = 4;
template <int kBits, bool kHigh, int kItems, class Load, class Sink>
__global__ void __launch_bounds__(kSortThreads, kSortBlocks)
    k_onesweep(Load load, Sink sink, uint64_t n, uint32_t shift, uint32_t bits, uint32_t epoch,
               const unsigned long long *__restrict__ hist, uint64_t *__restrict__ state,
               uint32_t *__restrict__ ticket, uint32_t *err) {
  constexpr int kTile = kSortThreads * kItems;
  static_assert(kSortThreads >= kRadix, "thread d owns digit d");
  extern __shared__ __align__(16) unsigned char s_raw[];
  uint64_t *s_key = reinterpret_cast<uint64_t *>(s_raw);
  uint64_t *s_goff = s_key + kTile;
  uint32_t *s_toff = reinterpret_cast<uint32_t *>(s_goff + kRadix);
  uint32_t *s_whist = s_toff + kRadix;
  __shared__ uint32_t s_warp[kSortWarps];
  __shared__ unsigned long long s_warp64[kSortWarps];
  __shared__ uint32_t s_ticket, s_bad;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    s_ticket = atomicAdd(ticket, 1u);
    s_bad = 0;
  }
  for (uint32_t i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads) s_whist[i] = 0;
  __syncthreads();
  const uint64_t tile = s_ticket;
  const uint64_t base = tile * kTile;
  const uint32_t count = n - base < kTile ? (uint32_t)(n - base) : kTile;
  const uint32_t mask = (1u << bits) - 1u;
  const uint32_t sub = warp * 32 * kItems + lane;
  uint32_t *wh = s_whist + warp * kRadix;
  uint64_t k[kItems];
  uint16_t rank[kItems];  // below 32 * kItems
  const uint32_t lt = (1u << lane) - 1u;
  if (count == kTile) {
#pragma unroll
    for (int j = 0; j < kItems; ++j) k[j] = load(base + sub + j * 32);
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t d = key_digit<kHigh>(k[j], shift, mask);
      const uint32_t peers = match_digit<kBits>(d, 0xffffffffu);
      const uint32_t leader = __ffs(peers) - 1;
      uint32_t before = 0;
      if (lane == leader) before = atomicAdd(&wh[d], (uint32_t)__popc(peers));
      rank[j] = (uint16_t)(__shfl_sync(0xffffffffu, before, leader) + __popc(peers & lt));
    }
  } else {
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      k[j] = sub + j * 32 < count ? load(base + sub + j * 32) : 0;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const bool valid = sub + j * 32 < count;
      const uint32_t d = key_digit<kHigh>(k[j], shift, mask);
      const uint32_t peers = match_digit<kBits>(d, __ballot_sync(0xffffffffu, valid));
      const uint32_t leader = valid ? __ffs(peers) - 1 : lane;
      uint32_t before = 0;
      if (valid && lane == leader) before = atomicAdd(&wh[d], (uint32_t)__popc(peers));
      rank[j] = (uint16_t)(__shfl_sync(0xffffffffu, before, leader) + __popc(peers & lt));
    }
  }
  __syncthreads();
  // digit d's count in the tile, its warps' offsets within it
  uint32_t c = 0;
  if (threadIdx.x < kRadix) {
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t x = s_whist[w * kRadix + threadIdx.x];
      s_whist[w * kRadix + threadIdx.x] = c;
      c += x;
    }
  }
  uint64_t *word = state + tile * kRadix + threadIdx.x;
  if (threadIdx.x < kRadix && tile > 0) st_tile(word, tile_word(epoch, kTileAgg, c));
  uint32_t total;
  const uint32_t incl = block_inclusive_scan<kSortThreads, uint32_t>(c, s_warp, &total);
  if (threadIdx.x < kRadix) s_toff[threadIdx.x] = incl - c;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    if (sub + j * 32 < count) {
      const uint32_t d = key_digit<kHigh>(k[j], shift, mask);
      s_key[s_toff[d] + wh[d] + rank[j]] = k[j];
    }
  }
  if (tile == 0) {
    // the first tile's inclusive words carry the digits' global starts
    unsigned long long t64;
    const unsigned long long h = threadIdx.x < kRadix ? hist[threadIdx.x] : 0;
    const unsigned long long i64 =
        block_inclusive_scan<kSortThreads, unsigned long long>(h, s_warp64, &t64);
    if (threadIdx.x < kRadix) {
      const bool on = *err == kDevOk;  // else the keys may not be there
      st_tile(word, tile_word(epoch, on ? kTileIncl : kTilePoison, i64 - h + c));
      s_goff[threadIdx.x] = i64 - h - (incl - c);
      if (!on) s_bad = 1;
    }
  } else if (threadIdx.x < kRadix) {
    uint64_t sum = 0;
    uint32_t spins = 0, done = 0;  // done: 1 = reached an inclusive word, 2 = gave up
    for (uint64_t at = tile; !done;) {
      // the words of the kLookAhead tiles before `at` (tile 0's is inclusive)
      uint64_t w[kLookAhead];
#pragma unroll
      for (int j = 0; j < kLookAhead; ++j) {
        const uint64_t q = at > (uint64_t)j ? at - 1 - j : 0;
        w[j] = ld_tile(state + q * kRadix + threadIdx.x);
      }
#pragma unroll
      for (int j = 0; j < kLookAhead; ++j) {
        const uint32_t f = tile_flag(w[j], epoch);
        if (f == 0) {
          if (++spins > kLookbackSpins) done = 2;
          break;
        }
        if (f == kTilePoison) {
          done = 2;
          break;
        }
        sum += w[j] & kTileValueMask;
        --at;
        if (f == kTileIncl) {
          done = 1;
          break;
        }
      }
    }
    if (done == 2) {
      atomicCAS(err, 0u, (uint32_t)kDevLookbackTimeout);
      s_bad = 1;
      st_tile(word, tile_word(epoch, kTilePoison, 0));
    } else {
      st_tile(word, tile_word(epoch, kTileIncl, sum + c));
      s_goff[threadIdx.x] = sum - (incl - c);
    }
  }
  __syncthreads();
  if (s_bad) return;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < count; i += kSortThreads) {
    const uint64_t key = s_key[i];
    sink(s_goff[key_digit<kHigh>(key, shift, mask)] + i, key);
  }
}

// Workspace of one sort of up to n keys, cleared: the digits' histograms, the
// passes' tickets and the look-back words. A part of a larger one (at), or
// its own (alloc).
struct SortSpace {
  Scratch<uint64_t> buf;
  unsigned long long *hist = nullptr;
  uint32_t *tickets = nullptr;
  uint64_t *state = nullptr;
  static constexpr uint64_t kHead = (uint64_t)kMaxPasses * kRadix + kMaxPasses;
  static uint64_t words(uint64_t n) { return kHead + sort_tiles(n) * kRadix; }
  void at(uint64_t *p) {
    hist = reinterpret_cast<unsigned long long *>(p);
    tickets = reinterpret_cast<uint32_t *>(p + kMaxPasses * kRadix);
    state = p + kHead;
  }
  int alloc(DeviceContext *ctx, cudaStream_t st, uint64_t n) {
    WETRIC_TRY(buf.alloc(ctx, st, words(n)));
    WETRIC_CUDA_TRY(cudaMemsetAsync(buf.ptr, 0, words(n) * sizeof(uint64_t), st));
    at(buf.ptr);
    return WETRIC_OK;
  }
};

template <int kBits, bool kHigh, int kItems, class Load, class Sink>
int onesweep_launch(cudaStream_t st, const Load &load, const Sink &sink, uint64_t n,
                    const DigitPlan &plan, uint32_t p, const SortSpace &ws, uint32_t *err) {
  const auto fn = k_onesweep<kBits, kHigh, kItems, Load, Sink>;
  constexpr size_t smem = sort_smem(kItems);
  if (smem > 48 * 1024)
    WETRIC_CUDA_TRY(
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  fn<<<(unsigned)ceil_div(n, kSortThreads * kItems), kSortThreads, smem, st>>>(
      load, sink, n, plan.shift[p], plan.bits[p], p + 1, ws.hist + (uint64_t)p * kRadix, ws.state,
      ws.tickets + p, err);
  WETRIC_LAUNCH_CHECK();
  return WETRIC_OK;
}

template <int kItems, class Load, class Sink>
int onesweep_items(cudaStream_t st, const Load &load, const Sink &sink, uint64_t n,
                   const DigitPlan &plan, uint32_t p, const SortSpace &ws, uint32_t *err) {
  const bool high = plan.shift[p] >= 32;
  if (plan.bits[p] > 7)
    return high ? onesweep_launch<8, true, kItems>(st, load, sink, n, plan, p, ws, err)
                : onesweep_launch<8, false, kItems>(st, load, sink, n, plan, p, ws, err);
  return high ? onesweep_launch<7, true, kItems>(st, load, sink, n, plan, p, ws, err)
              : onesweep_launch<7, false, kItems>(st, load, sink, n, plan, p, ws, err);
}

template <class Load, class Sink>
int onesweep_pass(cudaStream_t st, const Load &load, const Sink &sink, uint64_t n,
                  const DigitPlan &plan, uint32_t p, const SortSpace &ws, uint32_t *err) {
  return n <= kSortFewKeys
             ? onesweep_items<kSortFewItems>(st, load, sink, n, plan, p, ws, err)
             : onesweep_items<kSortItems>(st, load, sink, n, plan, p, ws, err);
}

// Loads the forms of a pass.
template <class Load, class Sink>
int load_onesweep() {
  return load_kernels({(const void *)k_onesweep<7, false, kSortItems, Load, Sink>,
                       (const void *)k_onesweep<7, true, kSortItems, Load, Sink>,
                       (const void *)k_onesweep<8, false, kSortItems, Load, Sink>,
                       (const void *)k_onesweep<8, true, kSortItems, Load, Sink>,
                       (const void *)k_onesweep<7, false, kSortFewItems, Load, Sink>,
                       (const void *)k_onesweep<7, true, kSortFewItems, Load, Sink>,
                       (const void *)k_onesweep<8, false, kSortFewItems, Load, Sink>,
                       (const void *)k_onesweep<8, true, kSortFewItems, Load, Sink>});
}

// Stable LSD sort of n keys on their bits [lo, lo + bits). `counted` gives
// the keys to the histogram pass (it may build and store them), `first` to
// the first pass, whose output goes to a; the passes then alternate between
// a and b, and the last one hands (position, key) to `sink`. Pass count:
// digit_plan(lo, bits).passes, at least 1 (bits >= 1). *err (device) receives
// a look-back that ran out. space: a workspace for n keys or more, fresh from
// alloc (none: the sort takes its own).
template <class Counted, class First, class Sink>
int radix_sort_into(DeviceContext *ctx, cudaStream_t st, const Counted &counted,
                    const First &first, uint64_t *a, uint64_t *b, const Sink &sink, uint64_t n,
                    uint32_t lo, uint32_t bits, uint32_t *err, const SortSpace *space = nullptr) {
  if (n == 0) return WETRIC_OK;
  const DigitPlan plan = digit_plan(lo, bits ? bits : 1);
  SortSpace own;
  if (!space) WETRIC_TRY(own.alloc(ctx, st, n));
  const SortSpace &ws = space ? *space : own;
  uint64_t blocks = ceil_div(n, 256 * (n <= kSortFewKeys ? kSortFewItems : kSortItems));
  const uint64_t cap = (uint64_t)ctx->sm_count * 8;
  if (blocks > cap) blocks = cap;
  const size_t hs = (size_t)plan.passes * kRadix * kHistCopies * sizeof(uint32_t);
  k_radix_hist<Counted><<<(unsigned)blocks, 256, hs, st>>>(counted, n, plan, ws.hist, err);
  WETRIC_LAUNCH_CHECK();
  if (plan.passes == 1) return onesweep_pass(st, first, sink, n, plan, 0, ws, err);
  WETRIC_TRY((onesweep_pass(st, first, KeysTo{a}, n, plan, 0, ws, err)));
  uint64_t *from = a, *to = b;
  for (uint32_t p = 1; p + 1 < plan.passes; ++p) {
    WETRIC_TRY((onesweep_pass(st, KeysFrom{from}, KeysTo{to}, n, plan, p, ws, err)));
    uint64_t *x = from;
    from = to;
    to = x;
  }
  return onesweep_pass(st, KeysFrom{from}, sink, n, plan, plan.passes - 1, ws, err);
}

// The buffer (a or b) that the sort above leaves its keys in when the last
// sink is KeysTo: the one its last pass does not read.
inline uint64_t *sorted_buffer(uint64_t *a, uint64_t *b, uint32_t lo, uint32_t bits) {
  return digit_plan(lo, bits ? bits : 1).passes % 2 == 1 ? a : b;
}

}  // namespace prim
}  // namespace wetric
