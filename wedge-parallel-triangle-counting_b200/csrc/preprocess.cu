// preprocess.cu -- device-side graph preprocessing.
//
// The reference builds its CSR on the host: symmetrise + drop self-loops
// (tc.cu:590-621), sort (CUB or qsort, 628-647), sequential dedup + row
// histogram (649-684), then relabels by ascending degree (688-723), keeps
// each edge once toward the higher new id (740-758) and sorts every row
// (763-784). Here all of that runs on the GPU with this library's own radix
// sort:
//
//   raw pairs --canonical (min,max) key--> sort --> unique + degrees
//     --> stable (degree, id) rank --> (rank lo, rank hi) key --> sort
//     --> oriented CSR (u64 row offsets, u32 columns)
//
// Keys pack two ids of b = bits(n-1) bits each into 2b bits, so a sort
// costs ceil(2b / 8) digit passes. Canonicalising to (min, max) before the
// first sort halves the keys compared with the reference's symmetrised
// list. The passes take their keys where they arise (the degree sort reads
// the degrees, the symmetric sort the unique keys, without an unsorted copy);
// the raw pairs, which are the caller's, are read once. The vertex order equals
// that of the reference's stable CUB sort (its -p 1 / -p 2 styles):
// ascending degree, ties by ascending id.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "common.cuh"
#include "preprocess.cuh"
#include "primitives.cuh"
#include "readback.cuh"

namespace wetric {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ uint64_t pack_key(uint32_t lo, uint32_t hi,
                                             uint32_t b) {
  return ((uint64_t)lo << b) | (uint64_t)hi;
}

__global__ void k_max_id(const uint32_t *__restrict__ src,
                         const uint32_t *__restrict__ dst, uint64_t P,
                         uint32_t *max_id, uint32_t *any_edge) {
  uint32_t local = 0, seen = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t s = src[i], d = dst[i];
    if (s != d) {
      local = max(local, max(s, d));
      seen = 1;
    }
  }
  local = __reduce_max_sync(0xffffffffu, local);
  seen = __reduce_or_sync(0xffffffffu, seen);
  if ((threadIdx.x & 31) == 0) {
    if (seen) {
      atomicMax(max_id, local);
      atomicOr(any_edge, 1u);
    }
  }
}

// Keys of the raw pairs: (min, max) packed, or the all-ones sentinel for a
// self-loop or an id >= n (which raises *err), made and stored while their
// digits are counted. The caller's arrays are read this once: a sort whose
// passes read them again would write past its buffers if another stream or
// thread changed them in between (counts and keys would not agree). R-MAT
// scale 22: 7.12 ms for the orientation, 7.02 with the pairs read twice.
struct CanonPairs {
  const uint32_t *__restrict__ src, *__restrict__ dst;
  uint64_t *__restrict__ out;
  uint32_t b;
  uint64_t n, sentinel;
  uint32_t *err;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const {
    const uint32_t s = __ldg(src + i), d = __ldg(dst + i);
    const uint32_t lo = min(s, d), hi = max(s, d);
    if (s != d && (uint64_t)hi >= n) atomicCAS(err, 0u, (uint32_t)kDevColumnRange);
    const uint64_t k = s == d || (uint64_t)hi >= n ? sentinel : pack_key(lo, hi, b);
    out[i] = k;
    return k;
  }
};

// Sorted keys -> the unique ones (no sentinel) in order, their number, and
// the degree of every vertex, in one pass: a warp's keys are consecutive,
// the block's offset comes by look-back. deg[hi] takes one atomic per edge
// and deg[lo] one per run of equal lo in a warp's 32 keys (equal addresses
// serialise: with one atomic per edge each side, in a kernel of its own
// after two more passes over the keys, this took 2.16 + 0.69 ms on R-MAT
// scale 22; now 0.77 ms, bound by the atomics on deg[hi]).
constexpr int kUniqueItems = 16;
constexpr int kUniqueTile = kThreads * kUniqueItems;
__global__ void __launch_bounds__(kThreads)
    k_unique_degrees(const uint64_t *__restrict__ keys, uint64_t N, uint64_t sentinel,
                     uint32_t b, uint64_t *__restrict__ out, uint32_t *__restrict__ deg,
                     uint64_t *__restrict__ state, uint32_t *__restrict__ ticket,
                     uint64_t *__restrict__ m_out, uint32_t *err) {
  __shared__ uint32_t s_warp[kThreads / 32];
  __shared__ uint64_t s_excl;
  __shared__ uint32_t s_ticket, s_ok;
  if (threadIdx.x == 0) s_ticket = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint64_t tile = s_ticket;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t sub = tile * kUniqueTile + (uint64_t)warp * 32 * kUniqueItems;
  const uint64_t mask = (1ull << b) - 1;
  uint64_t k[kUniqueItems];
  uint32_t keep[kUniqueItems];
#pragma unroll
  for (int j = 0; j < kUniqueItems; ++j) {
    const uint64_t i = sub + (uint64_t)j * 32 + lane;
    k[j] = i < N ? keys[i] : sentinel;
  }
  // the key before the warp's first (any key but it when there is none)
  uint64_t last = sub > 0 && sub - 1 < N ? keys[sub - 1] : ~k[0];
  last = __shfl_sync(0xffffffffu, last, 0);
  uint32_t mine = 0;
#pragma unroll
  for (int j = 0; j < kUniqueItems; ++j) {
    uint64_t prev = __shfl_up_sync(0xffffffffu, k[j], 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(0xffffffffu, k[j], 31);
    keep[j] = __ballot_sync(0xffffffffu, k[j] != sentinel && k[j] != prev);
    mine += __popc(keep[j]);
  }
  if (lane == 0) s_warp[warp] = mine;
  __syncthreads();
  if (warp == 0) {
    const uint32_t c = lane < kThreads / 32 ? s_warp[lane] : 0u;
    const uint32_t total = __reduce_add_sync(0xffffffffu, c);
    uint64_t excl = 0;
    const bool ok = prim::tile_prefix<false>(state, nullptr, tile, total, err, &excl);
    if (lane == 0) {
      s_excl = excl;
      s_ok = ok;
      if (ok && (tile + 1) * kUniqueTile >= N) *m_out = excl + total;
    }
  }
  __syncthreads();
  if (!s_ok) return;
  uint64_t pos = s_excl;
  for (uint32_t w = 0; w < warp; ++w) pos += s_warp[w];
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < kUniqueItems; ++j) {
    const bool mykeep = (keep[j] >> lane) & 1u;
    const uint32_t lo = (uint32_t)(k[j] >> b);
    if (mykeep) {
      out[pos + __popc(keep[j] & lt)] = k[j];
      atomicAdd(&deg[(uint32_t)(k[j] & mask)], 1u);
    }
    pos += __popc(keep[j]);
    // runs of equal lo: the run's first lane adds its kept keys
    const uint32_t before = __shfl_up_sync(0xffffffffu, lo, 1);
    const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || lo != before);
    if ((heads >> lane) & 1u) {
      const uint32_t later = heads & ~(lt | (1u << lane));
      const uint32_t upto = later ? (1u << (__ffs(later) - 1)) - 1u : 0xFFFFFFFFu;
      const uint32_t c = __popc(keep[j] & upto & ~lt);
      if (c) atomicAdd(&deg[lo], c);
    }
  }
}

__global__ void __launch_bounds__(kThreads)
    k_max_u32(const uint32_t *__restrict__ a, uint64_t n, uint64_t *out) {
  uint32_t local = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    local = max(local, a[i]);
  local = __reduce_max_sync(0xffffffffu, local);
  __shared__ uint32_t s_max[kThreads / 32];
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < kThreads / 32; ++w) local = max(local, s_max[w]);
    atomicMax(reinterpret_cast<unsigned long long *>(out), (unsigned long long)local);
  }
}

// The degree sort's keys (degree above, id below: the ids ride along) and
// what it is for: rank[id] = position.
struct DegreeKeys {
  const uint32_t *__restrict__ deg;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const {
    return ((uint64_t)deg[i] << 32) | i;
  }
};
struct RankTo {
  uint32_t *__restrict__ rank;
  __device__ __forceinline__ void operator()(uint64_t i, uint64_t k) const {
    rank[(uint32_t)k] = (uint32_t)i;
  }
};

// Keys of the oriented edges, (rank lower, rank higher), made and stored
// while their digits are counted.
struct OrientedKeys {
  const uint64_t *__restrict__ keys;
  const uint32_t *__restrict__ rank;
  uint64_t *__restrict__ out;
  uint32_t b;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const {
    const uint64_t k = __ldg(keys + i);
    const uint32_t ra = __ldg(rank + (uint32_t)(k >> b));
    const uint32_t rb = __ldg(rank + (uint32_t)(k & ((1ull << b) - 1)));
    const uint64_t o = pack_key(min(ra, rb), max(ra, rb), b);
    out[i] = o;
    return o;
  }
};

// Both directions of every unique key.
struct BothDirections {
  const uint64_t *__restrict__ keys;
  uint32_t b;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const {
    const uint64_t k = keys[i >> 1];
    return (i & 1) ? pack_key((uint32_t)(k & ((1ull << b) - 1)), (uint32_t)(k >> b), b) : k;
  }
};

// Sorted (row, col) keys -> columns and row offsets in one pass: the offset
// of every row in (row of key i - 1, row of key i] is i. The rows before the
// first key's (isolated vertices come first in the degree order) and after
// the last key's are filled by the whole grid, which is sized for rows and
// keys; longer gaps in between by the whole block, but for the chunks of
// kGapChunk rows that lie inside one: a block each finds such a chunk's
// offset by bisection. (One block alone writes 60 GB/s: orienting 3 pairs among
// 50,000,000 ids took 7.1 ms with a grid sized for the keys, now 0.8; with
// 20,000,000 rows in between 5.6, now 3.1; R-MAT scale 22 is unchanged.)
// Replaces a histogram by one atomic per edge on the row
// (equal addresses for a whole row: 0.73 ms on R-MAT scale 22), a scan and
// a pass for the columns: 0.93 -> 0.24 ms there.
constexpr uint32_t kGapByThread = 8, kGapChunk = 65536;
__global__ void __launch_bounds__(kThreads)
    k_keys_to_csr(const uint64_t *__restrict__ keys, uint64_t m, uint64_t n, uint32_t b,
                  uint64_t *__restrict__ rp, uint32_t *__restrict__ ci,
                  const uint32_t *__restrict__ err) {
  if (*err != kDevOk) return;  // the keys may not be there
  __shared__ uint32_t s_from[kThreads], s_to[kThreads], s_gaps;
  const uint64_t mask = (1ull << b) - 1;
  const uint64_t gid = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * kThreads;
  const uint64_t first = keys[0] >> b, end = keys[m - 1] >> b;
  for (uint64_t r = gid; r <= first; r += stride) rp[r] = 0;
  for (uint64_t r = end + 1 + gid; r <= n; r += stride) rp[r] = m;
  for (uint64_t c = first / kGapChunk + 1 + blockIdx.x; (c + 1) * kGapChunk <= end + 1;
       c += gridDim.x) {
    uint64_t lo = 0, hi = m - 1;  // the first key of row c * kGapChunk or more
    while (lo < hi) {
      const uint64_t mid = lo + (hi - lo) / 2;
      if (keys[mid] >> b < c * kGapChunk) lo = mid + 1;
      else hi = mid;
    }
    if (keys[lo] >> b < (c + 1) * kGapChunk - 1) continue;
    for (uint32_t r = threadIdx.x; r < kGapChunk; r += kThreads) rp[c * kGapChunk + r] = lo;
  }
  for (uint64_t i0 = (uint64_t)blockIdx.x * kThreads; i0 < m; i0 += stride) {
    __syncthreads();
    if (threadIdx.x == 0) s_gaps = 0;
    __syncthreads();
    const uint64_t i = i0 + threadIdx.x;
    if (i < m) {
      const uint64_t k = keys[i];
      ci[i] = (uint32_t)(k & mask);
      if (i > 0) {
        const uint32_t row = (uint32_t)(k >> b), prev = (uint32_t)(keys[i - 1] >> b);
        if (row - prev <= kGapByThread) {
          for (uint32_t r = prev; r < row; ++r) rp[r + 1] = i;
        } else {
          const uint32_t g = atomicAdd(&s_gaps, 1u);
          s_from[g] = prev;
          s_to[g] = threadIdx.x;
        }
      }
    }
    __syncthreads();
    for (uint32_t g = 0; g < s_gaps; ++g) {
      const uint64_t at = i0 + s_to[g];
      const uint64_t from = (uint64_t)s_from[g] + 1, to = (keys[at] >> b) + 1;
      // without the whole chunks inside, which are filled already
      const uint64_t c0 = (from + kGapChunk - 1) / kGapChunk * kGapChunk;
      const uint64_t c1 = to / kGapChunk * kGapChunk;
      const uint64_t stop = c0 < c1 ? c0 : to;
      for (uint64_t r = from + threadIdx.x; r < stop; r += kThreads) rp[r] = at;
      if (c0 < c1)
        for (uint64_t r = c1 + threadIdx.x; r < to; r += kThreads) rp[r] = at;
    }
  }
}

// Degrees of a CSR given by row offsets (the reference's num_edges of
// preprocess_vertex_t, tc.cu:694).
__global__ void k_row_lengths(const uint64_t *__restrict__ rp, uint64_t n,
                              uint32_t *__restrict__ deg) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    deg[v] = (uint32_t)(rp[v + 1] - rp[v]);
}

// Orientation of a CSR as the reference's preprocess loop does it
// (tc.cu:740-758): entry (v, w) is kept as (rank v, rank w) when
// rank w > rank v. One warp per row; pass 1 counts (the longest row to
// *most), pass 2 writes the rows or, when one is too long to be sorted in
// place, their keys.
__global__ void k_kept_per_row(const uint64_t *__restrict__ rp,
                               const uint32_t *__restrict__ ci, uint64_t n,
                               const uint32_t *__restrict__ rank,
                               uint32_t *__restrict__ kept, uint64_t *__restrict__ most,
                               const uint32_t *__restrict__ err) {
  if (*err != kDevOk) return;  // the ranks may not be there
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t top = 0;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint32_t rv = rank[v];
    uint32_t c = 0;
    for (uint64_t j = rp[v] + lane; j < rp[v + 1]; j += 32)
      c += rank[ci[j]] > rv ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) kept[rv] = c;
    top = c > top ? c : top;
  }
  __shared__ uint32_t s_top;
  if (threadIdx.x == 0) s_top = 0;
  __syncthreads();
  if (lane == 0) atomicMax(&s_top, top);
  __syncthreads();
  if (threadIdx.x == 0)
    atomicMax(reinterpret_cast<unsigned long long *>(most), (unsigned long long)s_top);
}

// The oriented rows of a symmetric CSR in place: a warp per row gathers the
// ranks of its kept columns in shared memory, finds each one's place by
// counting the smaller ones (equal ones in their order), and writes the row
// at its offset. Bound by the gathers of the ranks and, for long rows, by the
// counting (quadratic in the row), hence the limit; it takes the place of
// keys, their radix passes and the CSR from the keys: 131 us against 412 for
// a Chung-Lu graph of 500,000 vertices and 5.7M edges.
constexpr uint32_t kRowSortCols = 512;
__global__ void __launch_bounds__(256)
    k_kept_rows(const uint64_t *__restrict__ rp, const uint32_t *__restrict__ ci, uint64_t n,
                const uint32_t *__restrict__ rank, const uint64_t *__restrict__ row_ptr,
                uint32_t *__restrict__ col) {
  __shared__ __align__(16) uint32_t s_row[8][kRowSortCols];
  uint32_t *s = s_row[threadIdx.x >> 5];
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint32_t rv = rank[v];
    const uint64_t begin = rp[v], end = rp[v + 1], out = row_ptr[rv];
    // the last hub keeps nothing of the longest row (a star of 2,000,000
    // leaves, count with orientation: 47 ms, without its second gather 9.5; by
    // keys and radix passes 36)
    if (end - begin >= 128 && row_ptr[rv + 1] == out) continue;
    uint32_t c = 0;
    for (uint64_t j0 = begin; j0 < end; j0 += 32) {
      const uint64_t j = j0 + lane;
      const uint32_t rw = j < end ? rank[ci[j]] : 0u;
      const uint32_t bal = __ballot_sync(0xffffffffu, rw > rv);
      const uint32_t at = c + __popc(bal & lt);
      if (rw > rv && at < kRowSortCols) s[at] = rw;
      c += __popc(bal);
    }
    if (c > kRowSortCols) c = kRowSortCols;  // not when the caller checked
    __syncwarp();
    for (uint32_t i = lane; i < c; i += 32) {
      const uint32_t x = s[i];
      uint32_t at = 0, k = 0;
      for (; k + 4 <= c; k += 4) {
        const uint4 y = *reinterpret_cast<const uint4 *>(s + k);
        at += (y.x < x + (k < i)) + (y.y < x + (k + 1 < i)) + (y.z < x + (k + 2 < i)) +
              (y.w < x + (k + 3 < i));
      }
      for (; k < c; ++k) at += s[k] < x + (k < i);
      col[out + at] = x;
    }
    __syncwarp();
  }
}

__global__ void k_kept_write(const uint64_t *__restrict__ rp,
                             const uint32_t *__restrict__ ci, uint64_t n,
                             const uint32_t *__restrict__ rank, uint32_t b,
                             const uint64_t *__restrict__ off,
                             uint64_t *__restrict__ okeys) {
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint32_t rv = rank[v];
    uint64_t pos = off[rv];
    const uint64_t end = rp[v + 1];
    for (uint64_t j0 = rp[v]; j0 < end; j0 += 32) {
      const uint64_t j = j0 + lane;
      bool keep = false;
      uint32_t rw = 0;
      if (j < end) {
        rw = rank[ci[j]];
        keep = rw > rv;
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, keep);
      if (keep) okeys[pos + __popc(bal & lt)] = pack_key(rv, rw, b);
      pos += __popc(bal);
    }
  }
}

// Row offsets monotone from 0 to m, every column id < n.
__global__ void k_check_ids(const uint64_t *__restrict__ rp,
                            const uint32_t *__restrict__ ci, uint64_t n,
                            uint64_t m, uint32_t *err) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    if (ci[i] >= n) atomicCAS(err, 0u, (uint32_t)kDevColumnRange);
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x)
    if (rp[v + 1] < rp[v] || rp[v + 1] > m)
      atomicCAS(err, 0u, (uint32_t)kDevRowPtrRange);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    if (rp[0] != 0 || rp[n] != m) atomicCAS(err, 0u, (uint32_t)kDevRowPtrRange);
}

// Grid of a grid-stride element-wise kernel: at most 32 blocks per SM, so
// blocks stay short and a higher-priority stream's kernels get SMs soon.
unsigned grid_for(DeviceContext *ctx, uint64_t work) {
  const uint64_t cap = (uint64_t)ctx->sm_count * 32;
  uint64_t g = ceil_div(work, 256);
  if (g > cap) g = cap;
  if (g == 0) g = 1;
  return (unsigned)g;
}

// Grid of a kernel that ends in one atomic per block.
unsigned max_grid(DeviceContext *ctx, uint64_t n) {
  const uint64_t cap = (uint64_t)ctx->sm_count * 4;
  const uint64_t g = ceil_div(n, kThreads * 4);
  return (unsigned)(g == 0 ? 1 : g < cap ? g : cap);
}

// Words that the pipeline leaves for the host: read by one copy into pinned
// memory, so a read costs one round trip.
struct PrepWords {
  uint64_t m;       // unique (or kept) edges
  uint64_t maxdeg;  // largest degree
  uint32_t err, pad;
  uint32_t max_id, any_edge;
};
int read_words(cudaStream_t st, const PrepWords *d, PrepWords *h) {
  uint64_t *host = readback_words();
  if (!host) host = reinterpret_cast<uint64_t *>(h);
  WETRIC_CUDA_TRY(cudaMemcpyAsync(host, d, sizeof(PrepWords), cudaMemcpyDeviceToHost, st));
  WETRIC_CUDA_TRY(cudaStreamSynchronize(st));
  memcpy(h, host, sizeof(PrepWords));
  return WETRIC_OK;
}

// Reads the words and turns a device error into a status.
int checked_words(cudaStream_t st, const PrepWords *d, const char *what, PrepWords *h) {
  WETRIC_TRY(read_words(st, d, h));
  if (h->err == kDevLookbackTimeout) {
    set_error(WETRIC_ETIMEDOUT, "%s: a look-back did not complete in time", what);
    return WETRIC_ETIMEDOUT;
  }
  if (h->err != kDevOk) {
    set_error(WETRIC_EINVAL, "%s: invalid input (device check %u)", what, h->err);
    return WETRIC_EINVAL;
  }
  return WETRIC_OK;
}

int alloc_words(DeviceContext *ctx, cudaStream_t st, Scratch<PrepWords> *w) {
  WETRIC_TRY(w->alloc(ctx, st, 1));
  WETRIC_CUDA_TRY(cudaMemsetAsync(w->ptr, 0, sizeof(PrepWords), st));
  return WETRIC_OK;
}

// The group sort's keys, in degree order: group above (the g with
// group_base[g] <= v < group_base[g + 1]), id below.
struct GroupKeys {
  const uint64_t *__restrict__ by_degree;
  const uint64_t *__restrict__ group_base;
  uint32_t G;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const {
    const uint32_t v = (uint32_t)by_degree[i];
    uint32_t lo = 0, len = G;
    while (len > 1) {
      const uint32_t h = len >> 1;
      if (group_base[lo + h] <= v) lo += h;
      len -= h;
    }
    return ((uint64_t)lo << 32) | v;
  }
};

// rank[v] = position of v in the stable ascending-degree order. With groups
// (a disjoint union of G graphs) the order is (group, degree, id), so every
// group keeps its id range and the order inside a group is that of the
// group alone.
int degree_rank(DeviceContext *ctx, cudaStream_t st, const uint32_t *deg, uint64_t n,
                uint64_t maxdeg, uint32_t *rank, uint32_t *err,
                const uint64_t *group_base = nullptr, uint32_t G = 0,
                const prim::SortSpace *spaces = nullptr) {
  const uint32_t dbits = bits_for(maxdeg);
  const bool groups = group_base != nullptr && G > 1;
  const uint32_t passes = prim::digit_plan(32, dbits ? dbits : 1).passes;
  Scratch<uint64_t> a, b;
  if (groups || passes > 1) WETRIC_TRY(a.alloc(ctx, st, n));
  if (groups || passes > 2) WETRIC_TRY(b.alloc(ctx, st, n));
  const DegreeKeys keys{deg};
  if (!groups)
    return prim::radix_sort_into(ctx, st, keys, keys, a.ptr, b.ptr, RankTo{rank}, n, 32, dbits,
                                 err, spaces);
  uint64_t *by_degree = prim::sorted_buffer(a.ptr, b.ptr, 32, dbits);
  WETRIC_TRY((prim::radix_sort_into(ctx, st, keys, keys, a.ptr, b.ptr, prim::KeysTo{by_degree}, n,
                                    32, dbits, err, spaces)));
  const GroupKeys gkeys{by_degree, group_base, G};
  return prim::radix_sort_into(ctx, st, gkeys, gkeys, by_degree == a.ptr ? b.ptr : a.ptr,
                               by_degree, RankTo{rank}, n, 32, bits_for(G - 1), err,
                               spaces ? spaces + 1 : nullptr);
}

// Sorted packed (row, col) keys -> CSR arrays.
int keys_to_csr(DeviceContext *ctx, cudaStream_t st, const uint64_t *keys,
                uint64_t m, uint64_t n, uint32_t b, uint64_t *row_ptr,
                uint32_t *col_ind, const uint32_t *err) {
  if (m == 0) {
    WETRIC_CUDA_TRY(cudaMemsetAsync(row_ptr, 0, (n + 1) * sizeof(uint64_t), st));
    return WETRIC_OK;
  }
  k_keys_to_csr<<<grid_for(ctx, m > n ? m : n), kThreads, 0, st>>>(keys, m, n, b, row_ptr,
                                                                  col_ind, err);
  WETRIC_LAUNCH_CHECK();
  return WETRIC_OK;
}

}  // namespace

void DeviceCsr::release() {
  if (ctx) {
    if (row_ptr) dev_free(ctx, stream, row_ptr, (n + 1) * sizeof(uint64_t));
    if (col_ind) dev_free(ctx, stream, col_ind, (m ? m : 4) * sizeof(uint32_t));
  }
  row_ptr = nullptr;
  col_ind = nullptr;
  n = m = 0;
}

static int alloc_csr(DeviceContext *ctx, cudaStream_t st, uint64_t n,
                     uint64_t m, DeviceCsr *out) {
  out->release();
  out->ctx = ctx;
  out->stream = st;
  void *p = nullptr;
  WETRIC_TRY(dev_alloc(ctx, st, (n + 1) * sizeof(uint64_t), &p));
  out->row_ptr = static_cast<uint64_t *>(p);
  out->n = n;
  p = nullptr;
  int rc = dev_alloc(ctx, st, (m ? m : 4) * sizeof(uint32_t), &p);
  if (rc != WETRIC_OK) {
    out->release();
    return rc;
  }
  out->col_ind = static_cast<uint32_t *>(p);
  out->m = m;
  return WETRIC_OK;
}

// The cleared workspaces of a chain of sorts over P pairs and n vertices: one
// allocation and one memset (with its own for each sort and the unique pass
// the orientation of a 9,000-vertex graph took 197 us, so 182).
struct PrepSpace {
  Scratch<uint64_t> buf;
  prim::SortSpace pairs, vertices[2], last;  // vertices: by degree, by group
  uint64_t *unique = nullptr;                // [0] the ticket, then one word per tile
  int alloc(DeviceContext *ctx, cudaStream_t st, uint64_t n, uint64_t P, uint64_t last_keys,
            bool groups) {
    const uint64_t a = prim::SortSpace::words(P), u = ceil_div(P, kUniqueTile) + 1;
    const uint64_t v = prim::SortSpace::words(n), l = prim::SortSpace::words(last_keys);
    const uint64_t words = a + u + (groups ? 2 : 1) * v + l;
    WETRIC_TRY(buf.alloc(ctx, st, words));
    WETRIC_CUDA_TRY(cudaMemsetAsync(buf.ptr, 0, words * sizeof(uint64_t), st));
    pairs.at(buf.ptr);
    unique = buf.ptr + a;
    last.at(unique + u);
    vertices[0].at(unique + u + l);
    vertices[1].at(unique + u + l + (groups ? v : 0));
    return WETRIC_OK;
  }
};

// Raw pairs -> unique undirected edges as sorted canonical keys (P slots,
// words->m of them used) and the degrees of the n vertices. Reads m, the
// largest degree and the checks back.
static int unique_edges(DeviceContext *ctx, cudaStream_t st, const uint32_t *src,
                        const uint32_t *dst, uint64_t P, uint64_t n_hint,
                        const Scratch<PrepWords> &words, uint64_t *n_out, uint32_t *b_out,
                        Scratch<uint64_t> *ukeys, Scratch<uint32_t> *deg, PrepWords *h,
                        PrepSpace *space, uint32_t last_per_pair, bool groups) {
  uint64_t n = n_hint;
  if (n == 0) {
    if (P > 0) {
      k_max_id<<<grid_for(ctx, P), 256, 0, st>>>(src, dst, P, &words.ptr->max_id,
                                                 &words.ptr->any_edge);
      WETRIC_LAUNCH_CHECK();
    }
    WETRIC_TRY(read_words(st, words.ptr, h));
    n = (uint64_t)h->max_id + 1;  // tc.cu:625, max_vertex starts at 0
  }
  if (n > (1ull << 32)) {
    set_error(WETRIC_ERANGE, "n = %llu exceeds 2^32", (unsigned long long)n);
    return WETRIC_ERANGE;
  }
  uint32_t b = bits_for(n - 1);
  if (b == 0) b = 1;
  const uint64_t sentinel = (2 * b >= 64) ? ~0ull : ((1ull << (2 * b)) - 1);
  Scratch<uint64_t> keys, alt;
  WETRIC_TRY(keys.alloc(ctx, st, P));
  WETRIC_TRY(alt.alloc(ctx, st, P));
  WETRIC_TRY(deg->alloc(ctx, st, n));
  WETRIC_CUDA_TRY(cudaMemsetAsync(deg->ptr, 0, n * sizeof(uint32_t), st));
  WETRIC_TRY(space->alloc(ctx, st, n, P, last_per_pair * P, groups));
  const CanonPairs counted{src, dst, alt.ptr, b, n, sentinel, &words.ptr->err};
  uint64_t *sorted = prim::sorted_buffer(keys.ptr, alt.ptr, 0, 2 * b);
  WETRIC_TRY((prim::radix_sort_into(ctx, st, counted, prim::KeysFrom{alt.ptr}, keys.ptr, alt.ptr,
                                    prim::KeysTo{sorted}, P, 0, 2 * b, &words.ptr->err,
                                    &space->pairs)));
  uint64_t *spare = sorted == keys.ptr ? alt.ptr : keys.ptr;
  if (P > 0) {
    const uint64_t tiles = ceil_div(P, kUniqueTile);
    k_unique_degrees<<<(unsigned)tiles, kThreads, 0, st>>>(
        sorted, P, sentinel, b, spare, deg->ptr, space->unique + 1,
        reinterpret_cast<uint32_t *>(space->unique), &words.ptr->m, &words.ptr->err);
    WETRIC_LAUNCH_CHECK();
  }
  k_max_u32<<<max_grid(ctx, n), kThreads, 0, st>>>(deg->ptr, n, &words.ptr->maxdeg);
  WETRIC_LAUNCH_CHECK();
  // Keep the buffer that holds the unique keys; release the other.
  Scratch<uint64_t> &kept = spare == keys.ptr ? keys : alt;
  (spare == keys.ptr ? alt : keys).release();
  ukeys->ctx = kept.ctx;
  ukeys->stream = kept.stream;
  ukeys->bytes = kept.bytes;
  ukeys->ptr = kept.detach();
  WETRIC_TRY(checked_words(st, words.ptr, "edge ids", h));
  *n_out = n;
  *b_out = b;
  return WETRIC_OK;
}

int orient_pairs(DeviceContext *ctx, cudaStream_t st, const uint32_t *src,
                 const uint32_t *dst, uint64_t P, uint64_t n_hint,
                 DeviceCsr *out, const uint64_t *group_base, uint32_t G) {
  NvtxRange nvtx_("wetric orient");
  uint64_t n = 0;
  uint32_t b = 0;
  PrepWords h{};
  Scratch<PrepWords> words;
  Scratch<uint64_t> ukeys;
  Scratch<uint32_t> deg, rank;
  PrepSpace space;
  WETRIC_TRY(alloc_words(ctx, st, &words));
  WETRIC_TRY(unique_edges(ctx, st, src, dst, P, n_hint, words, &n, &b, &ukeys, &deg, &h, &space, 1,
                          group_base != nullptr && G > 1));
  const uint64_t m = h.m;
  uint32_t *err = &words.ptr->err;
  WETRIC_TRY(rank.alloc(ctx, st, n));
  WETRIC_TRY(degree_rank(ctx, st, deg.ptr, n, h.maxdeg, rank.ptr, err, group_base, G,
                         space.vertices));
  deg.release();
  // The oriented keys go to the sort's second buffer, so the peak stays at
  // input pairs + 2 key buffers (m > 2^32 fits 180 GB).
  Scratch<uint64_t> okeys;
  WETRIC_TRY(okeys.alloc(ctx, st, m));
  uint64_t *sorted = prim::sorted_buffer(ukeys.ptr, okeys.ptr, 0, 2 * b);
  WETRIC_TRY((prim::radix_sort_into(
      ctx, st, OrientedKeys{ukeys.ptr, rank.ptr, okeys.ptr, b}, prim::KeysFrom{okeys.ptr},
      ukeys.ptr, okeys.ptr, prim::KeysTo{sorted}, m, 0, 2 * b, err, &space.last)));
  rank.release();
  WETRIC_TRY(alloc_csr(ctx, st, n, m, out));
  WETRIC_TRY(keys_to_csr(ctx, st, sorted, m, n, b, out->row_ptr, out->col_ind, err));
  return checked_words(st, words.ptr, "orientation", &h);
}

int load_orient_kernels() {
  using prim::KeysFrom;
  using prim::KeysTo;
  WETRIC_TRY((prim::load_onesweep<KeysFrom, KeysTo>()));
  WETRIC_TRY((prim::load_onesweep<DegreeKeys, KeysTo>()));
  WETRIC_TRY((prim::load_onesweep<DegreeKeys, RankTo>()));
  WETRIC_TRY((prim::load_onesweep<KeysFrom, RankTo>()));
  WETRIC_TRY((prim::load_onesweep<GroupKeys, KeysTo>()));
  WETRIC_TRY((prim::load_onesweep<GroupKeys, RankTo>()));
  return load_kernels({(const void *)k_max_id, (const void *)k_unique_degrees,
                       (const void *)k_max_u32, (const void *)k_keys_to_csr,
                       (const void *)prim::k_radix_hist<CanonPairs>,
                       (const void *)prim::k_radix_hist<DegreeKeys>,
                       (const void *)prim::k_radix_hist<GroupKeys>,
                       (const void *)prim::k_radix_hist<OrientedKeys>});
}

int symmetric_from_pairs(DeviceContext *ctx, cudaStream_t st,
                         const uint32_t *src, const uint32_t *dst, uint64_t P,
                         uint64_t n_hint, DeviceCsr *out) {
  uint64_t n = 0;
  uint32_t b = 0;
  PrepWords h{};
  Scratch<PrepWords> words;
  Scratch<uint64_t> ukeys;
  Scratch<uint32_t> deg;
  PrepSpace space;
  WETRIC_TRY(alloc_words(ctx, st, &words));
  WETRIC_TRY(unique_edges(ctx, st, src, dst, P, n_hint, words, &n, &b, &ukeys, &deg, &h, &space, 2,
                          false));
  deg.release();
  const uint64_t m = h.m;
  Scratch<uint64_t> dkeys, dalt;
  WETRIC_TRY(dkeys.alloc(ctx, st, 2 * m));
  WETRIC_TRY(dalt.alloc(ctx, st, 2 * m));
  const BothDirections both{ukeys.ptr, b};
  uint64_t *sorted = prim::sorted_buffer(dkeys.ptr, dalt.ptr, 0, 2 * b);
  WETRIC_TRY((prim::radix_sort_into(ctx, st, both, both, dkeys.ptr, dalt.ptr,
                                    prim::KeysTo{sorted}, 2 * m, 0, 2 * b, &words.ptr->err,
                                    &space.last)));
  ukeys.release();
  WETRIC_TRY(alloc_csr(ctx, st, n, 2 * m, out));
  WETRIC_TRY(
      keys_to_csr(ctx, st, sorted, 2 * m, n, b, out->row_ptr, out->col_ind,
                  &words.ptr->err));
  return checked_words(st, words.ptr, "symmetric CSR", &h);
}

int orient_csr(DeviceContext *ctx, cudaStream_t st, const uint64_t *rp,
               const uint32_t *ci, uint64_t n, uint64_t m, DeviceCsr *out) {
  if (n == 0) {
    WETRIC_TRY(alloc_csr(ctx, st, 0, 0, out));
    WETRIC_CUDA_TRY(cudaMemsetAsync(out->row_ptr, 0, sizeof(uint64_t), st));
    return WETRIC_OK;
  }
  if (n > (1ull << 32)) {
    set_error(WETRIC_ERANGE, "n = %llu exceeds 2^32", (unsigned long long)n);
    return WETRIC_ERANGE;
  }
  PrepWords h{};
  Scratch<PrepWords> words;
  Scratch<uint32_t> deg, rank;
  WETRIC_TRY(alloc_words(ctx, st, &words));
  uint32_t *err = &words.ptr->err;
  k_check_ids<<<grid_for(ctx, m > n ? m : n), 256, 0, st>>>(rp, ci, n, m, err);
  WETRIC_LAUNCH_CHECK();
  WETRIC_TRY(deg.alloc(ctx, st, n));
  WETRIC_TRY(rank.alloc(ctx, st, n));
  k_row_lengths<<<grid_for(ctx, n), 256, 0, st>>>(rp, n, deg.ptr);
  WETRIC_LAUNCH_CHECK();
  k_max_u32<<<max_grid(ctx, n), kThreads, 0, st>>>(deg.ptr, n, &words.ptr->maxdeg);
  WETRIC_LAUNCH_CHECK();
  WETRIC_TRY(checked_words(st, words.ptr, "csr", &h));
  uint32_t b = bits_for(n - 1);
  if (b == 0) b = 1;
  WETRIC_TRY(degree_rank(ctx, st, deg.ptr, n, h.maxdeg, rank.ptr, err));
  // deg is reused as the kept count of every oriented row.
  const unsigned warps_grid = grid_for(ctx, n * 32);
  WETRIC_CUDA_TRY(cudaMemsetAsync(&words.ptr->maxdeg, 0, sizeof(uint64_t), st));
  k_kept_per_row<<<warps_grid, 256, 0, st>>>(rp, ci, n, rank.ptr, deg.ptr, &words.ptr->maxdeg,
                                          err);
  WETRIC_LAUNCH_CHECK();
  Scratch<uint64_t> off;
  WETRIC_TRY(off.alloc(ctx, st, n + 1));
  WETRIC_TRY((prim::exclusive_scan<uint32_t, uint64_t>(ctx, st, deg.ptr,
                                                       off.ptr, n, err)));
  WETRIC_CUDA_TRY(cudaMemcpyAsync(&words.ptr->m, off.ptr + n, sizeof(uint64_t),
                                  cudaMemcpyDeviceToDevice, st));
  WETRIC_TRY(checked_words(st, words.ptr, "csr", &h));
  const uint64_t kept = h.m;
  if (h.maxdeg <= kRowSortCols && n < (1ull << 32)) {
    WETRIC_TRY(alloc_csr(ctx, st, n, kept, out));
    WETRIC_CUDA_TRY(cudaMemcpyAsync(out->row_ptr, off.ptr, (n + 1) * sizeof(uint64_t),
                                    cudaMemcpyDeviceToDevice, st));
    k_kept_rows<<<warps_grid, 256, 0, st>>>(rp, ci, n, rank.ptr, off.ptr, out->col_ind);
    WETRIC_LAUNCH_CHECK();
    return WETRIC_OK;
  }
  Scratch<uint64_t> okeys, oalt;
  WETRIC_TRY(okeys.alloc(ctx, st, kept));
  WETRIC_TRY(oalt.alloc(ctx, st, kept));
  k_kept_write<<<warps_grid, 256, 0, st>>>(rp, ci, n, rank.ptr, b, off.ptr,
                                           okeys.ptr);
  WETRIC_LAUNCH_CHECK();
  deg.release();
  rank.release();
  off.release();
  const prim::KeysFrom from{okeys.ptr};
  uint64_t *sorted = prim::sorted_buffer(oalt.ptr, okeys.ptr, 0, 2 * b);
  WETRIC_TRY((prim::radix_sort_into(ctx, st, from, from, oalt.ptr, okeys.ptr,
                                    prim::KeysTo{sorted}, kept, 0, 2 * b, err)));
  WETRIC_TRY(alloc_csr(ctx, st, n, kept, out));
  WETRIC_TRY(
      keys_to_csr(ctx, st, sorted, kept, n, b, out->row_ptr, out->col_ind, err));
  return checked_words(st, words.ptr, "csr", &h);
}

}  // namespace wetric
