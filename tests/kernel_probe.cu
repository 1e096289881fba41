// Device code of the library as tests call it: the words that look-back
// scans publish, scans of given values, and the kernels that follow a scan or
// a sort, run with a given error word.
#include "pair_streams.cuh"
#include "primitives.cuh"
#include "stage_workers.h"
#include "walk.cuh"

using namespace wetric;

#define PROBE(call)                            \
  do {                                         \
    const int rc_ = (int)(call);               \
    if (rc_ != 0) return rc_;                  \
  } while (0)

// The words of a 64-bit value under `flag`, and what a reader makes of any
// two words.
extern "C" void probe_tile_words(uint32_t flag, uint64_t value, uint64_t *words) {
  words[0] = prim::tile_word(0, flag, value);
  words[1] = prim::tile_rest(flag, value);
}
extern "C" uint32_t probe_tile_read(const uint64_t *words, uint64_t *value) {
  *value = prim::tile_pair_value(words[0], words[1]);
  return prim::tile_pair_flag(words[0], words[1]);
}

// out[0..n] = exclusive prefix of in[0..n-1] (device arrays); *err: the error
// word afterwards.
extern "C" int probe_scan_u64(const uint64_t *in, uint64_t n, uint64_t *out, uint32_t *err) {
  DeviceContext *ctx = nullptr;
  PROBE(get_context(0, &ctx));
  Scratch<uint32_t> e;
  PROBE(e.alloc(ctx, ctx->stream, 1));
  PROBE(cudaMemsetAsync(e.ptr, 0, 4, ctx->stream));
  PROBE((prim::exclusive_scan<uint64_t, uint64_t>(ctx, ctx->stream, in, out, n, e.ptr)));
  PROBE(cudaMemcpyAsync(err, e.ptr, 4, cudaMemcpyDeviceToHost, ctx->stream));
  return (int)cudaStreamSynchronize(ctx->stream);
}

// The rest take device arrays and the device error word *err.

// keys[0..n) sorted on their bits [0, bits) into out, by way of a and b.
extern "C" int probe_sort(const uint64_t *keys, uint64_t n, uint32_t bits, uint64_t *a,
                          uint64_t *b, uint64_t *out, uint32_t *err) {
  DeviceContext *ctx = nullptr;
  PROBE(get_context(0, &ctx));
  const prim::KeysFrom from{keys};
  PROBE((prim::radix_sort_into(ctx, ctx->stream, from, from, a, b, prim::KeysTo{out}, n, 0, bits,
                               err)));
  return (int)cudaStreamSynchronize(ctx->stream);
}

// The kernels behind the scans of the wedge-check path; every output is an
// element of `out` (room for 4 n each).
extern "C" int probe_after_scan(const uint32_t *rp, uint64_t n, const uint32_t *active,
                                const uint64_t *pos, uint64_t *out, const uint32_t *err) {
  DeviceContext *ctx = nullptr;
  PROBE(get_context(0, &ctx));
  uint64_t *wp = out, *rb = out + n;
  k_compact_active<uint32_t><<<8, 256, 0, ctx->stream>>>(
      rp, n, active, pos, wp, rb, reinterpret_cast<uint32_t *>(out + 2 * n), err);
  CoreStarts cs{};
  cs.v0[cs.c++] = n / 2;
  k_core_prefix<<<1, 32, 0, ctx->stream>>>(wp, pos, cs, out + 3 * n, err);
  ChunkRows rows{};
  rows.v[rows.c++] = n / 2;
  k_chunk_prefix<<<1, 32, 0, ctx->stream>>>(wp, pos, rows, out + 3 * n + 2, err);
  PROBE(cudaGetLastError());
  return (int)cudaStreamSynchronize(ctx->stream);
}

// The walk behind its sort: `keys` are m sorted entries, one per middle
// vertex x = 0, 1, ... (its column row[x]), tails of one column each.
extern "C" int probe_walk(const uint32_t *rp, const uint32_t *split, const uint32_t *long_rows,
                          const uint32_t *ci, uint64_t m, const uint64_t *keys, uint32_t entries,
                          uint32_t rows, uint32_t bits_start, uint32_t bits_len, uint32_t *start,
                          uint32_t *items, uint32_t *counts, unsigned long long *out,
                          const uint32_t *err) {
  DeviceContext *ctx = nullptr;
  PROBE(get_context(0, &ctx));
  const WalkBits bits{1, bits_start, bits_len};
  uint2 *big = reinterpret_cast<uint2 *>(items), *small = big + 2 * rows;
  k_walk_starts<<<1, kWalkBlock, 0, ctx->stream>>>(keys, entries, 2 * rows, bits.shift(), start,
                                                   err);
  k_walk_plan<<<1, kWalkBlock, 0, ctx->stream>>>(rp, split, long_rows, start, 2 * rows, big, small,
                                                 counts, false, err);
  k_walk_count<kWalkSmallBlock, kWalkSmallBlocks, false><<<4, kWalkSmallBlock, 0, ctx->stream>>>(
      rp, split, long_rows, walk_columns(ci, m), 0, keys, start, bits, small, counts + 1,
      counts + 2, 0, out, WalkGroups{}, nullptr, err);
  PROBE(cudaGetLastError());
  return (int)cudaStreamSynchronize(ctx->stream);
}

// A vertex of two columns counted by pair streams (one tile of all columns).
extern "C" int probe_pairs(const uint32_t *rp, const uint32_t *ci, const uint32_t *pv,
                           const uint64_t *ps, const uint32_t *tile_k, uint64_t cols,
                           unsigned long long *total, const uint32_t *err) {
  DeviceContext *ctx = nullptr;
  PROBE(get_context(0, &ctx));
  k_count_pairs<false><<<1, kPairWarps * 32, 0, ctx->stream>>>(rp, ci, pv, ps, nullptr, 1, tile_k,
                                                               1, cols, total, nullptr, err);
  PROBE(cudaGetLastError());
  return (int)cudaStreamSynchronize(ctx->stream);
}

// The form that counts a graph: 0 intersections, 1 with the walk, 2 neither.
extern "C" int probe_walk_form(uint64_t n, uint64_t m, uint64_t edges, uint64_t long_rows,
                               uint64_t longest, uint64_t long_wedges) {
  return (int)walk_form(n, m, edges, long_rows, longest, long_wedges);
}

// One warp's hits, hits[lane] each, added to *sum (device).
__global__ void add_hits(const unsigned long long *hits, unsigned long long *sum) {
  walk_add_hits(sum, hits[threadIdx.x], threadIdx.x);
}
extern "C" int probe_add_hits(const unsigned long long *hits, unsigned long long *sum) {
  add_hits<<<1, 32>>>(hits, sum);
  PROBE(cudaGetLastError());
  return (int)cudaDeviceSynchronize();
}

// `callers` threads copy pieces of the given sizes at once, `rounds` times
// each, `gap_ms` apart; 0 when every copy is whole and nothing else changed.
extern "C" int probe_stage_copies(const uint64_t *sizes, int n, int callers, int rounds,
                                  int gap_ms) {
  StageWorkers workers;
  workers.start();
  std::atomic<int> bad{0};
  std::vector<std::thread> threads;
  for (int c = 0; c < callers; ++c)
    threads.emplace_back([&, c] {
      for (int r = 0; r < rounds; ++r)
        for (int i = 0; i < n; ++i) {
          const size_t size = sizes[i], pad = 64;
          std::vector<unsigned char> src(size), dst(size + 2 * pad, 0xAB);
          for (size_t k = 0; k < size; ++k) src[k] = (unsigned char)(k * 31 + (k >> 13) + c + r + i);
          workers.copy(src.data(), dst.data() + pad, size);
          bool ok = size == 0 || memcmp(src.data(), dst.data() + pad, size) == 0;
          for (size_t k = 0; k < pad; ++k) ok = ok && dst[k] == 0xAB && dst[pad + size + k] == 0xAB;
          if (!ok) ++bad;
          if (gap_ms) std::this_thread::sleep_for(std::chrono::milliseconds(gap_ms));
        }
    });
  for (std::thread &t : threads) t.join();
  return bad;
}
