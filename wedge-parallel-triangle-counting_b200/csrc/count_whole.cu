// count_whole.cu -- the default count: a whole graph with 32-bit row offsets
// (or a small one with any), by the dense core, row intersections and the
// column walk (walk.cuh).
//
// The reference counts every wedge by one edge check (tc.cu:173-293); here
// every edge (v, w) takes the cheapest of three forms of the same
// intersection, so nothing needs the wedge prefix, the tiles over it or
// per-row hash sets. A small graph is one kernel that writes its results to
// the host (k_small_count; with validation k_edge_vertices, k_validate,
// k_edge_merge and a copy), a large one
//
//   k_edge_vertices                                                 [read]
//   per row chunk: k_walk_split k_edge_merge k_core_bitmap k_core_count
//   the entries made                                                [read]
//   sort  k_walk_starts  k_walk_plan  k_walk_count (two block sizes) [read]
//
// Wedge ranges, u64 offsets of large graphs and the options that name another
// kernel (CountArgs::kernel, pair_streams off, a shell, l2_persist) keep to
// count.cu. So do graphs that are declined here: no room for a part, entries of
// more than 64 bits (walk_form), more entries than room, or too many wedges
// between rows of several hash sets (WalkFar).
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "count.cuh"
#include "count_kernels.cuh"
#include "primitives.cuh"
#include "readback.cuh"
#include "walk.cuh"

namespace wetric {

namespace {

// Below this many columns a graph takes no core and no walk: one kernel
// intersects the rows of all its edges.
constexpr uint64_t kSmallColumns = 1ull << 17;
constexpr uint64_t kSmallRows = 1ull << 20;  // and this many rows at most: one launch

// A word read by the core's row ANDs against a wedge counted below it (R-MAT
// scale 22, between neighbouring lengths: 0.21 ps per estimated word, 0.8 ps
// per wedge; the whole count at 16,384 / 32,768 / 49,152 / 65,536 vertices:
// 6.45 / 5.93 / 6.04 / 6.40 ms, scale 24 36.9 / 35.0 / 33.0 / 32.4, scale 20
// 1.50 / 1.55 / 1.68 / 1.90).
constexpr double kCoreWordsPerWalked = 4.0;

struct EventPair {
  cudaEvent_t a = nullptr, b = nullptr;
  ~EventPair() {
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
  }
  int start(cudaStream_t st) {
    if (!a) {
      WETRIC_CUDA_TRY(cudaEventCreate(&a));
      WETRIC_CUDA_TRY(cudaEventCreate(&b));
    }
    WETRIC_CUDA_TRY(cudaEventRecord(a, st));
    return WETRIC_OK;
  }
  int stop(cudaStream_t st) {
    WETRIC_CUDA_TRY(cudaEventRecord(b, st));
    return WETRIC_OK;
  }
  int add_to(double *ms) const {
    if (!a) return WETRIC_OK;
    float f = 0;
    WETRIC_CUDA_TRY(cudaEventElapsedTime(&f, a, b));
    *ms += f;
    return WETRIC_OK;
  }
};

int check_words(uint64_t err, uint64_t longest) {
  if (err == kDevLookbackTimeout || err == kDevStageTimeout) {
    set_error(WETRIC_ETIMEDOUT, "a bounded wait on the device ran out (code %u)", (uint32_t)err);
    return WETRIC_ETIMEDOUT;
  }
  if (err != kDevOk) {
    set_error(WETRIC_EINVAL, "oriented CSR check failed (device code %u)", (uint32_t)err);
    return WETRIC_EINVAL;
  }
  if (longest >= kMaxOutDegree) {
    set_error(WETRIC_ERANGE, "max out-degree %llu >= 2^30", (unsigned long long)longest);
    return WETRIC_ERANGE;
  }
  return WETRIC_OK;
}

}  // namespace

bool count_whole_takes(const CountArgs &a) {
  return a.n > 0 && a.kernel == 0 && a.pair_streams && !a.l2_persist && a.wedge_begin == 0 &&
         a.wedge_end == 0 && (a.shell_len == 0 || a.shell_len == kCoreOff) &&
         a.n < (1ull << 31) && a.m < (1ull << 31) &&
         (a.offsets32 || (a.m < kSmallColumns && (a.core_len == 0 || a.core_len == kCoreOff)));
}

// The small graph's single launch (k_small_count); false: no pinned words.
template <typename Off>
static int small_count(DeviceContext *ctx, cudaStream_t st, const CountArgs &a, CountResult *r,
                       bool *done) {
  static_assert(kSmallBlocks * kSmallWords <= kPinnedWords, "one word group per block");
  const unsigned long long *out = reinterpret_cast<unsigned long long *>(readback_words());
  *done = out != nullptr;
  if (!out) return WETRIC_OK;
  EventPair ev_all;
  WETRIC_TRY(ev_all.start(st));
  if (a.ci_ready) WETRIC_CUDA_TRY(cudaStreamWaitEvent(st, a.ci_ready, 0));
  const uint32_t n = (uint32_t)a.n, m = (uint32_t)a.m, warps = kWalkBlock / 32;
  const uint32_t T = 32 * (uint32_t)ceil_div(m ? m : 1, 32ull * warps * kSmallBlocks);
  const uint64_t for_rows = ceil_div(n, kWalkBlock), for_edges = ceil_div(m, T * warps);
  uint64_t grid = for_rows > for_edges ? for_rows : for_edges;
  if (grid > kSmallBlocks) grid = kSmallBlocks;
  k_small_count<Off><<<(unsigned)grid, kWalkBlock, 0, st>>>(
      static_cast<const Off *>(a.row_ptr), walk_columns(a.col_ind, m), n, m, T,
      const_cast<unsigned long long *>(out));
  WETRIC_LAUNCH_CHECK();
  WETRIC_TRY(ev_all.stop(st));
  WETRIC_CUDA_TRY(cudaEventSynchronize(ev_all.b));
  unsigned long long sum[3] = {}, longest = 0, bad = 0;
  for (uint64_t i = 0; i < grid; ++i) {
    const unsigned long long *w = out + i * kSmallWords;
    sum[0] += w[0];
    sum[1] += w[1];
    sum[2] += w[2] & ((1ull << 40) - 1);
    bad |= w[2] >> 40;
    longest = longest > w[3] ? longest : w[3];
  }
  r->max_out_degree = longest;
  WETRIC_TRY(check_words(bad ? (uint64_t)kDevRowPtrRange : 0, longest));
  r->triangles = sum[0];
  r->wedges = r->wedges_counted = r->pair_wedges = sum[1];
  r->pair_rows = sum[2];
  WETRIC_TRY(ev_all.add_to(&r->exec_ms));
  r->count_ms = r->pair_ms = r->exec_ms;
  r->block = kWalkBlock;
  r->grid = (uint32_t)grid;
  r->launches = 1;
  return WETRIC_OK;
}

template <typename Off>
static int whole_impl(DeviceContext *ctx, cudaStream_t st, const CountArgs &a, CountResult *r,
                      bool *declined) {
  NvtxRange nvtx_("wetric count");
  const Off *rp = static_cast<const Off *>(a.row_ptr);
  const uint64_t n = a.n, m = a.m;
  *r = CountResult();
  const uint32_t C_in = a.col_chunks, C = C_in ? C_in : 1u;
  if (C_in > kMaxColChunks || (C_in && a.validate)) {
    set_error(WETRIC_EINVAL, "bad column chunks");
    return WETRIC_EINVAL;
  }
  for (uint32_t i = 0; i < C_in; ++i) {
    const uint64_t hi = i ? a.chunk_lo[i - 1] : n;
    if (a.chunk_lo[i] >= hi || (i + 1 == C_in && a.chunk_lo[i] != 0)) {
      set_error(WETRIC_EINVAL, "column chunks must cover the rows top down");
      return WETRIC_EINVAL;
    }
  }
  const bool small = m < kSmallColumns && (a.core_len == 0 || a.core_len == kCoreOff);
  if (small && !a.validate && !C_in && n > 0 && n <= kSmallRows) {
    bool done = false;
    WETRIC_TRY(small_count<Off>(ctx, st, a, r, &done));
    if (done) return WETRIC_OK;
  }
  EventPair ev_all;
  WETRIC_TRY(ev_all.start(st));
  uint32_t launches = 0;
  uint64_t grid = 0;
  // [0] triangles, [1] wedges of the row intersections, [2] error word and,
  // above it, whether the graph is not walked after all, [3...]
  // k_edge_vertices' totals
  Scratch<unsigned long long> words;
  constexpr uint32_t kWords = 3 + kEdgeTotals;
  static_assert(kWords + kCoreNumCandidates <= kReadWords, "one read-back");
  WETRIC_TRY(words.alloc(ctx, st, kWords));
  WETRIC_CUDA_TRY(cudaMemsetAsync(words.ptr, 0, kWords * sizeof(uint64_t), st));
  uint32_t *err = reinterpret_cast<uint32_t *>(words.ptr + 2);

  EdgeCores cores{};
  if (!small && a.core_len != kCoreOff && n >= 64) {
    if (a.core_len == 0)
      for (; cores.count < kCoreNumCandidates; ++cores.count)
        cores.len[cores.count] = (uint32_t)(n < core_candidate(cores.count)
                                                ? n
                                                : core_candidate(cores.count));
    else
      cores.len[cores.count++] = (uint32_t)(n < a.core_len ? n : a.core_len < kCoreMaxLen
                                                                   ? a.core_len
                                                                   : kCoreMaxLen);
  }
  // No room for a part of this way: the wedge-check path counts (and searches
  // where it has no room for its sets).
  const auto without_room = [&](int rc) {
    if (rc != WETRIC_ENOMEM) return rc;
    clear_error();
    *declined = true;
    return (int)WETRIC_OK;
  };
  Scratch<uint32_t> number, long_rows, core;
  if (!small) {
    int rc = number.alloc(ctx, st, n);
    if (rc == WETRIC_OK) rc = long_rows.alloc(ctx, st, long_rows_room(m));
    if (rc != WETRIC_OK) return without_room(rc);
  }
  if (n > 0) {
    const uint64_t most = (uint64_t)ctx->sm_count * 8, need = ceil_div(n, kWalkBlock);
    k_edge_vertices<Off><<<(unsigned)(need < most ? need : most), kWalkBlock, 0, st>>>(
        rp, n, m, cores, words.ptr + 3, number.ptr, long_rows.ptr, err);
    WETRIC_LAUNCH_CHECK();
    ++launches;
  }
  if (a.ci_ready && (a.validate || small)) WETRIC_CUDA_TRY(cudaStreamWaitEvent(st, a.ci_ready, 0));
  if (a.validate && m > 0) {
    const uint64_t most = (uint64_t)ctx->sm_count * 32, need = ceil_div(n * 32, 256);
    k_validate<Off><<<(unsigned)(need < most ? need : most), 256, 0, st>>>(rp, a.col_ind, n, m,
                                                                           err);
    WETRIC_LAUNCH_CHECK();
    ++launches;
  }

  uint64_t core_h = 0, core_v0 = n, below_m = m, core_rows = 0, core_words = 0;
  uint32_t core_H4 = 0;
  uint64_t local[kReadWords];
  uint64_t W = 0, rows = 0;
  bool emit = false, sets = false;
  WalkRun walk;
  if (!small) {
    ReadPlan rd;
    rd.add(words.ptr, kWords, 8);
    for (uint32_t c = 0; c < cores.count; ++c) rd.add(rp + n - cores.len[c], 1, sizeof(Off));
    const uint64_t *w = nullptr;
    WETRIC_TRY(read_back(ctx, st, rd, local, &w));
    const uint64_t *tot = w + 3;
    WETRIC_TRY(check_words(w[2] & 0xFFFFFFFFu, tot[1]));
    W = tot[0];
    rows = tot[2];
    r->max_out_degree = tot[1];
    int pick = -1;
    if (a.core_len != 0) {
      pick = cores.count ? 0 : -1;
    } else if (cores.count) {
      unsigned long long plan[2 * kCoreNumCandidates];
      for (uint32_t c = 0; c < kCoreNumCandidates; ++c) {
        plan[2 * c] = tot[kEdgeCand + 3 * c];
        plan[2 * c + 1] = tot[kEdgeCand + 3 * c + 1];
      }
      pick = core_pick(plan, kCoreWordsPerWalked);
    }
    if (pick >= 0 && cores.len[pick] >= 32) {  // else too small to pay for its launches
      core_h = cores.len[pick];
      core_v0 = n - core_h;
      below_m = w[kWords + pick];
      r->core_wedges = tot[kEdgeCand + 3 * pick];
      core_rows = tot[kEdgeCand + 3 * pick + 2];
      r->core_len = (uint32_t)core_h;
    }
    const WalkForm form = walk_form(n, m, below_m, tot[3], tot[1], tot[4]);
    if (form == WalkForm::kNone) {
      *declined = true;
      return WETRIC_OK;
    }
    emit = form == WalkForm::kWalk;
    sets = row_sets_wanted(below_m, W - r->core_wedges, tot[1], emit ? tot[4] : 0);
    // Room for an entry per edge below the core and a quarter more: tails
    // with two entries are rare (they need a long row with more than 48
    // columns outside the window), and a graph with more of them starts over
    // on the wedge-check path.
    int rc = WETRIC_OK;
    if (emit) rc = walk.alloc(ctx, st, n, m, tot[3], tot[1], below_m + below_m / 4);
    if (core_h) core_H4 = (uint32_t)(4 * ceil_div(core_h, 128));
    core_words = core_h ? core_row_off(core_H4, (uint32_t)core_h) + 4 : 0;
    if (rc == WETRIC_OK && core_h) rc = core.alloc(ctx, st, core_words);
    if (rc != WETRIC_OK) return without_room(rc);
    r->copies_issued = a.issue_copies != nullptr;
    if (a.issue_copies) WETRIC_TRY(a.issue_copies(a.issue_ctx));
  }

  const bool tma_ok = (reinterpret_cast<uintptr_t>(a.col_ind) & 15) == 0;
  if (core_h) WETRIC_CUDA_TRY(cudaMemsetAsync(core.ptr, 0, core_words * sizeof(uint32_t), st));

  NvtxRange nvtx_launch("wetric count: structures and kernels");
  EventPair ev_merge[kMaxColChunks], ev_core[kMaxColChunks], ev_walk;
  struct Event {
    cudaEvent_t e = nullptr;
    ~Event() {
      if (e) cudaEventDestroy(e);
    }
  } ev_made;
  uint64_t *made = readback_words();
  if (!made) made = local;
  const WalkColumns cols = walk_columns(a.col_ind, m);
  const uint32_t *rp32 = reinterpret_cast<const uint32_t *>(rp);  // unless small
  const uint64_t most_far = walk_most_far(W - r->core_wedges);
  for (uint32_t i = 0; i < C && n > 0; ++i) {
    const uint64_t lo = C_in ? a.chunk_lo[i] : 0, hi = i ? a.chunk_lo[i - 1] : n;
    const cudaEvent_t ready = C_in ? a.chunk_ready[i] : a.ci_ready;
    if (ready && !small) WETRIC_CUDA_TRY(cudaStreamWaitEvent(st, ready, 0));
    if (emit) {
      k_walk_split<false><<<WalkRun::grid(ctx, hi - lo), kWalkBlock, 0, st>>>(
          rp32, a.col_ind, n, lo, hi, walk.split.ptr, WalkGroups{}, walk.far(), most_far,
          err + 1);
      WETRIC_LAUNCH_CHECK();
      ++launches;
    }
    const uint64_t top = hi < core_v0 ? hi : core_v0;
    if (top > lo && below_m > 0) {
      // the chunk's share of the edges: at most all of them
      const uint32_t T = merge_tile(below_m, ctx->sm_count);
      const uint64_t g = ceil_div(ceil_div(below_m, T), kMergeBlock / 32);
      if (g > grid) grid = g;
      WETRIC_TRY(ev_merge[i].start(st));
      const auto merge = [&](auto kernel, const auto *offsets) {
        kernel<<<(unsigned)g, kMergeBlock, 0, st>>>(
            offsets, cols, n, lo, top, T, number.ptr, walk.split.ptr, walk.bits, walk.keys.ptr,
            (uint32_t)walk.cap, walk.counts.ptr, words.ptr, err, WalkGroups{},
            kMergeCount | kMergeEmit);
      };
      const auto form = [&](auto search) {
        constexpr bool kSearch = decltype(search)::value;
        if (emit && sets)
          merge(k_edge_merge<uint32_t, true, false, true, kSearch>, rp32);
        else if (emit)
          merge(k_edge_merge<uint32_t, true, false, false, kSearch>, rp32);
        else if (sets)
          merge(k_edge_merge<uint32_t, false, false, true, kSearch>, rp32);
        else
          merge(k_edge_merge<Off, false, false, false, kSearch>, rp);
      };
      // (a small graph's longest row is not known here)
      if (small || r->max_out_degree > kSearchOver)
        form(std::true_type());
      else
        form(std::false_type());
      WETRIC_LAUNCH_CHECK();
      ++launches;
      WETRIC_TRY(ev_merge[i].stop(st));
    }
    if (emit && i + 1 == C) {
      WETRIC_CUDA_TRY(cudaMemcpyAsync(made, walk.counts.ptr, WalkRun::kCounts * 4,
                                      cudaMemcpyDeviceToHost, st));
      WETRIC_CUDA_TRY(cudaEventCreateWithFlags(&ev_made.e, cudaEventDisableTiming));
      WETRIC_CUDA_TRY(cudaEventRecord(ev_made.e, st));
    }
    if (core_h && hi > core_v0) {
      const uint64_t r0 = (lo > core_v0 ? lo : core_v0) - core_v0, r1 = hi - core_v0;
      k_core_bitmap<Off><<<WalkRun::grid(ctx, (r1 - r0) * 32), 256, 0, st>>>(
          rp, a.col_ind, core_v0, (uint32_t)core_h, core_H4, core.ptr, (uint32_t)r0,
          (uint32_t)r1);
      WETRIC_LAUNCH_CHECK();
      WETRIC_TRY(ev_core[i].start(st));
      k_core_count<Off, true><<<(unsigned)(r1 - r0), kCoreBlock, 0, st>>>(
          a.col_ind, core.ptr, core_v0, (uint32_t)core_h, core_H4, nullptr, nullptr, nullptr, 0, 0,
          0, ~0ull, words.ptr, tma_ok, err, rp, core_v0 + r0);
      WETRIC_LAUNCH_CHECK();
      launches += 2;
      WETRIC_TRY(ev_core[i].stop(st));
    }
  }
  if (emit) {
    WETRIC_CUDA_TRY(cudaEventSynchronize(ev_made.e));
    const uint64_t entries = (uint32_t)*made;
    const WalkFar far{made[WalkRun::kFar / 2], made[WalkRun::kFar / 2 + 1],
                      made[WalkRun::kFar / 2 + 2], 0};
    if (entries > walk.cap || far.past(most_far)) {
      *declined = true;
      return WETRIC_OK;
    }
    if (far.rows) walk.share(ctx, st);
    if (entries > 0) {
      WETRIC_TRY(walk.sort(ctx, st, rp32, long_rows.ptr, entries, err, &launches));
      WETRIC_TRY(ev_walk.start(st));
      WETRIC_TRY(walk.count(ctx, st, rp32, a.col_ind, long_rows.ptr, a.persistent, words.ptr,
                            err, &grid, &launches));
      WETRIC_TRY(ev_walk.stop(st));
    }
  }
  uint64_t *host = readback_words();
  if (!host) host = local;
  const uint32_t back = small ? kWords : 3;
  WETRIC_CUDA_TRY(cudaMemcpyAsync(host, words.ptr, back * sizeof(uint64_t),
                                  cudaMemcpyDeviceToHost, st));
  WETRIC_TRY(ev_all.stop(st));
  WETRIC_CUDA_TRY(cudaEventSynchronize(ev_all.b));
  if (small) {
    W = host[3];
    rows = host[5];
    r->max_out_degree = host[4];
  }
  WETRIC_TRY(check_words(host[2] & 0xFFFFFFFFu, r->max_out_degree));
  r->triangles = host[0];
  r->pair_wedges = host[1];
  r->pair_rows = host[1] ? rows - core_rows : 0;
  r->wedges = r->wedges_counted = W;
  for (uint32_t i = 0; i < C; ++i) {
    WETRIC_TRY(ev_merge[i].add_to(&r->pair_ms));
    WETRIC_TRY(ev_core[i].add_to(&r->core_ms));
  }
  WETRIC_TRY(ev_walk.add_to(&r->count_ms));
  r->count_ms += r->pair_ms + r->core_ms;
  WETRIC_TRY(ev_all.add_to(&r->exec_ms));
  r->block = kWalkBlock;
  r->grid = (uint32_t)grid;
  r->launches = launches;
  return WETRIC_OK;
}

int count_whole(DeviceContext *ctx, cudaStream_t st, const CountArgs &a, CountResult *r,
                bool *declined) {
  *declined = false;
  if (a.offsets32) return whole_impl<uint32_t>(ctx, st, a, r, declined);
  return whole_impl<uint64_t>(ctx, st, a, r, declined);
}

}  // namespace wetric
