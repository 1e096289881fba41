// readback.cuh -- device values brought to the host in one copy.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace wetric {

constexpr uint32_t kReadWords = 128;     // values of one read-back at most
constexpr uint32_t kPinnedWords = 1024;  // of a thread
// Pinned words for the calling thread's read-backs (portable: any device),
// made on first use and freed when the thread ends; null if pinned memory
// cannot be had (the caller then reads into its own array).
inline uint64_t *readback_words() {
  struct Holder {
    uint64_t *p = nullptr;
    bool tried = false;
    ~Holder() {
      if (p) cudaFreeHost(p);
    }
  };
  thread_local Holder h;
  if (!h.tried) {
    h.tried = true;
    if (cudaHostAlloc(reinterpret_cast<void **>(&h.p), kPinnedWords * sizeof(uint64_t),
                      cudaHostAllocPortable) != cudaSuccess) {
      h.p = nullptr;
      cudaGetLastError();
    }
  }
  return h.p;
}
namespace {

// Host read-backs: one gather kernel collects the values into a device
// array and one copy brings them to pinned host memory. A copy into
// pageable memory (a stack variable) returns only when it is done, so one
// copy per value cost a round trip each while the device sat idle.
struct ReadSpan {
  const void *src;
  uint32_t count, bytes;  // elements of 4 or 8 bytes
};
constexpr uint32_t kReadSpans = 24;
struct ReadPlan {
  ReadSpan s[kReadSpans];
  uint32_t n = 0, total = 0;
  // Returns the first word of the span in the gathered array.
  uint32_t add(const void *src, uint32_t count, uint32_t bytes) {
    s[n++] = ReadSpan{src, count, bytes};
    total += count;
    return total - count;
  }
};
__global__ void k_read_gather(const __grid_constant__ ReadPlan p, uint64_t *__restrict__ out) {
  uint32_t j = threadIdx.x;  // one word per thread: its span, its element
  if (j >= p.total) return;
  uint32_t i = 0;
  while (j >= p.s[i].count) j -= p.s[i++].count;
  const ReadSpan &sp = p.s[i];
  out[threadIdx.x] = sp.bytes == 4 ? (uint64_t)static_cast<const uint32_t *>(sp.src)[j]
                                   : static_cast<const uint64_t *>(sp.src)[j];
}

static_assert(kReadWords <= 128 && kReadWords <= kPinnedWords, "a thread of the gather per word");
// Gathers plan's values on st, copies them to the host and waits (for
// `done`, recorded after the copy, when given); *words points at them
// afterwards (valid until the calling thread's next read).
int read_back(DeviceContext *ctx, cudaStream_t st, const ReadPlan &plan, uint64_t *local,
              const uint64_t **words, cudaEvent_t done = nullptr) {
  Scratch<uint64_t> dev;
  WETRIC_TRY(dev.alloc(ctx, st, plan.total));
  k_read_gather<<<1, 128, 0, st>>>(plan, dev.ptr);
  WETRIC_LAUNCH_CHECK();
  uint64_t *host = readback_words();
  if (!host) host = local;
  WETRIC_CUDA_TRY(cudaMemcpyAsync(host, dev.ptr, plan.total * sizeof(uint64_t),
                                  cudaMemcpyDeviceToHost, st));
  if (done) {
    WETRIC_CUDA_TRY(cudaEventRecord(done, st));
    WETRIC_CUDA_TRY(cudaEventSynchronize(done));
  } else {
    WETRIC_CUDA_TRY(cudaStreamSynchronize(st));
  }
  *words = host;
  return WETRIC_OK;
}

}  // namespace
}  // namespace wetric
