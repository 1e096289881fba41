// The preprocessing's kernels behind a sort, as tests call them: on device
// arrays, with a given error word *err.
#include "preprocess.cu"

// The unique keys among N sorted ones of b bits each, the degrees they make,
// and the CSR of all N as (row, column).
extern "C" int probe_after_sort(const uint64_t *keys, uint64_t N, uint64_t n, uint32_t b,
                                uint64_t *state, uint64_t *unique, uint32_t *deg, uint64_t *made,
                                uint64_t *rp, uint32_t *ci, uint32_t *err) {
  using namespace wetric;
  const uint64_t tiles = ceil_div(N, kUniqueTile);
  k_unique_degrees<<<(unsigned)tiles, kThreads>>>(keys, N, ~0ull, b, unique, deg, state + 1,
                                                  reinterpret_cast<uint32_t *>(state), made, err);
  k_keys_to_csr<<<4, kThreads>>>(keys, N, n, b, rp, ci, err);
  if (cudaGetLastError() != cudaSuccess) return -1;
  return (int)cudaDeviceSynchronize();
}

// kept[rank[v]] = columns of row v whose rank is above its own.
extern "C" int probe_kept(const uint64_t *rp, const uint32_t *ci, uint64_t n, const uint32_t *rank,
                          uint32_t *kept, uint64_t *most, const uint32_t *err) {
  wetric::k_kept_per_row<<<4, 256>>>(rp, ci, n, rank, kept, most, err);
  if (cudaGetLastError() != cudaSuccess) return -1;
  return (int)cudaDeviceSynchronize();
}
