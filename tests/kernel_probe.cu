// Device code of the library as tests call it: the words that look-back
// scans publish, and scans of given values.
#include "primitives.cuh"

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
