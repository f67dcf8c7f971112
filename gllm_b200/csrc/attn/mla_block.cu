// The latent attention block of decoding sequences and short portions, from the hidden state to the heads' results, in one call from the
// host: both projections of the hidden state, their norms, the queries, W_UK per head, rotary + cache write, attention, W_UV per head.
// The kernels and their order are those of the separate entry points; this file only lays out the scratch and launches them.
//
// What bounds a decode batch that is launched eagerly is the host: eight launches of 15 to 18 us each through Python (asserts, an
// output tensor, some 20 converted arguments) against 109 us on the device for 128 sequences, 16 heads. From here a launch takes the
// driver's 3 us and the tensor maps. Block of 128 sequences, 16 heads, context up to 4096: 143 -> 103 us.
#include "../common/host_utils.h"

// The other families' entry points; null in a library that was built without them.
#define GLLM_WEAK extern "C" __attribute__((weak))
GLLM_WEAK int gllm_gemm_bf16(const void*, int64_t, const void*, int64_t, void*, int64_t, int, int, int, const void*, int, int,
                             const void*, void*, int64_t, void*, int, void*);
GLLM_WEAK int gllm_gemm_smallm(const void*, int64_t, const void*, int64_t, void*, int64_t, int, int, int, const void*, int, int, void*,
                               int64_t, void*, void*);
GLLM_WEAK int gllm_gemm_bf16_batched(const void*, int64_t, int64_t, const void*, void*, int64_t, int64_t, int, int, int, int, void*);
GLLM_WEAK int gllm_rmsnorm_two(const void*, int64_t, const void*, void*, int, const void*, int64_t, const void*, void*, int, int, float,
                               void*);
extern "C" int gllm_mla_attention(const void*, void*, const void*, int64_t, const void*, const void*, const void*, void*, void*, void*,
                                  int, int, int, int, int, float, int, const void*, void*);
extern "C" int gllm_mla_rope_cache(const void*, int64_t, int64_t, int, void*, int64_t, int64_t, const void*, int64_t, const void*,
                                   int64_t, const void*, const void*, const void*, void*, int, int, void*);

namespace {

constexpr int kLat = 512, kRot = 64, kNope = 128, kVal = 128, kFull = kLat + kRot, kHead = kNope + kRot;

// scratch of a call, each part on a 256-byte boundary
struct Parts {
  int64_t both, qa, kv_c, q, q_full, out_lat, part_o, part_lse, end;
};
Parts parts(int64_t t, int64_t heads, int64_t q_rank, int64_t ctas) {
  int64_t at = 0;
  auto take = [&](int64_t bytes) {
    const int64_t here = at;
    at += (bytes + 255) / 256 * 256;
    return here;
  };
  Parts p;
  p.both = take(t * (q_rank + kFull) * 2);
  p.qa = take(t * q_rank * 2);
  p.kv_c = take(t * kLat * 2);
  p.q = take(t * heads * kHead * 2);
  p.q_full = take(t * heads * kFull * 2);
  p.out_lat = take(t * heads * kLat * 2);
  p.part_o = take(ctas * 2 * 16 * kLat * 4);
  p.part_lse = take(ctas * (2 * 16 + 4) * 4);
  p.end = at;
  return p;
}

}  // namespace

// bytes of scratch that gllm_mla_block needs
GLLM_EXPORT int64_t gllm_mla_block_scratch(int t, int heads, int q_rank, int ctas) { return parts(t, heads, q_rank, ctas).end; }

// h [t, width] (rows ldh apart); qkv_a [q_rank + 576, width], q_b [heads * 192, q_rank], w_uk [heads, 512, 128], w_uv [heads, 128, 512];
// out [t, heads, 128]. few: the most rows that the kernel for a few rows takes (64 for K >= 8192). The others as in the entry points.
GLLM_EXPORT int gllm_mla_block(const void* h, int64_t ldh, int t, int width, int heads, int q_rank, const void* qkv_a, const void* q_norm,
                               const void* kv_norm, float eps, const void* q_b, const void* w_uk, const void* w_uv, const void* cos_sin,
                               const void* positions, const void* slots, void* cache, int64_t num_pages, int page_size,
                               const void* block_table, int max_blocks, const void* tok_seq, float scale, int ctas, void* out,
                               void* scratch, int64_t scratch_bytes, void* ws, int64_t ws_floats, void* few_cnt, void* tile_cnt,
                               int max_tiles, int few, void* stream) {
  if (t <= 0) return 0;
  if (gllm_gemm_bf16 == nullptr || gllm_gemm_smallm == nullptr || gllm_gemm_bf16_batched == nullptr || gllm_rmsnorm_two == nullptr) {
    fprintf(stderr, "[gllm_b200] mla_block: the library was built without the gemm or elemwise kernels\n");
    return 1;
  }
  const Parts at = parts(t, heads, q_rank, ctas);
  if (scratch_bytes < at.end) return 1;
  char* s = static_cast<char*>(scratch);
  auto linear = [&](const void* x, int64_t ldx, const void* w, void* y, int n, int k) {
    return t <= few || (t <= 64 && k >= 8192)
               ? gllm_gemm_smallm(x, ldx, w, k, y, n, t, n, k, nullptr, 0, 0, ws, ws_floats, few_cnt, stream)
               : gllm_gemm_bf16(x, ldx, w, k, y, n, t, n, k, nullptr, 0, 0, nullptr, ws, ws_floats * 4, tile_cnt, max_tiles, stream);
  };
  const int both_n = q_rank + kFull;
  char *both = s + at.both, *kv_a = both + q_rank * 2, *q = s + at.q, *q_full = s + at.q_full, *out_lat = s + at.out_lat;
  int rc = linear(h, ldh, qkv_a, both, both_n, width);
  if (rc == 0)
    rc = gllm_rmsnorm_two(both, both_n, q_norm, s + at.qa, q_rank, kv_a, both_n, kv_norm, s + at.kv_c, kLat, t, eps, stream);
  if (rc == 0) rc = linear(s + at.qa, q_rank, q_b, q, heads * kHead, q_rank);
  if (rc == 0)
    rc = gllm_gemm_bf16_batched(q, heads * kHead, kHead, w_uk, q_full, heads * kFull, kFull, t, heads, kLat, kNope, stream);
  if (rc == 0)
    rc = gllm_mla_rope_cache(q + kNope * 2, heads * kHead, kHead, heads, q_full + kLat * 2, heads * kFull, kFull, kv_a + kLat * 2, both_n,
                             s + at.kv_c, kLat, cos_sin, positions, slots, cache, page_size, t, stream);
  if (rc == 0)
    rc = gllm_mla_attention(q_full, out_lat, cache, num_pages, block_table, tok_seq, positions, s + at.part_o, s + at.part_lse,
                            s + at.part_lse + ctas * 32 * 4, t, max_blocks, heads, page_size, ctas, scale, 0, nullptr, stream);
  if (rc == 0) rc = gllm_gemm_bf16_batched(out_lat, heads * kLat, kLat, w_uv, out, heads * kVal, kVal, t, heads, kVal, kLat, stream);
  return rc;
}
