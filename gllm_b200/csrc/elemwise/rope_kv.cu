// Fused  [per-head q/k RMSNorm] -> RoPE (NeoX / GPT-J / partial / M-RoPE) -> paged KV-cache write.
//
// One pass over the QKV projection output replaces four kernels of the reference:
// q_norm/k_norm (gllm/models/qwen3.py:75-80), `_C.rotary_embedding`
// (gllm/layers/rotary_embedding.py:91-110), the Triton M-RoPE kernel (:342-506) and
// `reshape_and_cache_flash` (gllm/memory_manager.py:154-163).
//
// KV cache layout (ours, chosen for TMA): [num_pages, Hkv, D/64, page_size, 64] bf16 — each
// (page, head, 64-wide slice) is a contiguous page_size x 128 B slab that one TMA box with the
// 128-byte swizzle turns into a conflict-free tile for the attention kernels.
#include "../common/host_utils.h"
#include "../common/ptx.cuh"

namespace b200 {

struct RopeParams {
  __nv_bfloat16* q; int64_t q_ts, q_hs; int Hq;
  __nv_bfloat16* k; int64_t k_ts, k_hs; int Hkv;
  const __nv_bfloat16* v; int64_t v_ts, v_hs;
  const __nv_bfloat16* q_norm_w;
  const __nv_bfloat16* k_norm_w;
  const float* cos_sin;  // [max_pos, rot]: cos | sin
  int D, rot, neox, T;
  const int32_t* positions;  // [T] or [3, T] (mrope)
  const int32_t* slots;      // [T] or null
  float eps;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  int sec0, sec1, page_size;  // sec0 > 0: chunked M-RoPE [T|H|W]; sec0 < 0: interleaved (H = -sec0, W = sec1)
  int64_t pos_stride;         // row stride of a [3, T] positions tensor
};

// which of the (t, h, w) position rows rotary pair i uses
__device__ __forceinline__ int mrope_axis(int i, int sec0, int sec1) {
  if (sec0 > 0) return i < sec0 ? 0 : (i < sec0 + sec1 ? 1 : 2);
  if (sec0 < 0) {
    const int r = i % 3;
    if (r == 1 && i < -sec0 * 3) return 1;
    if (r == 2 && i < sec1 * 3) return 2;
  }
  return 0;
}

template <int C>  // elements per lane, D = 32 * C
__global__ void rope_kv_kernel(const RopeParams p) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int D = 32 * C;
  const int half = p.rot >> 1;
  const int e0 = lane * C;  // first element of this lane
  const bool do_rope = p.rot > 0;
  const int n_heads = p.Hq + p.Hkv + ((p.v != nullptr && p.slots != nullptr) ? p.Hkv : 0);

  int pos[3];
  if (p.sec0 != 0) {
    pos[0] = p.positions[t]; pos[1] = p.positions[p.pos_stride + t]; pos[2] = p.positions[2 * p.pos_stride + t];
  } else {
    pos[0] = pos[1] = pos[2] = p.positions != nullptr ? p.positions[t] : 0;
  }
  const int slot = p.slots != nullptr ? p.slots[t] : -1;

  // one head per warp: blockIdx.y strides the head list so a decode batch still fills the machine and no
  // warp walks several heads serially (the per-head chain of dependent global loads is the whole cost)
  for (int hh = blockIdx.y * nwarps + warp; hh < n_heads; hh += nwarps * gridDim.y) {
    const bool is_q = hh < p.Hq;
    const bool is_k = !is_q && hh < p.Hq + p.Hkv;
    const int h = is_q ? hh : (is_k ? hh - p.Hq : hh - p.Hq - p.Hkv);
    float x[C];
    if (is_q || is_k) {
      __nv_bfloat16* ptr = is_q ? p.q + t * p.q_ts + h * p.q_hs : p.k + t * p.k_ts + h * p.k_hs;
      const __nv_bfloat16* nw = is_q ? p.q_norm_w : p.k_norm_w;
#pragma unroll
      for (int e = 0; e < C; e += 2) {
        float2 f = unpack_bf16(*reinterpret_cast<const uint32_t*>(ptr + e0 + e));
        x[e] = f.x; x[e + 1] = f.y;
      }
      if (nw != nullptr) {
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < C; ++e) ss += x[e] * x[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = rsqrtf(ss / static_cast<float>(D) + p.eps);
#pragma unroll
        for (int e = 0; e < C; e += 2) {
          float2 wv = unpack_bf16(*reinterpret_cast<const uint32_t*>(nw + e0 + e));
          // round to bf16 after the norm like the unfused reference does
          x[e] = __bfloat162float(__float2bfloat16(x[e] * inv * wv.x));
          x[e + 1] = __bfloat162float(__float2bfloat16(x[e + 1] * inv * wv.y));
        }
      }
      if (do_rope) {
        if (p.neox) {
          // partner element lives `half` elements away -> lane +- half / C
          const int dl = half / C;
          const bool lo = e0 < half;
          const bool in_rot = e0 < p.rot;
          const int src = lo ? lane + dl : lane - dl;
          float y[C];
#pragma unroll
          for (int e = 0; e < C; ++e) y[e] = __shfl_sync(0xffffffffu, x[e], src & 31);
          if (in_rot) {
#pragma unroll
            for (int e = 0; e < C; ++e) {
              const int i = (e0 + e) % half;
              const int ps = pos[mrope_axis(i, p.sec0, p.sec1)];
              const float c = p.cos_sin[static_cast<size_t>(ps) * p.rot + i];
              const float s = p.cos_sin[static_cast<size_t>(ps) * p.rot + half + i];
              x[e] = lo ? x[e] * c - y[e] * s : x[e] * c + y[e] * s;
            }
          }
        } else {
          if (e0 < p.rot) {
#pragma unroll
            for (int e = 0; e < C; e += 2) {
              const int i = (e0 + e) >> 1;
              const int ps = pos[mrope_axis(i, p.sec0, p.sec1)];
              const float c = p.cos_sin[static_cast<size_t>(ps) * p.rot + i];
              const float s = p.cos_sin[static_cast<size_t>(ps) * p.rot + half + i];
              const float a = x[e], b = x[e + 1];
              x[e] = a * c - b * s;
              x[e + 1] = b * c + a * s;
            }
          }
        }
      }
      uint32_t packed[C / 2];
#pragma unroll
      for (int e = 0; e < C; e += 2) packed[e / 2] = pack_bf16(x[e], x[e + 1]);
#pragma unroll
      for (int e = 0; e < C / 2; ++e) *reinterpret_cast<uint32_t*>(ptr + e0 + 2 * e) = packed[e];
      if (is_k && slot >= 0 && p.k_cache != nullptr) {
        const int page = slot / p.page_size, off = slot - page * p.page_size;
        const size_t base = ((static_cast<size_t>(page) * p.Hkv + h) * (D / 64) + e0 / 64) * p.page_size * 64 +
                            static_cast<size_t>(off) * 64 + (e0 % 64);
#pragma unroll
        for (int e = 0; e < C / 2; ++e) *reinterpret_cast<uint32_t*>(p.k_cache + base + 2 * e) = packed[e];
      }
    } else if (slot >= 0) {
      const __nv_bfloat16* ptr = p.v + t * p.v_ts + h * p.v_hs;
      const int page = slot / p.page_size, off = slot - page * p.page_size;
      const size_t base = ((static_cast<size_t>(page) * p.Hkv + h) * (D / 64) + e0 / 64) * p.page_size * 64 +
                          static_cast<size_t>(off) * 64 + (e0 % 64);
#pragma unroll
      for (int e = 0; e < C; e += 2)
        *reinterpret_cast<uint32_t*>(p.v_cache + base + e) = *reinterpret_cast<const uint32_t*>(ptr + e0 + e);
    }
  }
}

// The same pass with 16-byte accesses: L = D / 8 lanes per head, 32 / L heads per warp, NB heads per lane group, all
// loaded before the first is written (the update is in place, so the compiler cannot move a later head's load over an
// earlier head's store), the rotation row read once for all of them. Memory-bound: every q / k element is read and
// written once, v and the cache rows once more. The kernel above has one head per warp and re-reads its cos / sin row for
// every head in 4-byte words. Cold L2, heads of 128, before and after: 4096 tokens x (32 + 8 + 8) heads 91 -> 43 us (2.7
// TB/s), 8192 x (64 + 8 + 8) 290 -> 114 us, 256 x (32 + 8 + 8) 13 -> 11 us; heads of 64, 4096 x 48: 68 -> 26 us. Whole NeoX heads of
// 64 and 128 take the kernel below.
template <int L, int NB>
__global__ void __launch_bounds__(128) rope_kv_vec_kernel(const RopeParams p) {
  griddep_launch();
  griddep_wait();
  constexpr int D = 8 * L, kHeadsPerWarp = 32 / L, kStep = 4 * kHeadsPerWarp;
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gl = lane % L, e0 = gl * 8;
  const int half = p.rot >> 1;
  const int n_qk = p.Hq + p.Hkv;
  const int n_heads = n_qk + ((p.v != nullptr && p.slots != nullptr) ? p.Hkv : 0);
  const int first = blockIdx.y * (kStep * NB) + warp * kHeadsPerWarp + lane / L;
  const int slot = p.slots != nullptr ? p.slots[t] : -1;

  uint4 raw[NB];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const int hh = first + n * kStep;
    raw[n] = make_uint4(0u, 0u, 0u, 0u);
    if (hh < n_heads) {
      const __nv_bfloat16* src = hh < p.Hq ? p.q + t * p.q_ts + hh * p.q_hs
                                 : hh < n_qk ? p.k + t * p.k_ts + (hh - p.Hq) * p.k_hs
                                             : p.v + t * p.v_ts + (hh - n_qk) * p.v_hs;
      if (hh < n_qk || slot >= 0) raw[n] = *reinterpret_cast<const uint4*>(src + e0);
    }
  }
  // this lane's rotation row: pair index of element e is (e0 + e) % half (NeoX) or (e0 + e) / 2 (adjacent pairs)
  float c[8], s[8];
  const bool in_rot = e0 < p.rot, lo = e0 < half;
  if (in_rot) {
    if (p.sec0 != 0) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = p.neox ? e0 + e - (lo ? 0 : half) : (e0 + e) >> 1;
        const int ax = mrope_axis(i, p.sec0, p.sec1);
        const float* row = p.cos_sin + static_cast<size_t>(p.positions[ax * p.pos_stride + t]) * p.rot;
        c[e] = row[i];
        s[e] = row[half + i];
      }
    } else {
      const float* row = p.cos_sin + static_cast<size_t>(p.positions != nullptr ? p.positions[t] : 0) * p.rot;
      if (p.neox) {
        const int i = e0 - (lo ? 0 : half);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const float4 cv = *reinterpret_cast<const float4*>(row + i + 4 * g);
          const float4 sv = *reinterpret_cast<const float4*>(row + half + i + 4 * g);
          c[4 * g] = cv.x; c[4 * g + 1] = cv.y; c[4 * g + 2] = cv.z; c[4 * g + 3] = cv.w;
          s[4 * g] = sv.x; s[4 * g + 1] = sv.y; s[4 * g + 2] = sv.z; s[4 * g + 3] = sv.w;
        }
      } else {
        const float4 cv = *reinterpret_cast<const float4*>(row + e0 / 2);
        const float4 sv = *reinterpret_cast<const float4*>(row + half + e0 / 2);
        c[0] = c[1] = cv.x; c[2] = c[3] = cv.y; c[4] = c[5] = cv.z; c[6] = c[7] = cv.w;
        s[0] = s[1] = sv.x; s[2] = s[3] = sv.y; s[4] = s[5] = sv.z; s[6] = s[7] = sv.w;
      }
    }
  }
  const int dl = half / 8;
  const int partner = (lane & ~(L - 1)) | ((lo ? gl + dl : gl - dl) & (L - 1));
  size_t cache_at = 0;
  if (slot >= 0) {
    const int page = slot / p.page_size, off = slot - page * p.page_size;
    cache_at = (static_cast<size_t>(page) * p.Hkv * (D / 64) + e0 / 64) * p.page_size * 64 + static_cast<size_t>(off) * 64 +
               (e0 % 64);
  }
  const size_t head_stride = static_cast<size_t>(D / 64) * p.page_size * 64;
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const int hh = first + n * kStep;
    const bool is_q = hh < p.Hq, is_qk = hh < n_qk;
    const uint32_t rw[4] = {raw[n].x, raw[n].y, raw[n].z, raw[n].w};
    float x[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack_bf16(rw[e]);
      x[2 * e] = f.x;
      x[2 * e + 1] = f.y;
    }
    const __nv_bfloat16* nw = is_q ? p.q_norm_w : p.k_norm_w;
    if (p.q_norm_w != nullptr || p.k_norm_w != nullptr) {
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += x[e] * x[e];
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (is_qk && nw != nullptr) {
        const float inv = rsqrtf(ss / static_cast<float>(D) + p.eps);
        const uint4 wv = *reinterpret_cast<const uint4*>(nw + e0);
        const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = unpack_bf16(ww[e]);
          // round to bf16 after the norm like the unfused reference does
          x[2 * e] = __bfloat162float(__float2bfloat16(x[2 * e] * inv * f.x));
          x[2 * e + 1] = __bfloat162float(__float2bfloat16(x[2 * e + 1] * inv * f.y));
        }
      }
    }
    if (p.rot > 0) {
      if (p.neox) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float y = __shfl_sync(0xffffffffu, x[e], partner);
          if (in_rot) x[e] = lo ? x[e] * c[e] - y * s[e] : x[e] * c[e] + y * s[e];
        }
      } else if (in_rot) {
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const float a = x[e], b = x[e + 1];
          x[e] = a * c[e] - b * s[e];
          x[e + 1] = b * c[e] + a * s[e];
        }
      }
    }
    if (hh >= n_heads) continue;
    if (is_qk) {
      const uint4 w = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
      __nv_bfloat16* dst = is_q ? p.q + t * p.q_ts + hh * p.q_hs : p.k + t * p.k_ts + (hh - p.Hq) * p.k_hs;
      *reinterpret_cast<uint4*>(dst + e0) = w;
      if (!is_q && slot >= 0 && p.k_cache != nullptr)
        *reinterpret_cast<uint4*>(p.k_cache + cache_at + (hh - p.Hq) * head_stride) = w;
    } else if (slot >= 0) {
      *reinterpret_cast<uint4*>(p.v_cache + cache_at + (hh - n_qk) * head_stride) = raw[n];
    }
  }
}

// NeoX rotation of whole heads (rot = D), the common form: a lane holds eight elements of the lower half and their partners of the
// upper one, so that nothing is exchanged for the rotation (eight shuffles per eight elements above) and its row (read once for NB
// heads) is half as long per lane. The projections come from L2, so the chain position -> row -> rotation and the issue slots bound it.
// Heads of 128 with norms, in an attention block, kernel above and this one: 4096 tokens x (32 + 8 + 8) heads 38.6 -> 24.1 us (4.2
// TB/s), 8192 x (64 + 8 + 8) without norms 106 -> 71 us, 256 x (32 + 8 + 8) 5.6 -> 3.6 us.
template <int L, int NB>
__global__ void __launch_bounds__(128) rope_kv_pair_kernel(const RopeParams p) {
  griddep_launch();
  griddep_wait();
  constexpr int D = 16 * L, H = D / 2, kHeadsPerWarp = 32 / L, kStep = 4 * kHeadsPerWarp;
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = (lane % L) * 8;
  const int n_qk = p.Hq + p.Hkv;
  const int n_heads = n_qk + ((p.v != nullptr && p.slots != nullptr) ? p.Hkv : 0);
  const int first = blockIdx.y * (kStep * NB) + warp * kHeadsPerWarp + lane / L;
  const int pos = p.positions != nullptr ? p.positions[t] : 0, slot = p.slots != nullptr ? p.slots[t] : -1;

  uint4 raw[NB][2];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const int hh = first + n * kStep;
    raw[n][0] = raw[n][1] = make_uint4(0u, 0u, 0u, 0u);
    if (hh < n_heads && (hh < n_qk || slot >= 0)) {
      const __nv_bfloat16* src = hh < p.Hq ? p.q + t * p.q_ts + hh * p.q_hs
                                 : hh < n_qk ? p.k + t * p.k_ts + (hh - p.Hq) * p.k_hs
                                             : p.v + t * p.v_ts + (hh - n_qk) * p.v_hs;
      raw[n][0] = *reinterpret_cast<const uint4*>(src + e0);
      raw[n][1] = *reinterpret_cast<const uint4*>(src + H + e0);
    }
  }
  float c[8], s[8];
  const float* row = p.cos_sin + static_cast<size_t>(pos) * D + e0;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const float4 cv = *reinterpret_cast<const float4*>(row + 4 * g), sv = *reinterpret_cast<const float4*>(row + H + 4 * g);
    c[4 * g] = cv.x; c[4 * g + 1] = cv.y; c[4 * g + 2] = cv.z; c[4 * g + 3] = cv.w;
    s[4 * g] = sv.x; s[4 * g + 1] = sv.y; s[4 * g + 2] = sv.z; s[4 * g + 3] = sv.w;
  }
  const size_t slab = static_cast<size_t>(p.page_size) * 64;
  size_t at = 0;                                           // of the lower eight elements in head 0 of the slot's page
  if (slot >= 0) {
    const int page = slot / p.page_size, off = slot - page * p.page_size;
    at = static_cast<size_t>(page) * p.Hkv * (D / 64) * slab + static_cast<size_t>(off) * 64 + e0;
  }
  const size_t upper = D == 64 ? 32 : slab;                // ... and from there to the upper eight
  const bool norm = p.q_norm_w != nullptr || p.k_norm_w != nullptr;
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const int hh = first + n * kStep;
    const bool is_q = hh < p.Hq;
    float x[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t rw[4] = {raw[n][i].x, raw[n][i].y, raw[n][i].z, raw[n][i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack_bf16(rw[e]);
        x[i][2 * e] = f.x;
        x[i][2 * e + 1] = f.y;
      }
    }
    if (norm) {
      float ss = 0.f, upper_ss = 0.f;                    // apart: the order of the sums is the kernel's above, and so are the bits
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        ss += x[0][e] * x[0][e];
        upper_ss += x[1][e] * x[1][e];
      }
      ss += upper_ss;
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const __nv_bfloat16* nw = is_q ? p.q_norm_w : p.k_norm_w;
      if (hh < n_qk && nw != nullptr) {
        const float inv = rsqrtf(ss / static_cast<float>(D) + p.eps);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 wv = *reinterpret_cast<const uint4*>(nw + i * H + e0);
          const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_bf16(ww[e]);
            // rounded to bf16 after the norm, as the unfused form does
            x[i][2 * e] = __bfloat162float(__float2bfloat16(x[i][2 * e] * inv * f.x));
            x[i][2 * e + 1] = __bfloat162float(__float2bfloat16(x[i][2 * e + 1] * inv * f.y));
          }
        }
      }
    }
    if (hh >= n_heads) continue;
    if (hh < n_qk) {
      uint32_t w[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float r[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int i = 2 * e + j;
          r[0][j] = x[0][i] * c[i] - x[1][i] * s[i];
          r[1][j] = x[1][i] * c[i] + x[0][i] * s[i];
        }
        w[0][e] = pack_bf16(r[0][0], r[0][1]);
        w[1][e] = pack_bf16(r[1][0], r[1][1]);
      }
      const uint4 a = make_uint4(w[0][0], w[0][1], w[0][2], w[0][3]), b = make_uint4(w[1][0], w[1][1], w[1][2], w[1][3]);
      __nv_bfloat16* dst = is_q ? p.q + t * p.q_ts + hh * p.q_hs : p.k + t * p.k_ts + (hh - p.Hq) * p.k_hs;
      *reinterpret_cast<uint4*>(dst + e0) = a;
      *reinterpret_cast<uint4*>(dst + H + e0) = b;
      if (!is_q && slot >= 0 && p.k_cache != nullptr) {
        __nv_bfloat16* k = p.k_cache + at + (hh - p.Hq) * (D / 64) * slab;
        *reinterpret_cast<uint4*>(k) = a;
        *reinterpret_cast<uint4*>(k + upper) = b;
      }
    } else if (slot >= 0) {
      __nv_bfloat16* v = p.v_cache + at + (hh - n_qk) * (D / 64) * slab;
      *reinterpret_cast<uint4*>(v) = raw[n][0];
      *reinterpret_cast<uint4*>(v + upper) = raw[n][1];
    }
  }
}

template <int L>
static cudaError_t launch_rope_pair(const RopeParams& p, int n_heads, cudaStream_t st) {
  constexpr int kStep = 4 * (32 / L);
  if (static_cast<int64_t>(p.T) * n_heads >= static_cast<int64_t>(num_sms()) * 16 * kStep * 2)
    return launch_pdl(rope_kv_pair_kernel<L, 2>, dim3(p.T, (n_heads + 2 * kStep - 1) / (2 * kStep)), dim3(128), 0, st, p);
  return launch_pdl(rope_kv_pair_kernel<L, 1>, dim3(p.T, (n_heads + kStep - 1) / kStep), dim3(128), 0, st, p);
}

template <int L>
static cudaError_t launch_rope_vec(const RopeParams& p, int n_heads, cudaStream_t st) {
  constexpr int kStep = 4 * (32 / L);
  // many tokens: NB heads per lane, fewer and longer blocks; a decode batch: one, so that it still fills the machine
  if (static_cast<int64_t>(p.T) * n_heads >= static_cast<int64_t>(num_sms()) * 16 * kStep * 4)
    return launch_pdl(rope_kv_vec_kernel<L, 4>, dim3(p.T, (n_heads + 4 * kStep - 1) / (4 * kStep)), dim3(128), 0, st, p);
  return launch_pdl(rope_kv_vec_kernel<L, 1>, dim3(p.T, (n_heads + kStep - 1) / kStep), dim3(128), 0, st, p);
}

}  // namespace b200

using namespace b200;

GLLM_EXPORT int gllm_rope_kv_write(void* q, int64_t q_ts, int64_t q_hs, int Hq, void* k, int64_t k_ts,
                                   int64_t k_hs, int Hkv, const void* v, int64_t v_ts, int64_t v_hs,
                                   const void* q_norm_w, const void* k_norm_w, const void* cos_sin, int D,
                                   int rot, int neox, int T, const void* positions, const void* slots,
                                   float eps, void* k_cache, void* v_cache, int sec0, int sec1,
                                   int page_size, int64_t pos_stride, void* stream) {
  if (T <= 0) return 0;
  RopeParams p;
  p.q = reinterpret_cast<__nv_bfloat16*>(q); p.q_ts = q_ts; p.q_hs = q_hs; p.Hq = Hq;
  p.k = reinterpret_cast<__nv_bfloat16*>(k); p.k_ts = k_ts; p.k_hs = k_hs; p.Hkv = Hkv;
  p.v = reinterpret_cast<const __nv_bfloat16*>(v); p.v_ts = v_ts; p.v_hs = v_hs;
  p.q_norm_w = reinterpret_cast<const __nv_bfloat16*>(q_norm_w);
  p.k_norm_w = reinterpret_cast<const __nv_bfloat16*>(k_norm_w);
  p.cos_sin = reinterpret_cast<const float*>(cos_sin);
  p.D = D; p.rot = rot; p.neox = neox; p.T = T;
  p.positions = reinterpret_cast<const int32_t*>(positions);
  p.slots = reinterpret_cast<const int32_t*>(slots);
  p.eps = eps;
  p.k_cache = reinterpret_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = reinterpret_cast<__nv_bfloat16*>(v_cache);
  p.sec0 = sec0; p.sec1 = sec1; p.page_size = page_size; p.pos_stride = pos_stride;
  const int C = D / 32;
  if (D % 64 != 0 || (rot > 0 && ((rot / 2) % C != 0 || rot > D))) {
    fprintf(stderr, "[gllm_b200] rope_kv_write: unsupported D=%d rot=%d\n", D, rot);
    return 1;
  }
  const int n_heads = Hq + 2 * Hkv;
  // 16-byte form: every row, the weights and the cache on 16-byte boundaries, and no lane of 8 elements astride the end of
  // the rotated part or of its halves
  auto al16 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
  const bool vec = (D == 64 || D == 128 || D == 256) && ((q_ts | q_hs | k_ts | k_hs) & 7) == 0 &&
                   (v == nullptr || ((v_ts | v_hs) & 7) == 0) && al16(q) && al16(k) && al16(v) && al16(q_norm_w) &&
                   al16(k_norm_w) && al16(cos_sin) && al16(k_cache) && al16(v_cache) &&
                   (rot == 0 || (neox ? rot % 16 == 0 : rot % 8 == 0));
  if (vec) {
    cudaStream_t vst = reinterpret_cast<cudaStream_t>(stream);
    if (neox && rot == D && D <= 128 && sec0 == 0 && cos_sin != nullptr) {
      CUDA_CHECK_RET(D == 64 ? launch_rope_pair<4>(p, n_heads, vst) : launch_rope_pair<8>(p, n_heads, vst));
      return 0;
    }
    CUDA_CHECK_RET(D == 64 ? launch_rope_vec<8>(p, n_heads, vst)
                           : D == 128 ? launch_rope_vec<16>(p, n_heads, vst) : launch_rope_vec<32>(p, n_heads, vst));
    return 0;
  }
  int warps = n_heads < 4 ? n_heads : 4;
  if (warps < 1) warps = 1;
  const dim3 grid(T, (n_heads + warps - 1) / warps);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (C) {
    case 2: CUDA_CHECK_RET(launch_pdl(rope_kv_kernel<2>, grid, dim3(warps * 32), 0, st, p)); break;
    case 4: CUDA_CHECK_RET(launch_pdl(rope_kv_kernel<4>, grid, dim3(warps * 32), 0, st, p)); break;
    case 8: CUDA_CHECK_RET(launch_pdl(rope_kv_kernel<8>, grid, dim3(warps * 32), 0, st, p)); break;
    default:
      fprintf(stderr, "[gllm_b200] rope_kv_write: unsupported head_dim %d\n", D);
      return 1;
  }
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}
