// MoE routing + token permutation kernels for sm_100a.
//
//   topk_softmax      softmax over experts + top-k (+renorm)            (ref: vLLM _moe_C.topk_softmax,
//                                                                         gllm/layers/moe/topk.py:141-171)
//   grouped_topk      DeepSeek group-limited routing (sigmoid/softmax scores, bias correction, top
//                     groups by sum of top-2 / max, renorm, scaling)     (gllm/layers/moe/topk.py:29-138)
//   moe_align         counting sort of the (token, k) slots by LOCAL expert into 128-row tiles:
//                     expert_count -> padded offsets -> per-tile expert id, slot -> row position
//                     (ref: moe_align_block_size, gllm/layers/moe/moe_align_block_size.py:10-78)
//   moe_gather        xs[row] = x[token(row)], as it is or quantised to e4m3; up to 4096 slots in one launch with the sort
//   moe_combine       out[t] = sum_j w[t,j] * y[pos[t,j]]   (ref: moe_sum, fused with the routing weight)
//
// The expert GEMMs themselves are the tcgen05 kernel in gemm/gemm_bf16.cu running in grouped mode
// (per-M-tile expert id selects the weight slab; the tile count is read from device memory so the
// whole MoE block is CUDA-graph capturable without a host sync).
#include "../common/fp8_quant.cuh"
#include "../common/host_utils.h"
#include "../common/ptx.cuh"

namespace b200 {

static constexpr int kTileM = 128;

// ---------------------------------------------------------------------------------------------
// top-k softmax: one warp per token, E <= 512
// ---------------------------------------------------------------------------------------------
template <int VPT>  // values per lane, E <= 32 * VPT
__global__ void topk_softmax_kernel(const __nv_bfloat16* __restrict__ logits, int64_t ld, float* __restrict__ w_out,
                                    int32_t* __restrict__ id_out, int T, int E, int K, int renorm) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= T) return;
  const __nv_bfloat16* row = logits + static_cast<size_t>(warp) * ld;
  float v[VPT];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int e = lane + i * 32;
    v[i] = e < E ? __bfloat162float(row[e]) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    v[i] = (lane + i * 32 < E) ? __expf(v[i] - mx) : 0.f;
    sum += v[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.f / sum;
  float wsum = 0.f;
  float my_w = 0.f;
  int my_id = 0;
  for (int k = 0; k < K; ++k) {
    float best = -1.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int e = lane + i * 32;
      if (v[i] > best) { best = v[i]; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if ((bi & 31) == lane) v[bi >> 5] = -1.f;  // remove the winner
    if (lane == k) { my_w = best * inv; my_id = bi; }
    wsum += best * inv;
  }
  if (lane < K) {
    w_out[static_cast<size_t>(warp) * K + lane] = renorm ? my_w / wsum : my_w;
    id_out[static_cast<size_t>(warp) * K + lane] = my_id;
  }
}

// ---------------------------------------------------------------------------------------------
// grouped top-k (DeepSeek): one warp per token, E <= 512, groups <= 32
// ---------------------------------------------------------------------------------------------
template <int VPT>
__global__ void grouped_topk_kernel(const __nv_bfloat16* __restrict__ logits, int64_t ld, const float* __restrict__ bias,
                                    float* __restrict__ w_out, int32_t* __restrict__ id_out, int T, int E, int K,
                                    int n_group, int topk_group, int renorm, int sigmoid, float scaling) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= T) return;
  const __nv_bfloat16* row = logits + static_cast<size_t>(warp) * ld;
  // expert e = lane * VPT + i  (contiguous per lane so a group maps to whole lanes when E/n_group >= VPT)
  float sc[VPT], sel[VPT];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int e = lane * VPT + i;
    sc[i] = e < E ? __bfloat162float(row[e]) : -INFINITY;
    mx = fmaxf(mx, sc[i]);
  }
  if (sigmoid) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) sc[i] = (lane * VPT + i < E) ? 1.f / (1.f + __expf(-sc[i])) : 0.f;
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) { sc[i] = (lane * VPT + i < E) ? __expf(sc[i] - mx) : 0.f; sum += sc[i]; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
    for (int i = 0; i < VPT; ++i) sc[i] /= sum;
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int e = lane * VPT + i;
    sel[i] = e < E ? sc[i] + (bias != nullptr ? bias[e] : 0.f) : -INFINITY;
  }
  // group score: sum of top-2 (bias-corrected) or max; lanes_per_group lanes cooperate
  const int epg = E / n_group;            // experts per group
  const int lpg = max(1, epg / VPT);      // lanes per group (epg multiple of VPT or lpg == 1)
  float t1 = -INFINITY, t2 = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    if (sel[i] > t1) { t2 = t1; t1 = sel[i]; } else if (sel[i] > t2) { t2 = sel[i]; }
  }
  for (int o = 1; o < lpg; o <<= 1) {
    const float o1 = __shfl_xor_sync(0xffffffffu, t1, o), o2 = __shfl_xor_sync(0xffffffffu, t2, o);
    if (o1 > t1) { t2 = fmaxf(t1, o2); t1 = o1; } else { t2 = fmaxf(t2, o1); }
  }
  float gscore = (bias != nullptr) ? t1 + t2 : t1;
  const int my_group = (lane * VPT) / epg;
  // rank of my group among groups: count groups with a strictly better score (ties: lower index wins)
  int better = 0;
  for (int g = 0; g < n_group; ++g) {
    const float gs = __shfl_sync(0xffffffffu, gscore, (g * epg) / VPT);
    if (gs > gscore || (gs == gscore && g < my_group)) ++better;
  }
  const bool group_on = (lane * VPT < E) && better < topk_group;
#pragma unroll
  for (int i = 0; i < VPT; ++i) if (!group_on) sel[i] = -INFINITY;
  float wsum = 0.f, my_w = 0.f;
  int my_id = 0;
  for (int k = 0; k < K; ++k) {
    float best = -INFINITY, bw = 0.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (sel[i] > best) { best = sel[i]; bi = lane * VPT + i; bw = sc[i]; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const float ow = __shfl_xor_sync(0xffffffffu, bw, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; bw = ow; }
    }
    if (bi / VPT == lane) sel[bi % VPT] = -INFINITY;
    if (lane == k) { my_w = bw; my_id = bi; }
    wsum += bw;
  }
  if (lane < K) {
    const float w = renorm ? my_w / (wsum + 1e-20f) : my_w;
    w_out[static_cast<size_t>(warp) * K + lane] = w * scaling;
    id_out[static_cast<size_t>(warp) * K + lane] = my_id;
  }
}

// ---------------------------------------------------------------------------------------------
// align: slots -> expert-sorted, 128-row padded tiles
// meta layout (int32): [0] num_tiles, [1] num_rows_padded, [2..2+E) counts, [2+E .. 2+2E) unused,
//                      [2+2E .. 2+3E+1) padded offsets
// ---------------------------------------------------------------------------------------------
// n_valid (optional device scalar): only the first *n_valid slots are live (EP receive pool, comm/ep_a2a.cu)
struct RouteParams {
  const int32_t *ids, *expert_map, *n_valid;
  int n_slots, top_k, E, max_tiles;
  int32_t *meta, *tile_expert, *slot_pos;
  const __nv_bfloat16* x;
  int64_t ldx;
  __nv_bfloat16* xs;        // rows as they are ...
  __nv_fp8_e4m3* q;         // ... or quantised, scales [H / 128][rows]
  float* scales;
  int H, rows;
};

__device__ __forceinline__ int local_expert(const RouteParams& p, int slot, int valid) {
  if (slot >= valid) return -1;
  int e = p.ids[slot];
  if (p.expert_map != nullptr) e = p.expert_map[e];
  return e >= 0 && e < p.E ? e : -1;
}

// Row offsets of the experts, padded to whole tiles, from their counts (both in shared memory; s_off has E + 1 entries). All threads
// of the block.
__device__ __forceinline__ void expert_offsets(const int* s_cnt, int* s_off, int E, int* s_warp) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int base = 0;
  for (int e0 = 0; e0 < E; e0 += blockDim.x) {
    const int e = e0 + static_cast<int>(threadIdx.x);
    const int own = e < E ? (s_cnt[e] + kTileM - 1) / kTileM * kTileM : 0;
    int sum = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 31) s_warp[warp] = sum;
    __syncthreads();
    int before = base, all = 0;
    for (int w = 0; w < nw; ++w) {
      if (w < warp) before += s_warp[w];
      all += s_warp[w];
    }
    if (e < E) s_off[e] = before + sum - own;
    base += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) s_off[E] = base;
  __syncthreads();
}

__device__ __forceinline__ void write_meta(const RouteParams& p, const int* s_cnt, const int* s_off) {
  const int E = p.E, total = s_off[E];
  for (int e = threadIdx.x; e <= E; e += blockDim.x) {
    p.meta[2 + 2 * E + e] = s_off[e];
    if (e == E) {
      p.meta[0] = total / kTileM;
      p.meta[1] = total;
      continue;
    }
    p.meta[2 + e] = s_cnt[e];
    for (int t = s_off[e] / kTileM; t < s_off[e + 1] / kTileM; ++t) p.tile_expert[t] = e;
  }
  for (int t = total / kTileM + threadIdx.x; t < p.max_tiles; t += blockDim.x) p.tile_expert[t] = -1;
}

// one warp: a token's row to its place in the expert's segment
template <bool QUANT>
__device__ __forceinline__ void gather_row(const RouteParams& p, int slot, int pos) {
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* src = p.x + static_cast<size_t>(slot / p.top_k) * p.ldx;
  if constexpr (!QUANT) {
    __nv_bfloat16* dst = p.xs + static_cast<size_t>(pos) * p.H;
    for (int i = lane * 8; i < p.H; i += 256) *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(src + i);
  } else {                                               // sixteen lanes per group of 128, four pairs of groups on their way
    for (int i0 = 0; i0 < p.H; i0 += 1024) {
      uint4 raw[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int i = i0 + n * 256 + lane * 8;
        raw[n] = i < p.H ? *reinterpret_cast<const uint4*>(src + i) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int i = i0 + n * 256 + lane * 8;
        float scale;
        const uint2 o8 = fp8_quant_lane(raw[n], scale);
        if (i >= p.H) continue;
        *reinterpret_cast<uint2*>(p.q + static_cast<size_t>(pos) * p.H + i) = o8;
        if ((lane & 15) == 0) p.scales[static_cast<size_t>(i / 128) * p.rows + pos] = scale;
      }
    }
  }
}

// Up to kOneLaunch slots: every block counts the whole batch for itself (a few KB of ids), so that routing is one launch instead of
// four with a memset; a slot's row is its rank among the slots of its expert. Then a warp per slot copies.
// 48 tokens x 8 of 128 experts, 2048 wide: 8.1 us, where the four took 12.5 and their launches as much again; 4096 tokens x 8, 32 of 256
// experts here, quantised on the way (the two kernels below): 33 us, with copies in bf16 and a quantiser behind them 68.
static constexpr int kOneLaunch = 4096, kRouteThreads = 256;

template <bool QUANT>
__global__ void __launch_bounds__(kRouteThreads) moe_route_kernel(const RouteParams p) {
  extern __shared__ int32_t s_route[];                   // counts [E], offsets [E + 1], then the slots' experts as 16 bits
  __shared__ int s_warp[kRouteThreads / 32];
  int *s_cnt = s_route, *s_off = s_route + p.E;
  int16_t* s_e = reinterpret_cast<int16_t*>(s_off + p.E + 1);
  griddep_launch();
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  griddep_wait();
  const int valid = p.n_valid != nullptr ? min(p.n_slots, *p.n_valid) : p.n_slots;
  for (int i = threadIdx.x; i < p.n_slots; i += blockDim.x) {
    const int e = local_expert(p, i, valid);
    s_e[i] = static_cast<int16_t>(e);
    if (e >= 0) atomicAdd(&s_cnt[e], 1);
  }
  __syncthreads();
  expert_offsets(s_cnt, s_off, p.E, s_warp);
  if (blockIdx.x == 0) write_meta(p, s_cnt, s_off);
  const int lane = threadIdx.x & 31;
  for (int slot = blockIdx.x * (kRouteThreads / 32) + (threadIdx.x >> 5); slot < p.n_slots; slot += gridDim.x * (kRouteThreads / 32)) {
    const int e = s_e[slot];
    int pos = -1;
    if (e >= 0) {
      int rank = 0;
      for (int i = lane; i < slot; i += 32) rank += s_e[i] == e;
      pos = s_off[e] + __reduce_add_sync(0xffffffffu, rank);
      gather_row<QUANT>(p, slot, pos);
    }
    if (lane == 0) p.slot_pos[slot] = pos;
  }
}

// More slots: one block counts and ranks them, or, beyond kOneBlock, the CTAs of a cluster take a part each, and to a slot's rank in its
// part come the counts of the parts before. slot_pos holds a slot's rank until the next kernel adds the offset. What bounds it is the
// latency of the ids and, behind them, of the map. With the copies behind it (2048 wide, 32 of 256 experts here), one block / a cluster:
// 8192 slots 8.2 / 9.9 us, 16,384 10.2 / 11.0, 32,768 14.6 / 12.2, 131,072 59 / 39 (32 of 256), 181 / 147 (all of 128); a receive pool
// of 131,072 slots of which 4096 live 31.7 / 23.6, 30,000 71.6 / 57.4.
static constexpr int kOneBlock = 16384, kAlignParts = 8, kAlignThreads = 1024, kAlignAtOnce = 8;

template <bool ONE>
__global__ void __launch_bounds__(kAlignThreads) moe_align_kernel(const RouteParams p) {
  constexpr int kU = ONE ? 4 : kAlignAtOnce, kStep = kU * kAlignThreads;
  __shared__ int s_cnt[1024], s_sum[ONE ? 1 : 1024], s_base[ONE ? 1 : 1024], s_off[1025], s_warp[32];
  griddep_launch();
  for (int e = threadIdx.x; e < p.E; e += kAlignThreads) s_cnt[e] = 0;
  __syncthreads();
  griddep_wait();
  const int valid = p.n_valid != nullptr ? min(p.n_slots, *p.n_valid) : p.n_slots;
  const int part = ONE ? 0 : blockIdx.x, parts = ONE ? 1 : gridDim.x;
  const int lo = static_cast<int>(static_cast<int64_t>(valid) * part / parts);
  const int hi = static_cast<int>(static_cast<int64_t>(valid) * (part + 1) / parts);
  const int first = lo + static_cast<int>(threadIdx.x);
  auto experts_of = [&](int i0, int (&e)[kU]) {
#pragma unroll
    for (int u = 0; u < kU; ++u) e[u] = i0 + u * kAlignThreads < hi ? local_expert(p, i0 + u * kAlignThreads, valid) : -1;
  };
  auto count = [&](int i0, const int (&e)[kU]) {
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (i0 + u * kAlignThreads < hi) p.slot_pos[i0 + u * kAlignThreads] = e[u] >= 0 ? atomicAdd(&s_cnt[e[u]], 1) : -1;
  };
  for (int i0 = first; i0 < hi; i0 += kStep) {
    int e[kU];
    experts_of(i0, e);
    count(i0, e);
  }
  for (int i = valid + part * kAlignThreads + static_cast<int>(threadIdx.x); i < p.n_slots; i += parts * kAlignThreads) p.slot_pos[i] = -1;
  if constexpr (ONE) {
    __syncthreads();
    expert_offsets(s_cnt, s_off, p.E, s_warp);
    write_meta(p, s_cnt, s_off);
  } else {
    __syncwarp();
    cluster_sync();                                      // every part is counted
    for (int e = threadIdx.x; e < p.E; e += kAlignThreads) {
      int before = 0, all = 0;
      for (int i = 0; i < parts; ++i) {
        int c;
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(c) : "r"(cluster_addr(&s_cnt[e], i)) : "memory");
        if (i < part) before += c;
        all += c;
      }
      s_base[e] = before;
      s_sum[e] = all;
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // the others' counts have been read
    __syncthreads();
    if (part == 0) {
      expert_offsets(s_sum, s_off, p.E, s_warp);
      write_meta(p, s_sum, s_off);
    }
    for (int i0 = part > 0 ? first : hi; i0 < hi; i0 += kStep) {           // this thread's own slots
      int e[kU], r[kU];
      experts_of(i0, e);
#pragma unroll
      for (int u = 0; u < kU; ++u) r[u] = e[u] >= 0 ? p.slot_pos[i0 + u * kAlignThreads] : 0;
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (e[u] >= 0) p.slot_pos[i0 + u * kAlignThreads] = s_base[e[u]] + r[u];
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");    // ... and they this CTA's
  }
}

// one warp per slot
template <bool QUANT>
__global__ void __launch_bounds__(256) moe_gather_kernel(const RouteParams p) {
  griddep_launch();
  griddep_wait();
  const int slot = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (slot >= p.n_slots) return;
  const int rank = p.slot_pos[slot];
  if (rank < 0) return;
  int e = p.ids[slot];
  if (p.expert_map != nullptr) e = p.expert_map[e];
  const int pos = p.meta[2 + 2 * p.E + e] + rank;
  gather_row<QUANT>(p, slot, pos);
  __syncwarp();                                          // every lane has read the rank
  if (lane == 0) p.slot_pos[slot] = pos;
}

__global__ void moe_combine_kernel(const __nv_bfloat16* __restrict__ y, const int32_t* __restrict__ slot_pos,
                                   const float* __restrict__ w, __nv_bfloat16* __restrict__ out, int top_k, int H) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = 0; j < top_k; ++j) {
      const int pos = slot_pos[t * top_k + j];
      if (pos < 0) continue;  // expert lives on another rank
      const float wt = w[t * top_k + j];
      const uint4 v = *reinterpret_cast<const uint4*>(y + static_cast<size_t>(pos) * H + i);
      const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), c = unpack_bf16(v.z), d = unpack_bf16(v.w);
      acc[0] += wt * a.x; acc[1] += wt * a.y; acc[2] += wt * b.x; acc[3] += wt * b.y;
      acc[4] += wt * c.x; acc[5] += wt * c.y; acc[6] += wt * d.x; acc[7] += wt * d.y;
    }
    uint4 o;
    o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
    o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
    *reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * H + i) = o;
  }
}

}  // namespace b200

using namespace b200;

GLLM_EXPORT int gllm_moe_topk_softmax(const void* logits, int64_t ld, void* w_out, void* id_out, int T, int E, int K,
                                      int renorm, void* stream) {
  if (T <= 0) return 0;
  if (E > 512 || K > 32) { fprintf(stderr, "[gllm_b200] topk_softmax: E<=512, K<=32 only\n"); return 1; }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int blocks = (T * 32 + 255) / 256;
  auto L = reinterpret_cast<const __nv_bfloat16*>(logits);
  auto W = reinterpret_cast<float*>(w_out);
  auto I = reinterpret_cast<int32_t*>(id_out);
  const int vpt = (E + 31) / 32;
  if (vpt <= 1) topk_softmax_kernel<1><<<blocks, 256, 0, st>>>(L, ld, W, I, T, E, K, renorm);
  else if (vpt <= 2) topk_softmax_kernel<2><<<blocks, 256, 0, st>>>(L, ld, W, I, T, E, K, renorm);
  else if (vpt <= 4) topk_softmax_kernel<4><<<blocks, 256, 0, st>>>(L, ld, W, I, T, E, K, renorm);
  else if (vpt <= 8) topk_softmax_kernel<8><<<blocks, 256, 0, st>>>(L, ld, W, I, T, E, K, renorm);
  else topk_softmax_kernel<16><<<blocks, 256, 0, st>>>(L, ld, W, I, T, E, K, renorm);
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

GLLM_EXPORT int gllm_moe_grouped_topk(const void* logits, int64_t ld, const void* bias, void* w_out, void* id_out,
                                      int T, int E, int K, int n_group, int topk_group, int renorm, int sigmoid,
                                      float scaling, void* stream) {
  if (T <= 0) return 0;
  const int vpt = (E + 31) / 32;
  const int epg = E / n_group;
  if (E > 512 || K > 32 || E % n_group != 0 || (epg % vpt != 0 && epg > vpt) || (epg < vpt && vpt % epg != 0) ||
      epg < vpt) {
    fprintf(stderr, "[gllm_b200] grouped_topk: unsupported E=%d groups=%d\n", E, n_group);
    return 1;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int blocks = (T * 32 + 255) / 256;
  auto L = reinterpret_cast<const __nv_bfloat16*>(logits);
  auto B = reinterpret_cast<const float*>(bias);
  auto W = reinterpret_cast<float*>(w_out);
  auto I = reinterpret_cast<int32_t*>(id_out);
#define GT(V) grouped_topk_kernel<V><<<blocks, 256, 0, st>>>(L, ld, B, W, I, T, E, K, n_group, topk_group, renorm, sigmoid, scaling)
  if (vpt <= 1) GT(1);
  else if (vpt <= 2) GT(2);
  else if (vpt <= 4) GT(4);
  else if (vpt <= 8) GT(8);
  else GT(16);
#undef GT
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

static int route(const RouteParams& p, cudaStream_t st) {
  if (p.n_slots <= 0) return 0;
  if (p.E < 0 || p.E > 1024) {                           // none: zero counts, no tile, no slot placed
    fprintf(stderr, "[gllm_b200] moe_align_gather: %d experts (0 to 1024)\n", p.E);
    return 1;
  }
  const bool quant = p.q != nullptr;
  if (p.n_slots <= kOneLaunch) {
    const size_t smem = (2 * p.E + 1) * 4 + p.n_slots * 2;
    const dim3 grid((p.n_slots + kRouteThreads / 32 - 1) / (kRouteThreads / 32));
    CUDA_CHECK_RET(launch_pdl(quant ? moe_route_kernel<true> : moe_route_kernel<false>, grid, dim3(kRouteThreads), smem, st, p));
    return 0;
  }
  const int parts = p.n_slots <= kAlignParts * kOneBlock / 2 ? (p.n_slots + kOneBlock / 2 - 1) / (kOneBlock / 2) : kAlignParts;
  CUDA_CHECK_RET(p.n_slots <= kOneBlock
                     ? launch_pdl(moe_align_kernel<true>, dim3(1), dim3(kAlignThreads), 0, st, p)
                     : launch_pdl_cluster(moe_align_kernel<false>, dim3(parts), parts, dim3(kAlignThreads), 0, st, p));
  CUDA_CHECK_RET(launch_pdl(quant ? moe_gather_kernel<true> : moe_gather_kernel<false>, dim3((p.n_slots + 7) / 8), dim3(256), 0, st, p));
  return 0;
}

static RouteParams route_params(const void* ids, const void* expert_map, int T, int top_k, int E, void* meta, void* tile_expert,
                                int max_tiles, void* slot_pos, const void* x, int64_t ldx, int H, const void* n_valid) {
  RouteParams p = {};
  p.ids = reinterpret_cast<const int32_t*>(ids);
  p.expert_map = reinterpret_cast<const int32_t*>(expert_map);
  p.n_valid = reinterpret_cast<const int32_t*>(n_valid);
  p.n_slots = T * top_k; p.top_k = top_k; p.E = E; p.max_tiles = max_tiles;
  p.meta = reinterpret_cast<int32_t*>(meta);
  p.tile_expert = reinterpret_cast<int32_t*>(tile_expert);
  p.slot_pos = reinterpret_cast<int32_t*>(slot_pos);
  p.x = reinterpret_cast<const __nv_bfloat16*>(x);
  p.ldx = ldx; p.H = H;
  return p;
}

// meta: int32[2 + 3*E_local + 1] (written here); tile_expert: int32[max_tiles]; slot_pos: int32[n_slots];
// xs: bf16 [max_tiles*128, H] (caller zero-fills padding rows once; stale finite rows are harmless).
GLLM_EXPORT int gllm_moe_align_gather(const void* ids, const void* expert_map, int T, int top_k, int E_local,
                                      void* meta, void* tile_expert, int max_tiles, void* slot_pos, const void* x,
                                      int64_t ldx, void* xs, int H, const void* n_valid, void* stream) {
  RouteParams p = route_params(ids, expert_map, T, top_k, E_local, meta, tile_expert, max_tiles, slot_pos, x, ldx, H, n_valid);
  p.xs = reinterpret_cast<__nv_bfloat16*>(xs);
  return route(p, reinterpret_cast<cudaStream_t>(stream));
}

// The same with the rows quantised on their way, as gllm_fp8_quant_group quantises them: q e4m3 [max_tiles*128, H], scales fp32
// [H/128, max_tiles*128]. Rows that no token goes to are not written.
GLLM_EXPORT int gllm_moe_align_gather_fp8(const void* ids, const void* expert_map, int T, int top_k, int E_local, void* meta,
                                          void* tile_expert, int max_tiles, void* slot_pos, const void* x, int64_t ldx, void* q,
                                          void* scales, int H, void* stream) {
  if (H % 128 != 0 || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0) {
    fprintf(stderr, "[gllm_b200] moe_align_gather_fp8: H %% 128 and rows on 16-byte boundaries required\n");
    return 1;
  }
  RouteParams p = route_params(ids, expert_map, T, top_k, E_local, meta, tile_expert, max_tiles, slot_pos, x, ldx, H, nullptr);
  p.q = reinterpret_cast<__nv_fp8_e4m3*>(q);
  p.scales = reinterpret_cast<float*>(scales);
  p.rows = max_tiles * kTileM;
  return route(p, reinterpret_cast<cudaStream_t>(stream));
}

GLLM_EXPORT int gllm_moe_combine(const void* y, const void* slot_pos, const void* w, void* out, int T, int top_k,
                                 int H, void* stream) {
  if (T <= 0) return 0;
  CUDA_CHECK_RET(launch_pdl(moe_combine_kernel, dim3(T), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                            reinterpret_cast<const __nv_bfloat16*>(y), reinterpret_cast<const int32_t*>(slot_pos),
                            reinterpret_cast<const float*>(w), reinterpret_cast<__nv_bfloat16*>(out), top_k, H));
  return 0;
}
