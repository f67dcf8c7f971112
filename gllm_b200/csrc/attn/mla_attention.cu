// Multi-head latent attention (DeepSeek V2 / V3 / R1, Kimi) over the paged LATENT cache, absorbed form:
//
//   q_full[t, h, :] = [ q_nope[t, h] · W_UK[h]  (512) | rope(q_pe[t, h]) (64) ]          (built by the caller)
//   s[t, h, j]      = q_full[t, h] · latent[j]            latent[j] = [ c_kv[j] (512) | rope(k_pe[j]) (64) ]
//   out_lat[t, h]   = softmax_j(s * scale) · c_kv[j]      (512)          -> caller applies W_UV[h]
//
// i.e. multi-query attention with one shared 576-wide key whose first 512 columns are also the value, so a KV
// tile is fetched ONCE (TMA page boxes, 128-byte swizzle, mbarrier ring, producer warp) and serves both GEMMs.
// This replaces the reference's Triton split-KV MQA decode kernels and its gather/up-project/FlashAttention
// prefill loop (gllm/layers/attention.py:129-391, gllm/layers/ops/triton_decode_attention.py).
//
// Work = the 64-key tiles of every (token, 16 heads), laid end to end and cut into equal shares, one per SM: a long sequence
// among short ones spreads over several CTAs and none idles, whatever the lengths. A (token, heads) inside one share is written
// as it is; the parts of one that crosses shares go to two slots per CTA and mla_merge_kernel adds them up. The lengths are read
// on the device (each CTA scans them), so a captured graph keeps the balance. The producer runs on from one (token, heads) into
// the next, two tiles ahead.
// Eight math warps: for S = Q K^T each takes 16 keys and half of the 576 columns, with its part of Q in registers (the two
// halves are added through shared memory); then the row maxima and the bf16 probabilities are exchanged and each warp takes 64
// value columns of O += P V. Warp 0 issues the copies itself: a ninth warp would hold the
// others to 168 registers, and the spills alone cost half the speed. Bound by the latent bytes at long contexts: 148 sequences of
// 4096 keys, 16 heads, 115 us (6.1 TB/s). 128 ragged sequences of up to 4096 keys, 16 heads: 96 -> 49 us, 32 x 1500 keys with 128
// heads 147 -> 80; before: four warps, Q in shared memory, one CTA per (token, heads, split).
// Every token is its own "sequence" with kv_len = position + 1, so the same kernel serves decode and short prompt portions.
//
// Latent cache layout: [num_pages, 1, 9, page_size, 64] bf16 (the generic paged layout with Hkv = 1, D = 576).
#include "attn_common.cuh"
#include "../common/bounded.cuh"

namespace b200 {

static constexpr int kLat = 576;        // kv_lora_rank (512) + qk_rope_head_dim (64)
static constexpr int kLatV = 512;       // value width = kv_lora_rank
static constexpr int kMlaStages = 3;
static constexpr int kMlaWarps = 8;
static constexpr int kMlaThreads = kMlaWarps * 32;
static constexpr int kMlaMinTiles = 2;  // a share is at least this long: below it the merge costs more than the split gains
static constexpr int kMlaTileBytes = kTileN * kLat * 2;                 // 73,728
static constexpr int kPStride = kTileN * 2 + 16;                        // padded row pitch of P in smem (bytes)
static constexpr int kMlaSmem = 1024 + kMlaStages * kMlaTileBytes + kMlaWarps * 32 * 16 + 16 * kPStride + 2 * 16 * kMlaWarps * 4 + 128;

struct MlaParams {
  const __nv_bfloat16* q;     // [tokens, H, 576]
  __nv_bfloat16* out;         // [tokens, H, 512]
  float* part_o;              // [2 * CTAs, 16, 512] parts of (token, heads) that cross shares
  float* part_lse;            // [2 * CTAs, 16]
  int4* meta;                 // [CTAs] (token, head group, last CTA, slot) of the one that starts here and goes on; token -1: none
  const int32_t* block_table; // [seqs, max_blocks]
  const int32_t* tok_seq;     // [tokens] sequence (block-table row) of every token; null => token index
  const int32_t* positions;   // [tokens] absolute position of the token (kv_len = position + 1)
  int tokens, max_blocks, H, page_size;
  float scale_log2;
  int window;                 // a token at position i sees keys j with i - j < window (0: the whole past)
  WaitConfig waits;
  const float* sink;          // [H] one more logit per head in the denominator, without a value (null: none)
};

struct MlaSpan {              // visible keys of one token: [win_lo, kv_len), tiles [tile_lo, tile_lo + n), n >= 1
  int kv_len, win_lo, tile_lo, n;
  __device__ __forceinline__ MlaSpan(const MlaParams& p, int tok) {
    kv_len = p.positions[tok] + 1;
    win_lo = p.window > 0 ? max(0, kv_len - p.window) : 0;
    tile_lo = win_lo / kTileN;
    n = max((kv_len + kTileN - 1) / kTileN - tile_lo, 1);
  }
};

__global__ void __launch_bounds__(kMlaThreads, 1)
mla_attn_kernel(const __grid_constant__ CUtensorMap tmap, const MlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float4* xch = reinterpret_cast<float4*>(smem + kMlaStages * kMlaTileBytes);       // [8 warps][32 lanes] half sums of S
  uint8_t* p_smem = reinterpret_cast<uint8_t*>(xch + kMlaWarps * 32);               // [16 rows][64 keys] bf16
  float* red_max = reinterpret_cast<float*>(p_smem + 16 * kPStride);                // [16 rows][8 warps]
  float* red_sum = red_max + 16 * kMlaWarps;                                        // [16 rows][8 warps]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(red_sum + 16 * kMlaWarps);
  uint32_t* dead = reinterpret_cast<uint32_t*>(full_bar + kMlaStages);
  int* first = reinterpret_cast<int*>(dead + 1);                                    // token, head group, tile of the share's start
  int* warp_sum = reinterpret_cast<int*>(xch);                                      // before the first tile only

  griddep_launch();
  griddep_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hg = (p.H + 15) / 16;
  const WaitGuard guard{dead, p.waits};

  // ---------------- this CTA's share [t0, t1) of all tiles ----------------
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMlaStages; ++i) mbar_init(&full_bar[i], 1);
    *dead = 0;
    fence_mbar_init();
  }
  int tok, grp, off, t0, t1, share, last_cta = -1;
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  if (p.tokens <= 32) {
    // A lane per token, every warp for itself. Where each (token, heads) can have whole shares, none begins inside another's: a CTA
    // that goes on into the next one waits for its queries once more (4 tokens of 300 keys, 16 heads: 14.6 us against 11.4).
    const int own = lane < p.tokens ? MlaSpan(p, lane).n : 0;
    auto upto = [&](int v) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      return v;
    };
    const int to = upto(own), total = __shfl_sync(0xffffffffu, to, 31) * hg;
    share = max((total + grid - 1) / grid, kMlaMinTiles);
    const int parts = (own + share - 1) / share, pto = upto(parts);
    const bool aligned = __shfl_sync(0xffffffffu, pto, 31) * hg <= grid;
    const int at = aligned ? cta : cta * share, from = (aligned ? pto - parts : to - own) * hg, width = aligned ? parts : own;
    const uint32_t mine = __ballot_sync(0xffffffffu, at >= from && at < from + width * hg);
    if (mine == 0) {                                                   // idle, and so all of the block
      if (threadIdx.x == 0) p.meta[cta] = make_int4(-1, 0, 0, 0);
      return;
    }
    tok = __ffs(mine) - 1;
    const int in = at - __shfl_sync(0xffffffffu, from, tok), w = __shfl_sync(0xffffffffu, width, tok),
              n = __shfl_sync(0xffffffffu, own, tok);
    grp = in / w;
    if (aligned) {
      off = in % w * share;
      t0 = 0;
      t1 = min(share, n - off);
      last_cta = cta + w - 1 - in % w;
    } else {
      off = in % w;
      t0 = at;
      t1 = min(t0 + share, total);
    }
    __syncthreads();                                                   // the barriers are initialised
  } else {
    const int per = (p.tokens + kMlaThreads - 1) / kMlaThreads;        // tokens scanned by one thread
    const int s0 = min(static_cast<int>(threadIdx.x) * per, p.tokens), s1 = min(s0 + per, p.tokens);
    int own = 0;
    for (int i = s0; i < s1; ++i) own += MlaSpan(p, i).n;
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (lane == 31) warp_sum[warp] = upto;
    __syncthreads();
    int total = 0, before = upto - own;
#pragma unroll
    for (int w = 0; w < kMlaWarps; ++w) {
      if (w < warp) before += warp_sum[w];
      total += warp_sum[w];
    }
    total *= hg;
    share = max((total + grid - 1) / grid, kMlaMinTiles);
    t0 = min(cta * share, total);
    t1 = min(t0 + share, total);
    if (t0 >= t1) {
      if (threadIdx.x == 0) p.meta[cta] = make_int4(-1, 0, 0, 0);
      return;
    }
    if (t0 >= before * hg && t0 < (before + own) * hg) {               // one thread: the token that the share starts in
      int at = s0, acc = before, n = MlaSpan(p, s0).n;
      while (t0 >= (acc + n) * hg) {
        acc += n;
        n = MlaSpan(p, ++at).n;
      }
      const int in = t0 - acc * hg;
      first[0] = at; first[1] = in / n; first[2] = in % n;
    }
    __syncthreads();
    tok = first[0];
    grp = first[1];
    off = first[2];
  }

  // ---------------- copies, issued by warp 0: one TMA box per page, K == V, two tiles ahead of the products ----------------
  const int page_bytes = p.page_size * kLat * 2, slab = p.page_size * 128;
  const int pages_per_tile = kTileN / p.page_size;                     // at most 8
  struct { int tok, grp, at, end, cur; uint32_t it; int page; } ld = {tok, grp, off, 0, t0, 0u, 0};
  auto fetch_page = [&] {                              // this lane's page of the next tile; the entry is used one tile later
    if (ld.cur >= t1) return;
    const MlaSpan span(p, ld.tok);
    const int32_t* bt = p.block_table + static_cast<size_t>(p.tok_seq != nullptr ? p.tok_seq[ld.tok] : ld.tok) * p.max_blocks;
    const int last_page = max(span.kv_len - 1, 0) / p.page_size;       // masked columns: finite data
    if (lane < pages_per_tile) ld.page = bt[min((span.tile_lo + ld.at) * pages_per_tile + lane, last_page)];
    ld.end = span.n;
  };
  auto load_tile = [&] {
    if (ld.cur >= t1) return;
    if (__any_sync(0xffffffffu, guard.gave_up())) {    // nothing more is issued: ld.it counts what was
      ld.cur = t1;
      return;
    }
    const int s = ld.it % kMlaStages;
    if (lane == 0) mbar_expect_tx(&full_bar[s], kMlaTileBytes);
    __syncwarp();
    if (lane < pages_per_tile)
      tma_load_3d(smem + s * kMlaTileBytes + lane * page_bytes, &tmap, &full_bar[s], 0, 0, ld.page * (kLat / 64));
    ++ld.it;
    ++ld.cur;
    if (++ld.at == ld.end) {
      ld.at = 0;
      if (++ld.grp == hg) { ld.grp = 0; ++ld.tok; }
    }
    fetch_page();
  };
  if (warp == 0) {
    fetch_page();
    for (int i = 0; i < kMlaStages - 1; ++i) load_tile();
    guard.first(&full_bar[1]);
  }

  const int g = lane >> 2, t = lane & 3;
  const int kg = warp & 3, kh = warp >> 2;           // S: keys [16 kg, +16) of a tile, columns [288 kh, +288)
  const uint32_t p_base = smem_u32(p_smem);
  uint32_t k_row[2], k_xor[2];                        // S: this lane's row of the two 8-key matrices, and its swizzle
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const int key = kg * 16 + nt * 8 + (lane & 7), pj = key / p.page_size, r = key - pj * p.page_size;
    k_row[nt] = pj * page_bytes + r * 128;
    k_xor[nt] = ((lane >> 3) ^ (r & 7)) << 4;
  }
  uint32_t v_row[kTileN / 16], v_xor[kTileN / 16];    // P V: this lane's row of each 16-key step, slab = warp
#pragma unroll
  for (int kk = 0; kk < kTileN / 16; ++kk) {
    const int key = kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), pj = key / p.page_size, r = key - pj * p.page_size;
    v_row[kk] = pj * page_bytes + warp * slab + r * 128;
    v_xor[kk] = ((lane >> 4) ^ (r & 7)) << 4;
  }
  int4 meta = make_int4(-1, 0, 0, 0);
  uint32_t it = 0;
  for (int cur = t0; cur < t1;) {
    const MlaSpan span(p, tok);
    const int len = min(span.n - off, t1 - cur);
    const bool whole = off == 0 && len == span.n;
    const int slot = 2 * blockIdx.x + (cur == t0 ? 0 : 1);
    if (off == 0 && !whole) meta = make_int4(tok, grp, last_cta >= 0 ? last_cta : (cur + span.n - 1) / share, slot);
    const int hbase = grp * 16, n_rows = min(16, p.H - hbase);
    uint32_t qa[kLat / 32][4];                        // Q fragments of this warp's columns; rows beyond the head count are zero
    {
      const __nv_bfloat16* qb = p.q + (static_cast<size_t>(tok) * p.H + hbase) * kLat + kh * (kLat / 2) + 2 * t;
#pragma unroll
      for (int ks = 0; ks < kLat / 32; ++ks)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = g + (e & 1) * 8;
          qa[ks][e] = row < n_rows ? *reinterpret_cast<const uint32_t*>(qb + row * kLat + ks * 16 + (e >> 1) * 8) : 0u;
        }
    }
    float o[8][4];  // this warp's 64 value columns: 8 n-tiles of 8
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY};
    float l_run[2] = {0.f, 0.f};  // partial row sums over THIS warp's keys (all warps share the same m_run)

    for (int i = 0; i < len; ++i, ++it) {
      const int s = it % kMlaStages;
      guard.wait<true>(&full_bar[s], (it / kMlaStages) & 1);   // polled: a wait per tile (256 tokens, 128 heads: 443 us, suspended 451)
      const uint32_t sk = smem_u32(smem + s * kMlaTileBytes);

      // S = Q K^T for 16 rows x 16 keys, k = this warp's half of 576; two chains per 8 keys
      float sc[2][2][4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int c = 0; c < 2; ++c) sc[nt][c][0] = sc[nt][c][1] = sc[nt][c][2] = sc[nt][c][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < kLat / 32; ks += 2) {
        const int u = ks / 2 + kh * (kLat / 64);                        // 32-column chunk: half (u & 1) of slab u >> 1
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4(sk + k_row[nt] + (u >> 1) * slab + (k_xor[nt] ^ ((u & 1) << 6)), b0, b1, b2, b3);
          mma_bf16_16816(sc[nt][0], qa[ks], b0, b1);
          mma_bf16_16816(sc[nt][1], qa[ks + 1], b2, b3);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[nt][0][e] += sc[nt][1][e];
      // the pair of warps with the same keys: each finishes 8 of them
      float (&mine)[4] = sc[0][0];
      xch[warp * 32 + lane] = kh == 0 ? make_float4(sc[1][0][0], sc[1][0][1], sc[1][0][2], sc[1][0][3])
                                      : make_float4(sc[0][0][0], sc[0][0][1], sc[0][0][2], sc[0][0][3]);
      if (kh == 1) {
#pragma unroll
        for (int e = 0; e < 4; ++e) mine[e] = sc[1][0][e];
      }
      asm volatile("bar.sync %0, 64;" ::"r"(2 + kg) : "memory");
      {
        const float4 x = xch[(warp ^ 4) * 32 + lane];
        mine[0] += x.x; mine[1] += x.y; mine[2] += x.z; mine[3] += x.w;
      }
      // mask, local row max over this warp's 8 keys
      const int key0 = (span.tile_lo + off + i) * kTileN + kg * 16 + kh * 8 + 2 * t;
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = key0 + (e & 1);
        float v = mine[e] * p.scale_log2;
        if (col >= span.kv_len || col < span.win_lo) v = -INFINITY;
        mine[e] = v;
        mx[e >> 1] = fmaxf(mx[e >> 1], v);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      }
      if (t == 0) {
        red_max[g * kMlaWarps + warp] = mx[0];
        red_max[(g + 8) * kMlaWarps + warp] = mx[1];
      }
      __syncthreads();
      if (warp == 0) load_tile();          // into the stage that every warp left before this barrier
      float alpha[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float4* rm = reinterpret_cast<const float4*>(red_max + (g + r * 8) * kMlaWarps);
        const float4 x = rm[0], y = rm[1];
        const float m_tile = fmaxf(fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)), fmaxf(fmaxf(y.x, y.y), fmaxf(y.z, y.w)));
        const float m_new = fmaxf(m_run[r], m_tile);
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        alpha[r] = exp2f(m_run[r] - m_use);
        m_run[r] = m_new;
        const float p0 = exp2f(mine[2 * r] - m_use), p1 = exp2f(mine[2 * r + 1] - m_use);
        l_run[r] = l_run[r] * alpha[r] + p0 + p1;
        *reinterpret_cast<uint32_t*>(p_smem + (g + r * 8) * kPStride + (kg * 16 + kh * 8 + 2 * t) * 2) = pack_bf16(p0, p1);
      }
#pragma unroll
      for (int nd = 0; nd < 8; ++nd) {
        o[nd][0] *= alpha[0]; o[nd][1] *= alpha[0];
        o[nd][2] *= alpha[1]; o[nd][3] *= alpha[1];
      }
      __syncthreads();
      // O[:, 64 * warp + ...] += P (16 x 64) * V (64 keys x 64 columns of the same tile)
#pragma unroll
      for (int kk = 0; kk < kTileN / 16; ++kk) {
        uint32_t pa[4];
        ldsm_x4(p_base + (lane & 15) * kPStride + (kk * 16 + (lane >> 4) * 8) * 2, pa[0], pa[1], pa[2], pa[3]);
#pragma unroll
        for (int nd = 0; nd < 8; nd += 2) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(sk + v_row[kk] + (v_xor[kk] ^ (nd << 4)), b0, b1, b2, b3);
          mma_bf16_16816(o[nd], pa, b0, b1);
          mma_bf16_16816(o[nd + 1], pa, b2, b3);
        }
      }
    }

    // total row sums across the warps, write this warp's value columns
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    }
    if (t == 0) {
      red_sum[g * kMlaWarps + warp] = l_run[0];
      red_sum[(g + 8) * kMlaWarps + warp] = l_run[1];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = g + r * 8;
      if (row >= n_rows) continue;
      const float4* rs = reinterpret_cast<const float4*>(red_sum + row * kMlaWarps);
      const float4 x = rs[0], y = rs[1];
      float l_all = ((x.x + x.y) + (x.z + x.w)) + ((y.x + y.y) + (y.z + y.w));
      // the sink joins the part with the first tile (which always has a key): its weight then carries it through the merge
      if (p.sink != nullptr && off == 0 && m_run[r] > -INFINITY)
        l_all += exp2f(p.sink[hbase + row] * 1.4426950408889634f - m_run[r]);
      const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
      const size_t th = static_cast<size_t>(tok) * p.H + hbase + row;
#pragma unroll
      for (int nd = 0; nd < 8; ++nd) {
        const int c = warp * 64 + nd * 8 + 2 * t;
        const float a = o[nd][2 * r] * inv, b = o[nd][2 * r + 1] * inv;
        if (whole) {
          *reinterpret_cast<uint32_t*>(p.out + th * kLatV + c) = pack_bf16(a, b);
        } else {
          *reinterpret_cast<float2*>(p.part_o + (static_cast<size_t>(slot) * 16 + row) * kLatV + c) = make_float2(a, b);
        }
      }
      if (!whole && warp == 0 && t == 0) p.part_lse[slot * 16 + row] = (l_all > 0.f) ? (m_run[r] + log2f(l_all)) : -INFINITY;
    }
    cur += len;
    off = 0;
    if (++grp == hg) { grp = 0; ++tok; }
  }
  if (threadIdx.x == 0) p.meta[blockIdx.x] = meta;
  if (warp == 0 && guard.gave_up()) {                                  // copies in flight end before the CTA does
    for (uint32_t k = ld.it < kMlaStages ? 0u : ld.it - kMlaStages; k < ld.it; ++k)
      guard.land(&full_bar[k % kMlaStages], (k / kMlaStages) & 1);
  }
}

// Adds up the parts of the (token, heads) that starts in share blockIdx.x and goes on into later ones: its first part lies in the
// slot that the share names, the others in the first slots of the shares behind. Four rows per block, four columns per thread.
__global__ void __launch_bounds__(512) mla_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse,
                                                        const int4* __restrict__ metas, __nv_bfloat16* __restrict__ out, int H) {
  griddep_launch();
  griddep_wait();
  const int4 meta = metas[blockIdx.x];                  // token, head group, last CTA, slot of the first part
  if (meta.x < 0) return;
  const int row = blockIdx.y * 4 + (threadIdx.x >> 7), head = meta.y * 16 + row, c = (threadIdx.x & 127) * 4;
  if (head >= H) return;
  auto slot_of = [&](int cta) { return (cta == static_cast<int>(blockIdx.x) ? meta.w : 2 * cta) * 16 + row; };
  const int lane = threadIdx.x & 31;
  float m = -INFINITY;
  for (int b = blockIdx.x + lane; b <= meta.z; b += 32) m = fmaxf(m, part_lse[slot_of(b)]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  float den = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int b0 = blockIdx.x; b0 <= meta.z; b0 += 32) {
    const int n = min(32, meta.z - b0 + 1);
    const float l = lane < n ? part_lse[slot_of(b0 + lane)] : -INFINITY;
    const float wl = l == -INFINITY ? 0.f : exp2f(l - m);
#pragma unroll 8
    for (int j = 0; j < n; ++j) {
      const float w = __shfl_sync(0xffffffffu, wl, j);
      const float4 v = *reinterpret_cast<const float4*>(part_o + static_cast<size_t>(slot_of(b0 + j)) * kLatV + c);
      den += w;
      acc.x += w * v.x; acc.y += w * v.y; acc.z += w * v.z; acc.w += w * v.w;
    }
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  *reinterpret_cast<uint2*>(out + (static_cast<size_t>(meta.x) * H + head) * kLatV + c) =
      make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
}

// Per token: interleaved-pair RoPE on the rope dims of every query head (written to q_out: the last 64 columns of the
// absorbed queries, or q_pe itself) and of the shared key, then the latent row [c_kv (512) | rope(k_pe) (64)] goes into its paged-cache slot.
// (reference: rotary_embedding + concat_and_cache_mla, gllm/layers/attention.py:443-451)
__global__ void mla_rope_cache_kernel(const __nv_bfloat16* q_pe, int64_t q_ts, int64_t q_hs, int H,
                                      __nv_bfloat16* q_out, int64_t o_ts, int64_t o_hs, const __nv_bfloat16* __restrict__ k_pe,
                                      int64_t k_ts, const __nv_bfloat16* __restrict__ kv_c, int64_t c_ts,
                                      const float* __restrict__ cos_sin, const int32_t* __restrict__ positions,
                                      const int32_t* __restrict__ slots, __nv_bfloat16* __restrict__ cache,
                                      int page_size) {
  griddep_launch();
  griddep_wait();
  const int tok = blockIdx.x;
  const int pos = positions[tok];
  const float* cs = cos_sin + static_cast<size_t>(pos) * 64;  // [cos (32) | sin (32)]
  for (int i = threadIdx.x; i < H * 32; i += blockDim.x) {
    const int h = i >> 5, pr = i & 31;
    const uint32_t raw = *reinterpret_cast<const uint32_t*>(q_pe + tok * q_ts + h * q_hs + 2 * pr);
    const float2 x = unpack_bf16(raw);
    const float c = cs[pr], sn = cs[32 + pr];
    *reinterpret_cast<uint32_t*>(q_out + tok * o_ts + h * o_hs + 2 * pr) =
        pack_bf16(x.x * c - x.y * sn, x.y * c + x.x * sn);
  }
  const int slot = slots != nullptr ? slots[tok] : -1;
  if (slot < 0) return;
  const int page = slot / page_size, off = slot - page * page_size;
  __nv_bfloat16* dst = cache + (static_cast<size_t>(page) * (kLat / 64) * page_size + off) * 64;
  const size_t slab_stride = static_cast<size_t>(page_size) * 64;
  for (int i = threadIdx.x; i < kLatV / 8; i += blockDim.x) {  // 64 chunks of 8 bf16
    const uint4 v = *reinterpret_cast<const uint4*>(kv_c + tok * c_ts + i * 8);
    *reinterpret_cast<uint4*>(dst + (i >> 3) * slab_stride + (i & 7) * 8) = v;
  }
  if (threadIdx.x < 32) {
    const int pr = threadIdx.x;
    const float2 x = unpack_bf16(*reinterpret_cast<const uint32_t*>(k_pe + tok * k_ts + 2 * pr));
    const float c = cs[pr], sn = cs[32 + pr];
    *reinterpret_cast<uint32_t*>(dst + 8 * slab_stride + 2 * pr) = pack_bf16(x.x * c - x.y * sn, x.y * c + x.x * sn);
  }
}

// First row of every sequence in the gathered latents (each takes whole 64-row tiles): rows[s] = sum of the lengths before it,
// rounded up to 64. Sequences of fewer than min_len new tokens, or of fewer than min_work / 2 (query, key) pairs, take none.
__global__ void mla_rows_kernel(const int32_t* __restrict__ seq_lens, const int32_t* __restrict__ q_start, int min_len, int min_work,
                                int nseq, int32_t* __restrict__ rows) {
  __shared__ int32_t part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (int s0 = 0; s0 <= nseq; s0 += blockDim.x) {
    const int s = s0 + threadIdx.x;
    const int len = s < nseq ? seq_lens[s] : 0, q = s < nseq ? q_start[s + 1] - q_start[s] : 0;
    const bool expand = s < nseq && q >= min_len && static_cast<int64_t>(q) * (2 * static_cast<int64_t>(len) - q) >= min_work;
    const int n = expand ? (len + 63) / 64 * 64 : 0;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    if (lane == 31) part[warp] = sum;
    __syncthreads();
    int before = base, all = base;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
      if (w < warp) before += part[w];
      all += part[w];
    }
    if (s <= nseq) rows[s] = before + sum - n;
    base = all;
    __syncthreads();
  }
}

// Latent rows of whole sequences out of their pages: lat [rows, 512] and the rotated key part pe [rows, 64], zeros behind a
// sequence's end. One warp per row, 16-byte accesses; memory-bound.
__global__ void __launch_bounds__(256) mla_gather_kernel(const __nv_bfloat16* __restrict__ cache,
                                                         const int32_t* __restrict__ block_table, int max_blocks,
                                                         const int32_t* __restrict__ seq_lens,
                                                         const int32_t* __restrict__ rows, int nseq, int total, int page_size,
                                                         __nv_bfloat16* __restrict__ lat, __nv_bfloat16* __restrict__ pe) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= total) return;
  int lo = 0, hi = nseq - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (rows[mid] <= r) lo = mid; else hi = mid - 1;
  }
  const int i = r - rows[lo];
  const bool ok = i < seq_lens[lo];
  const int page = ok ? block_table[static_cast<size_t>(lo) * max_blocks + i / page_size] : 0;
  const __nv_bfloat16* src = cache + (static_cast<size_t>(page) * (kLat / 64) * page_size + i % page_size) * 64;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int c = k * 32 + lane;                         // 16-byte chunk: 64 of the latent, 8 of the rotated part
    if (c < kLat / 8) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (ok) v = *reinterpret_cast<const uint4*>(src + static_cast<size_t>(c >> 3) * page_size * 64 + (c & 7) * 8);
      __nv_bfloat16* dst = c < kLatV / 8 ? lat + static_cast<size_t>(r) * kLatV + c * 8
                                         : pe + static_cast<size_t>(r) * 64 + (c - kLatV / 8) * 8;
      *reinterpret_cast<uint4*>(dst) = v;
    }
  }
}

}  // namespace b200

using namespace b200;

// q [tokens, H, 576] bf16 contiguous -> out [tokens, H, 512]; cache = latent pages [num_pages, 1, 9, page, 64].
// Runs on `ctas` CTAs; part_o [2 * ctas, 16, 512] fp32, part_lse [2 * ctas, 16] fp32 and meta [ctas] int4 are scratch.
// window (0: none) and sink (null: none): see MlaParams.
GLLM_EXPORT int gllm_mla_attention(const void* q, void* out, const void* cache, int64_t num_pages,
                                   const void* block_table, const void* tok_seq, const void* positions, void* part_o,
                                   void* part_lse, void* meta, int tokens, int max_blocks, int H, int page_size, int ctas,
                                   float scale, int window, const void* sink, void* stream) {
  if (tokens <= 0) return 0;
  if (page_size < 8 || kTileN % page_size != 0) {
    fprintf(stderr, "[gllm_b200] mla_attention: unsupported page_size=%d\n", page_size);
    return 1;
  }
  CUtensorMap tm;
  if (get_kv_tmap(cache, num_pages, 1, kLat, page_size, &tm)) return 1;
  MlaParams p;
  p.q = reinterpret_cast<const __nv_bfloat16*>(q);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.part_o = reinterpret_cast<float*>(part_o);
  p.part_lse = reinterpret_cast<float*>(part_lse);
  p.block_table = reinterpret_cast<const int32_t*>(block_table);
  p.tok_seq = reinterpret_cast<const int32_t*>(tok_seq);
  p.positions = reinterpret_cast<const int32_t*>(positions);
  p.meta = reinterpret_cast<int4*>(meta);
  p.tokens = tokens; p.max_blocks = max_blocks; p.H = H; p.page_size = page_size;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.window = window;
  p.waits = g_wait_config;
  p.sink = reinterpret_cast<const float*>(sink);
  static PerDeviceOnce configured;
  if (configured.need()) {
    CUDA_CHECK_RET(cudaFuncSetAttribute(mla_attn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMlaSmem));
    configured.done();
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUDA_CHECK_RET(launch_pdl(mla_attn_kernel, dim3(ctas), dim3(kMlaThreads), kMlaSmem, st, tm, p));
  CUDA_CHECK_RET(launch_pdl(mla_merge_kernel, dim3(ctas, 4), dim3(512), 0, st, static_cast<const float*>(p.part_o),
                            static_cast<const float*>(p.part_lse), static_cast<const int4*>(p.meta), p.out, H));
  return 0;
}

// rows [nseq + 1] int32 (written), lat [total, 512], pe [total, 64]; total = the lengths of the sequences with at least min_len
// new tokens and min_work / 2 pairs, each rounded up to 64
GLLM_EXPORT int gllm_mla_gather(const void* cache, const void* block_table, int max_blocks, const void* seq_lens,
                                const void* q_start, int min_len, int min_work, int nseq, int total, int page_size, void* rows,
                                void* lat, void* pe, void* stream) {
  if (nseq <= 0 || total <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  mla_rows_kernel<<<1, 256, 0, st>>>(reinterpret_cast<const int32_t*>(seq_lens), reinterpret_cast<const int32_t*>(q_start),
                                     min_len, min_work, nseq, reinterpret_cast<int32_t*>(rows));
  mla_gather_kernel<<<(total + 7) / 8, 256, 0, st>>>(
      reinterpret_cast<const __nv_bfloat16*>(cache), reinterpret_cast<const int32_t*>(block_table), max_blocks,
      reinterpret_cast<const int32_t*>(seq_lens), reinterpret_cast<const int32_t*>(rows), nseq, total, page_size,
      reinterpret_cast<__nv_bfloat16*>(lat), reinterpret_cast<__nv_bfloat16*>(pe));
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

// q_pe: strided view [T, H, 64] of the projected queries; k_pe [T, 64]; kv_c [T, 512] (normalised latent);
// cos_sin fp32 [max_pos, 64]; writes the rotated queries to q_out (token and head strides o_ts, o_hs; may be q_pe itself) and the
// cache rows at `slots`.
GLLM_EXPORT int gllm_mla_rope_cache(const void* q_pe, int64_t q_ts, int64_t q_hs, int H, void* q_out, int64_t o_ts,
                                    int64_t o_hs, const void* k_pe, int64_t k_ts, const void* kv_c, int64_t c_ts,
                                    const void* cos_sin, const void* positions, const void* slots, void* cache,
                                    int page_size, int tokens, void* stream) {
  if (tokens <= 0) return 0;
  CUDA_CHECK_RET(launch_pdl(mla_rope_cache_kernel, dim3(tokens), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream),
                            reinterpret_cast<const __nv_bfloat16*>(q_pe), q_ts, q_hs, H,
                            reinterpret_cast<__nv_bfloat16*>(q_out), o_ts, o_hs, reinterpret_cast<const __nv_bfloat16*>(k_pe), k_ts,
                            reinterpret_cast<const __nv_bfloat16*>(kv_c), c_ts, reinterpret_cast<const float*>(cos_sin),
                            reinterpret_cast<const int32_t*>(positions), reinterpret_cast<const int32_t*>(slots),
                            reinterpret_cast<__nv_bfloat16*>(cache), page_size));
  return 0;
}
