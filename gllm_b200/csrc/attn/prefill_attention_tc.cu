// tcgen05 / TMEM paged flash attention for prefill (chunked-prefill and prefix offsets included): the
// Blackwell-native successor of the mma.sync prefill kernel in paged_attention.cu (same arguments, same
// paged KV cache; reference call site: gllm/layers/attention.py:49-61, flash_attn_varlen_func on the paged cache).
//
// The default prefill kernel for head sizes 64 and 128; GLLM_ATTN_TC=0 selects the mma.sync kernel (ops/sm100.py).
//
// One CTA = two tiles of 128 query rows (128/GP tokens x GP heads that share one KV head, GQA-packed like the mma.sync
// kernel) x the causal prefix of one sequence, walked in tiles of 128 keys (64 for DK = 192):
//
//   warps 0-3, 4-7     softmax      : one warpgroup per query tile, one row per thread (tcgen05.ld 32x32b: a thread owns a
//                                     TMEM lane): row max / exp2 / row sum without shuffles; P (bf16) goes back into the
//                                     columns that S came from, as the A operand of the PV product; O rescaled in TMEM only
//                                     when a row max has grown by 2^8
//   warp 8             TMA producer : page boxes [page_size][64] of K and V -> smem tiles [D/64][keys][64] (SW128)
//   warp 9 (1 thread)  MMA issuer   : S  = Q K^T  (tcgen05.mma, A = Q smem K-major, B = K tile K-major, D in TMEM)
//                                     O += P V    (A = P in TMEM, B = V tile **MN-major**, D in TMEM)
//
// The schedule is the published one of FlashAttention on this generation (Dao and others, "FlashAttention-4"): two query tiles
// in turn, P over S in TMEM, and a reference of the exponentials that follows the row's maximum in steps.
// The tensor core runs one query tile's PV_j and S_j+1 while the other tile's softmax works on S_j. Products of one thread
// execute in order, so S_j+1 may take P_j's columns without a wait between the two, and the barrier that announces S_j+1 also
// says that PV_j is in O.
//
// What bounds it (heads of 128): per 128 keys and two query tiles 2048 cycles of tensor core and 2048 of the special-function
// unit. Shared memory would be the third: P through it costs 1500 cycles per tile of reads and writes, hence P in TMEM.
// Products of N = 64 take 48 cycles where 32 would be their share, and every commit and barrier wait of the issuing thread
// about 100, hence 128 keys at a time and two commits per step; the block-table entries are fetched one tile ahead by the
// lanes that use them (read in turn by one thread, they alone cost 470 cycles each).
// Back to back, before (one query tile, 64 keys, P through shared memory) and now: 8192 tokens over 8192 cached, 64 / 8 heads
// of 128: 5296 -> 2702 us (623 -> 1221 TFLOP/s); 8192 tokens, 32 / 8 heads: 961 -> 507 us; 4 x 2048: 332 -> 202 us; 64 x 128:
// 119 -> 91 us; heads of 64, 4 x 2048, 32 / 8: 254 -> 168 us.
//
// With DENSE the keys and values are not paged: the expanded heads of latent attention, keys [64 x 2 | 64] wide of which the
// last 64 columns are shared by all heads (DK = 192), values DV = 128 wide.
//
// The V operand: the cache stores V as [key][d] (d contiguous), i.e. the contraction dimension (keys) runs along
// ROWS of the tile. That is the MN-major canonical layout of the UMMA shared-memory descriptor
//     SW128, MN-major, in 16-byte units: ((8, n), (8, k)) : ((1, LBO), (8, SBO))
// -> 64 d-values (128 B) contiguous, next 64 d-values LBO bytes away (= one [64][64] slab), 8 keys are 8
// consecutive 128-byte rows, the next 8 keys SBO = 1024 B away; a K = 16 step advances the start address by 2048 B.
#include "../common/bounded.cuh"
#include "attn_common.cuh"

namespace b200 {

static constexpr int kTcRows = 128;                      // query rows of a tile (UMMA M)
static constexpr int kTcKeys = 128;                      // keys of a KV tile (64 where the keys are wider than 128)
static constexpr int kTcSoftmaxWarps = 8;                // four per query tile
static constexpr int kTcThreads = (kTcSoftmaxWarps + 4) * 32;
// Registers per thread after the split (a softmax thread holds a row of S): 128 x 72 + 256 x 216 is what 384 threads are
// launched with (168 each).
static constexpr int kTcRegsIssue = 72, kTcRegsSoftmax = 216;
static constexpr float kTcLazy = 8.f;                    // P stays below 2^8 between two rescales of O

struct TcAttnParams {
  const __nv_bfloat16* q;
  int64_t q_ts;
  __nv_bfloat16* out;
  const int32_t* block_table;
  const int32_t* seq_lens;
  const int32_t* q_start;
  int max_blocks, Hq, Hkv, G, GP, page_size, seq_offset, num_seqs, flat;
  float scale_log2;
  // score cap (kernel template CAP): a scaled score s becomes cap * tanh(s / cap); cap_log2 = cap * log2(e),
  // scale_over_cap = scale / cap. sink: one extra logit per query head in the softmax denominator that carries no
  // value (null = none)
  float cap_log2, scale_over_cap;
  const float* sink;
  int64_t out_ts;     // output row stride (elements)
  int window;         // sliding window: a query at i sees keys j with i - j < window (0 = the whole past)
  AttnExtras ex;      // distance bias or table (kernel template BIAS), turned values, output gate
  WaitConfig waits;
  int q_tiles;        // query tiles per CTA (2, or 1 where that gives every SM at most one CTA)
  const int32_t* kv_row;   // DENSE: first row of each sequence of this launch in the expanded keys and values
};

// BIAS of the kernel: none, the logarithmic distance bias, the distance table
enum TcBias : int { kNoBias = 0, kLogBias = 1, kTableBias = 2 };
static constexpr int kTabFloats = 8192;                  // staging of a distance table (fits beside four KV stages)

template <int DK, int DV, int BIAS>
struct TcSmem {
  static constexpr int KV = DK > 128 ? 64 : kTcKeys;
  static constexpr int kTabBytes = BIAS == kTableBias ? kTabFloats * 4 : 0;
  static constexpr int kQBytes = kTcRows * DK * 2;         // one query tile
  static constexpr int kKBytes = KV * DK * 2, kVBytes = KV * DV * 2;
  // as many stages as fit next to Q and the table (227 KB per CTA); K runs a tile ahead of V
  static constexpr int kKStages = DK == 128 && BIAS == kTableBias ? 2 : 3;
  static constexpr int kVStages = DK == 128 ? 2 : 3;
  static constexpr int kKOff = 2 * kQBytes, kVOff = kKOff + kKStages * kKBytes, kTabOff = kVOff + kVStages * kVBytes,
                       kBarOff = kTabOff + kTabBytes;
  static constexpr int kBytes = kBarOff + 256 + 1024;
  static_assert(kBytes <= 232448, "shared memory of a CTA");
  static constexpr int kTmemO = 2 * KV, kTmemCols = 512;   // S (and P) of the two tiles, then O of both
  static_assert(kTmemO + 2 * DV <= 512, "TMEM budget");
};

// tcgen05.mma with A (bf16 pairs, one row per lane) in TMEM
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
// two fp32 operations in one issue slot
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// SW128 descriptor with explicit LBO / SBO (MN-major operands use both)
__device__ __forceinline__ uint64_t make_sw128_desc(uint32_t smem_addr, uint32_t lbo16, uint32_t sbo16) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFF);
  d |= static_cast<uint64_t>(lbo16 & 0x3FFF) << 16;
  d |= static_cast<uint64_t>(sbo16 & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

template <int DK, int DV, bool DENSE, bool CAP, int BIAS>
__global__ void __launch_bounds__(kTcThreads, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                       const __grid_constant__ CUtensorMap tmap_pe, const __grid_constant__ CUtensorMap tmap_q,
                       const TcAttnParams p) {
  using SM = TcSmem<DK, DV, BIAS>;
  constexpr int KV = SM::KV;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::kBarOff);
  uint64_t* k_full = bars;                             // [kKStages] TMA -> MMA
  uint64_t* v_full = k_full + SM::kKStages;            // [kVStages]
  uint64_t* s_full = v_full + SM::kVStages;            // [1] tile 0: phase j = S_j written, PV_j-1 in O
  uint64_t* step = s_full + 1;                         // [4] step j = the same for tile 1; K_j and V_j-1 are free (producer).
                                                       // Step j is phase j / 4 of barrier j % 4: the producer lags up to two
  uint64_t* p_full = step + 4;                         // [2 tiles] softmax (4 warps) -> MMA: P_j written, S_j read
  uint64_t* q_full = p_full + 2;                       // [2 tiles] Q staged (TMA)
  uint64_t* mma_end = q_full + 2;                      // [1]       every product has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_end + 1);
  const WaitGuard guard{tmem_slot + 1, p.waits};
  volatile int* sees = reinterpret_cast<int*>(tmem_slot + 2);   // [2 tiles][low, end): keys that a query tile sees, from tile0 on

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Head groups first, then sequences, then from the last query block of each to the first: the CTAs that start late are the
  // ones with few keys. (One sequence of one head after the other left the last wave to the long blocks of the last head: expanded
  // latent heads, 5 prompts of 4096 tokens in all, 169 us for 145; 19 prompts, 32 / 8 heads of 128, 65.6 for 63.9; 8192 tokens over
  // 8192 cached, 64 / 8 heads, 2751 for 2703.)
  // The grid has them in this order; where a count is beyond its dimension it is flat (dividing there costs a short portion 0.4 us:
  // 16 of 64 tokens, 8 / 1 heads 8.2 us for 8.6).
  const int groups_per_kv = p.G / p.GP;
  int z = blockIdx.x, seq_in = blockIdx.y, back = blockIdx.z;
  if (p.flat) {
    z = blockIdx.x % (p.Hkv * groups_per_kv);
    const int rest = blockIdx.x / (p.Hkv * groups_per_kv);
    seq_in = rest % p.num_seqs;
    back = rest / p.num_seqs;
  }
  const int seq = seq_in + p.seq_offset;
  const int kvh = z / groups_per_kv;
  const int hbase = kvh * p.G + (z % groups_per_kv) * p.GP;
  const int q_begin = p.q_start[seq], q_len = p.q_start[seq + 1] - q_begin;
  if (DENSE && p.kv_row[seq_in + 1] == p.kv_row[seq_in]) return;      // no rows: not expanded
  const int toks_per_tile = kTcRows / p.GP;
  const int toks_per_cta = toks_per_tile * p.q_tiles;
  const int n_blocks = (q_len + toks_per_cta - 1) / toks_per_cta;
  if (back >= n_blocks) return;
  const int tok_cta = (n_blocks - 1 - back) * toks_per_cta;
  const int seq_len = p.seq_lens[seq];
  const int ctx_len = seq_len - q_len;
  // KV tiles [tile0, tile0 + n): with a window the first query's oldest visible key decides where they start; pipeline
  // indices (stages, phases, buffers) count from 0. A query tile ends at the causal horizon of its last token.
  const int tile0 = p.window > 0 ? max(0, ctx_len + tok_cta - p.window + 1) / KV : 0;
  auto tiles_of = [&](int t) {
    const int tok0 = tok_cta + t * toks_per_tile;
    if (t >= p.q_tiles || tok0 >= q_len) return 0;
    return (ctx_len + min(tok0 + toks_per_tile, q_len) + KV - 1) / KV - tile0;
  };
  const int n0 = tiles_of(0), n1 = tiles_of(1), n_max = max(n0, n1);

  // One lane per box (DENSE: per slab). The block-table entries are fetched one tile ahead: read where it is used, each
  // cost the copies of a tile some 470 cycles, and with 16-token pages that chain alone took as long as four softmax tiles.
  const int box = min(p.page_size, 64);                // rows of a box
  const int boxes = DENSE ? 1 : KV / box;
  const int j = lane % boxes, sl = lane / boxes;       // this lane's box and 64-wide slab
  const int32_t* bt = p.block_table + static_cast<size_t>(seq) * p.max_blocks;
  const int last_page = (seq_len - 1) / p.page_size;
  const int row0 = DENSE ? p.kv_row[seq_in] : 0;
  auto page_of = [&](int tile) {                       // masked columns read the last page: keep the data finite
    return DENSE ? 0 : bt[min(((tile0 + tile) * KV + j * box) / p.page_size, last_page)];
  };
  // Boxes of the last K / V tile that hold a key some query of this CTA sees, in steps of 16 keys (a step of the product with V); the
  // others stay out. (Worked out per tile, the division held the copies up by 6 to 9 % in long prompts.)
  const int rows_last = min((ctx_len + min(tok_cta + toks_per_cta, q_len) - (tile0 + n_max - 1) * KV + 15) & ~15, KV);
  const int boxes_last = DENSE ? 1 : min((rows_last + box - 1) / box, boxes);
  auto load = [&](int tile, int page, uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int width, bool is_v) {
    const int n = tile + 1 < n_max ? boxes : boxes_last;
    if (lane == 0) mbar_expect_tx(bar, (DENSE ? KV : n * box) * width * 2);
    __syncwarp();
    if (sl >= width / 64 || j >= n) return;
    if constexpr (DENSE) {
      const int row = row0 + (tile0 + tile) * KV;
      if (sl < 2) tma_load_2d(dst + sl * (KV * 128), map, bar, kvh * 256 + (is_v ? 128 : 0) + sl * 64, row, kEvictNormal);
      else tma_load_2d(dst + sl * (KV * 128), &tmap_pe, bar, 0, row, kEvictNormal);
    } else {
      tma_load_3d(dst + sl * (KV * 128) + j * box * 128, map, bar, 0, ((tile0 + tile) * KV + j * box) % p.page_size,
                  (page * p.Hkv + kvh) * (width / 64) + sl);
    }
  };
  auto load_q = [&](int t) {                           // rows tok * GP + head of a query tile, 64 columns per box
    if ((t ? n1 : n0) == 0) return;
    if (lane == 0) mbar_expect_tx(&q_full[t], SM::kQBytes);
    __syncwarp();
    if (lane < DK / 64)
      tma_load_3d(smem + t * SM::kQBytes + lane * (kTcRows * 128), &tmap_q, &q_full[t], lane * 64, hbase,
                  q_begin + tok_cta + t * toks_per_tile);
  };
  int page = 0;                                        // of the K tile to come
  if (warp == kTcSoftmaxWarps) {
    // The first copies are on their way while the others wait for tensor memory.
    if (lane < 3) tma_prefetch_desc(lane == 0 ? &tmap_q : lane == 1 ? &tmap_k : DENSE ? &tmap_pe : &tmap_v);
    if (n_max > 0) page = page_of(0);
    if (lane == 0) {
      for (int i = 0; i < SM::kKStages; ++i) mbar_init(&k_full[i], 1);
      for (int i = 0; i < SM::kVStages; ++i) mbar_init(&v_full[i], 1);
      mbar_init(s_full, 1);
      for (int i = 0; i < 4; ++i) mbar_init(&step[i], 1);
      for (int i = 0; i < 2; ++i) { mbar_init(&p_full[i], 4); mbar_init(&q_full[i], 1); }
      mbar_init(mma_end, 1);
      *guard.dead = 0;
      for (int t = 0; t < 2; ++t) {
        const int tok0 = tok_cta + t * toks_per_tile;
        sees[2 * t] = p.window > 0 ? max(ctx_len + tok0 - p.window + 1 - tile0 * KV, 0) : 0;
        sees[2 * t + 1] = ctx_len + min(tok0 + toks_per_tile, q_len) - tile0 * KV;
      }
      fence_mbar_init();
    }
    __syncwarp();
    if (n_max > 0) {
      load_q(0);
      load(0, page, smem + SM::kKOff, &tmap_k, &k_full[0], DK, false);
      load_q(1);
    }
  }
  if (warp == kTcSoftmaxWarps + 1) tmem_alloc<1>(tmem_slot, SM::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp >= kTcSoftmaxWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcRegsIssue));
    if (warp == kTcSoftmaxWarps) {
      // ------------------------------------------------------------------ TMA producer
      auto after_step = [&](int j) { return j < 0 || guard.wait<true>(&step[j & 3], (j >> 2) & 1); };
      int tk = n_max > 0 ? 1 : 0, tv = 0;                  // tiles issued
      bool ok = true;
      int page_v = page;
      page = n_max > 1 ? page_of(1) : 0;
      for (int tile = 1; tile <= n_max; ++tile) {
        const int next = tile + 1 < n_max ? page_of(tile + 1) : 0;
        if (tile < n_max) {                                // K_tile
          const int ks = tile % SM::kKStages;
          ok = __all_sync(0xffffffffu, after_step(tile - SM::kKStages));
          if (!ok) break;
          load(tile, page, smem + SM::kKOff + ks * SM::kKBytes, &tmap_k, &k_full[ks], DK, false);
          ++tk;
        }
        const int v = tile - 1, vs = v % SM::kVStages;     // V_tile-1
        ok = __all_sync(0xffffffffu, after_step(v - SM::kVStages + 1));
        if (!ok) break;
        load(v, page_v, smem + SM::kVOff + vs * SM::kVBytes, &tmap_v, &v_full[vs], DV, true);
        ++tv;
        page_v = page;
        page = next;
      }
      if (n_max > 0) {                                     // copies in flight land before the CTA ends, whichever role gave up
        for (int t = 0; t < 2; ++t)
          if ((t ? n1 : n0) > 0) guard.land(&q_full[t], 0);
        for (int i = max(0, tk - SM::kKStages); i < tk; ++i) guard.land(&k_full[i % SM::kKStages], (i / SM::kKStages) & 1);
        for (int i = max(0, tv - SM::kVStages); i < tv; ++i) guard.land(&v_full[i % SM::kVStages], (i / SM::kVStages) & 1);
      }
    } else if (warp == kTcSoftmaxWarps + 1 && lane == 0) {
      // ------------------------------------------------------------------ MMA issuer
      constexpr uint32_t idesc_s = make_idesc_bf16(kTcRows, KV);
      constexpr uint32_t idesc_pv = make_idesc_bf16(kTcRows, DV) | (1u << 16);
      auto issue_s = [&](int t, int tile) {
        const uint32_t q_addr = smem_u32(smem + t * SM::kQBytes),
                       k_addr = smem_u32(smem + SM::kKOff + (tile % SM::kKStages) * SM::kKBytes), d_tmem = tmem + t * KV;
#pragma unroll
        for (int kd = 0; kd < DK / 64; ++kd) {
          const uint64_t da = make_sw128_kmajor_desc(q_addr + kd * (kTcRows * 128));
          const uint64_t db = make_sw128_kmajor_desc(k_addr + kd * (KV * 128));
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_bf16<1>(d_tmem, da + kk * 2, db + kk * 2, idesc_s, (kd | kk) != 0);
        }
      };
      // Only the 16-key steps that some row of the query tile sees: a masked key has P = 0, but 0 times a value that is no
      // number is none either, so keys behind the tile's last token (or before its window) stay out of the product.
      // (The range is kept in shared memory: in registers it made this role spill.) DENSE takes its tiles of 64 keys whole, as the
      // absorbed form does: with a range the prompts of 4096 tokens, 16 heads, take 427 us instead of 419.
      auto issue_pv = [&](int t, int tile, int low, int end) {
        const uint32_t v_addr = smem_u32(smem + SM::kVOff + (tile % SM::kVStages) * SM::kVBytes);
        const uint64_t dv = make_sw128_desc(v_addr, (KV * 128) >> 4, 1024 >> 4);
        const uint32_t o_tmem = tmem + SM::kTmemO + t * DV, p_tmem = tmem + t * KV;
        const uint32_t acc = low < 0 ? 1u : 0u;          // an earlier tile wrote O
        if (DENSE || (end >= KV && low <= 0)) {          // all but the first and the last tiles
#pragma unroll
          for (int kk = 0; kk < KV / 16; ++kk)           // 16 keys per step: 8 columns of P, 16 rows of V
            umma_bf16_ts(o_tmem, p_tmem + kk * 8, dv + static_cast<uint64_t>(kk) * (2048 >> 4), idesc_pv, kk != 0 ? 1u : acc);
        } else {
          const int k0 = max(low, 0) / 16, k1 = min((end + 15) / 16, KV / 16);
#pragma unroll 1
          for (int kk = k0; kk < k1; ++kk)
            umma_bf16_ts(o_tmem, p_tmem + kk * 8, dv + static_cast<uint64_t>(kk) * (2048 >> 4), idesc_pv, kk != k0 ? 1u : acc);
        }
      };
      bool ok = n_max > 0 && guard.first(&k_full[0]);
      for (int t = 0; t < 2; ++t)
        if (t ? n1 : n0) ok = ok && guard.wait<true>(&q_full[t], 0);
      ok = ok && guard.wait<true>(&k_full[0], 0);
      if (ok) {
        tc_fence_after();
        if (n0 > 0) { issue_s(0, 0); umma_commit(s_full); }
        if (n1 > 0) issue_s(1, 0);
        umma_commit(&step[0]);
      }
      for (int tile = 0; tile < n_max && ok; ++tile) {
        if (tile + 1 < n_max) ok = guard.wait<true>(&k_full[(tile + 1) % SM::kKStages], ((tile + 1) / SM::kKStages) & 1);
        ok = ok && guard.wait<true>(&v_full[tile % SM::kVStages], (tile / SM::kVStages) & 1);
        for (int t = 0; t < 2 && ok; ++t) {
          const int n = t ? n1 : n0;
          if (tile < n) {
            const int low = DENSE ? -tile : sees[2 * t] - tile * KV, end = DENSE ? KV : sees[2 * t + 1] - tile * KV;
            ok = guard.wait<true>(&p_full[t], tile & 1);
            if (!ok) break;
            tc_fence_after();
            issue_pv(t, tile, low, end);
            if (tile + 1 < n) issue_s(t, tile + 1);
            if (t == 0) umma_commit(s_full);
          }
        }
        umma_commit(&step[(tile + 1) & 3]);
      }
      umma_commit(mma_end);                              // nothing is in flight when the columns are given back
      guard.land(mma_end, 0);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcRegsSoftmax));
    if ((warp >> 2 ? n1 : n0) > 0 || BIAS == kTableBias) {
      // ------------------------------------------------------------------ softmax warps: one row per thread
      const int qt = warp >> 2;                            // query tile
      const int n_tiles = qt ? n1 : n0;
      const int row = threadIdx.x & 127;                   // == TMEM lane
      const int tok_base = tok_cta + qt * toks_per_tile;
      const int last_tok = min(tok_base + toks_per_tile, q_len) - 1;
      const int tok = tok_base + row / p.GP;
      const int head = hbase + row % p.GP;
      const bool row_ok = tok < q_len && n_tiles > 0;
      const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
      const uint32_t tmem_o = tmem + SM::kTmemO + qt * DV;
      const int lim = ctx_len + tok;                       // last visible key of this row
      const int low = p.window > 0 ? lim - p.window + 1 : 0;          // first visible key of this row
      float b1 = 0.f, b2 = 0.f;
      if (BIAS == kLogBias) { b1 = p.ex.r1[head]; b2 = p.ex.r2[head]; }
      // distance table: staged once per CTA for every distance that its near tiles meet, [distance - dmin][GP heads], so the
      // lanes of a warp (tokens x heads) read neighbouring words
      float* stab = reinterpret_cast<float*>(smem + SM::kTabOff);
      const int dmin = 2 - KV - toks_per_tile;             // smallest distance of any tile (keys behind the diagonal)
      if (BIAS == kTableBias) {
        b1 = dist_table_log2(p.ex.dtab + head, p.ex.dtab_n, p.Hq, p.ex.dtab_n - 1);
        const int last_cta = min(tok_cta + toks_per_cta, q_len) - 1;
        const int dmax = min(p.ex.dtab_n + KV + toks_per_tile - 3, ctx_len + last_cta);
        const int total = (dmax - dmin + 1) * p.GP;
        const int dstep = 2 * kTcRows / p.GP;              // GP divides the row count: a thread keeps its head
        const float* col = p.ex.dtab + head;
        int d = dmin + static_cast<int>(threadIdx.x) / p.GP;
#pragma unroll 4
        for (int e = threadIdx.x; e < total; e += 2 * kTcRows, d += dstep) stab[e] = dist_table_log2(col, p.ex.dtab_n, p.Hq, d);
        asm volatile("bar.sync 1, 256;" ::: "memory");
      }
      float m_run = -INFINITY, l_run = 0.f;
      // phase j of the query tile: S_j is there and PV_j-1 is in O
      auto await = [&](int j) {
        if (qt == 0) guard.wait<true>(s_full, j & 1);
        else guard.wait<true>(&step[j & 3], (j >> 2) & 1);
        tc_fence_after();
      };
      const uint32_t t_s = tmem + lane_base + qt * KV, t_o = tmem_o + lane_base;
      constexpr bool kRaw = BIAS == kNoBias && !CAP;
      const int left_last = ctx_len + last_tok + 1 - (tile0 + n_tiles - 1) * KV;      // keys that the query tile sees of its last tile
      const bool short_last = !DENSE && left_last <= KV / 2;   // tiles of 64 keys gain nothing by it
      for (int tile = 0; tile < n_tiles; ++tile) {
        // smallest distance of the tile (uniform over the query tile); at the table's end every score gets the same entry
        const int d0 = ctx_len + tok_base - ((tile0 + tile) * KV + KV - 1);
        const bool far_tile = BIAS == kTableBias && d0 >= p.ex.dtab_n - 1;
        const float* trow = stab + (d0 - dmin) * p.GP + row;      // + (KV - 1 - c) GP: the entry of the tile's key c
        const int key0 = (tile0 + tile) * KV;
        // uniform over the query tile: a diagonal tile, or one that the window of some row starts in
        const bool need_mask = key0 + KV - 1 > ctx_len + tok_base ||
                               (p.window > 0 && key0 < ctx_len + last_tok - p.window + 1);
        await(tile);
        // the reference of the exponents follows the row's maximum only in steps of 2^8: P, l and O are all relative to it
        auto follow = [&](float m_new) {
          float alpha = 1.f;
          if (m_new > m_run + kTcLazy) {
            alpha = exp2f(m_run - m_new);
            m_run = m_new;
          }
          if (tile > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
            for (int c = 0; c < DV; c += 16) {
              uint32_t v[16];
              tmem_ld_32x16(t_o + c, v);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
              tmem_st_32x16(t_o + c, v);
            }
          }
          return alpha;
        };
        if (short_last && tile + 1 == n_tiles) {
          // A last tile that is half empty or more (all there is of a short prompt): 32 keys at a time, S read twice, nothing
          // done for the rest, which the product leaves out too.
          const int groups = (left_last + 31) / 32;
          auto score = [&](uint32_t raw, int c) {
            float x = __uint_as_float(raw);
            if (BIAS == kTableBias) x = fmaf(x, p.scale_log2, far_tile ? b1 : trow[(KV - 1 - c) * p.GP]);
            else if (BIAS == kLogBias) x = fmaf(x, p.scale_log2, -dist_bias_log2(b1, b2, lim - (key0 + c)));
            else if (CAP) x = p.cap_log2 * tanh_exp(x * p.scale_over_cap);
            return key0 + c > lim || key0 + c < low ? -INFINITY : x;
          };
          float mx = -INFINITY;
#pragma unroll 1
          for (int g = 0; g < groups; ++g) {
            uint32_t v[32];
            tmem_ld_32x32(t_s + g * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) mx = fmaxf(mx, score(v[e], g * 32 + e));
          }
          const float alpha = follow(fmaxf(m_run, kRaw ? mx * p.scale_log2 : mx));
          const float m_use = m_run == -INFINITY ? 0.f : m_run;
          float sum = 0.f;
#pragma unroll 1
          for (int g = 0; g < groups; ++g) {
            uint32_t v[32], pk[16];
            tmem_ld_32x32(t_s + g * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float y0 = exp2f(fmaf(score(v[2 * e], g * 32 + 2 * e), kRaw ? p.scale_log2 : 1.f, -m_use)),
                          y1 = exp2f(fmaf(score(v[2 * e + 1], g * 32 + 2 * e + 1), kRaw ? p.scale_log2 : 1.f, -m_use));
              sum += y0 + y1;
              pk[e] = pack_bf16(y0, y1);
            }
            tmem_st_32x16(t_s + g * 16, pk);               // into columns whose scores have been read
          }
          l_run = l_run * alpha + sum;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[qt]);
          continue;
        }
        // the whole row of the tile stays in registers: S leaves TMEM once
        float f[KV];
        {
          uint32_t v[KV / 32][32];
#pragma unroll
          for (int c = 0; c < KV / 32; ++c) tmem_ld_32x32(t_s + c * 32, v[c]);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < KV; ++e) f[e] = __uint_as_float(v[e / 32][e % 32]);
        }
        // scores in the base-2 domain of the softmax (raw without bias and cap: the scale rides on the exponent's fma); masked
        // ones are -inf
        if (BIAS == kTableBias && !far_tile) {
          const float* tr = trow + (KV - 1) * p.GP;
#pragma unroll
          for (int e = 0; e < KV; ++e) f[e] = fmaf(f[e], p.scale_log2, tr[-e * p.GP]);
        } else if (!kRaw) {
#pragma unroll
          for (int e = 0; e < KV; ++e)
            f[e] = BIAS == kTableBias ? fmaf(f[e], p.scale_log2, b1)
                   : BIAS == kLogBias ? fmaf(f[e], p.scale_log2, -dist_bias_log2(b1, b2, lim - (key0 + e)))
                                      : p.cap_log2 * tanh_exp(f[e] * p.scale_over_cap);
        }
        if (need_mask) {
#pragma unroll
          for (int e = 0; e < KV; ++e)
            if (key0 + e > lim || key0 + e < low) f[e] = -INFINITY;
        }
        float m4[4] = {f[0], f[1], f[2], f[3]};
#pragma unroll
        for (int e = 4; e < KV; e += 8) {
#pragma unroll
          for (int i = 0; i < 4; ++i) m4[i] = fmaxf(m4[i], e + 4 < KV ? fmaxf(f[e + i], f[e + 4 + i]) : f[e + i]);
        }
        const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        const float alpha = follow(fmaxf(m_run, kRaw ? mx * p.scale_log2 : mx));
        const float m_use = m_run == -INFINITY ? 0.f : m_run;
        const uint64_t sc2 = pack2(kRaw ? p.scale_log2 : 1.f, kRaw ? p.scale_log2 : 1.f), nm2 = pack2(-m_use, -m_use);
        uint64_t sum2[2] = {0, 0};
#pragma unroll
        for (int c = 0; c < KV; c += 32) {                 // 32 keys: 16 columns of P
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 x = unpack2(fma2(pack2(f[c + 2 * e], f[c + 2 * e + 1]), sc2, nm2));
            const float2 y = make_float2(exp2f(x.x), exp2f(x.y));
            sum2[e & 1] = add2(sum2[e & 1], pack2(y.x, y.y));
            pk[e] = pack_bf16(y.x, y.y);
          }
          tmem_st_32x16(t_s + c / 2, pk);
        }
        const float2 sa = unpack2(add2(sum2[0], sum2[1]));
        l_run = l_run * alpha + (sa.x + sa.y);
        tmem_st_wait();
        tc_fence_before();                                 // P and the rescaled O are in TMEM, S has been read
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[qt]);
      }
      // ---- epilogue: O / l -> bf16 -> global
      if (n_tiles > 0) {
        await(n_tiles);
        if (p.sink != nullptr && row_ok && m_run > -INFINITY) l_run += exp2f(p.sink[head] * 1.4426950408889634f - m_run);
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        __nv_bfloat16* op = p.out + static_cast<size_t>(q_begin + tok) * p.out_ts + static_cast<size_t>(head) * DV;
        const __nv_bfloat16* gp = p.ex.gate != nullptr && row_ok
                                      ? p.ex.gate + static_cast<size_t>(q_begin + tok) * p.ex.ldg + static_cast<size_t>(head) * DV
                                      : nullptr;
        // 32 finished columns from column c on: normalise, gate, round, store
        auto store32 = [&](int c, const float (&f)[32]) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = f[g * 8 + e] * inv;
            if (gp != nullptr) {
              const uint4 gv = *reinterpret_cast<const uint4*>(gp + c + g * 8);
              const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 z = unpack_bf16(gw[e]);
                x[2 * e] *= sigmoid_fast(z.x);
                x[2 * e + 1] *= sigmoid_fast(z.y);
              }
            }
            uint4 w;
            w.x = pack_bf16(x[0], x[1]);
            w.y = pack_bf16(x[2], x[3]);
            w.z = pack_bf16(x[4], x[5]);
            w.w = pack_bf16(x[6], x[7]);
            *reinterpret_cast<uint4*>(op + c + g * 8) = w;
          }
        };
        if (p.ex.v_turn != nullptr) {
          // turn the head's result back: columns m and m + D / 2 of this row, both in this thread's TMEM lane
          const float4* tr =
              reinterpret_cast<const float4*>(p.ex.v_turn + static_cast<size_t>(q_begin + (row_ok ? tok : 0)) * DV);
#pragma unroll 1
          for (int c = 0; c < DV / 2; c += 32) {
            uint32_t a[32], b[32];
            tmem_ld_32x32(t_o + c, a);
            tmem_ld_32x32(t_o + DV / 2 + c, b);
            tmem_ld_wait();
            if (row_ok) {
              float fa[32], fb[32];
#pragma unroll
              for (int g = 0; g < 8; ++g) {
                const float4 cv = tr[c / 4 + g], sv = tr[DV / 8 + c / 4 + g];
                const float cs[4] = {cv.x, cv.y, cv.z, cv.w}, sn[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float u = __uint_as_float(a[g * 4 + e]), w = __uint_as_float(b[g * 4 + e]);
                  fa[g * 4 + e] = u * cs[e] + w * sn[e];
                  fb[g * 4 + e] = w * cs[e] - u * sn[e];
                }
              }
              store32(c, fa);
              store32(c + DV / 2, fb);
            }
            __syncwarp();
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < DV; c += 32) {
            uint32_t v[32];
            tmem_ld_32x32(t_o + c, v);
            tmem_ld_wait();
            if (row_ok) {
              float f[32];
#pragma unroll
              for (int e = 0; e < 32; ++e) f[e] = __uint_as_float(v[e]);
              store32(c, f);
            }
            __syncwarp();
          }
        }
        tc_fence_before();
      }
    }
  }
  __syncthreads();
  if (warp == kTcSoftmaxWarps + 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc<1>(tmem, SM::kTmemCols);
  }
}

// tensor map over the paged cache with ONE 64-wide slab per box ([page_size][64]), so that a KV tile can be
// assembled slab-major ([D/64][keys][64]) — the layout both UMMA operand forms need (pages of 128 keys: two boxes)
static int get_kv_slab_tmap(const void* base, int64_t num_pages, int Hkv, int D, int page_size, CUtensorMap* out) {
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  static std::mutex mu;
  TmapKey key{base, num_pages, Hkv, D, page_size};
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return 0;
  }
  CUtensorMap m;
  cuuint64_t dims[3] = {64, (cuuint64_t)page_size, (cuuint64_t)(num_pages * Hkv * (D / 64))};
  cuuint64_t strides[2] = {128, (cuuint64_t)page_size * 128};
  cuuint32_t box[3] = {64, (cuuint32_t)(page_size < 64 ? page_size : 64), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = get_encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box,
                               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "[gllm_b200] KV slab tensor-map encode failed (%d)\n", (int)r);
    return 1;
  }
  cache.emplace(key, m);
  *out = m;
  return 0;
}

template <int DK, int DV, bool DENSE, bool CAP = false, int BIAS = kNoBias>
static int launch_prefill_tc(const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tpe, TcAttnParams p, int num_seqs,
                             int num_tokens, int max_q_len, cudaStream_t st) {
  using SM = TcSmem<DK, DV, BIAS>;
  static PerDeviceOnce configured;
  if (configured.need()) {
    CUDA_CHECK_RET(cudaFuncSetAttribute(attn_prefill_tc_kernel<DK, DV, DENSE, CAP, BIAS>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, SM::kBytes));
    configured.done();
  }
  // One query tile per CTA while that leaves at most one CTA per SM (short prompts): two would only halve the SMs at work
  p.waits = g_wait_config;
  const int toks = kTcRows / p.GP, z = p.Hkv * (p.G / p.GP);
  const int64_t single = static_cast<int64_t>((max_q_len + toks - 1) / toks) * num_seqs * z;
  p.q_tiles = single <= num_sms() ? 1 : 2;
  const int toks_per_cta = toks * p.q_tiles;
  CUtensorMap tq;                                        // queries [tok][head][DK]; a box is a query tile's 64 columns
  const cuuint64_t dims[3] = {DK, static_cast<cuuint64_t>(p.Hq), static_cast<cuuint64_t>(num_tokens)};
  const cuuint64_t strides[2] = {DK * 2, static_cast<cuuint64_t>(p.q_ts) * 2};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(p.GP), static_cast<cuuint32_t>(toks)}, estr[3] = {1, 1, 1};
  const CUresult r = get_encode_fn()(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(p.q), dims, strides,
                                     box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "[gllm_b200] query tensor-map encode failed (%d)\n", (int)r);
    return 1;
  }
  p.num_seqs = num_seqs;
  const int blocks = (max_q_len + toks_per_cta - 1) / toks_per_cta;
  const int64_t ctas = static_cast<int64_t>(blocks) * num_seqs * z;
  if (ctas > 0x7fffffff) {
    fprintf(stderr, "[gllm_b200] prefill attention: %lld blocks\n", static_cast<long long>(ctas));
    return 1;
  }
  p.flat = num_seqs > 65535 || blocks > 65535;
  const dim3 grid = p.flat ? dim3(static_cast<unsigned>(ctas)) : dim3(z, num_seqs, blocks);
  attn_prefill_tc_kernel<DK, DV, DENSE, CAP, BIAS><<<grid, kTcThreads, SM::kBytes, st>>>(tk, tv, tpe, tq, p);
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

}  // namespace b200

using namespace b200;

// Same contract as gllm_attn_prefill (paged_attention.cu). Returns 2 when the shape is outside this kernel's
// envelope (head_dim 64 / 128, page_size dividing the KV tile) — the caller then uses the mma.sync kernel.
// kv_tile (64 or 128) only bounds the page size; the kernel walks 128 keys at a time.
static int attn_prefill_tc_impl(const void* q, int64_t q_ts, void* out, const void* k_cache, const void* v_cache,
                                int64_t num_pages, const void* block_table, const void* seq_lens,
                                const void* q_start, int num_tokens, int num_seqs, int seq_offset, int max_q_len,
                                int max_blocks, int Hq, int Hkv, int D, int page_size, float scale, int kv_tile,
                                const void* sink, float softcap, void* stream, int window = 0, int64_t out_ts = 0,
                                const AttnExtras& ex = AttnExtras()) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  if ((D != 64 && D != 128) || (kv_tile != 64 && kv_tile != 128) || page_size < 8 || kv_tile % page_size != 0 ||
      q_ts % 8 != 0 || (reinterpret_cast<uintptr_t>(q) & 15) != 0 ||
      Hq % Hkv != 0 || ((ex.r1 != nullptr || ex.dtab != nullptr) && softcap > 0.f) ||
      (ex.dtab != nullptr && ex.r1 != nullptr))
    return 2;
  if (ex.dtab != nullptr && 64 % page_size != 0) return 2;
  CUtensorMap tk, tv;
  if (get_kv_slab_tmap(k_cache, num_pages, Hkv, D, page_size, &tk)) return 1;
  if (get_kv_slab_tmap(v_cache, num_pages, Hkv, D, page_size, &tv)) return 1;
  TcAttnParams p;
  p.q = reinterpret_cast<const __nv_bfloat16*>(q); p.q_ts = q_ts;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.block_table = reinterpret_cast<const int32_t*>(block_table);
  p.seq_lens = reinterpret_cast<const int32_t*>(seq_lens);
  p.q_start = reinterpret_cast<const int32_t*>(q_start);
  p.max_blocks = max_blocks; p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv;
  p.GP = 0;
  for (int d = (p.G < kTcRows ? p.G : kTcRows); d >= 1; --d) {
    // with a distance table: as many heads per CTA as its staged part allows
    if (p.G % d == 0 && kTcRows % d == 0 &&
        (ex.dtab == nullptr || (int64_t)(ex.dtab_n + 2 * (kTcKeys + kTcRows / d)) * d <= kTabFloats)) {
      p.GP = d;
      break;
    }
  }
  if (p.GP == 0) return 2;
  p.page_size = page_size; p.seq_offset = seq_offset;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  p.scale_over_cap = softcap > 0.f ? scale / softcap : 0.f;
  p.sink = reinterpret_cast<const float*>(sink);
  p.out_ts = out_ts > 0 ? out_ts : static_cast<int64_t>(Hq) * D;
  p.window = window;
  p.ex = ex;
  p.kv_row = nullptr;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define GLLM_TC(CAP, BIAS)                                                                                    \
  (D == 128 ? launch_prefill_tc<128, 128, false, CAP, BIAS>(tk, tv, tk, p, num_seqs, num_tokens, max_q_len, st) \
            : launch_prefill_tc<64, 64, false, CAP, BIAS>(tk, tv, tk, p, num_seqs, num_tokens, max_q_len, st))
  if (ex.dtab != nullptr) return GLLM_TC(false, kTableBias);
  if (ex.r1 != nullptr) return GLLM_TC(false, kLogBias);
  if (softcap > 0.f) return GLLM_TC(true, kNoBias);
  return GLLM_TC(false, kNoBias);
#undef GLLM_TC
}

GLLM_EXPORT int gllm_attn_prefill_tc(const void* q, int64_t q_ts, void* out, const void* k_cache, const void* v_cache,
                                     int64_t num_pages, const void* block_table, const void* seq_lens,
                                     const void* q_start, int num_tokens, int num_seqs, int seq_offset, int max_q_len,
                                     int max_blocks, int Hq, int Hkv, int D, int page_size, float scale, int kv_tile,
                                     void* stream) {
  return attn_prefill_tc_impl(q, q_ts, out, k_cache, v_cache, num_pages, block_table, seq_lens, q_start, num_tokens, num_seqs,
                              seq_offset, max_q_len, max_blocks, Hq, Hkv, D, page_size, scale, kv_tile, nullptr, 0.f,
                              stream);
}

// the same causal attention with a per-head softmax sink (null = none) and a tanh cap on the scaled scores
// (0 = none), a sliding window (0 = none) and the options of AttnExtras; output rows are out_ts elements apart (16-byte
// aligned), gate rows likewise
GLLM_EXPORT int gllm_attn_prefill_tc_cap(const void* q, int64_t q_ts, void* out, const void* k_cache,
                                         const void* v_cache, int64_t num_pages, const void* block_table,
                                         const void* seq_lens, const void* q_start, int num_tokens,
                                         int num_seqs, int seq_offset, int max_q_len, int max_blocks, int Hq, int Hkv, int D,
                                         int page_size, float scale, int kv_tile, const void* sink, float softcap, int window,
                                         int64_t out_ts, const void* r1, const void* r2, const void* gate, int64_t ldg,
                                         const void* v_turn, const void* dtab, int dtab_n, void* stream) {
  return attn_prefill_tc_impl(q, q_ts, out, k_cache, v_cache, num_pages, block_table, seq_lens, q_start, num_tokens, num_seqs,
                              seq_offset, max_q_len, max_blocks, Hq, Hkv, D, page_size, scale, kv_tile, sink, softcap,
                              stream, window, out_ts, make_extras(r1, r2, gate, ldg, v_turn, dtab, dtab_n));
}

// Causal attention of expanded latent heads: q [tokens, H, 192] (token stride q_ts), kv [rows, H, 256] = [128 key | 128 value
// columns], pe [rows, 64] = the key columns shared by all heads, both from kv_row[s] on for sequence s of this launch (64-row
// tiles); out [tokens, H, 128] with rows out_ts elements apart. Sequences seq_offset .. + num_seqs of seq_lens / q_start, those with
// rows (kv_row has one entry more than sequences). A slice of heads is passed by q, out and kv that start at it. Returns 2 for unaligned queries.
GLLM_EXPORT int gllm_attn_prefill_expanded(const void* q, int64_t q_ts, void* out, int64_t out_ts, const void* kv, const void* pe, int64_t rows,
                                           const void* kv_row, const void* seq_lens, const void* q_start, int num_tokens,
                                           int num_seqs, int seq_offset, int max_q_len, int H, float scale, void* stream) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  if (q_ts % 8 != 0 || (reinterpret_cast<uintptr_t>(q) & 15) != 0) return 2;
  CUtensorMap tkv, tpe;
  if (make_tmap_2d(&tkv, kv, rows, static_cast<uint64_t>(H) * 256, static_cast<uint64_t>(H) * 512, 64, 64,
                   CU_TENSOR_MAP_DATA_TYPE_BFLOAT16))
    return 1;
  if (make_tmap_2d(&tpe, pe, rows, 64, 128, 64, 64, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16)) return 1;
  TcAttnParams p = {};
  p.q = reinterpret_cast<const __nv_bfloat16*>(q); p.q_ts = q_ts;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.seq_lens = reinterpret_cast<const int32_t*>(seq_lens);
  p.q_start = reinterpret_cast<const int32_t*>(q_start);
  p.Hq = H; p.Hkv = H; p.G = 1; p.GP = 1;
  p.page_size = 64; p.seq_offset = seq_offset;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.out_ts = out_ts;
  p.kv_row = reinterpret_cast<const int32_t*>(kv_row);
  return launch_prefill_tc<192, 128, true>(tkv, tkv, tpe, p, num_seqs, num_tokens, max_q_len,
                                           reinterpret_cast<cudaStream_t>(stream));
}
