// Block-scaled FP8 (e4m3) GEMM for sm_100a, DeepSeek-V3 / Qwen3-FP8 checkpoint semantics
// (reference: gllm/layers/quantization/fp8.py:54-250 — Triton w8a8_block_fp8_matmul):
//
//   C[M,N] = sum_kb  (A8[M, kb] · W8[N, kb]^T) * a_s[M, kb] * w_s[N/128, kb]      (+ bias) -> bf16
//   A8: activations quantised per token per 128-wide K group (dynamic, amax/448), a_s fp32 [K/128, M]
//       (stored K-block-major so a warp's 32 rows read 32 consecutive floats)
//   W8: weights e4m3 [N, K] with fp32 scales per 128x128 block, w_s [N/128, K/128]
//
// The checkpoint scales are arbitrary fp32 values (not the power-of-two UE8M0 factors that
// `kind::mxf8f6f4.block_scale` applies in hardware), so each 128-deep K block is multiplied by
// `tcgen05.mma.kind::f8f6f4` into its own TMEM buffer (4 MMAs of K=32, the first one overwriting)
// and the epilogue warps promote it: acc += partial * a_s[row] * w_s[tile] in fp32 registers. Two
// TMEM buffers ping-pong per K block so the tensor core runs block kb+1 while the CUDA cores fold
// block kb. Same TMA (SWIZZLE_128B, 128 fp8 = one 128-byte row) / mbarrier ring as gemm_bf16.cu.
//
// What bounds it: its cycles, at a clock that power sets. 4096 x 36,864 x 7168 repeated for seconds takes 1.20 ms (1810 TFLOP/s) at the
// power limit, with the clock at 1.50 GHz; all-zero operands run at 1.965 GHz, 0.90 ms. Both are some 990 cycles per 128 x 256 x 128
// block, so what a change saves in cycles it may pay back in part in clock: without the fold a block took 880, where the product took 1.07
// ms for 1.22. The tensor core needs 512 of them; copies and products write and read 48 KB of shared memory, 768 at 128 bytes; a bare
// hand-over of products, fold (376 to 440 cycles of its own) and copies reaches 677. What mattered besides is who polls: threads that
// wait for a barrier without a suspend time took issue slots from the fold (some 65 cycles a block).
// No faster, each timed in a short loop, ahead of the power limit, in which this kernel with polling waits took 1110 us: sixteen fold warps (1290),
// scales copied by cp.async behind a barrier of their own (1230), boxes of 128 or 256 weight rows, tensor memory handed back before the last sums
// are added, pairs of SMs. The scales come from global memory (some 700 cycles away) and are therefore fetched kAhead blocks early. With
// 128-wide tiles, four fold warps and the scales loaded where they are used the product was 2.0 ms. 4096 x 18432 x 7168 gated + 4096 x
// 7168 x 18432 with their quantisers (one dense feed-forward): 3.16 -> 1.93 ms.
//
// Also here: the dynamic per-token-group activation quantiser (reference fp8.py:354-552).
#include <string.h>

#include "../common/bounded.cuh"
#include "../common/fp8_quant.cuh"
#include "../common/host_utils.h"
#include "../common/ptx.cuh"

namespace b200 {

static constexpr int kFBM = 128, kFBK = 128;  // K block = 128 fp8 = 128 B
static constexpr int kFEpiWarps = 8;
static constexpr int kFThreads = (4 + kFEpiWarps) * 32;   // one warpgroup for copies and products, two that fold
// Registers per thread after the split: the fold keeps 128 sums and 64 columns on their way from TMEM. 128 x 56 + 256 x 224 is
// exactly what 384 threads are launched with (168 each).
static constexpr int kFRegsIssue = 56, kFRegsFold = 224;
static constexpr int kAhead = 4;              // K blocks that the scales are fetched ahead of their use

struct Fp8Params {
  int M, N, K;
  __nv_bfloat16* C;
  int64_t ldc;
  const float* a_s;  // [K/128, M]
  int lda_s;         // = M (row pitch of a_s)
  const float* w_s;  // [N/128, K/128]  (grouped: [E][N/64][K/128], one scale row per 64 weight rows)
  const __nv_bfloat16* bias;
  // grouped (MoE) mode: M tile t multiplies the e4m3 slab of expert tile_expert[t]; the weight scales are
  // stored per 64-row half tile so a [64 gate | 64 up] interleaved tile can carry two different block scales
  const int32_t* tile_expert;
  const int32_t* num_m_tiles_ptr;
  int n_per_expert;      // rows of one expert slab
  int64_t ws_stride_e;   // floats per expert in w_s
  int silu;              // 1: out[:, j] = silu(gate[j]) * up[j]; the tile holds [64 gate | 64 up] boxes in turn
  WaitConfig waits;
  int up_row;            // > 0 (with silu): the weight is [gate rows ; up rows], up rows start here; the boxes are fetched
                         // from the two halves. 0: the rows are interleaved per 64 already
};

// d = a * b + d on two fp32 at once (one issue slot)
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return make_float2(__uint_as_float(lo), __uint_as_float(hi));
}

template <int BN>
struct Fp8Tile {
  static constexpr int kABytes = kFBM * kFBK, kBBytes = BN * kFBK, kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = BN == 256 ? 4 : BN == 128 ? 6 : 8;
  static constexpr int kBoxes = BN / 64;                 // TMA boxes of 64 weight rows, one weight scale each
  static constexpr int kCols = BN / 2;                   // columns of one epilogue warp
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
  // an epilogue warp of half h owns two runs of kCols / 2 columns; in gated mode the first are gates, the second their ups
  __device__ static int lo(int h) { return BN == 256 ? 128 * h : 32 * h; }
  __device__ static int hi(int h) { return BN == 256 ? 128 * h + 64 : BN == 128 ? 64 + 32 * h : 32 * h + 16; }
};

template <int BN>
__global__ void __launch_bounds__(kFThreads, 1)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const Fp8Params p) {
  using T = Fp8Tile<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + T::kStages * T::kStageBytes);
  uint64_t* empty_bar = full_bar + T::kStages;
  uint64_t* tmem_full = empty_bar + T::kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* mma_end = tmem_empty + 2;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(mma_end + 1);
  const WaitGuard guard{tmem_ptr_smem + 1, p.waits};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool grouped = p.tile_expert != nullptr;
  const int num_kb = p.K / kFBK;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int i = 0; i < T::kStages; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tmem_full[i], 1); mbar_init(&tmem_empty[i], kFEpiWarps); }
    mbar_init(mma_end, 1);
    *guard.dead = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc<1>(tmem_ptr_smem, 2 * BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  griddep_launch();
  griddep_wait();
  const int num_m = p.num_m_tiles_ptr != nullptr ? min(*p.num_m_tiles_ptr, (p.M + kFBM - 1) / kFBM)
                                                 : (p.M + kFBM - 1) / kFBM;
  const int num_n = (p.N + BN - 1) / BN;
  const int num_tiles = num_m * num_n;
  // weight row of box j of the tile that starts at column n0
  auto box_row = [&](int n0, int j) {
    return p.up_row > 0 ? (j & 1 ? p.up_row : 0) + n0 / 2 + (j >> 1) * 64 : n0 + j * 64;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFRegsIssue));
    if (warp == 0 && lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const int m0 = (tile % num_m) * kFBM, n0 = (tile / num_m) * BN;
        const int b_row_off = grouped ? p.tile_expert[tile % num_m] * p.n_per_expert : 0;
        for (int kb = 0; kb < num_kb && ok; ++kb, ++it) {
          const int s = it % T::kStages;
          if (!guard.wait(&empty_bar[s], ((it / T::kStages) & 1) ^ 1)) { ok = false; break; }
          uint8_t* sa = smem + s * T::kStageBytes;
          mbar_expect_tx(&full_bar[s], T::kStageBytes);
          tma_load_2d(sa, &tmap_a, &full_bar[s], kb * kFBK, m0, kEvictNormal);
#pragma unroll
          for (int j = 0; j < T::kBoxes; ++j)
            tma_load_2d(sa + T::kABytes + j * 64 * kFBK, &tmap_b, &full_bar[s], kb * kFBK, b_row_off + box_row(n0, j),
                        kEvictNormal);
        }
      }
      // copies in flight land before the CTA ends, whichever role gave up
      for (uint32_t i = it > T::kStages ? it - T::kStages : 0; i < it; ++i)
        guard.land(&full_bar[i % T::kStages], (i / T::kStages) & 1);
    }
    if (warp == 1 && lane == 0) {
      constexpr uint32_t idesc = make_idesc_e4m3(kFBM, BN);
      uint32_t it = 0;  // global k-block counter == TMEM hand-off counter
      bool ok = guard.first(&full_bar[0]);
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % T::kStages;
          const uint32_t buf = it & 1;
          ok = guard.wait(&tmem_empty[buf], ((it >> 1) & 1) ^ 1) && guard.wait(&full_bar[s], (it / T::kStages) & 1);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * T::kStageBytes);
          const uint64_t da = make_sw128_kmajor_desc(a_addr);
          const uint64_t db = make_sw128_kmajor_desc(a_addr + T::kABytes);
          const uint32_t d_tmem = tmem_base + buf * BN;
#pragma unroll
          for (int k = 0; k < kFBK / 32; ++k)  // UMMA K = 32 for 8-bit operands: +32 B per step
            umma_f8(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, k > 0 ? 1u : 0u);
          umma_commit(&empty_bar[s]);
          umma_commit(&tmem_full[buf]);
        }
      }
      umma_commit(mma_end);                               // nothing is in flight when the columns are given back
      guard.land(mma_end, 0);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFRegsFold));
    const int q = warp & 3, h = (warp - 4) >> 2;
    constexpr int kHalf = T::kCols / 2;                   // columns of one run
    constexpr int kLd = 16;                               // columns of one TMEM load (32 at a time: 1390 us in the short loop)
    const int c_lo = T::lo(h), c_hi = T::hi(h);
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      const int m0 = (tile % num_m) * kFBM, n0 = (tile / num_m) * BN;
      const int row = m0 + q * 32 + lane;
      const bool row_ok = row < p.M;
      // the scale rows of the two runs; a tile past the last column reads the last row instead
      const int r_lo = min(box_row(n0, c_lo / 64), p.N - 1), r_hi = min(box_row(n0, c_hi / 64), p.N - 1);
      const float* ws_lo;
      const float* ws_hi;
      if (grouped) {
        const float* ws = p.w_s + static_cast<size_t>(p.tile_expert[tile % num_m]) * p.ws_stride_e;
        ws_lo = ws + static_cast<size_t>(r_lo / 64) * num_kb;
        ws_hi = ws + static_cast<size_t>(r_hi / 64) * num_kb;
      } else {
        ws_lo = p.w_s + static_cast<size_t>(r_lo / 128) * num_kb;
        ws_hi = p.w_s + static_cast<size_t>(r_hi / 128) * num_kb;
      }
      const float* as = p.a_s + (row_ok ? row : 0);
      float sa[kAhead], sl[kAhead], sh[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int kb = min(i, num_kb - 1);
        sa[i] = as[static_cast<size_t>(kb) * p.lda_s];
        sl[i] = ws_lo[kb];
        sh[i] = ws_hi[kb];
      }
      uint64_t acc[kHalf];                                // [0, kHalf / 2): first run in pairs, then the second run
#pragma unroll
      for (int i = 0; i < kHalf; ++i) acc[i] = 0;
      for (int kb0 = 0; kb0 < num_kb && ok; kb0 += kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int kb = kb0 + i;
          if (kb < num_kb && ok) {
            const uint32_t buf = it & 1;
            const uint32_t wl = __float_as_uint(sa[i] * sl[i]), wh = __float_as_uint(sa[i] * sh[i]);
            const uint64_t w_lo = pack2(wl, wl), w_hi = pack2(wh, wh);
            const int next = min(kb + kAhead, num_kb - 1);
            sa[i] = as[static_cast<size_t>(next) * p.lda_s];
            sl[i] = ws_lo[next];
            sh[i] = ws_hi[next];
            ok = __all_sync(0xffffffffu, guard.wait(&tmem_full[buf], (it >> 1) & 1));
            tc_fence_after();
            const uint32_t t_row = tmem_base + buf * BN + (static_cast<uint32_t>(q * 32) << 16);
            // two loads on their way at a time; the next two are issued as their registers become free
            uint32_t v[2][kLd];
            tmem_ld_32x16(t_row + c_lo, v[0]);
            tmem_ld_32x16(t_row + (kLd < kHalf ? c_lo + kLd : c_hi), v[1]);
#pragma unroll
            for (int c = 0; c < T::kCols; c += kLd) {
              constexpr int kRuns = kHalf / kLd;
              const int n = c / kLd;
              if ((n & 1) == 0) tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < kLd / 2; ++j)
                fma2(acc[c / 2 + j], pack2(v[n & 1][2 * j], v[n & 1][2 * j + 1]), n < kRuns ? w_lo : w_hi);
              if (n + 2 < 2 * kRuns)
                tmem_ld_32x16(t_row + (n + 2 < kRuns ? c_lo + (n + 2) * kLd : c_hi + (n + 2 - kRuns) * kLd), v[n & 1]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
            ++it;
          }
        }
      }
      __nv_bfloat16* crow = p.C + static_cast<size_t>(row) * p.ldc;
      auto store8 = [&](int col, const float (&f)[8]) {
        st_v4(crow + col, make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                                     pack_bf16(f[6], f[7])));
      };
      if (row_ok && ok && p.silu) {
#pragma unroll
        for (int c = 0; c < kHalf; c += 8) {
          const int col = n0 / 2 + c_lo / (BN == 256 ? 2 : 1) + c;
          if (col < p.N / 2) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 gv = unpack2(acc[c / 2 + e]), uv = unpack2(acc[kHalf / 2 + c / 2 + e]);
              f[2 * e] = gv.x / (1.0f + __expf(-gv.x)) * uv.x;
              f[2 * e + 1] = gv.y / (1.0f + __expf(-gv.y)) * uv.y;
            }
            store8(col, f);
          }
        }
      } else if (row_ok && ok) {
#pragma unroll
        for (int c = 0; c < T::kCols; c += 8) {
          const int col = n0 + (c < kHalf ? c_lo + c : c_hi + c - kHalf);
          if (col < p.N) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 x = unpack2(acc[c / 2 + e]);
              f[2 * e] = x.x;
              f[2 * e + 1] = x.y;
            }
            if (p.bias != nullptr) {
              const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + col);
              const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 b = unpack_bf16(bw[e]);
                f[2 * e] += b.x;
                f[2 * e + 1] += b.y;
              }
            }
            store8(col, f);
          }
        }
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 2 * BN);
  }
}

// dynamic per-token-group quantisation: x bf16 [M, K] -> q e4m3 [M, K], scales fp32 [K/128, M]. Memory-bound. A block takes
// 8 rows x 8 groups: 16 lanes of 16 bytes per group, four groups per lane group in flight, and the eight rows of a group put
// their scales side by side (one 32-byte sector). `wide` = 0: rows on 8-byte boundaries only. `live_tiles` (null: all): only the first 128 * *live_tiles rows exist.
// 4096 x 18432: 47 us (2.4 TB/s read), one warp per group of 128 with 8-byte loads took 84.
__global__ void __launch_bounds__(256)
fp8_quant_group_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, __nv_fp8_e4m3* __restrict__ q,
                       float* __restrict__ scales, int M, int K, const int32_t* __restrict__ live_tiles,
                       int wide) {
  griddep_launch();
  griddep_wait();
  const int rows = live_tiles != nullptr ? min(M, *live_tiles * kFBM) : M;
  const int groups = K / 128, lane = threadIdx.x & 15;
  // one grid axis: the second one ends at 65,535 blocks, 524,280 rows
  const int across = (groups + 7) / 8, row0 = static_cast<int>(blockIdx.x / across) * 8, g0 = static_cast<int>(blockIdx.x % across) * 8;
  if (row0 >= rows) return;
  uint4 raw[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int pair = n * 16 + (threadIdx.x >> 4), row = row0 + (pair & 7), g = g0 + (pair >> 3);
    raw[n] = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows && g < groups) {
      const __nv_bfloat16* src = x + static_cast<size_t>(row) * ldx + g * 128 + lane * 8;
      if (wide) {
        raw[n] = ld_nc_v4(src);
      } else {
        const uint2 a = *reinterpret_cast<const uint2*>(src), b = *reinterpret_cast<const uint2*>(src + 4);
        raw[n] = make_uint4(a.x, a.y, b.x, b.y);
      }
    }
  }
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int pair = n * 16 + (threadIdx.x >> 4), row = row0 + (pair & 7), g = g0 + (pair >> 3);
    float scale;
    const uint2 o8 = fp8_quant_lane(raw[n], scale);
    if (row >= rows || g >= groups) continue;
    *reinterpret_cast<uint2*>(q + static_cast<size_t>(row) * K + g * 128 + lane * 8) = o8;
    if (lane == 0) scales[static_cast<size_t>(g) * M + row] = scale;
  }
}

template <int BN>
static int launch_fp8_tile(const CUtensorMap& ta, const CUtensorMap& tb, const Fp8Params& p, int64_t tiles, cudaStream_t st) {
  static PerDeviceOnce configured;
  if (configured.need()) {
    CUDA_CHECK_RET(cudaFuncSetAttribute(gemm_fp8_block_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        Fp8Tile<BN>::kSmem));
    configured.done();
  }
  const int grid = static_cast<int>(tiles < num_sms() ? tiles : num_sms());
  CUDA_CHECK_RET(launch_pdl(gemm_fp8_block_kernel<BN>, dim3(grid), dim3(kFThreads), Fp8Tile<BN>::kSmem, st, ta, tb, p));
  return 0;
}

// Tile width: the one with the least (waves x time of a tile's K block). A block of 128 rows takes 0.60 us 256 wide, 0.48 at 128
// and 0.43 at 64 (there the chain of copies, products and folds bounds it), so narrow tiles only pay when the wide ones leave SMs
// idle: a decode batch's 7168 columns are 28 tiles of 256. Over 80 shapes (1 to 1000 rows, 1536 to 36,864 columns, K 1536 to
// 18,432) timed at all three widths the choice is 0.3 % slower than the best on average. One to four rows of 7168 columns alone
// take 70 us 64 wide and 66.5 at 128 (K = 18432), but the whole MLP of one row 124.2 against 125.2. `live`: the most row tiles that can hold rows; grouped calls
// (256 or 128 wide) do not know more on the host.
static int launch_fp8(const void* A8, const void* W8, uint64_t w_rows, Fp8Params p, int64_t live, cudaStream_t st) {
  const int64_t m_tiles = (p.M + kFBM - 1) / kFBM;
  const int width[3] = {256, 128, 64}, cost[3] = {600, 480, 430};
  int bn = 256;
  int64_t best = -1;
  for (int i = 0; i < (p.silu || p.tile_expert != nullptr ? 2 : 3); ++i) {
    const int64_t tiles = live * ((p.N + width[i] - 1) / width[i]);
    const int64_t t = (tiles + num_sms() - 1) / num_sms() * cost[i];
    if (best < 0 || t < best) { best = t; bn = width[i]; }
  }
  p.waits = g_wait_config;
  CUtensorMap ta, tb;
  if (make_tmap_2d(&ta, A8, p.M, p.K, p.K, kFBM, kFBK, CU_TENSOR_MAP_DATA_TYPE_UINT8)) return 1;
  if (make_tmap_2d(&tb, W8, w_rows, p.K, p.K, 64, kFBK, CU_TENSOR_MAP_DATA_TYPE_UINT8)) return 1;
  const int64_t tiles = m_tiles * ((p.N + bn - 1) / bn);
  return bn == 256 ? launch_fp8_tile<256>(ta, tb, p, tiles, st)
         : bn == 128 ? launch_fp8_tile<128>(ta, tb, p, tiles, st) : launch_fp8_tile<64>(ta, tb, p, tiles, st);
}

}  // namespace b200

using namespace b200;

// live_tiles: device count of the 128-row tiles that exist (null: all M rows)
GLLM_EXPORT int gllm_fp8_quant_group(const void* x, int64_t ldx, void* q, void* scales, int M, int K, const void* live_tiles,
                                     void* stream) {
  if (M <= 0) return 0;
  if (K % 128 != 0) return 1;
  CUDA_CHECK_RET(launch_pdl(fp8_quant_group_kernel, dim3(static_cast<unsigned>((K / 128 + 7) / 8) * ((M + 7) / 8)), dim3(256), 0,
                            reinterpret_cast<cudaStream_t>(stream), reinterpret_cast<const __nv_bfloat16*>(x), ldx,
                            reinterpret_cast<__nv_fp8_e4m3*>(q), reinterpret_cast<float*>(scales), M, K,
                            reinterpret_cast<const int32_t*>(live_tiles),
                            static_cast<int>(ldx % 8 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0)));
  return 0;
}

// A8 [M,K] e4m3 contiguous, a_s [K/128, M]; W8 [N,K] e4m3 contiguous, w_s [ceil(N/128), K/128]. silu: the weight is
// [N/2 gate rows ; N/2 up rows] (N/2 a multiple of 128) and C [M, N/2] = silu(gate) * up.
GLLM_EXPORT int gllm_gemm_fp8_block(const void* A8, const void* a_s, const void* W8, const void* w_s, void* C,
                                    int64_t ldc, int M, int N, int K, const void* bias, int silu, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 128 != 0 || N % 8 != 0 || (silu && (N % 256 != 0 || bias != nullptr))) {
    fprintf(stderr, "[gllm_b200] gemm_fp8_block: K %% 128 and N %% 8 required (gated: N %% 256, no bias)\n");
    return 1;
  }
  if (ldc % 8 != 0 || ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(bias)) & 15) != 0) {
    fprintf(stderr, "[gllm_b200] gemm_fp8_block: output rows and bias must lie on 16-byte boundaries\n");
    return 1;
  }
  Fp8Params p;
  p.M = M; p.N = N; p.K = K;
  p.C = reinterpret_cast<__nv_bfloat16*>(C);
  p.ldc = ldc;
  p.a_s = reinterpret_cast<const float*>(a_s);
  p.lda_s = M;
  p.w_s = reinterpret_cast<const float*>(w_s);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.tile_expert = nullptr; p.num_m_tiles_ptr = nullptr; p.n_per_expert = 0; p.ws_stride_e = 0;
  p.silu = silu ? 1 : 0;
  p.up_row = silu ? N / 2 : 0;
  return launch_fp8(A8, W8, N, p, (M + kFBM - 1) / kFBM, reinterpret_cast<cudaStream_t>(stream));
}

// Grouped (MoE) block-scaled fp8 GEMM: A8 [max_tiles*128, K] e4m3 (expert-sorted, 128-row tiles), a_s
// [K/128, max_tiles*128]; W8 [E, N, K] e4m3, w_s [E, N/64, K/128] (one scale row per 64 weight rows);
// epi 1 = SiLU gate on [64 gate | 64 up] interleaved tiles -> C [rows, N/2]. At most max_live of the max_tiles tiles hold rows.
GLLM_EXPORT int gllm_moe_grouped_gemm_fp8(const void* A8, const void* a_s, const void* W8, const void* w_s, void* C,
                                          int64_t ldc, int max_tiles, int max_live, int N, int K, int E,
                                          const void* tile_expert, const void* num_tiles_ptr, int epi, void* stream) {
  if (max_tiles <= 0) return 0;
  if (K % 128 != 0 || N % 128 != 0) {
    fprintf(stderr, "[gllm_b200] moe_grouped_gemm_fp8: K %% 128 and N %% 128 required\n");
    return 1;
  }
  Fp8Params p;
  p.M = max_tiles * kFBM; p.N = N; p.K = K;
  p.C = reinterpret_cast<__nv_bfloat16*>(C);
  p.ldc = ldc;
  p.a_s = reinterpret_cast<const float*>(a_s);
  p.lda_s = p.M;
  p.w_s = reinterpret_cast<const float*>(w_s);
  p.bias = nullptr;
  p.tile_expert = reinterpret_cast<const int32_t*>(tile_expert);
  p.num_m_tiles_ptr = reinterpret_cast<const int32_t*>(num_tiles_ptr);
  p.n_per_expert = N;
  p.ws_stride_e = static_cast<int64_t>(N / 64) * (K / 128);
  p.silu = epi == 1 ? 1 : 0;
  p.up_row = 0;
  return launch_fp8(A8, W8, static_cast<uint64_t>(E) * N, p, max_live < max_tiles ? max_live : max_tiles,
                    reinterpret_cast<cudaStream_t>(stream));
}
