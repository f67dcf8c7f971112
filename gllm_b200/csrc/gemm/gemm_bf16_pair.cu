// bf16 GEMM on pairs of SMs (sm_100a):  C[M, N] = A[M, K] · W[N, K]^T (+ bias), the same products, sums and epilogues as
// gemm_bf16.cu, for prefill-sized M on one GPU (the fused collectives, expert tiles and K splits stay there).
//
// Two CTAs of a cluster share one output tile of 256 x 256: each stages its own 128 rows of A and its own half of the
// 256 weight rows, and one tcgen05.mma.cta_group::2 (256 x 256 x 16) reads both halves and leaves 128 rows of sums in each CTA's
// TMEM. So an SM copies 32 KB per 64-deep K block of a 256-wide tile instead of 48 KB and its tensor core reads 32 KB instead of
// 48 KB.
//
// What bounds it: the tensor cores at the power limit (1.5 to 1.58 PFLOP/s in long products, 1.40 PFLOP/s sustained is what the
// library reaches over seconds); in short ones the copies: a K block takes some 700 cycles instead of 512. Equal shares of the K
// blocks instead of whole tiles (parts of tiles summed through L2) gained nothing: the power limit evens a partly filled last
// round out, and pairs that walk K out of step no longer share their reads of L2. 8192 x 16384 x 4096: 716 us, on single SMs 808;
// 4096 x 6144 x 4096: 141 / 151; 8192 x 8192 x 256: 50 / 82 (with four warps to drain TMEM 58).
//
// Roles per CTA: warp 0 copies (both CTAs; every byte is counted by the leader's barrier of the stage), warp 1 issues products
// (leader only) and commits to both CTAs' barriers, warps 2-9 drain TMEM (each CTA its own rows). Sums are double buffered: the
// epilogue of a tile overlaps the products of the next.
#include <string.h>

#include "../common/bounded.cuh"
#include "../common/host_utils.h"
#include "../common/ptx.cuh"
#include "gemm_pair.h"

namespace b200 {

namespace {

constexpr int kPBK = 64;             // 64 bf16 = 128 B = one swizzle atom row
constexpr int kPEpi = 8;             // warps that drain TMEM
constexpr int kPThreads = (2 + kPEpi) * 32;
constexpr int kPBN = 256;            // columns of a tile (192: the same time per tile, 128: 1.6 times the time per column)
constexpr int kPStages = 6;
constexpr int kPABytes = 128 * kPBK * 2, kPStage = kPABytes + kPBN / 2 * kPBK * 2;
constexpr int kPSmem = kPStages * kPStage + 1024 + 256 + kPEpi * 4096;

struct PairParams {
  PairGemm g;
  WaitConfig waits;
  int num_m, num_n;                  // tiles down, across
};

// tile t -> (tile down, tile across): sweeps of eight tiles down, so that the 74 tiles worked on at one time share rows of A and W
// (8192 x 10240 x 8192: 913 us; sweeps of 2, 4, 16 tiles 1003, 942, 940)
constexpr int kSweep = 8;
__device__ __forceinline__ void tile_at(const PairParams& p, int t, int& mt, int& nt) {
  const int per = kSweep * p.num_n, sweep = t / per, r = t - sweep * per;
  const int rows = min(kSweep, p.num_m - sweep * kSweep);
  nt = r / rows;
  mt = sweep * kSweep + r - nt * rows;
}

template <bool GATED>
__global__ void __launch_bounds__(kPThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const PairParams p) {
  constexpr int BN = kPBN, S = kPStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S * kPStage);
  uint64_t* empty_bar = full_bar + S;
  uint64_t* tmem_full = empty_bar + S;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* mma_end = tmem_empty + 2;
  uint64_t* peer_end = mma_end + 1;                      // leader: the other CTA issues no more copies; how many stages it filled
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(peer_end + 1);
  uint32_t* peer_stages = tmem_ptr_smem + 2;
  const WaitGuard guard{tmem_ptr_smem + 1, p.waits};
  uint8_t* epi_smem = smem + S * kPStage + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int M = p.g.M, N = p.g.N;
  const int num_kb = (p.g.K + kPBK - 1) / kPBK;
  const int num_tiles = p.num_m * p.num_n, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  griddep_launch();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int i = 0; i < S; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tmem_full[i], 1); mbar_init(&tmem_empty[i], 2 * kPEpi); }
    mbar_init(mma_end, 1);
    mbar_init(peer_end, 1);
    *peer_stages = 0;
    *guard.dead = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_ptr_smem, 2 * BN);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                        // both CTAs' barriers are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0, pre = 0;
      bool ok = true;
      int mt, nt;
      // weights do not depend on the kernel before: the first stages' are on their way while it drains
      if (pair < num_tiles) {
        tile_at(p, pair, mt, nt);
        pre = static_cast<uint32_t>(min(S, num_kb));
        for (uint32_t i = 0; i < pre; ++i) {
          if (rank == 0) mbar_expect_tx(&full_bar[i], 2 * kPStage);
          tma_load_2d_pair(smem + i * kPStage + kPABytes, &tmap_b, cluster_addr(&full_bar[i], 0),
                           static_cast<int>(i) * kPBK, nt * BN + static_cast<int>(rank) * (BN / 2), kEvictNormal);
        }
      }
      griddep_wait();
      for (int t = pair; t < num_tiles && ok; t += pairs) {
        tile_at(p, t, mt, nt);
        const int m0 = mt * 256 + static_cast<int>(rank) * 128, n0 = nt * BN + static_cast<int>(rank) * (BN / 2);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % S;
          uint8_t* sa = smem + s * kPStage;
          const uint32_t bar = cluster_addr(&full_bar[s], 0);
          if (it >= pre) {
            if (!guard.wait(&empty_bar[s], ((it / S) & 1) ^ 1)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * kPStage);
            tma_load_2d_pair(sa + kPABytes, &tmap_b, bar, kb * kPBK, n0, kEvictNormal);
          }
          tma_load_2d_pair(sa, &tmap_a, bar, kb * kPBK, m0, kEvictNormal);
        }
      }
      // The commits that hand the last stages back arrive in both CTAs, and the cluster's barrier does not order them: the other
      // CTA sees its own before it ends (the leader's issuer waits for `mma_end`).
      if (rank == 1)
        for (uint32_t i = it > S ? it - S : 0; i < it && ok; ++i) ok = guard.wait(&empty_bar[i % S], (i / S) & 1);
      // Copies in flight land before the CTAs end, whichever role gave up (then the other CTA's waits end too). The leader's barriers
      // count both CTAs' copies, so it has to know how many stages the other one filled: a stage that only the leader filled is not
      // waited for in full, one that only the other CTA filled is counted after all.
      auto warn = [&] {
        if (guard.gave_up()) st_cluster(cluster_addr(const_cast<uint32_t*>(guard.dead), rank ^ 1), 1);
      };
      warn();
      if (rank == 1) {
        st_cluster(cluster_addr(peer_stages, 0), it);
        mbar_arrive_cluster(cluster_addr(peer_end, 0));
      } else {
        const uint32_t t0 = global_ns();
        bool told = mbar_try_wait_cluster(peer_end, 0);
        while (!told && global_ns() - t0 < 4000000000u) {
          warn();
          told = mbar_try_wait_cluster(peer_end, 0);
        }
        const uint32_t other = told ? *reinterpret_cast<volatile uint32_t*>(peer_stages) : it, most = other > it ? other : it;
        for (uint32_t i = other < it ? other : it; i < most; ++i) {
          if (i < it) mbar_complete_tx(&full_bar[i % S], kPStage);
          else mbar_expect_tx(&full_bar[i % S], kPStage);
        }
        for (uint32_t i = most > S ? most - S : 0; i < most; ++i) guard.land(&full_bar[i % S], (i / S) & 1);
      }
    }
  } else if (warp == 1) {
    griddep_wait();                                      // A is copied behind it: the limit of the waits does not count the kernel before
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(256, BN);
      uint32_t it = 0, n = 0;
      bool ok = guard.first(&full_bar[0]);
      for (int t = pair; t < num_tiles && ok; t += pairs, ++n) {
        const uint32_t buf = n & 1;
        ok = guard.wait(&tmem_empty[buf], ((n >> 1) & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % S;
          if (!guard.wait(&full_bar[s], (it / S) & 1)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * kPStage);
          const uint64_t da = make_sw128_kmajor_desc(a_addr), db = make_sw128_kmajor_desc(a_addr + kPABytes);
#pragma unroll
          for (int k = 0; k < kPBK / 16; ++k)
            umma_bf16_pair(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s]);
        }
        if (ok) umma_commit_pair(&tmem_full[buf]);
      }
      umma_commit_pair(mma_end);                         // nothing is in flight when the columns are given back
      guard.land(mma_end, 0);
    }
  } else {
    griddep_wait();
    const int q = warp & 3, half = (warp - 2) >> 2;      // TMEM lane quarter and half of the columns of this warp
    uint8_t* stg = epi_smem + (warp - 2) * 4096;
    constexpr int OUT = GATED ? BN / 2 : BN;             // output columns of a tile
    const int out_N = GATED ? N / 2 : N;
    uint32_t n = 0;
    bool ok = true;
    for (int t = pair; t < num_tiles && ok; t += pairs, ++n) {
      int mt, nt;
      tile_at(p, t, mt, nt);
      const int row0 = mt * 256 + static_cast<int>(rank) * 128 + q * 32, col0 = nt * OUT;
      const uint32_t buf = n & 1;
      ok = __all_sync(0xffffffffu, guard.wait(&tmem_full[buf], (n >> 1) & 1));
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + buf * BN + (static_cast<uint32_t>(q * 32) << 16);
      auto give_back = [&] {                             // the sums are read: the products may have the buffer
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(&tmem_empty[buf], 0));
      };
      if (row0 >= M) {
        give_back();
        continue;
      }
      // 32 rows x 64 columns at a time through shared memory, so that every store instruction writes whole 128-byte rows
      auto put = [&](int ch, const float (&f)[8]) {      // eight columns of this lane's row
        *reinterpret_cast<uint4*>(stg + lane * 128 + ((ch ^ (lane & 7)) * 16)) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
      };
#pragma unroll 1
      for (int c = half * (OUT / 2); c < (half + 1) * (OUT / 2); c += 64) {
        if constexpr (!GATED) {
          uint32_t v[2][32];
          tmem_ld_32x32(t_row + c, v[0]);
          tmem_ld_32x32(t_row + c + 32, v[1]);
          tmem_ld_wait();
          if (c + 64 >= (half + 1) * (OUT / 2)) give_back();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              const int col = col0 + c + h * 32 + j;
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[h][j + e]);
              if (p.g.bias != nullptr && col < out_N) {
                const uint4 bv = *reinterpret_cast<const uint4*>(p.g.bias + col);
                const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 b = unpack_bf16(bw[e]);
                  f[2 * e] += b.x;
                  f[2 * e + 1] += b.y;
                }
              }
              put(h * 4 + j / 8, f);
            }
          }
        } else {
#pragma unroll
          for (int h = 0; h < 64; h += 32) {
            uint32_t g[32], u[32];
            tmem_ld_32x32(t_row + c + h, g);
            tmem_ld_32x32(t_row + BN / 2 + c + h, u);
            tmem_ld_wait();
            if (c + h + 32 >= (half + 1) * (OUT / 2)) give_back();
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const float gv = __uint_as_float(g[j + e]), uv = __uint_as_float(u[j + e]);
                if (p.g.glu_limit > 0.f) {
                  const float gc = fminf(gv, p.g.glu_limit), uc = fminf(fmaxf(uv, -p.g.glu_limit), p.g.glu_limit);
                  f[e] = gc / (1.0f + __expf(-p.g.glu_alpha * gc)) * (uc + 1.0f);
                } else if (p.g.gelu) {
                  f[e] = gelu_tanh_fast(gv) * uv;
                } else {
                  f[e] = gv / (1.0f + __expf(-gv)) * uv;
                }
              }
              put((h + j) / 8, f);
            }
          }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3), ch = lane & 7, col = col0 + c + ch * 8;
          const uint4 o = *reinterpret_cast<const uint4*>(stg + r * 128 + ((ch ^ (r & 7)) * 16));
          if (row0 + r < M && col < out_N) st_v4(p.g.C + static_cast<size_t>(row0 + r) * p.g.ldc + col, o);
        }
        __syncwarp();
      }
    }
    // the very last commit as well
    if (rank == 1 && warp == 2 && lane == 0) WaitGuard::land(mma_end, 0);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                        // the other CTA's shared memory and barriers are in use until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * BN);
  }
}

template <bool GATED>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, PairParams p, cudaStream_t st) {
  auto kern = gemm_bf16_pair_kernel<GATED>;
  static PerDeviceOnce configured;
  if (configured.need()) {
    CUDA_CHECK_RET(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPSmem));
    configured.done();
  }
  p.num_m = (p.g.M + 255) / 256;
  p.num_n = (p.g.N + kPBN - 1) / kPBN;
  const int tiles = p.num_m * p.num_n, all = num_sms() / 2;
  CUDA_CHECK_RET(launch_pdl_cluster(kern, dim3(2 * (tiles < all ? tiles : all)), 2, dim3(kPThreads), kPSmem, st, ta, tb, p));
  return 0;
}

}  // namespace

int gemm_bf16_pair(const PairGemm& g, cudaStream_t st) {
  PairParams p;
  p.g = g;
  p.waits = g_wait_config;
  CUtensorMap ta, tb;
  if (make_tmap_2d(&ta, g.A, g.M, g.K, g.lda * 2, 128, kPBK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16)) return 1;
  if (make_tmap_2d(&tb, g.W, g.N, g.K, g.ldw * 2, kPBN / 2, kPBK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16)) return 1;
  return g.gated ? launch_pair<true>(ta, tb, p, st) : launch_pair<false>(ta, tb, p, st);
}

}  // namespace b200
