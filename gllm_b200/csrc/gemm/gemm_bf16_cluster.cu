// bf16 GEMM of a decode batch (a few to some hundred rows) for sm_100a:  C[M, N] = A[M, K] · W[N, K]^T (+ bias), optionally gated.
//
// The weights are the traffic, and N / 128 tiles of them are too few to draw it with all SMs, so K is cut over the CTAs of a cluster.
// A CTA multiplies 128 weight rows (the M operand) by all rows of A of its tile (the N operand, up to 256) over its part of K; the parts of a
// tile are exchanged through distributed shared memory, not through L2: each CTA of the cluster reads the sums of some rows of A from
// all others, adds them in order of K, and writes those rows.
//
// What bounds it: the weight bytes where there are many (64 rows, 4096 x 12,288: 21 us, 4.8 TB/s), else a chain of some 6 us: the
// first copy behind the kernel before 0.7, the last product 0.3, sums to shared memory 0.4, the cluster's barrier 0.6, reading the others'
// sums 1 to 2, stores 0.5. An SM copies at most some 60 bytes per cycle, so tiles are as tall as the batch, and where two CTAs fit an
// SM one's chain hides behind the other's copies (64 rows, 4096 x 12,288: 24 us with one CTA per SM). Pushing the sums to their
// CTAs took 3.2 us for 128 rows (and a barrier before it, because they land where the ring was); being read they take 2.1.
//
// Roles: warp 0 copies, warp 1 issues the products, warps 2-9 bring the sums from TMEM to shared memory; all add.
#include <mutex>

#include "../common/bounded.cuh"
#include "../common/host_utils.h"
#include "../common/ptx.cuh"
#include "gemm_cluster.h"

namespace b200 {

namespace {

constexpr int kCW = 128, kCK = 64;                       // weight rows of a tile, depth of a K block (128 bytes)
constexpr int kCEpi = 8, kCThreads = (2 + kCEpi) * 32;

struct ClusterParams {
  ClusterGemm g;
  WaitConfig waits;
  int bt, tiles_n, stages;                               // rows of A per tile (a multiple of 16), tiles across N, stages of the ring
  uint32_t tmem_cols;
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

template <int N>
struct Most {
  static constexpr int value = N;
};

template <bool GATED>
__global__ void __launch_bounds__(kCThreads, 2)
gemm_bf16_cluster_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const ClusterParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // barriers first: what follows is the ring, and the sums where the ring has been
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty_bar = full_bar + kClusterStages;
  uint64_t* done = empty_bar + kClusterStages;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(done + 1);
  const WaitGuard guard{tmem_ptr_smem + 1, p.waits};
  uint8_t* ring = smem + 1024;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.stages, BT = p.bt, stage_bytes = kCW * kCK * 2 + BT * kCK * 2;
  const uint32_t C = cluster_size(), rank = cluster_ctarank();
  const int tile = blockIdx.x / C, tn = tile % p.tiles_n, m0 = tile / p.tiles_n * BT;
  const int num_kb = (p.g.K + kCK - 1) / kCK;
  const int kb0 = num_kb * static_cast<int>(rank) / static_cast<int>(C), kb1 = num_kb * (static_cast<int>(rank) + 1) / static_cast<int>(C);

  griddep_launch();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int i = 0; i < S; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    mbar_init(done, 1);
    *guard.dead = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc<1>(tmem_ptr_smem, p.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr_smem;

  if (warp == 0) {
    if (lane == 0) {
      auto load_w = [&](int i, int kb) {
        uint8_t* dst = ring + i * stage_bytes;
        if constexpr (GATED) {                           // 64 gate rows, then their up rows; blocks of 128 alternate in the weight
          const int f = tn * 64, row = f / 128 * 256 + f % 128;
          tma_load_2d(dst, &tmap_w, &full_bar[i], kb * kCK, row, kEvictFirst);
          tma_load_2d(dst + 64 * kCK * 2, &tmap_w, &full_bar[i], kb * kCK, row + 128, kEvictFirst);
        } else {
          tma_load_2d(dst, &tmap_w, &full_bar[i], kb * kCK, tn * kCW, kEvictFirst);
        }
      };
      // weights do not depend on the kernel before: the first stages' are on their way while it drains
      const int n = kb1 - kb0, pre = min(S, n);
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(&full_bar[i], stage_bytes);
        load_w(i, kb0 + i);
      }
      griddep_wait();
      int it = 0;
      for (; it < n; ++it) {
        const int s = it % S;
        if (it >= pre) {
          if (!guard.wait(&empty_bar[s], ((it / S) & 1) ^ 1)) break;
          mbar_expect_tx(&full_bar[s], stage_bytes);
          load_w(s, kb0 + it);
        }
        tma_load_2d(ring + s * stage_bytes + kCW * kCK * 2, &tmap_x, &full_bar[s], (kb0 + it) * kCK, m0, kEvictLast);
      }
      // copies in flight land before the sums take their place, whichever role gave up
      for (int i = max(0, it - S); i < it; ++i) guard.land(&full_bar[i % S], (i / S) & 1);
    }
  } else if (warp == 1) {
    griddep_wait();                                      // A is copied behind it: the limit of the waits does not count the kernel before
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(kCW, BT);
      bool ok = guard.first(&full_bar[0]);
      for (int it = 0; it < kb1 - kb0 && ok; ++it) {
        const int s = it % S;
        ok = guard.wait(&full_bar[s], (it / S) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w_addr = smem_u32(ring + s * stage_bytes);
        const uint64_t dw = make_sw128_kmajor_desc(w_addr), dx = make_sw128_kmajor_desc(w_addr + kCW * kCK * 2);
#pragma unroll
        for (int k = 0; k < kCK / 16; ++k)
          umma_bf16<1>(tmem, dw + (uint64_t)(k * 2), dx + (uint64_t)(k * 2), idesc, (it | k) != 0 ? 1u : 0u);
        umma_commit(&empty_bar[s]);
      }
      umma_commit(done);                                 // every product has finished: the ring is free
      guard.land(done, 0);
    }
  } else {
    griddep_wait();
    WaitGuard::land(done, 0);
  }
  // This CTA's copies have landed (warp 0) and its products have finished: the ring holds the part's sums from here, [row of A / 4]
  // [weight row][4].
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp >= 2) {
    const int q = warp & 3, half = (warp - 2) >> 2;      // TMEM lane quarter; every other sixteen rows of A
    float4* to = reinterpret_cast<float4*>(ring) + q * 32 + lane;
    for (int c = half * 16; c < BT; c += 32) {
      uint32_t v[16];
      tmem_ld_32x16(tmem + c + (static_cast<uint32_t>(q * 32) << 16), v);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i)
        to[(c / 4 + i) * kCW] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]),
                                            __uint_as_float(v[4 * i + 3]));
    }
    tc_fence_before();
  }
  __syncwarp();
  cluster_sync();                                        // every part's sums are there
  // CTA r adds the rows of A in fours [fours r / C, fours (r + 1) / C).
  const int fours = BT / 4, my_lo = fours * static_cast<int>(rank) / static_cast<int>(C),
            my_n = fours * (static_cast<int>(rank) + 1) / static_cast<int>(C) - my_lo;
  constexpr int OUT = GATED ? 64 : 128;                  // columns of C of a tile
  const int out_N = GATED ? p.g.N / 2 : p.g.N, col0 = tn * OUT;
  __nv_bfloat16* stg = reinterpret_cast<__nv_bfloat16*>(ring + static_cast<size_t>(BT) * kCW * 4);           // [row][OUT + 8]
  constexpr int LD = OUT + 8;
  // P: at least C. Sixteen loads of a thread are on their way at a time (a remote one takes about 0.8 us); then they are added in order of K.
  auto add = [&](auto most) {
    constexpr int P = decltype(most)::value, U = 16 / P / (GATED ? 2 : 1), V = GATED ? 2 : 1;
    for (int i0 = threadIdx.x; i0 < my_n * OUT; i0 += U * kCThreads) {
      float4 x[U][V][P];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = min(i0 + u * kCThreads, my_n * OUT - 1), f = my_lo + i / OUT, w = i % OUT;
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
          for (int r = 0; r < P; ++r)
            if (r < static_cast<int>(C)) x[u][v][r] = ld_cluster_v4(cluster_addr(ring, r) + (f * kCW + w + v * 64) * 16);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kCThreads, f = i / OUT, w = i % OUT;
        if (i >= my_n * OUT) break;
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
          for (int r = 1; r < P; ++r)
            if (r < static_cast<int>(C)) {
              x[u][v][0].x += x[u][v][r].x; x[u][v][0].y += x[u][v][r].y;
              x[u][v][0].z += x[u][v][r].z; x[u][v][0].w += x[u][v][r].w;
            }
        float y[4] = {x[u][0][0].x, x[u][0][0].y, x[u][0][0].z, x[u][0][0].w};
        if constexpr (GATED) {
          const float up[4] = {x[u][V - 1][0].x, x[u][V - 1][0].y, x[u][V - 1][0].z, x[u][V - 1][0].w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            y[e] = p.g.gelu ? gelu_tanh_fast(y[e]) * up[e] : y[e] / (1.f + __expf(-y[e])) * up[e];
        } else if (p.g.bias != nullptr && col0 + w < out_N) {
          const float b = __bfloat162float(p.g.bias[col0 + w]);
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] += b;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) stg[(f * 4 + e) * LD + w] = __float2bfloat16(y[e]);
      }
    }
  };
  if (C <= 2) add(Most<2>{});
  else if (C <= 4) add(Most<4>{});
  else add(Most<8>{});
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");    // the others' sums have been read
  __syncthreads();
  for (int i = threadIdx.x; i < my_n * 4 * (OUT / 8); i += kCThreads) {
    const int r = i / (OUT / 8), ch = i % (OUT / 8) * 8, m = m0 + my_lo * 4 + r;
    if (m < p.g.M && col0 + ch < out_N)
      st_v4(p.g.C + static_cast<size_t>(m) * p.g.ldc + col0 + ch, *reinterpret_cast<const uint4*>(stg + r * LD + ch));
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, p.tmem_cols);
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // ... and they this CTA's
}

template <bool GATED>
int launch_cluster(const CUtensorMap& tw, const CUtensorMap& tx, const ClusterParams& p, int tiles, int parts, int smem, cudaStream_t st) {
  auto kern = gemm_bf16_cluster_kernel<GATED>;
  static PerDeviceOnce configured;
  if (configured.need()) {
    CUDA_CHECK_RET(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured.done();
  }
  CUDA_CHECK_RET(launch_pdl_cluster(kern, dim3(tiles * parts), parts, dim3(kCThreads), smem, st, tw, tx, p));
  return 0;
}

}  // namespace

namespace {

// shared memory of a CTA that has an SM for itself, and of one of two
constexpr int kAlone = 220 * 1024, kOfTwo = 108 * 1024, kMostOfTwo = 112 * 1024;

int stages_of(int bt, int smem) {
  const int n = (smem - 2048) / ((kCW + bt) * kCK * 2);
  return n > kClusterStages ? kClusterStages : n;
}
// the ring, or the sums and the rounded results that take its place
int smem_of(int bt, int parts, bool gated, int stages) {
  const int ring = stages * (kCW + bt) * kCK * 2, most = (bt / 4 + parts - 1) / parts;
  const int sums = bt * kCW * 4 + most * 4 * ((gated ? 64 : 128) + 8) * 2;
  return (ring > sums ? ring : sums) + 2048;
}

// Clusters that this device runs side by side: [1 or 2 CTAs per SM][CTAs of a cluster]. Asked for with an empty kernel of the same block: for one
// that allocates TMEM the query says one CTA per SM whatever it takes, yet two run there.
__global__ void __launch_bounds__(kCThreads, 2) cluster_slots_kernel() {}

struct Slots {
  bool known = false;
  int n[3][9];
};
const Slots* slots() {                                   // null: not known
  static std::mutex mu;
  static Slots table[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  Slots& s = table[dev];
  if (!s.known) {
    auto kern = cluster_slots_kernel;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return nullptr;
    for (int r = 1; r <= 2; ++r)
      for (int c = 1; c <= 8; ++c) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c * 64);
        cfg.blockDim = dim3(kCThreads);
        cfg.dynamicSmemBytes = r == 1 ? kAlone : kMostOfTwo;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        s.n[r][c] = 0;
        if (cudaOccupancyMaxActiveClusters(&s.n[r][c], kern, &cfg) != cudaSuccess) {
          cudaGetLastError();
          s.n[r][c] = 0;
        }
      }
    s.known = true;
  }
  return &s;                                             // not written again
}

}  // namespace

// The plan with the least modelled time (us): rounds of clusters, each 4.4 + 0.005 per row of A (start, exchange, stores), and the larger
// of what an SM copies (100 KB per us) and what the memory gives. Fitted to some 9000 timings (20 weights of 512 x 4096 to 57,344 x 8192,
// 1 to 512 rows, all plans, weights cold, launched back to back). Of clusters of three or five, fewer run at once than the query says (45
// of three on an SM each: 5760 x 4096, 128 rows 21.5 us, 16.2 with a plan that leaves two of them free; 26 of five: 3328 x 8192, 512 rows
// 40.6 / 31.5); 15 of eight, 33 of four and 22 of six do.
//
// Taken instead of the other kernels: over 3456 plain and 770 gated products (weights drawn between 512 and 24,576 rows and 768 and
// 14,336 columns, 3 to 512 rows of A) one takes 0.80 (gated 0.72) of the time that those took on average; 30 plain ones take 5 % more or
// worse, 1.16 at worst (without the rules (e) to (g) and with the slots as the query says 211, 1.56). Some (rows: weights, before -> now,
// us): 4: 24,576 x 4096 gated 37.9 -> 35.1; 16: 6144 x 4096 14.6 -> 11.8, 1024 x 3072 7.8 -> 5.8; 32: 4096 x 4096 14.2 -> 10.2; 64: 4096
// x 12,288 29 -> 21, 10,240 x 8192 50 -> 31; 128: 2112 x 7168 15.5 -> 13.8; 256: 6144 x 4096 24.3 -> 21.5. Not taken: (a) 592 and more
// tiles across (heads of 151,936 columns): persistent CTAs with one start lose less (16 rows 49 us, here 63). (b) As wide as the machine
// or wider, with more than 64 rows (57,344 x 8192 gated, 128 rows: 165, here 171), or gated tiles of 192 that fit one round, with more
// than 32 (24,576 x 4096, 64 rows: 37.3, here 38.2): nothing to cut, and those tiles read A less often. (c) A few rows on few tiles:
// sixteen parts draw more than eight (768 x 4096, 4 rows 5.7 us, here 6.3). (d) Over 256 rows, except for narrow products with enough K
// (512 rows, 4096 x 4096: 24.2 -> 20.8 taken; 6144 x 4096 31.0, here 32.7). Plain ones where the other tiles fill the machine in one
// round: (e) K is not cut here either, up to 32 rows on nearly as many tiles as SMs (16,896 x 832, 32 rows 8.8, here 10.3), or rows that
// nearly fill tiles of 128 (12,736 x 1856, 128 rows 14.0, here 16.7), or with more than 216 rows more than one round of a short K (10,432
// x 2496, 256 rows 17, here 21; 9664 x 9472 64.7 and 55.7); (f) K in four parts there (4608 x 2368, 128 rows 11.5, here 12.6; 3072 x
// 8192, 384 rows 25, here 30; with K below 4480 15.9 and 15.3); (g) a short K (11,008 x 960, 128 rows 9.7, here 11.3).
static bool others_are_faster(int M, int N, int K, int bn, int split, const ClusterPlan& plan, int rounds) {
  const int tiles_n = (N + kCW - 1) / kCW, sms = num_sms(), num_kb = (K + kCK - 1) / kCK, rows = (M + 127) / 128, spare = rows * 128 - M;
  if (M <= 32) return plan.parts == 1 && tiles_n <= sms && tiles_n * 8 > sms * 7;
  if (M <= 256 && ((plan.parts == 1 && M > 48 && spare <= 48) || (rounds > 1 && M > 216 && num_kb <= 48))) return true;
  if (bn == 0) return false;
  const int units = rows * ((N + bn - 1) / bn) * split;
  if (units > sms) return false;
  if (split == 4 && units * 8 > sms * 7) return M <= 256 ? bn == 128 && spare <= 16 : num_kb >= 70 && plan.parts <= 3;
  return split == 1 && M <= 256 && spare <= 16 && num_kb <= 24 && plan.parts <= 3 && units * 2 > sms - 8;
}

bool plan_gemm_cluster(int M, int N, int K, bool gated, int bn, int split, ClusterPlan* plan) {
  const int tiles_n = (N + kCW - 1) / kCW, sms = num_sms(), num_kb = (K + kCK - 1) / kCK;
  if (M > 512 || tiles_n >= 4 * sms) return false;
  if (M > 256 && (gated || N < 2560 || N > 4096 || K < 1536)) return false;
  if (tiles_n * 8 < sms && (M <= 4 || (M <= 8 && K >= 6144))) return false;
  if (tiles_n >= sms && M > 32 && (M > 64 || (gated && (N + 191) / 192 <= sms))) return false;
  const Slots* side_by_side = slots();
  if (side_by_side == nullptr) return false;
  double best = 1e30;
  int best_rounds = 0;
  for (int tm = 1; tm <= 4; ++tm) {
    const int bt = ((M + tm - 1) / tm + 15) / 16 * 16;
    if (bt > 256) continue;
    if (tm > 1 && (bt < 32 || (tm > 2 && tm > (M + 127) / 128))) break;
    for (int parts = 1; parts <= 8 && (parts == 1 || parts * 2 <= num_kb); ++parts)
      for (int per_sm = 1; per_sm <= 2; ++per_sm) {
        const int stages = stages_of(bt, per_sm == 1 ? kAlone : kOfTwo);
        if (per_sm == 2 && (stages < 3 || smem_of(bt, parts, gated, stages) > kMostOfTwo)) continue;
        const int side = side_by_side->n[per_sm][parts] - (parts == 3 ? 2 : parts == 5 ? per_sm : 0), tiles = tiles_n * tm;
        if (side <= 0) continue;
        const int rounds = (tiles + side - 1) / side;
        const double ctas = static_cast<double>(tiles < side ? tiles : side) * parts;
        double drawing = per_sm == 1 ? ctas : 1.46 * ctas;                  // SMs that draw on the memory
        if (drawing > sms) drawing = sms;
        const double copies = static_cast<double>(rounds) * per_sm * ((num_kb + parts - 1) / parts) * ((kCW + bt) * kCK * 2) * 1e-5;
        const double memory = 2.0 * N * K / 6.36e6 * (1.0 + 0.25 * (sms / drawing - 1.0));
        const double t = (copies > memory ? copies : memory) + rounds * (4.4 + 0.005 * bt) + (parts > 1 ? 0.0026 * bt : 0.0) +
                         (per_sm == 2 ? 0.0018 * bt : 0.0);
        if (t < best) {
          best = t;
          best_rounds = rounds;
          *plan = ClusterPlan{bt, parts, per_sm == 1 ? kAlone : kOfTwo};
        }
      }
  }
  return best < 1e30 && (gated || !others_are_faster(M, N, K, bn, split, *plan, best_rounds));
}

int gemm_bf16_cluster(const ClusterGemm& g, const ClusterPlan& plan, cudaStream_t st) {
  ClusterParams p;
  p.g = g;
  p.waits = g_wait_config;
  const int tiles_m = (g.M + plan.bt - 1) / plan.bt;
  p.bt = plan.bt;
  p.tiles_n = (g.N + kCW - 1) / kCW;
  p.stages = stages_of(p.bt, plan.smem);
  const int smem = smem_of(p.bt, plan.parts, g.gated, p.stages);
  if (p.stages < 2 || smem > 227 * 1024) return 1;
  p.tmem_cols = 32;
  while (p.tmem_cols < static_cast<uint32_t>(p.bt)) p.tmem_cols *= 2;
  CUtensorMap tw, tx;
  if (make_tmap_2d(&tw, g.W, g.N, g.K, g.ldw * 2, g.gated ? 64 : kCW, kCK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16)) return 1;
  if (make_tmap_2d(&tx, g.A, g.M, g.K, g.lda * 2, p.bt, kCK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16)) return 1;
  return g.gated ? launch_cluster<true>(tw, tx, p, tiles_m * p.tiles_n, plan.parts, smem, st)
                 : launch_cluster<false>(tw, tx, p, tiles_m * p.tiles_n, plan.parts, smem, st);
}

}  // namespace b200

using namespace b200;

// The kernel with a given plan: `bt` rows of A per tile, `parts` of K, shared memory per CTA (a tuning aid, and for tests)
GLLM_EXPORT int gllm_gemm_bf16_cluster(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int M, int N, int K,
                                       const void* bias, int gated, int gelu, int bt, int parts, int smem, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (K % 8 != 0 || N % 8 != 0 || lda % 8 != 0 || ldw % 8 != 0 || ldc % 8 != 0 || (gated && (N % 256 != 0 || bias != nullptr)) ||
      ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(bias)) & 15) != 0 || bt % 16 != 0 || bt < 16 || bt > 256 || parts < 1 ||
      parts > 8 || parts > (K + kCK - 1) / kCK) {
    fprintf(stderr, "[gllm_b200] gemm_bf16_cluster: M=%d N=%d K=%d with %d rows, %d parts\n", M, N, K, bt, parts);
    return 1;
  }
  const ClusterGemm g{A, W, lda, ldw, reinterpret_cast<__nv_bfloat16*>(C), ldc, M, N, K, reinterpret_cast<const __nv_bfloat16*>(bias),
                      gated != 0, gelu};
  return gemm_bf16_cluster(g, ClusterPlan{bt, parts, smem}, reinterpret_cast<cudaStream_t>(stream));
}
