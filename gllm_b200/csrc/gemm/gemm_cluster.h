// bf16 GEMM of decode batches with K cut over the CTAs of a cluster (gemm_bf16_cluster.cu)
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

static constexpr int kClusterStages = 12;    // most stages of the ring

struct ClusterGemm {
  const void *A, *W;                         // [M, K], [N, K]; rows lda / ldw elements apart, multiples of 8
  int64_t lda, ldw;
  __nv_bfloat16* C;                          // 16-byte aligned, rows ldc apart (a multiple of 8)
  int64_t ldc;
  int M, N, K;                               // N, K multiples of 8
  const __nv_bfloat16* bias;                 // [N] or null
  bool gated;                                // weight rows in blocks of 128 gate, 128 up rows: C [M, N / 2] = silu(gate) * up
  int gelu;                                  // gated: the tanh form of gelu instead
};

struct ClusterPlan {
  int bt;                                    // rows of A per tile: a multiple of 16, at most 256
  int parts;                                 // CTAs of a cluster = parts of K, 1 to 8
  int smem;                                  // shared memory per CTA that the ring may fill
};

// Whether this kernel is the faster one for a product of this size, and how. `bn`, `split`: the tile width and K split that gemm_bf16.cu
// would take instead (0: not that kernel).
bool plan_gemm_cluster(int M, int N, int K, bool gated, int bn, int split, ClusterPlan* plan);

// 0: launched
int gemm_bf16_cluster(const ClusterGemm& g, const ClusterPlan& plan, cudaStream_t st);

}  // namespace b200
