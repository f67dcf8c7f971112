// The bf16 GEMM on pairs of SMs (gemm_bf16_pair.cu) as gemm_bf16.cu calls it.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

struct PairGemm {
  const void *A, *W;
  int64_t lda, ldw;
  __nv_bfloat16* C;
  int64_t ldc;
  int M, N, K;
  const __nv_bfloat16* bias;
  int gated;                         // 1: weight rows interleaved per 128, C [M, N / 2]
  float glu_limit, glu_alpha;        // glu_limit > 0: the clamped gate; otherwise
  int gelu;                          // 1: the tanh form of gelu, 0: silu
};

// Needs K, N and the leading dimensions in multiples of 8, C and bias on 16-byte boundaries.
int gemm_bf16_pair(const PairGemm& g, cudaStream_t st);

}  // namespace b200
