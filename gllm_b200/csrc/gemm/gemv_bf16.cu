// bf16 GEMM of one or two rows (the decode step of a sequence or two) for sm_100a:
//
//     C[M, N] = A[M, K] · W[N, K]^T        M <= 2
//
// Bound by the weight bytes and, for the small matrices of a layer, by latency: launch, one trip to HBM, the sum. A warp owns one
// or two weight rows with the whole of K: no tensor core, no split of K, no second pass over partial sums. Its first 4 KB of
// weights are in flight before the previous kernel ends, the next 4 KB while one is multiplied; the rows of A wait in shared
// memory. Products and sums are fp32 (a lane's in order, then a tree over the lanes).
// Taken where the busiest SM streams at most 560 KB (one row) or 140 KB (two), whole rounds of its 16 warps counted, and the rows
// of A fit 48 KB. The tensor-core kernel has 192 KB per SM in flight before the previous kernel ends where this one has 64, and its
// last round is not partly empty, so it wins on large matrices; two rows unpack A again for every weight row. Timed on whole
// captured decode steps, all layers (ms, one row / two; 0: none, then up to 560 / 140 KB, then up to 800 / 400 KB):
//     0.6B shape          0.979 / 0.995    0.712 / 0.833    0.712 / 0.830
//     1.7B, 16 layers     0.872 / 0.895    0.741 / 0.852    0.737 / 0.836
//     4B, 16 layers       1.255 / 1.247    1.189 / 1.248    1.142 / 1.261
//     8B, 20 layers       2.065 / 2.062    2.009 / 2.060    2.081 / 2.116    (everything: +10 % / +15 %)
//     half of it          1.386 / 1.375    1.307 / 1.346    1.346 / 1.400
//     an eighth           0.775 / 0.782    0.640 / 0.739    0.638 / 0.747
//     70B, an eighth, 10  0.698 / 0.703    0.688 / 0.692    0.690 / 0.723
// One GEMM at a time says otherwise (4096 -> 2 x 12288, 12288 -> 4096 cold: 19.9 -> 16.7 us on average for a layer of the 8B shape).
// Three rows lose where the matrix is large (74 against 53 us): the arithmetic of the plain cores then outlasts the weights.
#include "../common/host_utils.h"
#include "../common/ptx.cuh"

namespace b200 {

struct GemvParams {
  const __nv_bfloat16* a;
  const __nv_bfloat16* w;
  __nv_bfloat16* c;
  const __nv_bfloat16* bias;
  int64_t lda, ldw, ldc;
  int N, K, units;
};

__device__ __forceinline__ uint4 ldg_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// bf16 pair -> two fp32 in one 64-bit register, and acc += a * b on both
__device__ __forceinline__ uint64_t pair_f32(uint32_t v) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(v << 16), "r"(v & 0xffff0000u));
  return d;
}
__device__ __forceinline__ void fma_pair(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// most bytes of weights that the busiest SM streams
static constexpr int64_t kMostOneRow = 560 * 1024, kMostTwoRows = 140 * 1024;

// MT: rows of A; R weight rows per warp, U 16-byte loads per lane and row at a time.
// ACT 0: plain (+ bias); 1: silu(gate) * up; 2: tanh gelu. Gated weights are interleaved per 128 rows (128 gate, 128 up), R = 2.
template <int MT, int R, int U, int ACT>
__global__ void __launch_bounds__(128) gemv_kernel(const GemvParams p) {
  extern __shared__ __align__(16) uint8_t gemv_smem[];
  __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(gemv_smem);      // [MT][K]
  const int lane = threadIdx.x & 31, wid = blockIdx.x * 4 + (threadIdx.x >> 5), nw = gridDim.x * 4;
  const int chunks = (p.K + 256 * U - 1) / (256 * U);
  griddep_launch();
  auto row_of = [&](int u, int r) { return ACT != 0 ? (u >> 7) * 256 + (u & 127) + r * 128 : u * R + r; };
  auto load = [&](int u, int c, uint4 (&v)[R][U]) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int n = row_of(u, r);
      const __nv_bfloat16* src = p.w + static_cast<size_t>(n) * p.ldw;
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int k = (c * U + i) * 256 + lane * 8;
        v[r][i] = n < p.N && k < p.K ? ldg_stream(src + k) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  uint4 cur[R][U], nxt[R][U];
  int u = wid, c = 0;
  if (u < p.units) load(u, 0, cur);
  griddep_wait();
  for (int i = threadIdx.x; i < MT * (p.K / 8); i += 128) {
    const int m = i / (p.K / 8), k = (i - m * (p.K / 8)) * 8;
    *reinterpret_cast<uint4*>(xs + m * p.K + k) = __ldcg(reinterpret_cast<const uint4*>(p.a + m * p.lda + k));
  }
  __syncthreads();
  uint64_t acc[R][MT];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m] = 0ull;
  while (u < p.units) {
    int nu = u, nc = c + 1;
    if (nc == chunks) { nc = 0; nu += nw; }
    if (nu < p.units) load(nu, nc, nxt);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = (c * U + i) * 256 + lane * 8;
      if (k < p.K) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const uint4 x = *reinterpret_cast<const uint4*>(xs + m * p.K + k);
          const uint64_t x0 = pair_f32(x.x), x1 = pair_f32(x.y), x2 = pair_f32(x.z), x3 = pair_f32(x.w);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            fma_pair(acc[r][m], pair_f32(cur[r][i].x), x0);
            fma_pair(acc[r][m], pair_f32(cur[r][i].y), x1);
            fma_pair(acc[r][m], pair_f32(cur[r][i].z), x2);
            fma_pair(acc[r][m], pair_f32(cur[r][i].w), x3);
          }
        }
      }
    }
    if (nc == 0) {                                      // the rows are done
      float sum[R][MT];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          float s = __uint_as_float(static_cast<uint32_t>(acc[r][m])) + __uint_as_float(static_cast<uint32_t>(acc[r][m] >> 32));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          sum[r][m] = s;
          acc[r][m] = 0ull;
        }
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (lane != m) continue;
        if (ACT != 0) {
          const float g = sum[0][m], up = sum[R - 1][m];
          p.c[m * p.ldc + u] = __float2bfloat16((ACT == 2 ? gelu_tanh_fast(g) : g / (1.f + __expf(-g))) * up);
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int n = row_of(u, r);
            if (n < p.N) p.c[m * p.ldc + n] = __float2bfloat16(sum[r][m] + (p.bias != nullptr ? __bfloat162float(p.bias[n]) : 0.f));
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < U; ++i) cur[r][i] = nxt[r][i];
    u = nu;
    c = nc;
  }
}

template <int MT, int R, int U, int ACT>
static int launch_gemv(GemvParams p, cudaStream_t st) {
  p.units = ACT != 0 ? p.N / 2 : (p.N + R - 1) / R;
  const int want = (p.units + 3) / 4, sms = num_sms(), grid = want < 4 * sms ? want : 4 * sms;
  // what the busiest SM streams: whole rounds of its warps, the last one included
  const int64_t rounds = (p.units + 4 * grid - 1) / (4 * grid), warps = (grid + sms - 1) / sms * 4;
  if (rounds * warps * R * p.K * 2 > (MT == 1 ? kMostOneRow : kMostTwoRows)) return -1;
  CUDA_CHECK_RET(launch_pdl(gemv_kernel<MT, R, U, ACT>, dim3(grid), dim3(128), MT * p.K * 2, st, p));
  return 0;
}

template <int MT>
static int launch_gemv_rows(const GemvParams& p, int act, cudaStream_t st) {
  if (act == 1) return launch_gemv<MT, 2, 4, 1>(p, st);
  if (act == 2) return launch_gemv<MT, 2, 4, 2>(p, st);
  // two short rows at a time share the reads of A; one row at a time while two would leave SMs without work
  if (p.K <= 1024 && p.N >= 4096) return launch_gemv<MT, 2, 4, 0>(p, st);
  return launch_gemv<MT, 1, 8, 0>(p, st);
}

// Called by gllm_gemm_smallm. Returns -1 for what this kernel does not take.
int gemv_bf16(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int M, int N, int K, const void* bias,
              int act, cudaStream_t st) {
  if (M > 2 || K <= 0 || (act != 0 && N % 256 != 0)) return -1;
  if (((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) != 0) return -1;
  if (M * K * 2 > 48 * 1024) return -1;                // the rows of A in shared memory
  GemvParams p = {};
  p.a = reinterpret_cast<const __nv_bfloat16*>(A);
  p.w = reinterpret_cast<const __nv_bfloat16*>(W);
  p.c = reinterpret_cast<__nv_bfloat16*>(C);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.lda = lda; p.ldw = ldw; p.ldc = ldc;
  p.N = N; p.K = K;
  return M == 1 ? launch_gemv_rows<1>(p, act, st) : launch_gemv_rows<2>(p, act, st);
}

}  // namespace b200
