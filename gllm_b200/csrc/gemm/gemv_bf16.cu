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
  // NORM: the rows of A are rmsnorm(a + residual) * norm_w; the sums go to residual_out ([M, K], as residual)
  const __nv_bfloat16 *residual, *norm_w;
  __nv_bfloat16* residual_out;
  float eps;
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
// NORM: every block forms the normed rows for itself (6 KB of reads at K = 1024), so that a decoding layer's norms are no launches of their
// own: decode step of one sequence, 8 layers of the 0.6B shape, 282 -> 270 us (sixteen launches of 1.8 less, the products 0.2 longer).
template <int MT, int R, int U, int ACT, bool NORM>
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
  if constexpr (NORM) {
    __shared__ float red[MT][4];                           // counted by gemv_takes
    float ss[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      ss[m] = 0.f;
      for (int k = threadIdx.x * 8; k < p.K; k += 128 * 8) {
        const uint4 a = __ldcg(reinterpret_cast<const uint4*>(p.a + m * p.lda + k));
        const uint4 b = __ldcg(reinterpret_cast<const uint4*>(p.residual + static_cast<size_t>(m) * p.K + k));
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = unpack_bf16(aw[e]), y = unpack_bf16(bw[e]);
          o[e] = pack_bf16(x.x + y.x, x.y + y.y);
          const float2 z = unpack_bf16(o[e]);              // the norm is of the rounded sum
          ss[m] += z.x * z.x + z.y * z.y;
        }
        const uint4 v = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(xs + m * p.K + k) = v;
        if (blockIdx.x == 0) *reinterpret_cast<uint4*>(p.residual_out + static_cast<size_t>(m) * p.K + k) = v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss[m] += __shfl_xor_sync(0xffffffffu, ss[m], o);
      if (lane == 0) red[m][threadIdx.x >> 5] = ss[m];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float inv = rsqrtf((red[m][0] + red[m][1] + red[m][2] + red[m][3]) / static_cast<float>(p.K) + p.eps);
      for (int k = threadIdx.x * 8; k < p.K; k += 128 * 8) {          // this thread's own values
        const uint4 v = *reinterpret_cast<const uint4*>(xs + m * p.K + k), g = *reinterpret_cast<const uint4*>(p.norm_w + k);
        const uint32_t vw[4] = {v.x, v.y, v.z, v.w}, gw[4] = {g.x, g.y, g.z, g.w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = unpack_bf16(vw[e]), y = unpack_bf16(gw[e]);
          o[e] = pack_bf16(x.x * inv * y.x, x.y * inv * y.y);
        }
        *reinterpret_cast<uint4*>(xs + m * p.K + k) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  } else {
    for (int i = threadIdx.x; i < MT * (p.K / 8); i += 128) {
      const int m = i / (p.K / 8), k = (i - m * (p.K / 8)) * 8;
      *reinterpret_cast<uint4*>(xs + m * p.K + k) = __ldcg(reinterpret_cast<const uint4*>(p.a + m * p.lda + k));
    }
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

template <int MT, int R, int U, int ACT, bool NORM>
static int launch_gemv(GemvParams p, cudaStream_t st) {
  p.units = ACT != 0 ? p.N / 2 : (p.N + R - 1) / R;
  const int want = (p.units + 3) / 4, sms = num_sms(), grid = want < 4 * sms ? want : 4 * sms;
  // what the busiest SM streams: whole rounds of its warps, the last one included
  const int64_t rounds = (p.units + 4 * grid - 1) / (4 * grid), warps = (grid + sms - 1) / sms * 4;
  if (rounds * warps * R * p.K * 2 > (MT == 1 ? kMostOneRow : kMostTwoRows)) return -1;
  CUDA_CHECK_RET(launch_pdl(gemv_kernel<MT, R, U, ACT, NORM>, dim3(grid), dim3(128), MT * p.K * 2, st, p));
  return 0;
}

template <int MT, bool NORM>
static int launch_gemv_rows(const GemvParams& p, int act, cudaStream_t st) {
  if (act == 1) return launch_gemv<MT, 2, 4, 1, NORM>(p, st);
  if (act == 2) return launch_gemv<MT, 2, 4, 2, NORM>(p, st);
  // two short rows at a time share the reads of A; one row at a time while two would leave SMs without work
  if (p.K <= 1024 && p.N >= 4096) return launch_gemv<MT, 2, 4, 0, NORM>(p, st);
  return launch_gemv<MT, 1, 8, 0, NORM>(p, st);
}

static bool gemv_takes(const void* A, const void* W, int M, int N, int K, int act, bool norm) {
  return M <= 2 && K > 0 && (act == 0 || N % 256 == 0) && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0 &&
         M * K * 2 + (norm ? M * 16 : 0) <= 48 * 1024;     // shared memory: the rows of A and, normed, the warps' sums
}

static GemvParams gemv_params(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int N, int K,
                              const void* bias) {
  GemvParams p = {};
  p.a = reinterpret_cast<const __nv_bfloat16*>(A);
  p.w = reinterpret_cast<const __nv_bfloat16*>(W);
  p.c = reinterpret_cast<__nv_bfloat16*>(C);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.lda = lda; p.ldw = ldw; p.ldc = ldc;
  p.N = N; p.K = K;
  return p;
}

// Called by gllm_gemm_smallm. Returns -1 for what this kernel does not take.
int gemv_bf16(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int M, int N, int K, const void* bias,
              int act, cudaStream_t st) {
  if (!gemv_takes(A, W, M, N, K, act, false)) return -1;
  const GemvParams p = gemv_params(A, lda, W, ldw, C, ldc, N, K, bias);
  return M == 1 ? launch_gemv_rows<1, false>(p, act, st) : launch_gemv_rows<2, false>(p, act, st);
}

}  // namespace b200

using namespace b200;

// C[M, N] = (rmsnorm(y + residual) * norm_w) · W[N, K]^T (+ bias, or gated by `act` as in gllm_gemm_smallm); residual_out = y + residual.
// residual, residual_out [M, K] contiguous and not the same. Returns 2 for what the kernel of one or two rows does not take.
GLLM_EXPORT int gllm_norm_gemv(const void* y, int64_t ldy, const void* residual, void* residual_out, const void* norm_w, float eps,
                               const void* W, int64_t ldw, void* C, int64_t ldc, int M, int N, int K, const void* bias, int act,
                               void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 8 != 0 || ldy % 8 != 0 || ldw % 8 != 0 || !gemv_takes(y, W, M, N, K, act, true) ||
      ((reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(residual_out) | reinterpret_cast<uintptr_t>(norm_w)) & 15) != 0)
    return 2;
  GemvParams p = gemv_params(y, ldy, W, ldw, C, ldc, N, K, bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.residual_out = reinterpret_cast<__nv_bfloat16*>(residual_out);
  p.norm_w = reinterpret_cast<const __nv_bfloat16*>(norm_w);
  p.eps = eps;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int rc = M == 1 ? launch_gemv_rows<1, true>(p, act, st) : launch_gemv_rows<2, true>(p, act, st);
  return rc < 0 ? 2 : rc;
}
