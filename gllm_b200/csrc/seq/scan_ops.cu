// Mamba-1 recurrence cut in time (selective_scan; csrc/seq/seq_ops.cu holds the token-serial form):
//     S_n <- exp(dt a_n) S_n + dt x B_n;  y = sum_n S_n C_n + D x;  out = y silu(z)          N states per channel, fp32
// The decays are diagonal, so a chunk of 64 tokens takes an entering state S_0 to exp(a_n sum dt) S_0 + (its own end state).
// Three kernels: every chunk's end state from zero and its sum of steps; the chain over a sequence's chunks (one thread per
// channel and state); every chunk again from its entering state, with the outputs. One thread per channel, all its states in
// registers, no shuffles. Same formulas, order and functions per token as the serial kernel.
//
// What bounds it: issue slots, about 11 per (token, channel, state) and pass, most of them the accurate expf. The serial kernel
// does the exponentials once, but its longest sequence is one chain of tokens on a part of the machine, and the four threads of
// a channel each form the same steps and gates.
// 8192 ragged tokens in 4 sequences, 8192 channels, 16 states: 527 + 29 + 740 us, token-serial 2999 us (B200); one sequence of
// 8192 tokens: 1.28 ms / 8.5 ms. The hardware's 2^x on an exponent in two parts would take 250 us off, but its error is up to
// 1.8 times that of expf (state of 2048 tokens against float64: 3.1e-7 / 1.8e-7).
#include <cuda_bf16.h>

#include "common/host_utils.h"
#include "seq/seq_common.cuh"

namespace {
using namespace seqk;

constexpr int kL = 64;                              // tokens of a chunk
constexpr int kNM = 16;                             // states a thread holds
constexpr int kRows = 2 * kL;                       // tokens of the longest sequence that is walked whole

// Chunk slots: sequence s owns slots from qsl[s] / 64 + s on (at least one per started 64 tokens); some stay empty.
__device__ __forceinline__ int chunk_base(const int* qsl, int s) { return qsl[s] / kL + s; }

// Channels [c0, c0 + CW) of the batch; ends [slot][n][CW]: end states (FINAL 0: written) or entering states (FINAL 1: read);
// steps [slot][CW]: sums of dt. Sequences of fewer than min_len tokens are not cut: FINAL walks them whole, from the carried
// state (a kernel of their own behind the three took as long again: 8 portions of 100 tokens and one of 150).
template <typename T, bool FINAL>
__global__ void __launch_bounds__(128, FINAL ? 6 : 7) scan_chunk_kernel(
    const T* __restrict__ xc, const T* __restrict__ dt_raw, const T* __restrict__ proj, long ldp, const T* __restrict__ xz,
    long ldxz, const float* __restrict__ A, const float* __restrict__ Dskip, const float* __restrict__ dt_bias,
    float* __restrict__ state, const int* __restrict__ rec_slots, const int* __restrict__ seq_lens, const int* __restrict__ qsl,
    int nseq, int C, int N, int R, int c0, int CW, int min_len, float* __restrict__ ends, float* __restrict__ steps, T* __restrict__ out) {
  constexpr int TCH = 8;
  __shared__ __align__(16) float sBC[FINAL ? kRows : kL][2 * kNM];
  const int u = blockIdx.y;
  int lo = 0, hi = nseq - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (chunk_base(qsl, mid) <= u) lo = mid; else hi = mid - 1;
  }
  const int q0 = qsl[lo], q1 = qsl[lo + 1];
  const int base = q0 + (u - chunk_base(qsl, lo)) * kL;
  const bool whole = q1 - q0 < min_len;
  if (base < q0 || base >= q1 || (whole && base != q0)) return;     // uniform over the block
  const bool last = whole || base + kL >= q1;
  if (!FINAL && last) return;                       // nobody continues from its end
  const int len = (FINAL && whole ? q1 : min(base + kL, q1)) - base;      // whole: fewer than min_len tokens, at most kRows
  const int w = blockIdx.x * 128 + threadIdx.x;     // channel inside this round's range
  const bool active = w < CW;
  const int c = c0 + (active ? w : CW - 1);         // idle threads mirror the last channel (loads only)
  float S[kNM], a[kNM];
  float* e0 = ends + ((size_t)u * N) * CW + (active ? w : CW - 1);
  const bool carried = whole && state != nullptr && seq_lens[lo] > q1 - q0;
  const float* from = carried ? state + (size_t)rec_slots[lo] * N * C + c : e0;
  const size_t step = carried ? C : CW;
#pragma unroll
  for (int n = 0; n < kNM; ++n) {
    a[n] = n < N ? A[(size_t)c * N + n] : 0.f;
    S[n] = FINAL && n < N && (carried || !whole) ? from[n * step] : 0.f;
  }
  const float dsk = Dskip[c], bias = dt_bias[c];
  float sum = 0.f;
  for (int i = threadIdx.x; i < len * 2 * kNM; i += 128) {
    const int k = i / (2 * kNM), n = i % kNM, half = (i / kNM) & 1;
    sBC[k][half * kNM + n] = n < N ? to_f(proj[(size_t)(base + k) * ldp + R + half * N + n]) : 0.f;
  }
  __syncthreads();
  for (int k0 = 0; k0 < len; k0 += TCH) {
    float dtv[TCH], xv[TCH], zv[TCH];
#pragma unroll
    for (int k = 0; k < TCH; ++k) {
      const size_t t = base + min(k0 + k, len - 1);
      dtv[k] = to_f(dt_raw[t * C + c]);
      xv[k] = to_f(xc[t * C + c]);
      if (FINAL) zv[k] = to_f(xz[t * ldxz + C + c]);
    }
#pragma unroll
    for (int k = 0; k < TCH; ++k) {
      if (k0 + k < len) {
        const float v = dtv[k] + bias;
        const float dt = v > 20.0f ? v : log1pf(expf(v));
        const float x = xv[k], dx = dt * x;
        const float4* bc = reinterpret_cast<const float4*>(sBC[k0 + k]);
        float y4[4] = {0.f, 0.f, 0.f, 0.f};
        sum += dt;
#pragma unroll
        for (int g = 0; g < kNM / 4; ++g) {
          const float4 bv = bc[g], cv = bc[kNM / 4 + g];
          const float b[4] = {bv.x, bv.y, bv.z, bv.w}, cc[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int n = 4 * g + e;
            S[n] = expf(dt * a[n]) * S[n] + dx * b[e];
            if (FINAL) y4[e] = fmaf(S[n], cc[e], y4[e]);
          }
        }
        if (FINAL) {
          const float z = zv[k], y = fmaf(dsk, x, (y4[0] + y4[1]) + (y4[2] + y4[3]));
          if (active) out[(size_t)(base + k0 + k) * C + c] = from_f<T>(y * (z / (1.0f + expf(-z))));
        }
      }
    }
  }
  if (!active) return;
  if (!FINAL) {
#pragma unroll
    for (int n = 0; n < kNM; ++n)
      if (n < N) e0[(size_t)n * CW] = S[n];
    steps[(size_t)u * CW + w] = sum;
  } else if (last && state != nullptr) {
    float* st = state + (size_t)rec_slots[lo] * N * C;
#pragma unroll
    for (int n = 0; n < kNM; ++n)
      if (n < N) st[(size_t)n * C + c] = S[n];
  }
}

// end states from zero -> entering states, along the chunks of each sequence
__global__ void __launch_bounds__(128) scan_carry_kernel(const float* __restrict__ A, const float* __restrict__ state,
                                                         const int* __restrict__ rec_slots, const int* __restrict__ seq_lens,
                                                         const int* __restrict__ qsl, int C, int N, int c0, int CW,
                                                         int min_len, float* __restrict__ ends,
                                                         const float* __restrict__ steps) {
  constexpr int U = 8;                              // chunks fetched at a time: the chain itself is two operations
  const int w = blockIdx.x * 128 + threadIdx.x, n = blockIdx.y, s = blockIdx.z;
  const int q0 = qsl[s], q1 = qsl[s + 1];
  if (w >= CW || q1 <= q0 || q1 - q0 < min_len) return;
  const int c = c0 + w, chunks = (q1 - q0 + kL - 1) / kL;
  const float a = A[(size_t)c * N + n];
  const bool carried = state != nullptr && seq_lens[s] > q1 - q0;
  float S = carried ? state[((size_t)rec_slots[s] * N + n) * C + c] : 0.f;
  const size_t u0 = chunk_base(qsl, s);
  float* e = ends + (u0 * N + n) * CW + w;
  const float* d = steps + u0 * CW + w;
  const size_t stride = (size_t)N * CW;
  for (int i0 = 0; i0 < chunks; i0 += U) {
    float g[U], end[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = i0 + i;
      const bool ok = k < chunks - 1;               // the last chunk hands nothing on
      g[i] = ok ? d[(size_t)k * CW] : 0.f;
      end[i] = ok ? e[k * stride] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = i0 + i;
      if (k < chunks) {
        e[k * stride] = S;
        S = expf(g[i] * a) * S + end[i];
      }
    }
  }
}

template <typename T>
int launch_scan(const void* xc, const void* dt_raw, const void* proj, long ldp, const void* xz, long ldxz, const float* A,
                const float* Dskip, const float* dt_bias, float* state, const int* rec_slots, const int* seq_lens,
                const int* qsl, int ntok, int nseq, int C, int N, int R, int min_len, int width, float* work, void* out,
                cudaStream_t st) {
  const int slots = ntok / kL + nseq;
  for (int c0 = 0; c0 < C; c0 += width) {
    const int cw = width < C - c0 ? width : C - c0;
    float* steps = work + (size_t)slots * N * cw;
    const dim3 grid((cw + 127) / 128, slots);
    scan_chunk_kernel<T, false><<<grid, 128, 0, st>>>((const T*)xc, (const T*)dt_raw, (const T*)proj, ldp, (const T*)xz, ldxz,
                                                      A, Dskip, dt_bias, state, rec_slots, seq_lens, qsl, nseq, C, N, R, c0, cw,
                                                      min_len, work, steps, (T*)out);
    scan_carry_kernel<<<dim3((cw + 127) / 128, N, nseq), 128, 0, st>>>(A, state, rec_slots, seq_lens, qsl, C, N, c0, cw,
                                                                       min_len, work, steps);
    scan_chunk_kernel<T, true><<<grid, 128, 0, st>>>((const T*)xc, (const T*)dt_raw, (const T*)proj, ldp, (const T*)xz, ldxz,
                                                     A, Dskip, dt_bias, state, rec_slots, seq_lens, qsl, nseq, C, N, R, c0, cw,
                                                     min_len, work, steps, (T*)out);
  }
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

}  // namespace

// Sequences with at least min_len new tokens are cut, the others walked whole, `width` channels at a time; returns 2 outside its
// envelope (the caller then uses the token-serial kernel): N <= 16. `work`: (ntok / 64 + nseq) * (N + 1) * min(width, C) floats.
GLLM_EXPORT int gllm_scan_chunk(const void* xc, const void* dt_raw, const void* proj, long ldp, const void* xz, long ldxz,
                                const void* A, const void* Dskip, const void* dt_bias, void* state, const void* rec_slots,
                                const void* seq_lens, const void* qsl, int ntok, int nseq, int C, int N, int R, int min_len,
                                int width, void* work, void* out, int is_f32, void* stream) {
  if (nseq <= 0 || ntok <= 0) return 0;
  if (N < 1 || N > kNM || width < 1 || min_len > kRows + 1 || nseq > 65535 || ntok / kL + nseq > 65535) return 2;
  auto go = is_f32 ? launch_scan<float> : launch_scan<__nv_bfloat16>;
  return go(xc, dt_raw, proj, ldp, xz, ldxz, (const float*)A, (const float*)Dskip, (const float*)dt_bias, (float*)state,
            (const int*)rec_slots, (const int*)seq_lens, (const int*)qsl, ntok, nseq, C, N, R, min_len, width, (float*)work,
            out, (cudaStream_t)stream);
}
