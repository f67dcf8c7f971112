// Mamba-1 recurrence of prompt portions (selective_scan; csrc/seq/seq_ops.cu holds the token-serial form for decoding):
//     S_n <- exp(dt a_n) S_n + dt x B_n;  y = sum_n S_n C_n + D x;  out = y silu(z)          N states per channel, fp32
// Two or four lanes share a channel and hold an equal part of its states in registers; a block of 128 threads walks its channels
// through one piece of a sequence, 16 tokens at a time. For each 16 tokens the block first forms the steps dt = softplus(.), dt x
// and B, C in shared memory (two channels of a row per thread), then walks them (no arithmetic but the recurrence's own), then
// forms the gated outputs; the next tokens' inputs are on their way during the walk.
//
// Usually a piece is a whole sequence: one launch, every exponential once. Where the sequences are too few to fill the machine
// (scan_piece in ops/sm100_seq.py), they are cut in pieces and three kernels run: every piece's end state from zero and its sum
// of steps (the decays are diagonal, so a piece takes an entering state S_0 to exp(a_n sum dt) S_0 + its own end state); the
// chain over a sequence's pieces; every piece again from its entering state, with the outputs. Short sequences beside those are walked
// whole in the last one, so that their states do not depend on the batch.
//
// What bounds it: the 2^x unit (8 cycles per warp and exponential: 64 of about 100 cycles per token of a warp with 16 channels)
// and issue slots. So the arithmetic is on pairs (f32x2), log2(e) is multiplied into A, softplus and silu are formed once per
// token and channel in forms of their own instead of expf, log1pf and a division, and the exponential is the bare instruction with
// its bias taken out (a quarter of them as polynomials on the fma units: 730 instead of 614 us). 128 registers, for the scheduler to
// overlap four tokens (at 96: 10 % more).
// 2048 tokens in each of 4 sequences, 8192 channels, 16 states, bf16: 1329 us as chunks of 64 tokens in two passes, a thread per channel,
// with expf; 661 so (556 with the exponents of softplus and silu rounded to one fp32, which cost up to ten times their error, and
// without `anchored`).
// Relative error of the steps / gates against float64, rms over inputs in (-20, 20): at most 5.1e-8 / 5.1e-8, with expf, log1pf and a
// division 4.8e-8 / 4.9e-8; largest 1.8e-7 / 1.7e-7 and 1.9e-7 / 2.3e-7.
#include <cuda_bf16.h>

#include "common/host_utils.h"
#include "seq/seq_common.cuh"

namespace {
using namespace seqk;

constexpr int kNM = 16;                             // most states of a channel
constexpr int kThreads = 128;
constexpr int kTile = 16;                           // tokens between two barriers
constexpr int kAnchor = 4;                          // tiles between two corrections of the states' decay

// 2^t of both halves on the 2^x unit. Its results lie below 2^t on average: by 0.5e-8 for t in (-0.004, 0), 1.6e-8 to 2.7e-8 in
// (-0.5, -0.004), 2.5e-8 down to -1, 5e-8 below. That adds up over the tokens between two corrections of a state (`anchored`), so the
// caller adds kBias = 2.1e-8 / ln 2 to t in the fma that forms it. Outputs of 2048 tokens against float64, decays around exp of
// -0.001 / -0.005 / -0.01 / -0.02 / -0.05 / -0.1: 1.04e-6 / 4.3e-7 / 3.5e-7 / 3.1e-7 / 1.9e-7 / 1.3e-7 (with 2.7e-8: 9.5e-7 / 4.7e-7 /
// 4.0e-7 / 3.6e-7 / 1.7e-7 / 1.3e-7, 3.3e-8: 1.13e-6 / 4.1e-7 / 3.3e-7 / 2.7e-7 / 2.0e-7 / 1.4e-7); chunks of 64 tokens with expf 9.7e-7 /
// 3.9e-7 / 3.5e-7 / 3.2e-7 / 2.1e-7 / 1.5e-7. States: 8.8e-7 / 3.9e-7 / 3.1e-7 / 2.8e-7 / 1.7e-7 / 1.1e-7; 1.53e-6 / 4.6e-7 / 4.0e-7 / 3.3e-7 /
// 2.0e-7 / 1.3e-7.
// A single decay: A log2(e) is rounded before the product, so that decays of e^-5 and less have 1.4 times the rms error of expf(dt A),
// of a value that is added to 150 times its size, and below 2^-126 they are 0. States that forget within a token or two, steps of 0.1
// and A = -16: 6.7e-8, with expf 5.7e-8, a rounding of fp32 being 6e-8; steps of 0.1 to 2, A to -24: 5.3e-8, 5.2e-8.
constexpr float kBias = 3.0e-8f;
__device__ __forceinline__ f2 exp2_unit(f2 t) {
  float t0, t1;
  un(t, t0, t1);
  return pk(ex2(t0), ex2(t1));
}
__device__ __forceinline__ f2 rcp2(f2 v) {
  float a, b;
  un(v, a, b);
  return pk(rcp(a), rcp(b));
}
// e^-|v| = e (1 + c) of both halves. The exponent |v| log2 e is formed in two parts: rounded to one it would cost |v| 2^-24, 9e-7
// at v = -20. Here 2^x keeps denormals: it is formed once per token and channel.
__device__ __forceinline__ void exp_neg2(f2 v, f2& e, f2& c) {
  float v0, v1, t0, t1;
  un(v, v0, v1);
  v0 = fabsf(v0);
  v1 = fabsf(v1);
  const f2 m = pk(v0 > 200.f ? 200.f : v0, v1 > 200.f ? 200.f : v1);       // finite, or NaN
  const f2 t = mul2(m, pk(1.4426950216293335f, 1.4426950216293335f));
  const f2 rest = fma2(m, pk(-1.925963033500011e-8f, -1.925963033500011e-8f), fma2(m, pk(-1.4426950216293335f, -1.4426950216293335f), t));
  c = fma2(rest, pk(0.6931472f, 0.6931472f), pk(1.9e-8f, 1.9e-8f));
  un(t, t0, t1);
  asm("ex2.approx.f32 %0, %1;" : "=f"(v0) : "f"(-t0));
  asm("ex2.approx.f32 %0, %1;" : "=f"(v1) : "f"(-t1));
  e = pk(v0, v1);
}
__device__ __forceinline__ f2 neg2(f2 v) { return v ^ 0x8000000080000000ull; }
// log(1 + e^v) of both halves = max(v, 0) + log1p(e), e = e^-|v|; log1p(e) = 2 atanh(s), s = e / (2 + e) <= 1/3, by the polynomial of
// least relative error (4.5e-9) in s^2. Two roundings (2^x, the last sum): what the division leaves over and the second part of e
// are added at the end, their factors need no accuracy.
__device__ __forceinline__ f2 softplus2(f2 v) {
  f2 e, c;
  exp_neg2(v, e, c);
  const f2 two = pk(2.f, 2.f), r = rcp2(add2(e, two));
  f2 s = mul2(e, r);
  s = fma2(r, fma2(neg2(s), e, fma2(neg2(s), two, e)), s);
  const f2 left = fma2(neg2(s), e, fma2(neg2(s), two, e));
  const f2 q = mul2(s, s), twice = add2(s, s);
  f2 w = fma2(q, pk(0.14005993f, 0.14005993f), pk(0.14000903f, 0.14000903f));
  w = fma2(q, w, pk(0.20010763f, 0.20010763f));
  w = fma2(q, w, pk(0.3333321f, 0.3333321f));
  const f2 l = add2(twice, fma2(twice, fma2(q, w, c), mul2(add2(r, r), left)));
  float v0, v1;
  un(v, v0, v1);
  return add2(pk(fmaxf(v0, 0.f), fmaxf(v1, 0.f)), l);
}
// z / (1 + e^-z) of both halves, as z / (1 + e) or z e / (1 + e) with e = e^-|z|: nothing overflows. What z e and the division leave
// over and the second part of e are added at the end.
__device__ __forceinline__ f2 silu2(f2 z) {
  f2 e, c;
  exp_neg2(z, e, c);
  float z0, z1, e0, e1, c0, c1;
  un(z, z0, z1);
  un(e, e0, e1);
  un(c, c0, c1);
  const f2 m = pk(z0 < 0.f ? e0 : 1.f, z1 < 0.f ? e1 : 1.f), g = pk(z0 < 0.f ? c0 : -c0 * e0, z1 < 0.f ? c1 : -c1 * e1);
  const f2 num = mul2(z, m), r = rcp2(add2(e, pk(1.f, 1.f))), q = mul2(num, r);
  const f2 left = add2(fma2(neg2(q), e, add2(num, neg2(q))), fma2(z, m, neg2(num)));
  const f2 better = fma2(r, fma2(q, g, left), q);                          // NaN where z is infinite
  float q0, q1, b0, b1;
  un(q, q0, q1);
  un(better, b0, b1);
  return pk(fabsf(z0) <= 3.4028235e38f ? b0 : q0, fabsf(z1) <= 3.4028235e38f ? b1 : q1);
}

constexpr float kMostF = 3.4028235e38f;
// What a state lacks after steps of `Dt` in all from S0 on, decays whose product was P: the unit's errors have one sign for decays of
// about the same size, and a state that keeps thousands of tokens adds them up. exp(A Dt), formed once in 64 tokens, does not. States
// of 2048 tokens whose decays lie around 0.9999 / 0.999 / 0.99, against float64: 1.4e-6 / 8.8e-7 / 3.1e-7, without it 2.3e-5 / 1.0e-5 /
// 5.5e-7, chunks of 64 tokens with expf 9e-7 / 1.5e-6 / 4.0e-7. It costs 8 % of the kernel.
__device__ __forceinline__ float anchored(float a, float Dt, float P, float S0) {
  const float lack = (exp2f(a * Dt) - P) * S0;
  return fabsf(lack) <= kMostF ? lack : 0.f;         // infinite states and growing ones stay as they are
}

// Piece slots: sequence s owns slots from qsl[s] / piece + s on (at least one per started piece); some stay empty.
__device__ __forceinline__ int piece_base(const int* qsl, int s, int piece) { return qsl[s] / piece + s; }

struct ScanArgs {
  const float *A, *Dskip, *dt_bias;
  float* state;
  const int *rec_slots, *seq_lens, *qsl;
  int nseq, C, N, R, c0, CW, piece, uncut;
  long ldp, ldxz;
  int wide;                                          // channels 2 i, 2 i + 1 of x, dt, z and out can be moved together
  float *ends, *steps;
};

template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> { using V = uint32_t; };
template <> struct Pair<float> { using V = float2; };
__device__ __forceinline__ f2 pair_f(uint32_t v) { return pk(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
__device__ __forceinline__ f2 pair_f(float2 v) { return pk(v.x, v.y); }
__device__ __forceinline__ void pair_make(uint32_t& v, __nv_bfloat16 a, __nv_bfloat16 b) {
  v = (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}
__device__ __forceinline__ void pair_make(float2& v, float a, float b) { v = make_float2(a, b); }

// Channels [c0, c0 + CW) of the batch; ends [slot][n][CW]: end states (FINAL 0: written) or entering states (FINAL 1: read, but a
// sequence of one piece starts from the carried state itself); steps [slot][CW]: sums of dt. LPC lanes per channel, NS states at most.
template <typename T, bool FINAL, int LPC, int NS>
__global__ void __launch_bounds__(kThreads, LPC == 2 ? 4 : 6)
scan_walk_kernel(const T* __restrict__ xc, const T* __restrict__ dt_raw, const T* __restrict__ proj, const T* __restrict__ xz,
                 T* __restrict__ out, const ScanArgs p) {
  using V = typename Pair<T>::V;
  constexpr int NL = NS / LPC, NP = NL / 2;                                // states and pairs of a lane
  constexpr int CH = kThreads / LPC;                                       // channels of the block
  constexpr int RP = 2 * kThreads / CH, RT = kTile / RP;                   // rows of the block at a time; rows of a thread
  __shared__ __align__(16) float4 sD[kTile][CH];                           // dt, dt, dt x, dt x
  __shared__ __align__(16) float sBC[kTile][2 * NS];
  __shared__ __align__(16) float sY[FINAL ? kTile : 1][CH];
  const int u = blockIdx.y;
  int lo = 0, hi = p.nseq - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (piece_base(p.qsl, mid, p.piece) <= u) lo = mid; else hi = mid - 1;
  }
  const int q0 = p.qsl[lo], q1 = p.qsl[lo + 1];
  const long off = (long)(u - piece_base(p.qsl, lo, p.piece)) * p.piece;
  if (off >= q1 - q0) return;                        // uniform over the block
  const bool whole = q1 - q0 <= max(p.piece, p.uncut);
  const int base = q0 + (int)off, len = whole ? q1 - q0 : min(q1 - base, p.piece);
  const bool last = base + len >= q1;
  if (whole ? off > 0 || !FINAL : !FINAL && last) return;                  // nobody continues from the end of a sequence
  const int tid = threadIdx.x, j = tid % LPC, ch = tid / LPC, C = p.C, N = p.N;
  const int w0 = blockIdx.x * CH, w = w0 + ch;       // channel inside this round's range
  const bool active = w < p.CW;
  const int wc = active ? w : p.CW - 1, c = p.c0 + wc;                     // idle threads mirror the last channel (loads only)

  f2 S[NP], a[NP];                                   // states; A log2(e), finite (a step of 0 leaves a state alone at any rate)
  f2 S0[NP], P[NP];                                  // states and product of the decays since the last anchor
  float Dt = 0.f;                                    // sum of the steps since then
  {
    const bool carried = whole && p.state != nullptr && p.seq_lens[lo] > q1 - q0;
    const float* from = carried ? p.state + (size_t)p.rec_slots[lo] * N * C + c : p.ends + (size_t)u * N * p.CW + wc;
    const size_t step = carried ? C : p.CW;
    float sv[NL], av[NL];
#pragma unroll
    for (int e = 0; e < NL; ++e) {
      const int n = j * NL + e;
      av[e] = n < N ? p.A[(size_t)c * N + n] * 1.4426950408889634f : 0.f;
      if (fabsf(av[e]) > kMostF) av[e] = copysignf(kMostF, av[e]);
      sv[e] = FINAL && n < N && (carried || !whole) ? from[n * step] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < NP; ++e) {
      S0[e] = S[e] = pk(sv[2 * e], sv[2 * e + 1]);
      a[e] = pk(av[2 * e], av[2 * e + 1]);
      P[e] = pk(1.f, 1.f);
    }
  }

  // the two channels and the rows (r0, r0 + RP, ...) of each tile whose steps and outputs this thread forms
  const int cp = 2 * (tid % (CH / 2)), r0 = tid / (CH / 2), cc = p.c0 + w0 + cp;
  const bool on0 = w0 + cp < p.CW, on1 = w0 + cp + 1 < p.CW;
  const f2 bias = pk(on0 ? p.dt_bias[cc] : 0.f, on1 ? p.dt_bias[cc + 1] : 0.f);
  const f2 dsk = pk(on0 ? p.Dskip[cc] : 0.f, on1 ? p.Dskip[cc + 1] : 0.f);
  f2 sum = 0;
  auto load = [&](const T* src) {                    // channels cc, cc + 1 of a row
    V v;
    if (p.wide) {
      v = *reinterpret_cast<const V*>(src);
    } else {
      pair_make(v, src[0], on1 ? src[1] : src[0]);
    }
    return v;
  };
  constexpr int kBC = kTile * 2 * NS / kThreads;     // B and C values of a thread
  V dv[RT], xv[RT], zv[RT];
  T bc[kBC];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const size_t t = base + min(t0 + r0 + i * RP, len - 1);
      if (on0) {
        dv[i] = load(dt_raw + t * C + cc);
        xv[i] = load(xc + t * C + cc);
        if (FINAL) zv[i] = load(xz + t * p.ldxz + C + cc);
      }
    }
#pragma unroll
    for (int i = 0; i < kBC; ++i) {
      const int k = i * kThreads + tid, r = k / (2 * NS), v = k % (2 * NS), half = v / NS, n = min(v % NS, N - 1);
      bc[i] = proj[(size_t)(base + min(t0 + r, len - 1)) * p.ldp + p.R + half * N + n];
    }
  };
#pragma unroll
  for (int i = 0; i < RT; ++i) dv[i] = xv[i] = zv[i] = V{};
  fetch(0);
  for (int t0 = 0; t0 < len; t0 += kTile) {
    // steps and scaled inputs; tokens past the end leave the states alone (dt = dt x = B = 0)
    f2 xf[RT], zf[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = r0 + i * RP;
      xf[i] = pair_f(xv[i]);
      zf[i] = pair_f(zv[i]);
      f2 step = softplus2(add2(pair_f(dv[i]), bias)), in = mul2(step, xf[i]);
      if (t0 + r >= len) step = in = 0;
      sum = add2(sum, step);
      float s0, s1, m0, m1;
      un(step, s0, s1);
      un(in, m0, m1);
      sD[r][cp] = make_float4(s0, s0, m0, m0);
      sD[r][cp + 1] = make_float4(s1, s1, m1, m1);
    }
#pragma unroll
    for (int i = 0; i < kBC; ++i) {
      const int k = i * kThreads + tid, r = k / (2 * NS), n = k % NS;
      (&sBC[0][0])[k] = t0 + r < len && n < N ? to_f(bc[i]) : 0.f;
    }
    __syncthreads();
    if (t0 + kTile < len) fetch(t0 + kTile);         // on their way during the walk
    const int rows = min(kTile, len - t0);
#pragma unroll 1
    for (int g = 0; g < rows; g += 4) {
      float y[4];
      const f2 bias2 = pk(kBias, kBias);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(&sD[g + k][ch]);
        const f2 dt2 = d.x, dx2 = d.y;
        Dt += __uint_as_float((uint32_t)dt2);
        f2 b[NP], cv[NP];
#pragma unroll
        for (int e = 0; e < NP; e += 2) {
          const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(&sBC[g + k][j * NL + 2 * e]);
          b[e] = bb.x;
          b[e + 1] = bb.y;
          if (FINAL) {
            const ulonglong2 c2 = *reinterpret_cast<const ulonglong2*>(&sBC[g + k][NS + j * NL + 2 * e]);
            cv[e] = c2.x;
            cv[e + 1] = c2.y;
          }
        }
        f2 y2 = 0;
#pragma unroll
        for (int e = 0; e < NP; ++e) {
          const f2 dec = exp2_unit(fma2(dt2, a[e], bias2));
          S[e] = fma2(dec, S[e], mul2(dx2, b[e]));
          P[e] = mul2(P[e], dec);
          if (FINAL) y2 = e == 0 ? mul2(S[e], cv[e]) : fma2(S[e], cv[e], y2);
        }
        if (FINAL) {
          float h0, h1;
          un(y2, h0, h1);
          y[k] = h0 + h1;
        }
      }
      if (FINAL) {
        // the lanes' partial sums of the four tokens, transposed
        const bool odd = j & 1;
        const float q_0 = __shfl_xor_sync(0xffffffffu, odd ? y[0] : y[1], 1), q_1 = __shfl_xor_sync(0xffffffffu, odd ? y[2] : y[3], 1);
        const float k0 = (odd ? y[1] : y[0]) + q_0, k1 = (odd ? y[3] : y[2]) + q_1;
        if (LPC == 2) {
          sY[g + j][ch] = k0;
          sY[g + 2 + j][ch] = k1;
        } else {
          const bool up = j & 2;
          sY[g + j][ch] = (up ? k1 : k0) + __shfl_xor_sync(0xffffffffu, up ? k0 : k1, 2);
        }
      }
    }
    if ((t0 / kTile + 1) % kAnchor == 0) {
#pragma unroll
      for (int e = 0; e < NP; ++e) {
        float a0, a1, s0, s1, p0, p1, o0, o1;
        un(a[e], a0, a1);
        un(S[e], s0, s1);
        un(P[e], p0, p1);
        un(S0[e], o0, o1);
        S[e] = S0[e] = pk(s0 + anchored(a0, Dt, p0, o0), s1 + anchored(a1, Dt, p1, o1));
        P[e] = pk(1.f, 1.f);
      }
      Dt = 0.f;
    }
    __syncthreads();
    if (FINAL && on0) {
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int r = r0 + i * RP;
        if (r < rows) {
          const f2 y = *reinterpret_cast<const f2*>(&sY[r][cp]);
          float y0, y1;
          un(mul2(fma2(dsk, xf[i], y), silu2(zf[i])), y0, y1);
          const T o0 = from_f<T>(y0), o1 = from_f<T>(y1);
          T* dst = out + (size_t)(base + t0 + r) * C + cc;
          if (p.wide) {
            V v;
            pair_make(v, o0, o1);
            *reinterpret_cast<V*>(dst) = v;
          } else {
            dst[0] = o0;
            if (on1) dst[1] = o1;
          }
        }
      }
    }
  }
  if (!FINAL) {                                      // sums of the rows that other threads formed
    float* part = &sD[0][0].x;
    un(sum, part[r0 * CH + cp], part[r0 * CH + cp + 1]);
    __syncthreads();
    if (tid < CH && w0 + tid < p.CW) {
      float all = 0.f;
      for (int r = 0; r < RP; ++r) all += part[r * CH + tid];
      p.steps[(size_t)u * p.CW + w0 + tid] = all;
    }
  }
  if (!active) return;
  float sv[NL];
#pragma unroll
  for (int e = 0; e < NP; ++e) un(S[e], sv[2 * e], sv[2 * e + 1]);
  if (!FINAL) {
#pragma unroll
    for (int e = 0; e < NL; ++e)
      if (j * NL + e < N) p.ends[((size_t)u * N + j * NL + e) * p.CW + w] = sv[e];
  } else if (last && p.state != nullptr) {
    float* st = p.state + (size_t)p.rec_slots[lo] * N * C + c;
#pragma unroll
    for (int e = 0; e < NL; ++e)
      if (j * NL + e < N) st[(size_t)(j * NL + e) * C] = sv[e];
  }
}

// end states from zero -> entering states, along the pieces of each sequence
__global__ void __launch_bounds__(128) scan_carry_kernel(const ScanArgs p) {
  constexpr int U = 8;                              // pieces fetched at a time: the chain itself is two operations
  const int w = blockIdx.x * 128 + threadIdx.x, n = blockIdx.y, s = blockIdx.z;
  const int q0 = p.qsl[s], q1 = p.qsl[s + 1];
  if (w >= p.CW || q1 - q0 <= max(p.piece, p.uncut)) return;               // walked whole: from the carried state itself
  const int c = p.c0 + w, pieces = (q1 - q0 + p.piece - 1) / p.piece;
  const float a = p.A[(size_t)c * p.N + n];
  const bool carried = p.state != nullptr && p.seq_lens[s] > q1 - q0;
  float S = carried ? p.state[((size_t)p.rec_slots[s] * p.N + n) * p.C + c] : 0.f;
  const size_t u0 = piece_base(p.qsl, s, p.piece);
  float* e = p.ends + (u0 * p.N + n) * p.CW + w;
  const float* d = p.steps + u0 * p.CW + w;
  const size_t stride = (size_t)p.N * p.CW;
  for (int i0 = 0; i0 < pieces; i0 += U) {
    float g[U], end[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = i0 + i;
      const bool ok = k < pieces - 1;               // the last piece hands nothing on
      g[i] = ok ? d[(size_t)k * p.CW] : 0.f;
      end[i] = ok ? e[k * stride] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = i0 + i;
      if (k < pieces) {
        e[k * stride] = S;
        S = expf(g[i] * a) * S + end[i];
      }
    }
  }
}

template <typename T, int LPC, int NS>
int launch_scan(const void* xc, const void* dt_raw, const void* proj, const void* xz, ScanArgs p, int ntok, int width, float* work,
                void* out, cudaStream_t st) {
  constexpr int CH = kThreads / LPC;
  const int C = p.C, slots = ntok / p.piece + p.nseq;
  const bool cut = ntok > p.piece;
  if (!cut) width = C;
  p.wide = C % 2 == 0 && width % 2 == 0 && p.ldxz % 2 == 0 &&
           (((uintptr_t)xc | (uintptr_t)dt_raw | (uintptr_t)xz | (uintptr_t)out) & (2 * sizeof(T) - 1)) == 0;
  for (p.c0 = 0; p.c0 < C; p.c0 += width) {
    p.CW = width < C - p.c0 ? width : C - p.c0;
    p.ends = work;
    p.steps = work + (size_t)slots * p.N * p.CW;
    const dim3 grid((p.CW + CH - 1) / CH, slots);
    if (cut) {
      scan_walk_kernel<T, false, LPC, NS><<<grid, kThreads, 0, st>>>((const T*)xc, (const T*)dt_raw, (const T*)proj, (const T*)xz, (T*)out, p);
      scan_carry_kernel<<<dim3((p.CW + 127) / 128, p.N, p.nseq), 128, 0, st>>>(p);
    }
    scan_walk_kernel<T, true, LPC, NS><<<grid, kThreads, 0, st>>>((const T*)xc, (const T*)dt_raw, (const T*)proj, (const T*)xz, (T*)out, p);
  }
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

template <typename T>
int pick_scan(int lanes, const void* xc, const void* dt_raw, const void* proj, const void* xz, const ScanArgs& p, int ntok,
              int width, float* work, void* out, cudaStream_t st) {
  auto go = p.N <= 8 ? launch_scan<T, 2, 8> : lanes == 2 ? launch_scan<T, 2, 16> : launch_scan<T, 4, 16>;
  return go(xc, dt_raw, proj, xz, p, ntok, width, work, out, st);
}

}  // namespace

// Sequences longer than both `piece` and `uncut` tokens are cut, `width` channels at a time; none is if piece >= ntok, and `work` is
// not used then.
// Returns 2 outside its envelope (the caller then uses the token-serial kernel): N <= 16. `work`: (ntok / piece + nseq) * (N + 1) *
// min(width, C) floats.
GLLM_EXPORT int gllm_scan_walk(const void* xc, const void* dt_raw, const void* proj, long ldp, const void* xz, long ldxz,
                               const void* A, const void* Dskip, const void* dt_bias, void* state, const void* rec_slots,
                               const void* seq_lens, const void* qsl, int ntok, int nseq, int C, int N, int R, int piece,
                               int uncut, int width, void* work, void* out, int is_f32, void* stream) {
  if (nseq <= 0 || ntok <= 0) return 0;
  if (N < 1 || N > kNM || width < 1 || piece < 1 || nseq > 65535 || ntok / piece + nseq > 65535) return 2;
  ScanArgs p{};
  p.A = (const float*)A; p.Dskip = (const float*)Dskip; p.dt_bias = (const float*)dt_bias;
  p.state = (float*)state;
  p.rec_slots = (const int*)rec_slots; p.seq_lens = (const int*)seq_lens; p.qsl = (const int*)qsl;
  p.nseq = nseq; p.C = C; p.N = N; p.R = R; p.piece = piece; p.uncut = uncut; p.ldp = ldp; p.ldxz = ldxz;
  // Two lanes per channel spend fewer instructions, four have twice the warps. With warps for every scheduler two are faster (8192
  // channels, 4 portions of 2048, 3.5 warps: 661 / 701 us; 2 of 2048, 1.7: 407 / 483; 4096 channels, 4 of 2048, 1.7: 407 / 405), with
  // few four (4096 channels, 700 tokens, 0.4 warps: 112 / 81; 2000, 300, 100 and 50 tokens, of which one is walked for long: 318 /
  // 272). Portions are counted as if they were equal, hence the line at three.
  const int pieces = piece < ntok ? ntok / piece : nseq;
  const int lanes = static_cast<int64_t>(C) / 16 * pieces >= 3 * 4 * b200::num_sms() ? 2 : 4;
  return (is_f32 ? pick_scan<float> : pick_scan<__nv_bfloat16>)(lanes, xc, dt_raw, proj, xz, p, ntok, width, (float*)work, out,
                                                                (cudaStream_t)stream);
}
