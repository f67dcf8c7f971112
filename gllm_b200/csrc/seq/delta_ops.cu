// Chunked form of the gated delta rule (linear_state_scan with `delta`; csrc/seq/state_ops.cu holds the token-serial one):
//     S <- g_t S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t          S [D, V] fp32 per head
// Inside a chunk of 64 tokens, with L_t the running sum of log g and k, q already scaled (unit length, q factor):
//     (I + A) U = B,  A_ts = beta_t exp(L_t - L_s) (k_t . k_s) for s < t,  B_t = beta_t (v_t - exp(L_t) S_0^T k_t)
//     o_t   = exp(L_t) S_0^T q_t + sum_{s <= t} P_ts u_s,  P_ts = exp(L_t - L_s) (q_t . k_s)
//     S_end = exp(L_63) S_0 + sum_s k_s (exp(L_63 - L_s) u_s)^T
// (the chunkwise form of Yang, Wang, Zhang, Shen and Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence
// Length", 2024, with the decays of Yang, Kautz and Hatamizadeh, "Gated Delta Networks", 2024).
// Two kernels. `delta_prep_kernel` does what does not depend on S, for all chunks at once: T = (I + A)^-1 (two 32-row
// triangles by substitution, the block between them by two products, in fp32) and P. `delta_chunk_kernel` walks the chunks
// of one (sequence, head, 64 value columns) with S in registers: K S and Q S, U = T B, P U, K^T U, all on the tensor cores.
//
// Precision: what was fp32 stays fp32. k, q and v are bf16 as given (scales are applied to rows of the fp32 results), so
// their products are exact; fp32 operands (S, B, T, U, P) are split into three bf16 parts, which hold all 24 bits: three
// products against an exact operand, six of the nine between two split ones. The three left out are 2^-24 of the product each,
// about an fp32 rounding; the test holds the error against float64 to 1.2 times the token-serial kernel's.
//
// Values that are no numbers: a product with a zero above the diagonal would carry a token's NaN or infinity to the tokens before
// it in its 16-row tile. Rows of B and U enter the products with zeros in such places; the place of the first one in each
// column is kept, and the column's results from that token on, and its state, are set to NaN. The token-serial kernel has NaN
// or an infinity there.
//
// What bounds it: the chain of chunks of a sequence; per chunk some 3200 mma.sync, the splits and three block barriers.
// 4 x 1500 tokens, 32 heads of 128 x 128: 437 us, token-serial 3943 us; 1 x 6000 tokens, 8 heads of 128 x 256: 680 / 7352 us
// (B200). The whole mixer on 6000 ragged tokens at width 4096: 7171 -> 1310 us.
#include <cuda_bf16.h>

#include "common/host_utils.h"
#include "seq/seq_common.cuh"
#include "seq/seq_mma.cuh"

namespace {
using namespace seqk;
typedef __nv_bfloat16 bf16_t;

constexpr int kC = 64;                              // tokens of a chunk
constexpr int kTiles = 10;                          // 16 x 16 tiles of a 64 x 64 matrix on and below the diagonal
// workspace of one (chunk, head), in 32-bit words: T and P as split mma A fragments [tile][part][lane][4], then per token
// (beta exp(L) / |k|, beta, q factor exp(L) / |q|, exp(L_63 - L) / |k|) and exp(L_63)
constexpr int kFrag = kTiles * 3 * 32 * 4;
constexpr int kUnit = 2 * kFrag + 4 * kC + 4;

__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// Chunk slots: sequence s owns slots from qsl[s] / 64 + s on (at least one per started 64 tokens), so that no scan over the
// sequences is needed; some slots stay empty.
__device__ __forceinline__ int chunk_base(const int* qsl, int s) { return qsl[s] / kC + s; }

// A, then K and Q, whose place T and the block product take
constexpr int prep_smem(int np) {
  const int kq = 2 * kC * (np + 8) * 2, tx = (kC * 68 + 32 * 36) * 4;
  return kC * 68 * 4 + (kq > tx ? kq : tx);
}

template <int NP>
__global__ void __launch_bounds__(128) delta_prep_kernel(
    const bf16_t* __restrict__ q, long ldq, const bf16_t* __restrict__ k, long ldk, const bf16_t* __restrict__ beta, long ldb,
    const bf16_t* __restrict__ a, long lda, const float* __restrict__ neg_a, const float* __restrict__ dt_bias,
    const int* __restrict__ qsl, int nseq, int H, int G, int D, int h0, int unit_qk, float q_scale, int min_len,
    uint32_t* __restrict__ work) {
  constexpr int LN = NP + 8, LA = 68, LX = 36;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* sA = reinterpret_cast<float*>(smem_raw);   // [64][LA]
  bf16_t* sKQ = reinterpret_cast<bf16_t*>(sA + kC * LA);
  __shared__ float sLh[kC], sLl[kC], sBeta[kC], sRk[kC], sRq[kC];
  const int u = blockIdx.x, h = h0 + blockIdx.y;
  int lo = 0, hi = nseq - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (chunk_base(qsl, mid) <= u) lo = mid; else hi = mid - 1;
  }
  const int q0 = qsl[lo], q1 = qsl[lo + 1], c = u - chunk_base(qsl, lo);
  const int t0 = q0 + c * kC;
  if (c < 0 || q1 - q0 < min_len || t0 >= q1) return;           // uniform over the block
  const int nt = min(kC, q1 - t0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g4 = lane >> 2, t4 = lane & 3, lq = lane >> 3, lr = lane & 7;
  const int grp = h / (H / G);
  bf16_t *sK = sKQ, *sQ = sKQ + kC * LN;
  for (int i = threadIdx.x; i < kC * (NP / 8); i += 128) {
    const int r = i / (NP / 8), e = (i % (NP / 8)) * 8;
    const bool ok = r < nt && e < D;
    const size_t row = t0 + (ok ? r : 0);
    cp16(sK + r * LN + e, k + row * ldk + (size_t)grp * D + (ok ? e : 0), ok);
    cp16(sQ + r * LN + e, q + row * ldq + (size_t)grp * D + (ok ? e : 0), ok);
  }
  asm volatile("cp.async.commit_group;");
  if (warp == 0) {                                  // tokens 2 lane, 2 lane + 1: write strengths and running log decays
    float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
    const float na = neg_a[h], db = dt_bias[h];
    if (2 * lane < nt) {
      a0 = na * softplus_f(to_f(a[(size_t)(t0 + 2 * lane) * lda + h]) + db);
      b0 = 1.0f / (1.0f + expf(-to_f(beta[(size_t)(t0 + 2 * lane) * ldb + h])));
    }
    if (2 * lane + 1 < nt) {
      a1 = na * softplus_f(to_f(a[(size_t)(t0 + 2 * lane + 1) * lda + h]) + db);
      b1 = 1.0f / (1.0f + expf(-to_f(beta[(size_t)(t0 + 2 * lane + 1) * ldb + h])));
    }
    // exp(-2000) is as much zero as exp(-inf), and differences of the sums stay numbers
    if (a0 < -2000.f) a0 = -2000.f;
    if (a1 < -2000.f) a1 = -2000.f;
    double run = (double)a0 + (double)a1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += up;
    }
    // not run - a1: a decay that is no number stays out of the token before it
    const double up = __shfl_up_sync(0xffffffffu, run, 1);
    const double l1 = run, l0 = (lane > 0 ? up : 0.0) + (double)a0;
    sLh[2 * lane] = (float)l0;
    sLl[2 * lane] = (float)(l0 - (double)(float)l0);
    sLh[2 * lane + 1] = (float)l1;
    sLl[2 * lane + 1] = (float)(l1 - (double)(float)l1);
    sBeta[2 * lane] = b0;
    sBeta[2 * lane + 1] = b1;
  }
  asm volatile("cp.async.wait_group 0;");
  __syncthreads();
  {                                                 // scales of the rows: two threads per token
    const int r = threadIdx.x >> 1, half = threadIdx.x & 1;
    float sk = 0.f, sq = 0.f;
    if (unit_qk) {
#pragma unroll 4
      for (int e = half * (NP / 2); e < (half + 1) * (NP / 2); e += 2) {
        const float2 kv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sK + r * LN + e));
        const float2 qv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sQ + r * LN + e));
        sk += kv.x * kv.x + kv.y * kv.y;
        sq += qv.x * qv.x + qv.y * qv.y;
      }
      sk += __shfl_xor_sync(0xffffffffu, sk, 1);
      sq += __shfl_xor_sync(0xffffffffu, sq, 1);
      sk = 1.0f / sqrtf(sk + 1e-6f);
      sq = q_scale / sqrtf(sq + 1e-6f);
    } else {
      sk = 1.0f;
      sq = q_scale;
    }
    if (half == 0) { sRk[r] = sk; sRq[r] = sq; }
  }
  __syncthreads();
  // ---- K K^T and Q K^T of this warp's 16 tokens against the tokens up to them
  float gk[8][4], gq[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) gk[i][0] = gk[i][1] = gk[i][2] = gk[i][3] = gq[i][0] = gq[i][1] = gq[i][2] = gq[i][3] = 0.f;
#pragma unroll 2
  for (int ks = 0; ks < NP / 16; ++ks) {
    uint32_t ak[4], aq[4];
    const int off = (warp * 16 + (lq & 1) * 8 + lr) * LN + ks * 16 + (lq >> 1) * 8;
    ldsm4(s_addr(sK + off), ak);
    ldsm4(s_addr(sQ + off), aq);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk <= warp) {
        uint32_t r[4];
        ldsm4(s_addr(sK + (kk * 16 + (lq >> 1) * 8 + lr) * LN + ks * 16 + (lq & 1) * 8), r);
        mma16816(gk[2 * kk], ak, r[0], r[1]);
        mma16816(gk[2 * kk + 1], ak, r[2], r[3]);
        mma16816(gq[2 * kk], aq, r[0], r[1]);
        mma16816(gq[2 * kk + 1], aq, r[2], r[3]);
      }
    }
  }
  uint32_t* unit = work + ((size_t)u * gridDim.y + blockIdx.y) * kUnit;
  const int ta = warp * 16 + g4, tb = ta + 8;
  auto put_frag = [&](uint32_t* at, int kk, const uint32_t (&fh)[4], const uint32_t (&fm)[4], const uint32_t (&fl)[4]) {
    uint4* dst = reinterpret_cast<uint4*>(at) + (warp * (warp + 1) / 2 + kk) * 96 + lane;
    dst[0] = make_uint4(fh[0], fh[1], fh[2], fh[3]);
    dst[32] = make_uint4(fm[0], fm[1], fm[2], fm[3]);
    dst[64] = make_uint4(fl[0], fl[1], fl[2], fl[3]);
  };
  {
    const float lha = sLh[ta], lla = sLl[ta], lhb = sLh[tb], llb = sLl[tb];
    const float ba = sBeta[ta] * sRk[ta], bb = sBeta[tb] * sRk[tb], qa = sRq[ta], qb = sRq[tb];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk <= warp) {
        uint32_t fh[4], fm[4], fl[4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float p[4];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = kk * 16 + half * 8 + 2 * t4 + e;
            const float lh = sLh[j], ll = sLl[j], rk = sRk[j];
            const float da = j <= ta ? expf((lha - lh) + (lla - ll)) * rk : 0.f;
            const float dbv = j <= tb ? expf((lhb - lh) + (llb - ll)) * rk : 0.f;
            sA[ta * LA + j] = j < ta ? ba * da * gk[2 * kk + half][e] : 0.f;
            sA[tb * LA + j] = j < tb ? bb * dbv * gk[2 * kk + half][2 + e] : 0.f;
            p[e] = j <= ta ? qa * da * gq[2 * kk + half][e] : 0.f;
            p[2 + e] = j <= tb ? qb * dbv * gq[2 * kk + half][2 + e] : 0.f;
          }
          split3(p[0], p[1], fh[2 * half], fm[2 * half], fl[2 * half]);
          split3(p[2], p[3], fh[2 * half + 1], fm[2 * half + 1], fl[2 * half + 1]);
        }
        put_frag(unit + kFrag, kk, fh, fm, fl);
      }
    }
  }
  __syncthreads();                                  // A is complete; K and Q are consumed
  // ---- T = (I + A)^-1: one column of a 32-row triangle per lane, then the block below
  float* sT = reinterpret_cast<float*>(sKQ);        // [64][LA]
  float* sX = sT + kC * LA;                         // [32][LX]
  if (warp < 2) {
    const float* Ad = sA + warp * 32 * (LA + 1);
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float s4[4] = {i == lane ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < i; ++j) s4[j & 3] = fmaf(-Ad[i * LA + j], x[j], s4[j & 3]);
      x[i] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) sT[(warp * 32 + i) * LA + warp * 32 + lane] = x[i];
  }
  __syncthreads();
  const int xi = threadIdx.x >> 2, xj = (threadIdx.x & 3) * 8;
  {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int s = 0; s < 32; ++s) {
      const float av = sA[(32 + xi) * LA + s];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(av, sT[s * LA + xj + e], acc[e]);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) sX[xi * LX + xj + e] = acc[e];
  }
  __syncthreads();
  {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // zero for s > xi, where sX[s] may be no number: a warp's eight rows end with its own eight columns
    for (int s0 = 0; s0 <= 8 * warp; s0 += 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int s = s0 + i;
        const float tv = sT[(32 + xi) * LA + 32 + s];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float x = sX[s * LX + xj + e];
          acc[e] = fmaf(-tv, s <= xi ? x : 0.f, acc[e]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) sT[(32 + xi) * LA + xj + e] = acc[e];
  }
  __syncthreads();
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    if (kk <= warp) {
      uint32_t fh[4], fm[4], fl[4];
#pragma unroll
      for (int f = 0; f < 4; ++f) {                 // rows ta, tb; columns 2 t4, then 8 + 2 t4
        const float* src = sT + (f & 1 ? tb : ta) * LA + kk * 16 + (f >> 1) * 8 + 2 * t4;
        split3(src[0], src[1], fh[f], fm[f], fl[f]);
      }
      put_frag(unit, kk, fh, fm, fl);
    }
  }
  if (threadIdx.x < kC) {
    const int t = threadIdx.x;
    const float end = sLh[kC - 1], endl = sLl[kC - 1], lh = sLh[t], ll = sLl[t], el = expf(lh + ll);
    float4* tok = reinterpret_cast<float4*>(unit + 2 * kFrag);
    tok[t] = make_float4(sBeta[t] * el * sRk[t], sBeta[t], el * sRq[t], expf((end - lh) + (endl - ll)) * sRk[t]);
    if (t == 0) reinterpret_cast<float*>(unit + 2 * kFrag + 4 * kC)[0] = expf(end + endl);
  }
}

template <int NP>
struct DeltaSmem {
  static constexpr int VT = 64, LN = NP + 8, LV = VT + 8;       // row strides that keep ldmatrix conflict-free
  static constexpr int K = 0, Q = K + 2 * kC * LN, V = Q + 2 * kC * LN, S = V + 2 * kC * LV, B = S + 3 * NP * LV,
                       U = B + 3 * kC * LV, W = U + 3 * kC * LV, kElems = W + 3 * kC * LV;
  static constexpr int kBytes = kElems * 2;
};

// products of a split A fragment with a split B operand: all but the three smallest of nine
__device__ __forceinline__ void mma_split(float (&d)[4], const uint4 (&a)[3], uint32_t h0, uint32_t h1, uint32_t m0,
                                          uint32_t m1, uint32_t l0, uint32_t l1) {
  const uint32_t ah[4] = {a[0].x, a[0].y, a[0].z, a[0].w}, am[4] = {a[1].x, a[1].y, a[1].z, a[1].w},
                 al[4] = {a[2].x, a[2].y, a[2].z, a[2].w};
  mma16816(d, al, h0, h1);
  mma16816(d, am, m0, m1);
  mma16816(d, ah, l0, l1);
  mma16816(d, am, h0, h1);
  mma16816(d, ah, m0, m1);
  mma16816(d, ah, h0, h1);
}

template <int NP>
__global__ void __launch_bounds__(256, 1) delta_chunk_kernel(
    const bf16_t* __restrict__ q, long ldq, const bf16_t* __restrict__ k, long ldk, const bf16_t* __restrict__ v, long ldv,
    float* __restrict__ state, const int* __restrict__ rec_slots, const int* __restrict__ seq_lens,
    const int* __restrict__ qsl, int H, int G, int D, int V, int h0, int min_len, const uint32_t* __restrict__ work,
    float* __restrict__ out) {
  using SM = DeltaSmem<NP>;
  constexpr int LN = SM::LN, LV = SM::LV, VT = SM::VT;
  constexpr int WM = NP / 16, WN = 8 / WM, NI = VT / 8 / WN;    // state: 16 rows x NI column tiles per warp
  extern __shared__ __align__(16) uint8_t smem_raw[];
  bf16_t* sm = reinterpret_cast<bf16_t*>(smem_raw);
  bf16_t *sS = sm + SM::S, *sB = sm + SM::B, *sU = sm + SM::U, *sW = sm + SM::W;
  __shared__ int s_bad[VT];                         // first token of the chunk whose B or U is no number, per column
  constexpr int kPS = NP * LV, kPT = kC * LV;       // one part of S, of a token operand

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // One block per SM, and a block is as long as its sequence: the longest start first (up to 32 sequences: each lane finds the rank
  // of one). 438, 989, 2093 and 2480 tokens, 32 heads of 128 x 128: 394 us in the batch's order, 351 so
  int s = blockIdx.z;
  if (gridDim.z <= 32) {
    const int n = gridDim.z, mine = lane < n ? qsl[lane + 1] - qsl[lane] : -1;
    int rank = 0;
    for (int i = 0; i < n; ++i) {
      const int other = __shfl_sync(0xffffffffu, mine, i);
      rank += other > mine || (other == mine && i < lane) ? 1 : 0;
    }
    s = __ffs(__ballot_sync(0xffffffffu, lane < n && rank == s)) - 1;
  }
  const int h = h0 + blockIdx.x, v0 = blockIdx.y * VT;
  const int q0 = qsl[s], q1 = qsl[s + 1];
  if (q1 <= q0 || q1 - q0 < min_len) return;        // uniform over the block
  const int g4 = lane >> 2, t4 = lane & 3, lq = lane >> 3, lr = lane & 7;
  const int grp = h / (H / G);
  const int wm = warp % WM, wn = warp / WM;
  const int tw = warp & 3, cb = (warp >> 2) * 4;    // token group, first of four column tiles
  const bool carried = state != nullptr && seq_lens[s] > q1 - q0;
  float* st = state != nullptr ? state + ((size_t)rec_slots[s] * H + h) * (size_t)D * V : nullptr;
  const bf16_t* kp = k + (size_t)grp * D;
  const bf16_t* qp = q + (size_t)grp * D;
  const bf16_t* vp = v + (size_t)h * V + v0;

  float S[NI][4];
#pragma unroll
  for (int ni = 0; ni < NI; ++ni)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = wm * 16 + g4 + 8 * (e >> 1), c = v0 + (wn * NI + ni) * 8 + 2 * t4 + (e & 1);
      S[ni][e] = (carried && n < D && c < V) ? st[(size_t)n * V + c] : 0.f;
    }
  auto put_state = [&]() {                          // the state as the products' operand
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t hi, mid, lo;
        split3(S[ni][2 * r], S[ni][2 * r + 1], hi, mid, lo);
        uint32_t* dst = reinterpret_cast<uint32_t*>(sS + (wm * 16 + g4 + 8 * r) * LV + (wn * NI + ni) * 8 + 2 * t4);
        dst[0] = hi;
        dst[kPS / 2] = mid;
        dst[kPS] = lo;
      }
  };
  auto fetch = [&](int t0, int buf) {
    const int nt = min(kC, q1 - t0);
    bf16_t *dK = sm + SM::K + buf * kC * LN, *dQ = sm + SM::Q + buf * kC * LN, *dV = sm + SM::V + buf * kC * LV;
    for (int i = threadIdx.x; i < kC * (NP / 8); i += 256) {
      const int r = i / (NP / 8), e = (i % (NP / 8)) * 8;
      const bool ok = r < nt && e < D;
      const size_t row = t0 + (ok ? r : 0);
      cp16(dK + r * LN + e, kp + row * ldk + (ok ? e : 0), ok);
      cp16(dQ + r * LN + e, qp + row * ldq + (ok ? e : 0), ok);
    }
    for (int i = threadIdx.x; i < kC * (VT / 8); i += 256) {
      const int r = i / (VT / 8), e = (i % (VT / 8)) * 8;
      const bool ok = r < nt && v0 + e < V;
      const size_t row = t0 + (ok ? r : 0);
      cp16(dV + r * LV + e, vp + row * ldv + (ok ? e : 0), ok);
    }
    asm volatile("cp.async.commit_group;");
  };
  if (threadIdx.x < VT) s_bad[threadIdx.x] = kC;    // visible to all after the first barrier of the loop
  put_state();
  fetch(q0, 0);
  const uint32_t* unit = work + ((size_t)chunk_base(qsl, s) * gridDim.x + blockIdx.x) * kUnit;
  const int ta = tw * 16 + g4, tb = ta + 8;

  for (int t0 = q0, buf = 0; t0 < q1; t0 += kC, buf ^= 1, unit += (size_t)gridDim.x * kUnit) {
    const int nt = min(kC, q1 - t0);
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();                                // this chunk's rows and S are in place, the last chunk is consumed
    if (t0 + kC < q1) fetch(t0 + kC, buf ^ 1);
    const bf16_t *sK = sm + SM::K + buf * kC * LN, *sQ = sm + SM::Q + buf * kC * LN, *sV = sm + SM::V + buf * kC * LV;
    const uint4* frag = reinterpret_cast<const uint4*>(unit) + (tw * (tw + 1) / 2) * 96 + lane;
    uint4 T[4][3];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      if (kk <= tw) { T[kk][0] = frag[kk * 96]; T[kk][1] = frag[kk * 96 + 32]; T[kk][2] = frag[kk * 96 + 64]; }
    const float4* tok = reinterpret_cast<const float4*>(unit + 2 * kFrag);
    const float4 wa = tok[ta], wb = tok[tb];
    const float g_end = reinterpret_cast<const float*>(unit + 2 * kFrag + 4 * kC)[0];
    // ---- K S and Q S of this warp's 16 tokens and 32 columns
    float ks_[4][4], qs_[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      ks_[i][0] = ks_[i][1] = ks_[i][2] = ks_[i][3] = qs_[i][0] = qs_[i][1] = qs_[i][2] = qs_[i][3] = 0.f;
#pragma unroll 2
    for (int kx = 0; kx < NP / 16; ++kx) {
      uint32_t ak[4], aq[4];
      const int off = (tw * 16 + (lq & 1) * 8 + lr) * LN + kx * 16 + (lq >> 1) * 8;
      ldsm4(s_addr(sK + off), ak);
      ldsm4(s_addr(sQ + off), aq);
#pragma unroll
      for (int part = 2; part >= 0; --part)
#pragma unroll
        for (int nv = 0; nv < 4; nv += 2) {
          uint32_t r[4];
          ldsm4_t(s_addr(sS + part * kPS + (kx * 16 + (lq & 1) * 8 + lr) * LV + (cb + nv) * 8 + (lq >> 1) * 8), r);
          mma16816(ks_[nv], ak, r[0], r[1]);
          mma16816(ks_[nv + 1], ak, r[2], r[3]);
          mma16816(qs_[nv], aq, r[0], r[1]);
          mma16816(qs_[nv + 1], aq, r[2], r[3]);
        }
    }
    uint32_t odd = 0;                               // places of this thread's 16 values that are no numbers
    auto number = [&](float x, int i, int e) {
      const bool ok = fabsf(x) <= 3.402823466e38f;
      odd |= ok ? 0u : 1u << (4 * i + e);
      return ok ? x : 0.f;
    };
    auto note = [&]() {
      for (uint32_t m = odd; m != 0; m &= m - 1) {
        const int at = __ffs(m) - 1;
        atomicMin(&s_bad[(cb + (at >> 2)) * 8 + 2 * t4 + (at & 1)], (at & 2) ? tb : ta);
      }
    };
    auto put_rows = [&](bf16_t* dst, int i, int row, float x, float y) {
      uint32_t hi, mid, lo;
      split3(x, y, hi, mid, lo);
      uint32_t* p = reinterpret_cast<uint32_t*>(dst + row * LV + (cb + i) * 8 + 2 * t4);
      p[0] = hi;
      p[kPT / 2] = mid;
      p[kPT] = lo;
    };
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int row = r ? tb : ta;
        const float bk = r ? wb.x : wa.x, be = r ? wb.y : wa.y;
        const float2 vv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sV + row * LV + (cb + i) * 8 + 2 * t4));
        put_rows(sB, i, row, number(be * vv.x - bk * ks_[i][2 * r], i, 2 * r),
                 number(be * vv.y - bk * ks_[i][2 * r + 1], i, 2 * r + 1));
      }
    if (odd != 0) note();
    const bool dirty = __syncthreads_or(odd != 0);  // B is complete
    uint4 P[4][3];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      if (kk <= tw) {
        const uint4* f = frag + kFrag / 4 + kk * 96;
        P[kk][0] = f[0]; P[kk][1] = f[32]; P[kk][2] = f[64];
      }
    // ---- U = T B
    float acc[4][4];
    auto tri = [&](const uint4 (&A)[4][3], const bf16_t* rhs) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        if (kk <= tw) {
#pragma unroll
          for (int nv = 0; nv < 4; nv += 2) {
            uint32_t rh[4], rm[4], rl[4];
            const bf16_t* src = rhs + (kk * 16 + (lq & 1) * 8 + lr) * LV + (cb + nv) * 8 + (lq >> 1) * 8;
            ldsm4_t(s_addr(src), rh);
            ldsm4_t(s_addr(src + kPT), rm);
            ldsm4_t(s_addr(src + 2 * kPT), rl);
            mma_split(acc[nv], A[kk], rh[0], rh[1], rm[0], rm[1], rl[0], rl[1]);
            mma_split(acc[nv + 1], A[kk], rh[2], rh[3], rm[2], rm[3], rl[2], rl[3]);
          }
        }
      }
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    tri(T, sB);
    if (dirty) {                                    // a decay or key that is no number is in T's rows, too
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = number(acc[i][e], i, e);
      if (odd != 0) note();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float w = r ? wb.w : wa.w;
        put_rows(sU, i, r ? tb : ta, acc[i][2 * r], acc[i][2 * r + 1]);
        put_rows(sW, i, r ? tb : ta, w * acc[i][2 * r], w * acc[i][2 * r + 1]);
      }
    __syncthreads();                                // U is complete
    // ---- o = exp(L) Q S + P U
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i][0] = wa.z * qs_[i][0]; acc[i][1] = wa.z * qs_[i][1];
      acc[i][2] = wb.z * qs_[i][2]; acc[i][3] = wb.z * qs_[i][3];
    }
    tri(P, sU);
    if (dirty) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if ((e < 2 ? ta : tb) >= s_bad[(cb + i) * 8 + 2 * t4 + (e & 1)]) acc[i][e] = __int_as_float(0x7fffffff);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int tk = r ? tb : ta, c = v0 + (cb + i) * 8 + 2 * t4;
        if (tk < nt && c < V)
          *reinterpret_cast<float2*>(out + (size_t)(t0 + tk) * H * V + (size_t)h * V + c) =
              make_float2(acc[i][2 * r], acc[i][2 * r + 1]);
      }
    // ---- S = exp(L_63) S + K^T W
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[ni][e] *= g_end;
#pragma unroll
    for (int kx = 0; kx < kC / 16; ++kx) {
      uint32_t ak[4];
      ldsm4_t(s_addr(sK + (kx * 16 + (lq >> 1) * 8 + lr) * LN + wm * 16 + (lq & 1) * 8), ak);
#pragma unroll
      for (int part = 2; part >= 0; --part)
#pragma unroll
        for (int ni = 0; ni < NI; ni += 2) {
          uint32_t r[4];
          ldsm4_t(s_addr(sW + part * kPT + (kx * 16 + (lq & 1) * 8 + lr) * LV + (wn * NI + ni) * 8 + (lq >> 1) * 8), r);
          mma16816(S[ni], ak, r[0], r[1]);
          mma16816(S[ni + 1], ak, r[2], r[3]);
        }
    }
    if (dirty) {
#pragma unroll
      for (int ni = 0; ni < NI; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (s_bad[(wn * NI + ni) * 8 + 2 * t4 + (e & 1)] < kC) S[ni][e] = __int_as_float(0x7fffffff);
    }
    put_state();
  }
  if (st != nullptr) {
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = wm * 16 + g4 + 8 * (e >> 1), c = v0 + (wn * NI + ni) * 8 + 2 * t4 + (e & 1);
        if (n < D && c < V) st[(size_t)n * V + c] = S[ni][e];
      }
  }
}

template <int NP>
int launch_delta(const bf16_t* q, long ldq, const bf16_t* k, long ldk, const bf16_t* v, long ldv, const bf16_t* beta,
                 long ldb, const bf16_t* a, long lda, const float* neg_a, const float* dt_bias, float* state,
                 const int* rec_slots, const int* seq_lens, const int* qsl, int ntok, int nseq, int H, int G, int D, int V,
                 int unit_qk, float q_scale, int min_len, int heads_at_once, uint32_t* work, float* out, cudaStream_t st) {
  using SM = DeltaSmem<NP>;
  static b200::PerDeviceOnce configured;
  if (configured.need()) {
    CUDA_CHECK_RET(cudaFuncSetAttribute(delta_chunk_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::kBytes));
    CUDA_CHECK_RET(cudaFuncSetAttribute(delta_prep_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem(NP)));
    configured.done();
  }
  const int slots = ntok / kC + nseq;
  for (int h0 = 0; h0 < H; h0 += heads_at_once) {
    const int nh = heads_at_once < H - h0 ? heads_at_once : H - h0;
    delta_prep_kernel<NP><<<dim3(slots, nh), 128, prep_smem(NP), st>>>(q, ldq, k, ldk, beta, ldb, a, lda, neg_a, dt_bias, qsl,
                                                                      nseq, H, G, D, h0, unit_qk, q_scale, min_len, work);
    delta_chunk_kernel<NP><<<dim3(nh, (V + SM::VT - 1) / SM::VT, nseq), 256, SM::kBytes, st>>>(
        q, ldq, k, ldk, v, ldv, state, rec_slots, seq_lens, qsl, H, G, D, V, h0, min_len, work, out);
  }
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}

}  // namespace

// bytes of workspace per (chunk slot, head); a batch has ntok / 64 + nseq slots
GLLM_EXPORT int gllm_delta_unit_bytes() { return kUnit * 4; }

// The gated delta rule of the sequences with at least min_len new tokens; returns 2 outside its envelope (the caller then
// uses the token-serial kernel): bf16 rows on 16-byte boundaries, D <= 128 and V multiples of 8.
// `work`: (ntok / 64 + nseq) * heads_at_once units.
GLLM_EXPORT int gllm_delta_chunk(const void* q, long ldq, const void* k, long ldk, const void* v, long ldv, const void* beta,
                                 long ldb, const void* a, long lda, const void* neg_a, const void* dt_bias, void* state,
                                 const void* rec_slots, const void* seq_lens, const void* qsl, int ntok, int nseq, int H,
                                 int G, int D, int V, int unit_qk, float q_scale, int min_len, int heads_at_once, void* work,
                                 void* out, void* stream) {
  if (nseq <= 0 || ntok <= 0) return 0;
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (D <= 0 || D > 128 || D % 8 != 0 || V % 8 != 0 || ldq % 8 != 0 || ldk % 8 != 0 || ldv % 8 != 0 || !al16(q) || !al16(k) ||
      !al16(v) || !al16(work) || (reinterpret_cast<uintptr_t>(out) & 7) != 0 || H % G != 0 || nseq > 65535)
    return 2;
  auto go = D <= 64 ? launch_delta<64> : launch_delta<128>;
  return go((const bf16_t*)q, ldq, (const bf16_t*)k, ldk, (const bf16_t*)v, ldv, (const bf16_t*)beta, ldb, (const bf16_t*)a,
            lda, (const float*)neg_a, (const float*)dt_bias, (float*)state, (const int*)rec_slots, (const int*)seq_lens,
            (const int*)qsl, ntok, nseq, H, G, D, V, unit_qk, q_scale, min_len, heads_at_once, (uint32_t*)work, (float*)out,
            (cudaStream_t)stream);
}
