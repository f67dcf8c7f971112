// Dynamic e4m3 quantisation of a group of 128 bf16 values with one fp32 scale (amax / 448): the step that gemm/gemm_fp8_block.cu and
// moe/moe_routing.cu share.
#pragma once

#include <cuda_fp8.h>

#include "ptx.cuh"

namespace b200 {

// Sixteen lanes hold a group, eight values each (bf16 pairs in `raw`): this lane's eight bytes; the same scale in all sixteen.
__device__ __forceinline__ uint2 fp8_quant_lane(const uint4& raw, float& scale) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  float f[8], amax = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 a = unpack_bf16(w[e]);
    f[2 * e] = a.x;
    f[2 * e + 1] = a.y;
    amax = fmaxf(amax, fmaxf(fabsf(a.x), fabsf(a.y)));
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  amax = fmaxf(amax, 1e-10f);
  scale = amax / 448.f;
  const float inv = 1.f / scale;
  __align__(8) __nv_fp8_e4m3 o8[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) o8[e] = __nv_fp8_e4m3(f[e] * inv);
  return *reinterpret_cast<uint2*>(o8);
}

}  // namespace b200
