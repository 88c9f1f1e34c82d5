// Expanding NVFP4 codes: shared by the packed-expert products (moe_fp4.cu, moe_fp4_tc.cu).
#pragma once
#include "ptx.cuh"
#include <cuda_fp8.h>

namespace ff {

// Eight codes of a word (low nibble first) times a scale: pairs (0, 4), (1, 5), (2, 6), (3, 7), one code per half. A code n alone in its half, times
// 2^6 + 2^12, has its magnitude at bits 8..6 and its sign at bit 15, and nothing of it reaches the other half: one multiplication, which the FMA pipe
// does, takes the place of two shifts and a merge on the ALU, whose half rate is what expanding is bound by (17 ALU operations a word
// with shifts, 9 so). The products of 32
// sequences over 128 experts of 4096 x 1536: 198 -> 187 us on average.
__device__ __forceinline__ void f4_expand8(uint32_t w, __nv_bfloat162 sv, uint32_t (&p)[4]) {
  constexpr uint32_t KEEP = 0x81C081C0u;
  const uint32_t h = w >> 8;
  p[0] = ((w & 0x000F000Fu) * 0x1040u) & KEEP;
  p[1] = ((w & 0x00F000F0u) * 0x0104u) & KEEP;
  p[2] = ((h & 0x000F000Fu) * 0x1040u) & KEEP;
  p[3] = ((h & 0x00F000F0u) * 0x0104u) & KEEP;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&p[i]), sv);
    p[i] = *reinterpret_cast<const uint32_t*>(&r);
  }
}

// two E4M3 scales -> BF16 pairs (each twice) times 2^118
__device__ __forceinline__ void f4_scale2(uint32_t c, __nv_bfloat162& s0, __nv_bfloat162& s1) {
  const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)c, __NV_E4M3);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
  constexpr float UP = 3.3230699894622897e35f;         // 2^118
  s0 = __float2bfloat162_rn(f.x * UP);
  s1 = __float2bfloat162_rn(f.y * UP);
}

}  // namespace ff
