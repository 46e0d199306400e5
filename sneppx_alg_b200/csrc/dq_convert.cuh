// Packed weights of the dequant GEMMs as bf16 values without scale, which is exact for both formats.
#pragma once
#include <cuda_fp8.h>
#include "tc_common.cuh"

namespace sx {

// Eight nibbles (low first) -> four packed bf16 pairs of q - 8. 0x4300 | q is 128 + q in bf16, exactly.
__device__ __forceinline__ void int4x8_to_bf16(uint32_t w, uint32_t* o) {
  const uint32_t lo = w & 0x0f0f0f0fu, hi = (w >> 4) & 0x0f0f0f0fu;      // elements 0 2 4 6 / 1 3 5 7
  const uint32_t a = __byte_perm(lo, hi, 0x5140), b = __byte_perm(lo, hi, 0x7362);   // 0 1 2 3 / 4 5 6 7
  const uint32_t m = 0x43434343u;
  uint32_t t[4] = {__byte_perm(a, m, 0x4140), __byte_perm(a, m, 0x4342), __byte_perm(b, m, 0x4140), __byte_perm(b, m, 0x4342)};
  const __nv_bfloat162 off = __floats2bfloat162_rn(136.f, 136.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 v = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&t[i]), off);
    o[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
}
// Four e4m3 bytes -> two packed bf16 pairs (e4m3 has three mantissa bits: exact).
__device__ __forceinline__ void e4m3x4_to_bf16(uint32_t w, uint32_t* o) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> (16 * i)), __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    o[i] = pack_bf16x2(f.x, f.y);
  }
}

}  // namespace sx
