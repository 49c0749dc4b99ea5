// int8 quantisation of bf16 rows, eight elements at a time (bitvla_lm.cu, bitvla_vit.cu).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace vb {

// clamp(rne(x), -128, 127) as int8 in the low byte; NaN -> -128.  One conversion saturates and rounds; the maximum in front of it is there
// for NaN, which the conversion alone would turn into 0.
__device__ __forceinline__ uint32_t sat_s8(float x) {
    uint32_t r;
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(r) : "f"(fmaxf(x, -128.0f)));
    return r;
}

// Eight bf16 -> eight int8, q = clamp(rne(y * qs), -128, 127).  The row passes around the ternary products are bound by issue slots
// (16 sequences x 300 tokens: 4,800 rows of up to 6,912), and this is their longest stretch: 3.75 instructions an element
// (mul, max, cvt, three byte permutations per four) instead of 8.
__device__ __forceinline__ uint2 quant8_bf16(const uint4 &y, float qs) {
    const uint32_t w[4] = {y.x, y.y, y.z, y.w};
    uint32_t p[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[e]));
        p[e] = __byte_perm(sat_s8(f.x * qs), sat_s8(f.y * qs), 0x0040);
    }
    return make_uint2(__byte_perm(p[0], p[1], 0x5410), __byte_perm(p[2], p[3], 0x5410));
}

}  // namespace vb
