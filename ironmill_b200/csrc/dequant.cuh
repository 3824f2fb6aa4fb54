// Codes of a quantisation group to the fp16 operands of the tensor-core projections (gemm_tc.cu, gemm_pair.cu).
#pragma once
#include "common.cuh"

namespace im {

// (v & m) | 0x6400 in both halves as one instruction: with two constants the compiler makes two of it, and the logic pipe runs at half rate.
__device__ __forceinline__ uint32_t half_exponent() {
    uint32_t e;
    asm volatile("mov.b32 %0, 0x64006400;" : "=r"(e));
    return e;
}
__device__ __forceinline__ __half2 place_codes(uint32_t v, uint32_t m, uint32_t e) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(v), "r"(m), "r"(e));
    return *reinterpret_cast<__half2 *>(&d);
}
// The conversions below are the published ones of mixed-precision GEMMs: a code in the mantissa of an fp16 exponent (Kim et al., "Who Says Elephants Can't
// Run", 2022), the upper nibble brought down by an fma (Frantar et al., MARLIN, 2024); here with zero points and the exactness that they leave.
// (scale, zero) of a row and group for them: c = 1024 + z, d = -(64 + z).  0x6400 | q is the fp16 number 1024 + q, 0x6400 | 16 q the number
// 1024 + 16 q; where z is a whole or half number of at most 512 (plain), q - z = (1024 + q) - c = (1024 + 16 q) / 16 + d is exact for every code,
// and the product with s is rounded once.
struct GroupScale {
    __half2 c, d, s;
    bool plain;
};
__device__ __forceinline__ GroupScale group_scale(__half2 sz) {
    const __half2 z = __high2half2(sz), k = __float2half2_rn(1024.0f), c = __hadd2(z, k);
    return GroupScale{c, __hsub2(__float2half2_rn(-64.0f), z), __low2half2(sz), __hbeq2(__hsub2(c, k), z) && __hble2(__habs2(z), __float2half2_rn(512.0f))};
}
// The same by way of f32, for 8-bit codes in the pair kernel (whole zero points only): 2048 tokens, 14336 x 4096, 218 us against 220.5 with the above.
__device__ __forceinline__ GroupScale group_scale_f32(__half2 sz) {
    const float z = __high2float(sz);
    const __half2 c = __float2half2_rn(1024.0f + z);
    return GroupScale{c, c, __low2half2(sz), z == rintf(z) && z >= -1024.0f && z <= 1023.0f};
}
// 8 nibbles of a word -> 8 fp16 values (q - z) * s in memory order.
__device__ __forceinline__ uint4 dequant8_fast(uint32_t w, const GroupScale &g, uint32_t e) {
    const __half2 c = g.c, d = g.d, s = g.s;
    constexpr uint32_t M = 0x000F000Fu, MH = 0x00F000F0u;
    const __half2 sixteenth = __float2half2_rn(0.0625f);
    const uint32_t u = w >> 8;
    const __half2 v04 = __hmul2(__hsub2(place_codes(w, M, e), c), s), v15 = __hmul2(__hfma2(place_codes(w, MH, e), sixteenth, d), s);
    const __half2 v26 = __hmul2(__hsub2(place_codes(u, M, e), c), s), v37 = __hmul2(__hfma2(place_codes(u, MH, e), sixteenth, d), s);
    const uint32_t a = *reinterpret_cast<const uint32_t *>(&v04), b = *reinterpret_cast<const uint32_t *>(&v15);
    const uint32_t cc = *reinterpret_cast<const uint32_t *>(&v26), dd = *reinterpret_cast<const uint32_t *>(&v37);
    return make_uint4(__byte_perm(a, b, 0x5410), __byte_perm(cc, dd, 0x5410), __byte_perm(a, b, 0x7632), __byte_perm(cc, dd, 0x7632));
}
// 8-bit codes: the 8 bytes of two words -> 8 fp16 values (q - z) * s in memory order.  0x6400 | q is 1024 + q for q < 1024.
__device__ __forceinline__ uint4 dequant8b_fast(uint32_t w0, uint32_t w1, const GroupScale &g) {
    const __half2 c = g.c, s = g.s;
    uint32_t h[4] = {__byte_perm(w0, 0x64u, 0x4140), __byte_perm(w0, 0x64u, 0x4342), __byte_perm(w1, 0x64u, 0x4140), __byte_perm(w1, 0x64u, 0x4342)};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __half2 v = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&h[i]), c), s);
        o[i] = *reinterpret_cast<const uint32_t *>(&v);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ uint4 dequant8b_slow(uint32_t w0, uint32_t w1, float z, float s) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t w = i < 2 ? w0 : w1;
        const float lo = ((float)((w >> (16 * (i & 1))) & 255u) - z) * s, hi = ((float)((w >> (16 * (i & 1) + 8)) & 255u) - z) * s;
        o[i] = (uint32_t)__half_as_ushort(__float2half_rn(lo)) | ((uint32_t)__half_as_ushort(__float2half_rn(hi)) << 16);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ uint4 dequant8_slow(uint32_t w, float z, float s) {  // any zero point: f32, one rounding
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float lo = ((float)((w >> (8 * i)) & 15u) - z) * s, hi = ((float)((w >> (8 * i + 4)) & 15u) - z) * s;
        o[i] = (uint32_t)__half_as_ushort(__float2half_rn(lo)) | ((uint32_t)__half_as_ushort(__float2half_rn(hi)) << 16);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace im
