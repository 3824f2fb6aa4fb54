// Codes of a quantisation group to the fp16 operands of the tensor-core projections (gemm_tc.cu, gemm_pair.cu).
#pragma once
#include "common.cuh"

namespace im {

// 8 nibbles of a word -> 8 fp16 values (q - z) * s in memory order.  c = 1024 + z, exact for integer z in
// [-1024, 1023]: 0x6400 | q is the fp16 number 1024 + q, the subtraction is exact, the product is rounded once.
__device__ __forceinline__ uint4 dequant8_fast(uint32_t w, __half2 c, __half2 s) {
    constexpr uint32_t M = 0x000F000Fu, E = 0x64006400u;
    uint32_t h04 = (w & M) | E, h15 = ((w >> 4) & M) | E, h26 = ((w >> 8) & M) | E, h37 = ((w >> 12) & M) | E;
    __half2 v04 = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&h04), c), s);
    __half2 v15 = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&h15), c), s);
    __half2 v26 = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&h26), c), s);
    __half2 v37 = __hmul2(__hsub2(*reinterpret_cast<__half2 *>(&h37), c), s);
    const uint32_t a = *reinterpret_cast<uint32_t *>(&v04), b = *reinterpret_cast<uint32_t *>(&v15);
    const uint32_t cc = *reinterpret_cast<uint32_t *>(&v26), d = *reinterpret_cast<uint32_t *>(&v37);
    return make_uint4(__byte_perm(a, b, 0x5410), __byte_perm(cc, d, 0x5410), __byte_perm(a, b, 0x7632), __byte_perm(cc, d, 0x7632));
}
// 8-bit codes: the 8 bytes of two words -> 8 fp16 values (q - z) * s in memory order.  0x6400 | q is 1024 + q for q < 1024.
__device__ __forceinline__ uint4 dequant8b_fast(uint32_t w0, uint32_t w1, __half2 c, __half2 s) {
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
