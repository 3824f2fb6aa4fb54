// Per-group affine quantization + INT4 packing on the GPU, bit-exact with the reference's
// CPU quantizer: quantize_affine / emit_per_group
// (crates/mil-rs/src/ir/passes/affine_quantize.rs:256-298,420-453), pack_int4
// (crates/mil-rs/src/ir/passes/int4_pack.rs:20-34) and the AWQ column pre-scale
// (crates/ironmill-compile/src/weights/quantized.rs:925-940).
//
// Every float operation is an explicit round-to-nearest intrinsic so that no multiply-add is
// contracted; roundf() is round-half-away-from-zero like Rust's f32::round.
#include <float.h>

#include "common.cuh"

namespace im {

__device__ __forceinline__ float load_weight(const __half *w, const __half *awq, size_t idx, size_t col) {
    float x = __half2float(w[idx]);
    if (awq) x = __fmul_rn(x, __half2float(awq[col]));
    return x;
}

// ---- one pass over the weights: groups of 8 * L columns, rows a multiple of 8 columns, 16-byte aligned ------------------
// Bound: HBM (2 bytes in, 0.5 or 1 byte and 8 bytes per group out), as long as issue keeps up: at 14336 x 4096 an instruction per element is
// 1.7 us of a floor of 23.  A lane owns C octets of a group (every P = L / C-th, so that neighbouring lanes read neighbouring octets): the
// group's scale and zero point - two divisions, and shuffles among P lanes - are worked out for 32 elements at a time.  (Two rows to a lane, so that a
// vector of AWQ factors serves both: 16 warps an SM instead of 32, 55 us against 47.)  Octets past the end of a row and rows past the last repeat the
// last one and are not stored.  4-bit with AWQ, 14336 x 4096: 90 us with one octet to a lane (about 27 instructions per element) -> 52 (about 17; issue slots 57 % busy).
//
// Codes without a division per element: t = x * (1 / scale) + zp differs from the defining fl(fl(x / scale) + zp) by less
// than 2^-20 (|x / scale| + |zp| + 1), so the two round to the same integer unless t lies that close to a half; an octet
// with such a value (or a magnitude past 2^21) is recomputed by the definition.  An octet without one needs no clamp: x lies between the group's
// extrema, so t is at most a half outside 0 .. qmax, give or take that error.  Groups with a value that is not finite take quantize_row_any.  Of a minimum
// of zero the first place counts (its sign shows in the zero point): looked for only in warps that have one.  Nothing but zeros, 14336 x 4096, 4-bit with AWQ:
// 176 us by quantize_row_any, 68 so.

__device__ __forceinline__ unsigned quantize_one(float x, float scale, float zp, float qmax);

__device__ __forceinline__ float min3(float a, float b, float c) {  // NaN if one of them is
    float d;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Weight times AWQ factor: a product of two fp16 values is exact in f32.
template <bool AWQ>
__device__ __forceinline__ void quantize_values(const uint4 w, const uint4 a, float (&x)[8]) {
    const unsigned u[4] = {w.x, w.y, w.z, w.w}, v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&u[j]));
        x[2 * j] = f.x;
        x[2 * j + 1] = f.y;
        if (AWQ) {
            const float2 g = __half22float2(*reinterpret_cast<const __half2 *>(&v[j]));
            x[2 * j] = __fmul_rn(f.x, g.x);
            x[2 * j + 1] = __fmul_rn(f.y, g.y);
        }
    }
}
__device__ __forceinline__ void quantize_scale(float mn, float mx, bool finite, float qmax, float &scale, float &zp) {
    if (!finite) {  // no finite value in the group
        scale = 1.0f;
        zp = 0.0f;
    } else if (fabsf(__fsub_rn(mx, mn)) < FLT_EPSILON) {
        scale = 1.0f;
        zp = roundf(-mn);
    } else {
        scale = __fdiv_rn(__fsub_rn(mx, mn), qmax);
        zp = roundf(__fdiv_rn(-mn, scale));
    }
}
template <int BITS>
__device__ __forceinline__ void store_codes(uint8_t *packed, size_t octet, const float (&c)[8]) {
    if (BITS == 4) {
        // four codes in one exact f32 sum, the lower column in the lower nibble
        const float lo = fmaf(fmaf(fmaf(c[3], 16.0f, c[2]), 16.0f, c[1]), 16.0f, c[0]), hi = fmaf(fmaf(fmaf(c[7], 16.0f, c[6]), 16.0f, c[5]), 16.0f, c[4]);
        reinterpret_cast<unsigned *>(packed)[octet] = __byte_perm(__float_as_uint(lo + 8388608.0f), __float_as_uint(hi + 8388608.0f), 0x5410);
    } else {
        const float s0 = fmaf(c[1], 256.0f, c[0]) + 8388608.0f, s1 = fmaf(c[3], 256.0f, c[2]) + 8388608.0f, s2 = fmaf(c[5], 256.0f, c[4]) + 8388608.0f,
                    s3 = fmaf(c[7], 256.0f, c[6]) + 8388608.0f;
        reinterpret_cast<uint2 *>(packed)[octet] = make_uint2(__byte_perm(__float_as_uint(s0), __float_as_uint(s1), 0x5410), __byte_perm(__float_as_uint(s2), __float_as_uint(s3), 0x5410));
    }
}

// A lane's octets of a group by the definition, whatever its values: all lanes of the warp.  live: how many of them lie in the row (the others repeat the last one).
template <int BITS, int C, bool AWQ>
__device__ __noinline__ void quantize_row_any(const uint4 (&w)[C], const uint4 (&a)[C], int lane_of_group, int P, int live, size_t octet0, bool store, float *scale_out,
                                              float *zp_out, uint8_t *packed) {
    constexpr float qmax = BITS == 4 ? 15.0f : 255.0f;
    float mn = INFINITY, mx = -INFINITY;
    unsigned imn = 0xffffffffu, imx = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < C; i++) {
        float x[8];
        quantize_values<AWQ>(w[i], a[i], x);
        const unsigned at = (unsigned)(lane_of_group + i * P) * 8;
        for (int j = 0; j < 8; j++)
            if (isfinite(x[j])) {
                if (x[j] < mn) { mn = x[j]; imn = at + j; }
                if (x[j] > mx) { mx = x[j]; imx = at + j; }
            }
    }
    for (int o = P >> 1; o > 0; o >>= 1) {
        const float omn = __shfl_xor_sync(0xffffffffu, mn, o), omx = __shfl_xor_sync(0xffffffffu, mx, o);
        const unsigned oimn = __shfl_xor_sync(0xffffffffu, imn, o), oimx = __shfl_xor_sync(0xffffffffu, imx, o);
        if (omn < mn || (omn == mn && oimn < imn)) { mn = omn; imn = oimn; }
        if (omx > mx || (omx == mx && oimx < imx)) { mx = omx; imx = oimx; }
    }
    const bool finite = isfinite(mn) && isfinite(mx);
    float scale, zp;
    quantize_scale(mn, mx, finite, qmax, scale, zp);
    if (!store) return;
    if (lane_of_group == 0) {
        *scale_out = scale;
        *zp_out = zp;
    }
#pragma unroll
    for (int i = 0; i < C; i++) {
        float x[8], c[8];
        quantize_values<AWQ>(w[i], a[i], x);
        for (int j = 0; j < 8; j++) c[j] = finite ? (float)quantize_one(x[j], scale, zp, qmax) : 0.0f;
        if (i < live) store_codes<BITS>(packed, octet0 + i * P, c);
    }
}

// Place of a group's first zero, its sign in the lowest bit: all lanes of the warp.  (Inlined, it takes ordinary groups 2 % of their time.)
template <int C, bool AWQ>
__device__ __noinline__ unsigned quantize_first_zero(const uint4 (&w)[C], const uint4 (&a)[C], unsigned lane_of_group, int P) {
    unsigned first = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < C; i++) {
        float x[8];
        quantize_values<AWQ>(w[i], a[i], x);
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (x[j] == 0.0f) first = min(first, ((lane_of_group + (unsigned)(i * P)) * 8 + j) * 2 + (__float_as_uint(x[j]) >> 31));
    }
    for (int o = P >> 1; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
    return first;
}

template <int BITS, int C, bool AWQ>
__global__ void __launch_bounds__(256, 4) quantize_groups_kernel(const __half *__restrict__ w, const __half *__restrict__ awq, size_t rows, unsigned K, int P,
                                                                              unsigned G, float *__restrict__ scales, float *__restrict__ zps, uint8_t *__restrict__ packed) {
    constexpr float qmax = BITS == 4 ? 15.0f : 255.0f;
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low mantissa bits
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, at = i >> (__ffs(P) - 1);  // the group's number
    const size_t row = (at >> 32) == 0 ? (unsigned)at / G : at / G;
    const unsigned g = (unsigned)(at - row * G), p = (unsigned)i & (unsigned)(P - 1);
    const bool store = row < rows;
    const unsigned octets = K / 8, o0 = g * (unsigned)(P * C) + p;  // this lane's octets of the row: o0, o0 + P, ...
    const int live = o0 >= octets ? 0 : min(C, (int)((octets - 1 - o0) / (unsigned)P) + 1);
    const uint4 *src = reinterpret_cast<const uint4 *>(w) + min(row, rows - 1) * octets;
    const size_t octet0 = row * octets + o0;
    uint4 a[C], raw[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
        raw[c] = ldg_stream_v4(src + min(o0 + c * (unsigned)P, octets - 1));
        a[c] = make_uint4(0, 0, 0, 0);
        if (AWQ) a[c] = __ldg(reinterpret_cast<const uint4 *>(awq) + min(o0 + c * (unsigned)P, octets - 1));
    }
    float mn = INFINITY, mx = -INFINITY;  // NaN or infinite with a value that is not finite
#pragma unroll
    for (int c = 0; c < C; c++) {
        float x[8];
        quantize_values<AWQ>(raw[c], a[c], x);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            mn = min3(mn, x[j], x[j + 1]);
            mx = max3(mx, x[j], x[j + 1]);
        }
    }
    for (int o = P >> 1; o > 0; o >>= 1) {
        mn = min3(mn, mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (__any_sync(0xffffffffu, !isfinite(mn) || !isfinite(mx) || mn == 0.0f)) {
        if (__any_sync(0xffffffffu, !isfinite(mn) || !isfinite(mx))) {
            quantize_row_any<BITS, C, AWQ>(raw, a, (int)p, P, live, octet0, store, scales + at, zps + at, packed);
            return;
        }
        const unsigned first = quantize_first_zero<C, AWQ>(raw, a, p, P);
        if (mn == 0.0f) mn = __uint_as_float(first << 31);
    }
    float scale, zp;
    quantize_scale(mn, mx, true, qmax, scale, zp);
    if (!store) return;
    if (p == 0) {
        scales[at] = scale;
        zps[at] = zp;
    }
    const float inv = __fdividef(1.0f, scale);
    // t is within [mn, mx] / scale + zp; the largest magnitude on the way bounds the rounding of both forms
    const float mag = fmaxf(fabsf(mn), fabsf(mx)) * inv + fabsf(zp) + 1.0f;
    const float near_half = mag < 2097152.0f ? 0.5f - mag * 0x1p-20f : 0.0f;
#pragma unroll
    for (int c = 0; c < C; c++) {
        float x[8], q[8], far = 0.0f;
        quantize_values<AWQ>(raw[c], a[c], x);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const float t0 = fmaf(x[j], inv, zp), t1 = fmaf(x[j + 1], inv, zp);
            q[j] = __fsub_rn(__fadd_rn(t0, kMagic), kMagic);
            q[j + 1] = __fsub_rn(__fadd_rn(t1, kMagic), kMagic);
            far = max3(far, fabsf(t0 - q[j]), fabsf(t1 - q[j + 1]));
        }
        if (!(far < near_half)) {
#pragma unroll
            for (int j = 0; j < 8; j++) q[j] = (float)quantize_one(x[j], scale, zp, qmax);
        }
        if (c < live) store_codes<BITS>(packed, octet0 + c * (unsigned)P, q);
    }
}

template <int BITS, int C>
static int quantize_groups(const __half *w, const __half *awq, size_t rows, size_t K, int P, size_t G, float *scales, float *zps, uint8_t *packed, cudaStream_t st) {
    const size_t blocks = (rows * G * P + 255) / 256;
    if (blocks > 0x7fffffff) return IM_ERR_BOUNDS;
    if (awq) quantize_groups_kernel<BITS, C, true><<<(unsigned)blocks, 256, 0, st>>>(w, awq, rows, (unsigned)K, P, (unsigned)G, scales, zps, packed);
    else quantize_groups_kernel<BITS, C, false><<<(unsigned)blocks, 256, 0, st>>>(w, awq, rows, (unsigned)K, P, (unsigned)G, scales, zps, packed);
    IM_CUDA_CHECK(cudaGetLastError());
    return IM_OK;
}
template <int BITS>
static int quantize_groups(const __half *w, const __half *awq, size_t rows, size_t K, int L, size_t G, float *scales, float *zps, uint8_t *packed, cudaStream_t st) {
    if (L >= 4) return quantize_groups<BITS, 4>(w, awq, rows, K, L / 4, G, scales, zps, packed, st);
    if (L == 2) return quantize_groups<BITS, 2>(w, awq, rows, K, 1, G, scales, zps, packed, st);
    return quantize_groups<BITS, 1>(w, awq, rows, K, 1, G, scales, zps, packed, st);
}

// ---- any other shape: parameters first, then the codes -------------------------------------------------------------------
// One warp per (row, group): min/max over the finite values, then scale and zero point.
// The CPU loop keeps the first of equal extrema (strict compares); that only matters for
// the sign of a zero, and is reproduced by carrying the element index through the reduction.
__global__ void quantize_params_kernel(const __half *__restrict__ w, const __half *__restrict__ awq,
                                       size_t rows, size_t K, int gs, int G, float qmax,
                                       float *__restrict__ scales, float *__restrict__ zps) {
    size_t gid = (size_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    int lane = threadIdx.x & 31;
    if (gid >= rows * (size_t)G) return;
    size_t r = gid / G;
    int g = (int)(gid % G);
    size_t c0 = (size_t)g * gs, c1 = c0 + gs < K ? c0 + gs : K;

    float mn = INFINITY, mx = -INFINITY;
    unsigned imn = 0xffffffffu, imx = 0xffffffffu;
    for (size_t c = c0 + lane; c < c1; c += 32) {
        float x = load_weight(w, awq, r * K + c, c);
        if (isfinite(x)) {
            if (x < mn) { mn = x; imn = (unsigned)(c - c0); }
            if (x > mx) { mx = x; imx = (unsigned)(c - c0); }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float omn = __shfl_xor_sync(0xffffffffu, mn, o);
        unsigned oimn = __shfl_xor_sync(0xffffffffu, imn, o);
        float omx = __shfl_xor_sync(0xffffffffu, mx, o);
        unsigned oimx = __shfl_xor_sync(0xffffffffu, imx, o);
        if (omn < mn || (omn == mn && oimn < imn)) { mn = omn; imn = oimn; }
        if (omx > mx || (omx == mx && oimx < imx)) { mx = omx; imx = oimx; }
    }
    if (lane == 0) {
        float scale, zp;
        if (!isfinite(mn) || !isfinite(mx)) {
            scale = 1.0f;
            zp = 0.0f;
        } else if (fabsf(__fsub_rn(mx, mn)) < FLT_EPSILON) {
            scale = 1.0f;
            zp = roundf(-mn);
        } else {
            scale = __fdiv_rn(__fsub_rn(mx, mn), qmax);
            zp = roundf(__fdiv_rn(-mn, scale));
        }
        scales[gid] = scale;
        zps[gid] = zp;
    }
}

// A group without any finite value quantizes to all zeros (the CPU routine returns early with
// a zero vector); a non-finite element of any other group saturates through the clamp.  Only
// non-finite elements take the rescan, so the common path stays one pass.
__device__ __noinline__ bool group_has_finite(const __half *w, const __half *awq, size_t row_base, size_t c0, size_t c1) {
    for (size_t c = c0; c < c1; c++)
        if (isfinite(load_weight(w, awq, row_base + c, c))) return true;
    return false;
}

__device__ __forceinline__ unsigned quantize_one(float x, float scale, float zp, float qmax) {
    float t = roundf(__fadd_rn(__fdiv_rn(x, scale), zp));
    if (t != t) return 0u;  // NaN saturates to 0 like Rust's `as u8`
    t = fminf(fmaxf(t, 0.0f), qmax);
    return (unsigned)t;
}

__device__ __forceinline__ unsigned quantize_elem(const __half *w, const __half *awq, size_t i, size_t K, int gs, int G,
                                                  const float *scales, const float *zps, float qmax) {
    // 64-bit division costs more than the rest of the element: 32 bits where they hold the index
    const bool narrow = ((i | K) >> 32) == 0;
    const size_t r = narrow ? (unsigned)i / (unsigned)K : i / K, c = i - r * K;
    const size_t g = narrow ? (unsigned)c / (unsigned)gs : c / gs, pi = r * G + g;
    const float x = load_weight(w, awq, i, c);
    if (!isfinite(x)) {
        const size_t c0 = g * gs, c1 = c0 + gs < K ? c0 + gs : K;
        if (!group_has_finite(w, awq, r * K, c0, c1)) return 0u;
    }
    return quantize_one(x, scales[pi], zps[pi], qmax);
}

// 4-bit: one thread per output byte = flat element pair (2p, 2p+1); the pair may straddle
// groups or rows when K is odd, so each element looks up its own group.
__global__ void quantize_codes_int4_kernel(const __half *__restrict__ w, const __half *__restrict__ awq,
                                           size_t total, size_t K, int gs, int G,
                                           const float *__restrict__ scales, const float *__restrict__ zps,
                                           uint8_t *__restrict__ packed) {
    size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t nbytes = (total + 1) / 2;
    if (p >= nbytes) return;
    unsigned byte = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        size_t i = 2 * p + h;
        if (i < total) {
            unsigned q = quantize_elem(w, awq, i, K, gs, G, scales, zps, 15.0f);
            byte |= (q & 0xFu) << (4 * h);
        }
    }
    packed[p] = (uint8_t)byte;
}

__global__ void quantize_codes_int8_kernel(const __half *__restrict__ w, const __half *__restrict__ awq,
                                           size_t total, size_t K, int gs, int G,
                                           const float *__restrict__ scales, const float *__restrict__ zps,
                                           uint8_t *__restrict__ out) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    out[i] = (uint8_t)quantize_elem(w, awq, i, K, gs, G, scales, zps, 255.0f);
}

}  // namespace im

IM_EXPORT int im_cuda_quantize_affine(const void *w_dev, const void *awq_dev, size_t rows, size_t K,
                                      int group_size, int bit_width, void *packed_dev, float *scales_dev,
                                      float *zps_dev, void *stream) {
    IM_GUARD_BEGIN
    IM_REQUIRE(bit_width == 4 || bit_width == 8, "bit_width must be 4 or 8, got %d", bit_width);
    IM_REQUIRE(group_size > 0, "group_size must be positive");
    size_t total = rows * K;
    if (total == 0) return IM_OK;  // empty input: nothing to write
    IM_REQUIRE(w_dev && packed_dev && scales_dev && zps_dev, "NULL device pointer");
    size_t G = (K + group_size - 1) / group_size;
    IM_REQUIRE(G <= 0x7fffffff && rows * G / 8 + 1 <= 0x7fffffff, "tensor too large");
    cudaStream_t st = im::as_stream(stream);
    const __half *w = static_cast<const __half *>(w_dev);
    const __half *awq = static_cast<const __half *>(awq_dev);
    // One pass where octets of columns never straddle a group: the group is 8 L columns with L a power of two up to 32, rows are
    // a multiple of 8 columns, and every vector access is aligned.  Anything else takes the two kernels below.
    const int L = group_size / 8;
    if (group_size % 8 == 0 && L <= 32 && (L & (L - 1)) == 0 && K % 8 == 0 && K < ((size_t)1 << 31) && reinterpret_cast<uintptr_t>(w_dev) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(awq_dev) % 16 == 0 && reinterpret_cast<uintptr_t>(packed_dev) % (bit_width == 4 ? 4 : 8) == 0) {
        uint8_t *packed = static_cast<uint8_t *>(packed_dev);
        const int rc = bit_width == 4 ? im::quantize_groups<4>(w, awq, rows, K, L, G, scales_dev, zps_dev, packed, st)
                                      : im::quantize_groups<8>(w, awq, rows, K, L, G, scales_dev, zps_dev, packed, st);
        if (rc != IM_ERR_BOUNDS) return rc;
    }
    size_t ngroups = rows * G;
    const int warps_per_block = 8;
    im::quantize_params_kernel<<<(unsigned)((ngroups + warps_per_block - 1) / warps_per_block), warps_per_block * 32, 0, st>>>(
        w, awq, rows, K, group_size, (int)G, bit_width == 4 ? 15.0f : 255.0f, scales_dev, zps_dev);
    if (bit_width == 4) {
        size_t nbytes = (total + 1) / 2;
        im::quantize_codes_int4_kernel<<<(unsigned)((nbytes + 255) / 256), 256, 0, st>>>(
            w, awq, total, K, group_size, (int)G, scales_dev, zps_dev, static_cast<uint8_t *>(packed_dev));
    } else {
        im::quantize_codes_int8_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
            w, awq, total, K, group_size, (int)G, scales_dev, zps_dev, static_cast<uint8_t *>(packed_dev));
    }
    IM_CUDA_CHECK(cudaGetLastError());
    return IM_OK;
    IM_GUARD_END
}
