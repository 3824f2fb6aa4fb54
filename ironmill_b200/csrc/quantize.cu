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
// Bound: HBM (2 bytes in, 0.5 or 1 byte and 8 bytes per group out).  A thread owns the same eight columns of kQRows
// consecutive rows, so that its loads are in flight together and one index division and one load of the AWQ vector serve
// them all; the L = group / 8 lanes of a group find its extrema by shuffles and the codes are formed from the values still in
// registers.  14336 x 4096, 4-bit with AWQ: 406 -> 90 us (1.7 TB/s; issue bounds it: about eight instructions per element).
//
// Codes without a division per element: t = x * (1 / scale) + zp differs from the defining fl(fl(x / scale) + zp) by less
// than 2^-20 (|x / scale| + |zp| + 1), so the two round to the same integer unless t lies that close to a half; a thread
// that meets such a value (or a non-finite one, or a magnitude past 2^21) recomputes its eight by the definition.
constexpr int kQRows = 4;

__device__ __forceinline__ unsigned quantize_one(float x, float scale, float zp, float qmax);

template <int BITS>
__global__ void __launch_bounds__(256) quantize_groups_kernel(const __half *__restrict__ w, const __half *__restrict__ awq, size_t rows, unsigned K, int L,
                                                              unsigned G, float *__restrict__ scales, float *__restrict__ zps, uint8_t *__restrict__ packed) {
    constexpr float qmax = BITS == 4 ? 15.0f : 255.0f;
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low mantissa bits
    const unsigned per_row = G * (unsigned)L;  // octets of a row, the short last group padded
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t rb = (i >> 32) == 0 ? (unsigned)i / per_row : i / per_row;
    const unsigned o = (unsigned)(i - rb * per_row), g = o >> (__ffs(L) - 1), col = o * 8;
    const size_t r0 = rb * kQRows;
    const int lane = threadIdx.x & 31;
    const unsigned seg = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (lane & ~(L - 1));  // the lanes of this group
    const bool in_row = col < K;  // a group is 8 L columns and K a multiple of 8: an octet is inside or outside
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = 1.0f;
    unsigned bad_awq = 0;
    if (awq && in_row) {
        const uint4 v = *reinterpret_cast<const uint4 *>(awq + col);
        const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&u[j]));
            a[2 * j] = f.x;
            a[2 * j + 1] = f.y;
            bad_awq |= ((u[j] & 0x7fff7fffu) + 0x04000400u) & 0x80008000u;  // an exponent of all ones
        }
    }
    uint4 raw[kQRows];
#pragma unroll
    for (int r = 0; r < kQRows; r++) {
        raw[r] = make_uint4(0, 0, 0, 0);
        if (in_row && r0 + r < rows) raw[r] = ldg_stream_v4(w + (r0 + r) * K + col);
    }
#pragma unroll
    for (int r = 0; r < kQRows; r++) {
        const bool live = in_row && r0 + r < rows;
        const unsigned u[4] = {raw[r].x, raw[r].y, raw[r].z, raw[r].w};
        float x[8];
        unsigned bad = bad_awq;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&u[j]));
            x[2 * j] = awq ? __fmul_rn(f.x, a[2 * j]) : f.x;
            x[2 * j + 1] = awq ? __fmul_rn(f.y, a[2 * j + 1]) : f.y;
            bad |= ((u[j] & 0x7fff7fffu) + 0x04000400u) & 0x80008000u;
        }
        // extrema of the finite values; of equal extrema the first counts (the sign of a zero can tell them apart)
        float mn = INFINITY, mx = -INFINITY;
        if (live) {
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (!bad || isfinite(x[j])) {
                    if (x[j] < mn) mn = x[j];
                    if (x[j] > mx) mx = x[j];
                }
        }
        float gmn = mn, gmx = mx;
        for (int d = L >> 1; d > 0; d >>= 1) {
            gmn = fminf(gmn, __shfl_xor_sync(0xffffffffu, gmn, d));
            gmx = fmaxf(gmx, __shfl_xor_sync(0xffffffffu, gmx, d));
        }
        const unsigned at_mn = __ballot_sync(0xffffffffu, mn == gmn) & seg, at_mx = __ballot_sync(0xffffffffu, mx == gmx) & seg;
        mn = __shfl_sync(0xffffffffu, mn, __ffs(at_mn) - 1);
        mx = __shfl_sync(0xffffffffu, mx, __ffs(at_mx) - 1);
        float scale, zp;
        const bool finite = isfinite(mn) && isfinite(mx);  // false: no finite value in the group
        if (!finite) {
            scale = 1.0f;
            zp = 0.0f;
        } else if (fabsf(__fsub_rn(mx, mn)) < FLT_EPSILON) {
            scale = 1.0f;
            zp = roundf(-mn);
        } else {
            scale = __fdiv_rn(__fsub_rn(mx, mn), qmax);
            zp = roundf(__fdiv_rn(-mn, scale));
        }
        if (!live) continue;
        if ((o & (unsigned)(L - 1)) == 0) {
            scales[(r0 + r) * G + g] = scale;
            zps[(r0 + r) * G + g] = zp;
        }
        const float inv = __fdividef(1.0f, scale);
        // t is within [mn, mx] / scale + zp; the largest magnitude on the way bounds the rounding of both forms
        const float mag = fmaxf(fabsf(mn), fabsf(mx)) * inv + fabsf(zp) + 1.0f;
        const float near_half = 0.5f - mag * 0x1p-20f;
        float c[8], far = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float t = fmaf(x[j], inv, zp), rr = __fsub_rn(__fadd_rn(t, kMagic), kMagic);
            far = fmaxf(far, fabsf(t - rr));
            c[j] = fminf(fmaxf(rr, 0.0f), qmax);
        }
        if (bad || !finite || !(far < near_half) || !(mag < 2097152.0f)) {
#pragma unroll
            for (int j = 0; j < 8; j++) c[j] = finite ? (float)quantize_one(x[j], scale, zp, qmax) : 0.0f;
        }
        if (BITS == 4) {
            // four codes in one exact f32 sum, the lower column in the lower nibble
            const float lo = fmaf(fmaf(fmaf(c[3], 16.0f, c[2]), 16.0f, c[1]), 16.0f, c[0]), hi = fmaf(fmaf(fmaf(c[7], 16.0f, c[6]), 16.0f, c[5]), 16.0f, c[4]);
            reinterpret_cast<unsigned *>(packed)[((r0 + r) * K + col) >> 3] = (unsigned)lo | ((unsigned)hi << 16);
        } else {
            const float lo = fmaf(c[1], 256.0f, c[0]), lo2 = fmaf(c[3], 256.0f, c[2]), hi = fmaf(c[5], 256.0f, c[4]), hi2 = fmaf(c[7], 256.0f, c[6]);
            reinterpret_cast<uint2 *>(packed)[((r0 + r) * K + col) >> 3] =
                make_uint2((unsigned)lo | ((unsigned)lo2 << 16), (unsigned)hi | ((unsigned)hi2 << 16));
        }
    }
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
        const size_t threads = (rows + im::kQRows - 1) / im::kQRows * G * L, blocks = (threads + 255) / 256;
        if (blocks <= 0x7fffffff) {
            if (bit_width == 4)
                im::quantize_groups_kernel<4><<<(unsigned)blocks, 256, 0, st>>>(w, awq, rows, (unsigned)K, L, (unsigned)G, scales_dev, zps_dev,
                                                                               static_cast<uint8_t *>(packed_dev));
            else
                im::quantize_groups_kernel<8><<<(unsigned)blocks, 256, 0, st>>>(w, awq, rows, (unsigned)K, L, (unsigned)G, scales_dev, zps_dev,
                                                                               static_cast<uint8_t *>(packed_dev));
            IM_CUDA_CHECK(cudaGetLastError());
            return IM_OK;
        }
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
