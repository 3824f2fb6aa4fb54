// Epilogues of the tcgen05 projections (dense.cu, gemm_pair.cu): sixteen tokens of one weight row per lane, from f32 sums to
// the rows that DenseEpi names.
#pragma once
#include <cuda_fp16.h>

#include "stack.cuh"

namespace im {

template <>
__device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

// bf16 epilogues: z sigmoid(z), and gelu_tanh(z) = z / (1 + exp(-2 u)), u = sqrt(2 / pi) (z + 0.044715 z^3); the error of the
// fast exponential and quotient (about 1e-6) is far below the bf16 result's rounding. few: fewer rows than kDenseGemmMinF32, for which
// the activations are those of the matvec (epi_pair), so that a row's result is as exact whichever kernel a batch takes.
__device__ __forceinline__ float silu_fast(float z) { return __fdividef(z, 1.0f + __expf(-z)); }
template <typename T>
__device__ __forceinline__ float pair_act(float z, float up, bool silu, bool few) {
    if (few) return (silu ? silu_f(z) : gelu_tanh_f(z)) * up;
    if (silu) return silu_fast(z) * up;
    const float w = -1.5957691216057308f * z * fmaf(0.044715f * z, z, 1.0f);
    return __fdividef(z * up, 1.0f + __expf(fminf(w, 80.0f)));
}
// fp16 (quantized blocks): gate and up are rounded before the activation, as the reference's separate kernels do
template <>
__device__ __forceinline__ float pair_act<__half>(float z, float up, bool, bool) {
    return silu_f(__half2float(__float2half_rn(z))) * __half2float(__float2half_rn(up));
}
// The same for the values of a lane side by side: the general quotient's branches keep them apart (a prompt of 5003 tokens through four layers of a 2048-wide model
// took 5.21 ms with them, 4.84 with the fast exponential and quotient, which are less exact, 4.93 like this). Quotient by Markstein's method (IBM J. Res. Dev. 34, 1990):
// reciprocal refined by Newton steps, remainder by fma, one correction; equal to silu_f, bit for bit, for every fp16 gate but those that set odd (zeros, -80 and less, infinities, NaN).
template <typename T>
__device__ __forceinline__ float pair_act_side(float z, float up, bool silu, bool few, bool &) { return pair_act<T>(z, up, silu, few); }
template <>
__device__ __forceinline__ float pair_act_side<__half>(float z, float up, bool, bool, bool &odd) {
    const float g = __half2float(__float2half_rn(z)), d = 1.0f + expf(-g);
    odd = odd || !(g > -80.0f && g < INFINITY) || g == 0.0f;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    y = fmaf(y, fmaf(-d, y, 1.0f), y);
    y = fmaf(y, fmaf(-d, y, 1.0f), y);
    const float q = g * y;
    return fmaf(fmaf(-d, q, g), y, q) * __half2float(__float2half_rn(up));
}

// One round of a transposition between lanes: of every two values the lane with bit X clear keeps the first and gets its
// partner's first, the other lane the second ones; the results lie in the order of the lanes.
template <int X, typename V>
__device__ __forceinline__ void swap_lanes(const V &a, const V &b, V &lo, V &hi) {
    const bool up = threadIdx.x & X;
    V keep, send, got;
    const uint32_t *pa = reinterpret_cast<const uint32_t *>(&a), *pb = reinterpret_cast<const uint32_t *>(&b);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(V) / 4); i++) {
        reinterpret_cast<uint32_t *>(&keep)[i] = up ? pb[i] : pa[i];
        reinterpret_cast<uint32_t *>(&send)[i] = up ? pa[i] : pb[i];
        reinterpret_cast<uint32_t *>(&got)[i] = __shfl_xor_sync(0xffffffffu, reinterpret_cast<uint32_t *>(&send)[i], X);
    }
    lo = up ? got : keep;
    hi = up ? keep : got;
}
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
    const T a = from_f<T>(lo), b = from_f<T>(hi);
    return (uint32_t)*reinterpret_cast<const uint16_t *>(&a) | ((uint32_t)*reinterpret_cast<const uint16_t *>(&b) << 16);
}
// Eight values of eight lanes (neighbours at distance X) -> eight columns of one value, 16 bytes: lane bits X, 2 X, 4 X choose it.
template <typename T, int X>
__device__ __forceinline__ uint4 gather8(const float *v) {
    uint32_t w[4];
    uint2 d[2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float lo, hi;
        swap_lanes<X>(v[2 * i], v[2 * i + 1], lo, hi);
        w[i] = pack_pair<T>(lo, hi);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) swap_lanes<2 * X>(w[2 * i], w[2 * i + 1], d[i].x, d[i].y);
    uint2 lo, hi;
    swap_lanes<4 * X>(d[0], d[1], lo, hi);
    return make_uint4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ bool aligned16(const void *p, long long row_bytes) { return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)row_bytes) & 15) == 0; }

// epi_store16 for a warp whose 32 rows lie in one part of the result, with 16-byte rows: the lanes exchange their values so that a store
// carries 16 bytes.  A two-byte store per lane takes the SM 13 clocks however narrow it is: 128 x 256 results as such took 14000 clocks, most of a
// tile's products (gemm_pair.cu, 2048 tokens x 4096 x 512: 20.8 us, now 17.4 us with the activation branch below, 9.7 us without any store).  false: not such a warp, nothing stored.
template <typename T>
__device__ __forceinline__ bool epi_store16_wide(const DenseEpi &e, int N, int M, int n, int n_warp, int m, const float (&v)[16], bool few) {
    const int lane = threadIdx.x & 31, left = M - m, end = n_warp + 32;
    if (end > N) return false;
    const bool proj = e.kind == kEpiProj;
    if (proj && n_warp >= e.pair0) {
        const int col = (n_warp - e.pair0) >> 1;
        T *act = static_cast<T *>(e.act) + (size_t)m * e.ldact + col;
        if (!aligned16(act, 2ll * e.ldact)) return false;
        const bool odd = lane & 1;
        float r[8], z[8], u[8];
        bool other = false;
#pragma unroll
        for (int i = 0; i < 16; i += 2) {  // (gate, up) in neighbouring lanes: the even lane takes token i, the odd lane token i + 1
            const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
            z[i / 2] = odd ? got : v[i];
            u[i / 2] = odd ? v[i + 1] : got;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) r[i] = pair_act_side<T>(z[i], u[i], e.pair_silu, few, other);
        if (other)
#pragma unroll
            for (int i = 0; i < 8; i++) r[i] = pair_act<T>(z[i], u[i], e.pair_silu, few);
        const uint4 q = gather8<T, 2>(r);
        const int tok = lane & 15;
        if (tok < left) *reinterpret_cast<uint4 *>(act + (size_t)tok * e.ldact + (lane >> 4) * 8) = q;
        return true;
    }
    if (proj && end <= min(e.pair0, e.f0)) {
        T *y = static_cast<T *>(e.y) + (size_t)m * e.ldy + n_warp;
        if (!aligned16(y, 2ll * e.ldy)) return false;
        float r[16];
#pragma unroll
        for (int i = 0; i < 16; i++) r[i] = v[i];
        if (n_warp < e.silu_end)  // a branch: evaluated for every value and then dropped, it took more time than the stores
#pragma unroll
            for (int i = 0; i < 16; i++) r[i] = n < e.silu_end ? few ? silu_f(v[i]) : silu_fast(v[i]) : v[i];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint4 q = gather8<T, 1>(r + 8 * k);
            const int tok = 8 * k + (lane & 7);
            if (tok < left) *reinterpret_cast<uint4 *>(y + (size_t)tok * e.ldy + (lane & ~7)) = q;
        }
        return true;
    }
    if (proj && (n_warp < e.f0 || end > e.pair0)) return false;
    float *x = e.xf + (size_t)m * e.ldx + (proj ? n_warp - e.f0 : n_warp);
    if (!aligned16(x, 4ll * e.ldx)) return false;
    const float bias = !proj && e.kind == kEpiF32 && e.bias ? e.bias[n] : 0.0f;
    const bool cap = !proj && e.kind == kEpiF32 && e.cap > 0.0f;
    float4 q[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float r[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            r[i] = v[4 * k + i] + bias;
            if (cap) r[i] = e.cap * tanhf(r[i] / e.cap);
        }
        float2 a, b, lo, hi;
        swap_lanes<1>(r[0], r[1], a.x, a.y);
        swap_lanes<1>(r[2], r[3], b.x, b.y);
        swap_lanes<2>(a, b, lo, hi);
        q[k] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    x += (size_t)(lane & 3) * e.ldx + (lane & ~3);
    if (e.kind == kEpiResidual) {
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (4 * k + (lane & 3) < left) {
                const float4 o = *reinterpret_cast<const float4 *>(x + (size_t)(4 * k) * e.ldx);
                q[k] = make_float4(o.x + q[k].x, o.y + q[k].y, o.z + q[k].z, o.w + q[k].w);
            }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (4 * k + (lane & 3) < left) *reinterpret_cast<float4 *>(x + (size_t)(4 * k) * e.ldx) = q[k];
    return true;
}

// 16 tokens m .. m + 15 of row n (one per lane; n_warp: that of lane 0) of a result of N rows and M tokens
template <typename T>
__device__ __forceinline__ void epi_store16(const DenseEpi &e, int N, int M, int n, int n_warp, int m, const float (&v)[16], bool few = false) {
    if (epi_store16_wide<T>(e, N, M, n, n_warp, m, v, few)) return;
    const int lane = threadIdx.x & 31, left = M - m;
    if (e.kind == kEpiProj) {
        if (n_warp + 31 >= e.pair0) {
            // (gate, up) sit in neighbouring lanes: of two tokens, the even lane takes the first, the odd lane the second
            // (pair0 is a multiple of eight: no pair straddles it)
            T *act = static_cast<T *>(e.act) + (size_t)m * e.ldact + ((n - e.pair0) >> 1);
            T *y = static_cast<T *>(e.y) + (size_t)m * e.ldy + n;
            const bool odd = lane & 1, pair = n >= e.pair0;
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
                if (pair) {
                    const float r = odd ? pair_act<T>(got, v[i + 1], e.pair_silu, few) : pair_act<T>(v[i], got, e.pair_silu, few);
                    if (n < N && i + odd < left) act[(size_t)(i + odd) * e.ldact] = from_f<T>(r);
                } else {
#pragma unroll
                    for (int j = 0; j < 2; j++)
                        if (i + j < left) {
                            if (n >= e.f0) e.xf[(size_t)(m + i + j) * e.ldx + (n - e.f0)] = v[i + j];
                            else y[(size_t)(i + j) * e.ldy] = from_f<T>(n < e.silu_end ? few ? silu_f(v[i + j]) : silu_fast(v[i + j]) : v[i + j]);
                        }
                }
            }
        } else {
            T *y = static_cast<T *>(e.y) + (size_t)m * e.ldy + n;
            const bool act = n < e.silu_end;
            if (n < N && n >= e.f0) {
                float *f = e.xf + (size_t)m * e.ldx + (n - e.f0);
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (i < left) f[(size_t)i * e.ldx] = v[i];
            } else if (n < N) {
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (i < left) y[(size_t)i * e.ldy] = from_f<T>(act ? few ? silu_f(v[i]) : silu_fast(v[i]) : v[i]);
            }
        }
    } else if (n < N) {
        float *x = e.xf + (size_t)m * e.ldx + n;
        if (e.kind == kEpiResidual) {
            float old[16];
#pragma unroll
            for (int i = 0; i < 16; i++) old[i] = i < left ? x[(size_t)i * e.ldx] : 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (i < left) x[(size_t)i * e.ldx] = old[i] + v[i];
        } else {
            const float b = e.bias ? e.bias[n] : 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                float r = v[i] + b;
                if (e.cap > 0.0f) r = e.cap * tanhf(r / e.cap);
                if (i < left) x[(size_t)i * e.ldx] = r;
            }
        }
    }
}

}  // namespace im
