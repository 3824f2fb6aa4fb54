// TurboQuant attention for prefill chunks (many query tokens against one sequence's cache).
//
// turboquant_attention (crates/ironmill-inference/src/metal/shaders/turboquant/turboquant.metal:202-462) scores every
// (token, head) against the cached positions one token at a time; with T tokens in flight the cache is dequantised T
// times.  Its score is bilinear in what the cache holds,
//     s[t, h, p] = attn_scale * ks_p * ( q~[t,h] . cbK[idx_p]  +  (r_norm_p * qjl_factor) * (S q~)[t,h] . sign_p ),
//     o[t, h]    = sum_p softmax(s)[p] * vs_p * cbV[idx_p]        (in the rotated space; rotated back afterwards),
// so a chunk dequantises the positions ONCE into fp16 rows K' = [cbK[idx] | sign] (256 wide) and V' = cbV[idx] (128 wide), puts the
// queries into rows [q~ | S q~], and the causal kernel of flash_tc.cu runs over them on the tcgen05 tensor cores: fp16 operands, f32
// accumulation, the per-position factors applied to the f32 scores and weights exactly where the decode kernel
// (tq_attention_tc_kernel) applies them, the outputs rotated back in its epilogue.
//
//   tq_prompt_encode_kernel   K and V of the chunk into the cache (norm, rotation, bit-exact encoding)
//   tq_dequant_rows_kernel    cached rows -> K', V' and the factors, tile by tile
//   tq_prompt_query_kernel    queries (norm, rotation) -> [q~ | S q~]
// 2048 tokens, 32 / 8 heads: the token-by-token preparation took 238 us, the mma.sync attention 382 and its normalisation 74; now the queries
// 36 us, the cached rows 6, attention 118 (the encoding: at its kernel).
#include "common.cuh"
#include "flash_tc.cuh"
#include "tq_device.cuh"

namespace im {

namespace {

constexpr int kPfN = 64;      // positions of a tile of flash_tc.cu

// Cache rows [0, npos) of one slot -> K' [nkv][npos][256] and V' [nkv][npos][128] fp16, one thread per 8 elements; and the positions'
// factors, tiles of [ks | r_norm * qjl_factor | vs] with zeros past npos (the grid covers whole tiles).
template <int BITS>
__global__ void tq_dequant_rows_kernel(const uint8_t *__restrict__ kc, const uint8_t *__restrict__ vc, const float *__restrict__ k_cb,
                                       const float *__restrict__ v_cb, const float *__restrict__ ks, const float *__restrict__ vs, const float *__restrict__ krn,
                                       float qjl_factor, __half *__restrict__ kd, __half *__restrict__ vd, float *__restrict__ factors, int slot, int nkv,
                                       int max_seq, int npos) {
    pdl_trigger();
    pdl_wait();
    constexpr int kRowB = BITS == 4 ? kHd / 2 : kHd;
    constexpr unsigned kIdx = (1u << (BITS - 1)) - 1u, kSign = 1u << (BITS - 1), kAll = (1u << BITS) - 1u;
    const int c = threadIdx.x & 15;                       // chunk of 8 elements
    const int pos = blockIdx.x * 16 + (threadIdx.x >> 4);
    const int kvh = blockIdx.y;
    const size_t row = ((size_t)slot * nkv + kvh) * max_seq + pos;
    if (c < 3) {
        const int tiles = (npos + kPfN - 1) / kPfN;
        const float f = pos >= npos ? 0.0f : c == 0 ? ks[row] : c == 1 ? krn[row] * qjl_factor : vs[row];
        factors[((size_t)kvh * tiles + pos / kPfN) * (3 * kPfN) + c * kPfN + pos % kPfN] = f;
    }
    if (pos >= npos) return;
    unsigned kb[8], vb[8];
    if (BITS == 8) {
        const uint2 kw = *reinterpret_cast<const uint2 *>(kc + row * kRowB + 8 * c), vw = *reinterpret_cast<const uint2 *>(vc + row * kRowB + 8 * c);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            kb[i] = ((i < 4 ? kw.x : kw.y) >> (8 * (i & 3))) & 255u;
            vb[i] = ((i < 4 ? vw.x : vw.y) >> (8 * (i & 3))) & 255u;
        }
    } else {
        const unsigned kw = *reinterpret_cast<const unsigned *>(kc + row * kRowB + 4 * c), vw = *reinterpret_cast<const unsigned *>(vc + row * kRowB + 4 * c);
#pragma unroll
        for (int i = 0; i < 8; i++) {  // element 2j in the low nibble of byte j
            kb[i] = (kw >> (4 * i)) & 15u;
            vb[i] = (vw >> (4 * i)) & 15u;
        }
    }
    __half kcv[8], ksv[8], vv[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        kcv[i] = __float2half_rn(k_cb[kb[i] & kIdx]);
        ksv[i] = __float2half_rn((kb[i] & kSign) ? 1.0f : -1.0f);
        vv[i] = __float2half_rn(v_cb[vb[i] & kAll]);
    }
    const size_t orow = (size_t)kvh * npos + pos;
    *reinterpret_cast<uint4 *>(kd + orow * 256 + 8 * c) = *reinterpret_cast<const uint4 *>(kcv);
    *reinterpret_cast<uint4 *>(kd + orow * 256 + 128 + 8 * c) = *reinterpret_cast<const uint4 *>(ksv);
    *reinterpret_cast<uint4 *>(vd + orow * 128 + 8 * c) = *reinterpret_cast<const uint4 *>(vv);
}

__device__ __forceinline__ void mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ unsigned pack2h(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const unsigned *>(&h);
}

// Positions of the chunk's tokens and the rotation of a head's 128 values.
struct PromptRope {
    const __half *cosc, *sinc;
    int rotary_dim, base_pos, slot;
    const int *pos_dev;
    __device__ __forceinline__ int first() const { return base_pos + (pos_dev ? pos_dev[slot] : 0); }
};

// ---- K and V of the chunk -------------------------------------------------------------------------------------------------
// A warp encodes four tokens of one head, lane l the elements l, l + 32, l + 64, l + 96: the same operands in the same order as
// tq_encode_body, whose 128 threads hold one element each (strides 32 and 64 of the butterflies and of the summation tree are in the
// lane's own registers), without block barriers.  The projection reads the matrix from shared memory, once for four tokens:
// 128 x 128 separate multiplies and adds per key row take about 15 us of issue for 2048 tokens of 8 heads, the table searches about as much;
// measured 87 us (116 with keys and values alternating: a stride of all warps then gave one warp only keys, another only values).
constexpr int kEncRows = 4, kEncWarps = 8;
struct PromptEncode {
    const __half *kv;        // token rows; K head h at k_off + 128 h, V at v_off + 128 h
    int stride, k_off, v_off;
    const __half *kw;        // norm weights or nullptr
    float eps;
    PromptRope rope;
    EncodeTables ktab, vtab;
    uint8_t *kc, *vc;
    float *ks, *vs, *krn;
    int nkv, max_seq, T;
};
constexpr int kEncSmem = (kHd * kHd + kEncWarps * kHd * kEncRows + 2 * 256 + 2 * 128) * 4;

__device__ __forceinline__ float enc_tree_sum(const float (&x)[4]) {  // the order of tq_tree_sum
    float r = __fadd_rn(__fadd_rn(x[0], x[2]), __fadd_rn(x[1], x[3]));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) r = __fadd_rn(r, __shfl_down_sync(0xffffffffu, r, s));
    return __shfl_sync(0xffffffffu, r, 0);
}

template <int BITS>
__global__ void __launch_bounds__(kEncWarps * 32, 2) tq_prompt_encode_kernel(const PromptEncode a) {
    extern __shared__ __align__(16) float enc_smem[];
    float *mat = enc_smem, *res = mat + kHd * kHd, *vbd = res + kEncWarps * kHd * kEncRows, *kbd = vbd + 256, *kcb = kbd + 128, *sgs = kcb + 128;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_trigger();
    for (int i = tid; i < kHd * kHd / 4; i += kEncWarps * 32) reinterpret_cast<float4 *>(mat)[i] = reinterpret_cast<const float4 *>(a.ktab.qjl_t)[i];
    for (int i = tid; i < a.vtab.n_levels - 1; i += kEncWarps * 32) vbd[i] = a.vtab.bounds[i];
    for (int i = tid; i < a.ktab.n_levels; i += kEncWarps * 32) {
        kcb[i] = a.ktab.cb[i];
        if (i + 1 < a.ktab.n_levels) kbd[i] = a.ktab.bounds[i];
    }
    for (int i = tid; i < kHd; i += kEncWarps * 32) sgs[i] = a.ktab.signs[i];
    pdl_wait();
    __syncthreads();
    const int P = a.rope.first(), groups = (a.T + kEncRows - 1) / kEncRows, items = groups * 2 * a.nkv;
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)kHd));
    float *rw = res + warp * kHd * kEncRows;  // residuals [dimension][row]
    float sg[4];
#pragma unroll
    for (int i = 0; i < 4; i++) sg[i] = sgs[lane + 32 * i];
    for (int item = blockIdx.x * kEncWarps + warp; item < items; item += gridDim.x * kEncWarps) {
        // every key before the first value: keys take several times as long, and each warp gets its share of both
        const bool is_k = item < groups * a.nkv;
        const int left = is_k ? item : item - groups * a.nkv, h = left % a.nkv, t0 = left / a.nkv * kEncRows;
        unsigned code[kEncRows][4];
        const float *bd = is_k ? kbd : vbd;
        const int levels = is_k ? a.ktab.n_levels : a.vtab.n_levels;
#pragma unroll
        for (int r = 0; r < kEncRows; r++) {
            const int t = min(t0 + r, a.T - 1);  // rows past the last token repeat it (not stored)
            const __half *src = a.kv + (size_t)t * a.stride + (is_k ? a.k_off : a.v_off) + h * kHd;
            const int pos = P + t;
            float x[4];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = __half2float(src[lane + 32 * i]);
            if (is_k) {
                float nrm = 1.0f;
                if (a.kw) {
                    float tot = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float ss = warp_sum(x[i] * x[i]);
                        tot = i == 0 ? ss : tot + ss;
                    }
                    nrm = rsqrtf(tot / (float)kHd + a.eps);
#pragma unroll
                    for (int i = 0; i < 4; i++) x[i] = x[i] * nrm * __half2float(a.kw[lane + 32 * i]);
                }
                const int half_rot = a.rope.rotary_dim / 2;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int d = lane + 32 * i;
                    if (d < a.rope.rotary_dim) {
                        const int ri = d < half_rot ? d : d - half_rot, o = d < half_rot ? d + half_rot : ri;
                        float other = __half2float(src[o]);
                        if (a.kw) other = other * nrm * __half2float(a.kw[o]);
                        const float rc = __half2float(a.rope.cosc[(size_t)pos * (kHd / 2) + ri]), rs = __half2float(a.rope.sinc[(size_t)pos * (kHd / 2) + ri]);
                        const float lo = d < half_rot ? x[i] : other, hi = d < half_rot ? other : x[i];
                        rw[d * kEncRows + r] = d < half_rot ? lo * rc - hi * rs : lo * rs + hi * rc;
                    } else {
                        rw[d * kEncRows + r] = x[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = __half2float(__float2half_rn(rw[(lane + 32 * i) * kEncRows + r]));
            }
            // rotation: signs, butterflies, signs / sqrt(128)
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = __fmul_rn(x[i], sg[i]);
#pragma unroll
            for (int step = 1; step < 32; step <<= 1)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float o = __shfl_xor_sync(0xffffffffu, x[i], step);
                    x[i] = (lane & step) ? __fsub_rn(o, x[i]) : __fadd_rn(x[i], o);
                }
#pragma unroll
            for (int s = 1; s < 4; s <<= 1)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (!(i & s)) {
                        const float p = x[i], q = x[i + s];
                        x[i] = __fadd_rn(p, q);
                        x[i + s] = __fsub_rn(p, q);
                    }
            float y[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                x[i] = __fmul_rn(x[i], __fmul_rn(sg[i], scale));
                y[i] = __fmul_rn(x[i], x[i]);
            }
            const float norm = __fsqrt_rn(fmaxf(enc_tree_sum(y), 1e-20f)), inv = __fdiv_rn(1.0f, fmaxf(norm, 1e-10f));
            const size_t row = ((size_t)a.rope.slot * a.nkv + h) * a.max_seq + pos % a.max_seq;
            if (lane == 0 && t0 + r < a.T) (is_k ? a.ks : a.vs)[row] = norm;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float u = __fmul_rn(x[i], inv);
                int lo = 0, hi = levels - 1;  // bounds: suffix minima (tq_encode_body)
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (u >= bd[mid]) lo = mid + 1;
                    else hi = mid;
                }
                code[r][i] = (unsigned)lo;
                if (is_k) {
                    const float d = __fsub_rn(u, kcb[lo]);
                    rw[(lane + 32 * i) * kEncRows + r] = d;
                    y[i] = __fmul_rn(d, d);
                }
            }
            if (is_k) {
                const float rs = enc_tree_sum(y);
                if (lane == 0 && t0 + r < a.T) a.krn[row] = __fsqrt_rn(fmaxf(rs, 1e-20f));
            }
        }
        if (is_k) {
            __syncwarp();
            float acc[kEncRows][4];
#pragma unroll
            for (int r = 0; r < kEncRows; r++) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.0f;
#pragma unroll 4
            for (int k = 0; k < kHd; k++) {
                const float4 v = *reinterpret_cast<const float4 *>(rw + k * kEncRows);
                const float vr[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float m = mat[k * kHd + lane + 32 * i];
#pragma unroll
                    for (int r = 0; r < kEncRows; r++) acc[r][i] = __fadd_rn(acc[r][i], __fmul_rn(m, vr[r]));
                }
            }
#pragma unroll
            for (int r = 0; r < kEncRows; r++)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (acc[r][i] >= 0.0f) code[r][i] |= 1u << (BITS - 1);
            __syncwarp();
        }
#pragma unroll
        for (int r = 0; r < kEncRows; r++) {
            const int pos = P + t0 + r;
            const bool live = t0 + r < a.T;
            uint8_t *dst = (is_k ? a.kc : a.vc) + (((size_t)a.rope.slot * a.nkv + h) * a.max_seq + pos % a.max_seq) * (size_t)(kHd * BITS / 8);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (BITS == 4) {
                    const unsigned up = __shfl_down_sync(0xffffffffu, code[r][i], 1);
                    if (live && !(lane & 1)) dst[(lane + 32 * i) >> 1] = (uint8_t)((code[r][i] & 15u) | ((up & 15u) << 4));
                } else if (live) {
                    dst[lane + 32 * i] = (uint8_t)code[r][i];
                }
            }
        }
    }
}

// ---- queries ----------------------------------------------------------------------------------------------------------------
// A warp takes 16 consecutive (token, head) rows.  Lane (g, t) holds dimensions 32 t .. 32 t + 31 of rows g and g + 8: norm and rotation
// read the row's own 64 bytes (and its partners'), the butterflies need two shuffles, and the values are the A fragments of
// S q~ as they lie (the matrix is staged with its rows in the fragments' order).  mma.sync issue bounds it (128 products per 16 rows).
constexpr int kQWarps = 8, kMatRowB = 272;
struct PromptQuery {
    const __half *q;         // token rows, head h at 128 h
    int stride;
    const __half *qw;
    float eps;
    PromptRope rope;
    const float *signs, *qjl_t;
    __half *out;             // [T * nh][256]
    int nh, T;
};

__global__ void __launch_bounds__(kQWarps * 32) tq_prompt_query_kernel(const PromptQuery a) {
    __shared__ __align__(16) unsigned char mat[kHd * kMatRowB];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    pdl_trigger();
    for (int i = tid; i < kHd * 16; i += kQWarps * 32) {
        // row 16 kk + e of the staged matrix is dimension 32 t + 4 kk + ..: e = 2 t, 2 t + 1 -> + 0, 1; e = 2 t + 8, 2 t + 9 -> + 2, 3
        const int r = i >> 4, c = i & 15, kk = r >> 4, e = r & 15, k = 32 * ((e & 7) >> 1) + 4 * kk + (e & 1) + 2 * (e >> 3);
        const float4 x = *reinterpret_cast<const float4 *>(a.qjl_t + k * kHd + 8 * c), y = *reinterpret_cast<const float4 *>(a.qjl_t + k * kHd + 8 * c + 4);
        *reinterpret_cast<uint4 *>(mat + r * kMatRowB + 16 * c) = make_uint4(pack2h(x.x, x.y), pack2h(x.z, x.w), pack2h(y.x, y.y), pack2h(y.z, y.w));
    }
    pdl_wait();
    __syncthreads();
    const int rows = a.T * a.nh, base = (blockIdx.x * kQWarps + warp) * 16;
    if (base >= rows) return;
    const int P = a.rope.first(), half_rot = a.rope.rotary_dim / 2;
    unsigned fr[2][16];  // rows g, g + 8: dimensions 32 t + 2 j, + 1
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int row = min(base + g + 8 * r, rows - 1), tok = row / a.nh, h = row - tok * a.nh;  // rows past the end repeat the last
        const __half *src = a.q + (size_t)tok * a.stride + h * kHd;
        float x[32];
        if (a.stride % 8 == 0 && reinterpret_cast<uintptr_t>(a.q) % 16 == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 u = *reinterpret_cast<const uint4 *>(src + 32 * t + 8 * i);
                const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[j]));
                    x[8 * i + 2 * j] = f.x;
                    x[8 * i + 2 * j + 1] = f.y;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 32; i++) x[i] = __half2float(src[32 * t + i]);
        }
        float nrm = 1.0f;
        if (a.qw) {
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < 32; i++) ss = fmaf(x[i], x[i], ss);
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            ss += __shfl_xor_sync(0xffffffffu, ss, 2);
            nrm = rsqrtf(ss / (float)kHd + a.eps);
#pragma unroll
            for (int i = 0; i < 32; i++) x[i] = x[i] * nrm * __half2float(a.qw[32 * t + i]);
        }
        const __half *rc = a.rope.cosc + (size_t)(P + tok) * (kHd / 2), *rs = a.rope.sinc + (size_t)(P + tok) * (kHd / 2);
        if (a.rope.rotary_dim == kHd) {
            // partners sit in lane t ^ 2: lanes 0, 1 hold the first half
            const bool first = t < 2;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 cu = *reinterpret_cast<const uint4 *>(rc + 32 * (t & 1) + 8 * i), su = *reinterpret_cast<const uint4 *>(rs + 32 * (t & 1) + 8 * i);
                const unsigned cw[4] = {cu.x, cu.y, cu.z, cu.w}, sw[4] = {su.x, su.y, su.z, su.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&cw[j])), s = __half22float2(*reinterpret_cast<const __half2 *>(&sw[j]));
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const int k = 8 * i + 2 * j + q;
                        const float other = __shfl_xor_sync(0xffffffffu, x[k], 2), cv = q ? c.y : c.x, sv = q ? s.y : s.x;
                        const float lo = first ? x[k] : other, hi = first ? other : x[k];
                        x[k] = first ? lo * cv - hi * sv : lo * sv + hi * cv;
                    }
                }
            }
        } else if (a.rope.rotary_dim > 0) {
            float y[32];
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const int d = 32 * t + i;
                y[i] = x[i];
                if (d < a.rope.rotary_dim) {
                    const int ri = d < half_rot ? d : d - half_rot, o = d < half_rot ? d + half_rot : ri;
                    float other = __half2float(src[o]);
                    if (a.qw) other = other * nrm * __half2float(a.qw[o]);
                    const float lo = d < half_rot ? x[i] : other, hi = d < half_rot ? other : x[i], c = __half2float(rc[ri]), s = __half2float(rs[ri]);
                    y[i] = d < half_rot ? lo * c - hi * s : lo * s + hi * c;
                }
            }
#pragma unroll
            for (int i = 0; i < 32; i++) x[i] = y[i];
        }
        // rounded as the reference's q buffer, then into the rotated space
#pragma unroll
        for (int i = 0; i < 32; i++) x[i] = __half2float(__float2half_rn(x[i])) * __ldg(a.signs + 32 * t + i);
#pragma unroll
        for (int step = 1; step < 32; step *= 2)
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (!(i & step)) {
                    const float p = x[i], q = x[i + step];
                    x[i] = p + q;
                    x[i + step] = p - q;
                }
#pragma unroll
        for (int step = 1; step < 4; step *= 2)
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const float o = __shfl_xor_sync(0xffffffffu, x[i], step);
                x[i] = (t & step) ? o - x[i] : x[i] + o;
            }
        constexpr float kRoot = 0.08838834764831845f;  // 1 / sqrt(128)
#pragma unroll
        for (int j = 0; j < 16; j++)
            fr[r][j] = pack2h(x[2 * j] * (__ldg(a.signs + 32 * t + 2 * j) * kRoot), x[2 * j + 1] * (__ldg(a.signs + 32 * t + 2 * j + 1) * kRoot));
        if (base + g + 8 * r < rows) {
            uint4 *dst = reinterpret_cast<uint4 *>(a.out + (size_t)row * 256 + 32 * t);
#pragma unroll
            for (int i = 0; i < 4; i++) dst[i] = make_uint4(fr[r][4 * i], fr[r][4 * i + 1], fr[r][4 * i + 2], fr[r][4 * i + 3]);
        }
    }
    const unsigned m_a = (unsigned)__cvta_generic_to_shared(mat + (lane & 15) * kMatRowB + (lane >> 4) * 16);
#pragma unroll 2
    for (int nd = 0; nd < 16; nd += 2) {
        float c0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, c1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int kk = 0; kk < 8; kk++) {
            unsigned b[4];
            ldsm_x4_t(b, m_a + kk * 16 * kMatRowB + nd * 16);
            mma16816(c0, fr[0][2 * kk], fr[1][2 * kk], fr[0][2 * kk + 1], fr[1][2 * kk + 1], b[0], b[1]);
            mma16816(c1, fr[0][2 * kk], fr[1][2 * kk], fr[0][2 * kk + 1], fr[1][2 * kk + 1], b[2], b[3]);
        }
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (base + g + 8 * r < rows) {
                __half *dst = a.out + (size_t)(base + g + 8 * r) * 256 + 128 + 8 * nd + 2 * t;
                *reinterpret_cast<unsigned *>(dst) = pack2h(c0[2 * r], c0[2 * r + 1]);
                *reinterpret_cast<unsigned *>(dst + 8) = pack2h(c1[2 * r], c1[2 * r + 1]);
            }
    }
}

}  // namespace

bool tq_prefill_takes(int nh, int nkv) {
    if (nkv <= 0 || nh % nkv != 0) return false;
    const int gq = nh / nkv;
    return gq == 1 || gq == 2 || gq == 4 || gq == 8;
}

// K', V' rows, then the factors of whole tiles
size_t tq_prefill_scratch_bytes(int nkv, int max_seq) {
    return (size_t)nkv * max_seq * (256 + 128) * sizeof(__half) + (size_t)nkv * ((max_seq + kPfN - 1) / kPfN) * (3 * kPfN) * sizeof(float);
}

// K and V of a chunk of one sequence into its cache slot, as tq_prep_launch does for any step.
int tq_prompt_encode_launch(const Tq *tq, const TqPrep &p, int slot, cudaStream_t st) {
    if (tq->hd != kHd) return fail(IM_ERR_INVALID, "the prompt's cache write is built for head_dim 128 (got %d)", tq->hd);
    PromptEncode a{};
    a.kv = p.kv ? p.kv : p.qkv; a.stride = p.kv ? p.kv_stride : p.stride; a.k_off = p.k_off; a.v_off = p.v_off;
    a.kw = p.with_norm ? p.kw : nullptr; a.eps = p.eps;
    a.rope = PromptRope{p.cosc, p.sinc, p.rotary_dim, p.base_pos, slot, p.pos_dev};
    a.ktab = EncodeTables{tq->signs, tq->k_cb, tq->k_bd, tq->qjl_t, tq->k_levels, 1, tq->n_bits};
    a.vtab = EncodeTables{tq->signs, tq->v_cb, tq->v_bd, tq->qjl_t, tq->v_levels, 0, tq->n_bits};
    a.kc = p.kc; a.vc = p.vc; a.ks = p.ks; a.vs = p.vs; a.krn = p.krn; a.nkv = p.nkv; a.max_seq = p.max_seq; a.T = p.T;
    static DeviceOnce once;
    if (once.first(tq->dev->ordinal)) {
        IM_CUDA_CHECK(cudaFuncSetAttribute(tq_prompt_encode_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kEncSmem));
        IM_CUDA_CHECK(cudaFuncSetAttribute(tq_prompt_encode_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kEncSmem));
    }
    const int items = (p.T + kEncRows - 1) / kEncRows * 2 * p.nkv, blocks = (items + kEncWarps - 1) / kEncWarps, most = 2 * tq->dev->sm_count;
    IM_CUDA_CHECK(launch_k(tq->n_bits == 4 ? tq_prompt_encode_kernel<4> : tq_prompt_encode_kernel<8>, dim3(blocks < most ? blocks : most), dim3(kEncWarps * 32),
                           (size_t)kEncSmem, st, a));
    return IM_OK;
}

// One sequence's prefill chunk: T tokens whose rows are already in the cache at positions pos_dev[slot] .. + T - 1;
// ctx_end = the host's count of cached positions after the chunk (bounds the dequantisation).  q_rows: T * nh * 256 halves of scratch;
// dq: tq_prefill_scratch_bytes(nkv, max_seq).  IM_ERR_BOUNDS when the head grouping is not 1, 2, 4 or 8.
int tq_prefill_attention_launch(const Tq *tq, void *q_rows, void *dq, const TqPromptQuery &q, const uint8_t *kc, const uint8_t *vc, const float *ks,
                                const float *vs, const float *krn, float attn_scale, __half *out, int slot, int nh, int nkv, int max_seq,
                                const int *pos_dev, int T, int ctx_end, cudaStream_t st, int base_pos) {
    if (!tq_prefill_takes(nh, nkv) || T <= 0) return IM_ERR_BOUNDS;
    const int npos = ctx_end < max_seq ? ctx_end : max_seq, tiles = (npos + kPfN - 1) / kPfN;
    __half *kd = static_cast<__half *>(dq), *vd = kd + (size_t)nkv * npos * 256;
    float *factors = reinterpret_cast<float *>(vd + (size_t)nkv * npos * 128);
    const dim3 dgrid(tiles * (kPfN / 16), nkv);
    const float qjl_factor = sqrtf(2.0f / 3.14159265f) / (float)tq->hd;
    IM_CUDA_CHECK(launch_k(tq->n_bits == 4 ? tq_dequant_rows_kernel<4> : tq_dequant_rows_kernel<8>, dgrid, dim3(256), 0, st, kc, vc, (const float *)tq->k_cb,
                           (const float *)tq->v_cb, ks, vs, krn, qjl_factor, kd, vd, factors, slot, nkv, max_seq, npos));
    PromptQuery pq{};
    pq.q = q.q; pq.stride = q.stride; pq.qw = q.qw; pq.eps = q.eps; pq.rope = PromptRope{q.cosc, q.sinc, q.rotary_dim, base_pos, slot, pos_dev};
    pq.signs = tq->signs; pq.qjl_t = tq->qjl_t; pq.out = static_cast<__half *>(q_rows); pq.nh = nh; pq.T = T;
    const int rows = T * nh;
    IM_CUDA_CHECK(launch_k(tq_prompt_query_kernel, dim3((rows + kQWarps * 16 - 1) / (kQWarps * 16)), dim3(kQWarps * 32), 0, st, pq));
    if (const int rc = flash_prepare(tq->dev); rc != IM_OK) return rc;
    FlashArgs f;
    f.T = T; f.heads = nh; f.group = nh / nkv;
    f.q.base = q_rows; f.q.rows = T; f.q.ld = (long long)nh * 256; f.q.head_cols = 256; f.q.blocks = 4;
    f.k.base = kd; f.k.rows = (long long)nkv * npos; f.k.ld = 256; f.k.head_rows = npos; f.k.blocks = 4;
    f.v.base = vd; f.v.rows = (long long)nkv * npos; f.v.ld = 128; f.v.head_rows = npos; f.v.blocks = 2;
    f.base_pos = base_pos; f.slot = slot; f.n_max = npos; f.pos_dev = pos_dev; f.scale = attn_scale;
    f.scales = factors; f.scale_tiles = tiles; f.signs = tq->signs;
    f.out = out; f.ldo = nh * kHd; f.out_head = kHd; f.err = tq->dev->err_flag;
    return flash_run(f, st);
}

}  // namespace im
