// Causal attention of a prompt chunk on the 5th-generation tensor cores: softmax(scale * Q K^T [, sink]) V [* sigmoid(gate)] of
// one sequence, a chunk of T tokens against the positions cached before them and themselves.
//
// A CTA owns 256 consecutive tokens of one head as two halves of 128 rows (UMMA M = 128). Positions come in tiles of PN rows by
// cp.async.bulk.tensor into the 128-byte swizzle, one tile serving both halves. Per half and tile
//     S = Q K^T    both operands K-major in shared memory, accumulator S in tensor memory (f32)
//     P = exp2(S)  one thread per row: scores to registers, running maximum and sum in f32, weights back to tensor memory as 16-bit
//                  pairs over the scores' own columns (two terms: the rounded weight and what the rounding left, side by side)
//     O += P V     A operand P from tensor memory, B operand V with the head dimension contiguous (MN-major), f32 accumulator
// The two halves take turns: while one half's four warps exponentiate, the other half's products run. Tensor memory is full:
// scores / weights of two halves in 256 columns, outputs in 256 more. An accumulator is rescaled only when a row's maximum has grown by
// more than 2^8 since the last time (weights up to 2^8 are representable and the normalisation uses the same maximum; the scheme, like that of two
// halves in turns, is known from published attention kernels for this architecture, FlashAttention-4).
//
// Order: every product is issued by one thread, so S of the next tile cannot overtake the P V product that still reads the same
// columns, and a score barrier (tcgen05.commit) says that the half's earlier P V product is complete too: its softmax warps may
// then rescale O. All waits are bounded: a wait that runs out sets the device error word, every warp then runs to its end.
//
// Bound: 2 x 128 x PN x (DK + 128 per term) products and 128 x PN exponentials (16 a clock and SM) per half and tile; both are about
// 1000 clocks at DK = PN = 128. 2048 tokens, 16 heads: 128 columns fp16 84 us, two bf16 terms 92 us, 192/128 columns 89 us (mma.sync kernels: 221, 255, 265).
#include <cuda_bf16.h>
#include <math.h>

#include <type_traits>

#include "flash_tc.cuh"
#include "tmap.cuh"
#include "v2_device.cuh"

namespace im {

namespace {

constexpr int kFM = 128;                 // rows of a half
constexpr int kFDV = 128;                // value columns
constexpr int kFThreads = 10 * 32;       // four softmax warps per half, one warp for the copies, one for the products
constexpr int kFCopyWarp = 8, kFMmaWarp = 9;
constexpr float kLazy = 8.0f;            // growth of a row's maximum (in powers of two) that is left in the weights

struct FlashParams {
    FlashArgs a;
    float scale2;                        // scale / ln 2: scores in powers of two
};

// TQ: rows of a quantized cache (KB = 4): two score accumulators, factors per position, outputs rotated back
template <int KB, int PN>
struct FlashShape {
    static constexpr bool kTq = KB == 4;
    static constexpr int kScore = kTq ? 2 * PN : PN;    // tensor-memory columns of a half's scores
    static constexpr int kFactors = kTq ? 3 * PN * 4 : 0;
    static constexpr int kQ = 2 * KB * kFM * 128;       // both halves' queries
    static constexpr int kK = KB * PN * 128, kV = 2 * PN * 128;
    static constexpr int kStages = KB == 3 ? 3 : 2;
    static constexpr int kSmem = 1024 + kQ + kStages * (kK + kV + kFactors) + (4 * kStages + 7) * 8 + 16;
};

__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr, uint32_t lbo_bytes) {
    // shared-memory matrix descriptor, 128-byte swizzle (layout type 2), version 1; stride offset 1024 B between groups of eight
    // rows of 128 B. The leading offset matters for MN-major operands only: bytes between 64-element column blocks.
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0)
                 : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {  // A operand in tensor memory
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0)
                 : "memory");
}
__device__ __forceinline__ void commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {  // x: a multiple of eight elements (flash_takes)
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)), "l"(map),
                 "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {  // 16-byte aligned
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t *r) {  // no wait: tmem_wait_ld
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32"
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
        " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void st32(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32],"
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
        " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};\n" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]),
        "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// The whole warp waits; the hardware suspends a try_wait for a while, so no back-off on these short waits.
__device__ __forceinline__ bool wait_for(uint64_t *bar, uint32_t parity, int *err) {
    bool ok = mbar_try_wait(bar, parity);
    if (!ok) {
        const unsigned long long t0 = global_ns();
        for (unsigned i = 1; !ok; i++) {
            ok = mbar_try_wait(bar, parity);
            if (!ok && (i & 255u) == 0 && global_ns() - t0 > kWaitLimitNs) {
                atomicExch(err, 1);
                break;
            }
        }
    }
    return __all_sync(0xffffffffu, ok);
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    if (BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
    if (BF16) return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
    return __half22float2(*reinterpret_cast<const __half2 *>(&u));
}
__device__ __forceinline__ int chunk_start(int chunk, int pos) { return chunk > 0 ? pos / chunk * chunk : 0; }

template <bool BF16>
__device__ __forceinline__ const uint32_t *row_words(const FlashRows &r, int head, int row) {
    return reinterpret_cast<const uint32_t *>(static_cast<const uint16_t *>(r.base) + (r.row0 + head * r.head_rows + row) * r.ld + r.col0 + (long long)head * r.head_cols);
}
// Stores 32 outputs of a row, columns c .. c + 31, o already normalised.
template <bool BF16>
__device__ __forceinline__ void store32(const FlashArgs &a, int tok, int h, int c, const float *o) {
    uint4 *dst = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(a.out) + (size_t)tok * a.ldo + (size_t)h * a.out_head + c);
    const uint4 *gate = a.gate ? reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(a.gate) + (size_t)tok * a.ldg + (size_t)h * a.gate_head + c) : nullptr;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = o[8 * i + j];
        if (gate) {
            const uint4 g = gate[i];
            const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 z = unpack2<BF16>(gw[j]);
                v[2 * j] *= 1.0f / (1.0f + expf(-z.x));
                v[2 * j + 1] *= 1.0f / (1.0f + expf(-z.y));
            }
        }
        dst[i] = make_uint4(pack2<BF16>(v[0], v[1]), pack2<BF16>(v[2], v[3]), pack2<BF16>(v[4], v[5]), pack2<BF16>(v[6], v[7]));
    }
}
// A row whose tensor-core result is not finite, from its own positions alone: a product with a weight of zero turns an infinite
// or missing value of a position the row does not see into a NaN, here such a position is not touched.
template <bool BF16>
__device__ __noinline__ void plain_row(const FlashParams &p, int h, int tok, int from, int lim, float sink) {
    const FlashArgs &a = p.a;
    const int kvh = h / a.group;
    float o[kFDV], m = -INFINITY, l = 0.0f;
    for (int c = 0; c < kFDV; c++) o[c] = 0.0f;
    const uint32_t *q = row_words<BF16>(a.q, h, tok);
    for (int pos = from; pos <= lim; pos++) {
        float s = 0.0f;
        const uint32_t *k = row_words<BF16>(a.k, kvh, pos);
        for (int j = 0; j < a.k.blocks * 32; j++) {
            const float2 x = unpack2<BF16>(q[j]), y = unpack2<BF16>(k[j]);
            s = fmaf(x.x, y.x, fmaf(x.y, y.y, s));
        }
        if (a.k2.blocks) {
            k = row_words<BF16>(a.k2, kvh, pos);
            for (int j = 0; j < a.k2.blocks * 32; j++) {
                const float2 x = unpack2<BF16>(q[a.k.blocks * 32 + j]), y = unpack2<BF16>(k[j]);
                s = fmaf(x.x, y.x, fmaf(x.y, y.y, s));
            }
        }
        s *= p.scale2;
        const float m_new = fmaxf(m, s), corr = m_new == -INFINITY ? 1.0f : exp2f(m - m_new), w = s == -INFINITY ? 0.0f : exp2f(s - m_new);
        m = m_new;
        l = l * corr + w;
        const uint32_t *v = row_words<BF16>(a.v, kvh, pos);
        for (int j = 0; j < kFDV / 2; j++) {
            const float2 y = unpack2<BF16>(v[j]);
            o[2 * j] = fmaf(w, y.x, o[2 * j] * corr);
            o[2 * j + 1] = fmaf(w, y.y, o[2 * j + 1] * corr);
        }
    }
    const float gm = fmaxf(m, sink), c = m == -INFINITY ? 0.0f : exp2f(m - gm);
    const float inv = c / fmaxf(l * c + (sink == -INFINITY ? 0.0f : exp2f(sink - gm)), 1e-10f);
    for (int i = 0; i < kFDV; i++) o[i] *= inv;
    for (int i = 0; i < kFDV; i += 32) store32<BF16>(a, tok, h, i, o + i);
}

// grid (heads, ceil(T / 256)). KB: 64-column blocks of a key; PN: positions of a tile; TERMS: 16-bit terms of a weight.
template <bool BF16, int KB, int PN, int TERMS>
__global__ void __launch_bounds__(kFThreads, 1)
    flash_tc_kernel(const __grid_constant__ FlashParams p, const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tk2,
                    const __grid_constant__ CUtensorMap tv) {
    using Shape = FlashShape<KB, PN>;
    constexpr int ST = Shape::kStages, kScore = Shape::kScore;
    constexpr bool TQ = Shape::kTq;
    static_assert(TERMS * PN / 2 <= PN, "the weights lie over the scores");
    static_assert(2 * kScore <= 256, "scores and outputs fill tensor memory");
    extern __shared__ __align__(1024) unsigned char flash_smem[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(flash_smem) + 1023) & ~(uintptr_t)1023);
    unsigned char *Qs = smem, *Ks = smem + Shape::kQ, *Vs = Ks + ST * Shape::kK;
    float *Fs = reinterpret_cast<float *>(Vs + ST * Shape::kV);
    uint64_t *kfull = reinterpret_cast<uint64_t *>(Vs + ST * (Shape::kV + Shape::kFactors)), *kempty = kfull + ST, *vfull = kempty + ST, *vempty = vfull + ST;
    uint64_t *qfull = vempty + ST, *sfull = qfull + 1, *pfull = sfull + 2, *ofull = pfull + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(ofull + 2);
    const FlashArgs &a = p.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tb = gridDim.y - 1 - blockIdx.y, h = blockIdx.x, kvh = h / a.group;  // every head's latest (longest) block first
    if (tid == 0) {
        for (int i = 0; i < ST; i++) {
            mbar_init(&kfull[i], 1);
            mbar_init(&kempty[i], 1);
            mbar_init(&vfull[i], 1);
            mbar_init(&vempty[i], 1);
        }
        mbar_init(qfull, 1);
        for (int i = 0; i < 2; i++) {
            mbar_init(&sfull[i], 1);
            mbar_init(&pfull[i], 4);
            mbar_init(&ofull[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kFMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();  // after the allocation: a successor on this SM cannot take the columns first
    pdl_wait();
    const int P = a.base_pos + (a.pos_dev ? a.pos_dev[a.slot] : 0);
    const int t0 = tb * 2 * kFM, halves = a.T - t0 > kFM ? 2 : 1;
    const int n_begin = chunk_start(a.chunk, P + t0);
    int lo[2], hi[2];  // tiles of each half, counted from n_begin
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int first = t0 + i * kFM, last = min(first + kFM, a.T) - 1;
        lo[i] = i < halves ? (chunk_start(a.chunk, P + first) - n_begin) / PN : 0;
        hi[i] = i < halves ? max((min(P + last + 1, a.n_max) - n_begin + PN - 1) / PN, lo[i] + 1) : 0;
    }
    const int n_end = min(P + min(t0 + halves * kFM, a.T), a.n_max), tiles = max(hi[0], hi[1]);
    bool ok = true;

    if (warp == kFCopyWarp) {
        if (lane == 0) {
            mbar_expect_tx(qfull, (uint32_t)(halves * KB * kFM * 128));
            for (int i = 0; i < halves; i++)
                for (int b = 0; b < KB; b++)
                    tma_2d(Qs + (size_t)(i * KB + b) * kFM * 128, &tq, a.q.col0 + h * a.q.head_cols + b * 64, (int)(a.q.row0 + h * a.q.head_rows) + t0 + i * kFM, qfull);
        }
        __syncwarp();
        const int kx = a.k.col0 + kvh * a.k.head_cols, k2x = a.k2.col0 + kvh * a.k2.head_cols, vx = a.v.col0 + kvh * a.v.head_cols;
        const int ky = (int)(a.k.row0 + kvh * a.k.head_rows) + n_begin, k2y = (int)(a.k2.row0 + kvh * a.k2.head_rows) + n_begin;
        const int vy = (int)(a.v.row0 + kvh * a.v.head_rows) + n_begin;
        for (int it = 0; it < tiles; it++) {
            const int s = it % ST, use = it / ST;
            if (ok && use > 0 && !wait_for(&kempty[s], (use - 1) & 1, a.err)) ok = false;
            if (lane == 0 && ok) {
                mbar_expect_tx(&kfull[s], (uint32_t)Shape::kK);
                for (int b = 0; b < KB; b++) {
                    unsigned char *dst = Ks + (size_t)s * Shape::kK + (size_t)b * PN * 128;
                    if (b < a.k.blocks) tma_2d(dst, &tk, kx + b * 64, ky + it * PN, &kfull[s]);
                    else tma_2d(dst, &tk2, k2x + (b - a.k.blocks) * 64, k2y + it * PN, &kfull[s]);
                }
            }
            __syncwarp();
            if (ok && use > 0 && !wait_for(&vempty[s], (use - 1) & 1, a.err)) ok = false;
            if (lane == 0 && ok) {
                mbar_expect_tx(&vfull[s], (uint32_t)(Shape::kV + Shape::kFactors));
                if constexpr (TQ) bulk_copy(Fs + s * 3 * PN, a.scales + ((size_t)kvh * a.scale_tiles + it) * (3 * PN), Shape::kFactors, &vfull[s]);
                for (int b = 0; b < 2; b++) tma_2d(Vs + (size_t)s * Shape::kV + (size_t)b * PN * 128, &tv, vx + b * 64, vy + it * PN, &vfull[s]);
            }
            __syncwarp();
        }
    } else if (warp == kFMmaWarp) {
        // instruction descriptors: f32 accumulator, fp16 (0) or bf16 (1) operands in bits 7-9 and 10-12, B MN-major in bit 16,
        // N >> 3 in bits 17-22, M >> 4 in bits 24-28
        constexpr uint32_t kType = (1u << 4) | (BF16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(kFM >> 4) << 24);
        constexpr uint32_t kS = kType | ((uint32_t)(PN >> 3) << 17), kPV = kType | (1u << 16) | ((uint32_t)(kFDV >> 3) << 17);
        if (ok && !wait_for(qfull, 0, a.err)) ok = false;
        int turns[2] = {0, 0};
        for (int it = 0; it <= tiles; it++) {
            const int s = it % ST, sp = (it + ST - 1) % ST;
            for (int i = 0; i < halves; i++) {
                if (it > lo[i] && it <= hi[i]) {  // P V of tile it - 1
                    if (ok && !wait_for(&pfull[i], turns[i] & 1, a.err)) ok = false;
                    turns[i]++;
                    if (ok && !wait_for(&vfull[sp], ((it - 1) / ST) & 1, a.err)) ok = false;
                    if (it == tiles && n_begin + tiles * PN > n_end && ok) {
                        // rows past the last position hold whatever the buffer held: their weights are zero, but zero times a NaN
                        // is none (done before the first product that reads the tile; the second half finds zeros already)
                        const int r0 = max(n_end - (n_begin + (tiles - 1) * PN), 0);
                        for (int x = lane; x < 2 * (PN - r0) * 8; x += 32) {
                            const int b = x / ((PN - r0) * 8), y = x % ((PN - r0) * 8);
                            *reinterpret_cast<uint4 *>(Vs + (size_t)sp * Shape::kV + (size_t)b * PN * 128 + (size_t)r0 * 128 + (size_t)y * 16) = make_uint4(0, 0, 0, 0);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                    }
                    fence_after();
                    if (lane == 0 && ok) {
                        const uint32_t v0 = smem_u32(Vs + (size_t)sp * Shape::kV), pw = tmem + (uint32_t)(i * kScore), o = tmem + 256u + (uint32_t)(i * kFDV);
#pragma unroll
                        for (int t = 0; t < TERMS; t++)
#pragma unroll
                            for (int j = 0; j < PN / 16; j++)
                                mma_ts(o, pw + (uint32_t)(t * PN / 2 + j * 8), desc_sw128(v0 + j * 2048, PN * 128), kPV, (it - 1 > lo[i] || t > 0 || j > 0) ? 1u : 0u);
                        if (it == hi[i]) commit(&ofull[i]);
                    }
                    __syncwarp();
                }
                if (it >= lo[i] && it < hi[i]) {
                    if (ok && !wait_for(&kfull[s], (it / ST) & 1, a.err)) ok = false;
                    fence_after();
                    if (lane == 0 && ok) {
                        const uint32_t q0 = smem_u32(Qs + (size_t)i * KB * kFM * 128), k0 = smem_u32(Ks + (size_t)s * Shape::kK);
#pragma unroll
                        for (int j = 0; j < KB * 4; j++)
                            mma_ss(tmem + (uint32_t)(i * kScore + (TQ && j >= 8 ? PN : 0)), desc_sw128(q0 + (j >> 2) * (kFM * 128) + (j & 3) * 32, 16),
                                   desc_sw128(k0 + (j >> 2) * (PN * 128) + (j & 3) * 32, 16), kS, (TQ ? j & 7 : j) > 0 ? 1u : 0u);
                        commit(&sfull[i]);
                    }
                    __syncwarp();
                }
            }
            if (lane == 0 && ok) {
                if (it > 0) commit(&vempty[sp]);
                if (it < tiles) commit(&kempty[s]);
            }
            __syncwarp();
        }
    } else {
        const int i = warp >> 2, row = (warp & 3) * 32 + lane, tok = t0 + i * kFM + row;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t ts = tmem + lanes + (uint32_t)(i * kScore), to = tmem + lanes + 256u + (uint32_t)(i * kFDV);
        const float sink = a.sink ? a.sink[h] * 1.4426950408889634f : -INFINITY;
        if (i < halves) {
            const int first = P + t0 + i * kFM, last = P + min(t0 + i * kFM + kFM, a.T) - 1;
            const int lim = min(P + min(tok, a.T - 1), a.n_max - 1), from = chunk_start(a.chunk, lim);  // rows past the last token repeat it (not stored)
            const int from_last = chunk_start(a.chunk, last);
            float m = -INFINITY, l = 0.0f;
            for (int it = lo[i]; it < hi[i]; it++) {
                if (ok && !wait_for(&sfull[i], (it - lo[i]) & 1, a.err)) ok = false;
                fence_after();
                const int p0 = n_begin + it * PN;
                float s[PN], lazy = kLazy;
                bool odd = false;  // (quantized caches) a factor of this tile is not finite
                const float *ks = Fs + (it % ST) * 3 * PN, *kr = ks + PN, *vs = kr + PN;
                if constexpr (TQ) {
                    if (ok && !wait_for(&vfull[it % ST], (it / ST) & 1, a.err)) ok = false;
                    // a weight times vs has to stay in fp16's range: where vs is large the maximum follows at once
                    const unsigned vm = __reduce_max_sync(0xffffffffu, max(__float_as_uint(fabsf(vs[lane])), __float_as_uint(fabsf(vs[lane + 32]))));
                    if (vm > __float_as_uint(128.0f)) lazy = 0.0f;
                    odd = vm >= 0x7f800000u;
#pragma unroll
                    for (int c = 0; c < PN; c += 32) {
                        float t[32];
                        ld32(ts + (uint32_t)c, reinterpret_cast<uint32_t *>(s) + c);
                        ld32(ts + (uint32_t)(PN + c), reinterpret_cast<uint32_t *>(t));
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 a4 = *reinterpret_cast<const float4 *>(ks + c + j), b4 = *reinterpret_cast<const float4 *>(kr + c + j);
                            s[c + j] = a4.x * fmaf(b4.x, t[j], s[c + j]);
                            s[c + j + 1] = a4.y * fmaf(b4.y, t[j + 1], s[c + j + 1]);
                            s[c + j + 2] = a4.z * fmaf(b4.z, t[j + 2], s[c + j + 2]);
                            s[c + j + 3] = a4.w * fmaf(b4.w, t[j + 3], s[c + j + 3]);
                        }
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < PN; c += 32) ld32(ts + (uint32_t)c, reinterpret_cast<uint32_t *>(s) + c);
                    tmem_wait_ld();
                }
                if (p0 + PN - 1 > first || p0 < from_last || p0 + PN > a.n_max) {  // some row does not see all of the tile
                    const float hide = p.scale2 > 0.0f ? -INFINITY : INFINITY;
#pragma unroll
                    for (int c = 0; c < PN; c++) s[c] = (p0 + c >= from && p0 + c <= lim) ? s[c] : hide;
                }
                float mx[4];
                if (p.scale2 > 0.0f) {
#pragma unroll
                    for (int c = 0; c < 4; c++) mx[c] = s[c];
#pragma unroll
                    for (int c = 4; c < PN; c++) mx[c & 3] = fmaxf(mx[c & 3], s[c]);
                    mx[0] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                } else {
#pragma unroll
                    for (int c = 0; c < 4; c++) mx[c] = s[c];
#pragma unroll
                    for (int c = 4; c < PN; c++) mx[c & 3] = fminf(mx[c & 3], s[c]);
                    mx[0] = fminf(fminf(mx[0], mx[1]), fminf(mx[2], mx[3]));
                }
                const float top = mx[0] * p.scale2;
                if (__any_sync(0xffffffffu, top > m + lazy)) {  // (-inf + anything is -inf: a row's first visible position is one)
                    const float m_new = fmaxf(m, top), corr = m_new == -INFINITY ? 1.0f : ex2(m - m_new);
                    m = m_new;
                    l *= corr;
                    if (it > lo[i]) {
#pragma unroll 1
                        for (int c = 0; c < kFDV; c += 32) {
                            uint32_t o[32];
                            ld32(to + (uint32_t)c, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int j = 0; j < 32; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
                            st32(to + (uint32_t)c, o);
                        }
                    }
                }
                const float base = m == -INFINITY ? 0.0f : m;
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                // 64 columns at a time: 32 words of weights and, with two terms, 32 words of what their rounding left. ODD: zero times a factor that is
                // not finite would be a NaN in rows that do not see its position
                auto weights = [&](auto ODD) {
#pragma unroll
                    for (int c = 0; c < PN; c += 64) {
                        uint32_t w[32], w2[32];
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const float x0 = ex2(fmaf(s[c + 2 * j], p.scale2, -base)), x1 = ex2(fmaf(s[c + 2 * j + 1], p.scale2, -base));
                            sum[(2 * j) & 3] += x0;
                            sum[(2 * j + 1) & 3] += x1;
                            if constexpr (TQ) {
                                float2 v2 = *reinterpret_cast<const float2 *>(vs + c + 2 * j);
                                if constexpr (ODD) {
                                    if (p0 + c + 2 * j > lim) v2.x = 0.0f;
                                    if (p0 + c + 2 * j + 1 > lim) v2.y = 0.0f;
                                }
                                w[j] = pack2<BF16>(x0 * v2.x, x1 * v2.y);
                            } else {
                                w[j] = pack2<BF16>(x0, x1);
                            }
                            if (TERMS > 1) {
                                const float2 r = unpack2<BF16>(w[j]);
                                w2[j] = pack2<BF16>(x0 - r.x, x1 - r.y);
                            }
                        }
                        st32(ts + (uint32_t)(c / 2), w);
                        if (TERMS > 1) st32(ts + (uint32_t)(PN / 2 + c / 2), w2);
                    }
                };
                if (TQ && odd) weights(std::bool_constant<TQ>());
                else weights(std::false_type());
                l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
                tmem_wait_st();
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&pfull[i]);
            }
            if (ok && !wait_for(&ofull[i], 0, a.err)) ok = false;
            fence_after();
            const float gm = fmaxf(m, sink), c0 = m == -INFINITY ? 0.0f : ex2(m - gm);
            const float inv = c0 / fmaxf(l * c0 + (sink == -INFINITY ? 0.0f : ex2(sink - gm)), 1e-10f);
            if constexpr (TQ) {
                // back from the rotated space: signs, butterflies over the row's 128 values, signs / sqrt(128); the widest butterfly first, so
                // that the rest works on 64 registers at a time
                const float4 *sg = reinterpret_cast<const float4 *>(a.signs);
#pragma unroll 1
                for (int c = 0; c < 64; c += 32) {
                    uint32_t x[32], y[32];
                    ld32(to + (uint32_t)c, x);
                    ld32(to + (uint32_t)c + 64u, y);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        const float u = __uint_as_float(x[j]) * (inv * __ldg(a.signs + c + j)), v = __uint_as_float(y[j]) * (inv * __ldg(a.signs + c + 64 + j));
                        x[j] = __float_as_uint(u + v);
                        y[j] = __float_as_uint(u - v);
                    }
                    st32(to + (uint32_t)c, x);
                    st32(to + (uint32_t)c + 64u, y);
                }
                tmem_wait_st();
                constexpr float kRoot = 0.08838834764831845f;  // 1 / sqrt(128)
#pragma unroll 1
                for (int c = 0; c < kFDV; c += 64) {
                    float o[64];
                    ld32(to + (uint32_t)c, reinterpret_cast<uint32_t *>(o));
                    ld32(to + (uint32_t)c + 32u, reinterpret_cast<uint32_t *>(o) + 32);
                    tmem_wait_ld();
#pragma unroll
                    for (int step = 1; step < 64; step *= 2)
#pragma unroll
                        for (int j = 0; j < 64; j++)
                            if (!(j & step)) {
                                const float x = o[j], y = o[j + step];
                                o[j] = x + y;
                                o[j + step] = x - y;
                            }
#pragma unroll
                    for (int j = 0; j < 64; j += 4) {
                        const float4 g = __ldg(sg + (c + j) / 4);
                        o[j] *= kRoot * g.x; o[j + 1] *= kRoot * g.y; o[j + 2] *= kRoot * g.z; o[j + 3] *= kRoot * g.w;
                    }
                    if (tok < a.T && ok) {
                        store32<BF16>(a, tok, h, c, o);
                        store32<BF16>(a, tok, h, c + 32, o + 32);
                    }
                }
            }
            bool finite = true;
#pragma unroll 1
            for (int c = 0; c < kFDV && !TQ; c += 32) {
                uint32_t o[32];
                ld32(to + (uint32_t)c, o);
                tmem_wait_ld();
                float v[32], worst = 0.0f;
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    v[j] = __uint_as_float(o[j]) * inv;
                    worst += v[j] * 0.0f;  // zero unless a value is not finite
                }
                finite = finite && worst == 0.0f;
                if (tok < a.T && ok) store32<BF16>(a, tok, h, c, v);
            }
            if (!finite && tok < a.T && ok) plain_row<BF16>(p, h, tok, from, lim, sink);
        }
    }
    fence_before();
    sync_and_settle(ok);
    if (warp == kFMmaWarp) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <bool BF16, int KB, int PN, int TERMS>
int launch(const FlashArgs &a, cudaStream_t st) {
    alignas(64) CUtensorMap tq, tk, tk2, tv;
    auto map = [&](const FlashRows &r, int rows, CUtensorMap *m) { return tmap_2d(r.base, BF16, r.rows, r.ld, r.ld, rows, m); };
    int rc = map(a.q, kFM, &tq);
    if (rc == IM_OK) rc = map(a.k, PN, &tk);
    if (rc == IM_OK) rc = map(a.k2.blocks ? a.k2 : a.k, PN, &tk2);
    if (rc == IM_OK) rc = map(a.v, PN, &tv);
    if (rc != IM_OK) return rc;
    FlashParams p;
    p.a = a;
    p.scale2 = a.scale * 1.4426950408889634f;
    if (p.scale2 == 0.0f) p.scale2 = 1e-30f;  // every position alike, without 0 * inf at the hidden ones
    IM_CUDA_CHECK(launch_k(flash_tc_kernel<BF16, KB, PN, TERMS>, dim3(a.heads, (a.T + 2 * kFM - 1) / (2 * kFM)), dim3(kFThreads), (size_t)FlashShape<KB, PN>::kSmem, st, p,
                           tq, tk, tk2, tv));
    return IM_OK;
}

}  // namespace

bool flash_takes(const FlashArgs &a) {
    auto fits = [](const FlashRows &r) {
        return reinterpret_cast<uintptr_t>(r.base) % 16 == 0 && r.ld % 8 == 0 && r.ld < (1ll << 31) && r.rows < (1ll << 31) && r.col0 % 8 == 0 && r.head_cols % 8 == 0;
    };
    const int kb = a.k.blocks + a.k2.blocks;
    const bool tq = a.scales != nullptr;
    return a.T > 0 && a.T <= 65535 * 2 * kFM && a.heads > 0 && a.group > 0 && a.heads % a.group == 0 && (tq ? kb == 4 && a.chunk == 0 && a.signs : kb == 2 || kb == 3) && a.q.blocks == kb && a.v.blocks == 2 && fits(a.q) &&
           fits(a.k) && (!a.k2.blocks || fits(a.k2)) && fits(a.v) && reinterpret_cast<uintptr_t>(a.out) % 16 == 0 && a.ldo % 8 == 0 && a.out_head % 8 == 0 &&
           (!a.gate || (reinterpret_cast<uintptr_t>(a.gate) % 16 == 0 && a.ldg % 8 == 0 && a.gate_head % 8 == 0));
}

int flash_prepare(const Device *dev) {
    static DeviceOnce once;
    if (!once.first(dev->ordinal)) return IM_OK;
#define IM_SMEM(B, KB, PN, TERMS) \
    IM_CUDA_CHECK(cudaFuncSetAttribute((flash_tc_kernel<B, KB, PN, TERMS>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FlashShape<KB, PN>::kSmem))
    IM_SMEM(false, 2, 128, 1);
    IM_SMEM(true, 2, 128, 2);
    IM_SMEM(true, 3, 64, 2);
    IM_SMEM(false, 4, 64, 1);
#undef IM_SMEM
    return IM_OK;
}

int flash_run(const FlashArgs &a, cudaStream_t st) {
    if (!flash_takes(a)) return IM_ERR_BOUNDS;
    const int kb = a.k.blocks + a.k2.blocks;
    if (!a.bf16 && !a.two_terms && kb == 2) return launch<false, 2, 128, 1>(a, st);
    if (a.bf16 && a.two_terms && kb == 2) return launch<true, 2, 128, 2>(a, st);
    if (a.bf16 && a.two_terms && kb == 3) return launch<true, 3, 64, 2>(a, st);
    if (!a.bf16 && !a.two_terms && kb == 4) return launch<false, 4, 64, 1>(a, st);
    return IM_ERR_BOUNDS;
}

}  // namespace im
