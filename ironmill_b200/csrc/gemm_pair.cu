// Projections of many tokens (prompts): D[256 weight rows x TN tokens] per pair of CTAs, tcgen05.mma.cta_group::2.
//
// The single-CTA kernels (dense.cu, gemm_tc.cu) pull 128 weight rows and 256 tokens into an SM per product of 128 x 256: at 48 KB per
// 64 columns the traffic from L2 (about 45 bytes a clock and SM measured) takes twice the time of the product.  A pair shares both
// operands: each CTA holds 128 of the 256 rows and half of the tokens, 32 KB for the same product (20 KB where the weights arrive as
// 4-bit codes).  Persistent: a pair walks its tiles with two accumulators in tensor memory, so that the epilogue warps store one tile while the
// next one's products run.
//
// Weights: bf16 by cp.async.bulk.tensor (BITS = 0), or codes that sixteen warps of each CTA dequantise into the operand layout
// (BITS = 4, 8; rounding as in gemm_tc.cu: f16((q - z) s)); with two weights, even rows come from the first (gate) and odd rows from the
// second (up), and the epilogue forms silu(gate) * up from neighbouring lanes.  Tokens: cp.async.bulk.tensor, each CTA its half.
//
// Hand-over: the leader's full barrier of a stage counts its own announcement of both CTAs' bytes (and the weight warps of both), the
// leader issues the products, tcgen05.commit frees the stage and publishes the accumulator in both CTAs.  Every wait is bounded; a wait that
// runs out sets the device error word, every warp then runs to its end and the tensor memory is freed.
//
// Bound: the tensor pipe (512 clocks per 64 columns of a 128 x 256 half tile).  Measured back to back, bf16 2048 tokens x
// 28672 x 4096: 343 us, 1404 TFLOP/s; 20032 x 2048: 131 us (128-row kernel 164 us alone); 4-bit codes 28672 x 4096: 411 us, 1172 TFLOP/s, 4096 x 14336: 216 us;
// there the weight warps bound: without any epilogue the same launches reach 1240 TFLOP/s.
//
// The weight warps of the second CTA arrive at the leader's barrier with the default scope. What that barrier has to order is the issue of the products: a
// weight tile lies in the shared memory of the CTA that converted it, only that SM's tensor core reads it, and fence.proxy.async.shared::cta, which every
// lane executes before its warp arrives, is complete when the stores are visible there. A proxy fence for all spaces and cluster-scope semantics made the warps wait
// for their own loads of codes in flight: 1.5 times the time.
#include <cuda.h>

#include <algorithm>

#include "dense_epi.cuh"
#include "dequant.cuh"
#include "gemm_pair.cuh"
#include "tmap.cuh"
#include "v2_device.cuh"

namespace im {

namespace {

constexpr int kPRows = 128;   // weight rows of a CTA
constexpr int kPAhead4 = 4, kPAhead8 = 2;  // stages of codes in flight in registers

template <int TN, int BITS>
struct PairShape {
    static constexpr int kK = BITS ? 128 : 64;                     // columns of a stage: a quantisation group, or one swizzle atom
    static constexpr int kA = kPRows * kK * 2, kB = TN / 2 * kK * 2;
    static constexpr int kStages = 192 * 1024 / (kA + kB);
    static constexpr int kWeightWarps = BITS ? 16 : 0, kEpiWarps = BITS ? 4 : 8;
    static constexpr int kThreads = (kWeightWarps + kEpiWarps + 2) * 32;
    static constexpr int kSmem = 1024 + kStages * (kA + kB) + (2 * kStages + 4) * 8 + 16;
};

struct PairGemm {
    int N, M, kstages;        // result rows (both weights' when there are two), tokens, stages per tile
    int mtiles, ntiles;       // tiles of TN tokens and of 256 rows
    const uint8_t *codes[2];  // BITS: [rows, K] codes and (scale, zero) pairs of the weight, of even and of odd rows when there are two
    const __half2 *sz[2];
    int K, paired;
    int *err;
    DenseEpi epi;
};

__device__ __forceinline__ uint64_t pair_desc(uint32_t smem_addr) {  // K-major, 128-byte swizzle (see gemm_tc.cu)
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n" ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc),
                 "r"(accumulate), "r"(0)
                 : "memory");
}
// arrives at the barrier of this offset in both CTAs once the products issued so far are complete
__device__ __forceinline__ void pair_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ uint32_t leader_addr(const void *p) {  // the same place in the pair's first CTA
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void arrive_at(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// into this CTA's shared memory, bytes counted on a barrier of the pair; x is a multiple of 64 elements (128 bytes)
__device__ __forceinline__ void pair_tma(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32"
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
// One thread waits, without back-off (the hardware suspends a try_wait for a while); arrivals may come from the other CTA.
__device__ __forceinline__ bool pair_wait(uint64_t *bar, uint32_t parity, int *err) {
    unsigned long long t0 = 0;
    for (unsigned i = 0;; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i == 0) t0 = global_ns();
        if ((i & 255u) == 255u && global_ns() - t0 > kWaitLimitNs) break;
    }
    atomicExch(err, 1);
    return false;
}
__device__ __forceinline__ bool pair_wait_warp(uint64_t *bar, uint32_t parity, int *err) { return __all_sync(0xffffffffu, pair_wait(bar, parity, err)); }

// The weight warps of one CTA: groups of its 128 rows into the ring, tile after tile.  Four neighbouring lanes own the 128 columns of a row
// (whole 32-byte sectors of codes, one (scale, zero) pair); in the upper 64 columns the words are taken in the order 2, 3, 0, 1,
// so that the eight lanes of a store phase hit eight different 16-byte columns of the swizzle.
template <int TN, int BITS>
__device__ __forceinline__ bool weight_warps(const PairGemm &p, unsigned char *As, uint64_t *full, uint64_t *empty, int rank, int pair, int npairs) {
    using S = PairShape<TN, BITS>;
    constexpr int kAhead = BITS == 4 ? kPAhead4 : kPAhead8, kVec = BITS == 4 ? 1 : 2;
    const int tid = threadIdx.x, lane = tid & 31, r = tid >> 2, q = tid & 3, G = p.kstages;
    const int tiles = p.mtiles * p.ntiles, mine = pair < tiles ? (tiles - 1 - pair) / npairs + 1 : 0, total = mine * G;
    const size_t row_bytes = (size_t)p.K * BITS / 8;
    const uint32_t row_off = (uint32_t)((q >> 1) * (kPRows * 128) + (r >> 3) * 1024 + (r & 7) * 128);
    const int c0 = 4 * (q & 1), swap = q & 2, x = r & 7;
    // cursor of the requests, kAhead stages before the conversion
    int at = 0, tile = pair, g = 0;
    const uint8_t *crow = nullptr;
    const __half2 *szrow = nullptr;
    auto point = [&]() {
        const int n = tile / p.mtiles * (2 * kPRows) + rank * kPRows + r, row = p.paired ? n >> 1 : n, which = p.paired ? n & 1 : 0;
        crow = nullptr;
        if (n < p.N) {
            crow = p.codes[which] + (size_t)row * row_bytes + q * (4 * BITS);
            szrow = p.sz[which] + (size_t)row * G;
        }
    };
    uint4 wb[kAhead][kVec];
    __half2 szb[kAhead];
    auto request = [&](int u) {
#pragma unroll
        for (int v = 0; v < kVec; v++) wb[u][v] = make_uint4(0, 0, 0, 0);
        szb[u] = __floats2half2_rn(0.0f, 0.0f);
        if (at < total) {
            if (crow) {
                const uint4 *src = reinterpret_cast<const uint4 *>(crow + (size_t)g * (16 * BITS));
#pragma unroll
                for (int v = 0; v < kVec; v++) wb[u][v] = __ldg(src + v);
                szb[u] = __ldg(szrow + g);
            }
            at++;
            if (++g == G) {
                g = 0;
                tile += npairs;
                if (at < total) point();
            }
        }
    };
    if (total > 0) point();
#pragma unroll
    for (int u = 0; u < kAhead; u++) request(u);
    const uint32_t full0 = leader_addr(full), e = half_exponent();
    auto hand_over = [&](int stage) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> visible to the tensor cores
        __syncwarp();
        if (lane == 0) arrive_at(full0 + stage * 8);
    };
    bool ok = true;
    int s = 0, use = 0, prev = 0;
    for (int base = 0; base < total; base += kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            if (base + u < total) {
                uint4 cw[kVec];
#pragma unroll
                for (int v = 0; v < kVec; v++) cw[v] = wb[u][v];
                const __half2 sz = szb[u];
                request(u);
                // 16-byte chunks c0 .. c0 + 3 of the row, in the order this lane stores them
                uint2 in[4];
                if (BITS == 4) {
                    in[0].x = swap ? cw[0].z : cw[0].x; in[1].x = swap ? cw[0].w : cw[0].y;
                    in[2].x = swap ? cw[0].x : cw[0].z; in[3].x = swap ? cw[0].y : cw[0].w;
                } else {
                    const uint4 a = swap ? cw[kVec - 1] : cw[0], b = swap ? cw[0] : cw[kVec - 1];
                    in[0] = make_uint2(a.x, a.y); in[1] = make_uint2(a.z, a.w); in[2] = make_uint2(b.x, b.y); in[3] = make_uint2(b.z, b.w);
                }
                const GroupScale gs = BITS == 4 ? group_scale(sz) : group_scale_f32(sz);
                uint4 v[4];
                if (__builtin_expect(gs.plain, 1)) {
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] = BITS == 4 ? dequant8_fast(in[i].x, gs, e) : dequant8b_fast(in[i].x, in[i].y, gs);
                } else {
                    const float zf = __high2float(sz), sf = __low2float(sz);
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] = BITS == 4 ? dequant8_slow(in[i].x, zf, sf) : dequant8b_slow(in[i].x, in[i].y, zf, sf);
                }
                // the previous stage is handed over only now: its stores have landed while this one was converted, and the fence does not wait
                if (base + u > 0) hand_over(prev);
                if (ok && use > 0 && !pair_wait_warp(&empty[s], (use - 1) & 1, p.err)) ok = false;
                unsigned char *dst = As + (size_t)s * S::kA + row_off;
#pragma unroll
                for (int i = 0; i < 4; i++) *reinterpret_cast<uint4 *>(dst + (((c0 + (i ^ swap)) ^ x) << 4)) = v[i];
                prev = s;
                if (++s == S::kStages) s = 0, use++;
            }
        }
    }
    if (total > 0) hand_over(prev);
    return ok;
}

template <typename T, int TN, int BITS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairShape<TN, BITS>::kThreads, 1)
    pair_gemm_kernel(const PairGemm p, const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb) {
    using S = PairShape<TN, BITS>;
    constexpr int kCopyWarp = S::kWeightWarps + S::kEpiWarps, kMmaWarp = kCopyWarp + 1, kCols = 2 * TN;
    extern __shared__ __align__(1024) unsigned char pair_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(pair_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *As = smem, *Bs = smem + S::kStages * S::kA;
    uint64_t *full = reinterpret_cast<uint64_t *>(Bs + S::kStages * S::kB), *empty = full + S::kStages, *tfull = empty + S::kStages, *tempty = tfull + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tempty + 2);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, npairs = gridDim.x >> 1, tiles = p.mtiles * p.ntiles;
    pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < S::kStages; i++) {
            mbar_init(&full[i], 1 + 2 * S::kWeightWarps);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], 2 * S::kEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();  // the other CTA's barriers and tensor memory exist
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *tmem_slot;
    if (warp >= S::kWeightWarps) pdl_wait();  // the weight warps read constants and write shared memory only

    bool ok = true;
    if (warp < S::kWeightWarps) {
        if constexpr (BITS != 0) ok = weight_warps<TN, BITS>(p, As, full, empty, rank, pair, npairs);
    } else if (warp == kCopyWarp) {
        if (lane == 0) {
            const uint32_t full0 = leader_addr(full);
            int s = 0, use = 0;
            for (int w = pair; w < tiles; w += npairs) {
                const int m0 = w % p.mtiles * TN + rank * (TN / 2), n0 = w / p.mtiles * (2 * kPRows) + rank * kPRows;
                for (int k = 0; k < p.kstages; k++) {
                    if (ok && use > 0 && !pair_wait(&empty[s], (use - 1) & 1, p.err)) ok = false;
                    if (ok) {
                        if (rank == 0) mbar_expect_tx(&full[s], 2u * (uint32_t)(S::kB + (BITS ? 0 : S::kA)));
                        unsigned char *b = Bs + (size_t)s * S::kB;
                        if constexpr (BITS == 0) pair_tma(As + (size_t)s * S::kA, &ta, k * 64, n0, full0 + s * 8);
                        pair_tma(b, &tb, k * S::kK, m0, full0 + s * 8);
                        if constexpr (BITS != 0) pair_tma(b + TN / 2 * 128, &tb, k * S::kK + 64, m0, full0 + s * 8);
                    }
                    if (++s == S::kStages) s = 0, use++;
                }
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        if (lane == 0 && rank == 0) {
            // f32 accumulator, fp16 (0) or bf16 (1) operands, both K-major, N >> 3 in bits 17-22, M = 256: M >> 4 in bits 24-28
            constexpr uint32_t fmt = BITS ? 0u : 1u;
            constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(2 * kPRows >> 4) << 24);
            int s = 0, ph = 0, cnt = 0;
            for (int w = pair; w < tiles; w += npairs, cnt++) {
                const int acc = cnt & 1, use = cnt >> 1;
                if (ok && use > 0 && !pair_wait(&tempty[acc], (use - 1) & 1, p.err)) ok = false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int k = 0; k < p.kstages; k++) {
                    if (ok && !pair_wait(&full[s], ph & 1, p.err)) ok = false;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (ok) {
                        const uint32_t a0 = smem_u32(As + (size_t)s * S::kA), b0 = smem_u32(Bs + (size_t)s * S::kB);
#pragma unroll
                        for (int j = 0; j < S::kK / 16; j++)
                            pair_mma(tmem_d + (uint32_t)(acc * TN), pair_desc(a0 + (j >> 2) * (kPRows * 128) + (j & 3) * 32),
                                     pair_desc(b0 + (j >> 2) * (TN / 2 * 128) + (j & 3) * 32), idesc, (k > 0 || j > 0) ? 1u : 0u);
                        pair_commit(&empty[s]);
                        if (k == p.kstages - 1) pair_commit(&tfull[acc]);
                    }
                    if (++s == S::kStages) s = 0, ph++;
                }
            }
        }
        __syncwarp();
    } else {
        const int ew = warp - S::kWeightWarps, lanes = (warp & 3) * 32, half = ew >> 2;  // a warp reads tensor-memory lanes 32 (warp % 4) ..
        constexpr int kSpan = TN / (S::kEpiWarps / 4);
        const uint32_t tempty0 = leader_addr(tempty);
        int cnt = 0;
        for (int w = pair; w < tiles; w += npairs, cnt++) {
            const int m0 = w % p.mtiles * TN, n_warp = w / p.mtiles * (2 * kPRows) + rank * kPRows + lanes, acc = cnt & 1;
            if (ok && !pair_wait_warp(&tfull[acc], (cnt >> 1) & 1, p.err)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok) {
#pragma unroll 1
                for (int c = half * kSpan; c < (half + 1) * kSpan && m0 + c < p.M; c += 16) {
                    float v[16];
                    tmem_ld16(tmem_d + ((uint32_t)lanes << 16) + (uint32_t)(acc * TN + c), v);
                    epi_store16<T>(p.epi, p.N, p.M, n_warp + lane, n_warp, m0 + c, v);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_at(tempty0 + acc * 8);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_and_settle(ok);
    cluster_sync();  // neither CTA leaves while the other may still signal it or read its operands
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(kCols) : "memory");
    }
}

template <typename T, int TN, int BITS>
int launch(const Device *dev, PairGemm p, const CUtensorMap &ta, const void *x, int ldx, int K, cudaStream_t st) {
    using S = PairShape<TN, BITS>;
    auto kern = pair_gemm_kernel<T, TN, BITS>;
    static DeviceOnce once;  // per instantiation
    if (once.first(dev->ordinal)) IM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem));
    alignas(64) CUtensorMap tb;
    if (const int rc = tmap_2d(x, BITS == 0, p.M, K, ldx, TN / 2, &tb); rc != IM_OK) return rc;
    p.kstages = (K + S::kK - 1) / S::kK;
    p.mtiles = (p.M + TN - 1) / TN;
    p.ntiles = (p.N + 2 * kPRows - 1) / (2 * kPRows);
    const int pairs = std::min(p.mtiles * p.ntiles, dev->sm_count / 2);
    IM_CUDA_CHECK(launch_k(kern, dim3(2 * pairs), dim3(S::kThreads), (size_t)S::kSmem, st, p, ta, tb));
    return IM_OK;
}

// 256-token tiles unless 128-token tiles save more of the last wave than they lose in operand traffic (a 128-token tile
// moves 1.5 times the operand bytes per product: it has to save an eighth of the waves)
bool wide_tiles(const Device *dev, int N, int M) {
    const int pairs = dev->sm_count / 2, nt = (N + 2 * kPRows - 1) / (2 * kPRows);
    const long long w256 = (nt * ((M + 255ll) / 256) + pairs - 1) / pairs * 2, w128 = (nt * ((M + 127ll) / 128) + pairs - 1) / pairs;
    return 8 * w256 <= 9 * w128;
}

}  // namespace

bool pair_gemm_takes(const Device *dev, int rows, int M) {
    return M > 128 && (long long)((rows + 255) / 256) * ((M + 127) / 128) >= dev->sm_count / 4;
}

int pair_gemm_bf16(const Device *dev, const void *w, int ldw, int N, int K, const void *x, int ldx, int M, const DenseEpi &epi, cudaStream_t st) {
    PairGemm p{};
    p.N = N; p.M = M; p.err = dev->err_flag; p.epi = epi;
    alignas(64) CUtensorMap ta;
    if (const int rc = tmap_2d(w, true, N, K, ldw, kPRows, &ta); rc != IM_OK) return rc;
    return wide_tiles(dev, N, M) ? launch<__nv_bfloat16, 256, 0>(dev, p, ta, x, ldx, K, st) : launch<__nv_bfloat16, 128, 0>(dev, p, ta, x, ldx, K, st);
}

int pair_gemm_affine(const AffineWeight *w, const AffineWeight *up, const __half *x, __half *y, int M, cudaStream_t st) {
    PairGemm p{};
    p.N = up ? 2 * w->N : w->N; p.M = M; p.K = w->K; p.err = w->dev->err_flag; p.paired = up ? 1 : 0;
    p.codes[0] = w->codes; p.sz[0] = w->sz;
    if (up) p.codes[1] = up->codes, p.sz[1] = up->sz;
    p.epi.kind = kEpiProj;
    p.epi.pair0 = up ? 0 : 1 << 30;
    p.epi.pair_silu = 1;
    p.epi.y = p.epi.act = y;
    p.epi.ldy = p.epi.ldact = w->N;
    const CUtensorMap none{};
    const bool wide = wide_tiles(w->dev, p.N, M);
    if (w->bits == 8)
        return wide ? launch<__half, 256, 8>(w->dev, p, none, x, w->K, w->K, st) : launch<__half, 128, 8>(w->dev, p, none, x, w->K, w->K, st);
    return wide ? launch<__half, 256, 4>(w->dev, p, none, x, w->K, w->K, st) : launch<__half, 128, 4>(w->dev, p, none, x, w->K, w->K, st);
}

}  // namespace im
