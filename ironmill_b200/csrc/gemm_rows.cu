// Projections of up to 48 tokens (32 with 8-bit codes) with group-128 weights: decode batches of 16 and more, short prompts.
//   crates/ironmill-inference/src/metal/shaders/quantized/affine_matmul.metal:10-290 (superblock_matmul_int4 / _int8):
//   C[m, n] = sum_k f16(A[m, k] / awq[k]) * f16((q[n, k] - z) * s), f32 accumulation, fp16 result.
//
// Bound: the codes, read once (HBM); at 24 tokens the conversion of a code takes about as many issue slots as its bytes take time.
// On tcgen05 the converted weights have to pass through shared memory (store, proxy fence, barrier, one MMA thread), which left a stage of
// 128 x 128 codes at 1 us and SM whatever the token count: five times its bytes' time.  Here a lane converts the codes of
// its own mma.sync fragment in registers and multiplies them at once: no store, no fence, no hand-over.  Back to back with the packing of
// the tokens, 4-bit, 24 tokens, tcgen05 -> here: 14336 x 4096 32.4 -> 19.9 us, 4096 x 14336 30.2 -> 21.2, 4096 x 4096 12.3 -> 10.4.  What is left
// of a launch: 5 us of start and end, the rest at 50 % of the issue slots (460 instructions for two tiles, a third of them the conversion).  An
// instruction serves eight tokens, so the gain ends at about 48 (14336 x 4096: 31.0 against 33.2 us; 64 tokens 36 against 33.3) and,
// with 8-bit codes, 32 (28.2 against 29.3; 48 tokens 32.5 against 30.5): more tokens stay on tcgen05 (gemm_tc.cu).
//   * weights: the tiles of the matvec (16 rows x 128 columns, matvec_v2.cu); lane (g, t) owns columns 32 t .. 32 t + 31 of rows g
//     and g + 8, so that 16 contiguous bytes are its fragments of eight k-steps.  A warp multiplies two row blocks (they share
//     the token fragments); it brings its tiles itself, cp.async into a ring of its own, several units ahead, the
//     first ones before the predecessor kernel has finished;
//   * tokens: packed for these fragments by the kernel that writes them (token_chunk below): the lane's four fragment registers
//     of a token and eight columns are 16 contiguous bytes.  One thread brings the slabs of a few groups by cp.async.bulk;
//   * a CTA works on 128 rows (four row-block pairs) with its warps on different groups of K.  Few row tiles: each belongs to a cluster
//     of up to eight CTAs on slices of K, which add their sums through distributed shared memory.  Many: a CTA takes an equal
//     share of the flattened [row tile][group] list, and row tiles cut by a CTA boundary are completed by whichever of their
//     CTAs arrives last (a counter, nobody waits), adding the parts in CTA order.
// The joint form multiplies gate rows and up rows as the pair of row blocks and leaves f16(silu(f16 gate) f16(up)), if asked
// divided by the next projection's activation scales and packed for it.
#include <algorithm>

#include "common.cuh"
#include "gemm_rows.cuh"
#include "v2_device.cuh"

namespace im {

namespace {

constexpr int kRRows = 128;     // weight rows of a CTA's tile: four pairs of row blocks
constexpr int kRPad = 132;      // floats of a token's row of sums in shared memory: conflict-free for fragment stores
constexpr int kRBStages = 3;    // token slabs: in use, on their way, and one that its slowest reader may still hold

// More than 24 tokens: half the warps, so that their sums fit a thread's registers (16 with 8-bit codes, whose rings are twice as large).
template <int NT, int BITS>
constexpr int rows_warps() { return NT <= (BITS == 4 ? 3 : 2) ? 16 : 8; }
template <int NT, int BITS>
constexpr int rows_klanes() { return rows_warps<NT, BITS>() / 4; }
template <int NT, int BITS>
constexpr int rows_depth() { return rows_warps<NT, BITS>() == 16 ? (BITS == 4 ? 3 : 2) : BITS == 4 ? 4 : 3; }  // units (two tiles) in flight per warp
template <int BITS>
constexpr int rows_unit_bytes() { return 2 * TileGeom<BITS>::kTileBytes; }

struct RowsParams {
    const uint8_t *tiles[2];  // joint: gate, up; else both the matrix
    const __half *xs;         // packed tokens
    __half *y;
    const __half *div;        // joint: activation scales of the next projection, or none
    float *partial;           // [grid][2][tokens][128]
    int *counters;            // [row tiles], zero between launches
    int *err;
    int N, G, M, nblk, total;
    int slices;               // CTAs of a cluster that share a row tile (1: equal shares of the whole list)
    int joint, packed, wide;  // packed: the result as the next projection reads it; wide: 16-byte stores of the result
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 u2h(uint32_t u) { return *reinterpret_cast<__half2 *>(&u); }

__device__ __forceinline__ void add4(float4 &a, const float4 b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// Scales and zero points of a lane's rows g and g + 8 as the conversion uses them.  Where z is a whole or half number of at most 512,
// q - z is exact in fp16 from either nibble position, (1024 + q) - (1024 + z) or (1024 + 16 q) / 16 - (64 + z), and the product
// with s is rounded once: f16((q - z) s).
struct RowScale {
    __half2 c, d, s;
};
__device__ __forceinline__ bool row_scales(uint32_t sz0, uint32_t sz1, RowScale (&r)[2]) {
    const __half2 z = u2h(__byte_perm(sz0, sz1, 0x7632)), k = __float2half2_rn(1024.0f);
    const __half2 c = __hadd2(z, k), d = __hsub2(__float2half2_rn(-64.0f), z);
    r[0] = RowScale{__low2half2(c), __low2half2(d), u2h(__byte_perm(sz0, sz0, 0x1010))};
    r[1] = RowScale{__high2half2(c), __high2half2(d), u2h(__byte_perm(sz1, sz1, 0x1010))};
    return __hbeq2(__hsub2(c, k), z) && __hble2(__habs2(z), __float2half2_rn(512.0f));
}
// Eight columns c .. c + 7 of a row as four registers: (c, c + 4), (c + 1, c + 5), (c + 2, c + 6), (c + 3, c + 7).
// 8-bit codes: w holds the even columns' bytes, w2 the odd ones'.  e: 0x64006400 in a register that the compiler cannot see through; with two constants
// the and-or below becomes two instructions (the logic pipe runs at half rate and sets the pace here).
template <int BITS>
__device__ __forceinline__ void rows_dequant(uint32_t w, uint32_t w2, const RowScale &r, uint32_t e, uint32_t (&o)[4]) {
    if (BITS == 4) {
        constexpr uint32_t M = 0x000F000Fu, MH = 0x00F000F0u;
        auto place = [&](uint32_t v, uint32_t m) {  // (v & m) | e
            uint32_t d;
            asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(v), "r"(m), "r"(e));
            return u2h(d);
        };
        const __half2 sixteenth = __float2half2_rn(0.0625f);
        const uint32_t u = w >> 8;
        o[0] = h2u(__hmul2(__hsub2(place(w, M), r.c), r.s));
        o[1] = h2u(__hmul2(__hfma2(place(w, MH), sixteenth, r.d), r.s));
        o[2] = h2u(__hmul2(__hsub2(place(u, M), r.c), r.s));
        o[3] = h2u(__hmul2(__hfma2(place(u, MH), sixteenth, r.d), r.s));
    } else {
        o[0] = h2u(__hmul2(__hsub2(u2h(__byte_perm(w, 0x64u, 0x4240)), r.c), r.s));
        o[1] = h2u(__hmul2(__hsub2(u2h(__byte_perm(w2, 0x64u, 0x4240)), r.c), r.s));
        o[2] = h2u(__hmul2(__hsub2(u2h(__byte_perm(w, 0x64u, 0x4341)), r.c), r.s));
        o[3] = h2u(__hmul2(__hsub2(u2h(__byte_perm(w2, 0x64u, 0x4341)), r.c), r.s));
    }
}
template <int BITS>
__device__ __forceinline__ void rows_dequant_any(uint32_t w, uint32_t w2, uint32_t sz, uint32_t (&o)[4]) {  // any zero point: f32, one rounding
    const float2 f = __half22float2(u2h(sz));
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t v = BITS == 4 ? w >> (4 * i) : (i & 1 ? w2 : w) >> (8 * (i >> 1)), m = BITS == 4 ? 15u : 255u;
        o[i] = h2u(__floats2half2_rn(((float)(v & m) - f.y) * f.x, ((float)((v >> 16) & m) - f.y) * f.x));
    }
}

// The list of units: CTA share [u0, u1) of the flattened [row tile][group] list, cut into runs within a row tile.
struct Runs {
    int u, u1, G, tile, g0, g1;
    __device__ Runs(int u0, int u1_, int G_) : u(u0), u1(u1_), G(G_), tile(0), g0(0), g1(0) {}
    __device__ bool next() {
        if (u >= u1) return false;
        tile = u / G;
        g0 = u - tile * G;
        g1 = min(G, g0 + (u1 - u));
        u += g1 - g0;
        return true;
    }
};

template <int NT, int BITS>
__global__ void __launch_bounds__(rows_warps<NT, BITS>() * 32, 1) gemm_rows_kernel(const RowsParams p) {
    constexpr int NW = rows_warps<NT, BITS>(), KQ = rows_klanes<NT, BITS>(), D = rows_depth<NT, BITS>(), MP = NT * 8;
    constexpr int kTile = TileGeom<BITS>::kTileBytes, kCodes = TileGeom<BITS>::kCodeBytes, kUnit = rows_unit_bytes<BITS>();
    constexpr int CV = BITS == 4 ? 2 : 4;         // 16-byte vectors of codes per lane and tile
    constexpr int kCopies = KQ / 2;               // sums of warps on different groups, halved once in registers
    extern __shared__ __align__(128) unsigned char rows_smem[];
    unsigned char *ring = rows_smem;                                              // [warp][D][unit]
    unsigned char *bs = ring + NW * D * kUnit;                                    // [stage][KQ groups][tokens * 256 bytes], read up to seven tokens past the end
    float *red = reinterpret_cast<float *>(bs + kRBStages * KQ * MP * 256 + 512);  // [copies][MP][kRPad]
    uint64_t *full = reinterpret_cast<uint64_t *>(red + kCopies * MP * kRPad), *empty = full + kRBStages;
    int *flag = reinterpret_cast<int *>(empty + kRBStages);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.G, M = p.M, slab = M * 256, stage_bytes = KQ * MP * 256;
    int u0 = (int)((long long)p.total * blockIdx.x / gridDim.x), u1 = (int)((long long)p.total * (blockIdx.x + 1) / gridDim.x), rank = 0;
    if (p.slices > 1) {  // a row tile per cluster, a slice of K per CTA
        const int tile = blockIdx.x / p.slices;
        rank = blockIdx.x % p.slices;
        u0 = tile * G + G * rank / p.slices;
        u1 = tile * G + G * (rank + 1) / p.slices;
    }

    pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < kRBStages; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], NW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    // warp = (pair of row blocks rp, lane kq of the groups)
    const int rp = warp & 3, kq = warp >> 2, g8 = lane >> 2, t = lane & 3;
    unsigned char *mine = ring + warp * D * kUnit;
    const uint32_t mine_u = smem_u32(mine) + lane * 16;
    Runs ahead(u0, u1, G);  // the unit to request next: groups left of its run, its two tiles
    int left = 0;
    const uint8_t *src[2] = {nullptr, nullptr};
    bool more = true;
    auto request_next = [&](int slot) {
        while (more && left <= 0) {
            more = ahead.next();
            left = ahead.g1 - ahead.g0 - kq;
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const int rb = min(p.joint ? ahead.tile * 4 + rp : ahead.tile * 8 + 2 * rp + b, p.nblk - 1);
                src[b] = p.tiles[b] + ((size_t)rb * G + ahead.g0 + kq) * kTile + lane * 16;
            }
        }
        if (more) {
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const uint32_t dst = mine_u + slot * kUnit + b * kTile;
#pragma unroll
                for (int v = 0; v < CV; v++) cp_async16(dst + v * 512, src[b] + v * 512);
                if (lane < 4) cp_async16(dst + kCodes, src[b] + kCodes);
                src[b] += KQ * kTile;
            }
            left -= KQ;
        }
        cp_commit();  // an empty group too: the count of groups is the count of units
    };
#pragma unroll
    for (int d = 0; d < D; d++) request_next(d);  // weights are constants: requested before the predecessor has finished
    pdl_wait();

    // Warp 0 asks for the token slabs, one stage ahead of its own: the slot's last tenant is then two stages old, and the wait for it short.
    Runs br(u0, u1, G);
    bool bmore = warp == 0 && br.next(), dead = false;
    int bg = br.g0, bit = 0;
    auto bring = [&]() {
        if (!bmore) return;
        const int sl = bit % kRBStages, n = min(KQ, br.g1 - bg);
        if (!dead && bit >= kRBStages && !mbar_wait_warp(&empty[sl], (bit / kRBStages - 1) & 1, p.err)) dead = true;
        if (dead) {
            bmore = false;
            return;
        }
        if (lane == 0) {
            mbar_expect_tx(&full[sl], (uint32_t)(n * slab));
            bulk_g2s(bs + sl * stage_bytes, reinterpret_cast<const unsigned char *>(p.xs) + (size_t)bg * slab, (uint32_t)(n * slab), &full[sl]);
        }
        __syncwarp();
        bit++;
        bg += KQ;
        if (bg >= br.g1) {
            bmore = br.next();
            bg = br.g0;
        }
    };
    bring();

    uint32_t e;
    asm volatile("mov.b32 %0, 0x64006400;" : "=r"(e));
    float acc[2][NT][4];
    int s = 0, par = 0, slot = 0, nrun = 0;
    for (Runs r(u0, u1, G); r.next(); nrun++) {
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[b][n][i] = 0.0f;
        for (int g0 = r.g0; g0 < r.g1; g0 += KQ) {
            bring();
            if (!dead && !mbar_wait_warp(&full[s], par, p.err)) dead = true;
            if (g0 + kq < r.g1) {
                cp_wait<D - 1>();
                __syncwarp();
                const unsigned char *tp = mine + slot * kUnit, *bp = bs + s * stage_bytes + kq * slab + g8 * 64 + t * 16;
                uint32_t sz[2][2];
                RowScale rs[2][2];
                bool fast = true;
#pragma unroll
                for (int b = 0; b < 2; b++) {
#pragma unroll
                    for (int h = 0; h < 2; h++) sz[b][h] = *reinterpret_cast<const uint32_t *>(tp + b * kTile + kCodes + g8 * 4 + 32 * h);
                    fast = row_scales(sz[b][0], sz[b][1], rs[b]) && fast;
                }
                // eight columns: two k-steps of both row blocks
                auto multiply = [&](int i, const uint32_t (&a)[2][2][4]) {
#pragma unroll
                    for (int n = 0; n < NT; n++) {
                        const uint4 x = *reinterpret_cast<const uint4 *>(bp + i * (M * 64) + n * 512);
#pragma unroll
                        for (int b = 0; b < 2; b++) mma_f16(acc[b][n], a[b][0][0], a[b][1][0], a[b][0][1], a[b][1][1], x.x, x.y);
#pragma unroll
                        for (int b = 0; b < 2; b++) mma_f16(acc[b][n], a[b][0][2], a[b][1][2], a[b][0][3], a[b][1][3], x.z, x.w);
                    }
                };
                uint32_t a[2][2][4];
                if (__builtin_expect(__all_sync(0xffffffffu, fast), 1)) {
                    uint4 w[2][CV];
#pragma unroll
                    for (int b = 0; b < 2; b++)
#pragma unroll
                        for (int v = 0; v < CV; v++) w[b][v] = *reinterpret_cast<const uint4 *>(tp + b * kTile + v * 512 + lane * 16);
                    __syncwarp();
                    request_next(slot);  // every lane has its codes in registers
                    if (!dead)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
#pragma unroll
                            for (int b = 0; b < 2; b++)
#pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    const uint4 q = BITS == 4 ? w[b][h] : w[b][(2 * h + (i >> 1)) % CV];
                                    if (BITS == 4) rows_dequant<BITS>(i == 0 ? q.x : i == 1 ? q.y : i == 2 ? q.z : q.w, 0u, rs[b][h], e, a[b][h]);
                                    else rows_dequant<BITS>(i & 1 ? q.z : q.x, i & 1 ? q.w : q.y, rs[b][h], e, a[b][h]);
                                }
                            multiply(i, a);
                        }
                } else {
#pragma unroll 1
                    for (int i = 0; i < 4; i++) {
#pragma unroll
                        for (int b = 0; b < 2; b++)
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const uint32_t *w = reinterpret_cast<const uint32_t *>(tp + b * kTile + (BITS == 4 ? h : 2 * h + (i >> 1)) * 512 + lane * 16);
                                if (BITS == 4) rows_dequant_any<BITS>(w[i], 0u, sz[b][h], a[b][h]);
                                else rows_dequant_any<BITS>(w[2 * (i & 1)], w[2 * (i & 1) + 1], sz[b][h], a[b][h]);
                            }
                        if (!dead) multiply(i, a);
                    }
                    __syncwarp();
                    request_next(slot);
                }
                if (++slot == D) slot = 0;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (++s == kRBStages) s = 0, par ^= 1;
        }
        // ---- the run's sums: warps on different groups together, through shared memory as [token][row]
        auto sync = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory"); };
        auto each = [&](auto f) {
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        f(acc[b][n][i], red + ((kq % kCopies) * MP + n * 8 + 2 * t + (i & 1)) * kRPad + (p.joint ? b * 64 + rp * 16 : rp * 32 + b * 16) + g8 + 8 * (i >> 1));
        };
        if (kq >= kCopies) each([](float v, float *q) { *q = v; });
        sync();
        if (kq < kCopies) each([](float v, float *q) { *q += v; });
        // What is added up for the result: this CTA's sums, those of the cluster's CTAs, or the parts that its CTAs left in memory.
        int c_first = 0, c_last = 0;
        bool finish = true;
        if (p.slices > 1) {
            cluster_sync();
        } else {
            sync();
            c_first = (int)((((long long)r.tile * G + 1) * gridDim.x + p.total - 1) / p.total) - 1;
            c_last = (int)(((long long)(r.tile + 1) * G * gridDim.x + p.total - 1) / p.total) - 1;
        }
        const bool parts = c_first != c_last;
        if (parts) {
            float4 *out = reinterpret_cast<float4 *>(p.partial + ((size_t)blockIdx.x * 2 + (nrun ? 1 : 0)) * (MP * kRRows));
            for (int i = tid; i < M * (kRRows / 4); i += NW * 32) {
                const float *q = red + (i / (kRRows / 4)) * kRPad + (i % (kRRows / 4)) * 4;
                float4 v = *reinterpret_cast<const float4 *>(q);
                if (kCopies > 1) add4(v, *reinterpret_cast<const float4 *>(q + MP * kRPad));
                __stcg(out + i, v);
            }
            sync();
            if (tid == 0) {
                int before;
                asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(before) : "l"(p.counters + r.tile) : "memory");
                *flag = before == c_last - c_first;
                if (before == c_last - c_first) p.counters[r.tile] = 0;  // ready for the next launch
            }
            sync();
            finish = *flag != 0;
        }
        if (finish && !dead) {
            // a task: eight neighbouring rows of a token; the CTAs of a cluster share them
            const int chunks = p.joint ? 8 : 16, share = (M * chunks + p.slices - 1) / p.slices, end = min((rank + 1) * share, M * chunks);
            for (int i = rank * share + tid; i < end; i += NW * 32) {
                const int m = i / chunks, c = i - m * chunks;
                float v[2][8];
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    if (b && !p.joint) break;
                    const int row = b * 64 + c * 8;
                    float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
                    if (parts) {
                        constexpr int kAtOnce = 4;  // parts on their way together
                        for (int c0 = c_first; c0 <= c_last; c0 += kAtOnce) {
                            float4 x[kAtOnce], z[kAtOnce];
#pragma unroll
                            for (int k = 0; k < kAtOnce; k++) {
                                const int cc = min(c0 + k, c_last), first_tile = (int)((long long)p.total * cc / gridDim.x) / G;
                                const float4 *q =
                                    reinterpret_cast<const float4 *>(p.partial + ((size_t)cc * 2 + (first_tile == r.tile ? 0 : 1)) * (MP * kRRows) + m * kRRows + row);
                                x[k] = __ldcg(q);
                                z[k] = __ldcg(q + 1);
                            }
#pragma unroll
                            for (int k = 0; k < kAtOnce; k++)
                                if (c0 + k <= c_last) {
                                    add4(lo, x[k]);
                                    add4(hi, z[k]);
                                }
                        }
                    } else {
                        const uint32_t q = smem_u32(red + m * kRPad + row);
                        for (int k = 0; k < p.slices; k++) {
                            const uint32_t qk = p.slices > 1 ? cluster_addr(q, k) : q;
#pragma unroll
                            for (int j = 0; j < kCopies; j++) {
                                add4(lo, ld_cluster(qk + j * MP * kRPad * 4));
                                add4(hi, ld_cluster(qk + j * MP * kRPad * 4 + 16));
                            }
                        }
                    }
                    v[b][0] = lo.x; v[b][1] = lo.y; v[b][2] = lo.z; v[b][3] = lo.w;
                    v[b][4] = hi.x; v[b][5] = hi.y; v[b][6] = hi.z; v[b][7] = hi.w;
                }
                const int n = r.tile * (p.joint ? 64 : 128) + c * 8;
                __half h[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    h[j] = __float2half_rn(v[0][j]);
                    if (p.joint) {
                        const float gv = __half2float(h[j]), uv = __half2float(__float2half_rn(v[1][j]));
                        h[j] = __float2half_rn((gv / (1.0f + expf(-gv))) * uv);
                        if (p.div && n + j < p.N) h[j] = __float2half_rn(__half2float(h[j]) / __half2float(p.div[n + j]));
                    }
                }
                if (p.packed) {
                    if (n < p.N) *reinterpret_cast<uint4 *>(p.y + token_chunk(n >> 3, m, M) * 8) = pack_chunk(h);
                } else if (p.wide) {
                    if (n < p.N) *reinterpret_cast<uint4 *>(p.y + (size_t)m * p.N + n) = *reinterpret_cast<const uint4 *>(h);
                } else {
                    for (int j = 0; j < 8; j++)
                        if (n + j < p.N) p.y[(size_t)m * p.N + n + j] = h[j];
                }
            }
        }
        if (p.slices > 1) cluster_sync();  // the sums have been read, by this CTA before the next run writes its own and by the others before it leaves
        else sync();
    }
    cp_wait<0>();
    // token copies that nobody waited for (a wait ran out) must land before the block leaves
    if (warp == 0 && dead)
        for (int i = max(0, bit - kRBStages); i < bit; i++) mbar_wait_warp(&full[i % kRBStages], (i / kRBStages) & 1, p.err);
}

// Packed tokens f16(x / awq) (or x): one thread per eight columns of a token.
__global__ void __launch_bounds__(256) token_pack_kernel(const __half *__restrict__ x, const __half *__restrict__ awq, __half *__restrict__ out, int M, int K8) {
    pdl_trigger();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M * K8) return;
    const int m = i / K8, c = i - m * K8;
    __half h[8];
    if (reinterpret_cast<uintptr_t>(x) % 16 == 0) {
        *reinterpret_cast<uint4 *>(h) = reinterpret_cast<const uint4 *>(x)[i];
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) h[j] = x[(size_t)i * 8 + j];
    }
    if (awq) {
        __half a[8];
        *reinterpret_cast<uint4 *>(a) = reinterpret_cast<const uint4 *>(awq)[c];
#pragma unroll
        for (int j = 0; j < 8; j++) h[j] = __float2half_rn(__half2float(h[j]) / __half2float(a[j]));
    }
    reinterpret_cast<uint4 *>(out)[token_chunk(c, m, M)] = pack_chunk(h);
}

constexpr int kRMaxCluster = 8;

// launch_k with a cluster size
int rows_start(void (*kern)(RowsParams), int grid, int cluster, int threads, size_t smem, cudaStream_t st, const RowsParams &p) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    IM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, p));
    return IM_OK;
}

// Clusters of a size that the GPU holds at once, one CTA on an SM (asked for once per device: a cluster lies within a GPC, whose SMs need not divide evenly)
int rows_clusters(void (*kern)(RowsParams), int size, int threads, size_t smem, const Device *dev) {
    static std::atomic<int> held[64][kRMaxCluster + 1];
    const int at = dev->ordinal >= 0 && dev->ordinal < 64 ? dev->ordinal : -1;
    if (at >= 0 && held[at][size].load() > 0) return held[at][size].load() - 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    if (at >= 0) held[at][size].store(n + 1);
    return n;
}

template <int NT, int BITS>
int rows_launch(RowsParams p, const Device *dev, cudaStream_t st) {
    constexpr int NW = rows_warps<NT, BITS>(), KQ = rows_klanes<NT, BITS>(), MP = NT * 8;
    constexpr size_t smem = (size_t)NW * rows_depth<NT, BITS>() * rows_unit_bytes<BITS>() + (size_t)kRBStages * KQ * MP * 256 + 512 +
                            (size_t)(KQ / 2) * MP * kRPad * 4 + 2 * kRBStages * 8 + 16;
    static_assert(smem <= 227 * 1024, "the rings of this form do not fit");
    if (smem > dev->smem_optin) return IM_ERR_BOUNDS;
    auto kern = gemm_rows_kernel<NT, BITS>;
    static DeviceOnce once;  // per instantiation
    if (once.first(dev->ordinal)) IM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // Few row tiles: a cluster of CTAs per tile, as many as the GPU holds (at least one stage of groups each).  Otherwise equal shares of the
    // list (two partial tiles of each CTA fit the scratch).  The two ends of a share cost about three stages, so slices that leave SMs idle win
    // as long as they are not that much longer.
    const int tiles = p.total / p.G;
    p.slices = std::min(std::min(dev->sm_count / tiles, kRMaxCluster), std::max(1, p.G / KQ));
    while (p.slices > 1 && rows_clusters(kern, p.slices, NW * 32, smem, dev) < tiles) p.slices--;
    const int grid = (int)std::min<size_t>(std::min(dev->sm_count, std::max(1, p.total / KQ)), kGemmPartialBytes / ((size_t)2 * MP * kRRows * sizeof(float)));
    const int stages_sliced = p.slices > 0 ? ((p.G + p.slices - 1) / p.slices + KQ - 1) / KQ : 0, stages_shared = ((p.total + grid - 1) / grid + KQ - 1) / KQ;
    if (p.slices < 1 || stages_sliced > stages_shared + 3) p.slices = 1;
    else if (p.slices == 1) return rows_start(kern, tiles, 1, NW * 32, smem, st, p);  // a tile per CTA
    return rows_start(kern, p.slices > 1 ? tiles * p.slices : grid, p.slices, NW * 32, smem, st, p);
}

template <int BITS>
int rows_run(const RowsParams &p, const Device *dev, cudaStream_t st) {
    const int nt = (p.M + 7) / 8;
    if (nt <= 1) return rows_launch<1, BITS>(p, dev, st);
    if (nt == 2) return rows_launch<2, BITS>(p, dev, st);
    if (nt == 3) return rows_launch<3, BITS>(p, dev, st);
    if (nt == 4) return rows_launch<4, BITS>(p, dev, st);
    return rows_launch<6, 4>(p, dev, st);
}

}  // namespace

// At least eight groups of K: with fewer there is nothing to stream, and the tcgen05 kernels, which do not split so short a sum, give a token the same bits
// whatever portion of a prompt it comes in.
bool gemm_rows_takes(const AffineWeight *w, int M) {
    return M >= 1 && w->G >= 8 && M <= (w->bits == 4 ? kRowsMaxTokens : kRowsMaxTokens8) && w->tiles && w->group_size == 128 && w->K % 128 == 0 && (w->bits == 4 || w->bits == 8) && w->nblk <= kSkMaxBlocks &&
           (long long)w->nblk * w->G < (1 << 30) && w->dev->gemm_partial && w->dev->sk_counters;
}

int token_pack(const __half *x, const __half *awq, __half *out, int M, int K, cudaStream_t st) {
    const int n = M * (K / 8);
    IM_CUDA_CHECK(launch_k(token_pack_kernel, dim3((n + 255) / 256), dim3(256), 0, st, x, awq, out, M, K / 8));
    return IM_OK;
}

int gemm_rows(const AffineWeight *w, const AffineWeight *up, const __half *packed, __half *y, int M, const __half *div, bool pack_out, cudaStream_t st) {
    RowsParams p{};
    p.tiles[0] = w->tiles;
    p.tiles[1] = up ? up->tiles : w->tiles;
    p.xs = packed; p.y = y; p.div = div; p.partial = w->dev->gemm_partial; p.counters = w->dev->sk_counters; p.err = w->dev->err_flag;
    p.N = w->N; p.G = w->G; p.M = M; p.nblk = w->nblk; p.joint = up ? 1 : 0; p.packed = pack_out ? 1 : 0;
    p.wide = w->N % 8 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
    p.total = (up ? (w->nblk + 3) / 4 : (w->nblk + 7) / 8) * w->G;
    return w->bits == 8 ? rows_run<8>(p, w->dev, st) : rows_run<4>(p, w->dev, st);
}

}  // namespace im
