// Projections of up to 48 tokens (32 with 8-bit codes) with group-128 weights: decode batches of 16 and more, short prompts.
//   crates/ironmill-inference/src/metal/shaders/quantized/affine_matmul.metal:10-290 (superblock_matmul_int4 / _int8):
//   C[m, n] = sum_k f16(A[m, k] / awq[k]) * f16((q[n, k] - z) * s), f32 accumulation, fp16 result.
//
// Bound: the codes, read once (HBM); at 24 tokens the conversion of a code takes about as many issue slots as its bytes take time.
// On tcgen05 the converted weights have to pass through shared memory (store, proxy fence, barrier, one MMA thread), which left a stage of
// 128 x 128 codes at 1 us and SM whatever the token count: five times its bytes' time.  Here a lane converts the codes of
// its own mma.sync fragment in registers and multiplies them at once: no store, no fence, no hand-over.  Back to back with the packing of
// the tokens, 4-bit, 24 tokens, tcgen05 -> here: 14336 x 4096 32.4 -> 20.1 us, 4096 x 14336 30.2 -> 20.8, 4096 x 4096 12.3 -> 9.9.  What is left
// of a launch: 4 us of start and end, the rest at 50 % of the issue slots (460 instructions for two tiles, a third of them the conversion).  An
// instruction serves eight tokens, so the gain ends at about 48 (14336 x 4096: 30.4 against 33.2 us; 64 tokens 36 against 33.3) and,
// with 8-bit codes, 32 (28.2 against 29.3; 48 tokens 32.5 against 30.5): more tokens stay on tcgen05 (gemm_tc.cu).
//   * weights: the tiles of the matvec (16 rows x 128 columns, matvec_v2.cu); lane (g, t) owns columns 32 t .. 32 t + 31 of rows g
//     and g + 8, so that 16 contiguous bytes are its fragments of eight k-steps.  A warp multiplies two row blocks (they share
//     the token fragments); it brings its tiles itself, cp.async into a ring of its own, several units ahead, the
//     first ones before the predecessor kernel has finished;
//   * tokens: packed for these fragments by the kernel that writes them (token_chunk below): the lane's four fragment registers
//     of a token and eight columns are 16 contiguous bytes.  One thread brings the slabs of a few groups by cp.async.bulk;
//   * a CTA works on 128 rows (four row-block pairs) with its warps on different groups of K.  Few row tiles: each belongs to a cluster
//     of up to eight CTAs on slices of K, which add their sums through distributed shared memory.  Many: a CTA each or,
//     where the last wave would leave too many SMs idle, an equal share of the flattened [row tile][group] list; row tiles cut by a CTA boundary are
//     completed by whichever of their CTAs arrives last (a counter, nobody waits), adding the parts in CTA order.
// The joint form multiplies gate rows and up rows as the pair of row blocks and leaves f16(silu(f16 gate) f16(up)), if asked
// divided by the next projection's activation scales and packed for it.
//
// Batches of up to 15 rows keep the matvec's arithmetic (matvec_v2.cu: activations as 24-bit integers per group of 128, three byte planes, exact integer
// sums, u8 x s8 products): the same kernel with INT = true, two rows to an instruction.  The matvec stages the planes again in every CTA, which
// for four rows of 4096 values took 20 of a launch's 30 us, and passes over the weights once per four rows.  Here the kernel in front writes the planes
// (rows_planes_kernel, norm_planes_kernel), one pass serves the batch, and gate, up and their activation or Q, K and V are one launch: a step of four
// sequences through four 8B layers 690 -> 495 us, projections 24 -> 14 us a launch on average.
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
template <int NT, int BITS, bool INT>
constexpr int rows_warps() { return INT || NT <= (BITS == 4 ? 3 : 2) ? 16 : 8; }
template <int NT, int BITS, bool INT>
constexpr int rows_klanes() { return rows_warps<NT, BITS, INT>() / 4; }
template <int NT, int BITS, bool INT>
constexpr int rows_depth() { return rows_warps<NT, BITS, INT>() == 16 ? (BITS == 4 ? 3 : 2) : BITS == 4 ? 4 : 3; }  // units (two tiles) in flight per warp
template <int NT, bool INT>
constexpr int rows_tokens() { return INT ? NT * 2 : NT * 8; }  // tokens that NT instructions of eight columns take: four columns a row of integers
template <int NT, bool INT>
constexpr int rows_slab_max() { return INT ? planes_slab(NT * 2) : NT * 8 * 256; }
template <int BITS>
constexpr int rows_unit_bytes() { return 2 * TileGeom<BITS>::kTileBytes; }
template <int NT, int BITS, bool INT>
constexpr size_t rows_smem_bytes() {  // rings of tiles, token slabs, sums, barriers and the flag
    return (size_t)rows_warps<NT, BITS, INT>() * rows_depth<NT, BITS, INT>() * rows_unit_bytes<BITS>() + (size_t)kRBStages * rows_klanes<NT, BITS, INT>() * rows_slab_max<NT, INT>() + 512 +
           (size_t)(rows_klanes<NT, BITS, INT>() / 2) * rows_tokens<NT, INT>() * kRPad * 4 + 2 * kRBStages * 8 + 16;
}

struct RowsParams {
    const uint8_t *tiles[2];  // joint: gate, up; else both the matrix
    const uint8_t *xs[2];     // packed tokens or planes, [group][slab]; the second set for rows from split_row on
    int slab, split_row;
    __half *y;
    const __half *div;        // joint: activation scales of the next projection, or none
    float *partial;           // [grid][2][tokens][128], or none: every tile has its CTAs to itself
    int *counters;            // [row tiles], zero between launches
    int *err;
    int N, G, M, nblk, total;
    int slices;               // CTAs of a cluster that share a row tile (1: equal shares of the whole list)
    int joint, packed, wide;  // joint: 1 rounds gate and up before the activation, 2 does not; packed: the result as the next projection reads it; wide: 8-byte stores of the result
};

// Weights are read once a pass and leave L2 first: kept like other lines they push out what the kernels between the projections read again for every layer
// (encoder and rotation tables, activations).  Four 8B layers: a prompt of 40 tokens 841 -> 748 us, a step of 24 rows 516 -> 479, of four 400 -> 385.
__device__ __forceinline__ uint64_t leave_first() {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    return policy;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
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

template <int NT, int BITS, bool INT>
__global__ void __launch_bounds__(rows_warps<NT, BITS, INT>() * 32, 1) gemm_rows_kernel(const RowsParams p) {
    constexpr int NW = rows_warps<NT, BITS, INT>(), KQ = rows_klanes<NT, BITS, INT>(), D = rows_depth<NT, BITS, INT>(), MP = rows_tokens<NT, INT>();
    constexpr int kTile = TileGeom<BITS>::kTileBytes, kCodes = TileGeom<BITS>::kCodeBytes, kUnit = rows_unit_bytes<BITS>();
    constexpr int kStage = KQ * rows_slab_max<NT, INT>();
    constexpr int CV = BITS == 4 ? 2 : 4;         // 16-byte vectors of codes per lane and tile
    constexpr int kCopies = KQ / 2;               // sums of warps on different groups, halved once in registers
    extern __shared__ __align__(128) unsigned char rows_smem[];
    unsigned char *ring = rows_smem;                                              // [warp][D][unit]
    unsigned char *bs = ring + NW * D * kUnit;                                    // [stage][KQ groups][slab], read up to seven tokens past the end
    float *red = reinterpret_cast<float *>(bs + kRBStages * kStage + 512);  // [copies][MP][kRPad]
    uint64_t *full = reinterpret_cast<uint64_t *>(red + kCopies * MP * kRPad), *empty = full + kRBStages;
    int *flag = reinterpret_cast<int *>(empty + kRBStages);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.G, M = p.M, slab = p.slab;
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
    const uint64_t policy = leave_first();
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
                for (int v = 0; v < CV; v++) cp_async16(dst + v * 512, src[b] + v * 512, policy);
                if (lane < 4) cp_async16(dst + kCodes, src[b] + kCodes, policy);
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
            bulk_g2s(bs + sl * kStage, (br.tile * kRRows >= p.split_row ? p.xs[1] : p.xs[0]) + (size_t)bg * slab, (uint32_t)(n * slab), &full[sl]);
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
    constexpr int A = INT ? 2 : 4;
    float acc[2][NT][A];
    int s = 0, par = 0, slot = 0, nrun = 0;
    for (Runs r(u0, u1, G); r.next(); nrun++) {
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < A; i++) acc[b][n][i] = 0.0f;
        for (int g0 = r.g0; g0 < r.g1; g0 += KQ) {
            bring();
            if (!dead && !mbar_wait_warp(&full[s], par, p.err)) dead = true;
            if (g0 + kq < r.g1) {
                cp_wait<D - 1>();
                __syncwarp();
                const unsigned char *tp = mine + slot * kUnit, *bp = bs + s * kStage + kq * slab;
                if constexpr (INT) {
                    uint4 w[2][CV];
                    float2 sz[2][2];
#pragma unroll
                    for (int b = 0; b < 2; b++) {
#pragma unroll
                        for (int v = 0; v < CV; v++) w[b][v] = *reinterpret_cast<const uint4 *>(tp + b * kTile + v * 512 + lane * 16);
#pragma unroll
                        for (int h = 0; h < 2; h++) sz[b][h] = __half22float2(*reinterpret_cast<const __half2 *>(tp + b * kTile + kCodes + g8 * 4 + 32 * h));
                    }
                    __syncwarp();
                    request_next(slot);
                    if (!dead)
#pragma unroll
                        for (int n = 0; n < NT; n++) {
                            // this lane's column: byte plane g % 4 of batch row 2 n + g / 4 (plane 3: zeros), its 32 columns as two vectors
                            uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
                            if ((g8 & 3) < 3) {
                                const unsigned char *xp = bp + (2 * n + (g8 >> 2)) * 192 + (g8 & 3) * 64 + t * 16;
                                x0 = *reinterpret_cast<const uint4 *>(xp);
                                x1 = *reinterpret_cast<const uint4 *>(xp + M * 192);
                            }
                            // constants of (group, row 2 n + t / 2): even lanes hold the high and middle planes' sums, odd ones the low plane's
                            const float2 m = *reinterpret_cast<const float2 *>(bp + M * 384 + (2 * n + (t >> 1)) * 8);
                            const float mx = t & 1 ? m.x * 0x1p-16f : m.x, my = t & 1 ? 0.0f : m.y;
#pragma unroll
                            for (int b = 0; b < 2; b++) {
                                int lo[4], hi[4];
                                float f[2];
                                if (BITS == 4) {
                                    constexpr unsigned ML = 0x0F0F0F0Fu, MH = 0xF0F0F0F0u;
                                    const uint4 a0 = w[b][0], a1 = w[b][1];
                                    mma_u8s8_z(lo, a0.x & ML, a1.x & ML, a0.y & ML, a1.y & ML, x0.x, x0.z);
                                    mma_u8s8_z(hi, a0.x & MH, a1.x & MH, a0.y & MH, a1.y & MH, x0.y, x0.w);
                                    mma_u8s8(lo, a0.z & ML, a1.z & ML, a0.w & ML, a1.w & ML, x1.x, x1.z);
                                    mma_u8s8(hi, a0.z & MH, a1.z & MH, a0.w & MH, a1.w & MH, x1.y, x1.w);
#pragma unroll
                                    for (int h = 0; h < 2; h++) f[h] = fmaf((float)(lo[2 * h] * 16 + hi[2 * h]), 256.0f, (float)(lo[2 * h + 1] * 16 + hi[2 * h + 1]));
                                } else {
                                    const uint4 a0 = w[b][0], a1 = w[b][1], c0 = w[b][2 % CV], c1 = w[b][3 % CV];
                                    mma_u8s8_z(lo, a0.x, c0.x, a0.z, c0.z, x0.x, x0.z);
                                    mma_u8s8_z(hi, a0.y, c0.y, a0.w, c0.w, x0.y, x0.w);
                                    mma_u8s8(lo, a1.x, c1.x, a1.z, c1.z, x1.x, x1.z);
                                    mma_u8s8(hi, a1.y, c1.y, a1.w, c1.w, x1.y, x1.w);
#pragma unroll
                                    for (int h = 0; h < 2; h++) f[h] = fmaf((float)(lo[2 * h] + hi[2 * h]), 4096.0f, (float)(lo[2 * h + 1] + hi[2 * h + 1]) * 16.0f);
                                }
#pragma unroll
                                for (int h = 0; h < 2; h++) acc[b][n][h] = fmaf(sz[b][h].x * mx, fmaf(-sz[b][h].y, my, f[h]), acc[b][n][h]);
                            }
                        }
                } else {
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
                            const uint4 x = *reinterpret_cast<const uint4 *>(bp + g8 * 64 + t * 16 + i * (M * 64) + n * 512);
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
            float *at = red + (kq % kCopies) * MP * kRPad + rp * (p.joint ? 16 : 32) + g8;
            const int second = p.joint ? 64 : 16;  // rows from the pair's first block to its second
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int i = 0; i < A; i++) {
                        if constexpr (INT) {
                            const float v = acc[b][n][i] + __shfl_xor_sync(0xffffffffu, acc[b][n][i], 1);
                            if (!(t & 1)) f(v, at + (2 * n + (t >> 1)) * kRPad + b * second + 8 * i);
                        } else {
                            f(acc[b][n][i], at + (n * 8 + 2 * t + (i & 1)) * kRPad + b * second + 8 * (i >> 1));
                        }
                    }
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
            // a task: four neighbouring rows of a token; the CTAs of a cluster share them
            const int sh = p.joint ? 4 : 5, share = ((M << sh) + p.slices - 1) / p.slices + 1 & ~1, end = min((rank + 1) * share, M << sh);
            for (int i0 = rank * share; i0 < end; i0 += NW * 32) {  // whole warps: two lanes hold eight rows
                const int i = min(i0 + tid, end - 1), m = i >> sh, c = i - (m << sh);
                const bool mine_too = i0 + tid < end;
                float4 v[2];
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    v[b] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (b && !p.joint) break;
                    const int row = b * 64 + c * 4;
                    if (parts) {
                        constexpr int kAtOnce = 4;  // parts on their way together
                        for (int c0 = c_first; c0 <= c_last; c0 += kAtOnce) {
                            float4 x[kAtOnce];
#pragma unroll
                            for (int k = 0; k < kAtOnce; k++) {
                                const int cc = min(c0 + k, c_last), first_tile = (int)((long long)p.total * cc / gridDim.x) / G;
                                x[k] = __ldcg(reinterpret_cast<const float4 *>(p.partial + ((size_t)cc * 2 + (first_tile == r.tile ? 0 : 1)) * (MP * kRRows) + m * kRRows + row));
                            }
#pragma unroll
                            for (int k = 0; k < kAtOnce; k++)
                                if (c0 + k <= c_last) add4(v[b], x[k]);
                        }
                    } else {
                        const float *q = red + m * kRPad + row;
                        if (p.slices == 1) {
                            v[b] = *reinterpret_cast<const float4 *>(q);
                            if (kCopies > 1) add4(v[b], *reinterpret_cast<const float4 *>(q + MP * kRPad));
                        } else {
                            const uint32_t qs = smem_u32(q);
                            constexpr int kAtOnce = 4;  // CTAs whose sums are on their way together
                            int k0 = 0;
                            for (; k0 + kAtOnce <= p.slices; k0 += kAtOnce) {
                                float4 x[kAtOnce][kCopies];
#pragma unroll
                                for (int k = 0; k < kAtOnce; k++)
#pragma unroll
                                    for (int j = 0; j < kCopies; j++) x[k][j] = ld_cluster(cluster_addr(qs, k0 + k) + j * MP * kRPad * 4);
#pragma unroll
                                for (int k = 0; k < kAtOnce; k++)
#pragma unroll
                                    for (int j = 0; j < kCopies; j++) add4(v[b], x[k][j]);
                            }
                            for (; k0 < p.slices; k0++)
#pragma unroll
                                for (int j = 0; j < kCopies; j++) add4(v[b], ld_cluster(cluster_addr(qs, k0) + j * MP * kRPad * 4));
                        }
                    }
                }
                const int n = r.tile * (p.joint ? 64 : 128) + c * 4;
                const float f[2][4] = {{v[0].x, v[0].y, v[0].z, v[0].w}, {v[1].x, v[1].y, v[1].z, v[1].w}};
                __half h[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    h[j] = __float2half_rn(f[0][j]);
                    if (p.joint == 2) {
                        h[j] = __float2half_rn((f[0][j] / (1.0f + expf(-f[0][j]))) * f[1][j]);
                    } else if (p.joint) {
                        const float gv = __half2float(h[j]), uv = __half2float(__float2half_rn(f[1][j]));
                        h[j] = __float2half_rn((gv / (1.0f + expf(-gv))) * uv);
                        if (p.div && n + j < p.N) h[j] = __float2half_rn(__half2float(h[j]) / __half2float(p.div[n + j]));
                    }
                }
                auto two = [](__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); };
                uint2 w = make_uint2(two(h[0], h[1]), two(h[2], h[3]));
                if (p.packed) {  // rows c .. c + 3 and c + 4 .. c + 7 of a chunk of eight, interleaved: the even lane writes the first two words of four
                    const uint2 o = make_uint2(__shfl_xor_sync(0xffffffffu, w.x, 1), __shfl_xor_sync(0xffffffffu, w.y, 1));
                    w = lane & 1 ? make_uint2(__byte_perm(o.y, w.y, 0x5410), __byte_perm(o.y, w.y, 0x7632)) : make_uint2(__byte_perm(w.x, o.x, 0x5410), __byte_perm(w.x, o.x, 0x7632));
                    if (mine_too && n < p.N) *reinterpret_cast<uint2 *>(p.y + token_chunk(n >> 3, m, M) * 8 + (lane & 1) * 4) = w;
                } else if (p.wide) {
                    if (mine_too && n < p.N) *reinterpret_cast<uint2 *>(p.y + (size_t)m * p.N + n) = w;
                } else if (mine_too) {
                    for (int j = 0; j < 4; j++)
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

// Eight values of a group of 128 (its sixteen chunks in sixteen consecutive lanes, chunk hl) of row m as 24-bit integers against the group's largest
// magnitude: rounding and digits of stage_chunk24 (v2_device.cuh), laid out for the fragments above.  scale: a factor of the row, into the constants.
__device__ __forceinline__ void plane_chunk(const float (&v)[8], bool live, int grp, int m, int M, int hl, float scale, uint8_t *__restrict__ out) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float sx = amax > 0.0f ? amax * (1.0f / (float)kActTop) : 1.0f, inv = amax > 0.0f ? (float)kActTop / amax : 0.0f;
    unsigned y[8];
    int lsum = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int xi = max(-kActTop, min(kActTop, __float2int_rn(v[i] * inv)));
        lsum += xi;
        y[i] = (unsigned)(xi + 0x808080) ^ 0x808080u;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (!live) return;
    uint8_t *slab = out + (size_t)grp * planes_slab(M);
    const int t = hl >> 2, j = hl & 3;
#pragma unroll
    for (int c = 0; c < 3; c++) {  // plane c: 0 high, 1 middle, 2 low = byte 2 - c of y; the even columns, then the odd ones
        const unsigned sel = (unsigned)(2 - c) | ((unsigned)(6 - c) << 4);
        const unsigned e = __byte_perm(__byte_perm(y[0], y[2], sel), __byte_perm(y[4], y[6], sel), 0x5410);
        const unsigned o = __byte_perm(__byte_perm(y[1], y[3], sel), __byte_perm(y[5], y[7], sel), 0x5410);
        *reinterpret_cast<uint2 *>(slab + (j >> 1) * (M * 192) + m * 192 + c * 64 + t * 16 + (j & 1) * 8) = make_uint2(e, o);
    }
    if (hl == 0) *reinterpret_cast<float2 *>(slab + M * 384 + m * 8) = make_float2(sx * 16.0f * scale, (float)lsum * 0.0625f);
}
__device__ __forceinline__ void half8(const __half *p, float (&v)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4 *>(p);
    const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 f = __half22float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

// Planes of x / awq (or x): grid (rows, groups / 8), two groups a warp.
__global__ void __launch_bounds__(128) rows_planes_kernel(const __half *__restrict__ x, const __half *__restrict__ awq, uint8_t *__restrict__ out, int G) {
    pdl_trigger();
    const int lane = threadIdx.x & 31, hl = lane & 15, m = blockIdx.x, want = blockIdx.y * 8 + (threadIdx.x >> 5) * 2 + (lane >> 4), grp = min(want, G - 1), k = grp * 128 + hl * 8;
    float v[8], a[8];
    if (awq) half8(awq + k, a);
    pdl_wait();
    half8(x + (size_t)m * G * 128 + k, v);
    if (awq)
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __fdiv_rn(v[i], a[i]);
    plane_chunk(v, want < G, grp, m, gridDim.x, hl, 1.0f, out);
}

// r = a + b, residual = f16(r), and r normed, as planes of what the next projections read (the reference's two forms, matvec.cu):
//   u: the unrounded r gamma / awq, the norm's factor in the constants;   n: f16(r rms_inv gamma) / awq.
// One CTA per row; a half-warp holds a group (two for rows longer than 4096) from the sums on.
constexpr int kNormPlaneChunks = 2;
__global__ void __launch_bounds__(512) norm_planes_kernel(const __half *__restrict__ a, const __half *__restrict__ b, const __half *__restrict__ gamma,
                                                          const __half *__restrict__ awq, __half *__restrict__ residual, uint8_t *__restrict__ u, uint8_t *__restrict__ n,
                                                          int G, float eps) {
    __shared__ float sh[16];
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, hl = lane & 15, m = blockIdx.x, M = gridDim.x, K = G * 128;
    float r[kNormPlaneChunks][8], ss = 0.0f;
    pdl_wait();
#pragma unroll
    for (int c = 0; c < kNormPlaneChunks; c++) {
        const int grp = c * 32 + warp * 2 + (lane >> 4), k = grp * 128 + hl * 8;
        if (grp < G) {
            float v[8];
            half8(a + (size_t)m * K + k, r[c]);
            half8(b + (size_t)m * K + k, v);
            uint4 out;
            __half2 *ho = reinterpret_cast<__half2 *>(&out);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                r[c][i] += v[i];
                ss = fmaf(r[c][i], r[c][i], ss);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) ho[i] = __floats2half2_rn(r[c][2 * i], r[c][2 * i + 1]);
            *reinterpret_cast<uint4 *>(residual + (size_t)m * K + k) = out;
        }
    }
    ss = warp_sum(ss);
    if (lane == 0) sh[warp] = ss;
    __syncthreads();
    float tot = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) tot += sh[w];
    const float ri = rsqrtf(tot / (float)K + eps);
#pragma unroll
    for (int c = 0; c < kNormPlaneChunks; c++) {
        if (c * 32 + warp * 2 >= G) break;  // warp-uniform
        const int want = c * 32 + warp * 2 + (lane >> 4), grp = min(want, G - 1), k = grp * 128 + hl * 8;
        float g[8], q[8], v[8];
        half8(gamma + k, g);
        if (awq) half8(awq + k, q);
        if (u) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                v[i] = r[c][i] * g[i];
                if (awq) v[i] = __fdiv_rn(v[i], q[i]);
            }
            plane_chunk(v, want < G, grp, m, M, hl, ri, u);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            v[i] = __half2float(__float2half_rn(r[c][i] * ri * g[i]));
            if (awq) v[i] = __fdiv_rn(v[i], q[i]);
        }
        plane_chunk(v, want < G, grp, m, M, hl, 1.0f, n);
    }
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

// Clusters of a size that the GPU holds at once (a cluster lies within a GPC, whose SMs need not divide evenly); asked for once per form and device
template <int NT, int BITS, bool INT>
int rows_clusters(int size, const Device *dev) {
    static std::atomic<int> held[64][kRMaxCluster + 1];
    const int at = dev->ordinal >= 0 && dev->ordinal < 64 ? dev->ordinal : -1;
    if (at >= 0 && held[at][size].load() > 0) return held[at][size].load() - 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(rows_warps<NT, BITS, INT>() * 32);
    cfg.dynamicSmemBytes = rows_smem_bytes<NT, BITS, INT>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_rows_kernel<NT, BITS, INT>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;  // (asked again next time)
    }
    if (at >= 0) held[at][size].store(n + 1);
    return n;
}

// How the row tiles are dealt out: a cluster of CTAs on slices of K for each, where there are few; a CTA for each; or equal shares of the list of all groups.
struct RowsPlan {
    int grid, slices;
};
// Counted in groups of K that the longest CTA takes.  The two ends of a share (sums and parts of two tiles through memory, a counter, the last CTA's
// sum) cost as much as 11 to 18 of a launch by itself (24 tokens, 28672 x 2048 in two waves of whole tiles 24.2 us, in shares 26.8; 12288 x 4096 19.7 and 22.9;
// 10240 x 8192 34.0 and 29.9), and 12 are the best line in whole steps (four 8B layers, 12 rows, gate and up: 64 groups or 49 in shares 662 and 649 us).
constexpr int kRShareEnds = 12;
template <int NT, int BITS, bool INT>
int rows_plan(int tiles, int G, bool shares, const Device *dev, RowsPlan *out) {
    constexpr int KQ = rows_klanes<NT, BITS, INT>(), MP = rows_tokens<NT, INT>();
    constexpr size_t smem = rows_smem_bytes<NT, BITS, INT>();
    static_assert(smem <= 227 * 1024, "the rings of this form do not fit");
    if (smem > dev->smem_optin) return IM_ERR_BOUNDS;
    static DeviceOnce once;  // per instantiation
    if (once.first(dev->ordinal)) IM_CUDA_CHECK(cudaFuncSetAttribute(gemm_rows_kernel<NT, BITS, INT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int sms = dev->sm_count, total = tiles * G;
    int slices = std::max(1, std::min(std::min(sms / tiles, kRMaxCluster), G / KQ));
    while (slices > 1 && rows_clusters<NT, BITS, INT>(slices, dev) < tiles) slices--;
    const int own = slices > 1 ? (G + slices - 1) / slices : (tiles + sms - 1) / sms * G;
    // two partial tiles of each CTA fit the scratch
    const int grid = (int)std::min<size_t>(std::min(sms, std::max(1, total / KQ)), kGemmScratchBytes / ((size_t)2 * MP * kRRows * sizeof(float)));
    *out = !shares || own <= (total + grid - 1) / grid + kRShareEnds ? RowsPlan{tiles * slices, slices} : RowsPlan{grid, 1};
    return IM_OK;
}

template <int NT, int BITS, bool INT>
int rows_launch(RowsParams p, const Device *dev, cudaStream_t st) {
    RowsPlan plan;
    if (const int rc = rows_plan<NT, BITS, INT>(p.total / p.G, p.G, p.partial != nullptr, dev, &plan); rc != IM_OK) return rc;
    p.slices = plan.slices;
    return rows_start(gemm_rows_kernel<NT, BITS, INT>, plan.grid, plan.slices, rows_warps<NT, BITS, INT>() * 32, rows_smem_bytes<NT, BITS, INT>(), st, p);
}

template <int BITS>
int rows_run(const RowsParams &p, const Device *dev, cudaStream_t st) {
    const int nt = (p.M + 7) / 8;
    if (nt <= 1) return rows_launch<1, BITS, false>(p, dev, st);
    if (nt == 2) return rows_launch<2, BITS, false>(p, dev, st);
    if (nt == 3) return rows_launch<3, BITS, false>(p, dev, st);
    if (nt == 4) return rows_launch<4, BITS, false>(p, dev, st);
    return rows_launch<6, 4, false>(p, dev, st);
}
template <int BITS>
int planes_run(const RowsParams &p, const Device *dev, cudaStream_t st) {
    if (p.M <= 2) return rows_launch<1, BITS, true>(p, dev, st);
    if (p.M <= 4) return rows_launch<2, BITS, true>(p, dev, st);
    if (p.M <= 8) return rows_launch<4, BITS, true>(p, dev, st);
    return rows_launch<8, BITS, true>(p, dev, st);
}

}  // namespace

// At least eight groups of K: the slices and warps of shorter sums have nothing to stream.
// The upper half of the token range (two groups to a stage, half the warps) only where the slices of K are not much longer than those of the tcgen05 kernel,
// whose number no cluster limits (gemm_tc.cu): a group is 0.5 us, the other's adding up 2 us, a packing pass 1.3.  40 tokens, tcgen05 / here, 4-bit:
// 4096 x 4096 (4 and 4 slices) 14.0 / 12.2 us, 2048 x 8192 (9 and 6) 13.7 / 14.4 with packing, 6144 x 4096 (3 and 2) 15.7 / 18.0; a wave of short whole tiles that need
// packing, 17920 x 1536, 48 tokens: 15.3 / 15.6.
bool gemm_rows_takes(const AffineWeight *w, int M, bool packs) {
    if (M < 1 || w->G < 8 || M > (w->bits == 4 ? kRowsMaxTokens : kRowsMaxTokens8) || !w->tiles || w->group_size != 128 || w->K % 128 != 0 || (w->bits != 4 && w->bits != 8) ||
        w->nblk > kSkMaxBlocks || (long long)w->nblk * w->G >= (1 << 30))
        return false;
    if (M <= (w->bits == 4 ? 32 : 16)) return true;
    const int tiles = (w->nblk + 7) / 8, sms = w->dev->sm_count, other = std::max(1, std::min(sms / tiles, w->G / 4));
    RowsPlan plan;
    if ((w->bits == 4 ? rows_plan<6, 4, false>(tiles, w->G, false, w->dev, &plan) : M <= 24 ? rows_plan<3, 8, false>(tiles, w->G, false, w->dev, &plan) : rows_plan<4, 8, false>(tiles, w->G, false, w->dev, &plan)) != IM_OK) return false;
    if (other == 1) return !packs || tiles > sms || w->G >= 16;
    return (w->G + plan.slices - 1) / plan.slices - (w->G + other - 1) / other <= (packs ? 0 : 4);
}

int token_pack(const __half *x, const __half *awq, __half *out, int M, int K, cudaStream_t st) {
    const int n = M * (K / 8);
    IM_CUDA_CHECK(launch_k(token_pack_kernel, dim3((n + 255) / 256), dim3(256), 0, st, x, awq, out, M, K / 8));
    return IM_OK;
}

static RowsParams rows_params(const AffineWeight *w, const AffineWeight *up, __half *y, int M, int joint, const GemmScratch *own) {
    RowsParams p{};
    p.tiles[0] = w->tiles;
    p.tiles[1] = up ? up->tiles : w->tiles;
    p.y = y; p.partial = own ? own->partial : nullptr; p.counters = own ? own->counters : nullptr; p.err = w->dev->err_flag;
    p.N = w->N; p.G = w->G; p.M = M; p.nblk = w->nblk; p.joint = up ? joint : 0;
    p.wide = w->N % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 8 == 0;
    p.total = (up ? (w->nblk + 3) / 4 : (w->nblk + 7) / 8) * w->G;
    return p;
}

int gemm_rows(const AffineWeight *w, const AffineWeight *up, const __half *packed, __half *y, int M, const __half *div, bool pack_out, const GemmScratch *own, cudaStream_t st) {
    RowsParams p = rows_params(w, up, y, M, 1, own);
    p.xs[0] = p.xs[1] = reinterpret_cast<const uint8_t *>(packed);
    p.slab = M * 256; p.split_row = 1 << 30; p.div = div; p.packed = pack_out ? 1 : 0;
    return w->bits == 8 ? rows_run<8>(p, w->dev, st) : rows_run<4>(p, w->dev, st);
}

bool planes_take(const AffineWeight *w, int M) { return M >= 1 && M <= kPlanesMaxRows && gemm_rows_takes(w, M); }

int rows_planes(const __half *x, const __half *awq, uint8_t *planes, int M, int K, cudaStream_t st) {
    const int G = K / 128;
    IM_CUDA_CHECK(launch_k(rows_planes_kernel, dim3(M, (G + 7) / 8), dim3(128), 0, st, x, awq, planes, G));
    return IM_OK;
}

int norm_planes(const __half *a, const __half *b, const __half *gamma, const __half *awq, __half *residual, uint8_t *u, uint8_t *n, int H, int M, float eps, cudaStream_t st) {
    const int G = H / 128;
    if (H % 128 != 0 || G > 32 * kNormPlaneChunks) return IM_ERR_BOUNDS;
    IM_CUDA_CHECK(launch_k(norm_planes_kernel, dim3(M), dim3(32 * std::min(16, (G + 1) / 2)), 0, st, a, b, gamma, awq, residual, u, n, G, eps));
    return IM_OK;
}

int matvec_planes(const AffineWeight *w, const AffineWeight *up, const uint8_t *planes, const uint8_t *planes_from, int split_row, __half *y, int M, bool round_gate_up,
                  const GemmScratch *own, cudaStream_t st) {
    RowsParams p = rows_params(w, up, y, M, round_gate_up ? 1 : 2, own);
    p.xs[0] = planes;
    p.xs[1] = planes_from ? planes_from : planes;
    p.slab = planes_slab(M); p.split_row = planes_from ? split_row : 1 << 30;
    return w->bits == 8 ? planes_run<8>(p, w->dev, st) : planes_run<4>(p, w->dev, st);
}

}  // namespace im
