// Shared helpers for the sm_100a decode kernels and their C ABI.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <atomic>
#include <string>
#include <utility>
#include <vector>

#include "../../include/ironmill_cuda.h"

#define IM_EXPORT extern "C" __attribute__((visibility("default")))

namespace im {

// Thread-local error text behind im_cuda_last_error().
std::string &last_error();
int fail(int code, const char *fmt, ...) __attribute__((format(printf, 2, 3)));

#define IM_CUDA_CHECK(expr)                                                                   \
    do {                                                                                      \
        cudaError_t _e = (expr);                                                              \
        if (_e != cudaSuccess)                                                                \
            return im::fail(_e == cudaErrorMemoryAllocation ? IM_ERR_ALLOC : IM_ERR_CUDA,     \
                            "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, \
                            __LINE__);                                                        \
    } while (0)

#define IM_REQUIRE(cond, ...)                               \
    do {                                                    \
        if (!(cond)) return im::fail(IM_ERR_INVALID, __VA_ARGS__); \
    } while (0)

// Wrap an entry point body so that no C++ exception crosses the C boundary.
#define IM_GUARD_BEGIN try {
#define IM_GUARD_END                                                        \
    }                                                                       \
    catch (const std::bad_alloc &) { return im::fail(IM_ERR_ALLOC, "host allocation failed"); } \
    catch (const std::exception &e) { return im::fail(IM_ERR_CUDA, "exception: %s", e.what()); } \
    catch (...) { return im::fail(IM_ERR_CUDA, "unknown exception"); }

struct Device {
    int ordinal = 0;
    int sm_count = 0;
    size_t smem_optin = 0;
    cudaDeviceProp prop{};
    size_t allocated = 0;  // bytes handed out through this handle
    // stream-K scratch of the tiled matvec: partial sums of row blocks cut by a CTA boundary and the
    // arrival counters of those blocks.  One matvec in flight per device handle at a time.
    float *sk_partial = nullptr;
    int *sk_counters = nullptr;
    int *err_flag = nullptr;  // set by a kernel whose bounded wait ran out
    // f32 slices of a K-split tensor-core GEMM (gemm_tc.cu; few tokens against few row tiles).  One GEMM in flight per
    // device handle at a time.
    float *gemm_partial = nullptr;
};
constexpr size_t kGemmPartialBytes = (size_t)10 << 20;  // ten slices of 128 tokens x 2048 rows (dense.cu)
// A model's own: partial sums of its projections of few tokens (K slices, gemm_tc.cu; row tiles cut by CTA boundaries, gemm_rows.cu) and the counters of cut
// tiles, zero between launches.  One of a model's projections in flight at a time.
struct GemmScratch {
    float *partial = nullptr;
    int *counters = nullptr;
};
constexpr size_t kGemmScratchBytes = (size_t)10 << 20;  // three slices of 128 tokens x 6144 rows; two tiles of 48 tokens x 128 rows for each SM
constexpr int kSkMaxBlocks = 1 << 17;  // row blocks the counters cover (2M rows)

// cudaFuncSetAttribute applies to the current device: remember per device ordinal (not per thread) whether a
// kernel's attribute has been set.  Usage: static DeviceOnce once; if (once.first(dev->ordinal)) { set attributes }.
struct DeviceOnce {
    std::atomic<bool> done[64];
    DeviceOnce() {
        for (auto &d : done) d.store(false);
    }
    bool first(int ordinal) {
        if (ordinal < 0 || ordinal >= 64) return true;  // outside the table: set every time
        return !done[ordinal].exchange(true);
    }
};

// Allocation bookkeeping shared by buffers, weights and models.
int dev_malloc(Device *dev, void **ptr, size_t bytes);
void dev_free(Device *dev, void *ptr, size_t bytes);

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// GPU-resident affine weight after the load-time repack.
struct AffineWeight {
    Device *dev = nullptr;
    int N = 0, K = 0, group_size = 0, bits = 0, G = 0;
    uint8_t *codes = nullptr;  // [N, K/2] (4-bit) or [N, K] (8-bit), row-major, 16-byte aligned rows
    __half2 *sz = nullptr;     // [N, G] interleaved (scale, zero) fp16
    __half *awq = nullptr;     // [K] or nullptr
    // 4-bit, group 128: tiles of 16 rows x 128 columns (1 KB of nibbles) in [row block][group] order and
    // the 16 (scale, zero) pairs of each tile; see matvec_v2.cu
    uint8_t *tiles = nullptr;
    int nblk = 0;
    // gate+up pair in one tile stream (tile rows 0-7 from this matrix, 8-15 from `pair_with`), built on first use
    uint8_t *pair_tiles = nullptr;
    const AffineWeight *pair_with = nullptr;
    int pair_nblk = 0;
    size_t bytes = 0;
};

// bytes of one tile of the tile-major weight stream: 16 rows x 128 columns of codes + 16 (scale, zero) fp16 pairs
inline size_t tile_bytes_of(int bits) { return bits == 4 ? 1088 : 2112; }

struct V2Params {
    const uint8_t *tiles;  // [nblk][G][1088]: 1024 bytes of nibbles + 16 (scale, zero) pairs per tile
    const __half *awq, *x, *b, *gamma;
    __half *y, *residual_out, *normed_out;
    float eps;
    int N;       // logical outputs per batch row
    int K, G, nblk;
    int nring;   // stages in the shared-memory ring
    int split_tiles;  // 1: CTAs split the flattened tile list (stream-K); 0: whole row blocks per CTA
    float *partial;  // [grid][2][64]
    int *counters;   // [nblk], zero between launches
    int *err;
};

// INT4 or INT8 g128 GEMM on the tensor cores (gemm_tc.cu; few tokens gemm_rows.cu, many gemm_pair.cu): y[M, N] = f16(x / awq) * dequant(w)^T; xs_scratch holds M * K halves.
// IM_ERR_BOUNDS when the weight is not INT4 or INT8 group-128.  pack: the scratch is 16-byte aligned and shares no memory with x and y.
// own: where partial sums may go; without it (the stand-alone call, on any stream) only up to 64 tokens over few rows are cut along K, in the device handle's scratch.
enum TokenForm { kTokensRaw, kTokensScaled, kTokensPacked };  // x as it is; f16(x / awq); that, packed for gemm_rows.cu (where gemm_rows_takes says so)
int gemm_affine_tc(const AffineWeight *w, const __half *x, __half *y, int M, __half *xs_scratch, cudaStream_t st, TokenForm form = kTokensRaw,
                   bool pack = true, const GemmScratch *own = nullptr);
// The gated activation y[M, N] = f16(silu(f16(gate x)) f16(up x)) in one launch, for two weights of the same form and activation scales;
// only where gemm_affine_joins() says so.
bool gemm_affine_joins(const AffineWeight *gate, int M);
int gemm_affine_gate_up(const AffineWeight *gate, const AffineWeight *up, const __half *x, __half *y, int M, __half *xs_scratch, cudaStream_t st, TokenForm form);
// y[M, N] = f16(x w^T) for fp16 weights [N, K] and rows x [M, K] on the tensor cores (dense.cu); IM_ERR_BOUNDS for rows that are not 16-byte aligned
int dense_rows_f16(const Device *dev, const __half *w, int N, int K, const __half *x, __half *y, int M, cudaStream_t st);
int residual_norm_scaled(const __half *a, const __half *b, const __half *gamma, const __half *scale, __half *out, __half *residual, int H, int T, float eps,
                         cudaStream_t st, bool packed = false);
// Gate/up pair as one tile stream (matvec.cu); built on first use.
int ensure_pair(const AffineWeight *gate, const AffineWeight *up, cudaStream_t st);
int v2_run(int mode, int nb, const V2Params &p, const Device *dev, cudaStream_t st, int bits = 4);
int v2_repack8(const uint8_t *codes, const __half2 *sz, int N, int K, int G, int nblk, uint8_t *tiles, cudaStream_t st);
int v2_repack(const uint8_t *codes0, const __half2 *sz0, const uint8_t *codes1, const __half2 *sz1, int N, int K, int G, int nblk,
              int rows_per_blk, uint8_t *tiles, cudaStream_t st);

// ---- programmatic dependent launch ------------------------------------------
// Decode is a chain of ~230 short kernels per token.  Launched with the programmatic-serialization
// attribute, a kernel may start while its predecessor is still draining: everything it does before
// pdl_wait() (barrier set-up, streaming constant weights into shared memory) overlaps the predecessor's
// tail; pdl_wait() returns once the predecessor has completed and its writes are visible.  Every kernel
// launched through launch_k() must therefore call pdl_wait() before it reads anything a predecessor wrote
// and before its first global write.

template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// ---- device helpers -------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Streaming 128-bit load that does not allocate in L1 (weights are read once).
__device__ __forceinline__ uint4 ldg_stream_v4(const void *p) {
    uint4 r;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

// 4-way byte dot products: unsigned codes against signed / unsigned activation bytes.
__device__ __forceinline__ int dp4a_us(unsigned a, unsigned b_signed, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b_signed), "r"(c));
    return d;
}
__device__ __forceinline__ int dp4a_uu(unsigned a, unsigned b, int c) {
    unsigned d;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"((unsigned)c));
    return (int)d;
}

// Arguments of the fused (QK-norm +) RoPE kernel (norm.cu), shared with the model engine.
struct QkRopeArgs {
    const __half *q_in, *k_in, *v_in;
    int q_stride, k_stride, v_stride;  // elements between consecutive tokens of the inputs
    __half *q_out, *k_out, *v_out;
    const __half *qw, *kw, *cosc, *sinc;
    int nh, nkv, hd, rotary_dim, seq_offset;
    const int *pos_dev;  // per-sequence base positions (tokens_per_seq tokens each) or nullptr
    int tokens_per_seq;
    float eps;
    int with_norm;
};

int launch_qk_rope(const QkRopeArgs &a, int T, cudaStream_t st);

// TurboQuant constants + scratch (turboquant.cu)
struct Tq {
    Device *dev = nullptr;
    int hd = 0, n_bits = 0, k_levels = 0, v_levels = 0;
    float *signs = nullptr, *qjl = nullptr, *qjl_t = nullptr, *k_cb = nullptr, *k_bd = nullptr, *v_cb = nullptr, *v_bd = nullptr;
    float *scratch = nullptr;
    size_t scratch_bytes = 0;
    bool scratch_used = false;  // some launch, perhaps a captured one, holds its address: outgrown, it stays until the handle goes
    std::vector<std::pair<float *, size_t>> outgrown;
    size_t const_bytes = 0;
};

int tq_auto_splits(const Device *dev, int nseq, int T, int nh, int nkv, int seq_len);
// Prefill chunks of one sequence: dequantise the cached rows once, causal flash attention on the tensor cores (tq_prefill.cu).
size_t tq_prefill_scratch_bytes(int nkv, int max_seq);
struct TqPromptQuery {       // query rows as projected: head h at column 128 h
    const __half *q;
    int stride;
    const __half *qw = nullptr;  // norm weights, or none
    float eps = 0.0f;
    const __half *cosc = nullptr, *sinc = nullptr;
    int rotary_dim = 0;
};
int tq_prefill_attention_launch(const Tq *tq, void *q_rows, void *dq, const TqPromptQuery &q, const uint8_t *kc, const uint8_t *vc, const float *ks,
                                const float *vs, const float *krn, float attn_scale, __half *out, int slot, int nh, int nkv, int max_seq,
                                const int *pos_dev, int T, int ctx_end, cudaStream_t st, int base_pos = 0);
struct TqPrep;
int tq_prompt_encode_launch(const Tq *tq, const TqPrep &a, int slot, cudaStream_t st);
bool tq_prefill_takes(int nh, int nkv);  // head groupings the prefill pass is built for
// Inputs of the fused RoPE + cache write + query rotation launch (turboquant.cu).
struct TqPrep {
    const __half *qkv;  // [nseq*T, stride]: q | k | v of one token
    int stride, k_off, v_off;
    const __half *kv = nullptr;  // optional: K and V rows live in their own buffer [nseq*T, kv_stride]; k_off / v_off index it
    int kv_stride = 0;
    const __half *qw, *kw, *cosc, *sinc;
    int nh, nkv, rotary_dim, with_norm, T, nseq, max_seq, base_pos;
    float eps;
    const int *pos_dev;
    const int *slot_map = nullptr;  // optional: sequence index -> cache slot
    float *qrot;    // out [nseq*T, nh, 2, hd]
    __half *q_out;  // optional out [nseq*T, nh, hd]
    uint8_t *kc, *vc;
    float *ks, *vs, *krn;
};
int tq_prep_launch(const Tq *tq, const TqPrep &a, cudaStream_t st);
int tq_attention_launch(const Tq *tq, float *scratch, const __half *q, const uint8_t *kc, const uint8_t *vc, const float *ks,
                        const float *vs, const float *krn, float attn_scale, __half *out, int nseq, int nh, int nkv, int max_seq,
                        int base_pos, const int *pos_dev, int T, int splits, bool own_parts, cudaStream_t st, const float *qrot = nullptr,
                        const int *slot_map = nullptr);  // own_parts: splits is an automatic count, each token takes what its context fills

// ---- fp16 (unquantized) KV cache: kv_f16.cu ----
struct Kv16Prep {
    __half *qkv;  // [nseq*T, stride]: q | k | v of one token; the query heads are normed / rotated in place
    int stride, k_off, v_off;
    const __half *kv;  // nullptr, or the buffer [nseq*T, kv_stride] that holds the K and V rows (k_off / v_off index it)
    int kv_stride;
    const __half *qw, *kw, *cosc, *sinc;
    int nh, nkv, rotary_dim, with_norm, T, nseq, max_seq, base_pos;
    float eps;
    const int *pos_dev;
    const int *slot_map;  // optional: sequence index -> cache slot
    __half *kc, *vc;      // [slots, nkv, max_seq, 128]
};
int kv16_prep_launch(const Kv16Prep &a, cudaStream_t st);
size_t kv16_scratch_bytes(int tokens, int nh, int splits);
int kv16_auto_splits(const Device *dev, int tokens, int nkv, int max_ctx);
int kv16_attention_launch(const Device *dev, float *scratch, size_t scratch_bytes, const __half *q, int q_stride, const __half *kc, const __half *vc,
                          float scale, __half *out, int nseq, int nh, int nkv, int max_seq, int base_pos, const int *pos_dev, int T, int splits,
                          int ctx_hint, cudaStream_t st, const int *slot_map, int prefill_slot = -1);  // prefill_slot >= 0: one sequence in that cache slot

}  // namespace im

// The opaque handle types of the C ABI are thin tags over the internal structs.
struct im_device : im::Device {};
struct im_affine_weight : im::AffineWeight {};
