// Projections of few tokens over quantized weights (gemm_rows.cu) and the token layout that they read.
#pragma once
#include "common.cuh"

namespace im {

constexpr int kRowsMaxTokens = 48, kRowsMaxTokens8 = 32;  // 4-bit, 8-bit codes

// Packed tokens, in 16-byte chunks of eight columns: [group of 128][eight columns i of a run of 32][token][run t].
// Chunk c of token m of M lies at this place; its halves in the order 0, 4, 1, 5, 2, 6, 3, 7.
__host__ __device__ __forceinline__ size_t token_chunk(int c, int m, int M) {
    const int grp = c >> 4, t = (c >> 2) & 3, i = c & 3;
    return ((size_t)(grp * 4 + i) * M + m) * 4 + t;
}
#ifdef __CUDACC__
__device__ __forceinline__ uint4 pack_chunk(const __half (&h)[8]) {
    auto two = [](__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); };
    return make_uint4(two(h[0], h[4]), two(h[1], h[5]), two(h[2], h[6]), two(h[3], h[7]));
}
#endif

// Byte planes of M rows for one group of 128 columns: [16 of a run of 32 columns][row][plane][run] x 16 bytes, then two constants a row.
__host__ __device__ constexpr int planes_slab(int M) { return M * 384 + (M + 1) / 2 * 16; }
constexpr int kPlanesMaxRows = 15;  // from 16 rows on a decode step's projections are the reference's matmul form (gemm_rows, gemm_affine_tc)

// packs: the tokens need a packing pass that the other kernel (gemm_tc.cu) would do without
bool gemm_rows_takes(const AffineWeight *w, int M, bool packs = false);
// f16(x / awq) (awq may be null) of M rows of K = a multiple of 128, packed; x anywhere, out 16-byte aligned and apart from it
int token_pack(const __half *x, const __half *awq, __half *out, int M, int K, cudaStream_t st);
// y[M, N] = packed tokens times w; with `up` (of w's form) the gated activation of both, divided by `div` if given; pack_out: packed for the next projection
// own: for parts of row tiles that CTAs share (null: none are)
int gemm_rows(const AffineWeight *w, const AffineWeight *up, const __half *packed, __half *y, int M, const __half *div, bool pack_out, const GemmScratch *own, cudaStream_t st);

// The same for rows as 24-bit integers.
bool planes_take(const AffineWeight *w, int M);
int rows_planes(const __half *x, const __half *awq, uint8_t *planes, int M, int K, cudaStream_t st);
// residual = f16(a + b); planes of the normed sum as the next projections read it: u (may be null) unrounded, n rounded.  IM_ERR_BOUNDS: H is not
// a multiple of 128 or too long.
int norm_planes(const __half *a, const __half *b, const __half *gamma, const __half *awq, __half *residual, uint8_t *u, uint8_t *n, int H, int M, float eps, cudaStream_t st);
// y[M, N]; rows from split_row on read planes_from (null: all read planes); with `up` the gated activation, of rounded or of f32 products
int matvec_planes(const AffineWeight *w, const AffineWeight *up, const uint8_t *planes, const uint8_t *planes_from, int split_row, __half *y, int M, bool round_gate_up,
                  const GemmScratch *own, cudaStream_t st);

}  // namespace im
