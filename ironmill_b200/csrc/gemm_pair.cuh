// Projection of many tokens by CTA pairs (gemm_pair.cu).
#pragma once
#include "stack.cuh"

namespace im {

// Projections of `rows` weight rows that run on CTA pairs: more than one tile of tokens, and enough tiles of 256 rows x 128 tokens to occupy half
// of the pairs; below that the 128-row kernels, with two CTAs per SM, keep more SMs busy.
bool pair_gemm_takes(const Device *dev, int rows, int M);
// y = W x for bf16 weights [N, K] of row stride ldw and tokens x [M, ldx] (both 16-byte aligned)
int pair_gemm_bf16(const Device *dev, const void *w, int ldw, int N, int K, const void *x, int ldx, int M, const DenseEpi &epi, cudaStream_t st);
// fp16 tokens [M, K] against 4- or 8-bit codes of groups of 128: y[M, N] = f16(x dequant(w)^T), or with `up` (same shape as w) the
// gated activation f16(silu(f16(gate)) f16(up)) [M, N]
int pair_gemm_affine(const AffineWeight *w, const AffineWeight *up, const __half *x, __half *y, int M, cudaStream_t st);

}  // namespace im
