// Causal attention of a prompt chunk on the tcgen05 tensor cores (flash_tc.cu), shared by the fp16 and quantized caches of the
// Llama family and by the latent and grouped attention of models given as a list of layers.
#pragma once
#include "common.cuh"

namespace im {

// 16-bit rows in device memory: the 64-column block b of head index i at row r starts at
// base + (row0 + i * head_rows + r) * ld + col0 + i * head_cols + 64 b.
struct FlashRows {
    const void *base = nullptr;
    long long rows = 0, ld = 0;  // of the whole matrix
    long long row0 = 0, head_rows = 0;
    int col0 = 0, head_cols = 0;
    int blocks = 0;              // 64-column blocks of a row
};

struct FlashArgs {
    bool bf16 = false;           // element type: bf16, otherwise fp16
    int two_terms = 0;           // softmax weights enter their product as a sum of two 16-bit terms
    int T = 0, heads = 0, group = 1;  // tokens; query heads; query heads that share a key / value head
    FlashRows q, k, k2, v;       // rows of q: tokens; of k, k2 (the rest of a key, if any) and v: positions
    int base_pos = 0, slot = 0, n_max = 0;  // position of the first token: base_pos + pos_dev[slot]; no position from n_max on
    const int *pos_dev = nullptr;
    int chunk = 0;               // a position sees its own chunk of so many positions (0: everything before it)
    float scale = 1.0f;
    const float *sink = nullptr; // a keyless logit per head
    // Quantized caches in the rotated space (fp16, keys of 256 columns): q rows [R q | S R q], k rows [centroids | signs], v rows centroids.
    // A score is ks (q . k over the first 128 columns + kr (q . k over the last 128)), a weight enters the outputs times vs, and the
    // outputs are rotated back with `signs`. scales: per key / value head and tile of 64 positions 64 of ks, 64 of kr, 64 of vs.
    const float *scales = nullptr, *signs = nullptr;
    int scale_tiles = 0;         // tiles per head
    const void *gate = nullptr;  // outputs times sigmoid(gate): [T, ldg], head h at column h * gate_head
    int ldg = 0, gate_head = 0;
    void *out = nullptr;         // [T, ldo], head h at column h * out_head
    int ldo = 0, out_head = 0;
    int *err = nullptr;
};

// Shapes it is built for: keys of 128, 192 or (with scales) 256 columns, values of 128, everything 16-byte aligned.
bool flash_takes(const FlashArgs &a);
int flash_prepare(const Device *dev);  // launch attributes, on the current device
int flash_run(const FlashArgs &a, cudaStream_t st);

}  // namespace im
