// 2-D tensor maps over row-major matrices of 16-bit elements, for cp.async.bulk.tensor copies into the 128-byte swizzle.
#pragma once
#include <cuda.h>

namespace im {

// [rows, cols] with row stride ld (elements, a multiple of 8; base 16-byte aligned): boxes of 64 columns x box_rows, zeros outside
int tmap_2d(const void *base, bool bf16, long long rows, long long cols, long long ld, int box_rows, CUtensorMap *out);

}  // namespace im
