// Tensor maps for cp.async.bulk.tensor.
#pragma once

#include <cuda.h>

#include "lutb_common.cuh"

namespace lutb {

// A row-major matrix [rows x cols] of bytes (element_bytes 1), fp16 (2) or fp32 (4) in boxes of box_rows x box_cols, swizzled over 128, 64 or 0 bytes.  The base and
// the pitch are multiples of 16 bytes; elements outside the matrix read as zero and are not written.
int tensor_map_2d(CUtensorMap *map, int element_bytes, const void *p, int64_t rows, int64_t cols, int64_t pitch_bytes, int box_rows, int box_cols,
                  int swizzle_bytes);

}  // namespace lutb
