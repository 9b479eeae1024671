// The three contractions of the histogram path of the product-mode layer on the tensor cores (tcgen05); see
// hist_gemm_sm100.cu.  Counters H are fp16 [rows][KT] (exact up to 2048), KT = detectors * table rows, row-major.
#pragma once

#include <cuda_fp16.h>

#include "lutb_common.cuh"

namespace lutb {

enum HistGemmKind {
    HG_FORWARD,      // y [rows x O] += H . W               W [KT x O]
    HG_TABLE_GRAD,   // target [KT x O] += lr * H^T . dY     dY [rows x O]
    HG_ROW_DOTS,     // Q [rows x KT] = dY . W^T
};

// Scratch bytes of one call; never less for fewer rows than for more.
size_t hist_gemm_workspace(HistGemmKind kind, int rows, int KT, int O);
// O is a multiple of 4, KT a multiple of 16, all pointers 16-byte aligned.
int hist_gemm_forward(int rows, int KT, int O, const __half *H, const float *W, float *y, void *workspace,
                      size_t workspace_bytes, cudaStream_t stream);
int hist_gemm_table_grad(int rows, int KT, int O, const __half *H, const float *dY, float *target, float lr, void *workspace,
                         size_t workspace_bytes, cudaStream_t stream);
int hist_gemm_row_dots(int rows, int KT, int O, const float *dY, const float *W, float *Q, void *workspace,
                       size_t workspace_bytes, cudaStream_t stream);

}  // namespace lutb
