// Forward gathers of large layers from tables staged in shared memory; see infer_staged.cu.
#pragma once

#include "lutb_common.cuh"

namespace lutb {

// Row indices as the staged gathers read them: one byte per (detector, sample), detector-major, `pitch` bytes apart.
size_t packed_index_pitch(int64_t batch);

// Whether a call takes the staged gather (the comments at the rules say where the lines lie).
bool infer_staged_fp32_applies(const lutb_layer_cfg *cfg, int64_t batch, const void *weights, const void *y);
bool infer_staged_int8_applies(const lutb_layer_cfg *cfg, int64_t batch, const void *q_tables);

// Samples of one pass (0: the staged gather does not run) and the workspace of a call: packed indices of a pass first
// (packed_index_bytes), then the partial sums of the detector blocks (fp32) or the integer form of the scales (int8), last the
// ordered anchors of the comparison (anchor_plan_bytes).
int64_t infer_staged_pass(const lutb_layer_cfg *cfg, int64_t batch, bool int8);
size_t packed_index_bytes(const lutb_layer_cfg *cfg, int64_t pass);
size_t anchor_plan_bytes(const lutb_layer_cfg *cfg);
size_t infer_staged_fp32_workspace(const lutb_layer_cfg *cfg, int64_t batch);
size_t infer_staged_int8_workspace(const lutb_layer_cfg *cfg, int64_t batch);

// y[b, :] += sum_t W[t, packed[t][b], :] for one pass
int launch_infer_staged_fp32(const lutb_layer_cfg *cfg, int64_t batch, const float *weights, const uint8_t *packed, float *partial,
                             float *y, cudaStream_t stream);
// scale_plan: the scales of every truncation block as integers (once per call)
int launch_int8_scale_plan(const lutb_layer_cfg *cfg, const float *scales, void *scale_plan, cudaStream_t stream);
// acc[b, :] += fixed-point block sums of scale[t] * q[t, packed[t][b], :] for one pass (exact de-quantisation)
int launch_infer_staged_int8(const lutb_layer_cfg *cfg, int64_t batch, const int8_t *q_tables, const float *scales,
                             const void *scale_plan, const uint8_t *packed, int32_t *acc, cudaStream_t stream);

}  // namespace lutb
