// Host interface of the kernel for batches that do not fill the GPU (mlp_wide.cu).
#pragma once

#include "hb_common.h"

struct hb_mlp;

namespace hb {
// G blocks per group (0: not for this batch), W columns per group, groups, queries per group.
struct WidePlan {
  int G, W, groups, per_group;
};
WidePlan wide_plan(int64_t Q, bool split, int sm_count);
// Queries that can travel as kernel parameters: no copy and no read over PCIe for the scalar API.
constexpr int kWideInline = 16;
// Queues the launch; *launched stays false when the stream has no scratch (see there).  host_inputs: feats
// and dev_row are ordinary host memory and Q <= kWideInline.
hb_status wide_predict(hb_mlp* h, const WidePlan& w, const float* feats, const uint8_t* dev_row, int64_t Q, float* out,
                       cudaStream_t stream, bool* launched, bool host_inputs = false);
// After a launch that gave up: every stream's scratch on the GPU is set up again before its next use.
void wide_start_over(int device);
void wide_handle_created(int device);
void wide_handle_destroyed(int device);
}  // namespace hb
