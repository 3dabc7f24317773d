// Host interface of the kernels for batches that do not fill the GPU (mlp_wide.cu, mlp_pairs.cu).
#pragma once

#include <cuda.h>

#include <mutex>

#include "hb_common.h"

struct hb_mlp;

namespace hb {
// Tensor maps of unswizzled bytes: a box of `box_rows` rows of `row_bytes`; a box of `box_rows` rows, at most 128, of
// `box_images` consecutive 16 KB images of 128-byte rows.
cudaError_t encode_rows(CUtensorMap* map, void* base, uint32_t row_bytes, uint64_t rows, uint32_t box_rows);
cudaError_t encode_images(CUtensorMap* map, void* base, uint64_t rows, uint32_t box_rows, uint32_t box_images);
// G blocks per group (0: not for this batch), groups, queries per group, shape of mlp_wide.cu's table.
struct WidePlan {
  int G, groups, per_group, shape;
};
// alone: no other batch that this kernel takes runs beside it (queries beyond full rounds of mlp_chain.cu's tiles are
// alone in this sense)
WidePlan wide_plan(int64_t Q, bool split, int sm_count, bool alone);
// Queries that can travel as kernel parameters: no copy and no read over PCIe for the scalar API.
constexpr int kWideInline = 16;
// A batch of queries.  Either every query has its own row of feats and of dev_row, or (grid_n > 0) the same
// grid_n feature rows are asked about for each of a list of device rows: query q is row q % grid_n on
// device grid_rows[q / grid_n], and nothing has to be repeated in memory.
constexpr int kMaxGridRows = 80;
struct MlpBatch {
  const float* feats = nullptr;
  const uint8_t* dev_row = nullptr;
  int64_t Q = 0;
  int64_t first = 0;                 // the batch is queries first .. first + Q - 1 of feats, dev_row or the grid
  float* out = nullptr;
  bool host_inputs = false;          // feats and dev_row are ordinary host memory, Q <= kWideInline
  int32_t grid_n = 0;
  const uint8_t* grid_rows = nullptr;   // host, Q / grid_n entries
  // Launches of one call that read nothing from one another: number `lane` of them (its own scratch), and
  // whether it may run beside the launch before it on the stream.
  int lane = 0;
  bool beside = false;
};
constexpr int kMaxLanes = 4;
// Replaces the plans of n <= kMaxLanes batches that are launched side by side, where others finish sooner; returns the time
// that they then take, in us.
int wide_plans_together(WidePlan* plans, const int64_t* Q, const bool* split, int n, int sm_count);
// One call's launches on `device` follow one another on their stream: the caller holds this from the first to the
// last of them.  A launch that runs beside the one before it relies on what its own call has queued; another
// thread's launch in between, on the same stream, could still be using the lane's scratch.
std::unique_lock<std::mutex> wide_queue(int device);
// Queues the launch; *launched stays false when the stream has no scratch (see there).  Call under wide_queue.
hb_status wide_predict(hb_mlp* h, const WidePlan& w, const MlpBatch& batch, cudaStream_t stream, bool* launched);
// After a launch that gave up: every stream's scratch on the GPU is set up again before its next use.
void wide_start_over(int device);
// Leaves the mark of a launch that gave up in the GPU's scratch (tests of the error path): 1, or ~b for block b of each group
// alone; synchronises.
hb_status wide_set_mark(int device, int32_t mark);
// The next launch of mlp_pairs.cu on each stream of the GPU takes what it exchanges for stale (tests).
void wide_expect_stale(int device);
// ... sends one word of a layer's output as if it were stale, in builds that can.
bool pairs_plant_words();
void wide_plant_stale(int device, int32_t layer, int32_t feature, int32_t word);
// Second runs of clusters in all streams' launches since their scratch was set up; synchronises.
hb_status wide_second_runs(int device, int64_t* runs);
void wide_handle_created(int device);
void wide_handle_destroyed(int device);
}  // namespace hb
