// Trace-level totals and the special-operation ratio: small reduction and
// elementwise kernels that follow the two big ones on the same stream.
//
// hb_segment_sum stands in for Trace.run_time_ms / RunTimePrediction.run_time_ms
// (analyzer/habitat/analysis/trace.py:26-36, run_time.py:49-58) over many
// segments at once; hb_special_scale for the last line of
// Predictor._{conv2d,linear,bmm,lstm}_scale and the clamp in _special_scale
// (analysis/predictor.py:132-148, :182).
//
// Sums are accumulated in float64 with a fixed assignment of elements to lanes
// and a fixed reduction tree, so the result does not depend on grid size or
// scheduling (no floating-point atomics).
#include <mutex>

#include "hb_common.h"
#include "reduce_stage1.cuh"

namespace {

// One block per segment.
__global__ void __launch_bounds__(kSumThreads)
segment_sum_kernel(const float* __restrict__ values, const int64_t* __restrict__ offsets,
                   int64_t n_segments, double* __restrict__ out) {
  for (int64_t s = blockIdx.x; s < n_segments; s += gridDim.x) {
    const int64_t lo = offsets[s], hi = offsets[s + 1];
    double acc = 0.0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += kSumThreads) acc += static_cast<double>(values[i]);
    const double t = block_sum(acc);
    if (threadIdx.x == 0) out[s] = t;
  }
}

template <int CLUSTER>
__global__ void __launch_bounds__(kFinalThreadsMax)
plane_final_kernel(const double* __restrict__ partial, int per_plane, double* __restrict__ out) {
  hb_grid_dependency_wait();
  const double t = plane_total<CLUSTER>(partial, per_plane);
  if (threadIdx.x == 0 && blockIdx.x % CLUSTER == 0) out[blockIdx.x / CLUSTER] = t;
}

__global__ void __launch_bounds__(256)
special_scale_kernel(const float* __restrict__ run_time_ms, const float* __restrict__ pred_dest,
                     const float* __restrict__ pred_orig, int64_t n, float* __restrict__ out_ms,
                     uint32_t* __restrict__ negative_count) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  bool neg = false;
  if (i < n) {
    // predictor.py:182: run_time_ms * pred_dest / pred_orig, left to right
    // (float64 there; the two predictions are float32 values)
    double v = static_cast<double>(run_time_ms[i]) * static_cast<double>(pred_dest[i]) /
               static_cast<double>(pred_orig[i]);
    neg = v < 0;
    if (neg) v = 0.0;  // predictor.py:135-141
    out_ms[i] = static_cast<float>(v);
  }
  if (negative_count) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, neg);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(negative_count, __popc(m));
  }
}

// Segment sums over several planes that share the offsets.  The passes of a trace hold a kernel or a few
// each, and a block of 256 threads per sum (segment_sum_kernel) spent its time in barriers: LANES lanes share
// a sum, one for short segments (neighbouring threads then read and write neighbouring values), else a warp.
// `copy`, if given, receives the values themselves: with both outputs in page-locked host memory a caller
// gets the times and their sums without a copy that the launches behind this one would wait for.
template <int LANES>
__global__ void __launch_bounds__(256)
segment_sum_planes_kernel(const float* __restrict__ values, int64_t plane_len, const int64_t* __restrict__ offsets,
                          int64_t n_segments, int64_t n_sums, double* __restrict__ out, int64_t n_values,
                          float* __restrict__ copy) {
  hb_grid_dependency_wait();
  const int lane = threadIdx.x % LANES;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * (256 / LANES);
  for (int64_t w = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / LANES; w < n_sums; w += stride) {
    const int64_t plane = w / n_segments, s = w - plane * n_segments;
    const int64_t lo = offsets[s], hi = offsets[s + 1];
    const float* v = values + plane * plane_len;
    double acc = 0.0;
    for (int64_t i = lo + lane; i < hi; i += LANES) acc += static_cast<double>(v[i]);
    if (LANES == 32) acc = warp_sum(acc);
    if (lane == 0) out[w] = acc;
  }
  if (copy)
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < n_values; i += gridDim.x * 256ll)
      copy[i] = values[i];
}

// special_scale_kernel over a grid of predictions [1 + T][n] (row 0: the origin's): ms[t][i] =
// run_time[i] pred[1 + t][i] / pred[0][i], for up to four operation kinds at a time (blockIdx.y).
struct ScaleGrid {
  const float* run_time_ms;
  const float* pred;
  float* out_ms;
  uint32_t* negative_count;
  int32_t n, T;
};
struct ScaleGrids {
  ScaleGrid g[4];
};
__global__ void __launch_bounds__(256) special_scale_grid_kernel(const __grid_constant__ ScaleGrids grids) {
  hb_grid_dependency_wait();
  const ScaleGrid& g = grids.g[blockIdx.y];
  const int64_t total = static_cast<int64_t>(g.n) * g.T;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * 256; i0 < total; i0 += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t i = i0 + threadIdx.x;
    bool neg = false;
    if (i < total) {
      const int64_t k = i % g.n;
      double v = static_cast<double>(g.run_time_ms[k]) * static_cast<double>(g.pred[g.n + i]) /
                 static_cast<double>(g.pred[k]);
      neg = v < 0;
      if (neg) v = 0.0;
      g.out_ms[i] = static_cast<float>(v);
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, neg);
    if (g.negative_count && (threadIdx.x & 31) == 0 && m) atomicAdd(g.negative_count, __popc(m));
  }
}

// Totals of iterations: a warp per (iteration, destination) adds the iteration's overheads, its kernels'
// times and, kind by kind, its special operations' times (formed here from the prediction grid and rounded to
// float32 as hb_special_scale stores them).  Nothing in between is written: the separate sums, ratios and
// repeats took about thirty launches per pass.  Reads each input once per destination, from L2.
constexpr int kIterKinds = 8;
struct IterKind {
  const float* rt;
  const float* pred;
  const int64_t* offsets;
  int64_t n;
};
struct IterParams {
  const float* overhead;
  const float* measured;
  const float* scaled;
  const int64_t* offsets;
  double* out;
  int64_t K, I;
  int32_t D, n_kinds, add;            // add: on top of what out holds
  int8_t plane[HB_MAX_DEVICES];       // row of the prediction grids, 0 for the origin itself
  IterKind kind[kIterKinds];
};
__global__ void __launch_bounds__(256) iteration_totals_kernel(const __grid_constant__ IterParams p) {
  hb_grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int64_t w = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (w >= p.I * p.D) return;
  const int64_t i = w / p.D;
  const int d = static_cast<int>(w - i * p.D), plane = p.plane[d];
  double total = 0.0;
  if (p.add) {
    total = p.out[w];
  } else {
    const float* t = plane == 0 ? p.measured : p.scaled + d * p.K;
    double over = 0.0, kern = 0.0;
    for (int64_t k = p.offsets[i] + lane; k < p.offsets[i + 1]; k += 32) {
      over += static_cast<double>(p.overhead[k]);
      kern += static_cast<double>(t[k]);
    }
    total = (warp_sum(over) + warp_sum(kern)) / 1e6;   // lane 0
  }
  for (int q = 0; q < p.n_kinds; ++q) {
    const IterKind& kind = p.kind[q];
    double acc = 0.0;
    for (int64_t k = kind.offsets[i] + lane; k < kind.offsets[i + 1]; k += 32) {
      float ms = kind.rt[k];
      if (plane != 0) {
        const double v = static_cast<double>(ms) * static_cast<double>(kind.pred[plane * kind.n + k]) /
                         static_cast<double>(kind.pred[k]);
        ms = static_cast<float>(v < 0 ? 0.0 : v);
      }
      acc += static_cast<double>(ms);
    }
    total += warp_sum(acc);
  }
  if (lane == 0) p.out[w] = total;
}

// Per-GPU scratch of the two-stage sums.  A buffer that a launch may still be reading (or
// that a captured graph refers to) is never freed: when more room is needed a larger buffer
// is allocated and the old one is kept until the process ends.
constexpr int kMaxCudaDevices = 64;
struct SumScratch {
  double* plane = nullptr;      // [planes][kPlaneBlocks]
  size_t planes = 0;
  double* group = nullptr;      // [kMaxGroups][kGroupBlocks]
};
SumScratch g_scratch[kMaxCudaDevices];
std::mutex g_scratch_mu;

// Scratch of the current GPU with room for `planes` plane sums (0: leave as is) and, when
// `want_group`, for the group sum.  Allocates on the first call that needs more.
hb_status scratch_for_current_device(size_t planes, bool want_group, SumScratch* out) {
  int dev = 0;
  HB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxCudaDevices) {
    hb::set_error("device ordinal %d out of range", dev);
    return HB_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  SumScratch& sc = g_scratch[dev];
  if (planes > sc.planes) {
    // at least 64 planes, then doubling: a handful of allocations over the life of the process
    size_t want = sc.planes ? sc.planes : 64;
    while (want < planes) want *= 2;
    double* fresh = nullptr;
    HB_CUDA_TRY(cudaMalloc(&fresh, sizeof(double) * kPlaneBlocks * want));
    sc.plane = fresh;   // the previous buffer stays allocated: launches in flight and graphs may hold it
    sc.planes = want;
  }
  if (want_group && !sc.group) HB_CUDA_TRY(cudaMalloc(&sc.group, sizeof(double) * kMaxGroups * kGroupBlocks));
  *out = sc;
  return HB_OK;
}

}  // namespace

// Current size, in planes, of the plane-sum scratch of CUDA device `device` (0: none yet).
// For tests of the per-GPU bookkeeping; no reference counterpart.
extern "C" int64_t hb_plane_sum_scratch_planes(int32_t device) {
  if (device < 0 || device >= kMaxCudaDevices) return -1;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  return static_cast<int64_t>(g_scratch[device].planes);
}

extern "C" hb_status hb_segment_sum(const float* values, const int64_t* offsets,
                                    int64_t n_segments, double* out, void* stream) {
  if (n_segments < 0 || (n_segments > 0 && (!values || !offsets || !out))) {
    hb::set_error("hb_segment_sum: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n_segments == 0) return HB_OK;
  const int64_t blocks = n_segments < 148 * 8 * 8 ? n_segments : 148 * 8 * 8;
  segment_sum_kernel<<<static_cast<unsigned>(blocks), kSumThreads, 0,
                       static_cast<cudaStream_t>(stream)>>>(values, offsets, n_segments, out);
  HB_CUDA_TRY(cudaGetLastError());
  return HB_OK;
}

extern "C" hb_status hb_plane_sum(const float* values, int64_t plane_len, int32_t n_planes,
                                  double* out, void* stream) {
  if (plane_len < 0 || n_planes < 0 || n_planes > 65535 || (n_planes > 0 && (!values || !out))) {
    hb::set_error("hb_plane_sum: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n_planes == 0) return HB_OK;
  SumScratch sc;
  const hb_status st = scratch_for_current_device(static_cast<size_t>(n_planes), false, &sc);
  if (st != HB_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  HB_CUDA_TRY(hb::launch_overlapped(plane_partial_kernel, dim3(n_planes, kPlaneBlocks), dim3(kSumThreads), 0, s,
                                    values, plane_len, sc.plane));
  HB_CUDA_TRY(hb::launch_overlapped(plane_final_kernel<1>, dim3(n_planes), dim3(kSumThreads), 0, s,
                                    static_cast<const double*>(sc.plane), kPlaneBlocks, out));
  return HB_OK;
}

extern "C" hb_status hb_partials_sum(const double* partials, int32_t per_plane, int32_t n_planes, double* out,
                                     void* stream) {
  if (per_plane < 0 || n_planes < 0 || n_planes > 65535 || (n_planes > 0 && (!out || (per_plane > 0 && !partials)))) {
    hb::set_error("hb_partials_sum: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n_planes == 0) return HB_OK;
  if (final_cluster(per_plane) == 1) {
    HB_CUDA_TRY(hb::launch_overlapped(plane_final_kernel<1>, dim3(n_planes), dim3(final_threads(per_plane)), 0,
                                      static_cast<cudaStream_t>(stream), partials, per_plane, out));
  } else {
    HB_CUDA_TRY(hb::launch_overlapped_cluster(plane_final_kernel<kFinalCluster>, dim3(n_planes * kFinalCluster),
                                              dim3(kFinalThreadsMax), kFinalCluster,
                                              static_cast<cudaStream_t>(stream), partials, per_plane, out));
  }
  return HB_OK;
}

extern "C" hb_status hb_group_sum(const float* values, const uint8_t* keys, int64_t n, int32_t n_groups,
                                  double* out, void* stream) {
  if (n < 0 || n_groups < 0 || n_groups > 256 || (n_groups > 0 && !out) || (n > 0 && (!values || !keys))) {
    hb::set_error("hb_group_sum: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n_groups == 0) return HB_OK;
  SumScratch sc;
  const hb_status st = scratch_for_current_device(0, true, &sc);
  if (st != HB_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // eight groups per pass; the passes share the scratch and follow one another on the stream
  for (int32_t g0 = 0; g0 < n_groups; g0 += kMaxGroups) {
    const int32_t ng = n_groups - g0 < kMaxGroups ? n_groups - g0 : kMaxGroups;
    HB_CUDA_TRY(hb::launch_overlapped(group_partial_kernel, dim3(kGroupBlocks), dim3(kSumThreads), 0, s, values,
                                      keys, n, g0, ng, sc.group));
    static_assert(kGroupBlocks == kPlaneBlocks, "the final stage is shared with the plane sum");
    HB_CUDA_TRY(hb::launch_overlapped(plane_final_kernel<1>, dim3(ng), dim3(kSumThreads), 0, s,
                                      static_cast<const double*>(sc.group), kGroupBlocks, out + g0));
  }
  return HB_OK;
}

extern "C" hb_status hb_special_scale(const float* run_time_ms, const float* pred_dest,
                                      const float* pred_orig, int64_t n, float* out_ms,
                                      uint32_t* negative_count, void* stream) {
  if (n < 0 || (n > 0 && (!run_time_ms || !pred_dest || !pred_orig || !out_ms))) {
    hb::set_error("hb_special_scale: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n == 0) return HB_OK;
  const int64_t blocks = (n + 255) / 256;
  special_scale_kernel<<<static_cast<unsigned>(blocks), 256, 0,
                         static_cast<cudaStream_t>(stream)>>>(run_time_ms, pred_dest, pred_orig, n,
                                                              out_ms, negative_count);
  HB_CUDA_TRY(cudaGetLastError());
  return HB_OK;
}

extern "C" hb_status hb_segment_sum_planes(const float* values, int64_t plane_len, int32_t n_planes,
                                           const int64_t* offsets, int64_t n_segments, double* out, float* copy,
                                           void* stream) {
  if (n_segments < 0 || n_planes < 0 || plane_len < 0 ||
      (n_segments > 0 && n_planes > 0 && (!values || !offsets || !out))) {
    hb::set_error("hb_segment_sum_planes: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  const int64_t sums = n_segments * n_planes;
  if (sums == 0) return HB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool small = plane_len <= 8 * n_segments;   // values per sum on average
  const int64_t want = small ? (sums + 255) / 256 : (sums + 7) / 8;
  const int64_t blocks = want < 148 * 8 ? want : 148 * 8;
  HB_CUDA_TRY(hb::launch_overlapped(small ? segment_sum_planes_kernel<1> : segment_sum_planes_kernel<32>,
                                    dim3(static_cast<unsigned>(blocks)), dim3(256), 0, s, values, plane_len, offsets,
                                    n_segments, sums, out, plane_len * n_planes, copy));
  return HB_OK;
}

extern "C" hb_status hb_iteration_totals(const float* overhead_ns, const float* run_time_ns, const float* scaled_ns,
                                         int64_t n_kernels, const int64_t* kernel_offsets, int64_t n_iterations,
                                         int32_t n_destinations, const uint8_t* same, const hb_iteration_kind* kinds,
                                         int32_t n_kinds, double* out, void* stream) {
  if (n_iterations < 0 || n_destinations < 0 || n_destinations > HB_MAX_DEVICES || n_kinds < 0 || n_kernels < 0 ||
      (n_kinds > 0 && !kinds) ||
      (n_iterations > 0 && n_destinations > 0 &&
       (!kernel_offsets || !same || !out || (n_kernels > 0 && (!overhead_ns || !run_time_ns || !scaled_ns))))) {
    hb::set_error("hb_iteration_totals: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n_iterations == 0 || n_destinations == 0) return HB_OK;
  IterParams p{};
  p.overhead = overhead_ns; p.measured = run_time_ns; p.scaled = scaled_ns; p.offsets = kernel_offsets; p.out = out;
  p.K = n_kernels; p.I = n_iterations; p.D = n_destinations;
  int other = 0;
  for (int d = 0; d < n_destinations; ++d) p.plane[d] = static_cast<int8_t>(same[d] ? 0 : ++other);
  const int64_t blocks = (n_iterations * n_destinations + 7) / 8;
  if (blocks > 0x7FFFFFFF) {
    hb::set_error("hb_iteration_totals: too many iterations for one launch");
    return HB_ERR_TOO_LARGE;
  }
  int done = 0;
  do {
    p.n_kinds = 0;
    for (; done < n_kinds && p.n_kinds < kIterKinds; ++done) {
      const hb_iteration_kind& k = kinds[done];
      if (k.n == 0) continue;
      if (k.n < 0 || !k.run_time_ms || !k.offsets || (other > 0 && !k.pred)) {
        hb::set_error("hb_iteration_totals: bad kind %d", done);
        return HB_ERR_INVALID_ARGUMENT;
      }
      p.kind[p.n_kinds++] = IterKind{k.run_time_ms, k.pred, k.offsets, k.n};
    }
    HB_CUDA_TRY(hb::launch_overlapped(iteration_totals_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0,
                                      static_cast<cudaStream_t>(stream), p));
    p.add = 1;
  } while (done < n_kinds);
  return HB_OK;
}

extern "C" hb_status hb_special_scale_grid(const hb_scale_grid* items, int32_t n_items, void* stream) {
  if (n_items < 0 || n_items > 4 || (n_items > 0 && !items)) {
    hb::set_error("hb_special_scale_grid: 0 to 4 kinds");
    return HB_ERR_INVALID_ARGUMENT;
  }
  ScaleGrids grids{};
  int kinds = 0;
  int64_t most = 0;
  for (int i = 0; i < n_items; ++i) {
    const hb_scale_grid& g = items[i];
    if (g.n < 0 || g.n > 0x7FFFFFFF || g.n_destinations < 0 ||
        (g.n > 0 && g.n_destinations > 0 && (!g.run_time_ms || !g.pred || !g.out_ms))) {
      hb::set_error("hb_special_scale_grid: bad kind %d", i);
      return HB_ERR_INVALID_ARGUMENT;
    }
    const int64_t total = g.n * g.n_destinations;
    if (total == 0) continue;
    grids.g[kinds++] = ScaleGrid{g.run_time_ms, g.pred, g.out_ms, g.negative_count, static_cast<int32_t>(g.n),
                                 g.n_destinations};
    most = total > most ? total : most;
  }
  if (kinds == 0) return HB_OK;
  const int64_t blocks = (most + 255) / 256 < 148 * 8 ? (most + 255) / 256 : 148 * 8;
  HB_CUDA_TRY(hb::launch_overlapped(special_scale_grid_kernel, dim3(static_cast<unsigned>(blocks), kinds), dim3(256), 0,
                                    static_cast<cudaStream_t>(stream), grids));
  return HB_OK;
}

// ---------------------------------------------------------------------------
// Plane sums for callers that must not allocate
// ---------------------------------------------------------------------------
// hb_plane_sum above keeps its stage-1 partial sums in a buffer it obtains with
// cudaMalloc on first use.  Some hosts cannot tolerate that: a serving process
// that hands the whole device to its own memory pool at start-up (a later
// driver allocation fails or fragments the pool), or one whose latency rules
// forbid driver allocations once initialisation is over.  For them the same two
// kernels run on a scratch array that is part of the library image: it occupies
// kStaticPlanes * kPlaneBlocks * 8 bytes = 128 KB on every GPU that loads the
// library, from load until the process exits.
constexpr int kStaticPlanes = 64;
static __device__ __align__(256) double g_static_partial[kStaticPlanes * kPlaneBlocks];

namespace {
// Device address of g_static_partial on each device, resolved on first use.  In
// host code the symbol's name is only a handle for the runtime, not an address a
// kernel could dereference, hence the look-up.
double* g_static_partial_ptr[kMaxCudaDevices] = {};
}  // namespace

extern "C" hb_status hb_plane_sum_static(const float* values, int64_t plane_len, int32_t n_planes,
                                         double* out, void* stream) {
  if (plane_len < 0 || n_planes < 0 || (n_planes > 0 && (!values || !out))) {
    hb::set_error("hb_plane_sum_static: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (n_planes > kStaticPlanes) {
    hb::set_error("hb_plane_sum_static: %d planes requested, the built-in scratch holds %d "
                  "(use hb_plane_sum, or split the call)", n_planes, kStaticPlanes);
    return HB_ERR_TOO_LARGE;
  }
  if (n_planes == 0) return HB_OK;
  int dev = 0;
  HB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxCudaDevices) {
    hb::set_error("hb_plane_sum_static: device ordinal %d out of range", dev);
    return HB_ERR_UNSUPPORTED;
  }
  if (!g_static_partial_ptr[dev]) {
    // once per device, with that device current
    void* ptr = nullptr;
    HB_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_static_partial));
    g_static_partial_ptr[dev] = static_cast<double*>(ptr);
  }
  double* scratch = g_static_partial_ptr[dev];
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // Stage 1 writes every partial that stage 2 reads, so nothing in the scratch
  // has to start at zero; whatever the previous call left there is overwritten.
  plane_partial_kernel<<<dim3(n_planes, kPlaneBlocks), kSumThreads, 0, s>>>(values, plane_len, scratch);
  HB_CUDA_TRY(cudaGetLastError());
  plane_final_kernel<1><<<n_planes, kSumThreads, 0, s>>>(scratch, kPlaneBlocks, out);
  HB_CUDA_TRY(cudaGetLastError());
  return HB_OK;
}
