// Shared by the kernels for batches that do not fill the GPU (mlp_wide.cu, mlp_pairs.cu).
#pragma once

#include <atomic>

#include "mlp_common.cuh"
#include "mlp_wide.h"

namespace hb {

// Tensor maps of mlp_pairs.cu's activations: bytes per row, and rows of a K quarter (256 rows of NC columns; 40 and 48 in panels).
constexpr uint32_t act_map_row(int NC) { return NC == 40 || NC == 48 ? 256u : 2u * NC; }
constexpr uint32_t act_map_box(int NC) { return 512u * NC / act_map_row(NC); }
constexpr int kGroupCols = 128;    // columns of a group's fc2 sums

struct SmallParams {
  const float* bias;
  const float* fc2_w;
  float fc2_b;
  const double* mu;
  const double* sigma;
  const double* dev_feat;
  int32_t n_dev, n_op_feat, layers;
  const float* feats;
  const uint8_t* dev_row;
  int32_t Q;
  int32_t per_group;          // queries per group
  float* out;
  int32_t* status;
  uint8_t* acts;              // [groups][2 buffers][2 halves][1024 K rows][row bytes] (mlp_pairs.cu)
  unsigned long long* halves; // [groups][64 sets of 16 features][kGroupCols]: fc2 sum, tag
  int32_t* poison;            // [0] the mark of a launch that gave up (below zero: block ~mark of each group alone heeds it, in
                              // tests), [1] second runs of clusters (mlp_pairs.cu)
  uint32_t tag;               // of this launch
  uint32_t expect_stale;      // 0x80008000: every word of the first run is taken for stale (tests)
  int32_t stale_layer, stale_feature, stale_word;   // (checked build) the first run sends one word with the wrong signs: a layer's,
                              // -1: none; a feature's; 0 .. NC - 1 over both halves of the queries
  unsigned long long parity[2];   // bit g: parity of the next use of group g's buffer 0, 1 (mlp_pairs.cu)
  int32_t beside;             // runs beside the launch before it: nothing to wait for
  int64_t first;              // of feats and dev_row
  int32_t grid_n;             // > 0: query q is feature row q % grid_n on device grid_rows[q / grid_n]
  uint8_t grid_rows[hb::kMaxGridRows];
  int32_t inline_q;           // > 0: the queries themselves, below, instead of feats and dev_row
  float inline_feats[kWideInline * (kMaxInFeat - 4)];
  uint8_t inline_row[kWideInline];
  CUtensorMap map_slot;       // a ring slot of weight rows
  CUtensorMap map_fc1;        // one K block of the block's rows
  CUtensorMap map_acts;       // 256 rows of acts
};

inline __device__ bool concerns(int32_t mark, uint32_t block) {
  return mark > 0 || (mark < 0 && ~mark == static_cast<int32_t>(block));
}

// Launches `groups` clusters of `ctas` blocks; *fits = false (nothing launched) where the GPU cannot hold one.
template <typename Kernel>
cudaError_t launch_clusters(Kernel kernel, int ctas, int threads, int smem, const SmallParams& p, int groups, cudaStream_t stream,
                            bool* fits, std::atomic<int>& known) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(groups * ctas));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;   // for the occupancy question
  int n = known.load(std::memory_order_acquire);   // 1 + clusters the GPU runs at a time, 0: not asked yet
  if (n == 0) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess && ctas > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    int active = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&active, kernel, &cfg);
    if (e != cudaSuccess) return e;
    n = 1 + active;
    known.store(n, std::memory_order_release);
  }
  *fits = n > 1;
  cfg.numAttrs = overlapped_launch_enabled() ? 2 : 1;
  return *fits ? cudaLaunchKernelEx(&cfg, kernel, p) : cudaSuccess;
}
// mlp_pairs.cu: the shapes that it has, P pairs and NC columns per CTA, and a launch of one of them.
constexpr bool has_pairs_shape(int P, int NC) {
  return P == 8 ? NC == 16 || NC == 32 || NC == 40 || NC == 48 : (P == 4 ? NC == 32 || NC == 48 || NC == 64 : P == 2 && NC == 64);
}
cudaError_t launch_pairs(int P, int NC, bool split, const SmallParams& p, int groups, int device, cudaStream_t stream,
                         bool* fits);
constexpr int kMaxCudaDevices = 64;

}  // namespace hb

namespace {

using hb::kWideInline;
using hb::SmallParams;

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Gives up on behalf of the whole block.
__device__ __forceinline__ void give_up(volatile int* abort_flag, int32_t* status, int32_t* poison, int code) {
  *abort_flag = 1;
  *static_cast<volatile int32_t*>(status) = code;
  atomicExch(poison, 1);
}
template <int W>
__device__ __forceinline__ void tc_ld_cols(uint32_t taddr, float (&v)[W]) {
  static_assert(W == 8 || W == 16 || W == 32 || W == 40 || W == 48, "columns per load");
  if constexpr (W > 32) {
    float x[32], y[W - 32];
    tc_ld32(taddr, x);
    if constexpr (W == 40) tc_ld8(taddr + 32, y);
    else tc_ld16(taddr + 32, y);
#pragma unroll
    for (int i = 0; i < W; ++i) v[i] = i < 32 ? x[i % 32] : y[i % (W - 32)];
  } else if constexpr (W == 8) tc_ld8(taddr, v);
  else if constexpr (W == 16) tc_ld16(taddr, v);
  else tc_ld32(taddr, v);
}

// Normalised feature f of query `own` of the launch, as bf16 hi and lo parts.
__device__ __forceinline__ void load_feature(const SmallParams& p, int own, int f, __nv_bfloat16& hi, __nv_bfloat16& lo) {
  int64_t fr = p.first + own;
  int dr;
  if (p.grid_n) {
    const uint32_t block = static_cast<uint32_t>(fr) / static_cast<uint32_t>(p.grid_n);
    fr -= static_cast<int64_t>(block) * p.grid_n;
    dr = p.grid_rows[block];
  } else {
    dr = p.inline_q ? p.inline_row[own] : p.dev_row[fr];
  }
  dr = dr < p.n_dev ? dr : p.n_dev - 1;
  const double x = f < p.n_op_feat ? static_cast<double>(p.inline_q ? p.inline_feats[own * p.n_op_feat + f]
                                                                         : p.feats[fr * p.n_op_feat + f])
                                   : p.dev_feat[dr * 4 + (f - p.n_op_feat)];
  const float xn = static_cast<float>((x - p.mu[f]) / p.sigma[f]);
  hi = __float2bfloat16_rn(xn);
  lo = __float2bfloat16_rn(xn - __bfloat162float(hi));
}

// The 64 sets of 16 features of column `col` of a group, added in mlp_chain.cu's order: per CTA rank there, eight
// warps (two groups of four) of two 32-feature sets each, 512 features apart.  rank 0 or 1: one of the two summands of
// the prediction.
__device__ __forceinline__ float fc2_sum(const SmallParams& p, const unsigned long long* h, int rank, uint32_t tag,
                                         volatile int* abort_flag) {
  float tot = 0.0f;
  const long long t0 = clock64();
  float x[32];   // all asked for at once: two rounds of 16 took another 600 cycles
#pragma unroll 1
  for (uint32_t tries = 1;; ++tries) {
    bool all = true;
#pragma unroll
    for (int m = 0; m < 32; ++m) {
      const int kk = m >> 2;
      const int set = ((kk >> 2) * 256 + rank * 128 + (kk & 3) * 32) / 16 + ((m >> 1) & 1) * 32 + (m & 1);
      const unsigned long long v = ld_relaxed_u64(h + set * hb::kGroupCols);
      all = all && static_cast<uint32_t>(v >> 32) == tag;
      x[m] = __uint_as_float(static_cast<uint32_t>(v));
    }
    if (all) break;
    if ((tries & 63u) == 0u && (*abort_flag || clock64() - t0 > kWaitCycles)) {
      if (*abort_flag == 0) give_up(abort_flag, p.status, p.poison, 0x542);
      break;
    }
  }
#pragma unroll
  for (int m = 0; m < 32; m += 4) tot += (x[m] + x[m + 1]) + (x[m + 2] + x[m + 3]);
  return tot;
}

}  // namespace
