// MLP inference for batches that do not fill the GPU: the layers' features are spread over the SMs.
//
// mlp_chain.cu gives 128 queries to two SMs, which stream all 16.8 MB of weights past them: 103 to 110 us
// whether the batch has one query or 9,472.  What bounds that is the weight stream of one SM pair, so
// here G = 16, 8 or 4 thread blocks form a group that owns up to 64 queries (32 in split precision);
// block c computes output features 1024 / G * c .. of every layer for all of the group's queries and
// streams only their weights.  Between layers a group's blocks exchange their activations through
// global memory (L2): an all-gather of 2 KB per query.  Groups of few queries use distributed shared memory
// instead (NEAR, see there).
//
// Formulation as in mlp_chain.cu, H^T = W . X^T with tcgen05.mma (cta_group::1): A = weight rows
// (M = 64 with 16 blocks, else 128), B = activations (MN-major, W = 16, 32 or 64 columns, swizzle width
// 2 W bytes, so that narrow batches move less), D = fp32 in TMEM.  K is walked in the same order and
// fc2 adds in the same order as there, so both kernels give the same bits and the choice of kernel
// never shows in a result.
//
// Exchange.  There are no flags and no fences on the way: an activation is never negative, so the sign
// bit of every 32-bit word a block writes (two bf16 activations, or one fp32 activation in split
// precision) carries the parity of the buffer's use, and a reader polls the data itself until all its
// words show the expected parity.  A release fence took 1,000 cycles, and 6,000 while other groups
// streamed weights.  Reading a word of an earlier use with the same parity is impossible: the same
// block has read the use in between (coherence of one location).  Two buffers alternate by layer: a
// block writes layer L only after it has read all of layer L - 1, which every block wrote after reading
// L - 2.  The host keeps the parity each group's buffers have reached.
//
// The blocks of a group are one thread-block cluster, which the hardware schedules as a whole: that is
// what makes waiting for one another safe, and a launch may have more groups than fit at a time.
//
// Weights arrive through a ring of 32 KB slots, 3 to 6 of them; they do not depend on the activations,
// so the ring is full again when an exchange ends.
//
// Warp roles: 0 MMA issuer (and TMEM), 1 weight producer, 2 the mark, 4-7 epilogue (one TMEM lane quadrant each),
// 8-15 (64 columns: 8-23, NEAR: none) receivers.  Every wait is bounded, as in mlp_chain.cu; a launch that gave up
// leaves a mark in the scratch, and launches that find it report an error instead of a result.
//
// After giving up no ring slot may be requested again that nobody has waited for: its copy could still be under way,
// and its barrier would be armed a second time in one phase.  So the MMA issuer, whose commits free the slots, waits
// for the producer to leave before it issues anything past a wait that ran out, and goes no further than the layer's end.
#include <atomic>
#include <cstring>

#include "mlp_common.cuh"
#include "mlp_wide.h"

namespace {

using hb::kWideInline;

struct WideParams {
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
  uint8_t* acts;              // [groups][2][1024 K rows][2 W bytes]
  unsigned long long* halves; // [groups][64 sets of 16 features][kWideCols]: fc2 sum, tag
  int32_t* poison;            // set by a launch that gave up
  uint32_t tag;               // of this launch
  unsigned long long parity[2];   // bit g: parity of the next use of group g's buffer 0, 1
  int32_t beside;             // runs beside the launch before it: nothing to wait for
  int64_t first;              // of feats and dev_row
  int32_t grid_n;             // > 0: query q is feature row q % grid_n on device grid_rows[q / grid_n]
  uint8_t grid_rows[hb::kMaxGridRows];
  int32_t inline_q;           // > 0: the queries themselves, below, instead of feats and dev_row
  float inline_feats[kWideInline * (kMaxInFeat - 4)];
  uint8_t inline_row[kWideInline];
  CUtensorMap map_slot;       // 32 KB of weight rows: a ring slot
  CUtensorMap map_fc1;        // one K block of the block's rows
};

// Receiver warps: enough that 64 columns, too, need only four 16-byte loads per thread and K quarter.
template <int W>
constexpr int wide_receivers() { return W == 64 ? 16 : 8; }
template <int W, bool NEAR>
constexpr int wide_threads() { return 256 + (NEAR ? 0 : 32 * wide_receivers<W>()); }
constexpr int kWideSlotBytes = 2 * kTileBytes;
constexpr int kWideCols = 64;    // queries per group at most

template <int W, bool NEAR>
constexpr int wide_slots() { return W == 64 ? 3 : (W == 32 || NEAR ? 5 : 6); }
template <int W, bool NEAR>
constexpr int wide_act_bytes() { return (NEAR ? 2 : 1) * 2048 * W; }
template <int W, bool NEAR>
constexpr int wide_smem() { return wide_act_bytes<W, NEAR>() + wide_slots<W, NEAR>() * kWideSlotBytes + 1024 + 512; }
static_assert(wide_smem<64, false>() <= 232448 && wide_smem<32, false>() <= 232448 &&
              wide_smem<16, false>() <= 232448 && wide_smem<16, true>() <= 232448, "shared memory");

__device__ __forceinline__ uint4 ld_relaxed_v4(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_v4(void* p, uint4 v) {
  asm volatile("st.relaxed.gpu.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
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
// mbar_wait that also leaves the mark in the scratch.
__device__ __forceinline__ bool wide_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, const WideParams& p,
                                          int code) {
  if (mbar_wait(bar, parity, abort_flag, p.status, code)) return true;
  atomicExch(p.poison, 1);
  return false;
}
// wide_wait for a whole warp: one lane polls, and every lane gets the same answer, so that the
// warp-wide instructions after it are reached together or not at all.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int lane, volatile int* abort_flag,
                                          const WideParams& p, int code) {
  bool ok = true;
  if (lane == 0) ok = wide_wait(bar, parity, abort_flag, p, code);
  __syncwarp();
  return __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int32_t row, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row)
      : "memory");
}
__device__ __forceinline__ void tma_3d(uint32_t dst, const CUtensorMap* map, int32_t row, int32_t image, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row), "r"(image)
      : "memory");
}
__device__ __forceinline__ void mma_one_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void commit_one(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <int W>
__device__ __forceinline__ void tc_ld_cols(uint32_t taddr, float (&v)[W]) {
  static_assert(W == 8 || W == 16 || W == 32, "columns per load");
  if constexpr (W == 8) tc_ld8(taddr, v);
  else if constexpr (W == 16) tc_ld16(taddr, v);
  else tc_ld32(taddr, v);
}
// Byte offset of 16-byte chunk `chunk` of K row k in a B operand of W columns (swizzle width 2 W bytes).
template <int W>
__device__ __forceinline__ uint32_t b_chunk(uint32_t k, uint32_t chunk) {
  const uint32_t x = W == 64 ? (k & 7u) : (W == 32 ? ((k >> 1) & 3u) : ((k >> 2) & 1u));
  return k * (2u * W) + ((chunk ^ x) << 4);
}

// NEAR: groups of up to six queries (split: three) exchange through distributed shared memory instead.  B is K-major,
// so that a block's share of a query is 128 contiguous bytes, which eight threads store into each of the other
// blocks (st.async, counted in bytes on the barrier of the buffer); two buffers alternate by layer, for the reason
// given above.  An all-gather of 128 bytes per block takes 750 cycles, of 1 KB 1,500, of 2 KB 2,400 (about 14 bytes
// a cycle), while the way through L2 moves whole rows of columns, filled or not: 1,140 cycles to the first K quarter and
// 600 to each further one.  At first one query 23.6 -> 19.1 us, 14: 23.6 -> 20.5, 42: 23.9 -> 23.8, 56: 24.0 -> 25.5
// (not taken); split, one 33.1 -> 28.9, 14: 33.4 -> 31.0, 28: 33.9 either way (not taken).  Now 18.9, 20.2 and 23.3, split
// 28.8 and 30.6.
template <int G, int W, bool SPLIT, bool NEAR>
__global__ void __launch_bounds__(wide_threads<W, NEAR>(), 1) mlp_wide_kernel(const __grid_constant__ WideParams p) {
  static_assert(!NEAR || (G == 16 && W == 16), "one K block of 64 features per block");
  constexpr int kM = G == 16 ? 64 : 128;              // weight rows per MMA
  constexpr int kBlocks = kWidth / G / kM;            // row blocks per thread block
  constexpr int kCols = SPLIT || NEAR ? W / 2 : W;    // queries a group can hold
  constexpr int kSlots = wide_slots<W, NEAR>();
  constexpr int kReceivers = wide_receivers<W>();
  constexpr int kParts = SPLIT ? 2 : 1;               // images per packed K block
  constexpr int kUnitBytes = kM * 128;                // one K block of the rows
  constexpr int kUnitsPerSlot = kWideSlotBytes / kUnitBytes;
  constexpr int kSlotsPerBlock = kNumKB * kParts / kUnitsPerSlot;
  constexpr uint32_t kQuarterBytes = 256u * 2u * W;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t act = base;
  const uint32_t ring = base + wide_act_bytes<W, NEAR>();
  const uint32_t bars = ring + kSlots * kWideSlotBytes;
  uint8_t* bars_ptr = base_ptr + (bars - base);
  const uint32_t bar_full = bars, bar_empty = bars + 64;      // [kSlots]
  const uint32_t bar_act = bars + 128;                        // [4] K quarter in place; NEAR: [2] buffer in place
  const uint32_t bar_acc = bars + 160;                        // [kBlocks] row block accumulated
  const uint32_t bar_tfree = bars + 192;                      // TMEM read out (4 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_ptr + 200);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars_ptr + 204);
  volatile int* mark_seen = reinterpret_cast<volatile int*>(bars_ptr + 208);
  volatile int* producer_left = reinterpret_cast<volatile int*>(bars_ptr + 212);
  const uint32_t bar_drain = bars + 216;                      // after giving up: the MMAs have ended

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = static_cast<int>(blockIdx.x) / G, c = static_cast<int>(blockIdx.x) % G;   // group = cluster

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int q = 0; q < 4; ++q) mbar_init(bar_act + 8 * q, NEAR ? 1 : kReceivers);
    for (int b = 0; b < kBlocks; ++b) mbar_init(bar_acc + 8 * b, 1);
    mbar_init(bar_tfree, 4);
    mbar_init(bar_drain, 1);
    *abort_flag = 0;
    *mark_seen = 0;
    *producer_left = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // (before the peers' first stores)
  if (NEAR) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  constexpr uint32_t kTmemCols = kBlocks * W < 32 ? 32 : kBlocks * W;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  grid_begin(p.beside != 0);
  if (NEAR) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int n_layers = p.layers + 1;
  uint32_t issued = 0;
  uint8_t* const group_acts = p.acts + static_cast<size_t>(group) * (2u * 2048u * W);
  unsigned long long* const group_halves = p.halves + static_cast<size_t>(group) * 64 * kWideCols;
  // sign bit of the words of the `use`-th exchange of this launch
  auto sign_of = [&](int use) -> uint32_t {
    return static_cast<uint32_t>(((p.parity[use & 1] >> group) + static_cast<unsigned>(use >> 1)) & 1ull) << 31;
  };

  const int64_t q0 = static_cast<int64_t>(group) * p.per_group;
  const int n_q = static_cast<int>(min(static_cast<int64_t>(p.per_group), static_cast<int64_t>(p.Q) - q0));
  // fc1's B operand: K rows 0..63 hold [hi | lo | hi] of the normalised features, one query per column.  Epilogue
  // and receivers, who have nothing else to do yet, share the work: a value takes two dependent loads and a float64
  // division, 1,100 cycles, and the epilogue's 128 threads alone took three rounds with 32 queries, six with 64
  // (100 queries 25.1 -> 24.3 us, 900 48.2 -> 46.5, 2,000 75.1 -> 74.1).  A function that both roles call: as a step
  // before the roles part it made every layer 30 % slower.  In split precision, with half the queries, it gained
  // nothing and cost 1 to 2 % from 150 queries on: epilogue alone.
  // So too in four blocks of 32 columns, which batches that fill the GPU side by side take: shared, the features made 480,
  // 480 and 6 queries 58.9 -> 61.0 us and an iteration batch with 636, 384 and 12 66.0 -> 68.0 (those three alone 50.0 ->
  // 49.8), 960 beside 96, 1,000 beside 12 and 800 beside 200 the same within 0.2, 961 to 1,056 alone 47.9 -> 47.7.
  constexpr bool kAllFeatures = !SPLIT && !NEAR && !(G == 4 && W == 32);
  auto features = [&]() {
    constexpr int kThreads = kAllFeatures ? wide_threads<W, NEAR>() - 128 : 128;
    auto feat_sync = [] { asm volatile("bar.sync 2, %0;" ::"n"(kThreads) : "memory"); };
    const int T = static_cast<int>(threadIdx.x) - 128;
    const int C_in = p.n_op_feat + 4;
    for (int i = T; i < 64 * 2 * W / 16; i += kThreads) *reinterpret_cast<uint4*>(base_ptr + 16 * i) = make_uint4(0, 0, 0, 0);
    feat_sync();
    for (int i = T; i < n_q * C_in; i += kThreads) {
      const int q = i / C_in, f = i - q * C_in;
      const int own = static_cast<int>(q0) + q;                 // of the launch's queries
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
      const __nv_bfloat16 hi = __float2bfloat16_rn(xn);
      const __nv_bfloat16 lo = __float2bfloat16_rn(xn - __bfloat162float(hi));
      const uint32_t ch = static_cast<uint32_t>(q) >> 3, in = 2u * (static_cast<uint32_t>(q) & 7u);
      auto at = [&](int k) { return NEAR ? swz_off(q, k) : b_chunk<W>(k, ch) + in; };
      *reinterpret_cast<__nv_bfloat16*>(base_ptr + at(f)) = hi;
      *reinterpret_cast<__nv_bfloat16*>(base_ptr + at(C_in + f)) = lo;
      *reinterpret_cast<__nv_bfloat16*>(base_ptr + at(2 * C_in + f)) = hi;
    }
    fence_proxy_async();
    feat_sync();
    if (T < (NEAR ? 1 : kReceivers)) mbar_arrive(bar_act);
    __syncwarp();
  };

  if (warp == 2) {
    // An earlier launch that gave up left the buffers in an unknown state: report, and give up as well (no result is
    // stored then).  Only that result waits for the mark, whose load takes 700 cycles.
    if (lane == 0) {
      if (*reinterpret_cast<volatile int32_t*>(p.poison) != 0) {
        *static_cast<volatile int32_t*>(p.status) = 0x5FF;
        *abort_flag = 1;
      }
      __threadfence_block();
      *mark_seen = 1;
    }
  } else if (warp == 1) {
    // ------------------------------ weight producer ------------------------------
    if (lane == 0) {
      uint32_t s = 0, ph = 0;
      bool ok = true;
      for (int L = 0; L < n_layers && ok; ++L) {
        for (int b = 0; b < kBlocks && ok; ++b) {
          const int row0 = (c * kBlocks + b) * kM;              // first output feature
          const int mt = row0 / kMTile;
          const int image0 = kParts * (L == 0 ? mt : kNumMT + ((L - 1) * kNumMT + mt) * kNumKB);
          const int n = L == 0 ? 1 : kSlotsPerBlock;
          for (int g = 0; g < n; ++g) {
            const uint32_t full = bar_full + 8 * s;
            if (!wide_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, p, 0x511)) { ok = false; break; }
            mbar_expect_tx(full, L == 0 ? kUnitBytes : kWideSlotBytes);
            const CUtensorMap* map = L == 0 ? &p.map_fc1 : &p.map_slot;
            const int image = image0 + g * kUnitsPerSlot;
            if (G == 16) tma_3d(ring + s * kWideSlotBytes, map, row0 % kMTile, image, full);
            else tma_2d(ring + s * kWideSlotBytes, map, image * kMTile, full);
            ++issued;
            ring_next<kSlots>(s, ph);
          }
        }
      }
      *producer_left = 1;
    }
  } else if (warp == 0) {
    // ------------------------------ MMA issuer ------------------------------
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (NEAR ? 0u : 1u << 16) |
                               (static_cast<uint32_t>(W >> 3) << 17) | (static_cast<uint32_t>(kM >> 4) << 24);
    // A: K-major, 128-byte swizzle, 8-row groups 1024 B apart; B: MN-major, one swizzle atom wide, 8-row
    // groups of K 16 W bytes apart; NEAR: K-major like A, 16 rows (queries) of 128 bytes per K block
    const uint64_t desc_a = (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                            (static_cast<uint64_t>(2) << 61) | (static_cast<uint64_t>(1) << 16);
    const uint64_t desc_b = NEAR ? desc_a
                                 : (static_cast<uint64_t>((16 * W) >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                                       (static_cast<uint64_t>(W == 64 ? 2 : (W == 32 ? 4 : 6)) << 61) |
                                       (static_cast<uint64_t>(1) << 16);
    // in 16-byte units: 16 K values of B, a K block of 64
    constexpr uint32_t kStepB = NEAR ? 2 : (32 * W) >> 4, kBlockB = (128 * W) >> 4;
    const uint32_t a_lo0 = (ring & 0x3FFFF) >> 4, b_lo0 = (act & 0x3FFFF) >> 4;
    // One elected lane runs the whole loop.  An MMA of these shapes takes 24 to 49 cycles and only a
    // couple of them queue up, so what stands between two MMAs shows: the wait for the next slot goes
    // between the MMAs of the current one, the commit that frees a slot behind the next slot's first
    // MMAs, and every loop of a layer runs its full count whatever the waits say, so that the descriptors depend
    // on uniform values alone (a wait that ran out has set the abort flag; what is issued after it reads
    // stale shared memory and is discarded).  16 MMAs of 64 x 16 took 1,150 cycles in the plain form.
    if (elect_one()) {
      auto gave_up = [&] {   // (the producer looks at the abort flag when a slot does not come)
        for (const long long t0 = clock64(); *producer_left == 0 && clock64() - t0 <= kWaitCycles;) {}
      };
      auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        if (!mbar_try_wait(bar, parity) && (*abort_flag || !wide_wait(bar, parity, abort_flag, p, code))) gave_up();
        tc_fence_after();
      };
      // layer L's input: its first K quarter (which has one phase more than the others, fc1's input); NEAR: the whole
      // of buffer L & 1, written by the peers
      auto wait_input = [&](int L) {
        if (!NEAR) {
          wait(bar_act, L & 1, 0x521);
          return;
        }
        if (!mbar_wait_cluster(bar_act + 8 * (L & 1), (L >> 1) & 1, abort_flag, p.status, 0x521)) {
          atomicExch(p.poison, 1);
          gave_up();
        }
        fence_proxy_async();
        tc_fence_after();
      };
      uint32_t s = 0, ph = 0;
      for (int b = 0; b < kBlocks; ++b) {                        // fc1: one K block
        if (b == 0) wait_input(0);
        wait(bar_full + 8 * s, ph, 0x522);
        const uint32_t d = tmem_base + static_cast<uint32_t>(b * W);
        const uint32_t a_lo = a_lo0 + s * (kWideSlotBytes >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_one_bf16(d, desc_a | (a_lo + 2 * k), desc_b | (b_lo0 + k * kStepB), idesc, k ? 1u : 0u);
        commit_one(bar_acc + 8 * b);
        commit_one(bar_empty + 8 * s);
        ring_next<kSlots>(s, ph);
      }
      constexpr int kMmas = 4 * kUnitsPerSlot;                   // per slot
      constexpr int kPerQuarter = kSlotsPerBlock / 4;            // slots; none spans two K quarters
#pragma unroll 1
      for (int L = 1; L < n_layers && *abort_flag == 0; ++L) {
        wait(bar_tfree, (L - 1) & 1, 0x523);
#pragma unroll 1
        for (int b = 0; b < kBlocks; ++b) {
          const uint32_t d = tmem_base + static_cast<uint32_t>(b * W);
          wait(bar_full + 8 * s, ph, 0x522);
          if (b == 0) wait_input(L);
          uint32_t prev = 0;
#pragma unroll 1
          for (int g = 0; g < kSlotsPerBlock; ++g) {
            uint32_t next = s, next_ph = ph;
            ring_next<kSlots>(next, next_ph);
            const uint32_t a_lo = a_lo0 + s * (kWideSlotBytes >> 4);
            const uint32_t b_lo = b_lo0 + (NEAR ? static_cast<uint32_t>(L & 1) * (kNumKB * kBlockB) : 0u) +
                                  static_cast<uint32_t>(g) * (kBlockB * kUnitsPerSlot / kParts);
#pragma unroll
            for (int u = 0; u < kMmas; ++u) {
              mma_one_bf16(d, desc_a | (a_lo + (u >> 2) * (kUnitBytes >> 4) + 2 * (u & 3)),
                           desc_b | (b_lo + (u >> 2) / kParts * kBlockB + (u & 3) * kStepB), idesc,
                           u == 0 ? static_cast<uint32_t>(g) : 1u);
              if (u == 1 && g > 0) commit_one(bar_empty + 8 * prev);
              if (u == kMmas / 2 && g + 1 < kSlotsPerBlock) {
                wait(bar_full + 8 * next, next_ph, 0x522);
                if (!NEAR && b == 0 && (g + 1) % kPerQuarter == 0)
                  wait(bar_act + 8 * ((g + 1) / kPerQuarter), (L - 1) & 1, 0x521);
              }
            }
            prev = s;
            s = next;
            ph = next_ph;
          }
          commit_one(bar_acc + 8 * b);
          commit_one(bar_empty + 8 * prev);
        }
      }
    }
    __syncwarp();
  } else if (warp >= 8) {
    // ------------------------------ receivers ------------------------------
    // A unit is what ends as 16 bytes of B (bf16) or as a hi and a lo chunk (split, from 32 bytes of fp32).
    // Every warp takes a share of each K quarter, in order, so that the tensor core starts on the first one
    // while the others arrive.  Only what is missing is asked for again, and no quarter before the one ahead of
    // it is complete: the exchange is bound by the rate of these loads (all four quarters in flight at once:
    // 39.0 us for 371 queries; one ahead: 36.4; none: 33.2).
    const int t = static_cast<int>(threadIdx.x) - 256;
    constexpr int kLoads = SPLIT ? 2 : 1;
    constexpr int kUnits = static_cast<int>(kQuarterBytes) / (16 * kLoads) / (32 * kReceivers);   // per thread
    static_assert(kUnits >= 1, "a unit per thread and quarter");
    if (kAllFeatures) features();
    for (int L = 1; L < n_layers; ++L) {
      // the tensor core has read the previous layer's input
      if (!warp_wait(bar_acc + 8 * (kBlocks - 1), (L - 1) & 1, lane, abort_flag, p, 0x531)) break;
      const uint32_t sign = sign_of(L - 1);
      const uint8_t* src = group_acts + ((L - 1) & 1) * (2048u * W) + 16 * kLoads * t;
      constexpr int N = kUnits * kLoads;
      auto addr = [&](int q, int i) {
        return src + q * kQuarterBytes + ((i / kLoads) * 32 * kReceivers * kLoads + i % kLoads) * 16;
      };
      bool ok = true;
      const long long t0 = clock64();
      if (W == 32) {
        // What is asked for before the others can have written it only delays what they write.  The two shapes of 32
        // columns gain (without and with, us: 300 queries 32.9 / 32.1, 480 32.6 / 32.2, 1,056 48.6 / 48.0; split, 150
        // 48.0 / 46.4, 500 77.9 / 77.2; 200 cycles gain less, 500 about as much).  With 16 columns the values come
        // sooner (one query 23.3 / 23.7), with 64 later than any pause (960 48.0 / 48.0).
        while (clock64() - t0 < 350) {}
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 x[N];
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = ld_relaxed_v4(addr(q, i));
#pragma unroll 1
        for (uint32_t tries = 1; ok; ++tries) {
          uint32_t bad = 0;
#pragma unroll
          for (int i = 0; i < N; ++i)
            bad |= (x[i].x ^ sign) | (x[i].y ^ sign) | (x[i].z ^ sign) | (x[i].w ^ sign);
          if ((bad >> 31) == 0u) break;
          if ((tries & 63u) == 0u && (*abort_flag || clock64() - t0 > kWaitCycles)) {
            if (*abort_flag == 0) give_up(abort_flag, p.status, p.poison, 0x532);
            ok = false;
          }
#pragma unroll
          for (int i = 0; i < N; ++i)
            if (((x[i].x ^ sign) | (x[i].y ^ sign) | (x[i].z ^ sign) | (x[i].w ^ sign)) >> 31)
              x[i] = ld_relaxed_v4(addr(q, i));
        }
#pragma unroll
        for (int i = 0; i < kUnits; ++i) {
          const uint32_t unit = static_cast<uint32_t>(i * 32 * kReceivers + t);
          uint4 a = x[i * kLoads];
          a.x &= 0x7FFFFFFFu; a.y &= 0x7FFFFFFFu; a.z &= 0x7FFFFFFFu; a.w &= 0x7FFFFFFFu;
          if (!SPLIT) {
            *reinterpret_cast<uint4*>(base_ptr + q * kQuarterBytes + 16 * unit) = a;   // already in the image's order
          } else {
            uint4 b = x[i * kLoads + kLoads - 1];
            b.x &= 0x7FFFFFFFu; b.y &= 0x7FFFFFFFu; b.z &= 0x7FFFFFFFu; b.w &= 0x7FFFFFFFu;
            constexpr uint32_t kPerRow = W / 16;
            const uint32_t k = q * 256 + unit / kPerRow, ch = unit % kPerRow;
            const float f8[8] = {__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w),
                                 __uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w)};
            uint32_t hi4[4], lo4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(f8[2 * j], f8[2 * j + 1]);
              const __nv_bfloat162 l = __floats2bfloat162_rn(f8[2 * j] - __low2float(h), f8[2 * j + 1] - __high2float(h));
              hi4[j] = *reinterpret_cast<const uint32_t*>(&h);
              lo4[j] = *reinterpret_cast<const uint32_t*>(&l);
            }
            *reinterpret_cast<uint4*>(base_ptr + b_chunk<W>(k, ch)) = make_uint4(hi4[0], hi4[1], hi4[2], hi4[3]);
            *reinterpret_cast<uint4*>(base_ptr + b_chunk<W>(k, ch + kPerRow)) = make_uint4(lo4[0], lo4[1], lo4[2], lo4[3]);
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(bar_act + 8 * q);
      }
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
    }
  } else if (warp >= 4) {
    // ------------------------------ epilogue ------------------------------
    const int quad = warp & 3;
    const int T = static_cast<int>(threadIdx.x) - 128;          // 0..127
    auto epi_sync = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    features();
    // M = 64 leaves 16 rows in the low lanes of every quadrant, M = 128 all 32
    const bool row_ok = kM == 128 || lane < 16;
    const int row = kM == 128 ? quad * 32 + lane : quad * 16 + (lane & 15);
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    bool ok = true;
    // a wait that ran out skips the work that is left but none of the block-wide barriers
    for (int L = 0; L < n_layers; ++L) {
      const bool last = L == n_layers - 1;
      uint8_t* dst = group_acts + (L & 1) * (2048u * W);
      const uint32_t sign = sign_of(L);
#pragma unroll 1
      for (int b = 0; b < kBlocks; ++b) {
        const int f = (c * kBlocks + b) * kM + row;
        const float bias = __ldg(p.bias + L * kWidth + f);
        const float w2 = last ? __ldg(p.fc2_w + f) : 0.0f;
        ok = ok && warp_wait(bar_acc + 8 * b, L & 1, lane, abort_flag, p, 0x541);
        if (!ok) {
          if (NEAR && !last) epi_sync();
          break;
        }
        tc_fence_after();
        // up to 32 columns at a time (split: 16 queries, their hi and their lo column)
        constexpr int kPiece = kCols < 16 ? 8 : (SPLIT || W < 32 ? 16 : 32);
        const uint32_t t_block = t_lane + static_cast<uint32_t>(b * W);
#pragma unroll 1
        for (int q1 = 0; q1 < kCols; q1 += kPiece) {
          float v[kPiece];
          if (SPLIT) {
            float lo[kPiece];
            tc_ld_cols<kPiece>(t_block + q1, v);
            tc_ld_cols<kPiece>(t_block + W / 2 + q1, lo);
#pragma unroll
            for (int i = 0; i < kPiece; ++i) v[i] += lo[i];
          } else {
            tc_ld_cols<kPiece>(t_block + q1, v);
          }
          if (b == kBlocks - 1 && q1 + kPiece == kCols) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_tfree);
          }
#pragma unroll
          for (int i = 0; i < kPiece; ++i) v[i] = fmaxf(v[i] + bias, 0.0f);
          if (NEAR && !last) {
            // own features first, then the group's other blocks: 128 bytes of every query
            const uint32_t mine = static_cast<uint32_t>((L + 1) & 1) * (2048u * W) + static_cast<uint32_t>(c) * (128u * W);
            const uint32_t in_bar = bar_act + 8 * ((L + 1) & 1);
#pragma unroll
            for (int q = 0; q < kPiece; ++q) {
              if (!row_ok || q >= n_q) continue;
              const __nv_bfloat16 hi = __float2bfloat16_rn(v[q]);
              *reinterpret_cast<__nv_bfloat16*>(base_ptr + mine + swz_off(q, row)) = hi;
              if (SPLIT)
                *reinterpret_cast<__nv_bfloat16*>(base_ptr + mine + swz_off(W / 2 + q, row)) =
                    __float2bfloat16_rn(v[q] - __bfloat162float(hi));
            }
            fence_proxy_async();
            epi_sync();
            // (after giving up the buffer's last phase may be incomplete: it is not armed again)
            if (T == 0 && *abort_flag == 0) mbar_expect_tx(in_bar, static_cast<uint32_t>((G - 1) * kParts * 128 * n_q));
            const uint32_t chunk = static_cast<uint32_t>(T) & 7u, to = static_cast<uint32_t>(c + (T >> 3)) % G;
            if (T >= 8) {   // eight threads per peer, 16 bytes of each query
              const uint32_t there = map_to_cta(base + mine, to), bar = map_to_cta(in_bar, to);
              for (uint32_t q = 0; q < static_cast<uint32_t>(n_q); ++q)
#pragma unroll
                for (uint32_t part = 0; part < kParts; ++part) {
                  const uint32_t at = (part * (W / 2) + q) * 128u + (((chunk ^ q) & 7u) << 4);
                  const uint4 x = *reinterpret_cast<const uint4*>(base_ptr + mine + at);
                  st_async_v4(there + at, x.x, x.y, x.z, x.w, bar);
                }
            }
            __syncwarp();
          } else if (!last) {
            constexpr int kWords = SPLIT ? kPiece : kPiece / 2;
            uint32_t w[kWords];
#pragma unroll
            for (int i = 0; i < kWords; ++i) {
              if (SPLIT) {
                w[i] = __float_as_uint(v[i]);
              } else {
                const __nv_bfloat162 pk = __floats2bfloat162_rn(v[(2 * i) % kPiece], v[(2 * i + 1) % kPiece]);
                w[i] = *reinterpret_cast<const uint32_t*>(&pk);
              }
              w[i] = (w[i] & 0x7FFFFFFFu) | sign;
            }
            // N lanes with N chunks of 16 bytes of their own row each trade chunks, so that every store writes
            // N chunks in a row of one row: whole sectors instead of halves.
            constexpr int N = kWords / 4;
            trade_chunks<N>(w, lane);
            if (row_ok) {
              const uint32_t ch = static_cast<uint32_t>(SPLIT ? q1 / 4 : q1 / 8) + static_cast<uint32_t>(lane % N);
#pragma unroll
              for (int g = 0; g < N; ++g) {
                const uint32_t k = static_cast<uint32_t>(f - lane % N + g);
                st_relaxed_v4(dst + (SPLIT ? k * (2u * W) + 16u * ch : b_chunk<W>(k, ch)),
                              make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]));
              }
            }
          } else {
            constexpr int kFold = kPiece < 16 ? 16 : kPiece;
            float s[kFold];
#pragma unroll
            for (int i = 0; i < kFold; ++i) s[i] = i < kPiece ? __fmul_rn(w2, v[i % kPiece]) : 0.0f;
            fold16(s, lane);
            if (row_ok) {
              const int half = ((c * kBlocks + b) * kM + quad * (kM / 4) + (lane & 16)) / 16;
              unsigned long long* h = group_halves + half * kWideCols + q1 + fold16_col<kFold>(lane);
#pragma unroll
              for (int i = 0; i < kFold / 16; ++i)
                st_relaxed_u64(h + i, static_cast<unsigned long long>(p.tag) << 32 | __float_as_uint(s[i]));
            }
          }
        }
      }
    }
    if (c == 0) {
      // the first block of the group adds the 64 sets of 16 features of every query, in mlp_chain.cu's order:
      // per CTA rank there, eight warps (two groups of four) of two 32-feature sets each, 512 features apart
      const int q = T & 63, rank = T >> 6;
      const unsigned long long* h = group_halves + q;
      float tot = 0.0f;
      if (q < n_q && ok) {
        const long long t0 = clock64();
#pragma unroll 1
        for (int k = 0; k < 8; k += 4) {
          float x[16];
#pragma unroll 1
          for (uint32_t tries = 1;; ++tries) {
            bool all = true;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
              const int kk = k + (m >> 2);
              const int set = ((kk >> 2) * 256 + rank * 128 + (kk & 3) * 32) / 16 + ((m >> 1) & 1) * 32 + (m & 1);
              const unsigned long long v = ld_relaxed_u64(h + set * kWideCols);
              all = all && static_cast<uint32_t>(v >> 32) == p.tag;
              x[m] = __uint_as_float(static_cast<uint32_t>(v));
            }
            if (all) break;
            if ((tries & 63u) == 0u && (*abort_flag || clock64() - t0 > kWaitCycles)) {
              if (*abort_flag == 0) give_up(abort_flag, p.status, p.poison, 0x542);
              break;
            }
          }
#pragma unroll
          for (int m = 0; m < 16; m += 4) tot += (x[m] + x[m + 1]) + (x[m + 2] + x[m + 3]);
        }
      }
      float* tots = reinterpret_cast<float*>(base_ptr);        // the tensor core is done with the activations
      tots[T] = tot;
      epi_sync();
      // (the mark is long there)
      for (const long long t0 = clock64(); *mark_seen == 0 && clock64() - t0 <= kWaitCycles;) {}
      if (T < n_q && *mark_seen != 0 && *abort_flag == 0) p.out[q0 + T] = tots[T] + tots[64 + T] + p.fc2_b;
    }
  }

  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && warp == 1 && lane == 0) {
    // weight copies in flight must land before the shared memory goes away (bounded)
    const long long t0 = clock64();
    for (uint32_t i = issued > kSlots ? issued - kSlots : 0; i < issued; ++i)
      while (!mbar_try_wait(bar_full + 8 * (i % kSlots), (i / kSlots) & 1u) && clock64() - t0 <= kWaitCycles) {}
  }
  if (*abort_flag && warp == 0 && elect_one()) {
    // and the MMAs, before the TMEM they write is somebody else's (the lane that issued them)
    commit_one(bar_drain);
    const long long t0 = clock64();
    while (!mbar_try_wait(bar_drain, 0) && clock64() - t0 <= kWaitCycles) {}
  }
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (NEAR && *abort_flag) {
    // A block that has everything it waited for has been sent all that will be.  One that gave up may still be
    // written to: it stays until the others have left or given up as well (their waits are bounded), and a
    // little longer for what is on its way.
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {}
  }
  grid_end(p.beside != 0);
}
}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {
constexpr int kMaxCudaDevices = 64;
// Scratch per stream: launches on one stream follow one another, so they can share it (those of one call
// that run side by side have a lane each).  It is kept between launches and freed with the GPU's last predictor.
// The first kMaxStreams streams and lanes keep theirs.  Later ones (a program with a stream per request) share
// kMoreStreams: each launch of theirs is followed by an event, and a new stream takes over what has been out of
// use for longest.  The events keep a launch from overlapping the end of the one before it, which is why
// the first streams go without.  While none of the shared ones is out of use, a launch takes the two-SM kernel,
// which needs no scratch.
constexpr int kMaxStreams = 16, kMoreStreams = 16;
constexpr int kMaxGroups = 37;
constexpr int kWidths = 3;        // W = 16, 32, 64 have their own buffers: a word's parity counts its own uses
constexpr size_t kActsBytes = static_cast<size_t>(kMaxGroups) * 2 * 2048 * (16 + 32 + 64);
constexpr size_t kHalvesBytes = static_cast<size_t>(kMaxGroups) * 64 * kWideCols * sizeof(unsigned long long);
constexpr size_t kScratchBytes = kActsBytes + kHalvesBytes + 256;   // and the mark of a launch that gave up
struct StreamScratch {
  unsigned long long stream_id = 0;
  int lane = 0;
  uint8_t* base = nullptr;
  bool fresh = false;                            // buffers and parities start over at the next launch
  uint32_t tag = 0;
  unsigned long long parity[kWidths][2] = {};    // bit g: parity of the next use of group g's buffers
  cudaEvent_t done = nullptr;                    // shared ones: behind the last launch
  uint64_t last_use = 0;
};
struct GpuScratch {
  std::mutex mu;
  int handles = 0;
  int used = 0;
  uint64_t uses = 0;
  StreamScratch s[kMaxStreams + kMoreStreams];
};
GpuScratch g_wide[kMaxCudaDevices];

// A thread's own calls while another stream is being captured: that capture does not mind them.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The scratch of `stream` on GPU `dev`, or null when there is none to be had (a stream that is being
// captured: a graph may be replayed anywhere; too many streams at work; no memory).  Call with the mutex held.
StreamScratch* scratch_of(GpuScratch& g, cudaStream_t stream, int lane) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
      cudaStreamGetId(stream, &id) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  for (int i = 0; i < g.used; ++i)
    if (g.s[i].stream_id == id && g.s[i].lane == lane) return &g.s[i];
  const RelaxedCapture relaxed;
  if (g.used == kMaxStreams + kMoreStreams) {
    StreamScratch* oldest = nullptr;
    for (int i = kMaxStreams; i < g.used; ++i) {
      StreamScratch& s = g.s[i];
      if (s.done && (!oldest || s.last_use < oldest->last_use) && cudaEventQuery(s.done) == cudaSuccess) oldest = &s;
    }
    cudaGetLastError();   // not an error of this call: some event is still ahead
    if (oldest) {
      oldest->stream_id = id;   // the buffers, their parities and their tag go on
      oldest->lane = lane;
    }
    return oldest;
  }
  StreamScratch& s = g.s[g.used];
  s = StreamScratch{};
  void* base = nullptr;
  if ((g.used >= kMaxStreams && cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming) != cudaSuccess) ||
      cudaMalloc(&base, kScratchBytes) != cudaSuccess) {
    cudaGetLastError();
    if (s.done) cudaEventDestroy(s.done);
    s.done = nullptr;
    return nullptr;
  }
  s.stream_id = id;
  s.lane = lane;
  s.base = static_cast<uint8_t*>(base);
  s.fresh = true;
  ++g.used;
  return &s;
}

// Launches one shape; *fits = false (nothing launched) where the GPU cannot hold one such cluster.
template <int G, int W, bool SPLIT, bool NEAR = false>
cudaError_t launch(const WideParams& p, int groups, int device, cudaStream_t stream, bool* fits) {
  static std::atomic<int> clusters[kMaxCudaDevices];   // 1 + clusters the GPU runs at a time, 0: not asked yet
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(groups * G));
  cfg.blockDim = dim3(wide_threads<W, NEAR>());
  cfg.dynamicSmemBytes = wide_smem<W, NEAR>();
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = G;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;   // for the occupancy question
  int n = clusters[device].load(std::memory_order_acquire);
  if (n == 0) {
    cudaError_t e = cudaFuncSetAttribute(mlp_wide_kernel<G, W, SPLIT, NEAR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         wide_smem<W, NEAR>());
    if (e == cudaSuccess && G > 8)
      e = cudaFuncSetAttribute(mlp_wide_kernel<G, W, SPLIT, NEAR>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    int active = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&active, mlp_wide_kernel<G, W, SPLIT, NEAR>, &cfg);
    if (e != cudaSuccess) return e;
    n = 1 + active;
    clusters[device].store(n, std::memory_order_release);
  }
  *fits = n > 1;
  cfg.numAttrs = hb::overlapped_launch_enabled() ? 2 : 1;
  return *fits ? cudaLaunchKernelEx(&cfg, mlp_wide_kernel<G, W, SPLIT, NEAR>, p) : cudaSuccess;
}
template <bool SPLIT>
cudaError_t launch(const hb::WidePlan& w, const WideParams& p, int device, cudaStream_t s, bool* fits) {
  if (w.near) return launch<16, 16, SPLIT, true>(p, w.groups, device, s, fits);
  switch (w.G * 100 + w.W) {
    case 1616: return launch<16, 16, SPLIT>(p, w.groups, device, s, fits);
    case 816: return launch<8, 16, SPLIT>(p, w.groups, device, s, fits);
    case 832: return launch<8, 32, SPLIT>(p, w.groups, device, s, fits);
    case 864: return launch<8, 64, false>(p, w.groups, device, s, fits);   // bf16 only, see wide_plan
    case 432: return launch<4, 32, SPLIT>(p, w.groups, device, s, fits);
    default: return launch<4, 64, SPLIT>(p, w.groups, device, s, fits);
  }
}
}  // namespace

namespace hb {

// The cheapest shape whose groups all run at a time.  Clusters stay inside a GPC, so a B200 runs 7, 15 or
// 33 of 16, 8 or 4 blocks.  Smaller groups hold more queries in all but stream more weights per block
// (L2 and shared-memory fill bound), wider ones exchange more per layer (L2 latency and bandwidth); the
// shapes below are those that no other one beats at its capacity.  Measured per launch, conv2d predictor,
// 8 hidden layers (capacity in queries: time), against 103 us (bf16) and 168 us (split) of one tile of the two-SM kernel:
//   bf16    42: 23 us (one: 19)   112: 24   240: 28   480: 32   960: 46   1,056: 48   2,112: 73
//   split   21: 32 (one: 29)       56: 34   120: 42   240: 46             528: 78     1,056: 126
// Eight blocks x 64 columns lose to four x 32 in split precision (86 us for 480).  Beyond the last shape
// the two-SM kernel of mlp_chain.cu is the faster one.
namespace {
// us: what a launch of the shape takes, full or not
struct Shape { int G, W, clusters, us, us_split; bool near; };
constexpr Shape kShapes[] = {{16, 16, 7, 22, 31, true},  {16, 16, 7, 25, 34, false}, {8, 16, 15, 29, 42, false},
                             {8, 32, 15, 32, 46, false}, {8, 64, 15, 48, 1000, false}, {4, 32, 33, 48, 77, false},
                             {4, 64, 33, 75, 128, false}};
int clusters_of(const Shape& s, int sm_count) { return sm_count >= 148 ? s.clusters : s.clusters * sm_count / 148; }
int cols_of(const Shape& s, bool split) { return s.near ? (split ? 3 : 6) : (split ? s.W / 2 : s.W); }   // near: see NEAR
WidePlan plan_in(const Shape& s, int64_t Q, bool split, int cols = 0) {
  // full groups while they last: fewer groups move the weights fewer times
  if (cols == 0) cols = cols_of(s, split);
  WidePlan w{s.G, s.W, static_cast<int>((Q + cols - 1) / cols), 0, s.near};
  w.per_group = static_cast<int>((Q + w.groups - 1) / w.groups);
  w.groups = static_cast<int>((Q + w.per_group - 1) / w.per_group);
  return w;
}
// Beside other batches near groups, which hold few queries, cost more of the GPU than they gain: 30 queries as six of them
// did not fit beside 1,590 (148.3 -> 153.5 us with 960 more), two groups of (16, 16) do.
bool fits_in_company(const WidePlan& w) { return !w.near || w.groups == 1; }
}  // namespace

WidePlan wide_plan(int64_t Q, bool split, int sm_count, bool alone) {
  for (const Shape& s : kShapes) {
    if (split && s.G == 8 && s.W == 64) continue;
    const int clusters = clusters_of(s, sm_count);
    if (Q > static_cast<int64_t>(clusters) * cols_of(s, split)) continue;
    const WidePlan w = plan_in(s, Q, split, s.near && alone ? static_cast<int>((Q + clusters - 1) / clusters) : 0);
    if (alone || fits_in_company(w)) return w;
  }
  return WidePlan{};
}

// Shapes for batches that run side by side.  The cheapest shape of each is the most spread out, and two of them
// rarely fit on the GPU together: the second then waits for the first.  A shape takes the same time with few
// groups as with many, so the shortest way through is the lowest time at which all batches fit when each takes
// the narrowest shape of that time or less, unless one after the other is shorter.  What is left of the GPU goes
// to cheaper shapes for the batches that start last.  Three predictors with 318, 192 and 6 queries: 60 -> 51 us.
void wide_plans_together(WidePlan* plans, const int64_t* Q, const bool* split, int n, int sm_count) {
  auto us_of = [&](const Shape& s, int b) { return split[b] ? s.us_split : s.us; };
  auto share_of = [&](const WidePlan& w, const Shape& s) {   // of the clusters that run at a time
    const int clusters = clusters_of(s, sm_count);
    return clusters ? static_cast<double>(w.groups) / clusters : 2.0;
  };
  int in_turn = 0;
  for (int b = 0; b < n; ++b)
    for (const Shape& s : kShapes)
      if (s.G == plans[b].G && s.W == plans[b].W && s.near == plans[b].near) in_turn += us_of(s, b);
  for (const Shape& level : kShapes) {
    WidePlan take[kMaxLanes];
    double least[kMaxLanes], all = 0.0;
    int us = 0;
    for (int b = 0; b < n; ++b) {
      least[b] = 2.0;
      for (const Shape& s : kShapes) {
        const WidePlan w = plan_in(s, Q[b], split[b]);
        if (!fits_in_company(w) || us_of(s, b) > us_of(level, b) || share_of(w, s) >= least[b]) continue;
        least[b] = share_of(w, s);
        take[b] = w;
      }
      all += least[b];
      us = us > us_of(level, b) ? us : us_of(level, b);
    }
    if (all > 1.0 || us >= in_turn) continue;
    for (int b = n - 1; b >= 0; --b) {
      plans[b] = take[b];
      for (const Shape& s : kShapes) {
        const WidePlan w = plan_in(s, Q[b], split[b]);
        const double with = all - least[b] + share_of(w, s);
        if (!fits_in_company(w) || us_of(s, b) > us_of(level, b) || with > 1.0) continue;
        plans[b] = w;
        all = with;
        break;
      }
    }
    return;
  }
}

void wide_handle_created(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return;
  std::lock_guard<std::mutex> lock(g_wide[device].mu);
  ++g_wide[device].handles;
}
void wide_handle_destroyed(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  if (--g.handles > 0) return;
  for (int i = 0; i < g.used; ++i) {
    cudaFree(g.s[i].base);   // waits for launches that still use it
    if (g.s[i].done) cudaEventDestroy(g.s[i].done);
    g.s[i].done = nullptr;
  }
  g.used = 0;
}

void wide_start_over(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  for (int i = 0; i < g.used; ++i) g.s[i].fresh = true;
}

hb_status wide_set_mark(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return HB_OK;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  HB_CUDA_TRY(cudaDeviceSynchronize());
  for (int i = 0; i < g.used; ++i)
    HB_CUDA_TRY(cudaMemset(g.s[i].base + kActsBytes + kHalvesBytes, 1, sizeof(int32_t)));
  HB_CUDA_TRY(cudaDeviceSynchronize());
  return HB_OK;
}

std::unique_lock<std::mutex> wide_queue(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return {};   // wide_predict launches nothing there
  return std::unique_lock<std::mutex>(g_wide[device].mu);
}

hb_status wide_predict(hb_mlp* h, const WidePlan& w, const MlpBatch& batch, cudaStream_t stream, bool* launched) {
  *launched = false;
  if (w.G == 0 || h->device >= kMaxCudaDevices || (batch.host_inputs && batch.Q > kWideInline)) return HB_OK;
  // parities and tags follow the stream's order: the caller holds the queue's lock
  GpuScratch& g = g_wide[h->device];
  StreamScratch* s = scratch_of(g, stream, batch.lane);
  if (!s) return HB_OK;
  s->last_use = ++g.uses;
  const bool split = h->precision == HB_PRECISION_BF16X3;
  WideParams p{};
  p.bias = h->bias; p.fc2_w = h->fc2_w; p.fc2_b = h->fc2_b; p.mu = h->mu; p.sigma = h->sigma; p.dev_feat = h->dev_feat;
  p.n_dev = h->n_dev; p.n_op_feat = h->n_op_feat; p.layers = h->layers;
  p.feats = batch.feats; p.dev_row = batch.dev_row; p.Q = static_cast<int32_t>(batch.Q);
  p.per_group = w.per_group; p.out = batch.out;
  p.status = h->status;
  p.beside = batch.beside && !s->fresh ? 1 : 0;   // (a fresh buffer's clearing has to be waited for)
  p.first = batch.first;
  p.grid_n = batch.grid_n;
  if (batch.grid_n) std::memcpy(p.grid_rows, batch.grid_rows, (batch.first + batch.Q) / batch.grid_n);
  if (batch.host_inputs) {
    p.inline_q = static_cast<int32_t>(batch.Q);
    std::memcpy(p.inline_feats, batch.feats, sizeof(float) * batch.Q * h->n_op_feat);
    std::memcpy(p.inline_row, batch.dev_row, batch.Q);
  }
  if (s->fresh) {
    // all words at parity 0, all tags at 0
    HB_CUDA_TRY(cudaMemsetAsync(s->base, 0, kScratchBytes, stream));
    for (auto& width : s->parity) width[0] = width[1] = ~0ull;
    s->tag = 0;
    s->fresh = false;
  }
  const int width = w.W == 16 ? 0 : (w.W == 32 ? 1 : 2);
  p.acts = s->base + static_cast<size_t>(kMaxGroups) * 2 * 2048 * (width == 0 ? 0 : (width == 1 ? 16 : 48));
  p.halves = reinterpret_cast<unsigned long long*>(s->base + kActsBytes);
  p.poison = reinterpret_cast<int32_t*>(s->base + kActsBytes + kHalvesBytes);
  if (++s->tag == 0) s->tag = 1;
  p.tag = s->tag;
  // exchange `use` (0 .. layers - 1) takes buffer use & 1; every group of the launch flips with it
  const unsigned long long groups = (1ull << w.groups) - 1;
  for (int b = 0; b < 2; ++b) {
    p.parity[b] = s->parity[width][b];
    if (!w.near && (((h->layers + 1 - b) / 2) & 1)) s->parity[width][b] ^= groups;
  }
  p.map_slot = w.G == 16 ? h->tmap_wide_slot : h->tmap_slot;
  p.map_fc1 = w.G == 16 ? h->tmap_wide_fc1 : h->tmap_tile;
  bool fits = false;
  const cudaError_t e = split ? launch<true>(w, p, h->device, stream, &fits)
                              : launch<false>(w, p, h->device, stream, &fits);
  s->fresh = e != cudaSuccess || !fits;   // not launched: the parities above did not happen
  if (s->done && cudaEventRecord(s->done, stream) != cudaSuccess) {
    cudaGetLastError();
    cudaEventDestroy(s->done);
    s->done = nullptr;         // nobody can tell any more when it is out of use: it stays with its stream
  }
  if (e != cudaSuccess) return cuda_fail(e, "mlp_wide_kernel launch");
  *launched = fits;
  return HB_OK;
}

}  // namespace hb
