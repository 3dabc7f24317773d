// MLP inference for batches between a few queries and full rounds of mlp_chain.cu's tiles: clusters of two-SM pairs.
//
// mlp_chain.cu gives a pair of SMs 128 queries and streams all weights past them: 103 to 110 us whether the batch has one
// query or 9,472.  Here P = 8, 4 or 2 pairs form a cluster that owns up to 2 NC queries (NC = 16, 32, 40, 48 or 64; split
// precision: NC).  Pair i computes 1024 / P output features of every layer for all of them and streams only their
// weights, and after each layer the cluster exchanges its activations.
//
// Formulation as in mlp_chain.cu, H^T = W . X^T with tcgen05.mma.cta_group::2: A = weight rows, half of them in each CTA
// of the pair (M = 128 or 256), B = activations, N = 2 NC columns, half of them in each CTA (MN-major, rows of 2 NC
// bytes), D = fp32 in TMEM.  Each CTA keeps, and each exchange moves, the activations of one half of the
// queries only: blocks that share no MMAs move twice as much for the same number.
// K is walked in the same order and fc2 adds in the same order as in mlp_chain.cu, so all kernels give the same bits
// and the choice of kernel never shows in a result.
//
// Exchange.  Distributed shared memory moves 17 bytes a cycle and SM whatever does it (st.async or bulk copies), L2 about
// 30 in and 85 out, so it goes through L2: an epilogue warp writes the next layer's rows of its 32 features, as they will
// lie in shared memory, into the activation buffer where the layer has read it, copies them to global memory (bulk
// store), waits until they are there and arrives at a barrier of each CTA that wants them, one per K quarter (256 rows); a
// CTA requests a quarter, one tiled load, when its rows have arrived (when all had, 112 queries took 24.9 us instead of 24.0, 371 26.6
// instead of 26.2, 1,200 40.6 instead of 39.9).  32 KB are there 730 cycles after the request, 128 KB after 1,540.
//
// The arrival should be a release: one more round trip to L2, 1,300 to 2,300 cycles in each layer.  The network is tried
// without first.  The arrival is a relaxed one, what has come is used at once, and warps look at it afterwards, while the
// next layer's is on its way.  An activation is never negative, so the high sign bit of every 32-bit word (two bf16
// activations, or the lo and the hi part of one in split precision) carries the parity of the buffer's use; with the
// parity 1 both halves are negated, and the instruction negates B.  A word of an earlier use with the same parity cannot
// come: the use in between, n, is ordered before the load of use n + 2, for in every second layer an epilogue warp passes
// a fence between two arrivals that the loader waits for first, while the MMAs run (371 queries 27.1 us without, 27.4 so,
// 27.6 with a fence in each layer; 4,224 63.7, 63.9, 64.5).  That a word comes whole, new or old, is what copies of 16
// bytes and more do; nothing else is taken for granted.  Where a word does not show the parity (in one launch of 40,000
// while other streams kept L2 busy, never alone), all CTAs of the cluster run the network once more, with releases; the
// words and their parities are those of the first run.  No result is stored before all CTAs have looked at everything.
// Two buffers alternate by layer: a CTA writes layer L only after its pair has read all of layer L - 1, which every CTA
// wrote after reading L - 2.  The host keeps the parity each group's buffers have reached.
// (Before the quarters had signals of their own: 448 queries 27.3 us so, 26.5 if nobody looked; with releases 32; by
// ordinary loads that poll the data in L2, 32 bytes a cycle, 34; bulk copies that are looked at before they are used 30.
// 1,920 queries 45.6, with releases 49.2; 4,224 65.1 and 68.2.)
//
// NC = 40, 48: rows of 80 or 96 bytes fit no swizzle, so B lies in panels of eight columns, 16 bytes a row, and a warp's rows go
// out as five or six copies of 512 bytes.  N is a multiple of 32, so with 40 the MMAs read a sixth panel per CTA, which is
// whatever lies behind the fifth; nobody reads the columns of D that come of it.  480 queries: 28.5 us in eight pairs with 40, 34.3 in
// four with 32; 600: 31.0 in eight with 48; 1,056: 40.5 in four pairs with 48, 45 with 64.
//
// NC = 64: a pair's features are two row blocks, one in K quarters 0 and 1 and one in 2 and 3.  The units (block b, K quarter
// q) of a layer are issued in the order (0,0) (0,1) (1,0) (0,2) (0,3) | (1,1) (1,2) (1,3): quarters 0 and 1 are
// exchanged under the last three units and quarters 2 and 3 under the first three of the next layer.  D alternates between two
// sets of TMEM columns.
//
// What bounds it: NC = 16 to 48 the latency of one exchange per layer (P = 8: 2,300 to 2,700 cycles from the last MMA to the next
// layer's first, of which 300 to 500 until the accumulators are there, 350 to take them and write them out, 400 for the
// store, 400 for the arrivals, 700 for the loads) next to 1,500 of MMAs; NC = 64 shared memory besides: a CTA's weights are
// written and read once per layer, B is read once per row block, and the exchange writes it, 1.5 MB a layer and CTA for P = 2
// and 1 MB for P = 4 at 128 bytes a cycle, and what the order of units leaves of the exchange.
//
// The blocks of a cluster are scheduled as a whole: that is what makes waiting for one another safe, and a launch may
// have more clusters than fit at a time.
//
// Warp roles: 0 TMEM, the mark, activation loads; 1 MMA issuer (the pair's leader); 2-3 weight producers; 4 and more:
// epilogue; NC = 16 to 48: eight more that look at what has come.  Every wait is bounded, as in mlp_chain.cu; a launch
// that gave up leaves a mark in the scratch, and launches that find it report an error instead of a result.  After giving
// up no ring slot is requested again whose copy could be under way: the MMA issuer, whose commits free the slots, waits
// for the producers of both CTAs to leave before it issues anything past a wait that ran out, and goes no further than
// the layer's end.
#include "mlp_small.cuh"

namespace {

// Two row blocks: the units of a layer, four bits each (4 b + q), first unit in the low bits
constexpr uint32_t kQuadOrder = 0x76532410u;
constexpr uint32_t kQuadFirstOfQuarter = 0x1Bu;   // units that read a K quarter for the first time
constexpr uint32_t kQuadLastOfQuarter1 = 5;       // the one that reads quarter 1 for the last time

template <int P, int NC, bool SPLIT>
struct PairShape {
  static constexpr int kCtas = 2 * P;
  static constexpr int kBlocks = NC == 64 ? 2 : 1;         // row blocks per pair
  static constexpr int kRows = 512 / P / kBlocks;          // A rows per CTA and block
  static constexpr bool kNarrow = kRows == 64;             // M = 128: D's second half of the columns is in TMEM lanes 64 and up
  static constexpr bool kPanels = NC == 40 || NC == 48;    // B without swizzle, in panels of eight columns
  static constexpr int kN = (2 * NC + 31) / 32 * 32;
  static constexpr int kHalfQ = SPLIT ? NC / 2 : NC;       // queries per CTA at most
  static constexpr int kRowBytes = 2 * NC;
  static constexpr int kActBytes = kWidth * kRowBytes;
  static constexpr int kSlotBytes = kNarrow ? 2 * kTileBytes : kTileBytes;
  static constexpr int kSlots = (NC >= 48 ? 6 : 8) * kTileBytes / kSlotBytes;
  static constexpr int kUnitBytes = kRows * 128;           // one K block of the rows
  static constexpr int kImages = kSlotBytes / kUnitBytes;  // per slot
  static constexpr int kParts = SPLIT ? 2 : 1;             // images per packed K block
  static constexpr int kUnits = 4 * kBlocks;               // (block, K quarter) per layer
  static constexpr int kSignals = kBlocks == 2 ? 2 : 4;    // per exchange: of row blocks, of K quarters
  static constexpr int kUnitSlots = 4 * kParts / kImages;
  // A K quarter of the activations is counted on the barrier of the slot that it is used with.
  static constexpr bool kApart = kBlocks == 1;             // there is room for the rows on their way out
  static constexpr bool kJoint = kApart && kNarrow && !SPLIT && kSlots == kUnits;
  static constexpr int kColGroups = NC == 64 ? 2 : 1;      // epilogue warps that share 32 rows
  static constexpr int kEpiWarps = (kNarrow ? 4 : 8) * kColGroups;
  static constexpr int kStores = kNarrow ? 4 : 8;          // bulk stores per block and CTA
  static constexpr int kLookWarps = kApart ? 8 : 0;        // those that look at what has come; else the epilogue's do
  static constexpr int kThreads = 128 + 32 * (kEpiWarps + kLookWarps);
  static constexpr int kDCols = kNarrow ? kN / 2 : kN;      // TMEM columns of a block
  static constexpr uint32_t kTmemCols = kBlocks == 2 ? 4 * kDCols : (kDCols <= 32 ? 32 : (kDCols <= 64 ? 64 : 128));
  static_assert(kRows == 64 || kRows == 128, "shapes");
  static_assert(!kJoint || (kUnitSlots == 1 && kSlots == kUnits), "a slot per quarter, each its own");
  static constexpr int kStageBytes = kApart ? 2 * kRows * kRowBytes : 0;   // this CTA's rows on their way out
  static constexpr int kSmem = kActBytes + kSlots * kSlotBytes + kStageBytes + 1024 + 1024;
  static_assert(kSmem <= 232448, "shared memory");
};

// A bounded wait that leaves the mark in the scratch: what this CTA's threads, copies and MMAs have done.
__device__ __forceinline__ bool pairs_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, const SmallParams& p,
                                           int code) {
  if (mbar_wait(bar, parity, abort_flag, p.status, code)) return true;
  atomicExch(p.poison, 1);
  return false;
}
// ... what other CTAs' threads have done.
__device__ __forceinline__ bool cluster_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, const SmallParams& p,
                                             int code) {
  if (mbar_wait_cluster(bar, parity, abort_flag, p.status, code)) return true;
  atomicExch(p.poison, 1);
  return false;
}
__device__ __forceinline__ void tma_2d_pair(uint32_t dst, const CUtensorMap* map, int32_t row, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row)
      : "memory");
}
__device__ __forceinline__ void tma_3d_pair(uint32_t dst, const CUtensorMap* map, int32_t row, int32_t image, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row), "r"(image)
      : "memory");
}
// Bulk store to global memory; returns when it is there.
__device__ __forceinline__ void store_rows(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile(
      "cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\t"
      "cp.async.bulk.commit_group;\n\t"
      "cp.async.bulk.wait_group 0;" ::"l"(dst),
      "r"(src), "r"(bytes)
      : "memory");
}
// An arrival that orders nothing.
__device__ __forceinline__ void mbar_arrive_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar, uint16_t ctas) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(ctas)
      : "memory");
}
// Byte offset of 16-byte chunk `chunk` of K row k in a B operand of NC columns per CTA (swizzle width 2 NC bytes); NC = 40, 48: in
// panels of `rows` K rows of 16 bytes, 256 in a K quarter.
template <int NC>
__device__ __forceinline__ uint32_t b_chunk(uint32_t k, uint32_t chunk, uint32_t rows = 256) {
  if (NC == 40 || NC == 48) return (chunk * rows + k) * 16u;
  const uint32_t x = NC == 64 ? (k & 7u) : (NC == 32 ? ((k >> 1) & 3u) : ((k >> 2) & 1u));
  return k * (2u * NC) + ((chunk ^ x) << 4);
}

template <int P, int NC, bool SPLIT>
__global__ void __launch_bounds__(PairShape<P, NC, SPLIT>::kThreads, 1)
mlp_pairs_kernel(const __grid_constant__ SmallParams p) {
  using S = PairShape<P, NC, SPLIT>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t act = base;
  const uint32_t ring = base + S::kActBytes;
  const uint32_t stage = ring + S::kSlots * S::kSlotBytes;
  const uint32_t bars = stage + S::kStageBytes;
  uint8_t* bars_ptr = base_ptr + (bars - base);
  const uint32_t bar_full = bars, bar_empty = bars + 64;   // [kSlots] full: leader only, both CTAs' boxes landed
  const uint32_t bar_sig = bars + 264;      // [2 buffers][kSignals] rows of this CTA's queries are in global memory
  const uint32_t bar_actq = bars + 160;     // [4] leader only: K quarter in place in both CTAs
  const uint32_t bar_acc = bars + 192;      // [kBlocks] row block accumulated
  const uint32_t bar_stored = bars + 208;   // [kBlocks] this CTA's rows of the block are in global memory
  const uint32_t bar_feat = bars + 224;     // leader only: fc1's input in place in both CTAs
  const uint32_t bar_q1 = bars + 232;       // two blocks: quarter 1 has been read
  const uint32_t bar_seen = bars + 240;     // first run: the layer's input has been looked at
  const uint32_t bar_drain = bars + 248;    // leader only, after giving up: the MMAs have ended
  const uint32_t bar_out = bars + 256;      // kApart: the output of a layer after the first is on its way (kEpiWarps)
  constexpr int kBars = 41, kAbort = 340, kStale = 344, kLeft = 352;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_ptr + 336);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars_ptr + kAbort);
  volatile int* stale = reinterpret_cast<volatile int*>(bars_ptr + kStale);           // some CTA of the cluster has seen stale words
  volatile int* producers_left = reinterpret_cast<volatile int*>(bars_ptr + kLeft);   // [4] leader only

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank(), r = cta & 1u, leader = cta & ~1u;
  const int pair = static_cast<int>(cta >> 1);
  const int group = static_cast<int>(blockIdx.x) / S::kCtas;      // = cluster
  const uint16_t both = static_cast<uint16_t>(3u << leader);

  auto init_barriers = [&] {
    for (int i = 0; i < kBars; ++i) mbar_init(bars + 8 * i, 1);
    if (S::kJoint)
      for (int s = 0; s < S::kSlots; ++s) mbar_init(bar_full + 8 * s, 2);
    for (int i = 0; i < 2 * S::kSignals; ++i) mbar_init(bar_sig + 8 * i, 32 / S::kSignals);
    for (int b = 0; b < S::kBlocks; ++b) mbar_init(bar_stored + 8 * b, S::kStores);
    mbar_init(bar_feat, 2);
    mbar_init(bar_seen, S::kApart ? S::kLookWarps : S::kEpiWarps);
    mbar_init(bar_out, S::kEpiWarps);
    for (int i = 0; i < 4; ++i) producers_left[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  };
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *stale = 0;
    init_barriers();
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(S::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  grid_begin(p.beside != 0);
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int n_layers = p.layers + 1;

  // This group's queries, the first half of them with the leaders.
  const int64_t g0 = static_cast<int64_t>(group) * p.per_group;
  const int in_group = static_cast<int>(min(static_cast<int64_t>(p.per_group), static_cast<int64_t>(p.Q) - g0));
  const int first_half = min((p.per_group + 1) / 2, in_group);
  const int64_t q0 = g0 + (r ? first_half : 0);
  const int n_q = r ? in_group - first_half : first_half;
  constexpr uint32_t kHalfBytes = S::kActBytes;
  // first output feature of the pair's row block b, as a K index of the next layer
  auto block_feature = [&](int b) { return b * 512 + pair * (2 * S::kRows); };
  auto saw_stale = [&] {
#pragma unroll 1
    for (uint32_t c = 0; c < S::kCtas; ++c) st_cluster_u32(map_to_cta(bars + kStale, c), 1u);
    __threadfence();
  };
  constexpr uint32_t kSigns = SPLIT ? 0x80000000u : 0x80008000u;   // those that carry the parity
  float result = 0.0f;

  // sure: with releases; the first run goes without
#pragma unroll 1
  for (bool sure = false;; sure = true) {
    uint8_t* const group_acts = p.acts + static_cast<size_t>(group) * (4u * kHalfBytes);
    // both signs of the words of the `use`-th exchange
    auto signs_of = [&](int use) -> uint32_t {
      return (((p.parity[use & 1] >> group) + static_cast<unsigned>(use >> 1)) & 1ull) ? 0x80008000u : 0u;
    };
    const uint32_t tag = sure ? p.tag | 0x80000000u : p.tag;
    if (warp == 0) {
      // ------------------------------ the mark; activation loads ------------------------------
      if (lane == 0) {
        // An earlier launch that gave up may still be writing: report, and give up as well (no result is stored then).
        if (hb::concerns(*reinterpret_cast<volatile int32_t*>(p.poison), cta)) {
          *static_cast<volatile int32_t*>(p.status) = 0x5FF;
          *abort_flag = 1;
        }
        bool ok = true;
        const int32_t row0 = (group * 4 + static_cast<int>(r)) * 4;   // in K quarters
        for (int L = 1; L < n_layers && ok; ++L) {
          const int u = L - 1, buf = u & 1;
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            if (q == 0 || (S::kBlocks == 2 && q == 2)) {
              // the buffer has been read, this CTA's rows copied from it (kApart: they are not in it), and it has been looked at;
              // then the rows of all CTAs
              const int b = S::kBlocks == 2 ? q >> 1 : 0;
              ok = S::kApart ? pairs_wait(bar_acc, u & 1, abort_flag, p, 0x531)
                             : pairs_wait(bar_stored + 8 * b, u & 1, abort_flag, p, 0x531);
              if (!sure && u > 0 && q == 0) ok = ok && pairs_wait(bar_seen, (u - 1) & 1, abort_flag, p, 0x534);
            } else if (S::kBlocks == 2 && q == 1 && u > 0) {
              ok = pairs_wait(bar_q1, (u - 1) & 1, abort_flag, p, 0x533);
            }
            if (S::kSignals == 4 || (q & 1) == 0) {
              ok = ok && cluster_wait(bar_sig + 8 * (buf * S::kSignals + q * S::kSignals / 4), (u >> 1) & 1, abort_flag, p, 0x532);
              asm volatile("fence.proxy.async.global;" ::: "memory");
            }
            if (!ok) break;
            const uint32_t bar = S::kJoint ? bar_full + 8 * ((S::kBlocks + q) % S::kSlots) : bar_actq + 8 * q;
            if (r == 0) mbar_expect_tx(bar, 2u * 256u * S::kRowBytes);
            tma_2d_pair(act + q * 256 * S::kRowBytes, &p.map_acts, (row0 + buf * 8 + q) * static_cast<int32_t>(hb::act_map_box(NC)),
                        map_to_cta(bar, leader));
          }
        }
        if (S::kBlocks == 2 && ok) pairs_wait(bar_q1, (p.layers - 1) & 1, abort_flag, p, 0x533);   // as the last slots below
      }
      __syncwarp();
    } else if (warp == 2 || warp == 3) {
      // ------------------------------ weight producers ------------------------------
      if (lane == 0) {
        const uint32_t w = static_cast<uint32_t>(warp - 2);
        constexpr uint32_t kLayerLoads = S::kUnits * S::kUnitSlots;
        const uint32_t loads = S::kBlocks + static_cast<uint32_t>(p.layers) * kLayerLoads;
        for (uint32_t n = w; n < loads; n += 2) {
          const bool fc1 = n < S::kBlocks;
          const uint32_t m = n - S::kBlocks, L = m / kLayerLoads, u = m % kLayerLoads / S::kUnitSlots, g = m % S::kUnitSlots;
          const uint32_t unit = S::kBlocks == 2 ? (kQuadOrder >> (4 * u)) & 15u : u, kq = unit & 3u;
          const uint32_t b = fc1 ? n : unit >> 2;
          const uint32_t mt = static_cast<uint32_t>(block_feature(b)) / kMTile + (S::kNarrow ? 0u : r);
          const uint32_t image =
              fc1 ? S::kParts * mt
                  : S::kParts * (kNumMT + (L * kNumMT + mt) * kNumKB + kq * 4) + g * S::kImages;
          const uint32_t s = n % S::kSlots, ph = (n / S::kSlots & 1u) ^ 1u;
          const uint32_t full = bar_full + 8 * s, full_leader = map_to_cta(full, leader), dst = ring + s * S::kSlotBytes;
          if (!pairs_wait(bar_empty + 8 * s, ph, abort_flag, p, 0x511)) break;
          if (r == 0) mbar_expect_tx(full, 2 * (fc1 ? S::kUnitBytes : S::kSlotBytes));
          if (S::kJoint && r == 0 && fc1) mbar_arrive(full);
          if (S::kNarrow) tma_3d_pair(dst, fc1 ? &p.map_fc1 : &p.map_slot, r * S::kRows, image, full_leader);
          else tma_2d_pair(dst, &p.map_slot, image * kMTile, full_leader);
        }
        // Every slot's last commit: it may still be on its way to this CTA when the layer's is there, and the barriers start over,
        // or the shared memory is somebody else's.
        for (uint32_t n = loads + w; n < loads + S::kSlots && *abort_flag == 0; n += 2)
          pairs_wait(bar_empty + 8 * (n % S::kSlots), (n / S::kSlots & 1u) ^ 1u, abort_flag, p, 0x512);
        st_cluster_u32(map_to_cta(bars + kLeft + 4 * (2 * r + w), leader), 1u);
      }
      __syncwarp();
    } else if (warp == 1) {
      // ------------------------------ MMA issuer ------------------------------
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) |
                                 (static_cast<uint32_t>(S::kN >> 3) << 17) |
                                 (static_cast<uint32_t>((2 * S::kRows) >> 4) << 24);
      constexpr uint32_t kNegateB = 1u << 14;
      // A: K-major, 128-byte swizzle, 8-row groups 1024 B apart; B: MN-major, one swizzle atom wide, 8-row
      // groups of K 16 NC bytes apart
      const uint64_t desc_a = (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                              (static_cast<uint64_t>(2) << 61) | (static_cast<uint64_t>(1) << 16);
      // (panels: no swizzle, 8-row groups 128 B apart and 8-column ones 4 KB)
      const uint64_t desc_b =
          S::kPanels ? (static_cast<uint64_t>(4096 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                           (static_cast<uint64_t>(128 >> 4) << 16)
                     : (static_cast<uint64_t>((16 * NC) >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                           (static_cast<uint64_t>(NC == 64 ? 2 : (NC == 32 ? 4 : 6)) << 61) |
                           (static_cast<uint64_t>(1) << 16);
      // in 16-byte units: 16 K values of B, a K block of 64, a K quarter
      constexpr uint32_t kStepB = (S::kPanels ? 256 : 32 * NC) >> 4, kBlockB = 4 * kStepB;
      constexpr uint32_t kQuarterB = (256 * S::kRowBytes) >> 4;
      const uint32_t a_lo0 = (ring & 0x3FFFF) >> 4, b_lo0 = (act & 0x3FFFF) >> 4;
      // One elected lane runs the whole loop, and no loop of a layer depends on what a wait returns (after a wait that
      // ran out the abort flag is set, and nothing that comes of stale operands is stored as a result), which keeps the descriptors in
      // uniform registers.  A try_wait holds up the issue for 90 cycles, so with M = 128 (21 to 32 cycles per MMA) slots
      // last 16 MMAs: with 8 an MMA took 33 cycles whatever N, with 16 it takes 23 to 25.
      if (r == 0 && elect_one()) {
        auto wait = [&](uint32_t bar, uint32_t parity, int code) {
          if (!mbar_try_wait(bar, parity) && (*abort_flag || !pairs_wait(bar, parity, abort_flag, p, code))) {
            // (the producers look at their CTA's abort flag when a slot does not come)
            st_cluster_u32(map_to_cta(bars + kAbort, leader + 1), 1u);
            __threadfence();
            const long long t0 = clock64();
            for (int i = 0; i < 4; ++i)
              while (producers_left[i] == 0 && clock64() - t0 <= kWaitCycles) {}
          }
          tc_fence_after();
        };
        uint32_t s = 0, ph = 0;
        if (!cluster_wait(bar_feat, 0, abort_flag, p, 0x521)) wait(bar_feat, 0, 0x521);
        tc_fence_after();
#pragma unroll 1
        for (int b = 0; b < S::kBlocks; ++b) {                     // fc1: one K block
          wait(bar_full + 8 * s, ph, 0x522);
          const uint32_t d = tmem_base + static_cast<uint32_t>(b * S::kDCols);
          const uint32_t a_lo = a_lo0 + s * (S::kSlotBytes >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc_mma_pair_bf16(d, desc_a | (a_lo + 2 * k), desc_b | (b_lo0 + k * kStepB), idesc, k ? 1u : 0u);
          commit_pair(bar_empty + 8 * s, both);
          ring_next<S::kSlots>(s, ph);
        }
        // (all at once: the blocks' rows are written over the input)
        for (int b = 0; b < S::kBlocks; ++b) commit_pair(bar_acc + 8 * b, both);
#pragma unroll 1
        for (int L = 1; L < n_layers && *abort_flag == 0; ++L) {
          bool landed = false;            // the barrier of slot s has been seen complete
          const uint32_t id = idesc | (signs_of(L - 1) & kNegateB << 1) >> 1;
#pragma unroll 1
          for (uint32_t u = 0; u < S::kUnits; ++u) {
            const uint32_t unit = S::kBlocks == 2 ? (kQuadOrder >> (4 * u)) & 15u : u, b = unit >> 2, kq = unit & 3u;
            if (!S::kJoint && (S::kBlocks == 1 || (kQuadFirstOfQuarter >> u) & 1u))
              wait(bar_actq + 8 * kq, (L - 1) & 1, 0x523);
            const uint32_t d = tmem_base + (S::kBlocks == 2 ? ((L & 1) * 2 + b) * S::kDCols : 0u);
#pragma unroll
            for (uint32_t g = 0; g < S::kUnitSlots; ++g) {
              uint32_t next = s, next_ph = ph;
              ring_next<S::kSlots>(next, next_ph);
              const uint32_t a_lo = a_lo0 + s * (S::kSlotBytes >> 4);
              if (!landed) wait(bar_full + 8 * s, ph, 0x522);
#pragma unroll
              for (uint32_t i = 0; i < 4 * S::kImages; ++i) {
                const uint32_t kb = (g * S::kImages + (i >> 2)) / S::kParts, k = i & 3u;
                tc_mma_pair_bf16(d, desc_a | (a_lo + (i >> 2) * (S::kUnitBytes >> 4) + 2 * k),
                                 desc_b | (b_lo0 + kq * kQuarterB + kb * kBlockB + k * kStepB), id,
                                 (g == 0 && i == 0) ? kq : 1u);
                if (i == 2 * S::kImages - 1) {
                  // (not past the layer's end: a try_wait that has to wait holds up the MMAs behind it)
                  landed = (u + 1 < S::kUnits || g + 1 < S::kUnitSlots) && mbar_try_wait(bar_full + 8 * next, next_ph);
                  tc_fence_after();
                }
              }
              commit_pair(bar_empty + 8 * s, both);
              s = next;
              ph = next_ph;
            }
            if (S::kBlocks == 2 && u == kQuadLastOfQuarter1) commit_pair(bar_q1, both);
            if (kq == 3) commit_pair(bar_acc + 8 * b, both);
          }
        }
      }
      __syncwarp();
    } else {
      // ------------------------------ fc1's input ------------------------------
      // K rows 0..63 hold [hi | lo | hi] of the normalised features, one query per column (split: the second of its two, see
      // below).  Those that look later help: a thread's two loads in a row and the division take some 1,500 cycles, and the
      // epilogue's warps alone went round two to five times (112 queries 25.2 -> 24.9 us, 371 27.7 -> 26.6).
      constexpr int kFeatThreads = S::kThreads - 128;
      const int T = static_cast<int>(threadIdx.x) - 128;
      auto feat_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kFeatThreads) : "memory"); };
      const int C_in = p.n_op_feat + 4, n_in = n_q * C_in;
      for (int i = T; i < 64 * S::kRowBytes / 16; i += kFeatThreads)
        *reinterpret_cast<uint4*>(base_ptr + (S::kPanels ? b_chunk<NC>(i & 63, i >> 6) : 16 * i)) = make_uint4(0, 0, 0, 0);
#pragma unroll 1
      for (int i0 = 0; i0 == 0 || i0 < n_in; i0 += kFeatThreads) {
        const int i = i0 + T, q = i / C_in, f = i - q * C_in;
        __nv_bfloat16 hi, lo;
        if (i < n_in) load_feature(p, static_cast<int>(q0) + q, f, hi, lo);
        if (i0 == 0) feat_sync();   // the zeros are there
        if (i < n_in) {
          const uint32_t col = static_cast<uint32_t>(SPLIT ? 2 * q + 1 : q), ch = col >> 3, in = 2u * (col & 7u);
          *reinterpret_cast<__nv_bfloat16*>(base_ptr + b_chunk<NC>(f, ch) + in) = hi;
          *reinterpret_cast<__nv_bfloat16*>(base_ptr + b_chunk<NC>(C_in + f, ch) + in) = lo;
          *reinterpret_cast<__nv_bfloat16*>(base_ptr + b_chunk<NC>(2 * C_in + f, ch) + in) = hi;
        }
      }
      fence_proxy_async();
      feat_sync();
      if (T == 0) {
        if (r == 0) mbar_arrive(bar_feat);
        else mbar_arrive_remote(map_to_cta(bar_feat, leader));
      }
      __syncwarp();
      if (S::kApart && warp >= 4 + S::kEpiWarps) {
        // ------------------------------ looking at what has been used ------------------------------
        constexpr int kShare = S::kApart ? S::kActBytes / S::kLookWarps : 0, kBatch = NC == 40 ? 10 : 8;
        static_assert(kShare % (512 * kBatch) == 0, "all of it");
        const uint8_t* const mine = base_ptr + (warp - 4 - S::kEpiWarps) * kShare + 16 * lane;
#pragma unroll 1
        for (int L = 1; L < n_layers && !sure; ++L) {
          // (not while the epilogue is at it: it took 500 cycles instead of 220)
          if (!pairs_wait(bar_out, (L - 1) & 1, abort_flag, p, 0x551)) break;
          const uint32_t want = signs_of(L - 1) ^ p.expect_stale;
          uint32_t bad = 0;
#pragma unroll 1
          for (int i = 0; i < kShare; i += 512 * kBatch) {
            uint4 x[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) x[k] = *reinterpret_cast<const uint4*>(mine + i + 512 * k);
#pragma unroll
            for (int k = 0; k < kBatch; ++k) bad |= (x[k].x ^ want) | (x[k].y ^ want) | (x[k].z ^ want) | (x[k].w ^ want);
          }
          if (bad & kSigns) saw_stale();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_seen);
        }
        __syncwarp();
      } else {
        // ------------------------------ epilogue ------------------------------
        // A warp drains 32 rows (features) of one half of the columns, or a part of them (kColGroups).  Split precision: a
        // query has two columns, of the lo and the hi part of its activations: one 32-bit word in a row of B.
        const int quad = warp & 3, rest = (warp - 4) >> 2;
        const uint32_t half = S::kNarrow ? quad >> 1 : rest & 1;
        const int part = S::kNarrow ? rest : rest >> 1;
        const int row0 = S::kNarrow ? (quad & 1) * 32 : quad * 32;
        constexpr int kPiece = S::kHalfQ / S::kColGroups;      // queries per warp
        constexpr int kCols = S::kParts * kPiece;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + (S::kNarrow ? 0u : half * (S::kN / 2)) +
                                static_cast<uint32_t>(part * kCols);
        unsigned long long* const group_halves = p.halves + static_cast<size_t>(group) * 64 * hb::kGroupCols;
        auto rows_sync = [&] {   // the warps of these rows
          if (S::kColGroups == 2) asm volatile("bar.sync %0, 64;" ::"r"(2 + quad + (S::kNarrow ? 0 : 4 * static_cast<int>(half))) : "memory");
          else __syncwarp();
        };
        // This warp's share of the input, without the first `from` rows of quarters 0 and 2.
        auto look = [&](uint32_t want, uint32_t from) {
          constexpr uint32_t kStep = 4096;              // 32 rows
          uint32_t bad = 0;
#pragma unroll 1
          for (uint32_t at = (warp - 4) * kStep; at < S::kActBytes; at += S::kEpiWarps * kStep) {
            if ((at / S::kRowBytes & 511u) < from) continue;
            uint4 x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = *reinterpret_cast<const uint4*>(base_ptr + at + 512 * k + 16 * lane);
#pragma unroll
            for (int k = 0; k < 8; ++k) bad |= (x[k].x ^ want) | (x[k].y ^ want) | (x[k].z ^ want) | (x[k].w ^ want);
          }
          if (bad & kSigns) saw_stale();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_seen);
        };
        bool ok = true;
        // a wait that ran out skips the work that is left but none of the barriers
#pragma unroll 1
        for (int L = 0; L < n_layers; ++L) {
          const bool last = L == n_layers - 1;
          const uint32_t signs = signs_of(L), want = L > 0 ? signs_of(L - 1) ^ p.expect_stale : 0u;
#pragma unroll 1
          for (int b = 0; b < S::kBlocks; ++b) {
            const int f0 = block_feature(b) + static_cast<int>(r) * S::kRows + row0, f = f0 + lane;
            const float bias = __ldg(p.bias + L * kWidth + f);
            const float w2 = last ? __ldg(p.fc2_w + f) : 0.0f;
            if (ok) {
              bool go = true;
              if (lane == 0) go = pairs_wait(bar_acc + 8 * b, L & 1, abort_flag, p, 0x541);
              ok = __shfl_sync(0xFFFFFFFFu, go ? 1 : 0, 0) != 0;
            }
            // where the rows are kept for the copy: in a place of their own, or the activation buffer, where it has been read
            // (quarter 2 b) and is loaded over after they have been copied
            const int at0 = (S::kApart ? 0 : b * 512) + static_cast<int>(half) * S::kRows + row0;
            const uint32_t rows = S::kApart ? stage : act;
            if (ok) {
              tc_fence_after();
              const uint32_t t_block = t_lane + (S::kBlocks == 2 ? static_cast<uint32_t>(((L & 1) * 2 + b) * S::kDCols) : 0u);
              float v[kPiece];
              if constexpr (SPLIT) {
                float d[kCols];
                tc_ld_cols<kCols>(t_block, d);
#pragma unroll
                for (int i = 0; i < kPiece; ++i) v[i] = d[2 * i + 1] + d[2 * i];
              } else {
                tc_ld_cols<kPiece>(t_block, v);
              }
              tc_fence_before();
#pragma unroll
              for (int i = 0; i < kPiece; ++i) v[i] = fmaxf(v[i] + bias, 0.0f);
              if (!last) {
                constexpr int kWords = kCols / 2;
                uint32_t w[kWords];
#pragma unroll
                for (int i = 0; i < kWords; ++i) {
                  if (SPLIT) {
                    const __nv_bfloat16 hi = __float2bfloat16_rn(v[i % kPiece]);
                    const __nv_bfloat16 lo = __float2bfloat16_rn(v[i % kPiece] - __bfloat162float(hi));
                    w[i] = static_cast<uint32_t>(__bfloat16_as_ushort(hi)) << 16 | __bfloat16_as_ushort(lo);
                  } else {
                    const __nv_bfloat162 pk = __floats2bfloat162_rn(v[(2 * i) % kPiece], v[(2 * i + 1) % kPiece]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&pk);
                  }
                  w[i] = (w[i] & (SPLIT ? 0x7FFFFFFFu : 0x7FFF7FFFu)) ^ signs;
                }
                uint32_t bad = 0;
#pragma unroll
                for (int c = 0; c < kWords / 4; ++c) {
                  uint4* const to = reinterpret_cast<uint4*>(
                      base_ptr + (rows - base) +
                      b_chunk<NC>(static_cast<uint32_t>(at0 + lane), static_cast<uint32_t>(part * (kWords / 4) + c), 2 * S::kRows));
                  if (!S::kApart && !sure && L > 0) {   // looked at before it goes
                    const uint4 x = *to;
                    bad |= (x.x ^ want) | (x.y ^ want) | (x.z ^ want) | (x.w ^ want);
                  }
                  *to = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
                }
#if defined(HB_BOUNDS_CHECK)   // (it costs 0.3 to 0.5 us)
                if (L == p.stale_layer && !sure && f == p.stale_feature)
                  for (int i = 0; i < kWords; ++i)
                    if (p.stale_word == static_cast<int>(half) * (NC / 2) + part * kWords + i)
                      *reinterpret_cast<uint32_t*>(base_ptr + (rows - base) + 4 * (i & 3) +
                                                   b_chunk<NC>(static_cast<uint32_t>(at0 + lane),
                                                               static_cast<uint32_t>(part * (kWords / 4) + (i >> 2)), 2 * S::kRows)) ^=
                          0x80008000u;
#endif
                fence_proxy_async();
                if (bad & kSigns) saw_stale();
              } else {
                constexpr int kFold = (kPiece + 15) / 16 * 16;
                float sum[kFold];
#pragma unroll
                for (int i = 0; i < kFold; ++i) sum[i] = i < kPiece ? __fmul_rn(w2, v[i % kPiece]) : 0.0f;
                fold16(sum, lane);
                const int set = (f0 + (lane & 16)) / 16, col = fold16_col<kFold>(lane);
                unsigned long long* h = group_halves + set * hb::kGroupCols + half * 64 + part * kPiece + col;
#pragma unroll
                for (int i = 0; i < kFold / 16 && (kPiece == kFold || col + i < kPiece); ++i)
                  st_relaxed_u64(h + i, static_cast<unsigned long long>(tag) << 32 | __float_as_uint(sum[i]));
              }
            }
            if (S::kApart && L > 0) {   // (each phase waits for the look of the one before: no parity comes round unseen)
              __syncwarp();
              if (lane == 0) mbar_arrive(bar_out);
            }
            if (last) continue;
            rows_sync();
            if (part == 0) {
              if (ok) {
                uint8_t* const to = group_acts + ((L & 1) * 2 + half) * kHalfBytes;
                if (S::kPanels) {
                  if (lane < NC / 8)
                    store_rows(to + (f0 >> 8) * (256 * S::kRowBytes) + b_chunk<NC>(f0 & 255, lane),
                               rows + b_chunk<NC>(at0, lane, 2 * S::kRows), 32 * 16);
                } else if (lane == 0) {
                  store_rows(to + static_cast<uint32_t>(f0) * S::kRowBytes, rows + static_cast<uint32_t>(at0) * S::kRowBytes,
                             32 * S::kRowBytes);
                  if (!S::kApart) mbar_arrive(bar_stored + 8 * b);
                }
                __syncwarp();
                if (lane < P) {
                  const uint32_t bar = map_to_cta(bar_sig + 8 * ((L & 1) * S::kSignals + (S::kBlocks == 2 ? b : f0 >> 8)), 2 * lane + half);
                  if (sure) mbar_arrive_remote(bar);
                  else mbar_arrive_relaxed(bar);
                }
              }
              __syncwarp();
            }
            // Block 0 has used all of the layer's input.  What the blocks' rows are not written over is looked at now.
            if (!S::kApart && b == 0 && L > 0 && ok && !sure) look(want, 2 * S::kRows);
          }
          // With the arrivals after it a release of this layer's and the last one's rows, before those places are read again; while
          // the next layer's MMAs run.
          if (!sure && part == 0 && (L & 1) && L + 2 < n_layers) asm volatile("fence.acq_rel.cluster;" ::: "memory");
          if (!S::kApart && last && ok && !sure) look(want, 0);
        }
        if (cta < 2 && warp < 8) {
          // the first CTA of each half adds the 64 sets of 16 features of its queries
          const int q = T & 63;
          float* tots = reinterpret_cast<float*>(bars_ptr + 512);
          tots[T] = q < n_q && ok ? fc2_sum(p, group_halves + r * 64 + q, T >> 6, tag, abort_flag) : 0.0f;
          asm volatile("bar.sync 10, 128;" ::: "memory");
          result = tots[T & 63] + tots[64 + (T & 63)] + p.fc2_b;
        }
      }
    }
    // No CTA leaves while another may still signal to it, all have looked at everything, and all know whether one gave up: what
    // it has sent since may be anything, a last layer with its sums included, so then no CTA stores a result or runs again, and all
    // go through the teardown.  (Flags that another CTA has to see were followed by a fence.)
    tc_fence_before();
    __syncwarp();
    if (lane == 0 && *abort_flag) {
#pragma unroll 1
      for (uint32_t c = 0; c < S::kCtas; ++c) st_cluster_u32(map_to_cta(bars + kAbort, c), 1u);
      __threadfence();
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    tc_fence_after();
    if (sure || *abort_flag || *stale == 0) break;   // (nobody sets them between the two barriers)
    if (threadIdx.x == 0) {
      if (cta == 0) atomicAdd(p.poison + 1, 1);
      for (int i = 0; i < kBars; ++i) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bars + 8 * i) : "memory");
      init_barriers();
    }
    __syncthreads();
    cluster_sync_all();
  }
  if (cta < 2 && threadIdx.x >= 128 && threadIdx.x < 256) {
    const int T = static_cast<int>(threadIdx.x) - 128;
    if (T < n_q && *abort_flag == 0) p.out[q0 + T] = result;
  }

  // ------------------------------ teardown ------------------------------
  if (*abort_flag) {
    __syncthreads();
    if (r == 0 && warp == 1 && elect_one()) {
      // the MMAs end before the TMEM they write is somebody else's
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_drain) : "memory");
      const long long t0 = clock64();
      while (!mbar_try_wait_cluster(bar_drain, 0) && clock64() - t0 <= kWaitCycles) {}
    }
    // and copies in flight land before the shared memory goes away: they take about a thousand cycles
    if (threadIdx.x == 0)
      for (const long long t0 = clock64(); clock64() - t0 < 200000;) {}
    __syncthreads();
    cluster_sync_all();
  }
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::kTmemCols) : "memory");
  }
  grid_end(p.beside != 0);
}

template <int P, int NC, bool SPLIT>
cudaError_t launch(const SmallParams& p, int groups, int device, cudaStream_t stream, bool* fits) {
  using S = PairShape<P, NC, SPLIT>;
  static std::atomic<int> clusters[hb::kMaxCudaDevices];
  return hb::launch_clusters(mlp_pairs_kernel<P, NC, SPLIT>, S::kCtas, S::kThreads, S::kSmem, p, groups, stream, fits,
                             clusters[device]);
}
template <bool SPLIT>
cudaError_t launch(int P, int NC, const SmallParams& p, int groups, int device, cudaStream_t stream, bool* fits) {
  switch (P * 100 + NC) {
    case 816: return launch<8, 16, SPLIT>(p, groups, device, stream, fits);
    case 840: return launch<8, 40, SPLIT>(p, groups, device, stream, fits);
    case 848: return launch<8, 48, SPLIT>(p, groups, device, stream, fits);
    case 832: return launch<8, 32, SPLIT>(p, groups, device, stream, fits);
    case 448: return launch<4, 48, SPLIT>(p, groups, device, stream, fits);
    case 432: return launch<4, 32, SPLIT>(p, groups, device, stream, fits);
    case 464: return launch<4, 64, SPLIT>(p, groups, device, stream, fits);
    case 264: return launch<2, 64, SPLIT>(p, groups, device, stream, fits);
    default: return cudaErrorInvalidConfiguration;
  }
}
}  // namespace

bool hb::pairs_plant_words() {
#if defined(HB_BOUNDS_CHECK)
  return true;
#else
  return false;
#endif
}

cudaError_t hb::launch_pairs(int P, int NC, bool split, const SmallParams& p, int groups, int device, cudaStream_t stream,
                             bool* fits) {
  return split ? launch<true>(P, NC, p, groups, device, stream, fits)
               : launch<false>(P, NC, p, groups, device, stream, fits);
}
