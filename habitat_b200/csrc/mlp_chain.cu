// Fused inference of Habitat's per-operation MLP runtime predictors on sm_100a.
//
// Stands in for RuntimePredictor.predict (analyzer/habitat/analysis/mlp/mlp.py:252-267
// of the reference) over a whole batch of queries: feature normalisation
// (mlp.py:258-261), fc1 + ReLU, `layers` x [Linear(1024,1024) + ReLU] and fc2
// (mlp.py:17-109) run as ONE persistent kernel; activations never leave the SM.
//
// Formulation.  Two CTAs of a cluster own a tile of queries and compute every layer
// transposed, H^T = W . X^T, so that
//   A (M = 256 output features x K) = weight tiles, streamed from global/L2 into a
//                                     shared-memory ring by tiled TMA loads (mbarrier
//                                     completion), half of the rows in each CTA;
//   B (N = 128 columns x K)         = the activations, resident in shared memory
//                                     (MN-major, 128-byte swizzle), half of the columns
//                                     in each CTA;
//   D (128 lanes x 128 columns)     = fp32 accumulators in tensor memory, one column
//                                     block per 256-feature block, so the whole layer
//                                     output lives in TMEM until it is drained.
// tcgen05.mma.cta_group::2 (kind::f16, bf16 inputs, fp32 accumulate) is issued by one
// elected lane of a warp that walks the issue loop as a whole; the epilogue warps read TMEM
// with tcgen05.ld, add the bias, apply ReLU, round to bf16 and overwrite the activation
// buffer in place while the tensor core works on the remaining blocks of the layer.  fc2 is
// a dot product over features (= TMEM lanes), reduced through shared memory.
//
// fc1 has K = F + 4 <= 12.  Its inputs are the normalised features, which need
// more than bf16's 8 bits, so both x and w are split into bf16 hi + lo parts and
// the three products hi.hi + lo.hi + hi.lo are laid side by side along K
// (3 (F+4) <= 36 of the 64 columns of one K block).
//
// Precision modes: HB_PRECISION_BF16 rounds hidden activations and weights to bf16 (128
// queries per tile); HB_PRECISION_BF16X3 keeps hi + lo parts of both (64 queries per tile,
// the two parts of an activation side by side along N, the two parts of a weight tile one
// after the other in the ring: see the comment at the kernel).
//
// Warp roles: warp 0 = TMEM allocation, warp 1 = barrier set-up + MMA issuer (leader CTA),
// warps 2-5 and 12-15 = two epilogue groups (one TMEM lane quadrant per warp), warps 6-8 =
// weight producers, warps 9 and 10 = features (warp 11 times a copy).
// Every mbarrier wait is bounded: when a wait runs out the kernel records a status word, the roles
// leave their loops or run them empty (the two epilogue groups keep meeting at their common barriers, which
// have no limit of their own), outstanding bulk copies and MMAs are waited for (bounded) and TMEM is released.
// No ring slot is requested again that nobody has waited for: its copy could still be under way, and its barrier would be
// armed a second time in one phase.  So the MMA issuer, whose commits free the slots of both CTAs, waits for all
// producers to leave before it issues anything past a wait that ran out, and goes no further than the tile's end.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "mlp_common.cuh"
#include "mlp_wide.h"

namespace {

// One predictor and its batch of queries.
struct MlpProblem {
  const float* bias;         // [layers + 1][1024]: fc1, hidden...
  const float* fc2_w;        // [1024]
  float fc2_b;
  int32_t first_tile;        // of the launch's tiles
  const double* mu;          // [F + 4]
  const double* sigma;       // [F + 4]
  const double* dev_feat;    // [n_dev][4]
  int32_t n_dev;
  int32_t n_op_feat;         // F
  int32_t layers;            // hidden layers
  int32_t grid_n;            // > 0: query q is feature row q % grid_n on device grid_rows[q / grid_n]
  const float* feats;        // [Q][F]
  const uint8_t* dev_row;    // [Q]
  int64_t Q;
  float* out;                // [Q]
  int32_t* status;           // 0 ok, else (role << 8 | site)
  uint8_t grid_rows[hb::kMaxGridRows];
  CUtensorMap tmap_tile;     // the weight pack as [rows][128 B], box of one tile image (16 KB)
};
// A launch takes the tiles of up to four predictors, one after the other in one list, so that only the
// list's end leaves SMs idle.
struct MlpParams {
  int32_t num_tiles;
  int32_t n_problems;
  int32_t beside;            // runs beside the launch before it on the stream: nothing to wait for
  long long* phase_cycles;   // [16] cluster 0: cycle counters of the roles (diagnostic), or null
  MlpProblem prob[hb::kMaxLanes];
};
__device__ __forceinline__ const MlpProblem& problem_of(const MlpParams& p, int tile) {
  int k = 0;
  for (int i = 1; i < p.n_problems; ++i) k += tile >= p.prob[i].first_tile ? 1 : 0;
  return p.prob[k];
}

// ---------------------------------------------------------------------------
// The kernel.  A single CTA can only keep 64 queries on chip,
// and an M = 128 MMA with N = 64 occupies the tensor core for the same 64 cycles
// as one with N = 128, so the one-CTA kernel tops out at half rate.  Here two
// CTAs of a cluster share one tile of 128 queries:
//   * tcgen05.mma.cta_group::2 with M = 256, N = 128: CTA c supplies the A rows
//     (weights) of features 256 j + 128 c .. and the B rows (activations) of
//     queries 64 c .. 64 c + 63; its TMEM receives the D rows of its features
//     for all 128 queries.  Each weight byte is fetched once per pair.
//   * The leader CTA (rank 0) issues every MMA.  A ring slot is ready when the
//     leader's weight box and the peer's have landed: both are tiled TMA loads
//     (cp.async.bulk.tensor with .cta_group::2, no multicast) whose bytes are
//     counted on the leader's barrier, so no thread of the peer has to forward
//     anything.  tcgen05.commit multicasts "slot free" and "output block j
//     accumulated" to both CTAs.
//   * The activations are the MN-major B operand here (one 128-byte row of 64
//     queries per K index): an epilogue thread owns one feature = one K row
//     and writes eight queries per 16-byte store.
//   * The epilogue of CTA c holds features x all 128 queries, but the next
//     layer needs, in each CTA, all features x its 64 queries: half of the
//     bf16 results are stored into the peer's shared memory (st.async, counted
//     in bytes on a barrier of the peer).
//   * Epilogue and tensor core overlap: a hidden layer is issued as 16 units
//     (output block, K quarter) in the order kPairOrder, so that output blocks
//     finish one after the other and each frees the K quarter it will replace.
//     The leader waits per K quarter (bar_actq) and per TMEM block (bar_tfree)
//     instead of per layer; only the drain of the last block is exposed.
//   * fc2: each CTA reduces its 512 features to 128 partial sums, hands the 64
//     that belong to the peer's queries over through the peer's shared memory,
//     and finishes its own 64 queries.
// ---------------------------------------------------------------------------
constexpr int kPairQ = 128;                 // queries per cluster tile
constexpr int kPairHalfQ = 64;              // activation rows resident per CTA
constexpr int kPairMT = kWidth / 256;       // 4 MMA row blocks per layer
// Ring of weight tiles, 96 KB in all.  From the commit that frees a slot to its next tile in place it takes 1,100 to
// 1,300 cycles (710 to 900 of them the copy), while a tile lasts the tensor core 256.  Three slots of 32 KB with a
// producer each did not cover that; six of 16 KB do, just: 65,536 split queries 3,251 -> 3,084 us, 4,194,304 of
// bf16 57.0 -> 55.8 ms.
constexpr int kPairStages = 6;
constexpr int kPairProducers = 3;            // warps 6-8, two slots each; six measured the same, two 2 % slower (split)
constexpr int kPairStageBytes = kTileBytes;
static_assert(kPairStages == 2 * kPairProducers && kPairProducers == 3, "warps 6-8, two slots each");
constexpr int kPairActKb = kPairHalfQ * 128;          // 8 KB per K block
constexpr int kPairActBytes = kNumKB * kPairActKb;    // 128 KB
// Order of the 16 (output block j, K quarter q) units of a hidden layer, four bits each
// (4 j + q), first unit in the low bits:
//   (0,0) (0,1) (1,0) (1,1) (2,0) (3,0) (0,2) (0,3) | (2,1) (3,1) (1,2) (1,3) | (2,2) (3,2) (2,3) | (3,3)
// Block j completes after 8, 12, 15, 16 units, and by then no later unit reads quarter j,
// so the epilogue of block j can replace quarter j of the activations in place while the
// tensor core works on the remaining blocks; the next layer consumes the quarters in the
// same order.  What the last epilogues of a layer hold up, TMEM blocks 2 and 3 and quarters 2 and 3, comes
// as late as that allows in the next one, after five to seven units of 1,024 cycles.
// 109.1 -> 106.3 us for one round of tiles (with (1,0) (2,0) (3,0) in units 1 to 3 the issuer waited 2,700 cycles a
// layer for TMEM blocks); split precision, whose units last twice as long, takes the same time either way.
constexpr uint64_t kPairOrder = 0xFBEA76D932C85410ull;
constexpr uint32_t kPairFirstOfBlock = 0x35;     // units that write a TMEM block for the first time in the layer
constexpr uint32_t kPairFirstOfQuarter = 0xC3;   // ... that read a K quarter for the first time
constexpr uint32_t kPairLastOfBlock = 0xC880;    // ... that complete a block
constexpr int kPairThreads = 512;              // warps: 0 alloc, 1 MMA, 2-5 + 12-15 epilogue, 6-8 producers, 9-10 features
constexpr int kPairSmemBytes = kPairActBytes + kPairStages * kPairStageBytes + 1024 + 1024;
static_assert(kPairSmemBytes <= 232448, "over the 227 KB shared-memory limit");

__device__ __forceinline__ void pair_epi_bar_sync() {
  asm volatile("bar.sync 1, 256;" ::: "memory");
}
// SPLIT = false: bf16 operands, 128 queries per cluster tile (64 per CTA).
// SPLIT = true (the 1e-4 mode): activations and weights are kept as bf16 hi + lo parts.  A CTA
// holds 32 queries and lays the hi and lo parts of an activation side by side along N (the 128-byte
// B row of K index k is [hi of 32 queries | lo of 32 queries]), so the same M = 256, N = 128 MMA
// multiplies a weight tile with both parts at once, at full rate; the hi and the lo image of a K block
// of weights follow one another through the ring and accumulate into the same TMEM columns:
// D = (W_hi + W_lo) [x_hi | x_lo], and the epilogue adds the two column halves of a query (all four
// partial products, fp32 accumulation).  Two MMAs per K step and 64 queries instead of one and 128:
// a quarter of the bf16 rate.
template <bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
mlp_chain_pair_kernel(const __grid_constant__ MlpParams p) {
  constexpr int kTileQ = SPLIT ? kPairQ / 2 : kPairQ;          // queries per cluster tile
  constexpr int kHalfQ = kTileQ / 2;                           // queries per CTA
  constexpr int kLoadsPerUnit = SPLIT ? 8 : 4;                 // ring slots per (block, K quarter) unit
  constexpr int kRowsPerImage = (SPLIT ? 2 : 1) * (kTileBytes / 128);   // 128-byte rows per packed K block
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);

  const uint32_t act = base;
  const uint32_t stage0 = base + kPairActBytes;
  const uint32_t bars = stage0 + kPairStages * kPairStageBytes;
  uint8_t* bars_ptr = base_ptr + (bars - base);
  // barrier block (same offsets in both CTAs)
  const uint32_t bar_full = bars;            // [stages <= 8] leader only: both CTAs' weight boxes landed
  const uint32_t bar_empty = bars + 64;      // [stages <= 8] slot consumed (multicast commit)
  const uint32_t bar_accj = bars + 128;      // [4] output block j accumulated (multicast commit)
  const uint32_t bar_actq = bars + 160;      // [4] leader only: K quarter q of the activations ready in both CTAs
  const uint32_t bar_inq = bars + 192;       // [4] peer's half of K quarter q landed here (bytes)
  const uint32_t bar_tfree = bars + 224;     // [4] leader only: TMEM block j read out in both CTAs (8 warps)
  const uint32_t bar_fc2 = bars + 256;       // peer's fc2 partial sums arrived
  const uint32_t bar_next = bars + 264;      // the tile is done with the activation buffer (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_ptr + 272);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars_ptr + 276);
  volatile int* epi_ok = reinterpret_cast<volatile int*>(bars_ptr + 280);   // [5]: per epilogue group, twice; the hand-over of fc2
  const uint32_t bar_drain = bars + 304;     // leader only, after giving up: the MMAs have ended
  volatile int* producers_left = reinterpret_cast<volatile int*>(bars_ptr + 312);   // [2 * kPairProducers] leader only
  float* fc2_mine = reinterpret_cast<float*>(bars_ptr + 512);    // [64] own queries, own features
  float* fc2_peer = reinterpret_cast<float*>(bars_ptr + 768);    // [64] own queries, peer's features

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const uint32_t peer = rank ^ 1u;

  if (threadIdx.x == 32) {
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(bar_full + 8 * s, 1);   // used in the leader only: its producer's arrive.expect_tx
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int q = 0; q < 4; ++q) {
      mbar_init(bar_accj + 8 * q, 1);
      mbar_init(bar_actq + 8 * q, 2);   // one arrive per CTA
      mbar_init(bar_inq + 8 * q, 1);
      mbar_init(bar_tfree + 8 * q, 8);  // one arrive per epilogue warp of the block, both CTAs
    }
    mbar_init(bar_fc2, 1);
    mbar_init(bar_next, 8);
    mbar_init(bar_drain, 1);
    *abort_flag = 0;
    for (int i = 0; i < 2 * kPairProducers; ++i) producers_left[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  grid_begin(p.beside != 0);   // the set-up above overlaps the end of the launch before it on the stream
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int n_pairs = static_cast<int>(gridDim.x >> 1);
  const int pair_id = static_cast<int>(blockIdx.x >> 1);
  int my_tiles = 0;
  if (pair_id < p.num_tiles) my_tiles = (p.num_tiles - 1 - pair_id) / n_pairs + 1;

  uint32_t issued = 0;
  auto publish = [&](uint32_t q) {   // "this CTA's share of K quarter q is in place"
    const uint32_t bar = bar_actq + 8 * q;
    if (rank == 0) mbar_arrive(bar);
    else mbar_arrive_remote(map_to_cta(bar, 0));
  };

  if (warp >= 6 && warp < 6 + kPairProducers) {
    // ------------------------------ producers -----------------------------
    // The pack is laid out per 128-feature block (layer -> block -> K block); this CTA streams blocks 2 j + rank,
    // a hidden layer as 16 (block, K quarter) units of four K blocks each (fc1 has only one).  What a load needs
    // is worked out before the wait for its slot, so that only the request stands between the two (a dozen
    // instructions more there cost the split mode 4 %).
    if (lane == 0) {
      constexpr int kLayerLoads = 16 * kLoadsPerUnit;
      const uint32_t w = static_cast<uint32_t>(warp - 6);
      uint32_t s = w, ph = 1;
      uint32_t n = w;              // load of the tile
      bool ok = true;
      const bool timed = p.phase_cycles != nullptr && blockIdx.x == 0 && w == 0;
      long long c_empty = 0;
      for (int t = 0; t < my_tiles && ok; ++t) {
        const MlpProblem& pb = problem_of(p, pair_id + t * n_pairs);
        const uint32_t tile_loads = static_cast<uint32_t>(kPairMT + pb.layers * kLayerLoads);
        for (; n < tile_loads; n += kPairProducers) {
          uint32_t image = 2 * n + rank, g = 0;              // fc1: block n
          if (n >= kPairMT) {
            const uint32_t m = n - kPairMT, L = m / kLayerLoads, u = m % kLayerLoads / kLoadsPerUnit;
            const uint32_t unit = static_cast<uint32_t>(kPairOrder >> (4 * u)) & 15u;
            g = m % kLoadsPerUnit;
            image = kNumMT + (L * kNumMT + 2 * (unit >> 2) + rank) * kNumKB + (unit & 3u) * 4;
          }
          // split: a K block's hi and lo image are stored back to back
          const int32_t row = static_cast<int32_t>(image * kRowsPerImage + g * (kTileBytes / 128));
          const uint32_t dst = stage0 + s * kPairStageBytes, full = bar_full + 8 * s;
          const uint32_t full_leader = map_to_cta(full, 0);   // both CTAs' boxes are counted there
          const long long c0 = timed ? clock64() : 0;
          if (!mbar_wait(bar_empty + 8 * s, ph, abort_flag, pb.status, 0x111)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(full, 2 * kPairStageBytes);
          tma_rows_2sm(dst, &pb.tmap_tile, row, full_leader);
          if (timed) c_empty += clock64() - c0;   // (a copy that is waited for here, to time it, holds up the ring)
          ++issued;
          s += kPairProducers;
          if (s >= kPairStages) { s = w; ph ^= 1u; }
        }
        n -= tile_loads;
      }
      st_cluster_u32(map_to_cta(bars + 312 + 4 * (kPairProducers * rank + w), 0), 1u);
      if (timed) { p.phase_cycles[9] = c_empty; p.phase_cycles[11] = issued; }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ------------------------------ MMA issuer (leader) -------------------
      // One elected lane (elect.sync) runs the whole loop, and no loop of a tile depends on what a wait returns
      // (after a wait that ran out the abort flag is set, and what is issued on stale operands is
      // discarded), which keeps the descriptors in uniform registers: four MMAs and their commit are
      // queued in about 100 cycles of the 256 they take.  The barrier of the next slot is tested while they run.
      // D fp32, A/B bf16, A K-major, B MN-major (bit 16), N = 128, M = 256
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) |
                                 (static_cast<uint32_t>(kPairQ >> 3) << 17) |
                                 (static_cast<uint32_t>(256 >> 4) << 24);
      const uint64_t desc_hi = (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                               (static_cast<uint64_t>(2) << 61) | (static_cast<uint64_t>(1) << 16);
      const uint32_t a_lo0 = (stage0 & 0x3FFFF) >> 4;
      const uint32_t b_lo0 = (act & 0x3FFFF) >> 4;
      if (elect_one()) {
        // par: bits 0-3 = parity of the next wait on bar_actq[q], bits 4-7 on bar_tfree[j]
        uint32_t s = 0, ph = 0, par = 0;
        const bool mtimed = p.phase_cycles != nullptr && blockIdx.x == 0;
        long long mc_act = 0, mc_full = 0, mc_tfree = 0, mc_n = 0;
        int32_t* status = nullptr;
        auto gave_up = [&] {   // (the producers look at their CTA's abort flag when a slot does not come)
          st_cluster_u32(map_to_cta(bars + 276, 1), 1u);
          const long long t0 = clock64();
          for (int i = 0; i < 2 * kPairProducers; ++i)
            while (producers_left[i] == 0 && clock64() - t0 <= kWaitCycles) {}
        };
        auto wait = [&](uint32_t bar, uint32_t parity, long long& acc, int code) {
          const long long m0 = mtimed ? clock64() : 0;
          if (!mbar_wait_cluster(bar, parity, abort_flag, status, code)) gave_up();
          tc_fence_after();
          if (mtimed) acc += clock64() - m0;
        };
        const long long k0 = clock64();
        const unsigned long long g0 = global_timer_ns();
#pragma unroll 1
        for (int t = 0; t < my_tiles && *abort_flag == 0; ++t) {
          const MlpProblem& pb = problem_of(p, pair_id + t * n_pairs);
          const int n_layers = pb.layers + 1;
          status = pb.status;
          // fc1 reads K block 0, written after the previous tile's TMEM was read out
          wait(bar_actq, par & 1u, mc_act, 0x211);
          par ^= 1u;
#pragma unroll 1
          for (int j = 0; j < kPairMT; ++j) {
            wait(bar_full + 8 * s, ph, mc_full, 0x212);
            const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(j * kPairQ);
            const uint32_t a_lo = a_lo0 + s * (kPairStageBytes >> 4);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tc_mma_pair_bf16(d_tmem, desc_hi | (a_lo + 2 * k), desc_hi | (b_lo0 + 128 * k), idesc, k ? 1u : 0u);
            tc_commit_pair(bar_accj + 8 * j);
            tc_commit_pair(bar_empty + 8 * s);
            ring_next<kPairStages>(s, ph);
          }
#pragma unroll 1
          for (int L = 1; L < n_layers; ++L) {
            bool landed = false;            // the barrier of slot s has been seen complete
#pragma unroll 1
            for (uint32_t u = 0; u < 16; ++u) {
              const uint32_t unit = ((u < 8 ? static_cast<uint32_t>(kPairOrder) : static_cast<uint32_t>(kPairOrder >> 32)) >>
                                     (4 * (u & 7u))) & 15u;
              const uint32_t j = unit >> 2, kq = unit & 3u;
              if (u < 8) {
                // (the previous layer's values must be out)
                if ((kPairFirstOfBlock >> u) & 1u) {
                  wait(bar_tfree + 8 * j, (par >> (4 + j)) & 1u, mc_tfree, 0x213);
                  par ^= 16u << j;
                }
                if ((kPairFirstOfQuarter >> u) & 1u) {
                  wait(bar_actq + 8 * kq, (par >> kq) & 1u, mc_act, 0x211);
                  par ^= 1u << kq;
                }
              }
              const uint32_t d_tmem = tmem_base + j * kPairQ;
#pragma unroll
              for (uint32_t g = 0; g < kLoadsPerUnit; ++g) {
                uint32_t next = s, next_ph = ph;
                ring_next<kPairStages>(next, next_ph);
                const uint32_t a_lo = a_lo0 + s * (kPairStageBytes >> 4);
                const uint32_t b_lo = b_lo0 + (kq * 4 + (SPLIT ? g >> 1 : g)) * (kPairActKb >> 4);
                if (!landed) wait(bar_full + 8 * s, ph, mc_full, 0x212);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  // a K step of 16: 32 bytes along an A row, 16 K rows (2 KB) of B
                  tc_mma_pair_bf16(d_tmem, desc_hi | (a_lo + 2 * k), desc_hi | (b_lo + 128 * k), idesc,
                                   (g == 0 && k == 0) ? kq : 1u);
                  if (k == 1) {
                    landed = mbar_try_wait_cluster(bar_full + 8 * next, next_ph);
                    tc_fence_after();
                  }
                }
                tc_commit_pair(bar_empty + 8 * s);
                s = next;
                ph = next_ph;
              }
              if ((kPairLastOfBlock >> u) & 1u) tc_commit_pair(bar_accj + 8 * j);
            }
            mc_n += 16 * kLoadsPerUnit;
          }
        }
        if (mtimed) {
          p.phase_cycles[4] = mc_act; p.phase_cycles[5] = mc_full; p.phase_cycles[6] = mc_tfree;
          p.phase_cycles[8] = mc_n;
          p.phase_cycles[12] = clock64() - k0;
          p.phase_cycles[7] = p.phase_cycles[12] - mc_act - mc_full - mc_tfree;
          p.phase_cycles[13] = static_cast<long long>(global_timer_ns() - g0);
        }
      }
      __syncwarp();
    }
  } else if (warp == 11) {
    // diagnostic: how long the first copy takes, requested about now
    if (lane == 0 && p.phase_cycles != nullptr && blockIdx.x == 0 && my_tiles > 0) {
      const long long t0 = clock64();
      mbar_wait(bar_full, 0, abort_flag, problem_of(p, pair_id).status, 0x112);
      p.phase_cycles[10] = clock64() - t0;
    }
  } else if (warp == 9 || warp == 10) {
    // ------------------------------ features ------------------------------
    // One B column (query) per thread.  The next tile's features are loaded, normalised (float64) and split
    // into bf16 hi + lo while the tensor core works on the current tile; at the tile's end only the stores
    // are left.  SPLIT: columns 32..63 are the lo parts of the hidden layers; fc1 carries its own hi/lo
    // expansion along K, so they are zero here.
    const int T = static_cast<int>(threadIdx.x) - 9 * 32;
    for (int t = 0; t < my_tiles; ++t) {
      const int tile = pair_id + t * n_pairs;
      const MlpProblem& pb = problem_of(p, tile);
      const int C_in = pb.n_op_feat + 4;
      const int64_t q = static_cast<int64_t>(tile - pb.first_tile) * kTileQ + static_cast<int64_t>(rank) * kHalfQ + T;
      uint32_t x2[kMaxInFeat];             // hi | lo << 16
#pragma unroll
      for (int c = 0; c < kMaxInFeat; ++c) x2[c] = 0;
      if (T < kHalfQ && q < pb.Q) {
        int64_t fr = q;
        int dr;
        if (pb.grid_n) {
          const uint32_t block = static_cast<uint32_t>(q) / static_cast<uint32_t>(pb.grid_n);
          fr -= static_cast<int64_t>(block) * pb.grid_n;
          dr = pb.grid_rows[block];
        } else {
          dr = pb.dev_row[q];
        }
        dr = dr < pb.n_dev ? dr : pb.n_dev - 1;
#pragma unroll
        for (int c = 0; c < kMaxInFeat; ++c) {
          if (c >= C_in) continue;
          const double x = c < pb.n_op_feat ? static_cast<double>(pb.feats[fr * pb.n_op_feat + c])
                                            : pb.dev_feat[dr * 4 + (c - pb.n_op_feat)];
          const float xn = static_cast<float>((x - pb.mu[c]) / pb.sigma[c]);
          const __nv_bfloat16 hi = __float2bfloat16_rn(xn);
          const __nv_bfloat16 lo = __float2bfloat16_rn(xn - __bfloat162float(hi));
          x2[c] = static_cast<uint32_t>(__bfloat16_as_ushort(hi)) | static_cast<uint32_t>(__bfloat16_as_ushort(lo)) << 16;
        }
      }
      if (t > 0) {
        if (lane == 0) mbar_wait(bar_next, (t - 1) & 1, abort_flag, pb.status, 0x411);
        __syncwarp();
      }
      // K rows: [hi | lo | hi], then zeros (row k, query n: 128 k + 16 ((n / 8) xor (k mod 8)) + 2 (n mod 8))
      for (int i = T; i < (kKBlk - 3 * C_in) * 8; i += 64)
        *reinterpret_cast<uint4*>(base_ptr + 3 * C_in * 128 + 16 * i) = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int c = 0; c < kMaxInFeat; ++c) {
        if (c >= C_in) continue;
        const uint16_t hi = static_cast<uint16_t>(x2[c]), lo = static_cast<uint16_t>(x2[c] >> 16);
        *reinterpret_cast<uint16_t*>(base_ptr + mn_off(c, T)) = hi;
        *reinterpret_cast<uint16_t*>(base_ptr + mn_off(C_in + c, T)) = lo;
        *reinterpret_cast<uint16_t*>(base_ptr + mn_off(2 * C_in + c, T)) = hi;
      }
      fence_proxy_async();
      asm volatile("bar.sync 4, 64;" ::: "memory");
      if (T == 0) publish(0);
    }
  } else if (warp >= 2 && (warp < 6 || warp >= 12)) {
    // ------------------------------ epilogue ------------------------------
    // Two groups of four warps (warps 2-5 and 12-15); a warp may only read the
    // TMEM lane quadrant (warp id mod 4).  Group g drains the 256-feature blocks
    // g and g + 2 of a hidden layer (2 g and 2 g + 1 under fc2).
    const int grp = warp >= 12 ? 1 : 0;
    const int e = (warp - (grp ? 12 : 2)) * 32 + lane;   // 0..127 inside the group
    const int T = grp * 128 + e;                         // 0..255 over both groups
    const int quad = warp & 3;
    const int r = quad * 32 + lane;            // feature row inside this CTA's 128-row block
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t act_peer = map_to_cta(act, peer);
    uint32_t in_phase = 0, lay = 0, tile_no = 0;
    bool ok = true, in_order = true;           // in_order (e == 0): no wait for the peer's half of a quarter has run out
    float* red = reinterpret_cast<float*>(base_ptr);   // [8 warps][queries of the tile], aliases activations
    const bool timed = p.phase_cycles != nullptr && blockIdx.x == 0 && T == 0;
    long long c_wait = 0, c_epi = 0, c_fc2 = 0, c_layers = 0, c_ld = 0, c_bias = 0, c_sync = 0, c_loc = 0, c_rem = 0;
    // named barrier of this group alone (ids 2 and 3; id 1 joins both groups)
    auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory"); };
    for (int t = 0; t < my_tiles; ++t, ++tile_no) {
      const int tile = pair_id + t * n_pairs;
      const MlpProblem& pb = problem_of(p, tile);
      const int n_layers = pb.layers + 1;
      const int64_t q0 = static_cast<int64_t>(tile - pb.first_tile) * kTileQ + static_cast<int64_t>(rank) * kHalfQ;

      for (int L = 0; L < n_layers; ++L, ++lay) {
        const float* bias = pb.bias + L * kWidth;
        const bool last = (L == n_layers - 1);
        if (!last) {
          if (!ok) continue;
          // Group g drains output blocks g and g + 2.  Block j becomes K quarter j of the next
          // layer and is written over the current activations in place: in the unit order of a
          // hidden layer nothing reads quarter j once block j is complete.  Under fc1 the input
          // sits in quarter 0 until the last block is done, so everything waits for that.
#pragma unroll 1
          for (int jj = 0; jj < 2; ++jj) {
            const int j = grp + 2 * jj;
            const int gate = L == 0 ? 3 : j;
            const long long c0 = timed ? clock64() : 0;
            if (e == 0) {
              const bool go = in_order && mbar_wait(bar_accj + 8 * gate, lay & 1u, abort_flag, pb.status, 0x311);
              epi_ok[grp] = go ? 1 : 0;
              // the peer sends 128 K rows x 128 B of this quarter into this CTA
              if (go) mbar_expect_tx(bar_inq + 8 * j, 128u * 128u);
            }
            group_sync();
            if (epi_ok[grp] == 0) { ok = false; break; }
            tc_fence_after();
            const long long c1 = timed ? clock64() : 0;
            const int f = j * 256 + static_cast<int>(rank) * 128 + r;   // feature = next layer's K index
            const long long d0 = timed ? clock64() : 0;
            const float b = __ldg(bias + f);
            if (timed) { c_bias += clock64() - d0 + static_cast<long long>(b == 12345.0f); }
            const uint32_t row_off = static_cast<uint32_t>(f) * 128u;   // K row f of the next layer's B operand
            const uint32_t sw = static_cast<uint32_t>(f) & 7u;
            const uint32_t bar_in_peer = map_to_cta(bar_inq + 8 * j, peer);
            const uint32_t bar_tfree_leader = map_to_cta(bar_tfree + 8 * j, 0);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {         // 64 queries = one CTA's share per load
              // the peer's half first: it has the longer way to go
              const bool mine = hh == 1;
              const uint32_t h = mine ? rank : peer;
              float v[64];
              const long long d1 = timed ? clock64() : 0;
              tc_ld64(t_lane + static_cast<uint32_t>(j * kPairQ) + h * 64u, v);
              if (timed) c_ld += clock64() - d1;
              if (mine) {
                // this warp has read all of its lanes of block j: the next layer may overwrite them
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                  if (rank == 0) mbar_arrive(bar_tfree + 8 * j);
                  else mbar_arrive_remote(bar_tfree_leader);
                }
              }
              if (SPLIT) {
                // columns 0..31 hold W x_hi, 32..63 W x_lo of the same 32 queries: add them, then split
                // the activation into bf16 hi (columns 0..31 of the new row) and lo (32..63)
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                  const float x = fmaxf((v[i] + v[32 + i]) + b, 0.0f);
                  const float hi = __bfloat162float(__float2bfloat16_rn(x));
                  v[i] = hi;
                  v[32 + i] = x - hi;
                }
              } else {
#pragma unroll
                for (int i = 0; i < 64; ++i) v[i] = fmaxf(v[i] + b, 0.0f);
              }
              uint32_t w[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const __nv_bfloat162 pk = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&pk);
              }
              if (mine) {
#pragma unroll
                for (uint32_t g = 0; g < 8; ++g)             // eight values per 16-byte store
                  *reinterpret_cast<uint4*>(base_ptr + row_off + ((g ^ sw) << 4)) =
                      make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
              } else {
                // Into the peer go whole 128-byte rows: eight lanes trade chunks so that each store of theirs
                // fills one row.  Chunks of 32 different rows per store arrived one by one and held the
                // peer's shared memory long enough to stall its tensor core (831 -> 740 cycles per slot).
                trade_chunks<8>(w, lane);
                const uint32_t c8 = static_cast<uint32_t>(lane) & 7u;
                const uint32_t row8 = act_peer + (row_off - c8 * 128u);
#pragma unroll
                for (uint32_t g = 0; g < 8; ++g)
                  st_async_v4(row8 + g * 128u + ((c8 ^ g) << 4), w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3],
                              bar_in_peer);
              }
              if (timed) { if (mine) c_loc += clock64() - d1; else c_rem += clock64() - d1; }
            }
            const long long d2 = timed ? clock64() : 0;
            tc_fence_before();
            asm volatile("fence.proxy.async;" ::: "memory");   // local and peer shared memory
            group_sync();
            if (e == 0) {
              // own stores are fenced above; the peer's arrive as counted bytes
              in_order = mbar_wait_cluster(bar_inq + 8 * j, in_phase, abort_flag, pb.status, 0x313);
              if (in_order) publish(static_cast<uint32_t>(j));
            }
            if (timed) { c_wait += c1 - c0; c_epi += clock64() - c1; c_sync += clock64() - d2; }
          }
          in_phase ^= 1u;
          if (timed) ++c_layers;
        } else {
          // fc2 over this CTA's 512 features, a group's two blocks as they complete (the tensor core still
          // works on the later ones), 32 queries at a time (bf16: the four column quarters of the 128
          // queries; split: the two CTAs' 32 queries, hi and lo columns added first).  A warp multiplies its
          // 32 features of a block and adds them over its lanes with the transposing tree (31 shuffles leave
          // one query per lane); the eight warps' sums of a query meet in shared memory once, after all
          // columns and blocks.
          constexpr int kChunks = SPLIT ? 2 : 4;
          float part[kChunks];
#pragma unroll
          for (int i = 0; i < kChunks; ++i) part[i] = 0.0f;
          long long c1 = 0;
#pragma unroll 1
          for (int jj = 0; jj < 3 && ok; ++jj) {
            // third round: everything has been accumulated, the activation buffer is free
            const int j = jj < 2 ? grp + 2 * jj : 3;
            const long long c0 = timed ? clock64() : 0;
            if (e == 0) epi_ok[grp + 2 * (jj & 1)] = mbar_wait(bar_accj + 8 * j, lay & 1u, abort_flag, pb.status, 0x311) ? 1 : 0;
            group_sync();
            if (epi_ok[grp + 2 * (jj & 1)] == 0) { ok = false; break; }
            tc_fence_after();
            c1 = timed ? clock64() : 0;
            if (timed) c_wait += c1 - c0;
            if (jj == 2) break;
            const int f = j * 256 + static_cast<int>(rank) * 128 + r;
            const float b = __ldg(bias + f);
            const float w = __ldg(pb.fc2_w + f);
#pragma unroll
            for (int qd = 0; qd < kChunks; ++qd) {
              float v[32];
              if (SPLIT) {
                float lo[32];
                tc_ld32(t_lane + static_cast<uint32_t>(j * kPairQ + qd * 64), v);
                tc_ld32(t_lane + static_cast<uint32_t>(j * kPairQ + qd * 64 + 32), lo);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] += lo[i];
              } else {
                tc_ld32(t_lane + static_cast<uint32_t>(j * kPairQ + qd * 32), v);
              }
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __fmul_rn(w, fmaxf(v[i] + b, 0.0f));
              fold16(v, lane);
              fold_lanes<2>(v, lane, 16);
              part[qd] += v[0];
            }
            if (timed) c_fc2 += clock64() - c1;
          }
          // from here on both groups take part, also one that gave up
          if (ok) {
#pragma unroll
            for (int qd = 0; qd < kChunks; ++qd)
              red[(grp * 4 + quad) * (kChunks * 32) + qd * 32 + fold16_col<32>(lane) + (lane >> 4)] = part[qd];
          }
          pair_epi_bar_sync();
          float tot = 0.0f;
          if (T < kChunks * 32) {
#pragma unroll
            for (int k2 = 0; k2 < 8; ++k2) tot += red[k2 * (kChunks * 32) + T];
          }
          // nothing of this tile is left in the activation buffer or in TMEM: the next tile's features may come
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_next);
          if (ok && T < kChunks * 32) {
            // which CTA owns the query, and its index among the owner's
            const uint32_t owner = static_cast<uint32_t>(T / kHalfQ);
            const int slot = T % kHalfQ;
            if (owner == rank) fc2_mine[slot] = tot;
            else st_cluster_f32(map_to_cta(smem_u32(fc2_peer + slot), peer), tot);
          }
          pair_epi_bar_sync();
          // hand-over of the partial sums, then the owner finishes its 64 queries
          if (T == 0) {
            const bool all = *abort_flag == 0;   // both groups' sums are there
            if (all) mbar_arrive_remote(map_to_cta(bar_fc2, peer));
            epi_ok[4] = all && mbar_wait_cluster(bar_fc2, tile_no & 1u, abort_flag, pb.status, 0x312) ? 1 : 0;
          }
          pair_epi_bar_sync();
          ok = epi_ok[4] != 0;
          if (ok && T < kHalfQ) {
            const int64_t q = q0 + T;
            if (q < pb.Q) pb.out[q] = fc2_mine[T] + fc2_peer[T] + pb.fc2_b;
          }
          if (timed) { c_fc2 += clock64() - c1; ++c_layers; }
        }
      }
    }
    if (timed) {
      p.phase_cycles[0] = c_wait; p.phase_cycles[1] = c_epi;
      p.phase_cycles[2] = c_fc2; p.phase_cycles[3] = c_layers;
      p.phase_cycles[14] = c_sync; p.phase_cycles[15] = c_rem;
    }
  }

  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (rank == 0 && warp >= 6 && warp < 6 + kPairProducers && lane == 0 && *abort_flag && issued > 0) {
    // this producer's last copies, one per slot of its own
    const long long t0 = clock64();
    for (uint32_t i = 0; i < 2 && i < issued; ++i) {
      const uint32_t own = issued - 1 - i;
      const uint32_t s = static_cast<uint32_t>(warp - 6) + own % 2 * kPairProducers;
      while (!mbar_try_wait(bar_full + 8 * s, (own / 2) & 1u))
        if (clock64() - t0 > kWaitCycles) break;
    }
  }
  if (rank == 0 && warp == 1 && *abort_flag && elect_one()) {
    // and the MMAs, before the TMEM they write is somebody else's (the lane that issued them)
    tc_commit_pair(bar_drain);
    const long long t0 = clock64();
    while (!mbar_try_wait_cluster(bar_drain, 0) && clock64() - t0 <= kWaitCycles) {}
  }
  if (*abort_flag && threadIdx.x == 0) {
    // copies that the peer requested and the leader did not count
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {}
  }
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves while the other may still touch its memory
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
  }
  grid_end(p.beside != 0);
}

// ---------------------------------------------------------------------------
// Host side: weight packing and launch
// ---------------------------------------------------------------------------
uint16_t f32_to_bf16(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7F800000u) == 0x7F800000u && (u & 0x007FFFFFu)) return static_cast<uint16_t>((u >> 16) | 0x40);
  const uint32_t lsb = (u >> 16) & 1u;
  u += 0x7FFFu + lsb;
  return static_cast<uint16_t>(u >> 16);
}
float bf16_to_f32(uint16_t h) {
  const uint32_t u = static_cast<uint32_t>(h) << 16;
  float f;
  std::memcpy(&f, &u, 4);
  return f;
}

void put(uint8_t* tile, int row, int col, uint16_t v) {
  std::memcpy(tile + swz_off(static_cast<uint32_t>(row), static_cast<uint32_t>(col)), &v, 2);
}

}  // namespace

namespace {
// A tensor map of unswizzled bytes; dims, strides and box as cuTensorMapEncodeTiled takes them.
cudaError_t encode_bytes(CUtensorMap* map, void* base, uint32_t rank, const cuuint64_t* dims, const cuuint64_t* strides,
                         const cuuint32_t* box) {
  using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                CUtensorMapFloatOOBfill);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
  if (e != cudaSuccess) return e;
  if (fn == nullptr || found != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
  const cuuint32_t elem[3] = {1, 1, 1};
  return reinterpret_cast<EncodeFn>(fn)(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, base, dims, strides, box, elem,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? cudaSuccess
             : cudaErrorInvalidValue;
}
}  // namespace

cudaError_t hb::encode_rows(CUtensorMap* map, void* base, uint32_t row_bytes, uint64_t rows, uint32_t box_rows) {
  const cuuint64_t dims[2] = {row_bytes, rows}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {row_bytes, box_rows};
  return encode_bytes(map, base, 2, dims, strides, box);
}

cudaError_t hb::encode_images(CUtensorMap* map, void* base, uint64_t rows, uint32_t box_rows, uint32_t box_images) {
  const cuuint64_t dims[3] = {128, kTileBytes / 128, rows / (kTileBytes / 128)}, strides[2] = {128, kTileBytes};
  const cuuint32_t box[3] = {128, box_rows, box_images};
  return encode_bytes(map, base, 3, dims, strides, box);
}

extern "C" void hb_mlp_destroy(hb_mlp* h) {
  if (!h) return;
  if (h->counted) hb::wide_handle_destroyed(h->device);
  cudaFree(h->wpack); cudaFree(h->bias); cudaFree(h->fc2_w); cudaFree(h->mu);
  cudaFree(h->sigma); cudaFree(h->dev_feat); cudaFree(h->phase_cycles);
  if (h->status) cudaFreeHost(h->status);
  delete h;
}

extern "C" hb_status hb_mlp_create(hb_mlp** handle, int32_t n_op_features, int32_t layers,
                                   int32_t width, const float* fc1_w, const float* fc1_b,
                                   const float* hidden_w, const float* hidden_b,
                                   const float* fc2_w, const float* fc2_b, const double* mu,
                                   const double* sigma, const double* device_features,
                                   int32_t n_device_rows, int32_t precision) {
  if (!handle || !fc1_w || !fc1_b || (layers > 0 && (!hidden_w || !hidden_b)) || !fc2_w || !fc2_b ||
      !mu || !sigma || !device_features) {
    hb::set_error("hb_mlp_create: NULL argument");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (width < 1 || width > kWidth || layers < 1 || layers > 64 || n_op_features < 1 ||
      n_op_features + 4 > kMaxInFeat || n_device_rows < 1 || n_device_rows > 256 ||
      (precision != HB_PRECISION_BF16 && precision != HB_PRECISION_BF16X3)) {
    hb::set_error("hb_mlp_create: unsupported shape (1 <= width <= 1024, 1 <= F <= 8, 1 <= layers <= 64)");
    return HB_ERR_UNSUPPORTED;
  }
  // The kernel is built for 1024-wide layers.  A narrower network runs as a 1024-wide one whose
  // extra features have zero weights and zero bias: they stay 0 through every ReLU and add
  // nothing to any sum, so the results are those of the narrow network.
  std::vector<float> pad_fc1_w, pad_fc1_b, pad_hidden_w, pad_hidden_b, pad_fc2_w;
  if (width < kWidth) {
    const int C = n_op_features + 4;
    pad_fc1_w.assign(static_cast<size_t>(kWidth) * C, 0.0f);
    pad_fc1_b.assign(kWidth, 0.0f);
    pad_hidden_w.assign(static_cast<size_t>(layers) * kWidth * kWidth, 0.0f);
    pad_hidden_b.assign(static_cast<size_t>(layers) * kWidth, 0.0f);
    pad_fc2_w.assign(kWidth, 0.0f);
    std::memcpy(pad_fc1_w.data(), fc1_w, sizeof(float) * width * C);
    std::memcpy(pad_fc1_b.data(), fc1_b, sizeof(float) * width);
    std::memcpy(pad_fc2_w.data(), fc2_w, sizeof(float) * width);
    for (int L = 0; L < layers; ++L) {
      std::memcpy(&pad_hidden_b[static_cast<size_t>(L) * kWidth], hidden_b + static_cast<size_t>(L) * width,
                  sizeof(float) * width);
      for (int r = 0; r < width; ++r)
        std::memcpy(&pad_hidden_w[(static_cast<size_t>(L) * kWidth + r) * kWidth],
                    hidden_w + (static_cast<size_t>(L) * width + r) * width, sizeof(float) * width);
    }
    fc1_w = pad_fc1_w.data(); fc1_b = pad_fc1_b.data();
    hidden_w = pad_hidden_w.data(); hidden_b = pad_hidden_b.data();
    fc2_w = pad_fc2_w.data();
  }
  const bool split = precision == HB_PRECISION_BF16X3;
  const int C_in = n_op_features + 4;
  const size_t img = split ? 2 * kTileBytes : kTileBytes;
  const size_t n_img = kNumMT + static_cast<size_t>(layers) * kNumMT * kNumKB;
  std::vector<uint8_t> pack(n_img * img, 0);
  uint8_t* dst = pack.data();
  // fc1: [w_hi | w_hi | w_lo] along K, matching the activations' [x_hi | x_lo | x_hi]
  for (int mt = 0; mt < kNumMT; ++mt, dst += img) {
    for (int rr = 0; rr < kMTile; ++rr) {
      const float* wrow = fc1_w + static_cast<size_t>(mt * kMTile + rr) * C_in;
      for (int c = 0; c < C_in; ++c) {
        const uint16_t hi = f32_to_bf16(wrow[c]);
        const uint16_t lo = f32_to_bf16(wrow[c] - bf16_to_f32(hi));
        put(dst, rr, c, hi);
        put(dst, rr, C_in + c, hi);
        put(dst, rr, 2 * C_in + c, lo);
      }
    }
  }
  for (int L = 0; L < layers; ++L) {
    const float* W = hidden_w + static_cast<size_t>(L) * kWidth * kWidth;
    for (int mt = 0; mt < kNumMT; ++mt) {
      for (int kb = 0; kb < kNumKB; ++kb, dst += img) {
        for (int rr = 0; rr < kMTile; ++rr) {
          const float* wrow = W + static_cast<size_t>(mt * kMTile + rr) * kWidth + kb * kKBlk;
          for (int c = 0; c < kKBlk; ++c) {
            const uint16_t hi = f32_to_bf16(wrow[c]);
            put(dst, rr, c, hi);
            if (split) put(dst + kTileBytes, rr, c, f32_to_bf16(wrow[c] - bf16_to_f32(hi)));
          }
        }
      }
    }
  }

  hb_mlp* h = new hb_mlp();
  h->n_op_feat = n_op_features;
  h->layers = layers;
  h->precision = precision;
  h->n_dev = n_device_rows;
  h->fc2_b = fc2_b[0];
  auto fail = [&](cudaError_t e, const char* what) {
    hb_status st = hb::cuda_fail(e, what);
    hb_mlp_destroy(h);
    return st;
  };
  cudaError_t e;
  if ((e = cudaGetDevice(&h->device)) != cudaSuccess) return fail(e, "cudaGetDevice");
  if ((e = cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, h->device)) != cudaSuccess)
    return fail(e, "cudaDeviceGetAttribute");
  std::vector<float> bias(static_cast<size_t>(layers + 1) * kWidth);
  std::memcpy(bias.data(), fc1_b, sizeof(float) * kWidth);
  std::memcpy(bias.data() + kWidth, hidden_b, sizeof(float) * kWidth * layers);
#define HB_UP(field, src, bytes)                                                        \
  if ((e = cudaMalloc(reinterpret_cast<void**>(&h->field), (bytes))) != cudaSuccess)    \
    return fail(e, "cudaMalloc " #field);                                               \
  if ((e = cudaMemcpy(h->field, (src), (bytes), cudaMemcpyHostToDevice)) != cudaSuccess) \
    return fail(e, "cudaMemcpy " #field);
  HB_UP(wpack, pack.data(), pack.size());
  HB_UP(bias, bias.data(), bias.size() * sizeof(float));
  HB_UP(fc2_w, fc2_w, sizeof(float) * kWidth);
  HB_UP(mu, mu, sizeof(double) * C_in);
  HB_UP(sigma, sigma, sizeof(double) * C_in);
  HB_UP(dev_feat, device_features, sizeof(double) * 4 * n_device_rows);
#undef HB_UP
  // The pack as rows of 128 bytes for the tiled TMA loads.  The tile images are stored already swizzled, so the maps use
  // no swizzle of their own.
  const uint64_t pack_rows = pack.size() / 128;
  if ((e = hb::encode_rows(&h->tmap_tile, h->wpack, 128, pack_rows, kTileBytes / 128)) != cudaSuccess ||
      (e = hb::encode_images(&h->tmap_slot, h->wpack, pack_rows, 64, 4)) != cudaSuccess ||
      (e = hb::encode_images(&h->tmap_half_tile, h->wpack, pack_rows, 64, 1)) != cudaSuccess)
    return fail(e, "cuTensorMapEncodeTiled");
  if ((e = cudaHostAlloc(reinterpret_cast<void**>(&h->status), sizeof(int32_t), cudaHostAllocDefault)) != cudaSuccess)
    return fail(e, "cudaHostAlloc status");
  *h->status = 0;
  if ((e = cudaMalloc(reinterpret_cast<void**>(&h->phase_cycles), 16 * sizeof(long long))) != cudaSuccess)
    return fail(e, "cudaMalloc phase_cycles");
  if ((e = cudaMemset(h->phase_cycles, 0, 16 * sizeof(long long))) != cudaSuccess) return fail(e, "cudaMemset");
  e = cudaFuncSetAttribute(mlp_chain_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kPairSmemBytes);
  if (e != cudaSuccess) return fail(e, "cudaFuncSetAttribute");
  e = cudaFuncSetAttribute(mlp_chain_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kPairSmemBytes);
  if (e != cudaSuccess) return fail(e, "cudaFuncSetAttribute");
  hb::wide_handle_created(h->device);
  h->counted = true;
  *handle = h;
  return HB_OK;
}

namespace {
// A launch of the two-SM kernel: batches of predictors of one precision.
class ChainLaunch {
 public:
  ChainLaunch(const hb_mlp* h, bool split) : split_(split), pairs_(h->sm_count / 2) { p_.phase_cycles = h->phase_cycles; }
  int tile_q() const { return split_ ? kPairQ / 2 : kPairQ; }
  int64_t tiles_of(int64_t Q) const { return (Q + tile_q() - 1) / tile_q(); }
  // Rounds of tiles the SMs would walk with `more` tiles on top.
  int64_t rounds(int64_t more) const { return (p_.num_tiles + more + pairs_ - 1) / pairs_; }
  hb_status add(const hb_mlp* h, const hb::MlpBatch& batch) {
    const int64_t tiles = tiles_of(batch.Q);
    if (p_.n_problems == hb::kMaxLanes || tiles + p_.num_tiles > 0x7FFFFFFF || (batch.grid_n && batch.Q > 0xFFFFFFFFll)) {
      hb::set_error("hb_mlp_predict: Q too large for one launch");
      return HB_ERR_TOO_LARGE;
    }
    MlpProblem& q = p_.prob[p_.n_problems++];
    q.bias = h->bias; q.fc2_w = h->fc2_w; q.fc2_b = h->fc2_b; q.first_tile = p_.num_tiles;
    q.mu = h->mu; q.sigma = h->sigma; q.dev_feat = h->dev_feat; q.n_dev = h->n_dev;
    q.n_op_feat = h->n_op_feat; q.layers = h->layers; q.feats = batch.feats;
    q.dev_row = batch.dev_row; q.Q = batch.Q; q.out = batch.out; q.status = h->status;
    q.grid_n = batch.grid_n;
    if (batch.grid_n) std::memcpy(q.grid_rows, batch.grid_rows, static_cast<size_t>(batch.Q / batch.grid_n));
    q.tmap_tile = h->tmap_tile;
    p_.num_tiles += static_cast<int32_t>(tiles);
    return HB_OK;
  }
  // The queries at the end of the first batch without which the list has one round less (0: none).
  int64_t tail() const {
    const int64_t over = p_.num_tiles % pairs_, tiles = tiles_of(p_.prob[0].Q);
    if (over == 0 || over == p_.num_tiles || over >= tiles) return 0;
    return p_.prob[0].Q - (tiles - over) * tile_q();
  }
  void drop(int64_t queries) {
    const int32_t tiles = static_cast<int32_t>(tiles_of(p_.prob[0].Q) - tiles_of(p_.prob[0].Q - queries));
    p_.prob[0].Q -= queries;
    p_.num_tiles -= tiles;
    for (int i = 1; i < p_.n_problems; ++i) p_.prob[i].first_tile -= tiles;
  }
  hb_status go(bool beside, cudaStream_t s) {
    p_.beside = beside ? 1 : 0;
    // one cluster of two CTAs per tile (128 queries, 64 in split precision), at most one cluster per SM pair
    const int pairs = p_.num_tiles < pairs_ ? p_.num_tiles : pairs_;
    HB_CUDA_TRY(hb::launch_overlapped(split_ ? mlp_chain_pair_kernel<true> : mlp_chain_pair_kernel<false>,
                                      dim3(2 * pairs), dim3(kPairThreads), kPairSmemBytes, s, p_));
    return HB_OK;
  }

 private:
  bool split_;
  int pairs_;
  MlpParams p_{};
};

hb_status check_device(const hb_mlp* h) {
  int cur = -1;
  HB_CUDA_TRY(cudaGetDevice(&cur));
  if (cur == h->device) return HB_OK;
  // the weight pack, the tensor maps and the scratch live on the GPU the handle was created on
  hb::set_error("hb_mlp_predict: the handle belongs to CUDA device %d but device %d is current", h->device, cur);
  return HB_ERR_INVALID_ARGUMENT;
}

// HB_MLP_WIDE=0 keeps every batch on the two-SM kernel
hb::WidePlan plan_of(const hb_mlp* h, int64_t Q, bool alone = true) {
  static const bool use_wide = [] { const char* e = std::getenv("HB_MLP_WIDE"); return !e || std::atoi(e) != 0; }();
  return use_wide ? hb::wide_plan(Q, h->precision == HB_PRECISION_BF16X3, h->sm_count, alone) : hb::WidePlan{};
}

// A last round of few tiles takes as long as a full one, and the kernel for small batches is quicker: it takes the
// queries of that round from the first batch of the list (`batch`), the list follows beside it.  9,572 queries:
// 220 -> 135 us, 28,916: 435 -> 348; split, 5,792: 376 -> 282.
hb_status queue_tail(ChainLaunch* launch, hb_mlp* h, hb::MlpBatch batch, cudaStream_t s, int* launches) {
  const int64_t n = launch->tail();
  const hb::WidePlan plan = n ? plan_of(h, n) : hb::WidePlan{};
  if (plan.G == 0) return HB_OK;
  batch.first = batch.Q - n;
  batch.Q = n;
  batch.out += batch.first;
  bool launched = false;
  const hb_status st = hb::wide_predict(h, plan, batch, s, &launched);
  if (st == HB_OK && launched) {
    launch->drop(n);
    ++*launches;
  }
  return st;
}

// What the two-SM kernel takes for batches of n predictors as one list of tiles per precision, in us (8 hidden layers, as the
// times of the small-batch shapes).  Measured for one round: 107, 108 to 112, 113 to 117 and 114 to 120 for one to four
// predictors; split 171, 195, 215 to 226 and 226 to 229, whose weights (34 MB each) do not stay in L2 together.  Two lists run
// side by side when they fit, some 10 us slower.
int list_us(const int64_t* Q, const bool* split, int n, int sm_count) {
  const int64_t pairs = sm_count / 2;
  int64_t tiles[2] = {0, 0};
  int us[2] = {100, 165};
  for (int b = 0; b < n; ++b) {
    const int tile_q = split[b] ? kPairQ / 2 : kPairQ;
    tiles[split[b]] += (Q[b] + tile_q - 1) / tile_q;
    us[split[b]] += split[b] ? 16 : 4;
  }
  for (int k = 0; k < 2; ++k) us[k] *= static_cast<int>((tiles[k] + pairs - 1) / pairs);   // rounds, 0 without tiles
  if (tiles[0] == 0 || tiles[1] == 0) return us[0] + us[1];
  return tiles[0] + tiles[1] <= pairs ? std::max(us[0], us[1]) + 10 : us[0] + us[1];
}

// Queues one batch (checked by the callers) on the kernel for its size.  Call under wide_queue.
hb_status queue_batch(hb_mlp* h, const hb::WidePlan& plan, const hb::MlpBatch& batch, cudaStream_t s) {
  bool launched = false;
  hb_status st = check_device(h);
  if (st == HB_OK) st = hb::wide_predict(h, plan, batch, s, &launched);
  if (st != HB_OK || launched) return st;
  ChainLaunch launch(h, h->precision == HB_PRECISION_BF16X3);
  st = launch.add(h, batch);
  int launches = 0;
  if (st == HB_OK) st = queue_tail(&launch, h, batch, s, &launches);
  return st != HB_OK ? st : launch.go(batch.beside || launches > 0, s);
}
}  // namespace

extern "C" hb_status hb_mlp_predict(hb_mlp* h, const float* op_features, const uint8_t* device_row,
                                    int64_t Q, float* out, void* stream) {
  if (!h || Q < 0 || (Q > 0 && (!op_features || !device_row || !out))) {
    hb::set_error("hb_mlp_predict: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (Q == 0) return HB_OK;
  hb::MlpBatch batch;
  batch.feats = op_features; batch.dev_row = device_row; batch.Q = Q; batch.out = out;
  const auto queue = hb::wide_queue(h->device);
  return queue_batch(h, plan_of(h, Q), batch, static_cast<cudaStream_t>(stream));
}

extern "C" hb_status hb_mlp_predict_grid(const hb_mlp_grid* items, int32_t n_items, void* stream) {
  if (n_items < 0 || n_items > hb::kMaxLanes || (n_items > 0 && !items)) {
    hb::set_error("hb_mlp_predict_grid: 0 to %d batches", hb::kMaxLanes);
    return HB_ERR_INVALID_ARGUMENT;
  }
  for (int i = 0; i < n_items; ++i) {
    const hb_mlp_grid& g = items[i];
    if (!g.handle || g.n < 0 || g.n > 0x7FFFFFFF || g.n_device_rows < 0 || g.n_device_rows > hb::kMaxGridRows ||
        (g.n > 0 && g.n_device_rows > 0 && (!g.op_features || !g.device_rows || !g.out))) {
      hb::set_error("hb_mlp_predict_grid: bad batch %d (at most %d device rows)", i, hb::kMaxGridRows);
      return HB_ERR_INVALID_ARGUMENT;
    }
  }
  // The largest first: its launch waits for what is on the stream, the others run beside it.  Batches that
  // fill SM pairs go into one launch per precision, as one list of tiles; a smaller one joins the list when
  // it fits into the list's last round, else it gets a launch of its own.
  int order[hb::kMaxLanes] = {0, 1, 2, 3};
  auto queries = [&](int i) { return items[i].n * items[i].n_device_rows; };
  for (int i = 1; i < n_items; ++i)
    for (int j = i; j > 0 && queries(order[j]) > queries(order[j - 1]); --j) {
      const int t = order[j];
      order[j] = order[j - 1];
      order[j - 1] = t;
    }
  hb::MlpBatch batches[hb::kMaxLanes];
  bool queued[hb::kMaxLanes] = {};
  for (int i = 0; i < n_items; ++i) {
    const hb_mlp_grid& g = items[i];
    hb::MlpBatch& batch = batches[i];
    batch.feats = g.op_features; batch.Q = queries(i); batch.out = g.out;
    batch.grid_n = static_cast<int32_t>(g.n); batch.grid_rows = g.device_rows;
    queued[i] = batch.Q == 0;
    const hb_status st = batch.Q ? check_device(g.handle) : HB_OK;
    if (st != HB_OK) return st;
  }
  hb::WidePlan plans[hb::kMaxLanes];
  int64_t sizes[hb::kMaxLanes];
  bool split[hb::kMaxLanes], all_wide = true;
  int some = 0;   // batches with queries, the first ones in `order`
  for (; some < n_items && !queued[order[some]]; ++some) {
    const int i = order[some];
    plans[some] = plan_of(items[i].handle, batches[i].Q, n_items < 2 || queued[order[1]]);
    sizes[some] = batches[i].Q;
    split[some] = items[i].handle->precision == HB_PRECISION_BF16X3;
    all_wide = all_wide && plans[some].G != 0;
  }
  if (some == 0) return HB_OK;
  const auto queue = hb::wide_queue(items[order[0]].handle->device);   // the current device, as are the others'
  // Batches that each take most of the GPU follow one another on the small-batch kernels; one list of tiles can be sooner:
  // 1,956, 582 and 3,972 queries 160 -> 112 us, 498, 684, 1,650 and 492 in split precision 309 -> 220.
  if (all_wide && some > 1 &&
      hb::wide_plans_together(plans, sizes, split, some, items[order[0]].handle->sm_count) >
          list_us(sizes, split, some, items[order[0]].handle->sm_count)) {
    for (int k = 0; k < some; ++k) plans[k] = hb::WidePlan{};
  } else if (all_wide && some > 1) {
    // large clusters first: small ones spread over all GPCs and would leave no room for them
    for (int i = 1; i < some; ++i)
      for (int j = i; j > 0 && plans[j].G > plans[j - 1].G; --j) {
        std::swap(plans[j], plans[j - 1]);
        std::swap(order[j], order[j - 1]);
      }
  }
  int lane = 0;
  for (int k = 0; k < some; ++k) {
    const int i = order[k];
    if (queued[i]) continue;
    hb_mlp* h = items[i].handle;
    batches[i].lane = lane;
    batches[i].beside = lane > 0;
    ++lane;
    hb_status st = HB_OK;
    if (plans[k].G != 0) {
      st = queue_batch(h, plans[k], batches[i], static_cast<cudaStream_t>(stream));
      if (st != HB_OK) return st;
      continue;
    }
    ChainLaunch launch(h, h->precision == HB_PRECISION_BF16X3);
    for (int m = k; m < some && st == HB_OK; ++m) {
      const int o = order[m];
      const hb_mlp* other = items[o].handle;
      if (queued[o] || other->precision != h->precision) continue;
      const bool fills = plans[m].G == 0;
      if (m > k && !fills && launch.rounds(launch.tiles_of(batches[o].Q)) > launch.rounds(0)) continue;
      st = launch.add(other, batches[o]);
      queued[o] = true;
    }
    if (st == HB_OK) st = queue_tail(&launch, h, batches[i], static_cast<cudaStream_t>(stream), &lane);
    if (st == HB_OK) st = launch.go(lane > 1, static_cast<cudaStream_t>(stream));
    if (st != HB_OK) return st;
  }
  return HB_OK;
}

namespace {
// What the status word says about the launches that have ended.
hb_status read_status(hb_mlp* h, int32_t* device_status) {
  volatile int32_t* word = h->status;
  *device_status = *word;
  if (*device_status == 0) return HB_OK;
  // reported once: the word is cleared so that later launches are judged on their own
  *word = 0;
  hb::wide_start_over(h->device);
  hb::set_error("mlp kernel: a bounded device-side wait ran out (site 0x%x)", *device_status);
  return HB_ERR_DEVICE_TIMEOUT;
}
}  // namespace

extern "C" hb_status hb_mlp_status(hb_mlp* h, int32_t* device_status) {
  if (!h || !device_status) {
    hb::set_error("hb_mlp_status: NULL argument");
    return HB_ERR_INVALID_ARGUMENT;
  }
  HB_CUDA_TRY(cudaDeviceSynchronize());   // launches on non-blocking streams included
  return read_status(h, device_status);
}

extern "C" hb_status hb_mlp_poll_status(hb_mlp* h, int32_t* device_status) {
  if (!h || !device_status) {
    hb::set_error("hb_mlp_poll_status: NULL argument");
    return HB_ERR_INVALID_ARGUMENT;
  }
  return read_status(h, device_status);
}

extern "C" hb_status hb_mlp_inject_status(hb_mlp* h, int32_t device_status) {
  if (!h) {
    hb::set_error("hb_mlp_inject_status: NULL handle");
    return HB_ERR_INVALID_ARGUMENT;
  }
  HB_CUDA_TRY(cudaDeviceSynchronize());
  *static_cast<volatile int32_t*>(h->status) = device_status;
  return HB_OK;
}

extern "C" hb_status hb_mlp_inject_mark(hb_mlp* h) {
  if (!h) {
    hb::set_error("hb_mlp_inject_mark: NULL handle");
    return HB_ERR_INVALID_ARGUMENT;
  }
  const hb_status st = check_device(h);
  return st != HB_OK ? st : hb::wide_set_mark(h->device, 1);
}

extern "C" hb_status hb_mlp_inject_mark_at(hb_mlp* h, int32_t block) {
  if (!h || block < 0) {
    hb::set_error("hb_mlp_inject_mark_at: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  const hb_status st = check_device(h);
  return st != HB_OK ? st : hb::wide_set_mark(h->device, ~block);
}

extern "C" hb_status hb_mlp_inject_stale(hb_mlp* h) {
  if (!h) {
    hb::set_error("hb_mlp_inject_stale: NULL handle");
    return HB_ERR_INVALID_ARGUMENT;
  }
  hb::wide_expect_stale(h->device);
  return HB_OK;
}

extern "C" hb_status hb_mlp_inject_stale_at(hb_mlp* h, int32_t layer, int32_t feature, int32_t word) {
  if (!h || layer < 0 || feature < 0 || word < 0) {
    hb::set_error("hb_mlp_inject_stale_at: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (!hb::pairs_plant_words()) {
    hb::set_error("hb_mlp_inject_stale_at: this build plants no words (build with -DHB_BOUNDS_CHECK)");
    return HB_ERR_UNSUPPORTED;
  }
  hb::wide_plant_stale(h->device, layer, feature, word);
  return HB_OK;
}

extern "C" hb_status hb_mlp_second_runs(hb_mlp* h, int64_t* runs) {
  if (!h || !runs) {
    hb::set_error("hb_mlp_second_runs: NULL argument");
    return HB_ERR_INVALID_ARGUMENT;
  }
  const hb_status st = check_device(h);
  return st != HB_OK ? st : hb::wide_second_runs(h->device, runs);
}

extern "C" hb_status hb_mlp_phase_cycles(hb_mlp* h, int64_t out[16]) {
  if (!h || !out) {
    hb::set_error("hb_mlp_phase_cycles: NULL argument");
    return HB_ERR_INVALID_ARGUMENT;
  }
  long long v[16];
  HB_CUDA_TRY(cudaMemcpy(v, h->phase_cycles, sizeof(v), cudaMemcpyDeviceToHost));
  for (int i = 0; i < 16; ++i) out[i] = v[i];
  return HB_OK;
}

extern "C" hb_status hb_mlp_predict_host(hb_mlp* h, const float* op_features,
                                         const uint8_t* device_row, int64_t Q, float* out) {
  if (!h || Q < 0 || (Q > 0 && (!op_features || !device_row || !out))) {
    hb::set_error("hb_mlp_predict_host: bad arguments");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (Q == 0) return HB_OK;
  // staged through the per-GPU block and stream the `_host` entry points share
  hb::HostArena* arena = nullptr;
  hb_status st = hb::arena_for_current_device(&arena);
  if (st != HB_OK) return st;
  std::lock_guard<std::mutex> lock(arena->mu);
  const size_t q = static_cast<size_t>(Q), f_bytes = sizeof(float) * q * h->n_op_feat;
  cudaStream_t s = arena->stream;
  int cur = -1;
  HB_CUDA_TRY(cudaGetDevice(&cur));
  if (cur != h->device) return hb_mlp_predict(h, op_features, device_row, Q, out, s);   // says what is wrong
  // Up to kPinnedBytes the results are stored by the kernel itself into page-locked memory, which the host
  // watches, and small batches are read from there as well (or travel as kernel parameters): no copy, no
  // event, no synchronisation.  One query took 166 us with copies and two synchronisations.
  constexpr size_t kPinnedBytes = 4 << 20;
  if (f_bytes + 5 * q <= kPinnedBytes) {
    st = hb::arena_reserve_pinned(arena, f_bytes + 5 * q);
    if (st != HB_OK) return st;
    float* p_o = reinterpret_cast<float*>(arena->pinned);
    std::memset(p_o, 0xFF, 4 * q);
    float* p_f = p_o + q;
    uint8_t* p_r = reinterpret_cast<uint8_t*>(p_f) + f_bytes;
    hb::MlpBatch batch;
    batch.Q = Q; batch.out = p_o;
    const hb::WidePlan plan = plan_of(h, Q);
    batch.host_inputs = plan.G != 0 && Q <= hb::kWideInline;
    if (batch.host_inputs) {
      batch.feats = op_features;
      batch.dev_row = device_row;
    } else {
      std::memcpy(p_f, op_features, f_bytes);
      std::memcpy(p_r, device_row, q);
      batch.feats = p_f;
      batch.dev_row = p_r;
    }
    {
      const auto queue = hb::wide_queue(h->device);
      bool launched = false;
      st = hb::wide_predict(h, plan, batch, s, &launched);
      if (st != HB_OK) return st;
      if (!launched) {
        // the two-SM kernel reads a tile's features when it gets to the tile: they have to be near
        if (batch.host_inputs) {
          std::memcpy(p_f, op_features, f_bytes);
          std::memcpy(p_r, device_row, q);
          batch.host_inputs = false;
        }
        st = hb::arena_reserve(arena, f_bytes + q);
        if (st != HB_OK) return st;
        batch.feats = static_cast<float*>(arena->base);
        batch.dev_row = static_cast<uint8_t*>(arena->base) + f_bytes;
        HB_CUDA_TRY(cudaMemcpyAsync(arena->base, p_f, f_bytes + q, cudaMemcpyHostToDevice, s));
        st = queue_batch(h, hb::WidePlan{}, batch, s);
        if (st != HB_OK) return st;
      }
    }
    st = hb::wait_written(p_o, q, s);
    if (st != HB_OK) return st;
    int32_t code = 0;
    st = read_status(h, &code);
    if (st == HB_OK) std::memcpy(out, p_o, 4 * q);
    return st;
  }
  hb::Carver sizes(nullptr);
  sizes.take<float>(q * h->n_op_feat); sizes.take<uint8_t>(q); sizes.take<float>(q);
  st = hb::arena_reserve(arena, sizes.used());
  if (st != HB_OK) return st;
  hb::Carver c(arena->base);
  float* d_f = c.take<float>(q * h->n_op_feat);
  uint8_t* d_r = c.take<uint8_t>(q);
  float* d_o = c.take<float>(q);
  HB_CUDA_TRY(cudaMemcpyAsync(d_f, op_features, sizeof(float) * q * h->n_op_feat, cudaMemcpyHostToDevice, s));
  HB_CUDA_TRY(cudaMemcpyAsync(d_r, device_row, q, cudaMemcpyHostToDevice, s));
  st = hb_mlp_predict(h, d_f, d_r, Q, d_o, s);
  if (st != HB_OK) return st;
  HB_CUDA_TRY(cudaMemcpyAsync(out, d_o, sizeof(float) * q, cudaMemcpyDeviceToHost, s));
  HB_CUDA_TRY(cudaStreamSynchronize(s));
  int32_t code = 0;
  return hb_mlp_status(h, &code);
}
