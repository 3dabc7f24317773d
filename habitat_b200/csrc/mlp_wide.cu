// MLP inference for few queries: the layers' features are spread over the SMs, and sixteen thread blocks exchange them
// through distributed shared memory; and the choice of kernel for every batch that does not fill the GPU.
//
// Sixteen thread blocks form a group (one cluster) that owns up to six queries (two in split precision); block c computes
// output features 64 c .. of every layer for them and streams only their weights.
//
// Formulation as in mlp_chain.cu, H^T = W . X^T with tcgen05.mma (cta_group::1): A = weight rows (M = 64), B =
// activations (K-major, 8 or 16 columns), D = fp32 in TMEM.  K is walked in the same order and fc2 adds in the same order as
// there, so all kernels give the same bits and the choice of kernel never shows in a result.
//
// Exchange.  B is K-major, so that a block's share of a query is 128 contiguous bytes, which eight threads store into each
// of the other blocks (st.async, counted in bytes on the barrier of the buffer).  (Straight from registers, 32 bytes per
// warp and block without a barrier between, it took 19.7 us for one query and 24.1 for 16 instead of 18.9 and 20.8.)
// Two buffers alternate by layer: a block writes layer L only after it has read all of layer L - 1, which every block wrote
// after reading L - 2.  An all-gather of 128 bytes per block takes 750 cycles, of 1 KB 1,500, of 2 KB 2,400 (about 17
// bytes a cycle); through L2, as in mlp_pairs.cu, whole rows of columns travel, filled or not, in 2,000 cycles.
//
// The blocks of a group are one thread-block cluster, which the hardware schedules as a whole: that is
// what makes waiting for one another safe, and a launch may have more groups than fit at a time.
//
// Weights arrive through a ring; they do not depend on the activations, so it is full again when an exchange ends.
//
// Warp roles: 0 MMA issuer (and TMEM), 1 weight producer, 2 the mark, 4-7 epilogue (one TMEM lane quadrant each).  Every
// wait is bounded, as in mlp_chain.cu; a launch that gave up leaves a mark in the scratch, and launches that find it
// report an error instead of a result.
//
// After giving up no ring slot may be requested again that nobody has waited for: its copy could still be under way,
// and its barrier would be armed a second time in one phase.  So the MMA issuer, whose commits free the slots, waits
// for the producer to leave before it issues anything past a wait that ran out, and goes no further than the layer's end.
#include <atomic>
#include <cstring>

#include "mlp_small.cuh"

namespace {

constexpr int kNearBlocks = 16;                       // of a group
// Columns of B: eight queries, split: their hi and their lo parts (with eight too many 14 queries took 19.1 instead of 18.7 us)
template <bool SPLIT>
constexpr int kNearCols = SPLIT ? 16 : 8;
constexpr int kNearM = 64;                            // weight rows per block
constexpr int kNearThreads = 256;
template <bool SPLIT>
constexpr int kNearQ = SPLIT ? 2 : 6;                 // queries per group at most (with eight 0.3 us more for all, 56: 22.9)
template <bool SPLIT>
constexpr int kNearActBytes = 2 * 2048 * kNearCols<SPLIT>;   // two buffers
// Ring of weights.  bf16: few slots, each wait holds up the issue of MMAs for 90 cycles (one query 18.9 -> 17.8 us against five
// of 32 KB); a layer in split precision does not fit, and there two large ones are refilled too late (28.9 -> 34.7).
template <bool SPLIT>
constexpr int kNearSlots = SPLIT ? 5 : 2;
template <bool SPLIT>
constexpr int kNearSlotBytes = (SPLIT ? 2 : 4) * kTileBytes;
template <bool SPLIT>
constexpr int kNearSmem = kNearActBytes<SPLIT> + kNearSlots<SPLIT> * kNearSlotBytes<SPLIT> + 1024 + 512;
static_assert(kNearSmem<false> <= 232448 && kNearSmem<true> <= 232448, "shared memory");

// mbar_wait that also leaves the mark in the scratch.
__device__ __forceinline__ bool near_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, const SmallParams& p,
                                          int code) {
  if (mbar_wait(bar, parity, abort_flag, p.status, code)) return true;
  atomicExch(p.poison, 1);
  return false;
}
// near_wait for a whole warp: one lane polls, and every lane gets the same answer, so that the
// warp-wide instructions after it are reached together or not at all.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int lane, volatile int* abort_flag,
                                          const SmallParams& p, int code) {
  bool ok = true;
  if (lane == 0) ok = near_wait(bar, parity, abort_flag, p, code);
  __syncwarp();
  return __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
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

template <bool SPLIT>
__global__ void __launch_bounds__(kNearThreads, 1) mlp_near_kernel(const __grid_constant__ SmallParams p) {
  constexpr int kSlots = kNearSlots<SPLIT>, kSlotBytes = kNearSlotBytes<SPLIT>;
  constexpr int kParts = SPLIT ? 2 : 1;               // images per packed K block
  constexpr int kUnitBytes = kNearM * 128;            // one K block of the rows
  constexpr int kUnitsPerSlot = kSlotBytes / kUnitBytes;
  constexpr int kSlotsPerLayer = kNumKB * kParts / kUnitsPerSlot;
  constexpr int kCols = kNearCols<SPLIT>, kBufferBytes = 2048 * kCols;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t act = base;
  const uint32_t ring = base + kNearActBytes<SPLIT>;
  const uint32_t bars = ring + kSlots * kSlotBytes;
  uint8_t* bars_ptr = base_ptr + (bars - base);
  const uint32_t bar_full = bars, bar_empty = bars + 64;      // [kSlots]
  const uint32_t bar_act = bars + 128;                        // [2] buffer in place
  const uint32_t bar_acc = bars + 160;                        // layer accumulated
  const uint32_t bar_tfree = bars + 192;                      // TMEM read out (4 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_ptr + 200);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars_ptr + 204);
  volatile int* mark_seen = reinterpret_cast<volatile int*>(bars_ptr + 208);
  volatile int* producer_left = reinterpret_cast<volatile int*>(bars_ptr + 212);
  const uint32_t bar_drain = bars + 216;                      // after giving up: the MMAs have ended

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = static_cast<int>(blockIdx.x) / kNearBlocks, c = static_cast<int>(blockIdx.x) % kNearBlocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int q = 0; q < 2; ++q) mbar_init(bar_act + 8 * q, 1);
    mbar_init(bar_acc, 1);
    mbar_init(bar_tfree, 4);
    mbar_init(bar_drain, 1);
    *abort_flag = 0;
    *mark_seen = 0;
    *producer_left = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // (before the peers' first stores)
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  constexpr uint32_t kTmemCols = 32;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  grid_begin(p.beside != 0);
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int n_layers = p.layers + 1;
  uint32_t issued = 0;
  unsigned long long* const group_halves = p.halves + static_cast<size_t>(group) * 64 * hb::kGroupCols;

  const int64_t q0 = static_cast<int64_t>(group) * p.per_group;
  const int n_q = static_cast<int>(min(static_cast<int64_t>(p.per_group), static_cast<int64_t>(p.Q) - q0));

  if (warp == 2) {
    // An earlier launch that gave up may still be writing: report, and give up as well (no result is
    // stored then).  Only that result waits for the mark, whose load takes 700 cycles.
    if (lane == 0) {
      if (hb::concerns(*reinterpret_cast<volatile int32_t*>(p.poison), static_cast<uint32_t>(c))) {
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
      const int mt = c * kNearM / kMTile, row = c * kNearM % kMTile;   // the block's rows
      for (int L = 0; L < n_layers && ok; ++L) {
        const int image0 = kParts * (L == 0 ? mt : kNumMT + ((L - 1) * kNumMT + mt) * kNumKB);
        const int n = L == 0 ? 1 : kSlotsPerLayer;
        for (int g = 0; g < n; ++g) {
          const uint32_t full = bar_full + 8 * s;
          if (!near_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, p, 0x511)) { ok = false; break; }
          mbar_expect_tx(full, L == 0 ? kUnitBytes : kSlotBytes);
          if (L == 0) {
            tma_3d(ring + s * kSlotBytes, &p.map_fc1, row, image0, full);
          } else {   // four images each
            tma_3d(ring + s * kSlotBytes, &p.map_slot, row, image0 + g * kUnitsPerSlot, full);
            if (!SPLIT) tma_3d(ring + s * kSlotBytes + kSlotBytes / 2, &p.map_slot, row, image0 + g * kUnitsPerSlot + 4, full);
          }
          ++issued;
          ring_next<kSlots>(s, ph);
        }
      }
      *producer_left = 1;
    }
  } else if (warp == 0) {
    // ------------------------------ MMA issuer ------------------------------
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kCols >> 3) << 17) |
                               (static_cast<uint32_t>(kNearM >> 4) << 24);
    // A and B: K-major, 128-byte swizzle, 8-row groups 1024 B apart; B: kCols rows of 128 bytes per K block
    const uint64_t desc = (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
                          (static_cast<uint64_t>(2) << 61) | (static_cast<uint64_t>(1) << 16);
    // in 16-byte units: 16 K values of B, a K block of 64
    constexpr uint32_t kStepB = 2, kBlockB = (128 * kCols) >> 4;
    const uint32_t a_lo0 = (ring & 0x3FFFF) >> 4, b_lo0 = (act & 0x3FFFF) >> 4;
    // One elected lane runs the whole loop.  An MMA of this shape takes 23 cycles and only a
    // couple of them queue up, so what stands between two MMAs shows: the wait for the next slot goes
    // between the MMAs of the current one, the commit that frees a slot behind the next slot's first
    // MMAs, and every loop of a layer runs its full count whatever the waits say, so that the descriptors depend
    // on uniform values alone (a wait that ran out has set the abort flag; what is issued after it reads
    // stale shared memory and is discarded).  16 MMAs took 1,150 cycles in the plain form.
    if (elect_one()) {
      auto gave_up = [&] {   // (the producer looks at the abort flag when a slot does not come)
        for (const long long t0 = clock64(); *producer_left == 0 && clock64() - t0 <= kWaitCycles;) {}
      };
      auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        if (!mbar_try_wait(bar, parity) && (*abort_flag || !near_wait(bar, parity, abort_flag, p, code))) gave_up();
        tc_fence_after();
      };
      // layer L's input, the whole of buffer L & 1, written by the peers
      auto wait_input = [&](int L) {
        if (!mbar_wait_cluster(bar_act + 8 * (L & 1), (L >> 1) & 1, abort_flag, p.status, 0x521)) {
          atomicExch(p.poison, 1);
          gave_up();
        }
        fence_proxy_async();
        tc_fence_after();
      };
      uint32_t s = 0, ph = 0;
      {                                                          // fc1: one K block
        wait_input(0);
        wait(bar_full + 8 * s, ph, 0x522);
        const uint32_t a_lo = a_lo0 + s * (kSlotBytes >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_one_bf16(tmem_base, desc | (a_lo + 2 * k), desc | (b_lo0 + k * kStepB), idesc, k ? 1u : 0u);
        commit_one(bar_acc);
        commit_one(bar_empty + 8 * s);
        ring_next<kSlots>(s, ph);
      }
      constexpr int kMmas = 4 * kUnitsPerSlot;                   // per slot
#pragma unroll 1
      for (int L = 1; L < n_layers && *abort_flag == 0; ++L) {
        wait(bar_tfree, (L - 1) & 1, 0x523);
        wait(bar_full + 8 * s, ph, 0x522);
        wait_input(L);
        uint32_t prev = 0;
#pragma unroll 1
        for (int g = 0; g < kSlotsPerLayer; ++g) {
          uint32_t next = s, next_ph = ph;
          ring_next<kSlots>(next, next_ph);
          const uint32_t a_lo = a_lo0 + s * (kSlotBytes >> 4);
          const uint32_t b_lo = b_lo0 + static_cast<uint32_t>(L & 1) * (kNumKB * kBlockB) +
                                static_cast<uint32_t>(g) * (kBlockB * kUnitsPerSlot / kParts);
#pragma unroll
          for (int u = 0; u < kMmas; ++u) {
            mma_one_bf16(tmem_base, desc | (a_lo + (u >> 2) * (kUnitBytes >> 4) + 2 * (u & 3)),
                         desc | (b_lo + (u >> 2) / kParts * kBlockB + (u & 3) * kStepB), idesc,
                         u == 0 ? static_cast<uint32_t>(g) : 1u);
            if (u == 1 && g > 0) commit_one(bar_empty + 8 * prev);
            if (u == kMmas / 2 && g + 1 < kSlotsPerLayer) wait(bar_full + 8 * next, next_ph, 0x522);
          }
          prev = s;
          s = next;
          ph = next_ph;
        }
        commit_one(bar_acc);
        commit_one(bar_empty + 8 * prev);
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------ epilogue ------------------------------
    const int quad = warp & 3;
    const int T = static_cast<int>(threadIdx.x) - 128;          // 0..127
    auto epi_sync = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    // fc1's B operand: K columns 0..63 hold [hi | lo | hi] of the normalised features, one query per row
    const int C_in = p.n_op_feat + 4;
    for (int i = T; i < 64 * 2 * kCols / 16; i += 128) *reinterpret_cast<uint4*>(base_ptr + 16 * i) = make_uint4(0, 0, 0, 0);
    epi_sync();
    for (int i = T; i < n_q * C_in; i += 128) {
      const int q = i / C_in, f = i - q * C_in;
      __nv_bfloat16 hi, lo;
      load_feature(p, static_cast<int>(q0) + q, f, hi, lo);
      *reinterpret_cast<__nv_bfloat16*>(base_ptr + swz_off(q, f)) = hi;
      *reinterpret_cast<__nv_bfloat16*>(base_ptr + swz_off(q, C_in + f)) = lo;
      *reinterpret_cast<__nv_bfloat16*>(base_ptr + swz_off(q, 2 * C_in + f)) = hi;
    }
    fence_proxy_async();
    epi_sync();
    if (T < 1) mbar_arrive(bar_act);
    __syncwarp();
    // M = 64 leaves 16 rows in the low lanes of every quadrant
    const bool row_ok = lane < 16;
    const int row = quad * 16 + (lane & 15), f = c * kNearM + row;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    constexpr int kPiece = 8;                                   // columns, queries
    bool ok = true;
    // a wait that ran out skips the work that is left but none of the block-wide barriers
    for (int L = 0; L < n_layers; ++L) {
      const bool last = L == n_layers - 1;
      const float bias = __ldg(p.bias + L * kWidth + f);
      const float w2 = last ? __ldg(p.fc2_w + f) : 0.0f;
      ok = ok && warp_wait(bar_acc, L & 1, lane, abort_flag, p, 0x541);
      if (!ok) {
        if (!last) epi_sync();
        continue;
      }
      tc_fence_after();
      float v[kPiece];
      tc_ld8(t_lane, v);
      if (SPLIT) {   // columns 8 to 15 are the lo parts
        float lo[kPiece];
        tc_ld8(t_lane + 8, lo);
#pragma unroll
        for (int i = 0; i < kPiece; ++i) v[i] += lo[i];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tfree);
#pragma unroll
      for (int i = 0; i < kPiece; ++i) v[i] = fmaxf(v[i] + bias, 0.0f);
      if (!last) {
        // own features first, then the group's other blocks: 128 bytes of every query
        const uint32_t mine = static_cast<uint32_t>((L + 1) & 1) * kBufferBytes + static_cast<uint32_t>(c) * (128u * kCols);
        const uint32_t in_bar = bar_act + 8 * ((L + 1) & 1);
#pragma unroll
        for (int q = 0; q < kNearQ<SPLIT>; ++q) {
          if (!row_ok || q >= n_q) continue;
          const __nv_bfloat16 hi = __float2bfloat16_rn(v[q]);
          *reinterpret_cast<__nv_bfloat16*>(base_ptr + mine + swz_off(q, row)) = hi;
          if (SPLIT)
            *reinterpret_cast<__nv_bfloat16*>(base_ptr + mine + swz_off(8 + q, row)) =
                __float2bfloat16_rn(v[q] - __bfloat162float(hi));
        }
        fence_proxy_async();
        epi_sync();
        // (after giving up the buffer's last phase may be incomplete: it is not armed again)
        if (T == 0 && *abort_flag == 0) mbar_expect_tx(in_bar, static_cast<uint32_t>((kNearBlocks - 1) * kParts * 128 * n_q));
        const uint32_t chunk = static_cast<uint32_t>(T) & 7u, to = static_cast<uint32_t>(c + (T >> 3)) % kNearBlocks;
        if (T >= 8) {   // eight threads per peer, 16 bytes of each query
          const uint32_t there = map_to_cta(base + mine, to), bar = map_to_cta(in_bar, to);
          for (uint32_t q = 0; q < static_cast<uint32_t>(n_q); ++q)
#pragma unroll
            for (uint32_t part = 0; part < kParts; ++part) {
              const uint32_t at = (part * 8 + q) * 128u + (((chunk ^ q) & 7u) << 4);
              const uint4 x = *reinterpret_cast<const uint4*>(base_ptr + mine + at);
              st_async_v4(there + at, x.x, x.y, x.z, x.w, bar);
            }
        }
        __syncwarp();
      } else {
        const int gave_up = *abort_flag;   // an issuer that did has gone on to the layer's end
        float s[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) s[i] = i < kPiece ? __fmul_rn(w2, v[i % kPiece]) : 0.0f;
        fold16(s, lane);
        if (row_ok && gave_up == 0) {   // (without the sums the block that adds them gives up as well)
          const int set = (c * kNearM + quad * 16) / 16;
          st_relaxed_u64(group_halves + set * hb::kGroupCols + fold16_col<16>(lane),
                         static_cast<unsigned long long>(p.tag) << 32 | __float_as_uint(s[0]));
        }
      }
    }
    if (c == 0) {
      // the first block of the group adds the 64 sets of 16 features of every query
      const int q = T & 63;
      float* tots = reinterpret_cast<float*>(base_ptr);        // the tensor core is done with the activations
      tots[T] = q < n_q && ok ? fc2_sum(p, group_halves + q, T >> 6, p.tag, abort_flag) : 0.0f;
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
  if (*abort_flag) {
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
using hb::kMaxCudaDevices;
// The shapes.  pairs: of mlp_pairs.cu, with NC columns per CTA; 0: mlp_near_kernel.  clusters: of the shape that a B200 runs at a
// time.  us: what a launch takes, full or not (measured, see wide_plan).
struct Shape { int pairs, NC, clusters, us, us_split; };
constexpr Shape kShapes[] = {{0, 16, 7, 21, 30}, {8, 16, 7, 25, 32}, {8, 32, 7, 26, 35}, {8, 40, 7, 29, 38}, {8, 48, 7, 31, 41},
                             {4, 32, 15, 34, 49}, {4, 48, 15, 40, 58},
                             {4, 64, 15, 45, 62}, {2, 64, 33, 64, 103}};
constexpr int kNumShapes = static_cast<int>(sizeof(kShapes) / sizeof(kShapes[0]));
constexpr int kMaxGroups = 33;
constexpr bool shapes_fit() {
  for (const Shape& s : kShapes)
    if (s.clusters > kMaxGroups || (s.pairs != 0 && !hb::has_pairs_shape(s.pairs, s.NC))) return false;
  return true;
}
static_assert(shapes_fit(), "parities are kept for 64 groups, sums for kMaxGroups, and every shape has a kernel");

// Scratch per stream: launches on one stream follow one another, so they can share it (those of one call
// that run side by side have a lane each).  It is kept between launches and freed with the GPU's last predictor.
// The first kMaxStreams streams and lanes keep theirs.  Later ones (a program with a stream per request) share
// kMoreStreams: each launch of theirs is followed by an event, and a new stream takes over what has been out of
// use for longest.  The events keep a launch from overlapping the end of the one before it, which is why
// the first streams go without.  While none of the shared ones is out of use, a launch takes the two-SM kernel,
// which needs no scratch.
constexpr int kMaxStreams = 16, kMoreStreams = 16;
constexpr size_t kHalvesBytes = static_cast<size_t>(kMaxGroups) * 64 * hb::kGroupCols * sizeof(unsigned long long);
constexpr size_t kBaseBytes = kHalvesBytes + 256;   // and the mark of a launch that gave up
// Activations of a shape of mlp_pairs.cu, 0.9 to 17 MB: made when the stream first has a batch for the shape.
constexpr size_t acts_bytes(const Shape& s) { return static_cast<size_t>(s.clusters) * 4 * kWidth * 2 * s.NC; }
struct Activations {
  uint8_t* base = nullptr;
  bool fresh = false;                            // words and parities start over at the next launch
  unsigned long long parity[2] = {};             // bit g: parity of the next use of group g's buffers
  CUtensorMap map{};
};
struct StreamScratch {
  unsigned long long stream_id = 0;
  int lane = 0;
  uint8_t* base = nullptr;                       // sums, mark
  bool fresh = false;                            // they start over at the next launch
  uint32_t tag = 0;
  Activations acts[kNumShapes];                  // (the near shape has none)
  bool expect_stale = false;                     // at the next launch that could (tests)
  int32_t stale[3] = {-1, -1, -1};               // then, too: SmallParams::stale_layer ..
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
      cudaMalloc(&base, kBaseBytes) != cudaSuccess) {
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

// The activations of a shape, or null when there is no memory for them.  Call with the mutex held.
Activations* acts_of(StreamScratch& s, int shape) {
  Activations& a = s.acts[shape];
  if (a.base) return &a;
  const RelaxedCapture relaxed;
  const Shape& form = kShapes[shape];
  void* base = nullptr;
  if (cudaMalloc(&base, acts_bytes(form)) != cudaSuccess ||
      hb::encode_rows(&a.map, base, hb::act_map_row(form.NC), acts_bytes(form) / hb::act_map_row(form.NC),
                      hb::act_map_box(form.NC)) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(base);
    return nullptr;
  }
  a.base = static_cast<uint8_t*>(base);
  a.fresh = true;
  return &a;
}

template <bool SPLIT>
cudaError_t launch_near(const SmallParams& p, int groups, int device, cudaStream_t stream, bool* fits) {
  static std::atomic<int> clusters[kMaxCudaDevices];
  return hb::launch_clusters(mlp_near_kernel<SPLIT>, kNearBlocks, kNearThreads, kNearSmem<SPLIT>, p, groups, stream, fits,
                             clusters[device]);
}
}  // namespace

namespace hb {

// The cheapest shape whose groups all run at a time.  Clusters stay inside a GPC, so a B200 runs 7, 15 or
// 33 of 16, 8 or 4 blocks.  Smaller clusters hold more queries in all but stream more weights per block, wider ones
// exchange more per layer.  Measured per launch, conv2d predictor, 8 hidden layers (capacity in queries: us), against 103 us
// (bf16) and 168 us (split) of one tile of mlp_chain.cu's kernel, which is the faster one beyond the last shape:
//   near               42: 21.6 (one: 17.8)   split    14: 29.6 (one: 27.5)
//   8 pairs x 16      224: 24.6 (43: 23.1)            112: 32.2 (15: 30.4)
//   8 pairs x 32      448: 26.3                       224: 35.2
//   8 pairs x 40      560: 28.6                       280: 37.8   (what 4 pairs x 32 take is 5.7 and 11 more)
//   8 pairs x 48      672: 31.0                       336: 41.5
//   4 pairs x 32      960: 34.3                       480: 48.9   (in two row blocks 4.0 and 0.7 more)
//   4 pairs x 48    1,440: 40.4                       720: 58.3
//   4 pairs x 64    1,920: 45.3                       960: 61.6   (in one row block, exchanged at once, 51.5 and 73.6)
//   2 pairs x 64    4,224: 63.6                     2,112: 103
// Blocks without partners (M = 64 or 128 each, all queries of a group in every block; data polled in L2) took 24 for 112,
// 28 for 240, 32 for 480, 46 for 960, 48 for 1,056 and 73 for 2,112 queries, split 34 for 56, 46 for 240, 78 for 528 and 126
// for 1,056: nowhere better than these.
namespace {
int clusters_of(const Shape& s, int sm_count) { return sm_count >= 148 ? s.clusters : s.clusters * sm_count / 148; }
int cols_of(const Shape& s, bool split) {
  return s.pairs == 0 ? (split ? kNearQ<true> : kNearQ<false>) : (split ? s.NC : 2 * s.NC);
}
WidePlan plan_in(const Shape& s, int64_t Q, bool split, int cols = 0) {
  // full groups while they last: fewer groups move the weights fewer times
  if (cols == 0) cols = cols_of(s, split);
  WidePlan w{s.pairs ? 2 * s.pairs : kNearBlocks, static_cast<int>((Q + cols - 1) / cols), 0, static_cast<int>(&s - kShapes)};
  w.per_group = static_cast<int>((Q + w.groups - 1) / w.groups);
  w.groups = static_cast<int>((Q + w.per_group - 1) / w.per_group);
  return w;
}
// Beside other batches near groups, which hold few queries, cost more of the GPU than they gain.
bool fits_in_company(const WidePlan& w) { return kShapes[w.shape].pairs != 0 || w.groups == 1; }
}  // namespace

WidePlan wide_plan(int64_t Q, bool split, int sm_count, bool alone) {
  for (const Shape& s : kShapes) {
    const int clusters = clusters_of(s, sm_count);
    if (Q > static_cast<int64_t>(clusters) * cols_of(s, split)) continue;
    // near groups are the faster the fewer queries they have
    const WidePlan w = plan_in(s, Q, split, s.pairs == 0 && alone ? static_cast<int>((Q + clusters - 1) / clusters) : 0);
    if (alone || fits_in_company(w)) return w;
  }
  return WidePlan{};
}

// Shapes for batches that run side by side.  The cheapest shape of each is the most spread out, and two of them
// rarely fit on the GPU together: the second then waits for the first.  A shape takes the same time with few
// groups as with many, so the shortest way through is the lowest time at which all batches fit when each takes
// the narrowest shape of that time or less, unless one after the other is shorter.  What is left of the GPU goes
// to cheaper shapes for the batches that start last.  Three predictors with 318, 192 and 6 queries take 33 us.
// (Clusters cannot be cut at will, as the sum of shares has it.  Measured on 108 random calls of two to four batches: with the list
// of tiles as the other choice, see hb_mlp_predict_grid, none took over 2 % longer than without the shapes for 2,113 to 4,224.)
int wide_plans_together(WidePlan* plans, const int64_t* Q, const bool* split, int n, int sm_count) {
  auto us_of = [&](const Shape& s, int b) { return split[b] ? s.us_split : s.us; };
  auto share_of = [&](const WidePlan& w, const Shape& s) {   // of the clusters that run at a time
    const int clusters = clusters_of(s, sm_count);
    return clusters ? static_cast<double>(w.groups) / clusters : 2.0;
  };
  int in_turn = 0;   // (what takes less than half of the GPU mostly runs beside the others all the same)
  for (int b = 0; b < n; ++b) {
    const Shape& s = kShapes[plans[b].shape];
    const double share = share_of(plans[b], s);
    in_turn += s.pairs == 2 || share >= 0.5 ? us_of(s, b) : static_cast<int>(share * us_of(s, b));
  }
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
    return us;
  }
  return in_turn + in_turn / 20;   // (measured: 0 to 9 % more than the sum)
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
    for (Activations& a : g.s[i].acts) cudaFree(a.base);
    if (g.s[i].done) cudaEventDestroy(g.s[i].done);
    g.s[i].done = nullptr;
  }
  g.used = 0;
}

void wide_start_over(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  for (int i = 0; i < g.used; ++i) {
    g.s[i].fresh = true;
    for (Activations& a : g.s[i].acts) a.fresh = true;
  }
}

hb_status wide_set_mark(int device, int32_t mark) {
  if (device < 0 || device >= kMaxCudaDevices) return HB_OK;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  HB_CUDA_TRY(cudaDeviceSynchronize());
  for (int i = 0; i < g.used; ++i)
    HB_CUDA_TRY(cudaMemcpy(g.s[i].base + kHalvesBytes, &mark, sizeof(mark), cudaMemcpyHostToDevice));
  HB_CUDA_TRY(cudaDeviceSynchronize());
  return HB_OK;
}

void wide_expect_stale(int device) {
  if (device < 0 || device >= kMaxCudaDevices) return;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  for (int i = 0; i < g.used; ++i) g.s[i].expect_stale = true;
}

void wide_plant_stale(int device, int32_t layer, int32_t feature, int32_t word) {
  if (device < 0 || device >= kMaxCudaDevices) return;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  for (int i = 0; i < g.used; ++i) {
    g.s[i].stale[0] = layer;
    g.s[i].stale[1] = feature;
    g.s[i].stale[2] = word;
  }
}

hb_status wide_second_runs(int device, int64_t* runs) {
  *runs = 0;
  if (device < 0 || device >= kMaxCudaDevices) return HB_OK;
  GpuScratch& g = g_wide[device];
  std::lock_guard<std::mutex> lock(g.mu);
  HB_CUDA_TRY(cudaDeviceSynchronize());
  for (int i = 0; i < g.used; ++i) {
    int32_t n = 0;
    if (g.s[i].fresh) continue;   // not cleared yet
    HB_CUDA_TRY(cudaMemcpy(&n, g.s[i].base + kHalvesBytes + sizeof(int32_t), sizeof(n), cudaMemcpyDeviceToHost));
    *runs += n;
  }
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
  const Shape& shape = kShapes[w.shape];
  Activations* const acts = shape.pairs ? acts_of(*s, w.shape) : nullptr;
  if (shape.pairs && !acts) return HB_OK;
  s->last_use = ++g.uses;
  const bool split = h->precision == HB_PRECISION_BF16X3;
  SmallParams p{};
  p.bias = h->bias; p.fc2_w = h->fc2_w; p.fc2_b = h->fc2_b; p.mu = h->mu; p.sigma = h->sigma; p.dev_feat = h->dev_feat;
  p.n_dev = h->n_dev; p.n_op_feat = h->n_op_feat; p.layers = h->layers;
  p.feats = batch.feats; p.dev_row = batch.dev_row; p.Q = static_cast<int32_t>(batch.Q);
  p.per_group = w.per_group; p.out = batch.out;
  p.status = h->status;
  p.beside = batch.beside && !s->fresh && !(acts && acts->fresh) ? 1 : 0;   // (a fresh buffer's clearing has to be waited for)
  p.first = batch.first;
  p.grid_n = batch.grid_n;
  if (batch.grid_n) std::memcpy(p.grid_rows, batch.grid_rows, (batch.first + batch.Q) / batch.grid_n);
  if (batch.host_inputs) {
    p.inline_q = static_cast<int32_t>(batch.Q);
    std::memcpy(p.inline_feats, batch.feats, sizeof(float) * batch.Q * h->n_op_feat);
    std::memcpy(p.inline_row, batch.dev_row, batch.Q);
  }
  if (s->fresh) {   // all tags at 0, no mark
    HB_CUDA_TRY(cudaMemsetAsync(s->base, 0, kBaseBytes, stream));
    s->tag = 0;
    s->fresh = false;
  }
  if (acts) {
    if (acts->fresh) {   // all words at parity 0
      HB_CUDA_TRY(cudaMemsetAsync(acts->base, 0, acts_bytes(shape), stream));
      acts->parity[0] = acts->parity[1] = ~0ull;
      acts->fresh = false;
    }
    p.acts = acts->base;
    p.map_acts = acts->map;
    p.parity[0] = acts->parity[0];
    p.parity[1] = acts->parity[1];
    p.expect_stale = s->expect_stale ? 0x80008000u : 0u;
    s->expect_stale = false;
    p.stale_layer = s->stale[0]; p.stale_feature = s->stale[1]; p.stale_word = s->stale[2];
    s->stale[0] = -1;
  }
  p.halves = reinterpret_cast<unsigned long long*>(s->base);
  p.poison = reinterpret_cast<int32_t*>(s->base + kHalvesBytes);
  s->tag = s->tag % 0x7FFFFFFFu + 1;   // the high bit is the second run's (mlp_pairs.cu)
  p.tag = s->tag;
  const bool narrow = shape.pairs == 0 || shape.pairs == 8 || (shape.pairs == 4 && shape.NC == 64);   // blocks of 64 weight rows
  p.map_slot = narrow ? h->tmap_slot : h->tmap_tile;
  p.map_fc1 = narrow ? h->tmap_half_tile : h->tmap_tile;
  bool fits = false;
  const cudaError_t e =
      shape.pairs ? launch_pairs(shape.pairs, shape.NC, split, p, w.groups, h->device, stream, &fits)
                  : (split ? launch_near<true>(p, w.groups, h->device, stream, &fits)
                           : launch_near<false>(p, w.groups, h->device, stream, &fits));
  if (acts && e == cudaSuccess && fits) {
    // exchange `use` (0 .. layers - 1) takes buffer use & 1; every group of the launch flips with it
    const unsigned long long groups = (1ull << w.groups) - 1;
    for (int b = 0; b < 2; ++b)
      if (((h->layers + 1 - b) / 2) & 1) acts->parity[b] ^= groups;
  }
  if (s->done && cudaEventRecord(s->done, stream) != cudaSuccess) {
    cudaGetLastError();
    cudaEventDestroy(s->done);
    s->done = nullptr;         // nobody can tell any more when it is out of use: it stays with its stream
  }
  if (e != cudaSuccess) return cuda_fail(e, "small-batch MLP launch");
  *launched = fits;
  return HB_OK;
}

}  // namespace hb
