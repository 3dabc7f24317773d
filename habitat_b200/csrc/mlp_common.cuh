// Shared by the MLP kernels (mlp_chain.cu, mlp_pairs.cu, mlp_wide.cu): sizes, PTX wrappers, the handle.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "hb_common.h"

namespace {

constexpr int kWidth = 1024;            // layer_size of every Habitat predictor
constexpr int kMTile = 128;             // output features per MMA (TMEM lanes)
constexpr int kKBlk = 64;               // bf16 per 128-byte swizzle row
constexpr int kNumMT = kWidth / kMTile; // 8
constexpr int kNumKB = kWidth / kKBlk;  // 16
constexpr int kTileBytes = kMTile * 128;// one weight tile image: 16 KB
constexpr int kMaxInFeat = 12;          // F + 4 (conv2d: 8 + 4)

// ---------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(pred)::"memory");
  return pred;
}
// Programmatic dependent launch of kernels of which some run side by side.  An ordinary one waits for the
// launch before it and only then lets the next one start; one that runs beside its predecessor does not
// wait at the start (it can only have started after an ordinary one before it had waited), but one of its
// blocks waits at the end, so that "this grid is complete" still means "and so are those before it".
__device__ __forceinline__ void hb_grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_begin(bool beside) {
  if (!beside) hb_grid_wait();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_end(bool beside) {
  if (beside && blockIdx.x == 0) hb_grid_wait();
}

// Slot arithmetic of the MMA issue loops.  The descriptors of tcgen05.mma live in uniform registers, and
// only some operations exist there: a ring position kept by compare and select (or by a remainder)
// went through vector registers and cost a transfer per MMA, 180 cycles per 16 of them.  Shifts and
// masks stay uniform: the successor of slot s is looked up in a constant.
template <int N>
constexpr uint32_t ring_table() {
  static_assert(N <= 8, "three bits per slot, 24 bits");
  uint32_t t = 0;
  for (int s = 0; s < N; ++s) t |= static_cast<uint32_t>((s + 1) % N) << (3 * s);
  return t;
}
template <int N>
__device__ __forceinline__ void ring_next(uint32_t& s, uint32_t& phase) {
  s = (ring_table<N>() >> (3 * s)) & 7u;
  phase ^= (1u >> s) & 1u;   // back at slot 0
}

// Transposes N x N chunks of four words over each N neighbouring lanes: lane l of them gives chunk j to lane j.
template <int N>
__device__ __forceinline__ void trade_chunks(uint32_t (&w)[4 * N], int lane) {
#pragma unroll
  for (int m = 1; m < N; m *= 2) {
    const bool upper = (lane & m) != 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (j & m) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t& lo = w[4 * j + i];
        uint32_t& hi = w[4 * (j + m) + i];
        const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, upper ? lo : hi, m);
        if (upper) lo = got;
        else hi = got;
      }
    }
  }
}

// One fold of the transposing reduction below: N values per lane and a lane mask become N / 2
// values, the sums over the pair of lanes that differ in `mask`; lanes with the bit keep the upper half.
template <int N, int W>
__device__ __forceinline__ void fold_lanes(float (&v)[W], int lane, int mask) {
  const bool upper = (lane & mask) != 0;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float keep = upper ? v[i + N / 2] : v[i];
    const float send = upper ? v[i] : v[i + N / 2];
    v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, mask);
  }
}
// Sums of W columns over the 16 lanes of each half warp, as a fixed tree (lane distances 8, 4, 2,
// 1).  Lane l is left with columns fold16_col<W>(l) + 0 .. W / 16 - 1 of its half, in v[0 ..].  fc2 adds
// its products in this order in every kernel, so a prediction does not depend on which one made it.
template <int W>
__device__ __forceinline__ void fold16(float (&v)[W], int lane) {
  fold_lanes<W>(v, lane, 8);
  fold_lanes<W / 2>(v, lane, 4);
  fold_lanes<W / 4>(v, lane, 2);
  fold_lanes<W / 8>(v, lane, 1);
}
template <int W>
__device__ __forceinline__ int fold16_col(int lane) {
  return ((lane & 8) ? W / 2 : 0) + ((lane & 4) ? W / 4 : 0) + ((lane & 2) ? W / 8 : 0) + ((lane & 1) ? W / 16 : 0);
}
__device__ __forceinline__ void tc_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane
// (quadrant base + t), registers = columns.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  tc_wait_ld();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 8 and x 16 consecutive 32-bit columns.
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 64 consecutive 32-bit columns in one instruction: halves the number of
// load round trips of the epilogue (each tcgen05.ld + wait costs several hundred cycles).
__device__ __forceinline__ void tc_ld64(uint32_t taddr, float (&v)[64]) {
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
      "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]),
        "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]),
        "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]),
        "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]),
        "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}

// Byte offset of element (row, col) inside a K-major 128-byte-swizzled block of
// 128-byte rows: 16-byte chunks are permuted by the row index modulo 8.
__host__ __device__ __forceinline__ uint32_t swz_off(uint32_t row, uint32_t col) {
  return row * 128u + ((((col >> 3) ^ row) & 7u) << 4) + ((col & 7u) << 1);
}

constexpr long long kWaitCycles = 4000000000LL;  // about two seconds

// Bounded wait.  Returns false when the wait ran out or another role gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int32_t* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t i = 1;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 0u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > kWaitCycles) {
        *abort_flag = 1;
        *static_cast<volatile int32_t*>(status) = code;
        return false;
      }
    }
  }
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same with cluster scope.  After another role gave up it returns at once (a try_wait lasts 7,800 cycles when
// nothing comes, 64 of them a quarter of a millisecond): mlp_chain.cu's MMA issuer goes on to the end of its tile
// whatever the waits say, several hundred of them.  (mbar_wait looks at it every 64 tries: the small-batch kernels' waits
// mostly last less than one, and looking first took 1 to 2 % more.)
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity,
                                                  volatile int* abort_flag, int32_t* status,
                                                  int code) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t i = 0;; ++i) {
    if ((i & 63u) == 0u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > kWaitCycles) {
        *abort_flag = 1;
        *static_cast<volatile int32_t*>(status) = code;
        return false;
      }
    }
    if (mbar_try_wait_cluster(bar, parity)) return true;
  }
}
// Asynchronous 16-byte store into a peer CTA's shared memory; completion is counted
// in bytes on an mbarrier of that CTA.  Unlike st.shared::cluster the issuing
// thread does not wait for the store to be acknowledged.
__device__ __forceinline__ void st_async_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c,
                                            uint32_t d, uint32_t cluster_mbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
      ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(cluster_mbar)
      : "memory");
}
// Byte offset of element (K row k, query n) of an MN-major, 128-byte-swizzled B
// operand holding 64 queries per row: rows are 128 B apart, the eight 16-byte
// groups of a row are permuted by the row index modulo 8.
__device__ __forceinline__ uint32_t mn_off(uint32_t k, uint32_t n) {
  return k * 128u + ((((n >> 3) ^ k) & 7u) << 4) + ((n & 7u) << 1);
}
__device__ __forceinline__ void st_cluster_f32(uint32_t cluster_addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Tiled TMA load of a box of 128-byte rows into this CTA's shared memory.  With
// .cta_group::2 the completion may be counted on a barrier of the other CTA of the pair
// (given as a shared::cluster address): both CTAs' weight copies report to the leader's
// barrier directly.  No multicast: each CTA fetches its own half of the weights.
__device__ __forceinline__ void tma_rows_2sm(uint32_t dst, const CUtensorMap* map, int32_t row,
                                             uint32_t cluster_mbar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_mbar), "r"(0), "r"(row)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void tc_mma_pair_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                 uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

}  // namespace

struct hb_mlp {
  int32_t n_op_feat = 0, layers = 0, precision = 0, n_dev = 0, sm_count = 0, device = 0;
  float fc2_b = 0.f;
  uint8_t* wpack = nullptr;
  CUtensorMap tmap_tile{};                         // one tile image
  CUtensorMap tmap_slot{}, tmap_half_tile{};       // 64 rows of four consecutive tile images, of one
  float* bias = nullptr;
  float* fc2_w = nullptr;
  double* mu = nullptr;
  double* sigma = nullptr;
  double* dev_feat = nullptr;
  int32_t* status = nullptr;          // page-locked host word that the kernels write when they give up
  long long* phase_cycles = nullptr;
  bool counted = false;      // among the GPU's predictors (mlp_wide.cu)
};
