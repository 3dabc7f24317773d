// Wave scaling of recorded kernels: one fused elementwise kernel over
// (kernel x destination-device) pairs.
//
// Stands in for the per-kernel Python loop of the reference
// (analyzer/habitat/analysis/predictor.py:111-130 calling
// wave_scaling/roofline.py:8-65, resimplified.py:7-40, common.py:3-20 and,
// through pybind, cpp/src/cuda/kernel.cpp:33-56).
//
// Layout: kernels arrive as structure-of-arrays, results leave as
// destination-major planes.  One thread owns VEC consecutive kernels and walks
// all D destinations, so each record is read once and the origin-side
// occupancy is computed once.  Device rows live in constant memory; the
// per-launch (origin, destination) log2 ratios travel as a kernel parameter.
// The kernel is HBM-bound by design: 20 B read + 5 B written per kernel and
// 9 B written per pair.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

#include "hb_common.h"
#include "occupancy.cuh"
#include "reduce_stage1.cuh"

namespace {

thread_local int32_t t_path = 0;   // kernel of the last launch, see hb_wave_scale_path

__constant__ hb_dev_pre c_dev[HB_MAX_DEVICES];

struct LaunchParams {
  int32_t D;
  int32_t origin_row;
  int64_t K;
  double origin_peak;          // origin peak GFLOP/s (metrics mode)
  uint8_t dest_row[HB_MAX_DEVICES];
  // large branch: log2 t' = log2 t + gamma * a + b, a = log2(bw) - b,
  // b = log2(clock ratio) + log2(SM ratio); small branch uses log2_clk.
  double a[HB_MAX_DEVICES];
  double b[HB_MAX_DEVICES];
  double log2_clk[HB_MAX_DEVICES];
  double ridge[HB_MAX_DEVICES];  // destination peak / bandwidth (metrics mode)
};

// log2(i) for the per-SM block counts of the small-kernel branch (<= 32
// because occupancy never exceeds the blocks-per-SM limit).
__constant__ double c_log2_int[65];

template <typename T, int N>
struct alignas(sizeof(T) * N) Vec {
  T v[N];
};

template <typename T, int N>
__device__ __forceinline__ Vec<T, N> load_vec(const T* p) {
  return *reinterpret_cast<const Vec<T, N>*>(p);
}
template <typename T, int N>
__device__ __forceinline__ void store_vec(T* p, const Vec<T, N>& v) {
  *reinterpret_cast<Vec<T, N>*>(p) = v;
}

struct Ptrs {
  const int32_t* num_blocks;
  const uint16_t* block_size;
  const uint16_t* regs;
  const uint32_t* smem;
  const float* time_ns;
  const float* gamma;
  const double* flop_eff;
  const double* dram_read;
  const double* dram_write;
  const uint8_t* has_metrics;
  const int16_t* dest_regs;
  float* scaled_ns;
  uint8_t* dest_occ;
  uint32_t* dest_waves;
  uint8_t* origin_occ;
  uint32_t* origin_waves;
  uint8_t* status;
  int32_t* limits;
  double* block_sums;   // table kernel with fused totals: [D][blocks] sums of each block's results
};

// Per-SM block count ceil(nb / sms) for a kernel that fits in one wave.
__device__ __forceinline__ int32_t ceil_div_sms(int32_t nb, int32_t sms) {
  return hb_div_small(nb + sms - 1, sms);
}

template <int VEC, bool METRICS, bool EXTRA>
__global__ void __launch_bounds__(256)
wave_scale_kernel(const Ptrs p, const __grid_constant__ LaunchParams lp) {
  const int64_t K = lp.K;
  const int64_t k0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * VEC;
  if (k0 >= K) return;

  const Vec<int32_t, VEC> nbv = load_vec<int32_t, VEC>(p.num_blocks + k0);
  const Vec<uint16_t, VEC> bsv = load_vec<uint16_t, VEC>(p.block_size + k0);
  const Vec<uint16_t, VEC> rgv = load_vec<uint16_t, VEC>(p.regs + k0);
  const Vec<uint32_t, VEC> smv = load_vec<uint32_t, VEC>(p.smem + k0);
  const Vec<float, VEC> tv = load_vec<float, VEC>(p.time_ns + k0);
  Vec<float, VEC> gv;
  if (!METRICS) gv = load_vec<float, VEC>(p.gamma + k0);

  const hb_dev_pre& od = c_dev[lp.origin_row];

  int32_t smem[VEC], wave_o[VEC], omax[VEC];
  double intensity[VEC];   // METRICS: GFLOP per GB, < 0 encodes the special cases
  Vec<uint8_t, VEC> oocc;
  Vec<uint32_t, VEC> owav;
  int32_t lim[4];

#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    smem[i] = smv.v[i] > 0x7FFF0000u ? -1 : static_cast<int32_t>(smv.v[i]);
    const int32_t occ = hb_occupancy(od, bsv.v[i], smem[i], rgv.v[i], lim);
    if (EXTRA && p.limits) {
#pragma unroll
      for (int j = 0; j < 4; ++j) p.limits[static_cast<int64_t>(j) * K + k0 + i] = lim[j];
    }
    wave_o[i] = od.num_sms * occ;
    oocc.v[i] = static_cast<uint8_t>(occ);
    const int32_t nb = nbv.v[i];
    owav.v[i] = (wave_o[i] > 0 && nb >= 1) ? static_cast<uint32_t>(nb / wave_o[i]) : 0xFFFFFFFFu;
    // only consulted when nb < wave_o, i.e. the value is <= occ <= 32
    omax[i] = (nb >= 1 && nb < wave_o[i]) ? ceil_div_sms(nb, od.num_sms) : 1;
    if (METRICS) {
      // wave_scaling/roofline.py:68-88, same operation order, fp64
      double g = -1.0;  // "no metrics": gamma = 1
      if (p.has_metrics[k0 + i]) {
        const double total_gb =
            (p.dram_read[k0 + i] + p.dram_write[k0 + i]) / 1024 / 1024 / 1024;
        const double gps = p.flop_eff[k0 + i] / 100 * lp.origin_peak;
        const double gf = gps * static_cast<double>(tv.v[i]) / 1e9;
        if (gf < 1e-9) g = -1.0;             // gamma = 1
        else if (total_gb == 0) g = -2.0;    // gamma = 0
        else g = gf / total_gb;
      }
      intensity[i] = g;
    }
  }
  store_vec<uint8_t, VEC>(p.origin_occ + k0, oocc);
  store_vec<uint32_t, VEC>(p.origin_waves + k0, owav);

  for (int d = 0; d < lp.D; ++d) {
    const hb_dev_pre& dd = c_dev[lp.dest_row[d]];
    const int64_t base = static_cast<int64_t>(d) * K + k0;
    Vec<float, VEC> outv;
    Vec<uint8_t, VEC> occv, stv;
    Vec<uint32_t, VEC> wavv;
    Vec<int16_t, VEC> drv;
    if (p.dest_regs) drv = load_vec<int16_t, VEC>(p.dest_regs + base);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int32_t nb = nbv.v[i];
      int32_t regs = rgv.v[i];
      if (p.dest_regs && drv.v[i] >= 0) regs = drv.v[i];
      const int32_t occ = hb_occupancy(dd, bsv.v[i], smem[i], regs, lim);
      if (EXTRA && p.limits) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          p.limits[(static_cast<int64_t>(d + 1) * 4 + j) * K + k0 + i] = lim[j];
      }
      const int32_t wave_d = dd.num_sms * occ;
      occv.v[i] = static_cast<uint8_t>(occ);
      wavv.v[i] = (wave_d > 0 && nb >= 1) ? static_cast<uint32_t>(nb / wave_d) : 0xFFFFFFFFu;

      double gamma;
      if (METRICS) {
        const double x = intensity[i];
        if (x == -1.0) gamma = 1.0;
        else if (x == -2.0) gamma = 0.0;
        else {
          const double r = lp.ridge[d];
          gamma = x > r ? 0.5 * r / x : -0.5 / r * x + 1.0;
        }
      } else {
        gamma = static_cast<double>(gv.v[i]);
      }

      // Mirrors the short-circuit of roofline.py:29-30: the destination wave
      // size is only examined when the kernel fits in one origin wave.
      int32_t st;
      double e = 0.0;  // log2 of the scale factor
      if (nb < 1) {
        st = HB_PAIR_BAD_INPUT;
      } else if (wave_o[i] == 0) {
        st = HB_PAIR_ZERO_WAVE;
      } else if (nb < wave_o[i]) {
        if (wave_d == 0) {
          st = HB_PAIR_ZERO_WAVE;
        } else if (nb < wave_d) {
          st = HB_PAIR_SMALL;
          const int32_t dmax = ceil_div_sms(nb, dd.num_sms);
          e = (1.0 - gamma) * (lp.log2_clk[d] + c_log2_int[dmax] - c_log2_int[omax[i]]);
        } else {
          st = HB_PAIR_LARGE;
        }
      } else {
        st = HB_PAIR_LARGE;
      }
      if (st == HB_PAIR_LARGE) e = fma(gamma, lp.a[d], lp.b[d]);
      outv.v[i] = st <= HB_PAIR_SMALL ? tv.v[i] * exp2f(static_cast<float>(e))
                                      : __int_as_float(0x7FC00000);
      stv.v[i] = static_cast<uint8_t>(st);
    }
    store_vec<float, VEC>(p.scaled_ns + base, outv);
    store_vec<uint8_t, VEC>(p.dest_occ + base, occv);
    store_vec<uint32_t, VEC>(p.dest_waves + base, wavv);
    if (EXTRA && p.status) store_vec<uint8_t, VEC>(p.status + base, stv);
  }
}


// ---------------------------------------------------------------------------
// Fast path.  The generic kernel above spends its time in the transcendental /
// conversion unit: every integer division compiles to reciprocal + conversion
// sequences, about ninety such operations per pair, and that unit issues sixteen
// lanes per clock.  When every row of the launch is "ordinary" (valid, warp size
// 32, fields small enough for 32-bit magic numbers - true of every real GPU) the
// divisions become multiply-high by magic numbers M[d] = floor(2^32 / d) + 1
// looked up in shared memory:
//   * divisors that depend on the kernel only (warps per block, register
//     allocation units, shared-memory allocation units) index one 512-entry
//     table loaded from global memory;
//   * the wave size of a pair is num_sms * occupancy with occupancy <= 32, so
//     each device gets a 33-entry table built at block start.
// ---------------------------------------------------------------------------
__device__ uint32_t g_magic[kMagicN];   // filled by hb_set_devices

template <int VEC, bool DEST_REGS>
__global__ void __launch_bounds__(256)
wave_scale_fast_kernel(const Ptrs p, const __grid_constant__ FastParams fp) {
  __shared__ uint32_t s_magic[kMagicN];
  __shared__ uint32_t s_wave_magic[HB_MAX_DEVICES / 2 + 1][33];
  __shared__ double s_log2[33];
  for (int i = threadIdx.x; i < kMagicN; i += blockDim.x) s_magic[i] = g_magic[i];
  for (int i = threadIdx.x; i < (fp.D + 1) * 33; i += blockDim.x) {
    const int d = i / 33, occ = i - d * 33;
    const uint32_t wave = static_cast<uint32_t>((d == 0 ? fp.origin.num_sms : fp.dest[d - 1].num_sms) * occ);
    s_wave_magic[d][occ] = wave >= 2u ? 0xFFFFFFFFu / wave + ((0xFFFFFFFFu % wave) + 1u == wave ? 1u : 0u) + 1u : 0u;
  }
  if (threadIdx.x < 33) s_log2[threadIdx.x] = c_log2_int[threadIdx.x];
  __syncthreads();

  const int64_t K = fp.K;
  const int64_t k0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * VEC;
  if (k0 >= K) return;

  const Vec<int32_t, VEC> nbv = load_vec<int32_t, VEC>(p.num_blocks + k0);
  const Vec<uint16_t, VEC> bsv = load_vec<uint16_t, VEC>(p.block_size + k0);
  const Vec<uint16_t, VEC> rgv = load_vec<uint16_t, VEC>(p.regs + k0);
  const Vec<uint32_t, VEC> smv = load_vec<uint32_t, VEC>(p.smem + k0);
  const Vec<float, VEC> tv = load_vec<float, VEC>(p.time_ns + k0);
  const Vec<float, VEC> gv = load_vec<float, VEC>(p.gamma + k0);

  FastKernel fk[VEC];
  uint32_t m_rpw[VEC];
  int32_t wave_o[VEC], omax[VEC];
  Vec<uint8_t, VEC> oocc;
  Vec<uint32_t, VEC> owav;
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    FastKernel& k = fk[i];
    k.block_size = bsv.v[i];
    k.wpb = (k.block_size + 31) >> 5;
    k.regs = rgv.v[i];
    k.rpw_units = (k.regs + 7) >> 3;               // roundup(regs * 32, 256) / 256
    k.smem = smv.v[i] > 0x7FFF0000u ? -1 : static_cast<int32_t>(smv.v[i]);
    k.m_wpb = s_magic[min(k.wpb, kMagicN - 1)];    // wpb <= 32 whenever the block can run
    m_rpw[i] = s_magic[min(k.rpw_units, kMagicN - 1)];
    const int32_t occ = fast_occupancy(fp.origin, k, k.regs, k.rpw_units, m_rpw[i], s_magic);
    const int32_t nb = nbv.v[i];
    wave_o[i] = fp.origin.num_sms * occ;
    oocc.v[i] = static_cast<uint8_t>(occ);
    owav.v[i] = (occ > 0 && nb >= 1)
                    ? udiv_magic_fix(static_cast<uint32_t>(nb), static_cast<uint32_t>(wave_o[i]),
                                     s_wave_magic[0][occ])
                    : 0xFFFFFFFFu;
    omax[i] = (nb >= 1 && nb < wave_o[i])
                  ? static_cast<int32_t>(udiv_magic(nb + fp.origin.num_sms - 1, fp.origin.num_sms,
                                                    fp.origin.sms_magic))
                  : 1;
  }
  store_vec<uint8_t, VEC>(p.origin_occ + k0, oocc);
  store_vec<uint32_t, VEC>(p.origin_waves + k0, owav);

  for (int d = 0; d < fp.D; ++d) {
    const FastDev& dd = fp.dest[d];
    const int64_t base = static_cast<int64_t>(d) * K + k0;
    Vec<float, VEC> outv;
    Vec<uint8_t, VEC> occv;
    Vec<uint32_t, VEC> wavv;
    Vec<int16_t, VEC> drv;
    if (DEST_REGS) drv = load_vec<int16_t, VEC>(p.dest_regs + base);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int32_t nb = nbv.v[i];
      int32_t regs = fk[i].regs, units = fk[i].rpw_units;
      uint32_t m = m_rpw[i];
      if (DEST_REGS && drv.v[i] >= 0) {
        regs = drv.v[i];
        units = (regs + 7) >> 3;
        m = s_magic[min(units, kMagicN - 1)];
      }
      const int32_t occ = fast_occupancy(dd, fk[i], regs, units, m, s_magic);
      const int32_t wave_d = dd.num_sms * occ;
      occv.v[i] = static_cast<uint8_t>(occ);
      wavv.v[i] = (occ > 0 && nb >= 1)
                      ? udiv_magic_fix(static_cast<uint32_t>(nb), static_cast<uint32_t>(wave_d),
                                       s_wave_magic[d + 1][occ])
                      : 0xFFFFFFFFu;
      const float gamma = gv.v[i];
      float e;
      bool ok = nb >= 1 && wave_o[i] != 0;
      if (ok && nb < wave_o[i] && nb < wave_d) {
        // small kernel (roofline.py:32-45); both per-SM block counts are <= 32
        const int32_t dmax = static_cast<int32_t>(udiv_magic(nb + dd.num_sms - 1, dd.num_sms, dd.sms_magic));
        e = static_cast<float>((1.0 - static_cast<double>(gamma)) *
                               (dd.log2_clk + s_log2[dmax] - s_log2[omax[i]]));
      } else {
        ok = ok && !(nb < wave_o[i] && wave_d == 0);
        e = fmaf(gamma, dd.a_hi, dd.b_hi) + fmaf(gamma, dd.a_lo, dd.b_lo);
      }
      outv.v[i] = ok ? tv.v[i] * exp2f(e) : __int_as_float(0x7FC00000);
    }
    store_vec<float, VEC>(p.scaled_ns + base, outv);
    store_vec<uint8_t, VEC>(p.dest_occ + base, occv);
    store_vec<uint32_t, VEC>(p.dest_waves + base, wavv);
  }
}


bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

bool vec4_ok(const Ptrs& p, int64_t K, bool need_gamma) {
  // The 4-wide path needs every plane base (d * K elements in) and every input
  // to sit on a 16-byte boundary for its widest type.
  return (K % 4 == 0) && aligned16(p.num_blocks) && aligned16(p.smem) && aligned16(p.time_ns) &&
         (!need_gamma || aligned16(p.gamma)) && aligned16(p.scaled_ns) && aligned16(p.dest_waves) &&
         aligned16(p.origin_waves) && (reinterpret_cast<uintptr_t>(p.block_size) % 8 == 0) &&
         (reinterpret_cast<uintptr_t>(p.regs) % 8 == 0) &&
         (reinterpret_cast<uintptr_t>(p.dest_occ) % 4 == 0) &&
         (reinterpret_cast<uintptr_t>(p.origin_occ) % 4 == 0) &&
         (!p.status || reinterpret_cast<uintptr_t>(p.status) % 4 == 0) &&
         (!p.dest_regs || reinterpret_cast<uintptr_t>(p.dest_regs) % 8 == 0);
}

// ---------------------------------------------------------------------------
// Table kernel.  Every device-dependent limit of a record is a function of small
// integers, so hb_set_devices tabulates, per device row and one byte each:
//   P[warps per block 0..33][256-register units per warp 0..33] =
//       min(register limit, warp limit, blocks-per-SM limit)
//   S[shared memory in 128-byte steps 0..2047] = shared-memory limit
// and, per occupancy 0..32, a 16-byte entry T[occ] = {M, sh, A_hi, A_lo}:
//   * floor(n / (SMs * occ)) = umulhi(n, M) >> sh for every 0 <= n < 2^31
//     (M = floor(2^(31+s) / wave) + 1 with s = ceil(log2 wave), sh = s - 1: the
//     error term n e / 2^(31+s) stays below 1 / wave because e <= wave <= 2^s),
//     so a pair's wave count is one table load, one multiply-high and a shift,
//     and "the kernel fits in one wave" is the test quotient == 0;
//   * A = log2(occ) - log2(clock MHz) as float hi + lo: the exponent of the
//     small-kernel rule (roofline.py:32-45) is (1 - gamma) (A_dest[blocks per SM
//     on the destination] - A_origin[blocks per SM on the origin]).
// Rows that agree on everything P (or S) reads form a class.  The tables of four classes lie interleaved in one
// table of words, so a record's bytes for up to four classes are one load (eight: two), and a destination picks
// its two bytes with a byte permute and takes one 16-bit-pair minimum for the two records a thread owns.  The
// tables a launch touches (a few KB) stay in L1.  The extended variant (EXT) adds, under launch-uniform branches,
// the status plane, per-destination register counts (another P word per pair that has one) and gamma from raw
// metrics (one float64 intensity per record, a compare and a multiply-add per pair).  Without classes (NW = 0, more
// than eight in a launch) it reads every device's own P and S bytes per pair.
// Conditions (checked on the host, else wave_scale_fast_kernel or the generic
// kernel runs): D <= 32, D K < 2^31, and per row 2 <= SMs <= 4096,
// blocks-per-SM limit <= 32, thread limit per block a multiple of 32 and <= 1024,
// shared-memory reserve a multiple of 128, shared-memory cap below the table's
// last step.
// ---------------------------------------------------------------------------
constexpr int kMaxWords = 2;     // class words per launch; table sizes, LutOcc and the table builder: occupancy.cuh

__device__ uint8_t g_lut_p[HB_MAX_DEVICES * kLutP];
__device__ uint8_t g_lut_s[HB_MAX_DEVICES * kLutS];
// The P (and S) tables of four classes in one word per index: one load brings a record's bytes of all four.
// Class c of the device table (classes are numbered as their first rows come) is byte c % 4 of word c / 4.
constexpr int kWords = HB_MAX_DEVICES / 4;
__device__ uint32_t g_lut_pw[kWords * kLutP];
__device__ uint32_t g_lut_sw[kWords * kLutS];
__device__ uint2 g_lut_m[HB_MAX_DEVICES * kLutOcc];    // {M, sh}
__device__ float2 g_lut_a[HB_MAX_DEVICES * kLutOcc];   // {A_hi, A_lo}

struct alignas(16) LutDev {       // three 16-byte groups, each fetched with one constant load
  uint32_t sel_p, sel_s;          // permute selectors: class byte of record 0 -> low half, record 1 -> high half
  uint32_t t_off;                 // byte offset of the row's T entries
  uint32_t p_off;                 // byte offset of the row's own P table (per-destination register counts)
  float a_hi, a_lo, b_hi, b_lo;   // large-kernel exponent gamma a + b, split float64 constants
  uint32_t sms_m1, sms_magic;     // SMs - 1 and floor(2^32 / SMs) + 1, for ceil(blocks / SMs)
  uint32_t s_off;                 // byte offset of the row's own S table (extended variant)
  uint32_t words;                 // bit 0 (1): the row's P (S) class is in the launch's second word
};
struct LutDevRegs {               // LutDev as read by a thread
  uint4 sel;
  float4 ab;
  uint4 sm;
};
__device__ __forceinline__ LutDevRegs load_lut_dev(const LutDev& d) {
  LutDevRegs r;
  r.sel = *reinterpret_cast<const uint4*>(&d.sel_p);
  r.ab = *reinterpret_cast<const float4*>(&d.a_hi);
  r.sm = *reinterpret_cast<const uint4*>(&d.sms_m1);
  return r;
}

struct LutParams {
  uint32_t K;
  uint32_t stride;                                   // elements from one output plane to the next
  int32_t D;
  uint32_t off_p[kMaxWords], off_s[kMaxWords];       // offsets of the class words' tables, in words
  double origin_peak;                                // metrics mode: origin peak GFLOP/s
  LutDev origin;
  LutDev dest[HB_MAX_DEVICES / 2];
  double ridge[HB_MAX_DEVICES / 2];                  // metrics mode: destination peak / bandwidth
  double slope[HB_MAX_DEVICES / 2];                  // -0.5 / ridge
  double half_ridge[HB_MAX_DEVICES / 2];
};

constexpr int kLutThreads = 128;

// prmt.b32 in its default mode: selector nibble n picks byte (n & 7) of {b, a}; with bit 3 set
// the byte's sign bit is replicated instead (0x00 for the values below 128 used here).
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

#if defined(HB_BOUNDS_CHECK)
// Checked build: every table index and element index is compared with its bound; a violation is
// recorded (first one wins) and the access redirected to element 0.  Nothing traps.
__device__ uint32_t g_bounds_word = 0;
__device__ __forceinline__ uint32_t hb_checked(uint32_t idx, uint32_t limit, uint32_t site) {
  if (idx >= limit) {
    atomicCAS(&g_bounds_word, 0u, (site << 24) | (idx & 0xFFFFFFu) | 0x80000000u);
    return 0u;
  }
  return idx;
}
#define HB_IDX(idx, limit, site) hb_checked((idx), (limit), (site))
#else
#define HB_IDX(idx, limit, site) (idx)
#endif

// Two records per thread (VEC = 2) need the inputs on 8-byte boundaries; GAP = 0 says that the output planes are
// too (K even), so results leave as 8-byte stores.  Otherwise (odd K: every other plane starts on an odd element) the
// same two-record arithmetic ends in scalar stores, and a thread with a single record loads it alone.  The records of
// a thread are then neighbours (GAP = 1), or (GAP = 32) so far apart that each of a warp's accesses is one piece
// of 32 elements: with metrics, four arrays of which are loaded one element at a time in any case, that is 2 to 5 %
// faster up to eight destinations (1,000,001 x 6: 33.6 -> 32.6 us, x 1: 14.9 -> 14.3; 4,000,001 x 6: 113.3 -> 111.5) and
// 1 % slower with thirteen; without metrics the vector loads are worth more (1,000,001 x 6: 19.4 against 21.1).  The line
// lies where middle batches change sides (every destination with a register count of its own: 1,000,001 x 8: 44.4 ->
// 44.2, x 9: 48.6 -> 48.4, x 10: 52.1 -> 52.3, x 13: 63.7 -> 64.3); small ones gain beyond it too (250,001 x 8: 15.2 ->
// 14.7, x 16: 24.4 -> 24.0), large ones lose below it already (4,000,001 x 6: 121.3 -> 121.8, x 8: 149.8 -> 150.9).
template <typename T, int VEC, uint32_t GAP>
__device__ __forceinline__ Vec<T, VEC> load_pair(const T* q, bool pair) {
  if (VEC == 1 || GAP == 0) return load_vec<T, VEC>(q);
  Vec<T, VEC> v;
  if (GAP == 1 && pair) {
    v = load_vec<T, VEC>(q);
  } else {
    v.v[0] = q[0];
    v.v[VEC - 1] = GAP > 1 && pair ? q[GAP] : q[0];
  }
  return v;
}
// The same without vector loads, for arrays of any alignment.
template <typename T, int VEC, uint32_t GAP>
__device__ __forceinline__ Vec<T, VEC> load_each(const T* q, bool pair) {
  Vec<T, VEC> v;
  v.v[0] = q[0];
  if (VEC == 2) v.v[VEC - 1] = pair ? q[GAP ? GAP : 1] : q[0];
  return v;
}
template <typename T, int VEC, uint32_t GAP>
__device__ __forceinline__ void store_pair(T* q, const Vec<T, VEC>& v, bool pair) {
  if (VEC == 1 || GAP == 0) {
    store_vec<T, VEC>(q, v);
  } else {
    q[0] = v.v[0];
    if (pair) q[GAP] = v.v[VEC - 1];
  }
}
// The low bytes of the two 16-bit halves of `pair_word` as one or two bytes at q.
template <int VEC, uint32_t GAP>
__device__ __forceinline__ void store_byte_pair(uint8_t* q, uint32_t pair_word, bool pair) {
  if (VEC == 2 && GAP == 0) {
    *reinterpret_cast<uint16_t*>(q) = static_cast<uint16_t>(__byte_perm(pair_word, 0u, 0x4420u));
  } else {
    q[0] = static_cast<uint8_t>(pair_word);
    if (VEC == 2 && pair) q[GAP] = static_cast<uint8_t>(pair_word >> 16);
  }
}

// TOT: every block also adds up its own results per destination (float64, fixed order, NaN results
// skipped like the plane sums do) and leaves the sums in p.block_sums[d * gridDim.x + block], so
// the totals of a launch need no second pass over the [D x K] plane.  A thread parks the float64
// sum of its two results per destination in shared memory; at the end TOT lanes per destination (sixteen up to eight
// destinations, eight up to kTotMaxD) add the block's 128 sums.  Needs a grid that covers the batch in one pass.
constexpr int kTotMaxD = 16;

// EXT: 0 plain, 1 with the status plane and per-destination registers, 2 and 3 with gamma from metrics as well,
// whose float64 values take 20 registers.  With 56 registers (2) nine blocks fit an SM, with 48 (3) ten.  Batches of
// more than two fills of the first take the second: with register counts it is 4 to 8 % faster (4,000,000 kernels x 6:
// 113.7 -> 105.4 us, 11,184,812 x 6: 310 -> 287), without them up to 5 % faster with one or two destinations (8,000,000
// x 1: 73.7 -> 69.9) and 1 to 4 % slower with more (4,000,000 x 6: 81.8 -> 84.8).  Smaller batches are slower with the
// second (500,000 x 6: 17.4 -> 18.2 us, 250,000 x 13: 21.0 -> 24.0, with register counts).
template <int VEC, int EXT, bool ALIGNED, int NW, int TOT = 0, bool FAR = false>
__global__ void __launch_bounds__(kLutThreads, EXT == 2 ? 8 : (EXT == 3 ? 10 : 12))
wave_scale_lut_kernel(const Ptrs p, const __grid_constant__ LutParams lp) {
  static_assert(!TOT || (VEC == 2 && EXT == 0), "fused totals: plain two-record variants only");
  extern __shared__ __align__(16) double s_tot_raw[];   // TOT: [D][kLutThreads]
  double(*s_tot)[kLutThreads] = reinterpret_cast<double(*)[kLutThreads]>(s_tot_raw);
  hb_grid_dependency_wait();
  const uint32_t K = lp.K;
  const int D = lp.D;
  static_assert(!FAR || (VEC == 2 && !ALIGNED), "two records per thread, scalar stores");
  constexpr uint32_t GAP = ALIGNED ? 0 : (FAR ? 32 : 1);
  // a warp owns 32 VEC records in a row
  const uint32_t k0 = GAP > 1 ? (blockIdx.x * kLutThreads + (threadIdx.x & ~31u)) * VEC + (threadIdx.x & 31u)
                              : (blockIdx.x * kLutThreads + threadIdx.x) * VEC;
  if (TOT && k0 >= K) {
    for (int d = 0; d < D; ++d) s_tot[d][threadIdx.x] = 0.0;   // threads past the end
  }
  const uint8_t* __restrict__ tab_m = reinterpret_cast<const uint8_t*>(g_lut_m);
  const uint8_t* __restrict__ tab_a = reinterpret_cast<const uint8_t*>(g_lut_a);
  const bool with_regs = EXT && p.dest_regs != nullptr;
  constexpr bool with_metrics = EXT >= 2;
  const bool with_status = EXT && p.status != nullptr;

  if (k0 < K) {
    const bool pair = VEC == 2 && (ALIGNED || k0 + GAP < K);   // false: a single record at the end of an odd batch
    const Vec<int32_t, VEC> nbv = load_pair<int32_t, VEC, GAP>(p.num_blocks + k0, pair);
    const Vec<uint16_t, VEC> bsv = load_pair<uint16_t, VEC, GAP>(p.block_size + k0, pair);
    const Vec<uint16_t, VEC> rgv = load_pair<uint16_t, VEC, GAP>(p.regs + k0, pair);
    const Vec<uint32_t, VEC> smv = load_pair<uint32_t, VEC, GAP>(p.smem + k0, pair);
    const Vec<float, VEC> tv = load_pair<float, VEC, GAP>(p.time_ns + k0, pair);
    Vec<float, VEC> gv;
    if (!with_metrics) gv = load_pair<float, VEC, GAP>(p.gamma + k0, pair);
    Vec<double, VEC> fev, rdv, wrv;
    Vec<uint8_t, VEC> hmv;
    if (with_metrics) {   // all on their way at once, not the values behind the flag (3,000,000 x 2: 39.1 -> 35.7 us)
      hmv = load_each<uint8_t, VEC, GAP>(p.has_metrics + k0, pair);
      fev = load_each<double, VEC, GAP>(p.flop_eff + k0, pair);
      rdv = load_each<double, VEC, GAP>(p.dram_read + k0, pair);
      wrv = load_each<double, VEC, GAP>(p.dram_write + k0, pair);
    }

    uint32_t P[2] = {0u, 0u}, S[2] = {0u, 0u};     // class bytes of the two records
    uint32_t P2[2] = {0u, 0u}, S2[2] = {0u, 0u};   // ... of the launch's second word
    // occupancies of the two records on a device, in the halves of a word
    auto occ_pair = [&](const LutDevRegs& r) {
      const bool p2 = NW == 2 && (r.sm.w & 1u), s2 = NW == 2 && (r.sm.w & 2u);
      return __vimin_s16x2_relu(prmt(p2 ? P2[0] : P[0], p2 ? P2[1] : P[1], r.sel.x),
                                prmt(s2 ? S2[0] : S[0], s2 ? S2[1] : S[1], r.sel.y));
    };
    uint32_t wrow[2] = {0u, 0u};                 // EXT: warps per block x row length (P index base)
    float omg[2] = {0.0f, 0.0f};
    double xint[2] = {0.0, 0.0}, xinv[2] = {0.0, 0.0};   // EXT: intensity and 1 / intensity
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const uint32_t wpb = min((static_cast<uint32_t>(bsv.v[i]) + 31u) >> 5, static_cast<uint32_t>(kLutW - 1));
      const uint32_t pidx = HB_IDX(lut_p_index(bsv.v[i], rgv.v[i]), kLutP, 1);
      const uint32_t steps = HB_IDX(lut_s_index(smv.v[i]), kLutS, 2);
      if (NW > 0) {
        P[i] = __ldg(g_lut_pw + (lp.off_p[0] + pidx));
        S[i] = __ldg(g_lut_sw + (lp.off_s[0] + steps));
        if (NW == 2) {
          P2[i] = __ldg(g_lut_pw + (lp.off_p[1] + pidx));
          S2[i] = __ldg(g_lut_sw + (lp.off_s[1] + steps));
        }
      } else {
        P[i] = pidx; S[i] = steps;   // every device's own tables are indexed directly (no class limit)
      }
      if (EXT) wrow[i] = wpb * kLutU;
      if (!with_metrics) omg[i] = 1.0f - gv.v[i];
      if (with_metrics) {
        // wave_scaling/roofline.py:68-92, float64.  The rule below gives gamma 1 for intensity 0 and gamma 0
        // for an infinite one, which is how its two special cases are written here: no metrics or next to no
        // floating-point work, and no memory traffic.  Reciprocals, not divisions: two of those per record were
        // 15 % of the kernel.
        if (hmv.v[i]) {
          const double total_gb = (rdv.v[i] + wrv.v[i]) / 1024 / 1024 / 1024;
          const double gf = fev.v[i] * (lp.origin_peak / 100 / 1e9) * static_cast<double>(tv.v[i]);
          if (!(gf < 1e-9)) {
            xint[i] = total_gb == 0 ? __longlong_as_double(0x7FF0000000000000ll) : gf * __drcp_rn(total_gb);
            xinv[i] = total_gb == 0 ? 0.0 : total_gb * __drcp_rn(gf);
          }
        }
      }
    }

    // origin: both records at once
    const LutDevRegs og = load_lut_dev(lp.origin);
    uint32_t o2;
    if (NW > 0) {
      o2 = occ_pair(og);
    } else {
      o2 = 0;
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const uint32_t pb = __ldg(g_lut_p + (og.sel.w + P[i]));
        const uint32_t sb = __ldg(g_lut_s + (og.sm.z + S[i]));
        o2 |= min(pb, sb) << (16 * i);
      }
    }
    bool nbok[2] = {false, false}, live[2] = {false, false}, fits_o[2] = {false, false};
    float2 lg_o[2];
    Vec<uint32_t, VEC> owav;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const uint32_t occ = i == 0 ? (o2 & 0xFFFFu) : (o2 >> 16);
      const int32_t nb = nbv.v[i];
      const uint2 w = __ldg(reinterpret_cast<const uint2*>(tab_m + (og.sel.z + HB_IDX(occ, kLutOcc, 3) * 8u)));
      const uint32_t q = __umulhi(static_cast<uint32_t>(nb), w.x) >> w.y;
      nbok[i] = nb >= 1;
      live[i] = nbok[i] && occ != 0u;
      owav.v[i] = live[i] ? q : 0xFFFFFFFFu;
      fits_o[i] = live[i] && q == 0u;            // num_blocks < origin wave size
      // ceil(num_blocks / SMs) <= occupancy <= 32 whenever the small-kernel rule applies; otherwise
      // the entry read here is never used, and the clamp only keeps the index inside the table.  Not
      // selecting on fits_o keeps this load independent of the one above.
      const uint32_t om = min(__umulhi(static_cast<uint32_t>(nb) + og.sm.x, og.sm.y), static_cast<uint32_t>(kLutOcc - 1));
      lg_o[i] = __ldg(reinterpret_cast<const float2*>(tab_a + (og.sel.z + HB_IDX(om, kLutOcc, 4) * 8u)));
    }
    store_byte_pair<VEC, GAP>(p.origin_occ + k0, o2, pair);
    store_pair<uint32_t, VEC, GAP>(p.origin_waves + k0, owav, pair);

    // The plain instances keep what they know about a record in masks: six predicates that live through the loop
    // leave none for the body, and the masks go into one logic operation per question (11,184,812 x 6 with totals:
    // 175 -> 173.8 us, 8,388,608 x 6: 117.5 -> 116.3).
    uint32_t no_blocks[2], not_live[2], not_fit[2];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      no_blocks[i] = nbok[i] ? 0u : ~0u;
      not_live[i] = live[i] ? 0u : ~0u;
      not_fit[i] = fits_o[i] ? 0u : ~0u;
    }

    // per-destination register counts of the two records (-1: the record's own)
    auto load_regs = [&](uint32_t at) {
      Vec<int16_t, VEC> r;
      if (VEC == 1 || ALIGNED) {
        r = load_vec<int16_t, VEC>(p.dest_regs + at);
      } else {
        r.v[0] = p.dest_regs[at];
        r.v[VEC - 1] = pair ? p.dest_regs[at + GAP] : static_cast<int16_t>(-1);
      }
      return r;
    };
    Vec<int16_t, VEC> drv;
    if (with_regs) drv = load_regs(k0);

#pragma unroll 1
    for (int d = 0; d < D; ++d) {
      const LutDevRegs dd = load_lut_dev(lp.dest[d]);
      const uint32_t base = static_cast<uint32_t>(d) * lp.stride + k0;   // D K < 2^31
      uint32_t occ2;
      if (!EXT) {
        occ2 = occ_pair(dd);
      } else {
        // the next destination's counts are on their way while this one is worked on
        const Vec<int16_t, VEC> now = drv;
        if (with_regs && d + 1 < D) drv = load_regs(base + lp.stride);
        uint32_t over[2] = {0u, 0u};   // P index of a record that MetadataManager.kernel_registers_for gave other registers
        bool other[2] = {false, false};
        if (with_regs) {
#pragma unroll
          for (int i = 0; i < VEC; ++i) {
            other[i] = now.v[i] >= 0;
            const uint32_t units = min((static_cast<uint32_t>(now.v[i]) + 7u) >> 3, static_cast<uint32_t>(kLutU - 1));
            over[i] = HB_IDX(wrow[i] + units, kLutP, 5);
          }
        }
        if (NW > 0) {
          const bool p2 = NW == 2 && (dd.sm.w & 1u), s2 = NW == 2 && (dd.sm.w & 2u);
          uint32_t pw[2] = {p2 ? P2[0] : P[0], p2 ? P2[1] : P[1]};
          if (with_regs) {
#pragma unroll
            for (int i = 0; i < VEC; ++i)
              if (other[i]) pw[i] = __ldg(g_lut_pw + (lp.off_p[p2 ? 1 : 0] + over[i]));
          }
          occ2 = __vimin_s16x2_relu(prmt(pw[0], pw[1], dd.sel.x), prmt(s2 ? S2[0] : S[0], s2 ? S2[1] : S[1], dd.sel.y));
        } else {
          occ2 = 0;
#pragma unroll
          for (int i = 0; i < VEC; ++i) {
            const uint32_t pb = __ldg(g_lut_p + (dd.sel.w + (other[i] ? over[i] : P[i])));
            const uint32_t sb = __ldg(g_lut_s + (dd.sm.z + S[i]));
            occ2 |= min(pb, sb) << (16 * i);
          }
        }
      }
      Vec<float, VEC> outv;
      Vec<uint32_t, VEC> wavv;
      uint32_t st2 = 0;
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const uint32_t occ = i == 0 ? (occ2 & 0xFFFFu) : (occ2 >> 16);
        const int32_t nb = nbv.v[i];
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(tab_m + (dd.sel.z + HB_IDX(occ, kLutOcc, 6) * 8u)));
        const uint32_t q = __umulhi(static_cast<uint32_t>(nb), w.x) >> w.y;
        const bool has_wave = occ != 0u;
        // roofline.py:29-30 with its short circuit: the destination is only looked at when the
        // kernel fits in one origin wave
        bool small, ok;
        if (EXT) {
          wavv.v[i] = (nbok[i] && has_wave) ? q : 0xFFFFFFFFu;
          small = fits_o[i] && has_wave && q == 0u;
          ok = live[i] && !(fits_o[i] && !has_wave);
        } else {
          const uint32_t waves = (has_wave ? q : 0xFFFFFFFFu) | no_blocks[i];
          wavv.v[i] = waves;
          small = (waves | not_fit[i]) == 0u;
          ok = (~not_live[i] & (~waves | not_fit[i])) != 0u;
        }
        // blocks per SM on the destination: meaningful (and <= occupancy) when `small`; computed from
        // the record alone so that this table load does not wait for the one above
        const uint32_t dm = min(__umulhi(static_cast<uint32_t>(nb) + dd.sm.x, dd.sm.y), static_cast<uint32_t>(kLutOcc - 1));
        const float2 lg_d = __ldg(reinterpret_cast<const float2*>(tab_a + (dd.sel.z + HB_IDX(dm, kLutOcc, 7) * 8u)));
        float gamma, one_minus;
        if (with_metrics) {
          const double gm = xint[i] > lp.ridge[d] ? lp.half_ridge[d] * xinv[i] : fma(lp.slope[d], xint[i], 1.0);
          gamma = static_cast<float>(gm);
          one_minus = static_cast<float>(1.0 - gm);
        } else {
          gamma = gv.v[i];
          one_minus = omg[i];
        }
        const float e_small = one_minus * ((lg_d.x - lg_o[i].x) + (lg_d.y - lg_o[i].y));
        const float e_large = fmaf(gamma, dd.ab.x, dd.ab.z) + fmaf(gamma, dd.ab.y, dd.ab.w);
        const float e = small ? e_small : e_large;
        outv.v[i] = ok ? tv.v[i] * ex2_approx(e) : __int_as_float(0x7FC00000);
        if (with_status) {
          const uint32_t st = !nbok[i] ? HB_PAIR_BAD_INPUT
                                       : (!ok ? HB_PAIR_ZERO_WAVE : (small ? HB_PAIR_SMALL : HB_PAIR_LARGE));
          st2 |= st << (16 * i);
        }
      }
      store_pair<float, VEC, GAP>(p.scaled_ns + base, outv, pair);
      store_pair<uint32_t, VEC, GAP>(p.dest_waves + base, wavv, pair);
      store_byte_pair<VEC, GAP>(p.dest_occ + base, occ2, pair);
      if (with_status) store_byte_pair<VEC, GAP>(p.status + base, st2, pair);
      if (TOT) {
        const float g0 = outv.v[0] == outv.v[0] ? outv.v[0] : 0.0f;                     // NaN: no prediction
        const float g1 = pair && outv.v[VEC - 1] == outv.v[VEC - 1] ? outv.v[VEC - 1] : 0.0f;
        s_tot[d][threadIdx.x] = static_cast<double>(g0) + static_cast<double>(g1);   // exact
      }
    }
  }
  if (TOT) {
    __syncthreads();
    constexpr int kLanes = TOT ? TOT : 16;
    const int d = threadIdx.x / kLanes, j = threadIdx.x % kLanes;
    double acc = 0.0;
    if (d < D) {
      const double2* row = reinterpret_cast<const double2*>(s_tot[d]);
#pragma unroll
      for (int i = 0; i < kLutThreads / (2 * kLanes); ++i) {
        const double2 x = row[j + kLanes * i];
        acc += x.x + x.y;
      }
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, o, kLanes);
    if (j == 0 && d < D) p.block_sums[static_cast<size_t>(d) * gridDim.x + blockIdx.x] = acc;
  }
}

// ---------------------------------------------------------------------------
// Host side: device table, per-GPU upload, launch selection
// ---------------------------------------------------------------------------
// The table hb_set_devices receives is kept on the host; every GPU of the process gets its own
// copy (constant rows, tabulated limits) the first time it is used after a change, so one
// process may drive several GPUs.  All of it is guarded by one mutex; hb_wave_scale only takes
// the lock when the current GPU's copy is stale.
constexpr int kMaxCudaDevices = 64;

struct HostTable {
  int n = 0;
  hb_device_spec rows[HB_MAX_DEVICES];
  hb_dev_pre pre[HB_MAX_DEVICES];
  bool lut_ok[HB_MAX_DEVICES] = {};
  uint64_t row_version[HB_MAX_DEVICES] = {};   // bumped when a row's specification changes
  std::vector<uint8_t> lut_p = std::vector<uint8_t>(static_cast<size_t>(HB_MAX_DEVICES) * kLutP);
  std::vector<uint8_t> lut_s = std::vector<uint8_t>(static_cast<size_t>(HB_MAX_DEVICES) * kLutS);
  std::vector<LutOcc> lut_t = std::vector<LutOcc>(static_cast<size_t>(HB_MAX_DEVICES) * kLutOcc);
  // classes of rows that agree on everything P (S) reads, and their tables four to a word
  FastDev fast[HB_MAX_DEVICES];
  std::vector<FastDev> p_reps, s_reps;
  int p_class[HB_MAX_DEVICES] = {}, s_class[HB_MAX_DEVICES] = {};
  std::vector<uint32_t> words_p = std::vector<uint32_t>(static_cast<size_t>(kWords) * kLutP);
  std::vector<uint32_t> words_s = std::vector<uint32_t>(static_cast<size_t>(kWords) * kLutS);
};
struct GpuCopy {
  std::atomic<bool> constants{false};          // row-independent tables uploaded (read without the lock)
  uint64_t row_version[HB_MAX_DEVICES] = {};   // version of each row this GPU holds
  int sm_count = 0;
};

std::mutex g_mu;
HostTable g_tab;
GpuCopy g_gpu[kMaxCudaDevices];
std::atomic<uint64_t> g_version{0};                       // bumped by every hb_set_devices that changed a row
std::atomic<uint64_t> g_gpu_version[kMaxCudaDevices];     // table version each GPU has seen

// Brings the current GPU's copy of the table up to date (rows that changed since its last
// upload, plus the row-independent tables on first use).  Synchronises the device when it
// uploads anything, so launches on any stream see the new rows.
hb_status sync_gpu(int* sm_count) {
  int dev = 0;
  HB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxCudaDevices) {
    hb::set_error("hb_wave_scale: device ordinal %d out of range", dev);
    return HB_ERR_UNSUPPORTED;
  }
  if (g_gpu_version[dev].load(std::memory_order_acquire) == g_version.load(std::memory_order_acquire) &&
      g_gpu[dev].constants.load(std::memory_order_acquire)) {
    if (sm_count) *sm_count = g_gpu[dev].sm_count;
    return HB_OK;
  }
  std::lock_guard<std::mutex> lock(g_mu);
  GpuCopy& gc = g_gpu[dev];
  bool uploaded = false;
  if (!gc.constants.load(std::memory_order_relaxed)) {
    HB_CUDA_TRY(cudaDeviceGetAttribute(&gc.sm_count, cudaDevAttrMultiProcessorCount, dev));
    double lg[65];
    lg[0] = 0.0;
    for (int i = 1; i <= 64; ++i) lg[i] = std::log2(static_cast<double>(i));
    HB_CUDA_TRY(cudaMemcpyToSymbol(c_log2_int, lg, sizeof(lg)));
    uint32_t magic[kMagicN];
    for (int i = 0; i < kMagicN; ++i) magic[i] = magic_of(static_cast<uint32_t>(i));
    HB_CUDA_TRY(cudaMemcpyToSymbol(g_magic, magic, sizeof(magic)));
    gc.constants.store(true, std::memory_order_release);
    uploaded = true;
  }
  for (int i = 0; i < g_tab.n; ++i) {
    if (gc.row_version[i] == g_tab.row_version[i]) continue;
    HB_CUDA_TRY(cudaMemcpyToSymbol(c_dev, &g_tab.pre[i], sizeof(hb_dev_pre), sizeof(hb_dev_pre) * i));
    HB_CUDA_TRY(cudaMemcpyToSymbol(g_lut_p, &g_tab.lut_p[static_cast<size_t>(i) * kLutP], kLutP,
                                   static_cast<size_t>(i) * kLutP));
    HB_CUDA_TRY(cudaMemcpyToSymbol(g_lut_s, &g_tab.lut_s[static_cast<size_t>(i) * kLutS], kLutS,
                                   static_cast<size_t>(i) * kLutS));
    uint2 m[kLutOcc];
    float2 a[kLutOcc];
    for (int occ = 0; occ < kLutOcc; ++occ) {
      const LutOcc& e = g_tab.lut_t[static_cast<size_t>(i) * kLutOcc + occ];
      m[occ] = make_uint2(e.magic, e.shift);
      a[occ] = make_float2(e.lg_hi, e.lg_lo);
    }
    HB_CUDA_TRY(cudaMemcpyToSymbol(g_lut_m, m, sizeof(m), sizeof(m) * i));
    HB_CUDA_TRY(cudaMemcpyToSymbol(g_lut_a, a, sizeof(a), sizeof(a) * i));
    gc.row_version[i] = g_tab.row_version[i];
    uploaded = true;
  }
  if (uploaded) {
    const size_t p_words = (g_tab.p_reps.size() + 3) / 4, s_words = (g_tab.s_reps.size() + 3) / 4;
    if (p_words) HB_CUDA_TRY(cudaMemcpyToSymbol(g_lut_pw, g_tab.words_p.data(), sizeof(uint32_t) * kLutP * p_words));
    if (s_words) HB_CUDA_TRY(cudaMemcpyToSymbol(g_lut_sw, g_tab.words_s.data(), sizeof(uint32_t) * kLutS * s_words));
  }
  if (uploaded) HB_CUDA_TRY(cudaDeviceSynchronize());
  g_gpu_version[dev].store(g_version.load(std::memory_order_acquire), std::memory_order_release);
  if (sm_count) *sm_count = gc.sm_count;
  return HB_OK;
}

uint32_t pair_selector(int c) {
  const uint32_t lo = static_cast<uint32_t>(c), hi = static_cast<uint32_t>(4 + c);
  return lo | ((8u | lo) << 4) | (hi << 8) | ((8u | hi) << 12);
}

bool same_p_class(const FastDev& a, const FastDev& b) {
  return same_regs_class(a, b) && same_warps_class(a, b) && a.blocks_limit == b.blocks_limit;
}

// The class of row `row` among `reps` (made now if it is new, its table put into the words); -1 when all
// numbers are taken.  A class keeps its number and its bytes for good, so a launch that was planned with an older
// table still finds them.  Call with g_mu held.
template <typename Same>
int class_of(std::vector<FastDev>& reps, std::vector<uint32_t>& words, const std::vector<uint8_t>& rows, int len, int row,
             Same same) {
  const FastDev& f = g_tab.fast[row];
  for (size_t c = 0; c < reps.size(); ++c)
    if (same(reps[c], f)) return static_cast<int>(c);
  if (reps.size() == HB_MAX_DEVICES) return -1;
  const size_t c = reps.size();
  reps.push_back(f);
  for (int i = 0; i < len; ++i)
    words[c / 4 * len + i] |= static_cast<uint32_t>(rows[static_cast<size_t>(row) * len + i]) << (8 * (c % 4));
  return static_cast<int>(c);
}

template <int VEC, int EXT, bool ALIGNED, int NW, int TOT = 0, bool FAR = false>
cudaError_t launch_lut(unsigned grid, cudaStream_t stream, const Ptrs& p, const LutParams& q) {
  return hb::launch_overlapped(wave_scale_lut_kernel<VEC, EXT, ALIGNED, NW, TOT, FAR>, dim3(grid), dim3(kLutThreads),
                               TOT ? sizeof(double) * kLutThreads * q.D : 0, stream, p, q);
}

// Everything about a launch that depends on the devices alone.  Callers ask for the same origin and
// destinations again and again, so a thread keeps its last few plans; a plan is of one version of the
// device table and holds no results.
struct LaunchPlan {
  uint64_t version = 0;
  LaunchParams lp{};
  bool lut_ok = false;         // every row can be tabulated
  int words = 1;               // class words the rows need; more than kMaxWords: every row's own tables (extended variant)
  LutParams q{};
};

void fill_lut(LaunchPlan* plan) {   // call with g_mu held
  const LaunchParams& lp = plan->lp;
  LutParams& q = plan->q;
  plan->lut_ok = lp.D <= HB_MAX_DEVICES / 2 && g_tab.lut_ok[lp.origin_row];
  for (int d = 0; d < lp.D && plan->lut_ok; ++d) plan->lut_ok = g_tab.lut_ok[lp.dest_row[d]];
  if (!plan->lut_ok) return;
  int words_p[HB_MAX_DEVICES], words_s[HB_MAX_DEVICES], n_p = 0, n_s = 0;
  auto slot_of = [](int* words, int* n, int word) {
    for (int i = 0; i < *n; ++i)
      if (words[i] == word) return i;
    words[*n] = word;
    return (*n)++;
  };
  for (int d = -1; d < lp.D; ++d) {
    const int row = d < 0 ? lp.origin_row : lp.dest_row[d];
    const int pc = g_tab.p_class[row], sc = g_tab.s_class[row];
    if (pc < 0 || sc < 0) plan->words = kMaxWords + 1;
    LutDev& o = d < 0 ? q.origin : q.dest[d];
    o.sel_p = pair_selector(pc & 3);
    o.sel_s = pair_selector(sc & 3);
    o.words = static_cast<uint32_t>((slot_of(words_p, &n_p, pc >> 2) & 1) | (slot_of(words_s, &n_s, sc >> 2) & 1) << 1);
    o.t_off = static_cast<uint32_t>(row * kLutOcc * sizeof(uint2));
    o.p_off = static_cast<uint32_t>(row * kLutP);
    o.s_off = static_cast<uint32_t>(row * kLutS);
    o.sms_m1 = static_cast<uint32_t>(g_tab.rows[row].num_sms - 1);
    o.sms_magic = magic_of(static_cast<uint32_t>(g_tab.rows[row].num_sms));
    if (d >= 0) {
      o.a_hi = static_cast<float>(lp.a[d]);
      o.a_lo = static_cast<float>(lp.a[d] - static_cast<double>(o.a_hi));
      o.b_hi = static_cast<float>(lp.b[d]);
      o.b_lo = static_cast<float>(lp.b[d] - static_cast<double>(o.b_hi));
      q.ridge[d] = lp.ridge[d];
      q.slope[d] = -0.5 / lp.ridge[d];
      q.half_ridge[d] = 0.5 * lp.ridge[d];
    }
  }
  plan->words = std::max({plan->words, n_p, n_s});
  for (int w = 0; w < kMaxWords; ++w) {   // a word that is not needed repeats the first
    q.off_p[w] = static_cast<uint32_t>(std::max(words_p[w < n_p ? w : 0], 0) * kLutP);
    q.off_s[w] = static_cast<uint32_t>(std::max(words_s[w < n_s ? w : 0], 0) * kLutS);
  }
  q.D = lp.D;
  q.origin_peak = lp.origin_peak;
}

// Launches wave_scale_lut_kernel when the launch qualifies; false = nothing launched.  *fused says
// whether the launch also wrote p.block_sums (one sum per destination and block of the grid).
// Output planes (and dest_regs) are `stride` >= K elements apart.
bool try_launch_lut(const Ptrs& p, const LaunchPlan& plan, int64_t K, int64_t stride, int sm_count, cudaStream_t stream,
                    hb_status* st, bool* fused, unsigned* fused_blocks, bool to_host = false) {
  *fused = false;
  static const bool use_lut = [] { const char* e = std::getenv("HB_WAVE_LUT"); return !e || std::atoi(e) != 0; }();
  const LaunchParams& lp = plan.lp;
  if (!use_lut || p.limits || !plan.lut_ok) return false;
  if (static_cast<int64_t>(lp.D) * stride >= (int64_t{1} << 31)) return false;   // 32-bit element indices
  LutParams q = plan.q;
  q.K = static_cast<uint32_t>(K);
  q.stride = static_cast<uint32_t>(stride);

  auto al = [](const void* ptr, uintptr_t a) { return (reinterpret_cast<uintptr_t>(ptr) & (a - 1)) == 0; };
  const bool metrics = p.has_metrics != nullptr;
  const bool ext = metrics || p.dest_regs != nullptr || p.status != nullptr || plan.words > kMaxWords;
  // two records per thread when the inputs sit on 8-byte boundaries; 8-byte stores when the
  // output planes do too (K even)
  const bool vec2 = al(p.num_blocks, 8) && al(p.smem, 8) && al(p.time_ns, 8) && (metrics || al(p.gamma, 8)) &&
                    al(p.block_size, 4) && al(p.regs, 4) && K >= 2 &&
                    // over PCIe every warp's store should be one piece: no two-record threads with odd planes
                    !(to_host && stride % 2 != 0);
  const bool aligned = vec2 && K % 2 == 0 && stride % 2 == 0 && al(p.scaled_ns, 8) && al(p.dest_waves, 8) && al(p.origin_waves, 8) &&
                       al(p.dest_occ, 2) && al(p.origin_occ, 2) && (!p.status || al(p.status, 2)) &&
                       (!p.dest_regs || al(p.dest_regs, 4));
  const int vec = vec2 ? 2 : 1;
  const int64_t blocks = ((K + vec - 1) / vec + kLutThreads - 1) / kLutThreads;
  // One block per 128 threads' worth of records measured fastest at every batch size: the block scheduler
  // balances the tail (persistent blocks that stride over the batch were slower throughout).
  const unsigned grid = static_cast<unsigned>(blocks);
  const bool two = plan.words == 2;
  cudaError_t le;
  if (ext) {
    auto launch_ext = [&](auto words) {
      constexpr int W = decltype(words)::value;
      const bool large = blocks > 18ll * sm_count;
      if (metrics && vec2 && !aligned && lp.D <= 8)   // see GAP
        return large ? launch_lut<2, 3, false, W, 0, true>(grid, stream, p, q) : launch_lut<2, 2, false, W, 0, true>(grid, stream, p, q);
      if (metrics && vec2 && large)
        return aligned ? launch_lut<2, 3, true, W>(grid, stream, p, q) : launch_lut<2, 3, false, W>(grid, stream, p, q);
      if (metrics)
        return !vec2 ? launch_lut<1, 2, true, W>(grid, stream, p, q)
                     : (aligned ? launch_lut<2, 2, true, W>(grid, stream, p, q) : launch_lut<2, 2, false, W>(grid, stream, p, q));
      return !vec2 ? launch_lut<1, 1, true, W>(grid, stream, p, q)
                   : (aligned ? launch_lut<2, 1, true, W>(grid, stream, p, q) : launch_lut<2, 1, false, W>(grid, stream, p, q));
    };
    le = plan.words > kMaxWords ? launch_ext(std::integral_constant<int, 0>{})
                                : (two ? launch_ext(std::integral_constant<int, 2>{}) : launch_ext(std::integral_constant<int, 1>{}));
  } else if (!vec2) {
    le = launch_lut<1, 0, true, 2>(grid, stream, p, q);
  } else {
    // Odd batches and nine to sixteen destinations are summed here from 131,073 records on, where reading the
    // results again is what the plane sum would spend its time on (table kernel and final stage, us, before and
    // after: 300,001 x 6 16.9 -> 13.4, 1,000,001 x 6 26.5 -> 20.6, 1,000,000 x 12 46.7 -> 34.9).  Smaller ones keep
    // the plane sum's 256 sums per destination, the number their callers see in per_plane; a launch is all that
    // would be saved there (70,001 x 6 15.6 -> 13.8).
    *fused = p.block_sums && ((aligned && lp.D <= 8) || (lp.D <= kTotMaxD && K > (1 << 17)));
    *fused_blocks = grid;
    auto launch_plain = [&](auto is_aligned, auto lanes) {
      constexpr bool A = decltype(is_aligned)::value;
      constexpr int T = decltype(lanes)::value;
      return two ? launch_lut<2, 0, A, 2, T>(grid, stream, p, q) : launch_lut<2, 0, A, 1, T>(grid, stream, p, q);
    };
    auto launch_totals = [&](auto lanes) {
      return aligned ? launch_plain(std::true_type{}, lanes) : launch_plain(std::false_type{}, lanes);
    };
    le = !*fused ? launch_totals(std::integral_constant<int, 0>{})
                 : (lp.D <= 8 ? launch_totals(std::integral_constant<int, 16>{}) : launch_totals(std::integral_constant<int, 8>{}));
  }
  t_path = 4;
  const cudaError_t ce = le != cudaSuccess ? le : cudaGetLastError();
  *st = ce == cudaSuccess ? HB_OK : hb::cuda_fail(ce, "wave_scale_lut_kernel launch");
  return true;
}

// Division-free kernel when every row of the launch is ordinary and only the five standard
// outputs are wanted; returns false (nothing launched) otherwise.
bool try_launch_fast(const Ptrs& p, const LaunchParams& lp, int64_t K, cudaStream_t stream, hb_status* st) {
  if (p.status || p.limits || lp.D > HB_MAX_DEVICES / 2) return false;
  FastParams fp{};
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!fast_row_ok(g_tab.rows[lp.origin_row], g_tab.pre[lp.origin_row])) return false;
    for (int d = 0; d < lp.D; ++d)
      if (!fast_row_ok(g_tab.rows[lp.dest_row[d]], g_tab.pre[lp.dest_row[d]])) return false;
    fp.D = lp.D;
    fp.K = K;
    fp.origin = fold_fast(g_tab.rows[lp.origin_row], g_tab.pre[lp.origin_row]);
    for (int d = 0; d < lp.D; ++d) {
      FastDev& f = fp.dest[d];
      f = fold_fast(g_tab.rows[lp.dest_row[d]], g_tab.pre[lp.dest_row[d]]);
      f.a_hi = static_cast<float>(lp.a[d]);
      f.a_lo = static_cast<float>(lp.a[d] - static_cast<double>(f.a_hi));
      f.b_hi = static_cast<float>(lp.b[d]);
      f.b_lo = static_cast<float>(lp.b[d] - static_cast<double>(f.b_hi));
      f.log2_clk = lp.log2_clk[d];
    }
  }
  const bool vec4 = vec4_ok(p, K, true);
  const int threads = 256, vec = vec4 ? 4 : 1;
  const int64_t blocks = ((K + vec - 1) / vec + threads - 1) / threads;
  if (blocks > 0x7FFFFFFF) {
    hb::set_error("hb_wave_scale: K too large for one launch");
    *st = HB_ERR_TOO_LARGE;
    return true;
  }
  const dim3 grid(static_cast<unsigned>(blocks));
  if (vec4) {
    if (p.dest_regs) wave_scale_fast_kernel<4, true><<<grid, threads, 0, stream>>>(p, fp);
    else wave_scale_fast_kernel<4, false><<<grid, threads, 0, stream>>>(p, fp);
  } else {
    if (p.dest_regs) wave_scale_fast_kernel<1, true><<<grid, threads, 0, stream>>>(p, fp);
    else wave_scale_fast_kernel<1, false><<<grid, threads, 0, stream>>>(p, fp);
  }
  t_path = 2;
  const cudaError_t e = cudaGetLastError();
  *st = e == cudaSuccess ? HB_OK : hb::cuda_fail(e, "wave_scale_fast_kernel launch");
  return true;
}

template <bool METRICS>
hb_status launch_kernel(const Ptrs& p, const LaunchPlan& plan, int64_t K, cudaStream_t stream, bool* fused,
                        unsigned* fused_blocks) {
  int sm_count = 0;
  const hb_status sync_st = sync_gpu(&sm_count);
  if (sync_st != HB_OK) return sync_st;
  const bool extra = p.status != nullptr || p.limits != nullptr;
  hb_status fast_st = HB_OK;
  *fused = false;
  if (try_launch_lut(p, plan, K, K, sm_count, stream, &fast_st, fused, fused_blocks)) return fast_st;
  if (!METRICS && try_launch_fast(p, plan.lp, K, stream, &fast_st)) return fast_st;
  LaunchParams lp = plan.lp;
  lp.K = K;
  const bool vec4 = vec4_ok(p, K, !METRICS);
  const int threads = 256;
  const int vec = vec4 ? 4 : 1;
  const int64_t nthreads = (K + vec - 1) / vec;
  const int64_t blocks = (nthreads + threads - 1) / threads;
  if (blocks > 0x7FFFFFFF) {
    hb::set_error("hb_wave_scale: K too large for one launch");
    return HB_ERR_TOO_LARGE;
  }
  const dim3 grid(static_cast<unsigned>(blocks));
  if (vec4) {
    if (extra) wave_scale_kernel<4, METRICS, true><<<grid, threads, 0, stream>>>(p, lp);
    else wave_scale_kernel<4, METRICS, false><<<grid, threads, 0, stream>>>(p, lp);
  } else {
    if (extra) wave_scale_kernel<1, METRICS, true><<<grid, threads, 0, stream>>>(p, lp);
    else wave_scale_kernel<1, METRICS, false><<<grid, threads, 0, stream>>>(p, lp);
  }
  t_path = 1;
  HB_CUDA_TRY(cudaGetLastError());
  return HB_OK;
}

// The wave-scaling kernel the launch qualifies for; with p.block_sums also the first stage of the
// per-destination totals: inside the table kernel when it can (per_plane = blocks of its grid),
// else by the plane-sum kernel over the results just written (per_plane = kPlaneBlocks).
template <bool METRICS>
hb_status launch(const Ptrs& p, const LaunchPlan& plan, int64_t K, cudaStream_t stream, int32_t* per_plane = nullptr) {
  bool fused = false;
  unsigned fused_blocks = 0;
  const hb_status st = launch_kernel<METRICS>(p, plan, K, stream, &fused, &fused_blocks);
  if (st != HB_OK || !p.block_sums) return st;
  if (fused) {
    *per_plane = static_cast<int32_t>(fused_blocks);
    return HB_OK;
  }
  HB_CUDA_TRY(hb::launch_overlapped(plane_partial_kernel, dim3(plan.lp.D, kPlaneBlocks), dim3(kSumThreads), 0, stream,
                                    static_cast<const float*>(p.scaled_ns), K,
                                    p.block_sums));
  *per_plane = kPlaneBlocks;
  return HB_OK;
}

hb_status fill_params(LaunchParams* lp, int64_t K, int32_t origin_row, const int32_t* dest_rows,
                      int32_t D) {   // call with g_mu held
  if (g_tab.n == 0) {
    hb::set_error("hb_wave_scale: no device table (call hb_set_devices first)");
    return HB_ERR_INVALID_ARGUMENT;
  }
  if (K < 0 || D < 1 || D > HB_MAX_DEVICES || !dest_rows || origin_row < 0 ||
      origin_row >= g_tab.n) {
    hb::set_error("hb_wave_scale: bad K/D/origin_row");
    return HB_ERR_INVALID_ARGUMENT;
  }
  std::memset(lp, 0, sizeof(*lp));
  lp->D = D;
  lp->origin_row = origin_row;
  const hb_device_spec& o = g_tab.rows[origin_row];
  lp->origin_peak = static_cast<double>(o.peak_gflops_per_second);
  for (int d = 0; d < D; ++d) {
    const int r = dest_rows[d];
    if (r < 0 || r >= g_tab.n) {
      hb::set_error("hb_wave_scale: destination row %d out of range", r);
      return HB_ERR_INVALID_ARGUMENT;
    }
    const hb_device_spec& t = g_tab.rows[r];
    lp->dest_row[d] = static_cast<uint8_t>(r);
    // wave_scaling/roofline.py:48-57: ratios of the integer device fields
    const double l_bw = std::log2(static_cast<double>(o.mem_bandwidth_gb) / t.mem_bandwidth_gb);
    const double l_clk = std::log2(static_cast<double>(o.base_clock_mhz) / t.base_clock_mhz);
    const double l_sm = std::log2(static_cast<double>(o.num_sms) / t.num_sms);
    lp->b[d] = l_clk + l_sm;
    lp->a[d] = l_bw - lp->b[d];
    lp->log2_clk[d] = l_clk;
    lp->ridge[d] = static_cast<double>(t.peak_gflops_per_second) / t.mem_bandwidth_gb;
  }
  return HB_OK;
}

// The plan of (origin, destinations), from this thread's last four or made now.
hb_status plan_for(const LaunchPlan** out, int64_t K, int32_t origin_row, const int32_t* dest_rows, int32_t D) {
  constexpr int kPlans = 4;
  thread_local LaunchPlan plans[kPlans];
  thread_local int oldest = 0;
  const uint64_t version = g_version.load(std::memory_order_acquire);
  if (K >= 0 && D >= 1 && D <= HB_MAX_DEVICES && dest_rows) {
    for (const LaunchPlan& plan : plans) {
      if (plan.version != version || version == 0 || plan.lp.origin_row != origin_row || plan.lp.D != D) continue;
      bool same = true;
      for (int d = 0; d < D && same; ++d) same = dest_rows[d] == plan.lp.dest_row[d];
      if (same) {
        *out = &plan;
        return HB_OK;
      }
    }
  }
  std::lock_guard<std::mutex> lock(g_mu);
  LaunchPlan& plan = plans[oldest];
  plan = LaunchPlan{};
  const hb_status st = fill_params(&plan.lp, K, origin_row, dest_rows, D);
  if (st != HB_OK) return st;
  fill_lut(&plan);
  plan.version = g_version.load(std::memory_order_acquire);   // changes only under the lock
  oldest = (oldest + 1) % kPlans;
  *out = &plan;
  return HB_OK;
}

hb_status check_io(const hb_kernel_soa* k, const hb_wave_out* out, bool need_gamma, int64_t K) {
  if (K == 0 && k && out) return HB_OK;  // nothing to read or write: pointers may be NULL
  if (!k || !out || !k->num_blocks || !k->block_size || !k->regs_per_thread || !k->smem_bytes ||
      !k->run_time_ns || (need_gamma && !k->gamma) || !out->scaled_ns || !out->dest_occupancy ||
      !out->dest_waves || !out->origin_occupancy || !out->origin_waves) {
    hb::set_error("hb_wave_scale: required pointer is NULL");
    return HB_ERR_INVALID_ARGUMENT;
  }
  return HB_OK;
}

Ptrs make_ptrs(const hb_kernel_soa* k, const hb_kernel_metrics* m, const int16_t* dest_regs,
               const hb_wave_out* out) {
  Ptrs p{};
  p.num_blocks = k->num_blocks;
  p.block_size = k->block_size;
  p.regs = k->regs_per_thread;
  p.smem = k->smem_bytes;
  p.time_ns = k->run_time_ns;
  p.gamma = k->gamma;
  if (m) {
    p.flop_eff = m->flop_efficiency_pct;
    p.dram_read = m->dram_read_bytes;
    p.dram_write = m->dram_write_bytes;
    p.has_metrics = m->has_metrics;
  }
  p.dest_regs = dest_regs;
  p.scaled_ns = out->scaled_ns;
  p.dest_occ = out->dest_occupancy;
  p.dest_waves = out->dest_waves;
  p.origin_occ = out->origin_occupancy;
  p.origin_waves = out->origin_waves;
  p.status = out->status;
  p.limits = out->limits;
  return p;
}

}  // namespace

extern "C" int32_t hb_wave_scale_path(void) { return t_path; }

extern "C" hb_status hb_set_devices(const hb_device_spec* rows, int32_t n) {
  if (!rows || n < 1 || n > HB_MAX_DEVICES) {
    hb::set_error("hb_set_devices: need 1..%d rows", HB_MAX_DEVICES);
    return HB_ERR_INVALID_ARGUMENT;
  }
  for (int i = 0; i < n; ++i) {
    if (rows[i].mem_bandwidth_gb <= 0 || rows[i].base_clock_mhz <= 0 || rows[i].num_sms <= 0 ||
        rows[i].peak_gflops_per_second <= 0) {
      hb::set_error("hb_set_devices: row %d has a non-positive bandwidth/clock/SM/peak field", i);
      return HB_ERR_INVALID_ARGUMENT;
    }
  }
  {
    std::lock_guard<std::mutex> lock(g_mu);
    uint32_t magic[kMagicN];
    for (int i = 0; i < kMagicN; ++i) magic[i] = magic_of(static_cast<uint32_t>(i));
    bool changed = n != g_tab.n;
    for (int i = 0; i < n; ++i) {
      // a row is folded and tabulated again only when its specification changed (callers append
      // rows one at a time and pass the whole table); rows already on a GPU are left alone
      if (i < g_tab.n && g_tab.row_version[i] != 0 &&
          std::memcmp(&g_tab.rows[i], &rows[i], sizeof(hb_device_spec)) == 0)
        continue;
      g_tab.rows[i] = rows[i];
      g_tab.pre[i] = hb_fold_device(rows[i]);
      g_tab.lut_ok[i] = lut_row_ok(g_tab.rows[i], g_tab.pre[i]);
      uint8_t* pt = &g_tab.lut_p[static_cast<size_t>(i) * kLutP];
      uint8_t* st = &g_tab.lut_s[static_cast<size_t>(i) * kLutS];
      LutOcc* tt = &g_tab.lut_t[static_cast<size_t>(i) * kLutOcc];
      if (g_tab.lut_ok[i]) {
        g_tab.fast[i] = fold_fast(g_tab.rows[i], g_tab.pre[i]);
        build_row_lut(g_tab.rows[i], g_tab.fast[i], pt, st, tt, magic);
        g_tab.p_class[i] = class_of(g_tab.p_reps, g_tab.words_p, g_tab.lut_p, kLutP, i, same_p_class);
        g_tab.s_class[i] = class_of(g_tab.s_reps, g_tab.words_s, g_tab.lut_s, kLutS, i, same_smem_class);
      } else {
        std::memset(pt, 0, kLutP);
        std::memset(st, 0, kLutS);
        std::memset(tt, 0, sizeof(LutOcc) * kLutOcc);
      }
      ++g_tab.row_version[i];
      changed = true;
    }
    g_tab.n = n;
    if (changed) g_version.fetch_add(1, std::memory_order_acq_rel);
  }
  // the current GPU gets its copy now; the others on their first launch.  A process without a
  // GPU keeps the host table only (hb_thread_block_occupancy needs no more).
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    cudaGetLastError();   // not an error of this call
    return HB_OK;
  }
  return sync_gpu(nullptr);
}

extern "C" hb_status hb_wave_scale(const hb_kernel_soa* kernels, int64_t K, int32_t origin_row,
                                   const int32_t* dest_rows_host, int32_t D,
                                   const int16_t* dest_regs, const hb_wave_out* out,
                                   void* stream) {
  hb_status st = check_io(kernels, out, true, K);
  if (st != HB_OK) return st;
  const LaunchPlan* plan = nullptr;
  st = plan_for(&plan, K, origin_row, dest_rows_host, D);
  if (st != HB_OK) return st;
  if (K == 0) return HB_OK;
  return launch<false>(make_ptrs(kernels, nullptr, dest_regs, out), *plan, K,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int64_t hb_wave_scale_partials_len(int64_t K) {
  if (K < 0) return -1;
  const int64_t blocks = ((K + 1) / 2 + kLutThreads - 1) / kLutThreads;
  return blocks > kPlaneBlocks ? blocks : kPlaneBlocks;
}

extern "C" hb_status hb_wave_scale_partials(const hb_kernel_soa* kernels, int64_t K, int32_t origin_row,
                                            const int32_t* dest_rows_host, int32_t D,
                                            const int16_t* dest_regs, const hb_wave_out* out,
                                            double* partials, int32_t* per_plane, void* stream) {
  hb_status st = check_io(kernels, out, true, K);
  if (st != HB_OK) return st;
  if (!per_plane || (K > 0 && !partials)) {
    hb::set_error("hb_wave_scale_partials: partials / per_plane is NULL");
    return HB_ERR_INVALID_ARGUMENT;
  }
  const LaunchPlan* plan = nullptr;
  st = plan_for(&plan, K, origin_row, dest_rows_host, D);
  if (st != HB_OK) return st;
  *per_plane = 0;
  if (K == 0) return HB_OK;
  Ptrs p = make_ptrs(kernels, nullptr, dest_regs, out);
  p.block_sums = partials;
  return launch<false>(p, *plan, K, static_cast<cudaStream_t>(stream), per_plane);
}

extern "C" hb_status hb_wave_scale_metrics(const hb_kernel_soa* kernels,
                                           const hb_kernel_metrics* metrics, int64_t K,
                                           int32_t origin_row, const int32_t* dest_rows_host,
                                           int32_t D, const int16_t* dest_regs,
                                           const hb_wave_out* out, void* stream) {
  hb_status st = check_io(kernels, out, false, K);
  if (st != HB_OK) return st;
  if (!metrics || (K > 0 && (!metrics->flop_efficiency_pct || !metrics->dram_read_bytes ||
                             !metrics->dram_write_bytes || !metrics->has_metrics))) {
    hb::set_error("hb_wave_scale_metrics: metrics pointer is NULL");
    return HB_ERR_INVALID_ARGUMENT;
  }
  const LaunchPlan* plan = nullptr;
  st = plan_for(&plan, K, origin_row, dest_rows_host, D);
  if (st != HB_OK) return st;
  if (K == 0) return HB_OK;
  return launch<true>(make_ptrs(kernels, metrics, dest_regs, out), *plan, K,
                      static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// Host buffers.  The kernels read staged records from, and write results to, page-locked host memory
// directly: at 65,536 kernels x 6 destinations (1.3 MB in, 3.9 MB out) that is as fast over PCIe as eleven
// copies around the launch (114 against 155 us) and for a few kernels it saves all of their latency.  What
// is left is the host's own copying, 16 GB/s for one core: 82 us to stage those records and 230 us to bring the
// results to ordinary memory.  So
//   * records are staged chunk by chunk, and a chunk's launch runs while the next one is staged;
//   * results in page-locked memory of the caller (batched.wave_scale_host gives such arrays) are written there;
//   * otherwise large batches go through four threads, each with its part of the staging block and a
//     stream: stage, launch, wait, copy out, next chunk.
// ---------------------------------------------------------------------------
namespace {

// The planes of one call, as (element size, whether per destination).
struct HostPlanes {
  static constexpr int kIn = 7, kOut = 7;
  const uint8_t* in[kIn];
  uint8_t* out[kOut];
  size_t in_size[kIn] = {4, 2, 2, 4, 4, 4, 2};     // num_blocks, block, regs, smem, time, gamma | dest_regs [D][K]
  size_t out_size[kOut] = {4, 1, 4, 1, 4, 1, 4};   // scaled, occ, waves [D][K] | origin occ, waves [K] | status [D][K] | limits
  int in_rows[kIn], out_rows[kOut];
  int64_t K;

  HostPlanes(const hb_kernel_soa* k, const int16_t* regs, const hb_wave_out* o, int64_t K_, int D) : K(K_) {
    const void* i[kIn] = {k->num_blocks, k->block_size, k->regs_per_thread, k->smem_bytes, k->run_time_ns, k->gamma, regs};
    void* q[kOut] = {o->scaled_ns, o->dest_occupancy, o->dest_waves, o->origin_occupancy, o->origin_waves, o->status, o->limits};
    for (int j = 0; j < kIn; ++j) {
      in[j] = static_cast<const uint8_t*>(i[j]);
      in_rows[j] = in[j] ? (j < 6 ? 1 : D) : 0;
    }
    for (int j = 0; j < kOut; ++j) {
      out[j] = static_cast<uint8_t*>(q[j]);
      out_rows[j] = !out[j] ? 0 : (j == 3 || j == 4 ? 1 : (j == 6 ? 4 * (D + 1) : D));
    }
  }
  static size_t up(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }
  size_t in_bytes(int64_t n) const {
    size_t b = 0;
    for (int j = 0; j < kIn; ++j) b += up(in_size[j] * in_rows[j] * n);
    return b;
  }
  size_t out_bytes(int64_t n) const {
    size_t b = 0;
    for (int j = 0; j < kOut; ++j) b += up(out_size[j] * out_rows[j] * n);
    return b;
  }
  // Copies records [lo, lo + n) into `slot` and points p at them; dest_regs rows end up n apart.
  uint8_t* stage(uint8_t* slot, int64_t lo, int64_t n, Ptrs* p) const {
    uint8_t* at[kIn];
    for (int j = 0; j < kIn; ++j) {
      at[j] = in_rows[j] ? slot : nullptr;
      const size_t row = in_size[j] * n;
      for (int r = 0; r < in_rows[j]; ++r) std::memcpy(slot + r * row, in[j] + in_size[j] * (r * K + lo), row);
      slot += up(row * in_rows[j]);
    }
    p->num_blocks = reinterpret_cast<const int32_t*>(at[0]);
    p->block_size = reinterpret_cast<const uint16_t*>(at[1]);
    p->regs = reinterpret_cast<const uint16_t*>(at[2]);
    p->smem = reinterpret_cast<const uint32_t*>(at[3]);
    p->time_ns = reinterpret_cast<const float*>(at[4]);
    p->gamma = reinterpret_cast<const float*>(at[5]);
    p->dest_regs = reinterpret_cast<const int16_t*>(at[6]);
    return slot;
  }
  static void set_out(Ptrs* p, uint8_t* const (&at)[kOut]) {
    p->scaled_ns = reinterpret_cast<float*>(at[0]);
    p->dest_occ = at[1];
    p->dest_waves = reinterpret_cast<uint32_t*>(at[2]);
    p->origin_occ = at[3];
    p->origin_waves = reinterpret_cast<uint32_t*>(at[4]);
    p->status = at[5];
    p->limits = reinterpret_cast<int32_t*>(at[6]);
  }
  // The caller's own result planes from record lo on (rows K apart).
  void out_there(int64_t lo, Ptrs* p) const {
    uint8_t* at[kOut];
    for (int j = 0; j < kOut; ++j) at[j] = out[j] ? out[j] + out_size[j] * lo : nullptr;
    set_out(p, at);
  }
  // Result planes of n records in `slot` (rows n apart).
  void out_in_slot(uint8_t* slot, int64_t n, Ptrs* p) const {
    uint8_t* at[kOut];
    for (int j = 0; j < kOut; ++j) {
      at[j] = out_rows[j] ? slot : nullptr;
      slot += up(out_size[j] * out_rows[j] * n);
    }
    set_out(p, at);
  }
  // ... and from there to the caller's planes.
  void fetch(const uint8_t* slot, int64_t lo, int64_t n) const {
    for (int j = 0; j < kOut; ++j) {
      const size_t row = out_size[j] * n;
      for (int r = 0; r < out_rows[j]; ++r) std::memcpy(out[j] + out_size[j] * (r * K + lo), slot + r * row, row);
      slot += up(row * out_rows[j]);
    }
  }
  // Whether the GPU can write every result plane where it is: page-locked at both ends (a caller may have registered
  // the beginning of an array only).
  bool results_page_locked() const {
    for (int j = 0; j < kOut; ++j) {
      if (!out[j]) continue;
      uint8_t* const last = out[j] + out_size[j] * out_rows[j] * K - 1;
      for (uint8_t* p : {out[j], last}) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
          cudaGetLastError();
          return false;
        }
        if (a.type != cudaMemoryTypeHost || a.devicePointer != p) return false;
      }
    }
    return true;
  }
};

constexpr int kHostThreads = 4;
constexpr size_t kHostDirectBytes = 32u << 20;   // of staged records

// Results to ordinary memory.  Each thread takes the next chunk, so it works with as many threads as start (where
// a limit on threads is reached, with this one alone).
hb_status host_in_threads(hb::HostArena* arena, const HostPlanes& io, const LaunchPlan& plan, int64_t K, int64_t chunk,
                          int threads, int device) {
  const size_t slot_bytes = io.in_bytes(chunk) + io.out_bytes(chunk);
  hb_status st = hb::arena_reserve_pinned(arena, slot_bytes * threads);
  if (st != HB_OK) return st;
  hb_status got[kHostThreads] = {};
  char text[kHostThreads][256];
  std::atomic<int64_t> next{0};
  auto work = [&](int w) {
    cudaStream_t s = w == 0 ? arena->stream : arena->more[w - 1];
    uint8_t* slot = arena->pinned + slot_bytes * w;
    hb_status mine = cudaSetDevice(device) == cudaSuccess ? HB_OK : HB_ERR_CUDA;
    for (int64_t lo = next.fetch_add(chunk); lo < K && mine == HB_OK; lo = next.fetch_add(chunk)) {
      const int64_t n = K - lo < chunk ? K - lo : chunk;
      Ptrs p{};
      uint8_t* results = io.stage(slot, lo, n, &p);
      io.out_in_slot(results, n, &p);
      mine = launch<false>(p, plan, n, s);
      const cudaError_t e = cudaStreamSynchronize(s);
      if (mine == HB_OK && e != cudaSuccess) mine = hb::cuda_fail(e, "hb_wave_scale_host");
      if (mine == HB_OK) io.fetch(results, lo, n);
    }
    got[w] = mine;
    if (mine != HB_OK) std::snprintf(text[w], sizeof(text[w]), "%s", hb_last_error());
  };
  std::thread helpers[kHostThreads];
  int started = 1;
  try {
    for (; started < threads; ++started) helpers[started] = std::thread(work, started);
  } catch (const std::exception&) {   // no further thread to be had
  }
  work(0);
  for (int w = 1; w < started; ++w) helpers[w].join();
  for (int w = 0; w < started; ++w) {
    if (got[w] == HB_OK) continue;
    hb::set_error("%s", text[w]);   // the text of another thread
    return got[w];
  }
  return HB_OK;
}

// Results straight into the caller's page-locked planes; two streams, so that a chunk's launch does not wait for
// the last writes of the one before it.  Only the table kernel knows planes that are further apart than its
// records; other launches take the batch as one chunk.
hb_status host_direct(hb::HostArena* arena, const HostPlanes& io, const LaunchPlan& plan, int64_t K, int64_t chunk) {
  hb_status st = hb::arena_reserve_pinned(arena, io.in_bytes(K) + HostPlanes::kIn * 256 * (K / chunk + 1));
  if (st != HB_OK) return st;
  int sm_count = 0;
  st = sync_gpu(&sm_count);
  if (st != HB_OK) return st;
  uint8_t* slot = arena->pinned;
  int used = 0;
  for (int64_t lo = 0, c = 0; lo < K && st == HB_OK; lo += chunk, ++c) {
    const int64_t n = K - lo < chunk ? K - lo : chunk;
    cudaStream_t s = c & 1 ? arena->more[0] : arena->stream;
    Ptrs p{};
    slot = io.stage(slot, lo, n, &p);
    io.out_there(lo, &p);
    {
      bool fused = false;
      unsigned blocks = 0;
      if (!try_launch_lut(p, plan, n, K, sm_count, s, &st, &fused, &blocks, true)) {
        // not for the table kernel (the first chunk says so): everything at once
        slot = io.stage(arena->pinned, 0, K, &p);
        io.out_there(0, &p);
        st = launch<false>(p, plan, K, s);
        lo = K;
      }
    }
    used |= 1 << (c & 1);
  }
  for (int i = 0; i < 2; ++i) {
    if (!(used >> i & 1)) continue;
    const cudaError_t e = cudaStreamSynchronize(i ? arena->more[0] : arena->stream);
    if (st == HB_OK && e != cudaSuccess) st = hb::cuda_fail(e, "hb_wave_scale_host");
  }
  return st;
}

}  // namespace

extern "C" hb_status hb_wave_scale_host(const hb_kernel_soa* kernels, int64_t K,
                                        int32_t origin_row, const int32_t* dest_rows_host,
                                        int32_t D, const int16_t* dest_regs,
                                        const hb_wave_out* out) {
  hb_status st = check_io(kernels, out, true, K);
  if (st != HB_OK) return st;
  const LaunchPlan* plan = nullptr;
  st = plan_for(&plan, K, origin_row, dest_rows_host, D);
  if (st != HB_OK) return st;
  if (K == 0) return HB_OK;
  int device = 0;
  HB_CUDA_TRY(cudaGetDevice(&device));
  // one page-locked staging block per GPU, kept between calls, and the library's own streams
  hb::HostArena* arena = nullptr;
  st = hb::arena_for_current_device(&arena);
  if (st != HB_OK) return st;
  std::lock_guard<std::mutex> lock(arena->mu);
  const HostPlanes io(kernels, dest_regs, out, K, D);
  const LaunchPlan mine = *plan;   // other threads' calls replace theirs, not ours; the helpers have none
  cudaStream_t s;
  // per-destination registers keep rows of their own, block limits are written by the generic kernel alone
  if (!dest_regs && !out->limits && io.in_bytes(K) <= kHostDirectBytes && io.results_page_locked()) {
    // at most eight chunks, of at least 8,192 records: 10 us of staging each
    int64_t chunk = (K / 8 + 255) & ~int64_t{255};
    if (chunk < 8192) chunk = 8192;
    st = hb::arena_stream(arena, 1, &s);
    return st == HB_OK ? host_direct(arena, io, mine, K, chunk) : st;
  }
  // Chunks of 0.5 to 2 MB of records and results, sixteen if the batch is large enough, and no thread for less
  // than two chunks (starting one costs about 40 us).  1,048,576 kernels x 6: 3.3 ms into memory in use, 5.4 ms
  // into fresh pages, against 4.1 and 15.8 ms with pageable copies; 65,536: 0.31 against 0.42 ms.
  const size_t per_record = io.in_bytes(4096) / 4096 + io.out_bytes(4096) / 4096 + 1;
  const int64_t least = static_cast<int64_t>((512u << 10) / per_record), most = 4 * least;
  int64_t chunk = K / 16 < least ? least : (K / 16 > most ? most : K / 16);
  chunk = (chunk + 255) & ~int64_t{255};
  if (chunk > K) chunk = K;
  int64_t threads = (K + 2 * chunk - 1) / (2 * chunk);
  if (threads > kHostThreads) threads = kHostThreads;
  for (int w = 0; w < threads; ++w) {
    st = hb::arena_stream(arena, w, &s);
    if (st != HB_OK) return st;
  }
  return host_in_threads(arena, io, mine, K, chunk, static_cast<int>(threads), device);
}

// The occupancy rules are plain integer code that also compiles for the host
// (occupancy.cuh), so a single record needs no GPU: no allocation, no launch, no
// synchronisation, and the call is legal during a stream capture.
extern "C" hb_status hb_thread_block_occupancy(int32_t device_row, int32_t block_size,
                                               uint32_t smem_bytes, int32_t regs_per_thread,
                                               int32_t* occupancy, int32_t limits[4]) {
  if (!occupancy || block_size < 0 || block_size > 0xFFFF || regs_per_thread < 0 ||
      regs_per_thread > 0xFFFF) {
    hb::set_error("hb_thread_block_occupancy: argument out of range");
    return HB_ERR_INVALID_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(g_mu);
  if (device_row < 0 || device_row >= g_tab.n) {
    hb::set_error("hb_thread_block_occupancy: device row %d is not in the table (hb_set_devices)", device_row);
    return HB_ERR_INVALID_ARGUMENT;
  }
  int32_t lim[4];
  const int32_t smem = smem_bytes > 0x7FFF0000u ? -1 : static_cast<int32_t>(smem_bytes);
  *occupancy = hb_occupancy(g_tab.pre[device_row], block_size, smem, regs_per_thread, lim);
  if (limits) for (int j = 0; j < 4; ++j) limits[j] = lim[j];
  return HB_OK;
}

#if defined(HB_BOUNDS_CHECK)
extern "C" hb_status hb_bounds_check_word(uint32_t* word, int32_t reset) {
  if (!word) return HB_ERR_INVALID_ARGUMENT;
  HB_CUDA_TRY(cudaDeviceSynchronize());
  HB_CUDA_TRY(cudaMemcpyFromSymbol(word, g_bounds_word, sizeof(uint32_t)));
  if (reset) {
    const uint32_t zero = 0;
    HB_CUDA_TRY(cudaMemcpyToSymbol(g_bounds_word, &zero, sizeof(uint32_t)));
  }
  return HB_OK;
}
#else
extern "C" hb_status hb_bounds_check_word(uint32_t* word, int32_t reset) {
  (void)word; (void)reset;
  hb::set_error("hb_bounds_check_word: this build has no index checks (build with -DHB_BOUNDS_CHECK)");
  return HB_ERR_UNSUPPORTED;
}
#endif
