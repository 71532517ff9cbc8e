// fs_kernels.cu -- sm_103a kernels of the FastScape timestep, over a batch
// of realizations (a single model is a batch of one).
//
// A timestep starts with k_receivers_filter + k_receivers_fixup: D8 steepest
// descent over the interior (fastscape_RB.cpp:160-182), an FP32 proof of the
// receiver and the FP64 reference formula for the cells the proof cannot
// settle. Its other kernels, from the receivers on, are the tile walk
// (fs_tile.cu).
//
// k_donors_level0 writes donor masks (pull form of fastscape_RB.cpp:188-203)
// and the level-0 frontier (fastscape_RB.cpp:221-227), for the
// per-realization walk of large batches (k_cta_order_accum, k_cta_erode) and
// for callers that read the masks. Levels and the depth-first order are read
// back by fs_network.cu.
//
// Floating point follows the reference's operation order exactly; the whole
// file is compiled with -fmad=false so no multiply-add is contracted, every
// FP64 division is correctly rounded, and the additions and subtractions
// done in integer arithmetic (fs_bits.h) give the bits of the FP64 ones.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "fastscape_gb300.h"
#include "fs_bits.h"
#include "fs_device.h"
#include "fs_internal.h"

namespace fs {

namespace {

constexpr int kLevelCache = 2048;  // level offsets a realization's walk keeps in shared memory

// ---------------------------------------------------------------------------
// 1. Receivers: fastscape_RB.cpp:160-182. slope = (h[c]-h[n])/dr[n], strict
// '>' against a running maximum that starts at 0, so the first maximum in
// neighbour order wins and a cell with no strictly lower neighbour keeps
// NO_FLOW. k_receivers_exact is that formula verbatim in FP64 (kept to test
// the fast path against); k_receivers_filter + k_receivers_fixup is the fast
// path.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int receiver_fp64(const double *h, int c, int W, double dr_orth,
                                             double dr_diag) {
  const double hc = h[c];
  double max_slope = 0;
  int max_n = FS_NO_FLOW;
#pragma unroll
  for (int n = 0; n < 8; n++) {
    const double slope = (hc - h[c + nbr_off(n, W)]) / ((n & 1) ? dr_diag : dr_orth);
    if (slope > max_slope) {
      max_slope = slope;
      max_n = n;
    }
  }
  return max_n == FS_NO_FLOW ? kPit : max_n;
}

// The same formula for the cells the FP32 filter leaves open -- mostly
// flat ground, where neighbours are equal or differ by less than the
// filter's bound. Only a strictly lower neighbour can have a slope above the
// running maximum (which starts at 0), so the others are skipped by an
// integer comparison of order-preserving keys of the bit patterns: a flat
// cell costs no FP64 operation. (Keys order -0 below +0 where FP64 calls
// them equal; that lets through a slope of +0, which never wins. A NaN
// neighbour is skipped or yields a NaN slope, which never wins either.)
__device__ __forceinline__ uint64_t order_key(uint64_t x) {
  return (x >> 63) ? ~x : (x | 0x8000000000000000ull);
}

__device__ __forceinline__ int receiver_fp64_lower(const double *h, int c, const RealDesc &d) {
  const unsigned long long *hb = reinterpret_cast<const unsigned long long *>(h);
  const uint64_t hcb = hb[c];
  if ((hcb & ~kSignBit) > 0x7FF0000000000000ull) return kPit;  // NaN: every slope NaN
  const uint64_t kc = order_key(hcb);
  uint64_t max_slope = 0;  // bits of +0; slopes compared as non-negative bit patterns
  int max_n = FS_NO_FLOW;
#pragma unroll
  for (int n = 0; n < 8; n++) {
    const uint64_t hnb = hb[c + nbr_off(n, d.W)];
    if (order_key(hnb) >= kc || (hnb & ~kSignBit) > 0x7FF0000000000000ull) continue;
    const uint64_t db = sub_sterbenz(hcb, hnb);  // RN(hc - hn) > 0 (or +0)
    const double dr = (n & 1) ? d.dr_diag : d.dr_orth;
    const double rn = (n & 1) ? d.rdr_diag_n : d.rdr_orth_n;
    uint64_t slope;
    if (__double_as_longlong(rn) != 0) {
      slope = neg_div_rn_bits(db, dr, rn) ^ kSignBit;  // RN(d / dr)
    } else {
      slope = (uint64_t)__double_as_longlong(__longlong_as_double(db) / dr);
    }
    if (slope > max_slope) {
      max_slope = slope;
      max_n = n;
    }
  }
  return max_n == FS_NO_FLOW ? kPit : max_n;
}

__global__ void __launch_bounds__(256) k_receivers_exact(StepArgs a) {
  if (stopped(a.ctl)) return;
  const Tile t = a.rtiles[blockIdx.x];
  const RealDesc &d = a.desc[t.r];
  const double *h = a.h + d.off;
  int8_t *rec = a.rec + d.off;
  const int x = t.x0 + threadIdx.x;
#pragma unroll 1
  for (int y = t.y0 + threadIdx.y; y < t.y0 + a.rrows; y += 8) {
    if (x < d.W - 2 && y < d.H - 2) {
      const int c = y * d.W + x;
      rec[c] = (int8_t)receiver_fp64(h, c, d.W, d.dr_orth, d.dr_diag);
    }
  }
}

// GB300 runs FP64 at ~1.6 lanes/clock/SM against ~113 for FP32, so the eight
// FP64 divides per cell of the reference formula would dominate the
// timestep. The filter decides the receiver from FP32 approximations with a
// rigorous error bound and queues the rare cells it cannot prove for the
// FP64 formula. The result is identical to k_receivers_exact for every input.
//
// Bound: f = h truncated to FP32 (|f-h| <= 2^-23|h| + 2^-126),
// a_n = fl(fl(f_c - f_n) * g_n) with g_n = fl(1/dr_n); then for the exact
// reference slope q_n = RN(RN(h_c-h_n)/dr_n):
//   |a_n - q_n| <= 2^-20 * gmax * (M + 2^-100) =: E/2,
// M >= max |f| over the 3x3 window (the kernel takes the maximum over the
// whole staged tile, which only widens the bound), gmax = max g_n. So
//   best - second > 2E  and best > E  => q_best is the unique maximum > 0;
//   best < -E                         => every q_n < 0 (NO_FLOW);
// otherwise (near-ties, zero slopes, NaN, |h| >= 2^128) the cell is queued.
//
// High ground: the bound grows with the elevations themselves, so a tile
// whose largest |h| reaches 2^(kRelEmin-1023) is staged a second time,
// relative to its first cell: X = fixed_in_binade(h, et) (fs_bits.h; et the
// tile's largest biased exponent, unit u = 2^(et-1084), truncation error
// below u), f = RN32(X - X_ref) * u. Then
// |f - (h - X_ref*u)| <= 2^-24 |h - X_ref*u| + 1.01 u, a common offset that
// cancels in every difference h_c - h_n, so the same bound holds with M the
// largest |f| of the relative values plus 2^22 u for the truncation:
//   E/2 = 2^-20 * gmax * (M + 2^22 u),
// and M is taken per cell over its own 3x3 window (the proof needs no
// more), so a jump inside the tile -- base level beside high ground --
// widens the bound only next to it. Tiles below 2^(kRelEmax-1022) qualify
// (f and u stay normal FP32); others, and tiles below 2^(kRelEmin-1023),
// where truncation is already tight, keep the truncated values and the
// tile's M. tests/native/filter_bound_check.cpp restates these decisions on
// the host and checks them against the FP64 formula.

// trunc_bits_to_float (fs_bits.h): truncation of a double to FP32 with
// integer operations only (no FP64 pipe).
constexpr int kRelEmin = 1030;  // |h| >= 128
constexpr int kRelEmax = 1123;  // |h| < 2^101

// TMA staging of a single grid's tile (TMA variant): one box of FP64 values,
// columns x0-2 .. x0+33 (the box's x must be even: 16-byte aligned) and rows
// y0-1 .. y0+96 (y0+32), into shared memory; the staging then reads the values from
// there (column offset 1) instead of loading them from global memory.
constexpr int kRtW = kRxTile + 4;

__device__ __forceinline__ uint32_t rf_smem(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Loads the box of `rows` rows into dst with the transaction counted on bar
// (thread 0).
__device__ __forceinline__ void rf_tma_tile(int rows, void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int x, int y) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(rf_smem(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(rf_smem(bar)),
               "r"(static_cast<uint32_t>(kRtW * rows * 8))
               : "memory");
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(rf_smem(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(rf_smem(bar)), "r"(x), "r"(y)
      : "memory");
}

// Waits for the box (phase 0 of bar); false after limit_ns.
__device__ __forceinline__ bool rf_wait(uint64_t *bar, unsigned long long limit_ns) {
  const unsigned long long t0 = globaltimer_ns();
  for (int it = 0;; it++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(rf_smem(bar))
        : "memory");
    if (ok) return true;
    if ((it & 15) == 15 && globaltimer_ns() - t0 > limit_ns) return false;
  }
}

template <bool TMA, int ROWS>
__global__ void __launch_bounds__(256)
    k_receivers_filter(const __grid_constant__ CUtensorMap hmap, StepArgs a) {
  if (stopped(a.ctl)) return;
  __shared__ float s[ROWS + 2][kRxTile + 3];
  __shared__ alignas(128) unsigned long long s64[TMA ? ROWS + 2 : 1][TMA ? kRtW : 1];
  __shared__ uint64_t s_bar;
  __shared__ unsigned s_wmax[8];
  const Tile t = a.rtiles[blockIdx.x];
  const RealDesc &d = a.desc[t.r];
  const int W = d.W, H = d.H;
  const double *h = a.h + d.off;
  int8_t *rec = a.rec + d.off;
  const int x0 = t.x0 - 1, y0 = t.y0 - 1;  // grid coordinates of s[0][0]
  // Stage the tile and its halo; M = max |f| and whether any value is NaN
  // (|h| >= 2^128, Inf, NaN) are taken over the whole tile.
  float m = 0.f;
  bool bad = false;
  constexpr int kSw = kRxTile + 2, kSn = (ROWS + 2) * kSw;
  constexpr int kSPer = (kSn + 255) / 256;  // staged values per thread
  // all of a thread's loads in flight before the first is used
  const int t0 = threadIdx.y * 32 + threadIdx.x;
  if (TMA) {
    if (t0 == 0) rf_tma_tile(ROWS + 2, &s64[0][0], &hmap, &s_bar, x0 - 1, y0);
    __syncthreads();  // the barrier is initialised
    if (!rf_wait(&s_bar, a.timeout_ns)) {
      raise_err(a.ctl, FS_ERR_TIMEOUT, kPhaseNone);
      return;
    }
  }
  auto load_value = [&](int tb, int k) -> unsigned long long {  // staged value tb + 256k
    const int i = tb + 256 * k;
    const int ly = i / kSw, lx = i - ly * kSw;
    if (TMA) return i < kSn ? s64[ly][lx + 1] : 0ull;  // zero-filled outside the grid
    const int gx = x0 + lx, gy = y0 + ly;
    if (i < kSn && gx < W && gy < H)
      return __ldg(reinterpret_cast<const unsigned long long *>(h) + (gy * W + gx));
    return 0;  // bits of +0.0
  };
  // Truncated values first, with the tile's largest biased exponent, which
  // decides whether the tile is staged again relative to its first cell.
  __shared__ int s_wexp[8];
  int ew = 0;
  {
    unsigned long long hv[kSPer];
#pragma unroll
    for (int k = 0; k < kSPer; k++) hv[k] = load_value(t0, k);
#pragma unroll
    for (int k = 0; k < kSPer; k++) {
      const int i = t0 + 256 * k;
      if (i < kSn) {
        const int ly = i / kSw, lx = i - ly * kSw;
        const float f = trunc_bits_to_float(hv[k]);
        s[ly][lx] = f;
        m = fmaxf(m, fabsf(f));
        bad |= !(f == f);
        ew = max(ew, (int)(hv[k] >> 52) & 0x7FF);
      }
    }
  }
  const unsigned wm = __reduce_max_sync(kFull, __float_as_uint(m));  // m >= 0: bits order
  ew = __reduce_max_sync(kFull, ew);
  if (threadIdx.x == 0) {
    s_wmax[threadIdx.y] = wm;
    s_wexp[threadIdx.y] = ew;
  }
  const bool tile_bad = __syncthreads_or(bad) != 0;
  float M = 0.f;
  int et = 0;
#pragma unroll
  for (int w = 0; w < 8; w++) {
    M = fmaxf(M, __uint_as_float(s_wmax[w]));
    et = max(et, s_wexp[w]);
  }
  float absterm = 0x1p-100f;
  const bool rel = et >= kRelEmin && et <= kRelEmax;  // block-uniform; no NaN then
  if (rel) {
    // Staged again relative to the tile's first cell (interior: tiles start
    // at x, y >= 2), from a second read of the tile (cached). No thread
    // reads s before the barrier below.
    const long long xr = fixed_in_binade(
        __ldg(reinterpret_cast<const unsigned long long *>(h) + (t.y0 * W + t.x0)), et);
    const float unit = float_from_bits((uint32_t)(et - 1084 + 127) << 23);  // u
    absterm = float_from_bits((uint32_t)(et - 1062 + 127) << 23);           // 2^22 u
    // an opaque copy of t0: the indices are recomputed here instead of
    // being kept in registers across the first pass
    int tb;
    asm volatile("mov.u32 %0, %1;" : "=r"(tb) : "r"(t0));
    // two batches of loads in flight (one loop body: fewer registers)
    constexpr int kHalf = (kSPer + 1) / 2;
#pragma unroll 1
    for (int k0 = 0; k0 < kSPer; k0 += kHalf) {
      unsigned long long hv[kHalf];
#pragma unroll
      for (int k = 0; k < kHalf; k++) hv[k] = k0 + k < kSPer ? load_value(tb, k0 + k) : 0;
#pragma unroll
      for (int k = 0; k < kHalf; k++) {
        const int i = tb + 256 * (k0 + k);
        if (k0 + k < kSPer && i < kSn) {
          const int ly = i / kSw, lx = i - ly * kSw;
          s[ly][lx] = (float)(fixed_in_binade(hv[k], et) - xr) * unit;
        }
      }
    }
    __syncthreads();
  }
  const float g_orth = d.g_orth, g_diag = d.g_diag;
  const float cE = 0x1p-19f * d.gmax;
  const int lx = threadIdx.x + 1;
  const int gx = x0 + lx;
  unsigned qbits = 0;  // bit r: the cell of row lyb + r is queued
  // Each thread takes kRows consecutive rows of its column, sliding a 3x3
  // window down: 3 new shared loads per row. LOCAL (relative tiles): M is
  // the largest |f| of each cell's own window instead of the tile's, so a
  // jump inside the tile (base level next to high ground) widens the bound
  // only where it is.
  constexpr int kRows = ROWS / 8;
  const int lyb = kRows * threadIdx.y + 1;
  auto rows = [&](auto local) {
    constexpr bool LOCAL = decltype(local)::value;
    float u0 = s[lyb - 1][lx - 1], u1 = s[lyb - 1][lx], u2 = s[lyb - 1][lx + 1];
    float m0 = s[lyb][lx - 1], m1 = s[lyb][lx], m2 = s[lyb][lx + 1];
    float E = cE * (M + absterm);
    float cu = 0.f, cm = 0.f;  // LOCAL: largest |f| of the window's upper and middle rows
    if (LOCAL) {
      cu = fmaxf(fabsf(u0), fmaxf(fabsf(u1), fabsf(u2)));
      cm = fmaxf(fabsf(m0), fmaxf(fabsf(m1), fabsf(m2)));
    }
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      const int ly = lyb + r;
      const float d0 = s[ly + 1][lx - 1], d1 = s[ly + 1][lx], d2 = s[ly + 1][lx + 1];
      if (LOCAL) {
        const float cd = fmaxf(fabsf(d0), fmaxf(fabsf(d1), fabsf(d2)));
        E = cE * (fmaxf(cu, fmaxf(cm, cd)) + absterm);
        cu = cm;
        cm = cd;
      }
      const int gy = y0 + ly;
      if (gx < W - 2 && gy < H - 2) {
        const float fc = m1;
        // Largest and second largest approximate slope. Within a direction
        // class (orthogonal W N E S = codes 0 2 4 6, diagonal NW NE SE SW =
        // 1 3 5 7) a_n = fl(fl(fc - f_n) * g) does not increase with f_n
        // (rounding is monotone), so the class's largest and second largest
        // slopes are those of its smallest and second smallest f -- the same
        // values as over all eight slopes. bn is the direction of the
        // largest; it is used only when the largest exceeds every other
        // slope, when its f is the unique minimum of its class (a tie leaves
        // best == second, which queues the cell). Without NaN in the tile no
        // slope is NaN (an overflowing difference is +-Inf, and Inf - Inf
        // below only queues).
        const float lo1 = fminf(m0, m2), hi1 = fmaxf(m0, m2);  // W, E
        const float lo2 = fminf(u1, d1), hi2 = fmaxf(u1, d1);  // N, S
        const float lo3 = fminf(u0, u2), hi3 = fmaxf(u0, u2);  // NW, NE
        const float lo4 = fminf(d2, d0), hi4 = fmaxf(d2, d0);  // SE, SW
        const float omin = fminf(lo1, lo2), osec = fminf(fmaxf(lo1, lo2), fminf(hi1, hi2));
        const float dmin = fminf(lo3, lo4), dsec = fminf(fmaxf(lo3, lo4), fminf(hi3, hi4));
        const int oi = lo2 < lo1 ? (d1 < u1 ? 6 : 2) : (m2 < m0 ? 4 : 0);
        const int di = lo4 < lo3 ? (d0 < d2 ? 7 : 5) : (u2 < u0 ? 3 : 1);
        const float bo = (fc - omin) * g_orth, so = (fc - osec) * g_orth;
        const float bd = (fc - dmin) * g_diag, sd = (fc - dsec) * g_diag;
        const float best = fmaxf(bo, bd);
        const float second = fmaxf(fminf(bo, bd), fmaxf(so, sd));
        const int bn = bo > bd ? oi : di;
        int code = -1;
        if (!tile_bad) {
          if (best - second > 2.f * E && best > E) code = bn;
          else if (best < -E) code = kPit;
        }
        if (code != -1) rec[gy * W + gx] = (int8_t)code;
        else qbits |= 1u << r;
      }
      u0 = m0; u1 = m1; u2 = m2;
      m0 = d0; m1 = d1; m2 = d2;
    }
  };
  if (rel) rows(std::true_type{});
  else rows(std::false_type{});
  // The queued cells of the tile, placed with one atomic per tile (a
  // counter shared by the whole grid would serialise on one address).
  int total;
  const int tt = threadIdx.y * 32 + threadIdx.x;
  const int excl = block_excl_scan(__popc(qbits), total, tt, 256);
  if (total == 0) return;
  __shared__ int s_qbase;
  if (tt == 0) s_qbase = atomicAdd(&a.ctl->amb, total);
  __syncthreads();
  int q = s_qbase + excl;
#pragma unroll 1
  for (int r = 0; r < kRows; r++) {
    if (qbits >> r & 1u) {
      const int gy = y0 + kRows * threadIdx.y + r + 1;
      a.amb[q] = d.off + gy * W + gx;
      a.amb_r[q] = t.r;
      ++q;
    }
  }
}

// receiver_fp64_lower by eight threads, one per neighbour (whole warps).
__device__ __forceinline__ int receiver_fp64_eight(const double *h, int c, const RealDesc &d) {
  const unsigned long long *hb = reinterpret_cast<const unsigned long long *>(h);
  const int n = threadIdx.x & 7;
  const uint64_t hcb = hb[c], hnb = hb[c + nbr_off(n, d.W)];
  const bool nan = (hcb & ~kSignBit) > 0x7FF0000000000000ull ||
                   (hnb & ~kSignBit) > 0x7FF0000000000000ull;
  uint64_t slope = 0;
  if (!nan && order_key(hnb) < order_key(hcb)) {
    const uint64_t db = sub_sterbenz(hcb, hnb);
    const double dr = (n & 1) ? d.dr_diag : d.dr_orth;
    const double rn = (n & 1) ? d.rdr_diag_n : d.rdr_orth_n;
    slope = __double_as_longlong(rn) != 0
                ? neg_div_rn_bits(db, dr, rn) ^ kSignBit
                : (uint64_t)__double_as_longlong(__longlong_as_double(db) / dr);
  }
  int best = n;
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) {  // the steepest, of equals the first
    const uint64_t other = __shfl_xor_sync(kFull, slope, s);
    const int at = __shfl_xor_sync(kFull, best, s);
    if (other > slope || (other == slope && at < best)) {
      slope = other;
      best = at;
    }
  }
  return slope == 0 ? kPit : best;
}

// The queued cells of k_receivers_filter, with the reference formula in FP64.
// A thread per cell divides up to eight times in a row (500 clocks each); a
// queue that leaves seven of eight threads idle gets eight threads per cell
// (1000^2: 82 us a timestep instead of 86), a longer one is bound by the issue
// slots, where the skipped neighbours count.
__global__ void __launch_bounds__(256) k_receivers_fixup(StepArgs a) {
  if (stopped(a.ctl)) return;
  const int n_amb = ld_volatile_i32(&a.ctl->amb);
  if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->queued = n_amb;
  if (n_amb <= (int)(gridDim.x * blockDim.x / 8)) {
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 3);
    if (i - (int)((threadIdx.x & 31) >> 3) >= n_amb) return;  // whole warps
    const int q = i < n_amb ? i : n_amb - 1;
    const RealDesc &d = a.desc[a.amb_r[q]];
    const int c = a.amb[q] - d.off;
    const int code = receiver_fp64_eight(a.h + d.off, c, d);
    if (i < n_amb && (threadIdx.x & 7) == 0) a.rec[d.off + c] = (int8_t)code;
    return;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_amb; i += gridDim.x * blockDim.x) {
    const RealDesc &d = a.desc[a.amb_r[i]];
    const int c = a.amb[i] - d.off;
    a.rec[d.off + c] = (int8_t)receiver_fp64_lower(a.h + d.off, c, d);
  }
}

// ---------------------------------------------------------------------------
// 2. Donor masks + level 0.
// Bit k of mask[c] is set when neighbour c+nshift[k] has receiver code
// (k+4)%8, i.e. drains into c (the pull form of fastscape_RB+GPU.cpp:155-182).
// Level 0 = every cell without a receiver (fastscape_RB.cpp:221-227): the
// two outer rings, which never change and sit at ent[0, nring) of their
// realization from creation on, and the interior pits, appended here with
// one atomic per tile.
//
// Four cells per thread, as bytes of one 32-bit word: a tile's rows are
// staged as aligned words of rec, each thread extracts the words of its
// cells' left, centre and right neighbours with funnel shifts, and a
// byte-wise equality test against the direction code gives the eight mask
// bits of four cells at once.
// ---------------------------------------------------------------------------

// 0x80 in every byte of x equal to the byte t, 0 in the others (no carry
// crosses a byte: (y & 0x7F) + 0x7F <= 0xFE).
__device__ __forceinline__ unsigned bytes_eq(unsigned x, unsigned t) {
  const unsigned y = x ^ (t * 0x01010101u);
  return ~(((y & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | y) & 0x80808080u;
}

constexpr int kDRows = kDyTile / 8;       // consecutive rows per thread
constexpr int kDWords = kDxTile / 4 + 4;  // staged words per row

__global__ void __launch_bounds__(256) k_donors_level0(StepArgs a) {
  if (stopped(a.ctl)) return;
  __shared__ unsigned S[kDyTile + 2][kDWords];
  __shared__ int s_sh[kDyTile + 2];
  __shared__ int s_base;
  const Tile t = a.dtiles[blockIdx.x];
  const RealDesc &d = a.desc[t.r];
  const int W = d.W, H = d.H;
  const int8_t *rec = a.rec + d.off;
  const int tt = threadIdx.y * 32 + threadIdx.x;
  // Staged row ly = grid row y0-1+ly (clamped to the grid: rows past it only
  // feed cells that are not written), as the aligned words from the one
  // holding byte x0-4 on; s_sh = position of byte x0-4 in the first word.
  // The reads stay within kRecPad bytes of the realization.
  // (all of a thread's loads in flight before the first is stored)
  constexpr int kSRows = (kDyTile + 2 + 7) / 8;
  static_assert(kDWords > 32 && kDWords <= 64, "two words per lane and row");
  unsigned wv[kSRows][2];
  int shv[kSRows];
#pragma unroll
  for (int k = 0; k < kSRows; k++) {
    const int ly = threadIdx.y + 8 * k;
    wv[k][0] = wv[k][1] = 0;
    shv[k] = 0;
    if (ly < kDyTile + 2) {
      const int gy = min(t.y0 - 1 + ly, H - 1);
      const uintptr_t first = reinterpret_cast<uintptr_t>(rec + (size_t)gy * W + t.x0) - 4;
      const unsigned *src = reinterpret_cast<const unsigned *>(first & ~(uintptr_t)3);
      wv[k][0] = __ldg(src + threadIdx.x);
      if (threadIdx.x + 32 < kDWords) wv[k][1] = __ldg(src + 32 + threadIdx.x);
      shv[k] = (int)(first & 3);
    }
  }
#pragma unroll
  for (int k = 0; k < kSRows; k++) {
    const int ly = threadIdx.y + 8 * k;
    if (ly < kDyTile + 2) {
      S[ly][threadIdx.x] = wv[k][0];
      if (threadIdx.x + 32 < kDWords) S[ly][32 + threadIdx.x] = wv[k][1];
      if (threadIdx.x == 0) s_sh[ly] = shv[k];
    }
  }
  __syncthreads();
  const int gx0 = t.x0 + 4 * threadIdx.x;   // the thread's first cell
  const int ly0 = 1 + kDRows * threadIdx.y;  // its first staged row
  // left / centre / right neighbour words of the four cells in staged row ly
  auto words = [&](int ly, unsigned &L, unsigned &C, unsigned &R) {
    const int p = 3 + s_sh[ly] + 4 * threadIdx.x;  // byte of the first left neighbour
    const int sh = (p & 3) * 8;
    const unsigned *w = &S[ly][p >> 2];
    const unsigned w0 = w[0], w1 = w[1], w2 = w[2];
    L = __funnelshift_r(w0, w1, sh);
    C = __funnelshift_rc(w0, w1, sh + 8);
    R = sh <= 16 ? __funnelshift_rc(w0, w1, sh + 16) : __funnelshift_r(w1, w2, sh - 16);
  };
  unsigned vx = 0;  // 0xFF in the bytes of cells with 1 <= x <= W-2
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (gx0 + j >= 1 && gx0 + j <= W - 2) vx |= 0xFFu << (8 * j);
  unsigned UL, UC, UR, ML, MC, MR, DL, DC, DR;
  words(ly0 - 1, UL, UC, UR);
  words(ly0, ML, MC, MR);
  uint8_t *mask = a.mask + d.off;
  unsigned pits[kDRows];
  int npit = 0;
#pragma unroll
  for (int i = 0; i < kDRows; i++) {
    const int gy = t.y0 + kDRows * threadIdx.y + i;
    words(ly0 + i + 1, DL, DC, DR);
    const unsigned m = (bytes_eq(ML, 4) >> 7) | (bytes_eq(UL, 5) >> 6) |   // W, NW
                       (bytes_eq(UC, 6) >> 5) | (bytes_eq(UR, 7) >> 4) |   // N, NE
                       (bytes_eq(MR, 0) >> 3) | (bytes_eq(DR, 1) >> 2) |   // E, SE
                       (bytes_eq(DC, 2) >> 1) | bytes_eq(DL, 3);           // S, SW
    const unsigned v = gy <= H - 2 ? vx : 0u;
    pits[i] = bytes_eq(MC, (unsigned)(uint8_t)kPit) & v;
    npit += __popc(pits[i]);
    if (v) {
      uint8_t *row = mask + (size_t)gy * W + gx0;
      if (v == 0xFFFFFFFFu && (reinterpret_cast<uintptr_t>(row) & 3) == 0) {
        *reinterpret_cast<unsigned *>(row) = m;
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if ((v >> (8 * j)) & 1u) row[j] = (uint8_t)(m >> (8 * j));
      }
    }
    UL = ML; UC = MC; UR = MR;
    ML = DL; MC = DC; MR = DR;
  }
  int total;
  const int excl = block_excl_scan(npit, total, tt, 256);
  if (total == 0) return;
  if (tt == 0) s_base = d.off + d.nring + atomicAdd(&a.rctl[t.r].top, total);
  __syncthreads();
  int pos = s_base + excl;
#pragma unroll
  for (int i = 0; i < kDRows; i++) {
    const int gy = t.y0 + kDRows * threadIdx.y + i;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if ((pits[i] >> (8 * j + 7)) & 1u) a.ent[pos++] = gy * W + gx0 + j;
  }
}

// ---------------------------------------------------------------------------
// Per-realization level walk, the timestep of batches of many small
// realizations late in a long run, whose tiles do not fit the GPU at once.
// There the tile walk (fs_tile.cu) finds narrow levels, some 30 cells of a
// tile, and takes most cells in rounds of the whole GPU (256 realizations of
// eroded 512^2: 7.5 ms); one CTA that walks a whole realization's levels, some
// 1000 cells wide, with block barriers only, keeps its threads busy (3.6). Same
// per-cell arithmetic, counts and elevations bit for bit.
//   k_cta_order_accum: level ordering (fastscape_RB.cpp:213-254: level k+1 =
//     the donors of level k, each entry's donors contiguous in direction
//     order) and the accumulation back down the levels (fastscape_RB.cpp:
//     262-279, counts pushed into the receivers' positions); a count beyond
//     the realization's erosion table raises the batch-wide abort, so the
//     next kernel leaves every elevation unchanged and the timestep is redone.
//   k_cta_erode: uplift of the pits, then uplift + erosion level by level
//     (fastscape_RB.cpp:285-328 in the level order of fastscape_RB+P.cpp:
//     319-350).
// The CTAs are as wide as the batch leaves room for: a batch of up to two
// realizations per SM gives each 1024 threads for the ordering (512 for the
// erosion), one of more than four 256 (128), so that the realizations walk
// at once and the latency of one's levels is hidden by the others'.
// ---------------------------------------------------------------------------
template <int T>
__global__ void __launch_bounds__(T, 2048 / T) k_cta_order_accum(StepArgs a) {
  Ctl *ctl = a.ctl;
  if (stopped(ctl)) return;
  const int t = threadIdx.x;
  __shared__ int s_lvl[kLevelCache + 1];
  for (int r = blockIdx.x; r < a.nreal; r += gridDim.x) {
    const RealDesc d = a.desc[r];
    int32_t *ent = a.ent + d.off;
    uint8_t *pdir = a.pdir + d.off;
    uint32_t *acc = a.acc + d.off;
    int32_t *par = a.par + d.off;
    const uint8_t *mask = a.mask + d.off;
    int *lvl = a.lvl_off + d.lvl_base;
    int lo = 0, hi = d.nring + ld_volatile_i32(&a.rctl[r].top);
    if (t == 0) {
      lvl[0] = 0;
      lvl[1] = hi;
      s_lvl[0] = 0;
      s_lvl[1] = hi;
    }
    int nlev = 1;
    bool ovf = false;
    for (;;) {
      int next = hi;
      for (int cs = lo; cs < hi; cs += T) {
        const int i = cs + t;
        int cell = 0;
        unsigned m = 0;
        if (i < hi) {
          cell = __ldcg(&ent[i]);
          m = mask[cell];
          acc[i] = 1u;  // the cell itself; donors add theirs below
        }
        int total;
        const int excl = block_excl_scan(__popc(m), total, t, T);
        if (next + total > d.size) {  // block-uniform
          ovf = true;
          break;
        }
        int pos = next + excl;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          if (m >> k & 1u) {
            ent[pos] = cell + nbr_off(k, d.W);
            pdir[pos] = (uint8_t)((k + 4) & 7);
            par[pos] = i;  // the receiver's position
            ++pos;
          }
        }
        next += total;
      }
      __syncthreads();  // the next level's entries are written
      if (ovf || next == hi) break;
      lo = hi;
      hi = next;
      ++nlev;
      if (t == 0) {
        lvl[nlev] = hi;
        if (nlev <= kLevelCache) s_lvl[nlev] = hi;
      }
    }
    if (t == 0) {
      a.rctl[r].nlevels = nlev;
      if (ovf) raise_err(ctl, FS_ERR_LEVEL_OVERFLOW, kPhaseOrder);
      else if (hi != d.size) raise_err(ctl, FS_ERR_ORDER, kPhaseOrder);  // a cycle
    }
    __syncthreads();
    if (ovf || hi != d.size) continue;
    for (int Lv = nlev - 1; Lv >= 1; --Lv) {
      const int l0 = Lv <= kLevelCache ? s_lvl[Lv] : __ldcg(&lvl[Lv]);
      const int l1 = Lv + 1 <= kLevelCache ? s_lvl[Lv + 1] : __ldcg(&lvl[Lv + 1]);
      // two entries per thread load before their pushes (which go one level
      // down, so they cannot change the counts read here)
      for (int i = l0 + t; i < l1; i += 2 * T) {
        const int i2 = i + T;
        const uint32_t v = __ldcg(&acc[i]);
        const int q = __ldcg(&par[i]);
        const uint32_t v2 = i2 < l1 ? __ldcg(&acc[i2]) : 0u;
        const int q2 = i2 < l1 ? __ldcg(&par[i2]) : 0;
        atomicAdd(&acc[q], v);
        if (i2 < l1) atomicAdd(&acc[q2], v2);
        const uint32_t vm = v > v2 ? v : v2;
        if (a.do_erode && vm >= (uint32_t)d.tab_cap) {
          if (atomicMax(&ctl->abort_k, (int)vm) < (int)vm) ctl->abort_r = d.id;
        }
      }
      __syncthreads();  // this level's counts are final before the next reads them
    }
  }
}

// The erosion walk keeps two entries per thread in flight:
// the entry after next is loaded and the next one's own elevation gathered
// while a cell erodes; only the receiver's elevation waits for the level
// below, and the next level's first entries are loaded before the barrier
// (a cell's own elevation is written only in its own level).
template <int NMODE, int VAR, int T>
__global__ void __launch_bounds__(T, T == 128 ? 7 : 1024 / T) k_cta_erode(StepArgs a) {
  constexpr bool ISUB = VAR == 1, GENERIC = VAR == 2;
  Ctl *ctl = a.ctl;
  if (stopped(ctl)) return;  // an error, or a count beyond a table: nothing changes
  const int t = threadIdx.x;
  struct Entry {
    int c, dir;
    uint32_t k;
    bool ok;
  };
  for (int r = blockIdx.x; r < a.nreal; r += gridDim.x) {
    const RealDesc d = a.desc[r];
    const int nlev = __ldcg(&a.rctl[r].nlevels);
    const int *lvl = a.lvl_off + d.lvl_base;
    unsigned long long *hh = reinterpret_cast<unsigned long long *>(a.h + d.off);
    const int32_t *ent = a.ent + d.off;
    const uint8_t *pdir = a.pdir + d.off;
    const uint32_t *acc = a.acc + d.off;
    const uint64_t udt = (uint64_t)__double_as_longlong(d.u_dt);
    // the pits (level 0 after the rings) are uplifted, not eroded
    const int p1 = __ldcg(&lvl[1]);
    for (int i = d.nring + t; i < p1; i += T) {
      const int c = __ldcg(&ent[i]);
      hh[c] = fadd_bits(__ldcg(&hh[c]), udt);
    }
    auto load_entry = [&](int i, int hi) -> Entry {
      Entry e{0, 0, 0u, false};
      if (i < hi) {
        e.ok = true;
        e.c = __ldcg(&ent[i]);
        e.dir = __ldcg(&pdir[i]);
        e.k = __ldcg(&acc[i]);
      }
      return e;
    };
    auto gather_hc = [&](const Entry &e) -> uint64_t { return e.ok ? __ldcg(&hh[e.c]) : 0ull; };
    auto gather_hn = [&](const Entry &e) -> uint64_t {
      return e.ok ? __ldcg(&hh[e.c + nbr_off(e.dir & 7, d.W)]) : 0ull;
    };
    int lo = p1, hi = nlev > 1 ? __ldcg(&lvl[2]) : p1;
    Entry e1 = load_entry(lo + t, hi), e2 = load_entry(lo + t + T, hi);
    uint64_t hc1 = gather_hc(e1);
    __syncthreads();  // the pits are uplifted
    for (int Lv = 1; Lv < nlev; ++Lv) {
      uint64_t hn1 = gather_hn(e1);
      for (int i = lo + t; i < hi; i += T) {
        const Entry e = e1;
        const uint64_t hc = hc1, hn = hn1;
        e1 = e2;
        e2 = load_entry(i + 2 * T, hi);
        hc1 = gather_hc(e1);
        hn1 = gather_hn(e1);
        const uint64_t h0 = uplift_bits(hc, udt);
        const size_t rec_at = (size_t)e.k * kTabStride + 4 * (e.dir & 1);
        uint64_t hnew;
        if (NMODE == kNOne && !GENERIC) {
          const unsigned long long *Tb = reinterpret_cast<const unsigned long long *>(d.tab) + rec_at;
          hnew = erode_cell_n1<ISUB>(d.tol, ctl, Tb, load_tab_n1(Tb), h0, hn);
        } else if (NMODE == kNTwo && !GENERIC) {
          hnew = erode_cell_n2<ISUB>(d.tol, a.neq, ctl,
                                     __ldg(reinterpret_cast<const unsigned long long *>(d.tab) + rec_at),
                                     h0, hn);
        } else {
          hnew = (uint64_t)__double_as_longlong(erode_cell<NMODE>(
              d.tol, a.neq, ctl, d.tab + rec_at, __longlong_as_double(h0), __longlong_as_double(hn)));
        }
        if (((hnew >> 52) & 0x7FF) == 0x7FF)  // Inf or NaN
          raise_err(ctl, FS_ERR_NONFINITE, kPhaseErode);
        hh[e.c] = hnew;
      }
      if (Lv + 1 < nlev) {  // the next level's first entries
        lo = hi;
        hi = __ldcg(&lvl[Lv + 2]);
        e1 = load_entry(lo + t, hi);
        e2 = load_entry(lo + t + T, hi);
        hc1 = gather_hc(e1);
      }
      __syncthreads();  // this level's elevations are final before the next reads them
    }
  }
  if (blockIdx.x == 0 && t == 0) atomicAdd(&ctl->steps_done, 1);
}

__global__ void k_check_finite(const double *__restrict__ h, long long n, Ctl *ctl) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  bool bad = false;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    bad |= !isfinite(h[i]);
  if (__syncthreads_or(bad) && threadIdx.x == 0) raise_err(ctl, FS_ERR_NONFINITE, kPhaseNone);
}

// Philox4x32-10 (Salmon, Moraes, Dror & Shaw, SC'11), counter = cell index,
// key = seed. Two 32-bit outputs give one U[0,1) double with 53 random bits.
__device__ __forceinline__ void philox4x32_10(uint32_t ctr[4], uint32_t key[2]) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
  uint32_t k0 = key[0], k1 = key[1];
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t hi0 = __umulhi(M0, ctr[0]), lo0 = M0 * ctr[0];
    const uint32_t hi1 = __umulhi(M1, ctr[2]), lo1 = M1 * ctr[2];
    const uint32_t n0 = hi1 ^ ctr[1] ^ k0;
    const uint32_t n1 = lo1;
    const uint32_t n2 = hi0 ^ ctr[3] ^ k1;
    const uint32_t n3 = lo0;
    ctr[0] = n0; ctr[1] = n1; ctr[2] = n2; ctr[3] = n3;
    k0 += W0;
    k1 += W1;
  }
}

__global__ void k_philox_field(double *__restrict__ h, int W, int H, uint32_t key0,
                               uint32_t key1) {
  const long long size = (long long)W * H;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < size; c += stride) {
    uint32_t ctr[4] = {(uint32_t)c, (uint32_t)((unsigned long long)c >> 32), 0u, 0u};
    uint32_t key[2] = {key0, key1};
    philox4x32_10(ctr, key);
    const unsigned long long bits =
        ((unsigned long long)(ctr[0] >> 5) << 26) | (unsigned long long)(ctr[1] >> 6);
    double v = (double)bits * (1.0 / 9007199254740992.0);
    const int y = (int)(c / W);
    const int x = (int)(c - (long long)y * W);
    if (x <= 1 || y <= 1 || x >= W - 2 || y >= H - 2) v = 0.0;
    h[c] = v;
  }
}

// ent[0, nring) = the cells of rings 0 and 1 in ascending order: rows 0 and
// 1, then x = 0, 1, W-2, W-1 of rows 2..H-3, then rows H-2 and H-1.
__global__ void k_place_rings(int32_t *ent, int W, int H) {
  const int mid_rows = H > 4 ? H - 4 : 0;
  const int top = 2 * W;
  const int nring = W * H - (W > 4 ? W - 4 : 0) * mid_rows;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nring; i += gridDim.x * blockDim.x) {
    int c;
    if (H <= 4 || W <= 4) {
      c = i;  // no interior: every cell is a ring cell
    } else if (i < top) {
      c = i;
    } else if (i < top + 4 * mid_rows) {
      const int jj = i - top, row = 2 + jj / 4, q = jj % 4;
      const int x = q < 2 ? q : W - 4 + q;
      c = row * W + x;
    } else {
      c = (H - 2) * W + (i - top - 4 * mid_rows);
    }
    ent[i] = c;
  }
}

// rec of a grid without receivers: -1 on the rings, kPit inside; and its counts.
__global__ void k_no_receivers(int8_t *rec, uint32_t *count, int W, int H) {
  const int size = W * H;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < size; i += gridDim.x * blockDim.x) {
    const int y = i / W, x = i - y * W;
    rec[i] = (int8_t)(x >= 2 && y >= 2 && x < W - 2 && y < H - 2 ? kPit : FS_NO_FLOW);
    count[i] = 1;
  }
}

// A wait on a count that no block ever completes; the bounded wait must give
// up after timeout_ns and report FS_ERR_TIMEOUT. Used by the tests of the
// failure path only.
__global__ void k_test_wait(Ctl *ctl, unsigned long long timeout_ns) {
  if (threadIdx.x == 0) {
    const unsigned target = gridDim.x + 1;  // never reached
    atomicAdd(&ctl->bar, 1u);
    const unsigned long long t0 = globaltimer_ns();
    unsigned spins = 0;
    while (ld_acquire_u32(&ctl->bar) < target) {
      if (ld_volatile_i32(&ctl->err) != 0) break;
      if ((++spins & 255u) == 0 && globaltimer_ns() - t0 > timeout_ns) {
        raise_err(ctl, FS_ERR_TIMEOUT, kPhaseTest);
        break;
      }
      __nanosleep(64);
    }
  }
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

double neg_recip_dr(double dr) {
  return dr >= 1.0 && dr <= 0x1p60 ? -(1.0 / dr) : 0.0;
}

Tolerance make_tolerance(double tol) {
  Tolerance r{};
  r.tol = tol;
  std::memcpy(&r.bits, &tol, sizeof(double));
  const double t = tol * (1.0 - 0x1p-20);
  float f = (float)t;
  while ((double)f > t) f = nextafterf(f, 0.f);
  r.lo_f = f;
  auto upper = [](double x) {  // x >= 0: a double whose upper word is below x's is below x
    uint64_t b;
    std::memcpy(&b, &x, sizeof(b));
    return (uint32_t)(b >> 32);
  };
  r.q_hi = upper(tol * (1.0 - 0x1p-8));
  r.y_hi = upper(tol * 0x1p39);
  r.above_hi = upper(tol * (1.0 + 0x1p-7));
  return r;
}

int ring_cells(int W, int H) {
  return W * H - (W > 4 ? W - 4 : 0) * (H > 4 ? H - 4 : 0);
}

int receiver_rows(int n, const int *W, const int *H) {
  long long tiles = 0;
  for (int r = 0; r < n; r++)
    if (W[r] > 4 && H[r] > 4)
      tiles += (long long)((W[r] - 4 + kRxTile - 1) / kRxTile) * ((H[r] - 4 + kRyTile - 1) / kRyTile);
  return tiles < 152 ? kRySmall : kRyTile;
}

int append_tiles(int rows, int r, int W, int H, Tile *out, int cap) {
  const int kind = rows ? 0 : 1;
  // receivers: interior x, y in [2, W-3]; donors: x, y in [1, W-2]
  // (donor tiles start at x = 0 and cover x in [0, W-2]; x = 0 is skipped)
  const int lo = kind == 0 ? 2 : 1;
  const int xlo = kind == 0 ? 2 : 0;
  const int iw = W - 2 * lo, ih = H - 2 * lo;
  if (iw <= 0 || ih <= 0) return 0;
  const int tx = kind == 0 ? kRxTile : kDxTile, ty = kind == 0 ? rows : kDyTile;
  const int xw = W - lo - xlo;  // columns [xlo, W-1-lo]
  const int nx = (xw + tx - 1) / tx, ny = (ih + ty - 1) / ty;
  if ((long long)nx * ny > cap) return -1;
  int n = 0;
  for (int y = 0; y < ny; y++)
    for (int x = 0; x < nx; x++) out[n++] = Tile{r, xlo + x * tx, lo + y * ty, 0};
  return n;
}

void fill_table_range(double keq, double neq, double meq, double dt, double dr_orth,
                      double dr_diag, double cell_area, long long k0, long long k1,
                      double *rec) {
  const double kd = keq * dt;
  const double pl[2] = {std::pow(dr_orth, neq), std::pow(dr_diag, neq)};
  for (long long k = k0; k < k1; k++) {
    const double A = static_cast<double>(k) * cell_area;
    const double pa = std::pow(A, meq);
    double *r = rec + (k - k0) * kTabStride;
    for (int cls = 0; cls < 2; cls++) {
      const double F = kd * pa / pl[cls];
      const double D = 1. + F;
      r[4 * cls + 0] = F;
      r[4 * cls + 1] = D;
      r[4 * cls + 2] = 1. / D;
      r[4 * cls + 3] = -(1. / D);
    }
  }
}

cudaError_t launch_receivers_exact(const StepArgs &a, cudaStream_t s) {
  if (a.nrtiles == 0) return cudaSuccess;
  k_receivers_exact<<<a.nrtiles, dim3(32, 8), 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_receivers_fast(const StepArgs &a, cudaStream_t s, const CUtensorMap *hmap) {
  if (a.nrtiles == 0) return cudaSuccess;
  CUtensorMap map;
  if (hmap) map = *hmap;
  else std::memset(&map, 0, sizeof(map));
  const auto kernel = a.rrows == kRySmall ? (hmap ? &k_receivers_filter<true, kRySmall>
                                                  : &k_receivers_filter<false, kRySmall>)
                                          : (hmap ? &k_receivers_filter<true, kRyTile>
                                                  : &k_receivers_filter<false, kRyTile>);
  kernel<<<a.nrtiles, dim3(32, 8), 0, s>>>(map, a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_receivers_fixup<<<8 * sm_count(), 256, 0, s>>>(a);
  return cudaGetLastError();
}

bool make_receiver_map(CUtensorMap *m, const double *h, int W, int H, int rows) {
  typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                             const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode enc = nullptr;
  if (!enc) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return false;
    enc = reinterpret_cast<Encode>(fn);
  }
  // row stride a multiple of 16 bytes; the tiles' boxes start at even x
  if (W % 2 || W < kRxTile + 4 || H < 5) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(W), static_cast<cuuint64_t>(H)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(W) * 8};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kRtW), static_cast<cuuint32_t>(rows + 2)};
  const cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<double *>(h), dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_donors_level0(const StepArgs &a, cudaStream_t s) {
  if (a.ndtiles == 0) return cudaSuccess;
  k_donors_level0<<<a.ndtiles, dim3(32, 8), 0, s>>>(a);
  return cudaGetLastError();
}

// Threads of a CTA by the realizations an SM has to hold.
int cta_width(int nreal, int sms) {
  const int per = (nreal + sms - 1) / sms;
  return per <= 2 ? 2 : per <= 4 ? 1 : 0;
}

template <int NMODE, int VAR>
const void *cta_erode_ptr(int width) {
  return width == 2   ? reinterpret_cast<const void *>(&k_cta_erode<NMODE, VAR, 512>)
         : width == 1 ? reinterpret_cast<const void *>(&k_cta_erode<NMODE, VAR, 256>)
                      : reinterpret_cast<const void *>(&k_cta_erode<NMODE, VAR, 128>);
}

cudaError_t launch_cta_order(const StepArgs &a, int sms, cudaStream_t s) {
  switch (cta_width(a.nreal, sms)) {
    case 2: k_cta_order_accum<1024><<<a.nreal, 1024, 0, s>>>(a); break;
    case 1: k_cta_order_accum<512><<<a.nreal, 512, 0, s>>>(a); break;
    default: k_cta_order_accum<256><<<a.nreal, 256, 0, s>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_cta_erode(const StepArgs &a, int sms, cudaStream_t s) {
  StepArgs args = a;
  void *params[] = {&args};
  const int w = cta_width(a.nreal, sms), var = a.erode_generic ? 2 : a.erode_isub ? 1 : 0;
  const void *k = a.nmode == kNOne ? (var == 2   ? cta_erode_ptr<kNOne, 2>(w)
                                      : var == 1 ? cta_erode_ptr<kNOne, 1>(w)
                                                 : cta_erode_ptr<kNOne, 0>(w))
                  : a.nmode == kNTwo ? (var == 2   ? cta_erode_ptr<kNTwo, 2>(w)
                                        : var == 1 ? cta_erode_ptr<kNTwo, 1>(w)
                                                   : cta_erode_ptr<kNTwo, 0>(w))
                                     : cta_erode_ptr<kNGeneral, 2>(w);
  return cudaLaunchKernel(k, dim3(a.nreal), dim3(w == 2 ? 512 : w == 1 ? 256 : 128), params, 0, s);
}

cudaError_t launch_check_finite(const double *h, long long n, Ctl *ctl, cudaStream_t s) {
  long long blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  if (blocks < 1) blocks = 1;
  k_check_finite<<<(int)blocks, 256, 0, s>>>(h, n, ctl);
  return cudaGetLastError();
}

cudaError_t launch_philox_field(double *h, int W, int H, uint64_t seed, cudaStream_t s) {
  long long blocks = ((long long)W * H + 255) / 256;
  if (blocks > 8192) blocks = 8192;
  if (blocks < 1) blocks = 1;
  k_philox_field<<<(int)blocks, 256, 0, s>>>(h, W, H, (uint32_t)seed, (uint32_t)(seed >> 32));
  return cudaGetLastError();
}

cudaError_t launch_place_rings(int32_t *ent, int W, int H, cudaStream_t s) {
  k_place_rings<<<64, 256, 0, s>>>(ent, W, H);
  return cudaGetLastError();
}

cudaError_t launch_no_receivers(int8_t *rec, uint32_t *count, int W, int H, cudaStream_t s) {
  const long long blocks = ((long long)W * H + 255) / 256;
  k_no_receivers<<<(int)(blocks < 4096 ? blocks : 4096), 256, 0, s>>>(rec, count, W, H);
  return cudaGetLastError();
}

cudaError_t launch_test_wait(Ctl *ctl, int blocks, unsigned long long timeout_ns,
                             cudaStream_t s) {
  k_test_wait<<<blocks, 32, 0, s>>>(ctl, timeout_ns);
  return cudaGetLastError();
}

}  // namespace fs
