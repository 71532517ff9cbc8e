// fs_device.h -- device helpers shared by the timestep's kernel files
// (fs_kernels.cu, fs_tile.cu): clocks and barriers, FP64 arithmetic on bit
// patterns, and the erosion of one cell. Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fastscape_gb300.h"
#include "fs_bits.h"
#include "fs_internal.h"

namespace fs {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kNewtonMaxIt = 1000;

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Asynchronous 8-byte copy into shared memory; cp_async_wait waits for all of
// the thread's copies.
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

// Barrier number id (1 to 15) of n threads of the block (a multiple of 32),
// beside __syncthreads.
__device__ __forceinline__ void group_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ int ld_volatile_i32(const int *p) {
  return *reinterpret_cast<const volatile int *>(p);
}

__device__ __forceinline__ void raise_err(Ctl *ctl, int code, int phase) {
  if (atomicCAS(&ctl->err, 0, code) == 0) ctl->err_detail = phase;
}

// Barrier of all blocks of a cooperative launch, with a limit: false after an
// error, whoever raised it. epoch counts the caller's barriers.
__device__ __forceinline__ bool grid_barrier(Ctl *ctl, unsigned &epoch,
                                             unsigned long long timeout_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned target = ++epoch * gridDim.x;
    __threadfence();  // the block's writes before its arrival
    atomicAdd(&ctl->bar, 1u);
    int ok = 1;
    unsigned long long t0 = 0;
    for (unsigned n = 1; ld_acquire_u32(&ctl->bar) < target; ++n) {
      if ((n & 15u) == 0) {
        const unsigned long long now = globaltimer_ns();
        if (n == 16) t0 = now;
        if (now - t0 > timeout_ns) raise_err(ctl, FS_ERR_TIMEOUT, kPhaseBarrier);
        if (ld_volatile_i32(&ctl->err) != 0) {
          ok = 0;
          break;
        }
      }
      __nanosleep(32);
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ bool stopped(const Ctl *ctl) {
  return (ld_volatile_i32(&ctl->err) | ld_volatile_i32(&ctl->abort_k)) != 0;
}

// nshift[k] (fastscape_RB.cpp:137) for a run-time k without a local array:
// dx+1 and dy+1 of the 8 directions packed two bits per direction
// (W, NW, N, NE, E, SE, S, SW).
__device__ __forceinline__ int nbr_off(int k, int W) {
  const int dx = ((0x1A90 >> (2 * k)) & 3) - 1;
  const int dy = ((0xA901 >> (2 * k)) & 3) - 1;
  return dy * W + dx;
}

// Exclusive block scan of one int per thread; t is the thread's linear index
// in the block and nthreads the block size (a multiple of 32, at most 1024).
// Returns the prefix and the block total.
__device__ __forceinline__ int block_excl_scan(int v, int &total, int t, int nthreads) {
  __shared__ int s_w[32];
  const int lane = t & 31, wid = t >> 5;
  const int nw = nthreads >> 5;
  int incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int x = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += x;
  }
  if (lane == 31) s_w[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int w = lane < nw ? s_w[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int x = __shfl_up_sync(kFull, w, d);
      if (lane >= d) w += x;
    }
    if (lane < nw) s_w[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  total = s_w[nw - 1];
  const int before = wid ? s_w[wid - 1] : 0;
  __syncthreads();  // s_w may be reused by the caller's next scan
  return before + incl - v;
}

__device__ __forceinline__ long long abs_bits(double x) {
  return __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll;
}

// FP64 add / multiply of bit patterns held in integer registers. Keeping
// elevations as integers between the FP64 instructions avoids the FP64
// moves the compiler otherwise emits for merges, selects and negations of
// doubles (each an instruction on this part's narrow FP64 pipe).
__device__ __forceinline__ uint64_t fadd_bits(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("{\n\t.reg .f64 x, y;\n\tmov.b64 x, %1;\n\tmov.b64 y, %2;\n\t"
      "add.rn.f64 x, x, y;\n\tmov.b64 %0, x;\n\t}"
      : "=l"(r)
      : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ uint64_t fmul_bits(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("{\n\t.reg .f64 x, y;\n\tmov.b64 x, %1;\n\tmov.b64 y, %2;\n\t"
      "mul.rn.f64 x, x, y;\n\tmov.b64 %0, x;\n\t}"
      : "=l"(r)
      : "l"(a), "l"(b));
  return r;
}

constexpr uint64_t kSignBit = 0x8000000000000000ull;

// FP64 addition in a branch taken by few cells: volatile, so that the
// compiler does not execute it speculatively for the others.
__device__ __forceinline__ uint64_t fadd_bits_volatile(uint64_t a, uint64_t b) {
  uint64_t r;
  asm volatile(
      "{\n\t.reg .f64 x, y;\n\tmov.b64 x, %1;\n\tmov.b64 y, %2;\n\t"
      "add.rn.f64 x, x, y;\n\tmov.b64 %0, x;\n\t}"
      : "=l"(r)
      : "l"(a), "l"(b));
  return r;
}

// The erosion's FP64 pipe is its bottleneck while its integer pipes idle, so
// some of its additions run in integer arithmetic (fs_bits.h, each
// bit-identical to the hardware's RN operation on the operands it accepts;
// the rest take the FP64 addition).
//
// The uplift h + U*dt of an eroded cell: a positive elevation at least as
// large as the uplift's binade, as nearly every cell of a landscape a few
// timesteps old has. Off the cell's critical path (it does not wait for the
// receiver's elevation), so always worth it.
__device__ __forceinline__ uint64_t uplift_bits(uint64_t h, uint64_t udt) {
  if (add_pos_operand(udt) && (udt >> 52) <= 1900) {
    const uint64_t r = add_const_rn_bits(h, udt);
    if (r) return r;
  }
  return fadd_bits_volatile(h, udt);
}

// RN(x - y) of a cell's and its receiver's elevation: the exact integer
// difference when y >= x/2 (sub_near_bits), else in FP64.
__device__ __forceinline__ uint64_t sub_near(uint64_t x, uint64_t y) {
  if (add_pos_operand(x) && add_pos_operand(y) && x > y) {
    const uint64_t r = sub_near_bits(x, y);
    if (r) return r;
  }
  return fadd_bits_volatile(x, y ^ kSignBit);
}

// RN(x - y) of an elevation and its erosion: in integer arithmetic when y's
// exponent is at least 2 below x's (sub_far_bits), else in FP64.
__device__ __forceinline__ uint64_t sub_far(uint64_t x, uint64_t y) {
  if (add_pos_operand(x) && add_pos_operand(y)) {
    const uint64_t r = sub_far_bits(x, y);
    if (r) return r;
  }
  return fadd_bits_volatile(x, y ^ kSignBit);
}

// RN(x - y) for any two elevations: the exact integer difference when both
// are positive normal and within a factor 2 of each other (Sterbenz), else
// in FP64.
__device__ __forceinline__ uint64_t sub_sterbenz(uint64_t x, uint64_t y) {
  if (add_pos_operand(x) && add_pos_operand(y) && x != y) {
    const bool gt = x > y;
    const uint64_t r = sub_near_bits(gt ? x : y, gt ? y : x);
    if (r) return gt ? r : (r ^ kSignBit);
  }
  return fadd_bits_volatile(x, y ^ kSignBit);
}

// -RN(num/D) on bit patterns, given Rn = -R, R = RN(1/D), in one FP64
// operation: q0n = RN(num*Rn) = -RN(num*R) (RN is symmetric), then
// quotient_tabled_bits (fs_bits.h). tests/native/tile_arith_check.cpp replays it
// on the host against the IEEE division, near rounding midpoints included. It
// replaces Markstein's correction q1 = RN(q0 + r0*R) with r0 = num - q0*D by a
// fused multiply-add (P. Markstein, IBM J. Res. Dev. 34(1), 1990), which cost
// two more FP64 operations. Anything else takes the IEEE division (550 clocks
// for a warp that holds one such cell), volatile PTX in a branch; the
// numerator and result stay in integer registers.
__device__ __forceinline__ uint64_t neg_div_rn_bits(uint64_t numb, double D, double Rn) {
  const uint64_t Db = (uint64_t)__double_as_longlong(D);
  const uint64_t q =
      quotient_tabled_bits((uint64_t)__double_as_longlong(__longlong_as_double(numb) * Rn), numb, Db);
  if (q) return q;
  uint64_t r;
  asm volatile(
      "{\n\t.reg .f64 x, y;\n\tmov.b64 x, %1;\n\tmov.b64 y, %2;\n\t"
      "div.rn.f64 x, x, y;\n\tmov.b64 %0, x;\n\t}"
      : "=l"(r)
      : "l"(numb), "l"(Db));
  return r ^ kSignBit;
}

// ---------------------------------------------------------------------------
// 3. Erosion of one cell and the division it needs.
// ---------------------------------------------------------------------------

// Correctly rounded num/D for D > 0 given R = RN(1/D), without the FP64
// divide routine: Markstein's correction q1 = q0 + (num - q0*D)*R with
// fused multiply-adds (P. Markstein, IBM J. Res. Dev. 34(1), 1990), then an
// exact check of the remainder r1 = num - q1*D: q1 is accepted only if
// |r1| < D*ulp(q1)/2 (then |num/D - q1| < ulp(q1)/2, so q1 = RN(num/D)),
// q1 is not a power of two (where the spacing below halves) and its
// exponent is far from the subnormal/overflow range. Anything else -- zero
// numerators included -- takes the IEEE division. 4 FP64 operations against
// ~7.5 for the divide routine on this part.
__device__ __forceinline__ double div_rn(double num, double D, double R) {
  const double q0 = num * R;
  const double r0 = fma(-q0, D, num);
  const double q1 = fma(r0, R, q0);
  const double r1 = fma(-q1, D, num);
  const long long qb = abs_bits(q1);
  const int e = (int)(qb >> 52);
  if (e >= 64 && e <= 1980 && (qb & 0x000FFFFFFFFFFFFFll) != 0) {
    const long long thr = __double_as_longlong(D) + ((long long)(e - 1076) << 52);
    if (abs_bits(r1) < thr) return q1;
  }
  return num / D;
}

// pow(x, n) and pow(x, n-1) for the Newton update of fastscape_RB.cpp:322.
template <int NMODE>
__device__ __forceinline__ void powers(double x, double neq, double &pn, double &pn1) {
  if (NMODE == kNOne) {
    pn = x;
    pn1 = 1.0;
  } else if (NMODE == kNTwo) {
    pn = x * x;
    pn1 = x;
  } else {
    pn = pow(x, neq);
    pn1 = pow(x, neq - 1.0);
  }
}

// The fields of a table record the n = 1 erosion reads up front.
struct TabN1 {
  uint64_t fact, D, Rn;
};

__device__ __forceinline__ TabN1 load_tab_n1(const unsigned long long *Tb) {
  const ulonglong2 p = __ldg(reinterpret_cast<const ulonglong2 *>(Tb));
  const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2 *>(Tb) + 1);
  return TabN1{p.x, p.y, q.y};
}

// True when |RN(x - y)| <= tol is proven for x = RN(y - q), y the previous
// iterate and qn = -q: |RN(x - y)| <= (|q| + 2^-51(|y|+|q|))(1+2^-53), and
// an FP32 test on truncated magnitudes (each within 2^-23 relative, flushed
// below 2^-126) with 2^-21 of slack proves it for almost every cell without
// the subtraction.
__device__ __forceinline__ bool step_below_tol(uint64_t qn, uint64_t y, const Tolerance &tl) {
  const float qf = fabsf(trunc_bits_to_float(qn));
  const float yf = fabsf(trunc_bits_to_float(y));
  return qf * (1.f + 0x1p-21f) + yf * 0x1p-48f <= tl.lo_f;
}

// Most steps are settled by the upper words alone, with |y| 2^-48 < tol 2^-9:
// 1: |RN(x - y)| <= tol, as |q| < tol (1 - 2^-8) (the bound above); -1: it is
// above, as |q| > tol (1 + 2^-7) and |RN(x - y)| >= (|q| - 2^-52 (|y| + |q|))
// (1 - 2^-53); 0: not settled.
__device__ __forceinline__ int step_against_tol(uint64_t q, uint64_t y, const Tolerance &tl) {
  const uint32_t qh = (uint32_t)(q >> 32) & 0x7FFFFFFFu;
  if (((uint32_t)(y >> 32) & 0x7FFFFFFFu) >= tl.y_hi) return 0;
  return qh < tl.q_hi ? 1 : qh > tl.above_hi && qh < 0x7FF00000u ? -1 : 0;
}

// RN(x + y), y = -q with |q| far below x > 0 (a Newton correction): in
// integer arithmetic when the operands allow, else in FP64.
__device__ __forceinline__ uint64_t add_correction(uint64_t x, uint64_t y) {
  return (y & kSignBit) ? sub_far(x, y ^ kSignBit) : uplift_bits(x, y);
}

// RN(x / y) of bit patterns on the FP64 pipe.
// IEEE division in a branch taken by few cells (volatile: not executed
// speculatively for the others).
__device__ __forceinline__ uint64_t fdiv_bits_volatile(uint64_t a, uint64_t b) {
  uint64_t r;
  asm volatile(
      "{\n\t.reg .f64 x, y;\n\tmov.b64 x, %1;\n\tmov.b64 y, %2;\n\t"
      "div.rn.f64 x, x, y;\n\tmov.b64 %0, x;\n\t}"
      : "=l"(r)
      : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ uint64_t ffma_bits(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("{\n\t.reg .f64 x, y, z;\n\tmov.b64 x, %1;\n\tmov.b64 y, %2;\n\tmov.b64 z, %3;\n\t"
      "fma.rn.f64 x, x, y, z;\n\tmov.b64 %0, x;\n\t}"
      : "=l"(r)
      : "l"(a), "l"(b), "l"(c));
  return r;
}

// RN(num/den) on bit patterns for a denominator with no tabled reciprocal
// (the n = 2 erosion's), in three FP64 operations: the IEEE FP32 reciprocal
// of |den| truncated to FP32 (within 1.5*2^-23 of 1/|den|), one Newton step
// r1 = r0 + r0*(1 - |den|*r0) by fused multiply-adds (within ~2^-44.8),
// q0 = RN(|num|*r1) (within ~2^8.2 ulp of the quotient), and the rounding
// from the exact integer residual (round_quotient_bits, fs_bits.h). Newton's
// iteration for the reciprocal and the residual check are the published
// methods (e.g. P. Markstein, IBM J. Res. Dev. 34(1), 1990);
// tests/native/division_check.cpp replays the sequence on the host against
// the IEEE division. Operands outside [2^-99, 2^102) and the rare cases the
// rounding leaves open take the IEEE division.
__device__ __forceinline__ uint64_t fdiv_rn_bits(uint64_t nb, uint64_t db) {
  const uint64_t an = nb & ~kSignBit, ad = db & ~kSignBit;
  if ((unsigned)((int)(an >> 52) - 924) <= 200u && (unsigned)((int)(ad >> 52) - 924) <= 200u) {
    // |den| truncated to FP32: its exponent is in range
    const uint32_t hi = (uint32_t)(ad >> 32);
    const uint32_t rb = __float_as_uint(__frcp_rn(__uint_as_float(
        (((hi >> 20) - 896u) << 23) | __funnelshift_l((uint32_t)ad, hi & 0xFFFFFu, 3))));
    // widen the positive normal FP32 reciprocal to FP64 bits
    const uint64_t r0 = ((uint64_t)((rb >> 23) + 896) << 52) | ((uint64_t)(rb & 0x7FFFFFu) << 29);
    const uint64_t e = ffma_bits(ad ^ kSignBit, r0, 0x3FF0000000000000ull);  // 1 - |den| r0
    const uint64_t r1 = ffma_bits(r0, e, r0);
    const uint64_t q = round_quotient_bits(an, ad, fmul_bits(an, r1));
    if (q) return q | ((nb ^ db) & kSignBit);
  }
  return fdiv_bits_volatile(nb, db);
}

// RN(x - y) for any operands: in integer arithmetic when both are positive
// normal (sub_near_bits within a factor 2, sub_far_bits from an exponent gap
// of 2) or x is positive and y negative (add_pos_rn_bits), else in FP64.
__device__ __forceinline__ uint64_t sub_gen(uint64_t x, uint64_t y) {
  if (add_pos_operand(x)) {
    if (add_pos_operand(y)) {
      if (x != y) {
        const bool gt = x > y;
        const uint64_t hi = gt ? x : y, lo = gt ? y : x;
        const uint64_t r = ((int)(hi >> 52) - (int)(lo >> 52) >= 2) ? sub_far_bits(hi, lo)
                                                                     : sub_near_bits(hi, lo);
        if (r) return gt ? r : (r ^ kSignBit);
      }
    } else if (add_pos_operand(y ^ kSignBit)) {
      return add_pos_rn_bits(x, y ^ kSignBit);
    }
  }
  return fadd_bits_volatile(x, y ^ kSignBit);
}

// Erosion of one cell for n = 2 (fastscape_RB.cpp:315-326; pow(x,2) as x*x,
// pow(x,1) = x) on bit patterns, iterate by iterate in the reference's
// operation order: x' = RN(x - RN(num/den)) with
//   num = RN(RN(x - h0) + RN(fact*RN(RN(x-hn)^2))),
//   den = RN(1 + RN(RN(fact*n)*RN(x-hn))),
// RN(fact*n) hoisted (the reference's grouping), the first iterate's
// x - h0 = +0 dropped, and |x' - x| <= tol proven in FP32 for most
// iterates without the subtraction. With ISUB the subtractions run in
// integer arithmetic.
template <bool ISUB>
__device__ __forceinline__ uint64_t erode_cell_n2(const Tolerance &tl, double neq, Ctl *ctl,
                                                  uint64_t factb, uint64_t h0, uint64_t hn) {
  auto sub = [](uint64_t x, uint64_t y) { return ISUB ? sub_gen(x, y) : fadd_bits(x, y ^ kSignBit); };
  constexpr uint64_t kOne = 0x3FF0000000000000ull;
  const uint64_t fact2 = fmul_bits(factb, (uint64_t)__double_as_longlong(neq));
  uint64_t x = h0;
  for (int it = 1;; ++it) {
    const uint64_t dx = sub(x, hn);
    const uint64_t fpn = fmul_bits(factb, fmul_bits(dx, dx));
    uint64_t num;
    if (it == 1) {
      num = (fpn << 1) == 0 ? 0 : fpn;  // RN(+0 + fpn)
    } else {
      const uint64_t a = sub(x, h0);
      num = ISUB ? sub_gen(fpn, a ^ kSignBit) : fadd_bits(a, fpn);
    }
    const uint64_t den = fadd_bits(kOne, fmul_bits(fact2, dx));
    const uint64_t q = fdiv_rn_bits(num, den);
    const uint64_t xn = sub(x, q);
    const int step = step_against_tol(q, x, tl);
    if (step > 0 || (step == 0 && step_below_tol(q ^ kSignBit, x, tl))) return xn;
    if (step < 0) {  // surely not the last
      x = xn;
      if (it < kNewtonMaxIt) continue;
      raise_err(ctl, FS_ERR_NEWTON, kPhaseErode);
      return x;
    }
    const uint64_t df = sub(xn, x);
    x = xn;
    // fabs(diff) > tol as an integer compare (a NaN diff stops the loop)
    const long long m = (long long)(df & ~kSignBit);
    if (!(m > tl.bits && m <= 0x7FF0000000000000ll)) return x;
    if (it >= kNewtonMaxIt) {
      raise_err(ctl, FS_ERR_NEWTON, kPhaseErode);
      return x;
    }
  }
}

// Erosion of one cell for n = 1 (fastscape_RB.cpp:315-326) on bit
// patterns: h0 the uplifted elevation, hn the receiver's final elevation,
// t the table record of the cell's drainage count and direction class
// (fact, D = 1 + fact, -1/D; Tb the record itself for 1/D).
//
// The reference's loop for n = 1 (pow(x,1) = x, pow(x,0) = 1):
//   x' = RN(x - RN(RN(RN(x - h0) + RN(fact*RN(x - hn))) / D)),
//   stop when |RN(x' - x)| <= tol.
// First iterate (x = h0): RN(h0 - h0) = +0, so x1 = RN(h0 - RN(RN(fact*
// RN(h0-hn)) / D)). Cells whose erosion exceeds tol take a second iterate,
// unrolled here too; its residual num2 is often exactly 0 (then x2 = x1).
// Rarer third iterates follow the generic loop. With ISUB the subtractions
// of elevations run in integer arithmetic: that relieves the FP64 pipe but
// lengthens the cell's dependency chain after the receiver's elevation
// arrives, which pays where the pipe, not latency, limits the erosion (the
// autotuner decides per workload).
template <bool ISUB>
__device__ __forceinline__ uint64_t erode_cell_n1(const Tolerance &tl, Ctl *ctl,
                                                  const unsigned long long *Tb, TabN1 t,
                                                  uint64_t h0, uint64_t hn) {
  const uint64_t factb = t.fact;
  const double D = __longlong_as_double(t.D), Rn = __longlong_as_double(t.Rn);
  const uint64_t dh = ISUB ? sub_near(h0, hn) : fadd_bits(h0, hn ^ kSignBit);
  const uint64_t num = fmul_bits(factb, dh);
  const uint64_t qn = neg_div_rn_bits(num, D, Rn);  // -q
  const uint64_t x1 = ISUB ? sub_far(h0, qn ^ kSignBit) : fadd_bits(h0, qn);
  const int step = step_against_tol(qn, h0, tl);
  if (step > 0 || (step == 0 && step_below_tol(qn, h0, tl))) return x1;
  // diff = RN(x1 - h0); |diff| > tol as an integer compare of the
  // magnitudes' bits (a NaN diff stops the loop, as fabs(NaN) > tol is false)
  const uint64_t a = ISUB ? sub_sterbenz(x1, h0) : fadd_bits(x1, h0 ^ kSignBit);
  auto more = [&](uint64_t df) {
    const long long m = (long long)(df & ~kSignBit);
    return m > tl.bits && m <= 0x7FF0000000000000ll;
  };
  if (!more(a)) return x1;
  // second iterate: num2 = RN(a + RN(fact * RN(x1 - hn)))
  const uint64_t b = ISUB ? sub_sterbenz(x1, hn) : fadd_bits(x1, hn ^ kSignBit);
  const uint64_t c = fmul_bits(factb, b);
  const uint64_t num2 = ISUB ? sub_sterbenz(c, a ^ kSignBit) : fadd_bits(a, c);
  if ((num2 << 1) == 0) return x1;  // RN(0/D) = +0 and x1 - 0 = x1: diff = 0
  // The correction is a residual of x1's rounding: x2 is x1 or a neighbour,
  // decided from an FP32 estimate of the quotient (newton_step_in_spacing),
  // and a step of at most one spacing <= tol ends the loop.
  if (add_pos_operand(x1)) {
    const float qe = __fdividef(fabsf(trunc_bits_to_float(num2)), trunc_bits_to_float(t.D));
    int places;
    float ulp;
    if (newton_step_in_spacing(num2, t.D, x1, qe, &places, &ulp) && ulp <= tl.lo_f)
      return x1 + (uint64_t)(int64_t)places;
  }
  const uint64_t q2n = neg_div_rn_bits(num2, D, Rn);
  const uint64_t x2 = ISUB ? add_correction(x1, q2n) : fadd_bits(x1, q2n);
  if (step_below_tol(q2n, x1, tl)) return x2;
  // third and later iterates: the reference's loop in FP64
  const double R = __longlong_as_double(__ldg(Tb + 2));
  const double fact = __longlong_as_double(factb), h0d = __longlong_as_double(h0),
               hnd = __longlong_as_double(hn);
  double x = __longlong_as_double(x2);
  double diff = x - __longlong_as_double(x1), hp = x;
  int it = 2;
  while (more((uint64_t)__double_as_longlong(diff))) {
    const double n3 = (x - h0d) + fact * (x - hnd);
    x -= div_rn(n3, D, R);
    diff = x - hp;
    hp = x;
    if (++it >= kNewtonMaxIt) {
      raise_err(ctl, FS_ERR_NEWTON, kPhaseErode);
      break;
    }
  }
  return (uint64_t)__double_as_longlong(x);
}

// Erosion of one cell for n != 1: fastscape_RB.cpp:315-326 with h0 the
// uplifted elevation, hn the receiver's final elevation and T the table
// record of the cell's drainage count and direction class (T[0] = fact).
template <int NMODE>
__device__ __forceinline__ double erode_cell(const Tolerance &tl, double neq, Ctl *ctl,
                                             const double *T, double h0, double hn) {
  const double fact = T[0];
  double hnew, hp, diff;
  int it;
  hnew = h0;
  hp = h0;
  diff = 2 * tl.tol;
  it = 0;
  while (fabs(diff) > tl.tol) {
    double pn, pn1;
    powers<NMODE>(hnew - hn, neq, pn, pn1);
    hnew -= (hnew - h0 + fact * pn) / (1. + fact * neq * pn1);
    diff = hnew - hp;
    hp = hnew;
    if (++it >= kNewtonMaxIt) {
      raise_err(ctl, FS_ERR_NEWTON, kPhaseErode);
      break;
    }
  }
  return hnew;
}

}  // namespace

}  // namespace fs
