// gp_exact.cuh -- correctly rounded FP64 division and square root without
// branches, for the Riemann solvers (sm_100a).
//
// The reference's bits need every quotient and root correctly rounded.  The
// language's operators give that, but each one carries its own range test
// and branch, so a solver with some forty of them is a chain of short basic
// blocks whose latencies do not overlap, and quotients with a common divisor
// repeat the divisor's reciprocal.  Here the range test is only accumulated
// in a flag (`bad`), the arithmetic is straight-line, and the caller redoes
// the few faces whose flag is set with the operators.
//
// Methods (published): Newton's iteration on the reciprocal and the
// correction of a quotient by its exact remainder, P. Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34 (1990); division by a divisor whose correctly rounded reciprocal is
// known in one product and two FMAs, N. Brisebarre, J.-M. Muller, S. K.
// Raina, IEEE Trans. Comput. 53 (2004).  The seeds are PTX's rcp.approx.ftz.f64
// and rsqrt.approx.ftz.f64.
//   * y1 = y0 + y0 (e + e^2), e = 1 - b y0, is 1/b to 2^-58; one more Newton
//     step from there rounds correctly (Markstein), also for the all-ones
//     significand that his theorem leaves out once y1 is rounded upwards:
//     1/b then lies just above a midpoint, and only y1 = the lower neighbour
//     would take the step to it.
//   * q = a y, q + y (a - b q) with y = RN(1/b) is RN(a/b) (no exception while
//     nothing under- or overflows).
//   * s + h (a - s^2), s = RN(a y), h = y/2 with y within 0.55 ulp of a^(-1/2) is
//     RN(sqrt(a)) (Markstein's correction of a root).  That y is one step from the
//     seed y0 with e = 1 - a y0^2: a^(-1/2) = y0 (1 - e)^(-1/2), whose binomial
//     series is 1 + e/2 + 3 e^2/8 + 5 e^3/16 + ...  The seed holds 21 significand
//     bits, so y0^2 is exact and e good to 2^-53 |e|; the rounding of y adds 0.5 ulp
//     and the omitted term 5/16 |e|^3 <= 2^-57.4, or 0.05 ulp, for |e| <= 2^-18.6.
// All three hold for every significand of 4 to 12 bits (tests/test_exact_small.py);
// tests/test_gpu_exact.py measures the seeds (|e| up to 2^-19.9 and 2^-19.0, all upper
// 20 bits) and compares the results with the operators.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gp {

// The language's operators, with the interface of FastArith: the faces that leave
// its range, and what is not in a sweep.
struct PlainArith {
  static constexpr bool FAST = false;
  __device__ __forceinline__ double inv(double b) { return 1.0 / b; }
  __device__ __forceinline__ double quot(double a, double b, double) { return a / b; }
  __device__ __forceinline__ double div(double a, double b) { return a / b; }
  __device__ __forceinline__ double root(double a) { return sqrt(a); }
  __device__ __forceinline__ double root0(double a) { return sqrt(a); }
};

struct FastArith {
  static constexpr bool FAST = true;
  bool bad = false;

  // |b| in [2^-200, 2^200]: no intermediate of inv or quot leaves the normal
  // range when the dividend is 0 or in [2^-700, 2^700]
  static constexpr unsigned kDivLo = (1023u - 200u) << 20, kDivSpan = 400u << 20;
  static constexpr unsigned kNumLo = (1023u - 700u) << 20, kNumSpan = 1400u << 20;
  // root: a in [2^-400, 2^400]
  static constexpr unsigned kRootLo = (1023u - 400u) << 20, kRootSpan = 800u << 20;

  // RN(1/b), b > 0 (a negative b sets the flag)
  __device__ __forceinline__ double inv_pos(double b) {
    bad |= (unsigned)__double2hiint(b) - kDivLo > kDivSpan;
    return inv_in(b);
  }
  // the same without the test, for a divisor the caller's bounds cover
  __device__ __forceinline__ double inv_in(double b) {
    double y0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
    const double e = __fma_rn(-b, y0, 1.0);
    const double y1 = __fma_ru(__fma_rn(e, e, e), y0, y0);
    return __fma_rn(__fma_rn(-b, y1, 1.0), y1, y1);
  }
  // RN(1/b)
  __device__ __forceinline__ double inv(double b) {
    const int hi = __double2hiint(b), s = hi & (int)0x80000000;
    const double y = inv_pos(__hiloint2double(hi & 0x7fffffff, __double2loint(b)));
    return __hiloint2double(__double2hiint(y) | s, __double2loint(y));
  }
  // RN(a/b) with y = inv(b); a zero keeps the sign the operator gives
  __device__ __forceinline__ double quot(double a, double b, double y) {
    // a = 0 passes, a denormal does not: its low word is not 0
    const unsigned lo = (unsigned)__double2loint(a);
    const unsigned k = ((unsigned)__double2hiint(a) & 0x7fffffffu) | (lo < 1u ? lo : 1u);
    bad |= (k - kNumLo > kNumSpan) & (k != 0u);
    const double q = __dmul_rn(a, y);
    const double p = __fma_rn(__fma_rn(-b, q, a), y, q);
    const int s = __double2hiint(q) & (int)0x80000000;
    return __hiloint2double((__double2hiint(p) & 0x7fffffff) | s, __double2loint(p));
  }
  // the same for a > 0 and b > 0 (anything else sets the flag)
  __device__ __forceinline__ double quot_pos(double a, double b, double y) {
    bad |= (unsigned)__double2hiint(a) - kNumLo > kNumSpan;
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
  }
  __device__ __forceinline__ double div(double a, double b) { return quot(a, b, inv(b)); }
  // A dividend used with quot_bpos: 0 or in [2^-700, 2^700]
  __device__ __forceinline__ void check(double a) {
    const unsigned lo = (unsigned)__double2loint(a);
    const unsigned k = ((unsigned)__double2hiint(a) & 0x7fffffffu) | (lo < 1u ? lo : 1u);
    bad |= (k - kNumLo > kNumSpan) & (k != 0u);
  }
  // RN(a/b), b > 0, for a dividend that check() or the caller's bounds cover.
  // The remainder is rounded downwards, which leaves the quotient's rounding
  // as it is (checked exhaustively for 4 to 12 bits) and gives a zero
  // dividend the remainder -0, so that a zero quotient keeps its sign.
  __device__ __forceinline__ double quot_bpos(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rd(-b, q, a), y, q);
  }
  // RN(a/b), both checked, b of either sign
  __device__ __forceinline__ double div_any(double a, double b) {
    check(a);
    const int hi = __double2hiint(b), s = hi & (int)0x80000000;
    const double m = __hiloint2double(hi & 0x7fffffff, __double2loint(b));
    const double t = __hiloint2double(__double2hiint(a) ^ s, __double2loint(a));
    return quot_bpos(t, m, inv_pos(m));
  }
  // RN(sqrt(a)), a > 0
  __device__ __forceinline__ double root(double a) {
    bad |= (unsigned)__double2hiint(a) - kRootLo > kRootSpan;
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(a));
    const double e = __fma_rn(-a, __dmul_rn(y0, y0), 1.0);
    const double y1 = __fma_rn(__dmul_rn(e, __fma_rn(e, 0.375, 0.5)), y0, y0);
    const double g = __dmul_rn(a, y1);
    return __fma_rn(__fma_rn(-g, g, a), __dmul_rn(0.5, y1), g);
  }
  // root of a >= +0
  __device__ __forceinline__ double root0(double a) {
    const bool zero = __double_as_longlong(a) == 0;
    const double r = root(zero ? 1.0 : a);
    return zero ? a : r;
  }
};

static __device__ __noinline__ double quot_call(double a, double b) { return a / b; }

// RN(a/b) for a divisor fixed over a launch, y = RN(1/b) formed once; the
// operator where the dividend is not 0 or in [2^-700, 2^700].  The caller
// vouches for b in [2^-200, 2^200] (y = 0 otherwise: the operator).
__device__ __forceinline__ double fixed_quot(double a, double b, double y) {
  FastArith f;
  f.check(a);
  const double p = f.quot_bpos(a, b, y);
  return (f.bad || y == 0.0) ? quot_call(a, b) : p;
}
__device__ __forceinline__ float fixed_quot(float a, float b, float) { return a / b; }

// 1/b for fixed_quot (host side), 0 when b is outside its range
__host__ __device__ inline double fixed_inv(double b) {
  return (b >= 0x1p-200 && b <= 0x1p200) ? 1.0 / b : 0.0;
}
// 1/(gamma - 1) for the solvers, 0 (the operators) for a gamma out of
// [1 + 2^-40, 2^40]: a pressure whose gamma p passed its test is then a
// dividend that needs none
__host__ __device__ inline double gamma_inv(double gamma) {
  const double b = gamma - 1.0;
  return (b >= 0x1p-40 && gamma <= 0x1p40) ? 1.0 / b : 0.0;
}

}  // namespace gp
