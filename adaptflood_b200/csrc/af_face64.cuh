// af_face64.cuh -- the FP64 face law without branches.
//
// The reference's face law (src/kernels.cpp:60-84) takes three divisions, a
// square root and a pow per face, each rounded correctly (pow as af_pow.cuh).
// The library forms of division and square root test their operands and
// branch to a slow path, so the faces of a lane cannot overlap: the FP64
// pipe sat at a third of its rate, waiting for one dependent chain at a time.
// Here every operation is straight-line code on operands known to be in
// range, so the faces of a lane interleave; one test per face collects what
// is out of range (infinities, NaN, magnitudes near the ends of the format)
// and sends the warp to the library forms, which give the same values.
//
// Results are the correctly rounded ones, bit for bit:
//  * Division by a constant d (div_const) with d's reciprocal as rh + rl, rh
//    = RN(1/d): a*rl, then a*rh + a*rl in one fma is within one ulp of a/d,
//    and one remainder step with rh rounds correctly (Markstein's theorem;
//    Brisebarre, Muller and Raina, "Accelerating correctly rounded
//    floating-point division when the divisor is known in advance", 2004).
//  * Division (div_near): a Newton quotient q within half an ulp and 2^-26
//    ulp of a/b, so it is RN(a/b) unless a/b is that close to a midpoint.
//    The remainder r = a - b q is exact (fma) and says how far: |r| is b
//    ulp(q)/2 at a midpoint, so |r| within 2^-19 of that (by its high word)
//    goes to the library division.  One face in some 10^5 does.
//  * Square root (sqrt_near): the same with d = x - g^2, which is g ulp(g) at
//    a midpoint; below a power of two the spacing, and so the bound, halves.
#pragma once

#include <cuda_runtime.h>

#include "af_pow.cuh"

namespace af {

// a / d for a zero or 2^-900 <= |a| <= 2^900, 2^-60 <= d <= 2^60.
__device__ __forceinline__ double div_const(double a, double d, double rh, double rl) {
  const double q = __fma_rn(a, rh, a * rl);
  const double r = __fma_rn(-q, d, a);
  return __fma_rn(r, rh, q);
}

// a / b for a zero or 2^-900 <= |a| <= 2^500, 2^-300 <= b <= 2^300; `bad` is
// set when the result may be an ulp off.
__device__ __forceinline__ double div_near(double a, double b, bool& bad) {
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
  const double y1 = __fma_rn(y0, __fma_rn(-b, y0, 1.0), y0);
  const double q0 = a * y1;
  const double q = __fma_rn(__fma_rn(-b, q0, a), y1, q0);
  const int rh = __double2hiint(__fma_rn(-b, q, a)) & 0x7fffffff;
  // high word of b ulp(q)/2, less one (q = 0: r = 0 and a negative bound, so
  // the test is on both as unsigned numbers)
  const int th = __double2hiint(b) + (__double2hiint(q) & 0x7ff00000) - ((1023 + 53) << 20) - 1;
  bad = bad | ((unsigned)rh >= (unsigned)th);
  return q;
}

// sqrt(x) for 2^-500 <= x <= 2^500, `bad` as above.
__device__ __forceinline__ double sqrt_near(double x, bool& bad) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
  const double g0 = x * y0, h0 = 0.5 * y0;
  const double r0 = __fma_rn(-g0, h0, 0.5);
  const double g1 = __fma_rn(g0, r0, g0), h1 = __fma_rn(h0, r0, h0);
  const double g = __fma_rn(__fma_rn(-g1, g1, x), h1, g1);
  const int dh = __double2hiint(__fma_rn(-g, g, x)) & 0x7fffffff;
  const int gh = __double2hiint(g);
  // high word of g ulp(g) (of half that when g may be a power of two), less one
  bad = bad | (dh >= gh + ((gh - 1) & 0x7ff00000) - ((1023 + 52) << 20) - 1);
  return g;
}

// Whether face_fast may be used for a step's constants: with the flow depth
// between depth_thresh and max_hflow these keep every intermediate of the
// face law inside the ranges above.
__host__ __device__ __forceinline__ bool face_range_ok(double dx, double fn, double depth_thresh,
                                              double max_hflow, double gdt) {
  const double lo = 9.313225746154785e-10, hi = 1073741824.0;  // 2^-30, 2^30
  return dx >= lo && dx <= hi && depth_thresh >= lo && max_hflow <= hi && (fn == 0.0 || fn >= lo) &&
         fn <= 1024.0 && gdt >= lo * 9.765625e-4 && gdt <= hi * 1024.0;
}

// The discharge through one wet face (src/kernels.cpp:60-84 with theta = 1;
// the same operations in the same order): x = |Qvect|^2, base = the old
// discharge's part of the numerator.  `bad` is set when an operand is
// out of range and the value must come from the library forms instead.  Ranges: dh is
// 0 or a multiple of 2^-260 here (depths and beds that make a face wet above
// 2^-30 are), so only its upper bound is tested; below x = 2^-500 the
// friction term is under 2^-60 and the denominator is 1 whatever sqrt(x) is,
// so x is raised to 2^-500 (its high word; the low word may stay).  A dry
// face's value means nothing, nor does its `bad`.
__device__ __forceinline__ double face_fast(double dh, double hflow, double x, double base,
                                            double dx, double rh, double rl, double gdt, double fn,
                                            bool& bad) {
  bad = false;
  const double Sf = div_const(-dh, dx, rh, rl);
  const int xh = __double2hiint(x);
  const double xs = __hiloint2double(max(xh, (1023 - 500) << 20), __double2loint(x));
  const double gh = gdt * hflow;
  const double num = base - gh * Sf;
  const double den = 1.0 + div_near(gh * fn * fn * sqrt_near(xs, bad), pw::pow_depth(hflow), bad);
  // Both below 2^100.  x >= 0 or a NaN, which as an unsigned number is above
  // with either sign.
  const unsigned top = max((unsigned)__double2hiint(dh) & 0x7fffffffu, (unsigned)xh);
  const unsigned low = (unsigned)__double2hiint(num) << 1;    // num is 0 or at least 2^-900
  bad = bad | (top >= (1023u + 100u) << 20) | (low - 1u < ((unsigned)(1023 - 900) << 21) - 1u);
  return div_near(num, den, bad) * dx;
}

}  // namespace af
