// Branch-free FP64 arithmetic of the orbit step.
//
// The compiler's division and square root and gmath.h's functions test their
// arguments for zeros, subnormals, infinities and NaN, and the tests end basic
// blocks: the step's four logs, atan2, sincos, nine divisions and four square
// roots then run one after the other (a lone warp took 4.1 cycles per
// instruction, 6800 per step; measured alone a division takes 110 cycles, a
// square root 78, gm_log 275, gm_atan2 610, gm_sincos 280).  The versions here
// contain no branch and no conversion instruction, so that the compiler
// interleaves them: a lone orbit's step 4360 -> 2950 cycles, the pass of 1e5
// halo orbits (one long orbit sets its time) 32.4 -> 22.5 ms, the halo + disk
// pass of 1.2e6 378 -> 300 ms.  They return the same bits for arguments in the ranges
// stated; the orbit step checks its operands (step_safe, step_ones) and takes
// the general functions otherwise (model.cuh:orbit_step).
#ifndef GALIC_STEPMATH_CUH
#define GALIC_STEPMATH_CUH

#include <stdint.h>

#include "gmath.h"

// floor of 0 <= x < 2^31 (any x of [-0, 2^31)): added to 2^52 rounding down,
// the sum's low word is the integer and the sum minus 2^52 its double
struct StepFloor {
  int i;
  double d;
};
__device__ __forceinline__ StepFloor step_floor(double x)
{
  const double big = 4503599627370496.0;  // 2^52
  const double w = __dadd_rd(x, big);
  return {__double2loint(w), w - big};
}

// a / b, correctly rounded: the reciprocal by two Newton steps from the
// hardware's approximation (2^-20 relative or better), the quotient and one
// fused correction with the exact remainder (Markstein, IBM J. Res. Develop.
// 34(1), 1990).  2^-500 <= |b| <= 2^500; a = 0 (for b > 0 the quotient is +0,
// whichever zero a is) or both |a| and |a / b| in [2^-960, 2^960].  Divisors
// whose significand is next to 2 are the method's exception (their reciprocals
// lie next to rounding boundaries, and Newton's steps approach them from
// below): `ones` collects the largest top 20 fraction bits, and the quotient
// may be off by an ulp when step_ones(ones).
__device__ __forceinline__ double step_div(double a, double b, unsigned &ones)
{
  ones = max(ones, __double2hiint(b) & 0xfffffu);
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  const double q = a * y;
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
__device__ __forceinline__ bool step_ones(unsigned ones) { return ones == 0xfffffu; }

// sqrt(a), correctly rounded: Goldschmidt's coupled iteration for sqrt(a) and
// 1 / (2 sqrt(a)) and one correction with the exact remainder (Markstein, as
// above; Cornea, Harrison & Tang, Scientific Computing on Itanium-based
// Systems, 2002).  2^-900 <= a <= 2^900.
__device__ __forceinline__ double step_sqrt(double a)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  double g = a * y, h = 0.5 * y;
  double r = __fma_rn(-h, g, 0.5);
  g = __fma_rn(g, r, g);
  h = __fma_rn(h, r, h);
  r = __fma_rn(-h, g, 0.5);
  g = __fma_rn(g, r, g);
  h = __fma_rn(h, r, h);
  return __fma_rn(__fma_rn(-g, g, a), h, g);
}

// gm_log(x) for 1 <= x < 2^1000: the same table entry (j = round(128 (m - 1))
// from the significand's top eight bits), polynomial and sums
__device__ __forceinline__ double step_log(double x)
{
  const double ln2_hi = 0x1.62e42fee00000p-1, ln2_lo = 0x1.a39ef35793c76p-33;
  const int hi = __double2hiint(x);
  const int j = (((hi >> 12) & 0xff) + 1) >> 1;
  const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
  const double dk = __hiloint2double(0x43300000, (hi >> 20) - 1023) - 4503599627370496.0;
  const double r = __fma_rn(m, gm_log_inv_dev[j], -1.0);
  double p = -0x1.0000000000000p-3;
  p = __fma_rn(r, p, 0x1.2492492492492p-3);
  p = __fma_rn(r, p, -0x1.5555555555555p-3);
  p = __fma_rn(r, p, 0x1.999999999999ap-3);
  p = __fma_rn(r, p, -0x1.0000000000000p-2);
  p = __fma_rn(r, p, 0x1.5555555555555p-2);
  p = __fma_rn(r, p, -0.5);
  const double head = __fma_rn(dk, ln2_hi, gm_log_th_dev[j]);  // exact, as the product is
  return head + (r + ((r * r) * p + (dk * ln2_lo + gm_log_tl_dev[j])));
}

// gm_sincos(gm_atan2(y, x)) for 2^-100 <= |x|, |y| <= 2^100 (ones: see step_div)
__device__ __forceinline__ void step_direction(double y, double x, double *s, double *c, unsigned &ones)
{
  const double pio2_hi = 0x1.921fb54442d18p+0, pio2_lo = 0x1.1a62633145c07p-54;
  const double pi_hi = 0x1.921fb54442d18p+1, pi_lo = 0x1.1a62633145c07p-53;
  const double ax = gm_fabs(x), ay = gm_fabs(y);
  // gm_atan2
  const bool swap = ay > ax;
  const double t = step_div(swap ? ax : ay, swap ? ay : ax, ones);
  const StepFloor k = step_floor(t * 8.0 + 0.5);  // 0..8
  const double ck = k.d * 0.125;
  const double u = step_div(t - ck, 1.0 + t * ck, ones);
  const double zu = u * u;
  double p = -0x1.1111111111111p-4;
  p = __fma_rn(zu, p, 0x1.3b13b13b13b14p-4);
  p = __fma_rn(zu, p, -0x1.745d1745d1746p-4);
  p = __fma_rn(zu, p, 0x1.c71c71c71c71cp-4);
  p = __fma_rn(zu, p, -0x1.2492492492492p-3);
  p = __fma_rn(zu, p, 0x1.999999999999ap-3);
  p = __fma_rn(zu, p, -0x1.5555555555555p-2);
  double a = gm_atan_hi_dev[k.i] + (gm_atan_lo_dev[k.i] + (u + u * (zu * p)));
  a = swap ? (pio2_hi - a) + pio2_lo : a;
  a = x < 0 ? (pi_hi - a) + pi_lo : a;
  // gm_sincos of phi = copysign(a, y), 0 <= a <= pi: n = round(a 2/pi) in
  // 0..2, the signs put in afterwards (the reduction and the polynomials are
  // odd or even in phi exactly); the products with n are exact, so the fused
  // reduction rounds as gm_reduce_pio2's separate one
  const StepFloor n = step_floor(a * 0x1.45f306dc9c883p-1 + 0.5);
  const double r = __fma_rn(-n.d, 0x1.3198a2e037073p-69,
                            __fma_rn(-n.d, 0x1.0b4611a600000p-34, __fma_rn(-n.d, 0x1.921fb54400000p+0, a)));
  const double ps = gm_sin_poly(r), pc = gm_cos_poly(r);
  const double sv = (n.i & 1) ? pc : ps, cv = (n.i & 1) ? ps : pc;
  const bool tiny = a < 0x1.0p-27;
  const double sr = tiny ? a : ((n.i & 2) ? -sv : sv);
  *s = gm_copysign(1.0, y) * sr;
  *c = tiny ? 1.0 : (((n.i + 1) & 2) ? -cv : cv);
}

// __frcp_rn(x) with flushed subnormals (-ftz=true) without its branch: one
// Newton step from the hardware's approximation is the correctly rounded
// reciprocal of every normal x (tests/test_step_math.py compares all 2^32
// arguments); 0 and infinity, whose residual is NaN, keep the approximation.
__device__ __forceinline__ float step_rcp32(float x)
{
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  const float r = __fmaf_rn(-x, y, 1.f);
  return r == r ? __fmaf_rn(r, y, y) : y;
}

// true when every |c[i]| is in [2^-100, 2^100)
__device__ __forceinline__ bool step_safe(const double *c)
{
  const unsigned a = __double2hiint(c[0]) & 0x7fffffff, b = __double2hiint(c[1]) & 0x7fffffff,
                 d = __double2hiint(c[2]) & 0x7fffffff;
  return min(min(a, b), d) >= (1023u - 100u) << 20 && max(max(a, b), d) < (1023u + 100u) << 20;
}
// true when 2^-400 <= v < 2^400
__device__ __forceinline__ bool step_safe_wide(double v)
{
  return (unsigned) __double2hiint(v) - ((1023u - 400u) << 20) < (800u << 20);
}

#endif
