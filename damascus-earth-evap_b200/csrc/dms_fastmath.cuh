// FP64 division and square root as straight-line code, equal to IEEE `/` and sqrt() bit for bit.
//
// Why: an RK45 attempt holds forty-odd divisions, and the trajectory kernel is bound by instruction
// supply: its step has to fit the SM's 32 KB instruction cache.  `/` has to allow for every operand at every
// place it is used.  Here the quotients of one stage share a divisor, so one correctly rounded reciprocal (10
// operations) serves all of them at 4 operations each, without a branch, and the compiler can interleave
// independent stages.
//
// Method (published, restated here from the mathematics):
//  * reciprocal: Newton's iteration for 1/y - b = 0, y <- y + y (1 - b y), which squares the relative error,
//    written with fused multiply-add and started from the hardware approximation (PTX
//    rcp.approx.ftz.f64, error at most 2^-23 by its documentation): 2^-46 after one step, and after two within
//    one ulp of 1/b.  The third step then returns RN(1/b) unless the significand of b is all
//    ones (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
//    processor", IBM J. Res. Dev. 34, 1990; J.-M. Muller et al., "Handbook of Floating-Point
//    Arithmetic", 2010, sec. 4.7).
//  * quotient: with y = RN(1/b) and its residual l = (1 - b y) y, q0 = RN(a y + RN(a l)) is within one ulp of
//    a / b, and Markstein's theorem then gives q = RN(q0 + (a - b q0) y) = RN(a / b).  No operand,
//    quotient or remainder may leave the normal range: see in_division_range.  A zero dividend gives +0.
//  * square root: Goldschmidt iterations from rsqrt.approx.ftz.f64 and Markstein's correction step
//    s = RN(g + (x - g^2) h), with a certificate instead of a theorem: the rounding error of that
//    last sum, which is exactly representable, must stay below half the spacing of the doubles
//    around s by a relative margin of 2^-40, far above the error of (x - g^2) h.
// Where a condition does not hold, `ok` is cleared and the caller repeats its whole unit of work
// (one RK45 attempt) with IEEE arithmetic.
#pragma once

#include <cstdint>

namespace dms
{
namespace fast
{

__device__ __forceinline__ double rcp_approx(double x)
{
	double y;
	asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
	return y;
}

__device__ __forceinline__ double rsqrt_approx(double x)
{
	double y;
	asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
	return y;
}

// RN(1/b) and its residual, shared by every quotient with divisor b.  `ok` is cleared when the
// significand of b may be all ones (its low word is: one divisor in 2^32).
struct Recip
{
	double b, y, l;
};

__device__ __forceinline__ Recip recip(double b, bool& ok)
{
	Recip r;
	r.b = b;
	double y = rcp_approx(b);
	y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
	y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
	r.y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
	r.l = __dmul_rn(__fma_rn(-b, r.y, 1.0), r.y);
	ok &= __double2loint(b) != -1;
	return r;
}

// Whether (a, b) lie in the range of div: 2^-200 < |b| < 2^400, a = 0 or 2^-700 <= |a| <= 2^400, and a quotient of at
// least 2^-900, so that the remainder a - b q and its products stay normal.  The callers divide by radii and
// speeds in [1, 2^100), by norms in (2^-100, 2^100), by rates in (2^-200, 2^100) and by errors of an RK45
// attempt in [1e-14, 2^400).
__device__ __forceinline__ bool in_division_range(double a, double b)
{
	const double aa = fabs(a), ab = fabs(b);
	return (ab > 0x1p-200) & (ab < 0x1p400) & ((a == 0.0) | ((aa >= 0x1p-700) & (aa <= 0x1p400) & (aa >= 0x1p-900 * ab)));
}

// RN(a / b) for operands in that range.
__device__ __forceinline__ double div(double a, const Recip& d)
{
	const double q = __fma_rn(a, d.y, __dmul_rn(a, d.l));
	return __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
}

// RN(a / b) for a constant divisor with the residual l of its correctly rounded reciprocal.
__device__ __forceinline__ double div_const(double a, double b)
{
	const double y = 1.0 / b;
	const double q = __dmul_rn(a, y);
	const double q1 = __fma_rn(__fma_rn(-b, q, a), y, q);
	return __fma_rn(__fma_rn(-b, q1, a), y, q1);
}

// Whether 1 <= x < 2^100, from the exponent alone.
__device__ __forceinline__ bool in_radius_range(double x)
{
	return static_cast<unsigned int>(__double2hiint(x)) - 0x3ff00000u < 100u << 20;
}

// RN(sqrt(x)) when ok stays set.
__device__ __forceinline__ double sqrt(double x, bool& ok)
{
	const double y = rsqrt_approx(x);
	double g = __dmul_rn(x, y);
	double h = __dmul_rn(0.5, y);
	double e = __fma_rn(-g, h, 0.5);
	g = __fma_rn(g, e, g);
	h = __fma_rn(h, e, h);
	e = __fma_rn(-g, h, 0.5);
	g = __fma_rn(g, e, g);
	h = __fma_rn(h, e, h);
	const double d = __fma_rn(-g, g, x);
	const double s = __fma_rn(d, h, g);
	// the distance of the unrounded sum g + d h from s, against half the spacing above s; at a
	// power of two the spacing below is smaller, so only an exact root passes there
	const double off = __dsub_rn(__dmul_rn(d, h), __dsub_rn(s, g));
	const double power = __hiloint2double(__double2hiint(s) & 0x7ff00000, 0);
	ok &= (x > 0x1p-800) & (x < 0x1p+1000) & ((d == 0.0) | ((fabs(off) < power * (0x1p-53 * (1.0 - 0x1p-40))) & (s != power)));
	return s;
}

// The integer part of 0 <= x < 2^31 as an integer and as a double (the bits of x rounded down to a
// multiple of 1 by an addition; no conversion instruction).  Other x give some integer.
__device__ __forceinline__ unsigned int floor_index(double x, double& whole)
{
	const double t = __dadd_rd(x, 4503599627370496.0);
	whole = __dsub_rn(t, 4503599627370496.0);
	return static_cast<unsigned int>(__double2loint(t));
}

}	// namespace fast
}	// namespace dms
