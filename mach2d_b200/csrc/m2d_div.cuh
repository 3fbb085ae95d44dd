// m2d_div.cuh -- FP64 quotients for recurrences: without a branch, and an
// exact check of them afterwards.
#pragma once

namespace m2d {

// Quotients without a branch, from the hardware's reciprocal approximation y0
// of d (about 2^-19 relative error): with e = 1 - d y0, y0 (1 + e) (1 + e^2)
// is 1/d to about one ulp, and n y0 (1 + e) is n/d to 2^-38 (Goldschmidt's
// iteration, AFIPS 1964); one exact-remainder correction of the latter with
// the former (Markstein, IBM J. Res. Dev. 34, 1990) leaves a relative error near 2^-89 before
// the last rounding, so the result is the IEEE quotient but for about one
// in 2^36 operand pairs, and outside the normal range.  The caller checks
// every result.
struct Rcp { double y0, e, y2; };
__device__ __forceinline__ Rcp rcp_start(double d)
{
    Rcp r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r.y0) : "d"(d));
    r.e = fma(-d, r.y0, 1.0);
    const double y1 = fma(r.y0, r.e, r.y0);
    r.y2 = fma(y1, r.e * r.e, y1);
    return r;
}
__device__ __forceinline__ double div_fast(double n, double d, const Rcp &r)
{
    const double t = n * r.y0;
    const double t1 = fma(t, r.e, t);
    return fma(fma(-t1, d, n), r.y2, t1);
}
// The same quotient by way of a remainder scaled by 2^128, for quotients that
// decay through the subnormals: an unscaled remainder is rounded to whole units
// of 2^-1074 there, and one quotient in ten or so misses the nearest value.
// As many dependent operations; s = 2^128 d is made beside y0, and y2 here is
// 2^-128 / d.
__device__ __forceinline__ Rcp rcp_start_scaled(double d)
{
    Rcp r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r.y0) : "d"(d));
    r.e = fma(-d, r.y0, 1.0);
    const double ys = r.y0 * 0x1p-128, y1 = fma(ys, r.e, ys);
    r.y2 = fma(y1, r.e * r.e, y1);
    return r;
}
__device__ __forceinline__ double div_scaled(double n, double s, const Rcp &r)
{
    const double t = n * r.y0;
    const double t1 = fma(t, r.e, t);
    return fma(fma(-t1, s, n * 0x1p128), r.y2, t1);
}
// the same quotient where the reciprocal is ready before the dividend: one
// dependent operation less
__device__ __forceinline__ double div_ready(double n, double d, const Rcp &r)
{
    const double t = n * r.y2;
    return fma(fma(-t, d, n), r.y2, t);
}
// the same quotient with the sign of a zero right for d > 0, where div_fast's
// sums give -0 + 0 = 0 (four outer iterations of 203x77 cells with the signs
// set in the check alone 6.02 ms, 5.94 so)
__device__ __forceinline__ double div_plus(double n, double d, const Rcp &r)
{
    const double t = n * r.y0;
    const double t1 = t * fma(-d, r.y0, 2.0);
    return fma(fma(t1, d, -n), -r.y2, t1);
}
// whether q has the IEEE quotient's sign
__device__ __forceinline__ bool quot_sign_ok(double n, double d, double q)
{
    return (__double2hiint(n) ^ __double2hiint(d) ^ __double2hiint(q)) >= 0;
}
// RN(1/d), the same way
__device__ __forceinline__ double rcp_fast(double d, const Rcp &r) { return fma(fma(-d, r.y2, 1.0), r.y2, r.y2); }

// Is q the IEEE quotient n / d, in the common case?  The remainder
// r = n - q d is exact for |n| in [2^-900, 2^900), and q is the nearest value
// if |r| <= ulp/2 |d|, ulp the spacing just below |q| (half of that above it
// when q is a power of two).  Below 2^-969 half an ulp is taken as zero, so
// that q must be exact; the same bound makes q = 0 right for n = 0 alone (it
// is what a divisor above 2^1022, whose reciprocal is flushed, gives for every
// n).  An infinite or NaN q makes the difference of the two sides a NaN or
// positive.  q comes from the functions above, which give 0 or a NaN for n = 0
// and a NaN or Inf for an infinite, zero or subnormal d.  The sign of a zero is
// not looked at.  No branch, so it can ride along a recurrence.
__device__ __forceinline__ bool quot_common(double n, double d, double q)
{
    const int hn = __double2hiint(n) & 0x7fffffff, hq = __double2hiint(q) & 0x7fffffff;
    const int below = (hq - (__double2loint(q) == 0 ? 1 : 0)) & ~0xfffff;   // negative for q = 0
    const double half = __hiloint2double(max(below - (53 << 20), 0), 0);
    const bool range = ((unsigned)(hn - ((1023 - 900) << 20)) < (1800u << 20)) | ((hn | __double2loint(n)) == 0);
    return (fma(-fabs(d), half, fabs(fma(-q, d, n))) <= 0.0) & range;
}
// The rest.  Below 2^-900, n and q are scaled up first (exact), so that no
// bit of r underflows.  A subnormal quotient's ulp is 2^-1074; a tie, which
// only there can be one, answers no, and r < ulp/2 |d| holds for the rounded r
// only if it does for the exact one (a divisor above 2^52 need not leave r
// exact).  Other values outside the normal range, NaN and Inf answer no, which
// costs a repeat, not a wrong quotient.
static __device__ __noinline__ bool quot_ok_rare(double n, double d, double q)
{
    const bool tiny = fabs(n) < 0x1p-900;
    const bool subnormal = (__double2hiint(q) & 0x7ff00000) == 0;
    const double up = tiny ? 0x1p300 : 1.0;
    const double ns = n * up, qs = q * up;
    const int hq = __double2hiint(qs) & 0x7fffffff, exq = hq & 0x7ff00000;
    const bool pow2 = hq == exq && __double2loint(qs) == 0;
    const double half = __hiloint2double(exq - (pow2 ? 54 << 20 : 53 << 20), 0);
    const double r = fabs(fma(-qs, d, ns));
    if (tiny && subnormal) return fabs(d) >= 0x1p-200 && r < fabs(d) * 0x1p-775;
    return exq > (54 << 20) && exq < 0x7ff00000 && fabs(ns) >= 0x1p-900 && fma(-fabs(d), half, r) <= 0.0;
}
__device__ __forceinline__ bool quot_ok(double n, double d, double q)
{
    return quot_common(n, d, q) || quot_ok_rare(n, d, q);
}

}  // namespace m2d
