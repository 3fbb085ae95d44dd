// m2d_div.cuh -- FP64 quotients for recurrences: without a branch, and an
// exact check of them afterwards.
#pragma once

namespace m2d {

// Quotients without a branch, from the hardware's reciprocal approximation y0
// of d (about 2^-19 relative error): with e = 1 - d y0, y0 (1 + e) (1 + e^2)
// is 1/d to about one ulp, and n y0 (1 + e) is n/d to 2^-38 (Goldschmidt's
// iteration, AFIPS 1964); one exact-remainder correction of the latter with
// the former (Markstein, as above) leaves a relative error near 2^-89 before
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
// RN(1/d), the same way
__device__ __forceinline__ double rcp_fast(double d, const Rcp &r) { return fma(fma(-d, r.y2, 1.0), r.y2, r.y2); }

// Is q the IEEE quotient n / d?  The remainder r = n - q d is exact, and q
// is the nearest value if and only if |r| <= ulp(q)/2 |d|.  The common case
// first: |n| in [2^-900, 2^900) and q in the normal range and not a power of
// two (below which the spacing halves) unless r = 0, or a zero dividend that
// gave a zero.
static __device__ __noinline__ bool quot_ok_rare(double n, double d, double q)
{
    // Below 2^-900, n and q are scaled up first (exact), so that no bit of r
    // underflows.  A subnormal quotient may be off by one unit, 2^-1074:
    // along walls the fill-in of the factorisation decays through that range,
    // and such a unit reaches nothing above it.  Other values outside the
    // normal range, NaN and Inf answer no, which costs a repeat, not a wrong
    // quotient.
    const bool tiny = fabs(n) < 0x1p-900;
    const bool subnormal = (__double2hiint(q) & 0x7ff00000) == 0;
    const double up = tiny ? 0x1p300 : 1.0;
    const double ns = n * up, qs = q * up;
    const int hq = __double2hiint(qs) & 0x7fffffff, exq = hq & 0x7ff00000;
    const bool pow2 = hq == exq && __double2loint(qs) == 0;
    const double half = __hiloint2double(exq - (pow2 ? 54 << 20 : 53 << 20), 0);
    const double r = fabs(fma(-qs, d, ns));
    if (tiny && subnormal) return fabs(d) >= 0x1p-200 && r <= fabs(d) * 0x1p-774;
    return exq > (54 << 20) && exq < 0x7ff00000 && fabs(ns) >= 0x1p-900 && r <= fabs(d) * half;
}
__device__ __forceinline__ bool quot_ok(double n, double d, double q)
{
    const int hq = __double2hiint(q) & 0x7fffffff, exq = hq & 0x7ff00000, hn = __double2hiint(n) & 0x7fffffff;
    const double r = fabs(fma(-q, d, n));
    const bool near = r <= fabs(d) * __hiloint2double(exq - (53 << 20), 0);
    const bool plain = ((unsigned)(hn - ((1023 - 900) << 20)) < (1800u << 20)) &
                       ((unsigned)(exq - (55 << 20)) < (1900u << 20)) &
                       ((hq != exq) | (__double2loint(q) != 0) | (r == 0.0));
    const bool zero = (n == 0.0) & (q == 0.0) & (fabs(d) > 0.0);
    return ((plain & near) | zero) || quot_ok_rare(n, d, q);
}

}  // namespace m2d
