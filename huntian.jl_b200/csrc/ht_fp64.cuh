// FP64 arithmetic of the ellipsoid collapse (ht_collapse.cu): straight-line quotients, roots
// and Carlson's RD.  For use without contraction of products and sums (-fmad=false).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace {

// a / b, correctly rounded, from y = 1 / b correctly rounded: q = a y is within one unit in
// the last place, the remainder a - b q is exact in one fused operation, and q plus the
// remainder times y rounds to the quotient (P. Markstein, IBM J. Res. Dev. 34 (1990) 111).
// For quotients well inside the exponent range; quot_any divides outside it.
__device__ __forceinline__ double quot(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// 1 / b and sqrt(x), correctly rounded, for arguments in the range kind() admits.  They are
// straight-line, so that the six roots and two reciprocals of an RD round overlap (default RK4
// table: 220 ms with the operators / and sqrt(), 138 with these).  Reciprocal: Newton's
// iteration and a last correction with the exact remainder (Markstein, as above; where b's
// significand is all ones, one value in 2^52, it comes out one unit low, and quot is one unit
// low if besides a is a power of two).  Root: Goldschmidt's iteration for g = sqrt(x),
// h = 1 / (2 sqrt(x)), then g plus the exact remainder x - g g times h (P. Markstein,
// "Software division and square root using Goldschmidt's algorithms", RNC 6, 2004).
__device__ __forceinline__ bool kind(double x) { return x > 1e-60 && x < 1e60; }
__device__ __forceinline__ double recip(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));   // about 20 bits
    y = fma(y, fma(-b, y, 1.0), y);
    y = fma(y, fma(-b, y, 1.0), y);
    return fma(y, fma(-b, y, 1.0), y);
}
__device__ __forceinline__ double root(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));   // about 20 bits
    double g = x * y, h = 0.5 * y;
    double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    return fma(fma(-g, g, x), h, g);
}
// Either of the two forms, chosen where a call has looked at its arguments.
template <bool kKind>
__device__ __forceinline__ double root_t(double x) { return kKind ? root(x) : sqrt(x); }
template <bool kKind>
__device__ __forceinline__ double div_t(double a, double b) {
    return kKind ? quot(a, b, recip(b)) : a / b;
}

__device__ __forceinline__ double ratio(double a, double b) {
    return kind(a) && kind(b) ? quot(a, b, recip(b)) : a / b;
}
__device__ __forceinline__ double quot_any(double a, double b, double y) {
    const double m = fabs(a);
    return b > 1e-30 && b < 1e30 && m < 1e250 && m > 1e-250 ? quot(a, b, y) : a / b;
}

constexpr int kRdMaxIt = 200;   // Carlson RD: rounds before the loop gives up (see below)

// Carlson's RD (EllipsoidalCollapse.jl:62-106), two argument sets side by side: each set
// runs its own duplication rounds until its own stopping test holds (a finished set stops
// changing) and then the final formula, so both results are those of two separate calls,
// while the two square-root chains overlap: a round computes both sets without a branch and
// keeps the unfinished ones.  Finite positive arguments converge in a few dozen rounds; a
// set stops after kRdMaxIt rounds at the latest (the reference loops for ever on NaN
// arguments), as the CPU restatement does.
struct RdState {
    double xt, yt, zt, sum, fac, ave;
    bool done;
};

__device__ __forceinline__ void rd_init(RdState& r, double x, double y, double z) {
    r.xt = x; r.yt = y; r.zt = z; r.sum = 0.0; r.fac = 1.0; r.ave = 0.0;
    r.done = false;
}

constexpr double kRdErrTol = 0.05;

// The stopping test: max |ave - v| / ave, each quotient rounded, within kRdErrTol.  Beyond
// 1e-14 of the line a product decides it (rounding moves either side by a few 1e-16); on
// the line, and where a value is not finite, rd_stop takes the quotients.
struct RdTest { bool yes, open; };
__device__ __forceinline__ RdTest rd_test(const RdState& r) {
    const double e = fmax(fmax(fabs(r.ave - r.xt), fabs(r.ave - r.yt)), fabs(r.ave - r.zt));
    const double line = kRdErrTol * fabs(r.ave);
    const bool yes = e < line * (1.0 - 1e-14) && line < 1e300;
    const bool no = e > line * (1.0 + 1e-14) && e < 1e300;
    return RdTest{yes || r.done, !yes && !no && !r.done};
}
__device__ __forceinline__ bool rd_stop(const RdState& r) {
    const double ave = r.ave;
    return fmax(fmax(fabs((ave - r.xt) / ave), fabs((ave - r.yt) / ave)),
                fabs((ave - r.zt) / ave)) <= kRdErrTol;
}

template <bool kKind>
__device__ __forceinline__ void rd_round(RdState& r) {
    const double sqrtx = root_t<kKind>(r.xt), sqrty = root_t<kKind>(r.yt),
                 sqrtz = root_t<kKind>(r.zt);
    const double alamb = sqrtx * (sqrty + sqrtz) + sqrty * sqrtz;
    // (r.fac is a power of two: r.fac times the rounded reciprocal is the rounded quotient)
    const double den = sqrtz * (r.zt + alamb);
    const double sum = r.sum + (kKind ? r.fac * recip(den) : r.fac / den);
    const double xt = 0.25 * (r.xt + alamb), yt = 0.25 * (r.yt + alamb),
                 zt = 0.25 * (r.zt + alamb);
    const double ave = 0.2 * (xt + yt + 3.0 * zt);
    const bool keep = r.done;
    r.sum = keep ? r.sum : sum;
    r.fac = keep ? r.fac : r.fac * 0.25;
    r.xt = keep ? r.xt : xt;
    r.yt = keep ? r.yt : yt;
    r.zt = keep ? r.zt : zt;
    r.ave = keep ? r.ave : ave;
}

template <bool kKind>
__device__ __forceinline__ double rd_final(const RdState& r) {
    const double C1 = 3.0 / 14.0, C2 = 1.0 / 6.0, C3 = 9.0 / 22.0, C4 = 3.0 / 26.0,
                 C5 = 0.25 * C3, C6 = 1.5 * C4;
    const double ave = r.ave, delx = div_t<kKind>(ave - r.xt, ave),
                 dely = div_t<kKind>(ave - r.yt, ave), delz = div_t<kKind>(ave - r.zt, ave);
    const double ea = delx * dely, eb = delz * delz, ec = ea - eb, ed = ea - 6.0 * eb,
                 ee = ed + ec + ec;
    return 3.0 * r.sum +
           div_t<kKind>(r.fac * (1.0 + ed * (-C1 + C5 * ed - C6 * delz * ee) +
                                 delz * (C2 * ee + delz * (-C3 * ec + delz * C4 * ea))),
                        ave * root_t<kKind>(ave));
}

template <bool kKind>
__device__ __forceinline__ void rd_pair(RdState& a, RdState& b, double* r1, double* r2) {
    for (int it = 0; it < kRdMaxIt && !(a.done && b.done); ++it) {
        rd_round<kKind>(a);
        rd_round<kKind>(b);
        const RdTest ta = rd_test(a), tb = rd_test(b);
        a.done = ta.yes;
        b.done = tb.yes;
        if (ta.open || tb.open) {
            if (ta.open) a.done = rd_stop(a);
            if (tb.open) b.done = rd_stop(b);
        }
    }
    *r1 = rd_final<kKind>(a);
    *r2 = rd_final<kKind>(b);
}

__device__ __forceinline__ void elliptic_rd2(double x1, double y1, double z1, double x2,
                                             double y2, double z2, double* r1, double* r2) {
    RdState a, b;
    rd_init(a, x1, y1, z1);
    rd_init(b, x2, y2, z2);
    // a round keeps the arguments between a quarter of the least and the largest of them
    auto fits = [](double x) { return x > 1e-12 && x < 1e12; };
    if (fits(x1) && fits(y1) && fits(z1) && fits(x2) && fits(y2) && fits(z2))
        rd_pair<true>(a, b, r1, r2);
    else
        rd_pair<false>(a, b, r1, r2);
}

}  // namespace
