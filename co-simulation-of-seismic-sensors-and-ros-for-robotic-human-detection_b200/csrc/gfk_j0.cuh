// gfk_j0.cuh — Bessel J0 in FP64 for the wavenumber sums.
//
// The sums over wavenumber evaluate J0(k r) once per (wavenumber, range), at
// arguments mostly far above 25. There J0 is written in modulus-phase form,
//     J0(x) = M(x) cos(x - pi/4 + phi(x)),   H0(x) = M e^{i (x - pi/4 + phi)},
// (Watson, "A Treatise on the Theory of Bessel Functions", 13.75): one cosine
// instead of two, and M sqrt(x) and x phi are smooth functions of w = 1/x^2.
// Their polynomials are the degree-5 Chebyshev interpolants on
// [0, 1/625], computed from 60-digit values of J0 and Y0; absolute errors
// 6e-17 / sqrt(x) and 5e-18. The phase is reduced by a multiple of pi/2 in two
// parts (Cody and Waite) with fused multiply-adds, the multiple chosen with
// the offset included, so the remainder stays in [-pi/4, pi/4]; sine and cosine
// are degree-7 Chebyshev interpolants in its square (errors 6e-18), the
// quadrant picking which set of coefficients one Horner chain runs on.
// Below 25, and from 2^30 on, CUDA's j0.
//
// About 35 FP64 instructions against about 130 issue slots measured for CUDA's
// j0 (16.7M values in 0.12 ms): the FP64 pipe bounds every sum that evaluates
// it in the loop. Absolute error against 40-digit values at 6200 points of
// [25, 1e9] (compiled for the host): at most 6e-17, as glibc's j0 there.
#pragma once
#include "gfk_math.cuh"

namespace gfk {

constexpr double kJ0Asymptotic = 25.0;       // from here the modulus-phase form
constexpr double kJ0Largest = 1073741824.0;  // below this the quadrant fits an int

GFK_HD double j0_modulus_phase(double x) {
#ifdef __CUDA_ARCH__
    const double y = rsqrt_(x);
#else
    const double y = 1.0 / sqrt(x);
#endif
    const double u = y * y, w = u * u;  // 1/x, 1/x^2
    double p = fma(460.30608499789054, w, -23.345134131630825);
    p = fma(p, w, 1.6379601386715872);
    p = fma(p, w, -0.20957027324986877);
    p = fma(p, w, 0.0651041666613103);
    p = fma(p, w, -0.12499999999999988);
    const double off = fma(p, u, -0.78539816339744828);  // phi - pi/4
    double m = fma(-75.10534415095299, w, 4.648920550540045);
    m = fma(m, w, -0.4331145740700393);
    m = fma(m, w, 0.08259351363283507);
    m = fma(m, w, -0.04986778504944759);
    m = fma(m, w, 0.7978845608028653);
    // quadrant: round((x + off) 2/pi) by adding 1.5 2^52
    const double t = fma(x, 0.63661977236758138, off * 0.63661977236758138) + 6755399441055744.0;
    const double q = t - 6755399441055744.0;
#ifdef __CUDA_ARCH__
    const int iq = __double2loint(t);
#else
    const int iq = (int)(long long)q;
#endif
    double r = fma(-q, 1.5707963267948966, x);
    r = fma(-q, 6.123233995736766e-17, r) + off;
    const double z = r * r;
    const bool odd = iq & 1;
    double s = odd ? -7.578072323942544e-13 : -1.1353349346012276e-11;
    s = fma(s, z, odd ? 1.605835207122322e-10 : 2.0875581773272987e-09);
    s = fma(s, z, odd ? -2.505210477629445e-08 : -2.7557313093033837e-07);
    s = fma(s, z, odd ? 2.7557319213551425e-06 : 2.4801587283862812e-05);
    s = fma(s, z, odd ? -0.00019841269841253456 : -0.0013888888888861058);
    s = fma(s, z, odd ? 0.008333333333333321 : 0.04166666666666645);
    s = fma(s, z, odd ? -0.16666666666666666 : -0.5);
    s = fma(s, z, 1.0);
    const double a = odd ? r * m : m;  // cos(r + q pi/2): cos, -sin, -cos, sin
    const double v = (a * y) * s;
    return ((iq + 1) & 2) ? -v : v;
}

GFK_HD double j0_(double x) {
    if (x >= kJ0Asymptotic && x < kJ0Largest) return j0_modulus_phase(x);
    return j0(x);
}

}  // namespace gfk
