// gfk_j0.cuh — Bessel J0 in FP64 for the wavenumber sums.
//
// The sums over wavenumber evaluate J0(k r) once per (wavenumber, range), at
// arguments mostly far above 25. There J0 is written in modulus-phase form,
//     J0(x) = M(x) cos(x - pi/4 + phi(x)),   H0(x) = M e^{i (x - pi/4 + phi)},
// (Watson, "A Treatise on the Theory of Bessel Functions", 13.75): one cosine
// instead of two, and M sqrt(x) and x phi are smooth functions of w = 1/x^2.
// Their polynomials are the degree-5 Chebyshev interpolants on
// [0, 1/625], computed from 60-digit values of J0 and Y0; absolute errors
// 6e-17 / sqrt(x) and 5e-18. The phase is reduced by a multiple of pi in two
// parts (Cody and Waite) with fused multiply-adds, the multiple chosen with
// the offset included, so the remainder stays in [-pi/2, pi/2]; its cosine is
// the degree-9 Chebyshev interpolant in its square (error 1.6e-17). Reducing
// by pi/2 needs two FP64 steps fewer, but picking sine's or cosine's
// coefficients costs 28 moves and selects.
// Below 25, and from 2^30 on, CUDA's j0.
//
// 38 FP64 instructions against about 130 issue slots measured for CUDA's
// j0 (16.7M values in 0.12 ms): the FP64 pipe bounds every sum that evaluates
// it in the loop. Absolute error against 40-digit values at 6200 points of
// [25, 1e9] (compiled for the host): at most 7e-17 (glibc's j0: 6e-17).
#pragma once
#include "gfk_math.cuh"

namespace gfk {

constexpr double kJ0Asymptotic = 25.0;       // from here the modulus-phase form
constexpr double kJ0Largest = 1073741824.0;  // below this the multiple of pi fits an int

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
    // round((x + off)/pi) by adding 1.5 2^52
    const double t = fma(x, 0.3183098861837907, off * 0.3183098861837907) + 6755399441055744.0;
    const double q = t - 6755399441055744.0;
    double r = fma(-q, 3.141592653589793, x);
    r = fma(-q, 1.2246467991473532e-16, r) + off;
    const double z = r * r;
    double c = fma(-1.5119729481048052e-16, z, 4.77687121758436e-14);
    c = fma(c, z, -1.1470670120398209e-11);
    c = fma(c, z, 2.0876755665527946e-09);
    c = fma(c, z, -2.7557319209640205e-07);
    c = fma(c, z, 2.480158730149253e-05);
    c = fma(c, z, -0.001388888888888853);
    c = fma(c, z, 0.04166666666666666);
    c = fma(c, z, -0.5);
    c = fma(c, z, 1.0);
    const double v = (m * y) * c;
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(v) ^ (__double2loint(t) << 31), __double2loint(v));
#else
    return ((long long)q & 1) ? -v : v;
#endif
}

GFK_HD double j0_(double x) {
    if (x >= kJ0Asymptotic && x < kJ0Largest) return j0_modulus_phase(x);
    return j0(x);
}

}  // namespace gfk
