// FP64 building blocks of the Green-kernel samples: reciprocal square root and
// sine/cosine without the special-case paths of the library functions.
//
// A sample spends most of its FP64 instructions here. The library's rsqrt and
// sincos carry branches for denormal, infinite and very large arguments that
// no sample meets (distances are checked by the caller, and k*r stays far below
// kSinCosLimit between panels, whose areas are at least 1e-14 of the mesh's
// extent squared; observers may lie anywhere, so the fields check it), and those branches keep the compiler from interleaving the samples of
// an unrolled loop. Both functions are within 1.5 units in the last place
// (measured: root 0.99, sine 1.44, cosine 1.45 over 1e-12 .. 1e7), like the
// library's.
#pragma once

#include <cuda_runtime.h>

namespace hsb {

// 1/sqrt(x) for normal positive x: the hardware's approximation (over 20 bits)
// and one Householder step of third order, which leaves less than 2^-58.
// Zero, negative, infinite and NaN arguments give NaN or infinity.
__device__ __forceinline__ double reciprocalRoot(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(fma(e, 0.375, 0.5), e * y, y);
}

// sin(x) and cos(x) for |x| < kSinCosLimit: Cody-Waite reduction by pi/2 in two parts
// (the first product is exact inside its fma, because the difference has no bit
// below 2^-52 and is smaller than one), then minimax polynomials on
// [-pi/4, pi/4] fitted with the Remez exchange in 60 digits: relative error
// 3.5e-18 of sin(r)/r, absolute 4.7e-20 of cos(r).
constexpr double kSinCosLimit = 0x1p31;
__device__ __forceinline__ void sinCos(double x, double &sine, double &cosine) {
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    const double shifted = fma(x, 0x1.45f306dc9c883p-1, kRound);
    const int quadrant = __double2loint(shifted);
    const double turns = shifted - kRound;
    const double r = fma(-turns, 0x1.1a62633145c07p-54, fma(-turns, 0x1.921fb54442d18p+0, x));
    const double t = r * r;
    double s = 0x1.5d9300537b9efp-33, c = -0x1.8fae9c8e18ca4p-37;
    s = fma(s, t, -0x1.ae5e663807f5fp-26);
    c = fma(c, t, 0x1.1ee9ebe95c282p-29);
    s = fma(s, t, 0x1.71de3577b2fa4p-19);
    c = fma(c, t, -0x1.27e4f809f0e80p-22);
    s = fma(s, t, -0x1.a01a019c1194ap-13);
    c = fma(c, t, 0x1.a01a019cb1be1p-16);
    s = fma(s, t, 0x1.111111110f87ap-7);
    c = fma(c, t, -0x1.6c16c16c1517ep-10);
    s = fma(s, t, -0x1.5555555555549p-3);
    c = fma(c, t, 0x1.555555555554cp-5);
    c = fma(c, t, -0.5);
    s = fma(r * t, s, r);
    c = fma(c, t, 1.0);
    const bool swap = quadrant & 1;
    const double a = swap ? c : s, b = swap ? s : c;
    // signs: sine negative in quadrants 2, 3, cosine in 1, 2
    sine = __hiloint2double(__double2hiint(a) ^ ((quadrant & 2) << 30), __double2loint(a));
    cosine = __hiloint2double(__double2hiint(b) ^ (((quadrant + 1) & 2) << 30), __double2loint(b));
}

// Distance check on squared distances without FP64 compares: collects the
// smallest and largest high words, which order like the values for r^2 >= 0.
struct DistanceCheck {
    unsigned low = 0x7fffffffu, high = 0;
    __device__ __forceinline__ void add(double r2) {
        const unsigned h = unsigned(__double2hiint(r2));
        low = min(low, h);
        high = max(high, h);
    }
    // some value was zero (or denormal), infinite or NaN
    __device__ __forceinline__ bool bad() const { return low < 0x00100000u || high >= 0x7ff00000u; }
};

}  // namespace hsb
