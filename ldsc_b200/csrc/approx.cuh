// approx.cuh -- roots, quotients and reciprocals from the hardware's
// approximations and one correction step, without the branches that the IEEE
// operations take for special cases.  ldsc_debug_approx counts where they differ
// from those operations.
#pragma once
#include <cstdint>

namespace ldsc {

// Square root and quotient of normal f32 numbers well inside the range: the
// hardware's approximation and one correction from the exact remainder
// (Newton's step for the root, Markstein's final correction for the quotient),
// with no branch for special cases.  Against the IEEE operations: all 226
// million x in [8, 2^30) equal; 6 of 3 billion quotients differ, by one place.
__device__ __forceinline__ float sqrt_nr(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float s = x * y;
    return fmaf(fmaf(-s, s, x), 0.5f * y, s);
}
__device__ __forceinline__ float div_nr(float a, float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    const float q = a * y;
    return fmaf(fmaf(-q, b, a), y, q);
}

// 1 / d for positive d from the hardware's approximation of the upper word
// (about 20 bits) by one step of Halley's iteration, which triples the bits:
// with e = 1 - d r, 1/d = r / (1 - e) = r (1 + e + e^2 + ...), so r + r (e + e^2)
// leaves e^3 (1 of 3,400 results is one place from the IEEE quotient).  Without
// the division's own range checks the chains of a step interleave.  Values
// outside the normal range's middle take the division.
__device__ __forceinline__ bool recip_plain(double d) {
    const uint32_t e = ((uint32_t)__double2hiint(d) >> 20);   // sign and exponent: 0x3FF at 1
    return e - 2u < 2042u;
}
__device__ __forceinline__ double recip_halley(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

}  // namespace ldsc
