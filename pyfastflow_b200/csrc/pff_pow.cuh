// h^(5/3) as the reference forms it: the exponent rounded to f32, the power correctly
// rounded to f32 from double.
//
// The double-precision pow cost about two thirds of the Manning update (58 us at 2048^2,
// where its bytes take 18).  Here r = h^(-1/3) starts from the hardware's f32 log2 and
// exp2 (relative error below 1e-5) and takes one third-order step in double,
// r (1 + e/3 + 2 e^2/9) with e = 1 - h r^3, leaving about 1e-15; h^(5/3) = h^2 r; the
// exponent's rounding d = 5.0f/3.0f - 5/3 (about -4e-8) multiplies by exp(d ln h) =
// 1 + g + g^2/2, whose error is at most 1e-12 (log2's absolute error of 2.4e-5 times d).
// A result within 2^-36 of halfway between two floats, where that error could decide the
// rounding (one in 4096), and arguments outside [2^-70, 2^70] (zero, negative, NaN
// among them) take pow.  pff_pow53_selfcheck compares the two over ranges of floats.
#pragma once
#include <cuda_runtime.h>

namespace pff {

static __device__ __noinline__ float pow53_full(float h) { return (float)pow((double)h, (double)(5.0f / 3.0f)); }

__device__ __forceinline__ float pow53(float h)
{
    if (h >= 0x1p-70f && h <= 0x1p70f) {
        float l, r0;
        asm("lg2.approx.f32 %0, %1;" : "=f"(l) : "f"(h));
        asm("ex2.approx.f32 %0, %1;" : "=f"(r0) : "f"(__fmul_rn(l, -1.0f / 3.0f)));
        const double H = (double)h, r = (double)r0;
        const double e = fma(-H, r * r * r, 1.0);
        const double q = fma(r, e * fma(e, 2.0 / 9.0, 1.0 / 3.0), r);
        constexpr double d_ln2 = ((double)(5.0f / 3.0f) - 5.0 / 3.0) * 0.69314718055994530942;
        const double g = (double)l * d_ln2;
        const double v0 = H * H * q;
        const double v = fma(v0, fma(g, 0.5 * g, g), v0);
        const int tail = (__double2loint(v) & 0x1FFFFFFF) - 0x10000000;  // from halfway, in 2^-52 steps
        if (tail > 65536 || tail < -65536) return __double2float_rn(v);
    }
    return pow53_full(h);
}

}  // namespace pff
