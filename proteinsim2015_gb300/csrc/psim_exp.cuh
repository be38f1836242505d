// psim_exp.cuh -- exp(x) in FP64 from a table, for passes bound by the FP64 unit.
#pragma once

#include <cmath>

#include <cuda_runtime.h>

namespace psim {

constexpr int kExpTable = 256;

// 2^(k/256), k = 0 .. 255, and its rounding
inline void exp_table_values(double2* e2) {
    for (int k = 0; k < kExpTable; ++k) {
        const long double v = exp2l(k / (long double)kExpTable);
        e2[k].x = (double)v;
        e2[k].y = (double)(v - (long double)e2[k].x);
    }
}

// exp(x) by the table-driven method (Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM TOMS 15, 1989):
// x = (256 e + k) ln2/256 + r, e^x = 2^e 2^(k/256) (1 + r + r^2/2 + c r^3 + r^4/24)
// with |r| <= h = ln2/512; the table holds each value's rounding too.  r^5/120, up to
// 0.34 x 2^-53, is left to the cubic term: c = 1/6 + 0.869 h^2/120, as 0.869 x^3 comes
// closest to x^5 on [-1, 1] (0.131 away at most), which leaves 0.045 x 2^-53.  Eleven FP64
// operations against exp()'s ~18, in passes that take as long as they have FP64
// operations; largest error 1.04 and rms 0.425 x 2^-53 of the value over 2^20 x in [-14, 0]
// and in [-689, 689] (exp() 1.22 and 0.441; with c = 1/6 1.32 and 0.436).
__device__ __forceinline__ double exp_table(double x, const double2* e2) {
    if ((__double2hiint(x) & 0x7fffffff) >= 0x40859000) return exp(x);   // |x| >= 690, NaN
    // rounding to an integer by adding 1.5 2^52, which leaves it in the low word
    const double magic = 6755399441055744.0;
    const double t = __fma_rn(x, 369.3299304675746271, magic);   // 256 / ln2
    const double k = __dadd_rn(t, -magic);
    const int n = __double2loint(t);
    // ln2/256 in two parts, the first short enough for an exact product with k
    double r = __fma_rn(k, -0x1.62e42fefap-9, x);
    r = __fma_rn(k, -0x1.cf79abc9e3b3ap-48, r);
    constexpr double h = 0.69314718055994531 / 512.0, c = 1.0 / 6.0 + 0.869 * h * h / 120.0;
    const double q = __fma_rn(r, __fma_rn(r, 1.0 / 24.0, c), 0.5);
    const double p = __fma_rn(__dmul_rn(r, r), q, r);
    const double2 f = __ldg(e2 + (n & 255));
    const double v = __dadd_rn(f.x, __fma_rn(f.x, p, f.y));
    return __hiloint2double(__double2hiint(v) + ((n >> 8) << 20), __double2loint(v));
}

}  // namespace psim
