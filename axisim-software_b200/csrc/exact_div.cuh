// exact_div.cuh -- a / b for many a and one b, correctly rounded.
//
// P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990): with y = 1/b correctly
// rounded and q within an ulp of a/b, the remainder r = a - b q is exact in one
// FMA and q + r y rounds to the correctly rounded quotient. q0 = a y may be two
// ulps off, so one such step brings it within an ulp and a second one rounds it.
// The steps need no over- or underflow in b q, 1/b and q: exponents outside
// the ranges below (infinities and NaN included) take the division operator, and
// a zero keeps its sign in a y. The reciprocal is formed once per divisor; a quotient is then five
// dependent FMA-pipe operations (54 cycles in FP64, 35 in FP32 on a B200)
// where the division operator measures 114 and 47.
#pragma once

#include <cuda_runtime.h>

namespace axisim {

template <class T>
struct ExactDiv;

template <>
struct ExactDiv<double> {
    double b, y;
    bool ok;
    __device__ __forceinline__ explicit ExactDiv(double d) : b(d), y(1.0 / d) {
        const int e = (__double2hiint(d) >> 20) & 0x7ff;
        ok = (unsigned)(e - (1023 - 100)) <= 200u;  // 2^-100 .. 2^101
    }
    __device__ __forceinline__ double operator()(double a) const {
        const int e = (__double2hiint(a) >> 20) & 0x7ff;
        const double q0 = a * y;
        const double q1 = fma(fma(-b, q0, a), y, q0);
        double q = a == 0.0 ? q0 : fma(fma(-b, q1, a), y, q1);
        if (!ok || ((unsigned)(e - (1023 - 900)) > 1700u && a != 0.0)) q = a / b;  // outside 2^-900 .. 2^801
        return q;
    }
};

template <>
struct ExactDiv<float> {
    float b, y;
    bool ok;
    __device__ __forceinline__ explicit ExactDiv(float d) : b(d), y(1.0f / d) {
        const int e = (__float_as_int(d) >> 23) & 0xff;
        ok = (unsigned)(e - (127 - 60)) <= 90u;  // 2^-60 .. 2^31
    }
    __device__ __forceinline__ float operator()(float a) const {
        const int e = (__float_as_int(a) >> 23) & 0xff;
        const float q0 = a * y;
        const float q1 = fmaf(fmaf(-b, q0, a), y, q0);
        float q = a == 0.0f ? q0 : fmaf(fmaf(-b, q1, a), y, q1);
        if (!ok || ((unsigned)(e - (127 - 90)) > 150u && a != 0.0f)) q = a / b;  // outside 2^-90 .. 2^61
        return q;
    }
};

}  // namespace axisim
