// widen.cuh -- float32 -> float64 in integer arithmetic (conversions run at the FP64 pipe's
// rate, 1.7 a clock and SM).
#pragma once

namespace pbi4g {

__device__ __forceinline__ double widen(float q) {
    const unsigned u = __float_as_uint(q);
    unsigned m = u & 0x7fffffffu;
    long long bias = 896;
    if (m < 0x00800000u) {  // zero or subnormal: scaled into the normal range, exactly
        m = __float_as_uint(fabsf(q) * 0x1p64f);
        bias = m ? 896 - 64 : 0;
    } else if (m >= 0x7f800000u) {  // inf, NaN: exponent 2047
        bias = 2047 - 255;
    }
    return __longlong_as_double(((long long)(u >> 31) << 63) | (((long long)m << 29) + (bias << 52)));
}

}  // namespace pbi4g
