// fixed.cuh -- fixed-point conversion of the mass assignment's contributions.
#pragma once

namespace pbi4g {

// c 2^S rounded to the nearest integer, ties to even: __double2ll_rn((double)c * 2^S) from
// the bits of c.  The product is exact (a power of two) and the conversion is a shift; on
// the FP64 pipe (a 64th of the FP32 rate) the widening, the product and the conversion of
// every contribution took much of the assignment's time (FP64 form, 262,144 particles in 128^3,
// order 4 on two grids: 592 -> 527 us).  `s` is S; values at or beyond
// 2^63, infinities and NaN give what the conversion gives.
__device__ __forceinline__ long long to_fixed(double c, int s) {
    const long long u = __double_as_longlong(c);
    const int e = (int)(u >> 52) & 2047, sh = e - 1075 + s;
    const unsigned long long m = ((unsigned long long)u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    unsigned long long q;
    if (sh < 0) {
        const int r = -sh;
        q = r > 54 || e == 0 ? 0ull : (m + (1ull << (r - 1)) - 1 + ((m >> r) & 1)) >> r;
    } else if (sh <= 10 && e != 2047) {
        q = m << sh;
    } else {
        return u < 0 || (e == 2047 && (u << 12) != 0) ? (long long)(1ull << 63) : (long long)(~0ull >> 1);
    }
    return u < 0 ? -(long long)q : (long long)q;
}
__device__ __forceinline__ long long to_fixed(float c, int s) {
    const int u = __float_as_int(c);
    const int e = (u >> 23) & 255, sh = e - 150 + s;
    const unsigned m = ((unsigned)u & 0x7FFFFFu) | 0x800000u;
    unsigned long long q;
    if (sh < 0) {
        const int r = -sh;
        q = r > 25 || e == 0 ? 0u : (m + (1u << (r - 1)) - 1 + ((m >> r) & 1)) >> r;
    } else if (sh <= 39 && e != 255) {
        q = (unsigned long long)m << sh;
    } else {
        return u < 0 || (e == 255 && (u << 9) != 0) ? (long long)(1ull << 63) : (long long)(~0ull >> 1);
    }
    return u < 0 ? -(long long)q : (long long)q;
}

}  // namespace pbi4g
