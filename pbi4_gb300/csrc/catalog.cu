// catalog.cu -- catalogue positions to the [0, 1] positions the assignment
// reads, on the device (IO.read_catalogues, pbi4.py:121-245).
//
// The reference (numpy) does, for a catalogue of dtype T (float32 or float64):
//   pos[:] += Vel[:] * los / Hz * (1 + z)      (pbi4.py:158, 170, 214; Minerva
//                                               pbi4.py:184: pos += Vel * los)
//   pos = (pos + box) % box                     (pbi4.py:242)
//   pos = np.minimum(1 - nextafter(0, 1), pos / box)   (pbi4.py:243)
// with numpy's promotion rules: Vel * los is float64 (los is a float64 array), so
// the shift is computed in float64 and rounded once into T by the in-place add;
// box is a Python float, so the wrap and the division run in T; the clip
// compares with a float64 scalar (1 - 5e-324 == 1.0), so the result is float64.
// np.remainder for floats is fmod plus b where fmod's sign differs from b's.
//
// What bounds it: HBM, once the FP64 pipe is kept out (0.5 TFMA/s here: the chain
// product, division, product, sum of one float32 component, its division by hz alone ten
// FP64 operations, took 1.27 ms for 10^7 particles against 71 us of traffic; this form takes 103 us).
//  * A line-of-sight component that is zero shifts by an exact zero: no arithmetic.
//  * float32: the shifted position is formed in float32 pairs (shift_f32), whose error is
//    far below half an ulp of the rounded result; only where it could decide the rounding
//    does the lane run the reference's FP64 operations.
//  * divisions by hz and box as products with their reciprocals and residual corrections
//    (div_by): 5 operations, in float64 on the slow pipe.
//  * the wrap of a value in [0, 2 box) is at most one exact subtraction, not an fmod.
// Loads run over the catalogue as it lies (any alignment) into shared memory, a thread then
// takes whole particles: both sides are coalesced, and the branch on a zero component is
// uniform.
#include <float.h>
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "widen.cuh"

namespace pbi4g {

namespace {

constexpr int kPer = 6;  // components a thread loads: a tile is two particles a thread

struct CatArgs {
    double l[3];         // line of sight
    double hz, opz;      // rsd_mode 1: the shift is vel l / hz (1 + z)
    double rhz, rbox;    // correctly rounded reciprocals; 0: divide
    float rboxf;         // the same in float32
    float ch[3], cl[3];  // the shift's factor of vel as a float32 pair
    bool zero[3];        // the factor is zero: no shift
    int mode;
};

template <class V> __device__ __forceinline__ V pick(const V (&v)[3], int d) { return d == 0 ? v[0] : (d == 1 ? v[1] : v[2]); }

template <class T>
__device__ __forceinline__ T remainder_np(T a, T b) {
    if (a >= (T)0 && a < b) return a;
    if (a >= b && a < (T)2 * b) return a - b;  // exact (Sterbenz), as fmod is
    T m = fmod(a, b);
    if (m != (T)0 && ((b < (T)0) != (m < (T)0))) m += b;
    return m;
}

// a / b correctly rounded, from r = 1 / b correctly rounded: a quotient within one ulp,
// corrected twice by its exact residual (Markstein 1990: the last correction of a quotient
// within one ulp rounds correctly).  Needs b and the quotient far from the ends of the
// exponent range: |a| in [2^-700, 2^700] here, else (and for 0, inf, NaN) the division.
__device__ __forceinline__ double div_by(double a, double b, double r) {
    const int e = (__double2hiint(a) >> 20) & 2047;
    if (r == 0.0 || e < 1023 - 700 || e > 1023 + 700) return __ddiv_rn(a, b);
    double q = __dmul_rn(a, r);
    q = __fma_rn(__fma_rn(-q, b, a), r, q);
    return __fma_rn(__fma_rn(-q, b, a), r, q);
}

// the same in float32, for a = +0 or in [2^-40, 2^40] (the quotients of a wrapped position)
__device__ __forceinline__ float div_by(float a, float b, float r) {
    const unsigned u = __float_as_uint(a);
    if (r == 0.f || (u != 0u && u - ((127u - 40u) << 23) > (80u << 23))) return __fdiv_rn(a, b);
    float q = __fmul_rn(a, r);
    q = __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
    return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// the reference's operations: the shift in FP64 (one rounding each, no contraction), the
// in-place add rounded to T
template <class T>
__device__ __forceinline__ T shift_ref(T p, T v, const CatArgs &a, int d) {
    double t = __dmul_rn((double)v, pick(a.l, d));
    if (a.mode == 1) t = __dmul_rn(div_by(t, a.hz, a.rhz), a.opz);
    return (T)__dadd_rn((double)p, t);
}

// float32: p + v c with c = ch + cl to 2^-47, in float32 pairs.  s + e is the sum to
// 2^-45 (|s| + |th|): the product's error by FMA, the sum's by Knuth's two-sum, and the
// reference's own FP64 roundings are below 2^-50 of either.  Rounding s + e gives the
// reference's result unless a tie between two float32 values lies within that error of
// it; the test takes 2^-42 for it, and zeros, tiny values, inf and NaN go the FP64 way too.
__device__ __forceinline__ float shift_f32(float p, float v, const CatArgs &a, int d) {
    const float ch = pick(a.ch, d), cl = pick(a.cl, d);
    const float th = __fmul_rn(v, ch);
    const float tl = __fmaf_rn(v, cl, __fmaf_rn(v, ch, -th));
    const float s = __fadd_rn(p, th);
    const float bb = __fsub_rn(s, p);
    const float es = __fadd_rn(__fsub_rn(p, __fsub_rn(s, bb)), __fsub_rn(th, bb));
    const float e = __fadd_rn(es, tl);
    const float r = __fadd_rn(s, e);
    const float off = __fadd_rn(__fsub_rn(s, r), e);  // what the rounding left
    const int rb = __float_as_int(r);
    // half an ulp of r on its closer side
    const float h = __int_as_float((rb & 0x7f800000) - ((rb & 0x7fffff) ? 24 : 25) * (1 << 23));
    const float room = h - 0x1p-42f * (fabsf(s) + fabsf(th));
    if (fabsf(r) > 0x1p-60f && fabsf(r) < 0x1p100f && fabsf(off) < room) return r;
    return shift_ref<float>(p, v, a, d);
}

// one component: shift, wrap, scale, clip
__device__ __forceinline__ double position(float p, float v, bool shift, float box, const CatArgs &a, int d) {
    if (shift && !(pick(a.zero, d) && isfinite(v))) p = shift_f32(p, v, a, d);
    const float q = div_by(remainder_np<float>(__fadd_rn(p, box), box), box, a.rboxf);
    return q < 1.f || isnan(q) ? widen(q) : 1.0;  // np.minimum keeps NaN
}
__device__ __forceinline__ double position(double p, double v, bool shift, double box, const CatArgs &a, int d) {
    if (shift && !(pick(a.zero, d) && isfinite(v))) p = shift_ref<double>(p, v, a, d);
    const double q = div_by(remainder_np<double>(__dadd_rn(p, box), box), box, a.rbox);
    return q < 1.0 || isnan(q) ? q : 1.0;
}

template <class T, bool SHIFT, int kThreads>
__global__ void __launch_bounds__(kThreads) catalog_positions_kernel(int64_t n, const T *__restrict__ pos,
                                                                    const T *__restrict__ vel, const CatArgs a, T box,
                                                                    double *__restrict__ out) {
    constexpr int kTile = 2 * kThreads;
    __shared__ T sp[3 * kTile], sv[SHIFT ? 3 * kTile : 1];
    const int t = threadIdx.x;
    const int64_t ntiles = (n + kTile - 1) / kTile;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t base = tile * kTile;
        const int np = (int)(n - base < kTile ? n - base : kTile), ne = 3 * np;
        T p[kPer], v[SHIFT ? kPer : 1];
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            const int e = t + j * kThreads;
            p[j] = e < ne ? __ldcs(pos + 3 * base + e) : (T)0;
            if (SHIFT) v[j] = e < ne ? __ldcs(vel + 3 * base + e) : (T)0;
        }
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            sp[t + j * kThreads] = p[j];
            if (SHIFT) sv[t + j * kThreads] = v[j];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTile / kThreads; k++) {
            const int i = t + k * kThreads;
            if (i >= np) break;
#pragma unroll
            for (int d = 0; d < 3; d++)
                __stcs(out + (size_t)d * n + base + i,
                       position(sp[3 * i + d], SHIFT ? sv[3 * i + d] : (T)0, SHIFT, box, a, d));
        }
        __syncthreads();
    }
}

// 1 / b for div_by, or 0 where b is too near the ends of the exponent range for it
double reciprocal(double b) { return fabs(b) > 0x1p-300 && fabs(b) < 0x1p300 ? 1.0 / b : 0.0; }
float reciprocal(float b) { return fabsf(b) > 0x1p-30f && fabsf(b) < 0x1p30f ? 1.0f / b : 0.0f; }

}  // namespace

}  // namespace pbi4g

using namespace pbi4g;

extern "C" {

int pbi4g_catalog_positions(int64_t npart, const void *d_pos, const void *d_vel, int32_t is_double,
                            const double *los, int32_t rsd_mode, double hz, double z, double box, double *d_out,
                            void *stream) {
    if (npart < 0 || (npart > 0 && (!d_pos || !d_out)) || !(box > 0) || (d_vel && !los) ||
        (d_vel && (rsd_mode < 0 || rsd_mode > 1)) || (d_vel && rsd_mode == 1 && !(hz != 0)))
        return set_error(PBI4G_ERR_INVALID, "catalogue positions: npart=%lld box=%g rsd_mode=%d hz=%g",
                         (long long)npart, box, rsd_mode, hz);
    if (npart == 0) return PBI4G_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    CatArgs a = {};
    a.hz = hz;
    a.opz = 1.0 + z;
    a.mode = rsd_mode;
    a.rhz = reciprocal(hz);
    a.rbox = reciprocal(box);
    a.rboxf = reciprocal((float)box);
    for (int d = 0; d < 3; d++) {
        a.l[d] = d_vel ? los[d] : 0;
        // a zero shift: 0 / hz (1 + z) is a zero for finite hz and 1 + z
        a.zero[d] = a.l[d] == 0 && (rsd_mode == 0 || (isfinite(hz) && isfinite(a.opz)));
        const double c = rsd_mode == 1 ? a.l[d] / hz * a.opz : a.l[d];
        a.ch[d] = (float)c;
        a.cl[d] = (float)(c - (double)a.ch[d]);
        // a factor whose float32 pair is not that accurate: NaN sends every lane the FP64 way
        if (!(fabs(c) > 0x1p-60 && fabs(c) < 0x1p60)) a.ch[d] = NAN;
    }
    auto launch = [&](auto kern, auto box_t, int threads) {
        using T = decltype(box_t);
        kern<<<grid_blocks((size_t)npart, 2 * threads, 152 * 16), threads, 0, st>>>(
            npart, static_cast<const T *>(d_pos), static_cast<const T *>(d_vel), a, box_t, d_out);
    };
    auto sized = [&](auto box_t, auto threads) {
        using T = decltype(box_t);
        constexpr int TH = decltype(threads)::value;
        launch(d_vel ? catalog_positions_kernel<T, true, TH> : catalog_positions_kernel<T, false, TH>, box_t, TH);
    };
    // small tiles where large ones would be fewer than four an SM (42,836 float64 particles were
    // 84 CTAs on 152 SMs: 2.5 us more)
    const std::integral_constant<int, 256> large;
    const std::integral_constant<int, 64> little;
    const bool few = npart < (int64_t)152 * 4 * 512;
    if (is_double) few ? sized(box, little) : sized(box, large);
    else few ? sized((float)box, little) : sized((float)box, large);
    PBI4G_LAUNCH_CHECK();
    return PBI4G_OK;
}

}  // extern "C"
