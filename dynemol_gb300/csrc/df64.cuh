// Double-float (DF64) arithmetic on the FP32 pipes.  A value is the unevaluated
// sum hi + lo of two FP32 numbers (48-bit significand, about 4e-15 relative).
// Products use Dekker's exact product error by FMA, sums Knuth's TwoSum; every
// step is a round-to-nearest intrinsic so that the compiler contracts nothing.
// GB300's FP64 pipe runs at 1/58 of its FP32 rate, so about a dozen FP32
// instructions per FP64-equivalent operation still leaves DF64 5x ahead.
#pragma once

#include <cuda_runtime.h>

namespace elhl {

__device__ __forceinline__ float2 df_split(double x) {
    const float h = __double2float_rn(x);
    return make_float2(h, __double2float_rn(x - (double)h));
}

// (sh, sl) += (ah + al)(bh + bl), dropping al bl (2^-48 relative)
__device__ __forceinline__ void df_fma(float &sh, float &sl, float ah, float al, float bh, float bl) {
    const float p = __fmul_rn(ah, bh);
    float e = __fmaf_rn(ah, bh, -p);
    e = __fmaf_rn(ah, bl, e);
    e = __fmaf_rn(al, bh, e);
    const float t = __fadd_rn(sh, p);
    const float z = __fsub_rn(t, sh);
    const float y = __fadd_rn(__fsub_rn(sh, __fsub_rn(t, z)), __fsub_rn(p, z));
    sl = __fadd_rn(sl, __fadd_rn(y, e));
    sh = t;
}

// (ah, al) + (bh, bl) in FP32 pairs (TwoSum of the high parts, low parts added)
__device__ __forceinline__ void df_add(float &ah, float &al, float bh, float bl) {
    const float t = __fadd_rn(ah, bh);
    const float z = __fsub_rn(t, ah);
    const float y = __fadd_rn(__fsub_rn(ah, __fsub_rn(t, z)), __fsub_rn(bh, z));
    al = __fadd_rn(al, __fadd_rn(y, bl));
    ah = t;
}

// s + e = a + b exactly (Knuth's TwoSum), s in a, e in b
__device__ __forceinline__ void two_sum(float &a, float &b) {
    const float s = __fadd_rn(a, b);
    const float z = __fsub_rn(s, a);
    b = __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));
    a = s;
}

// FP32 triples s[0] + s[1] + s[2]: sums of FP32 numbers with less error (2^-70 of the largest
// partial sum) than FP64 makes, without the FP64 pipe.
__device__ __forceinline__ void ts_add(float (&s)[3], float y) {
    two_sum(s[0], y);
    two_sum(s[1], y);
    s[2] = __fadd_rn(s[2], y);
}
// A triple rounded to FP32, to nearest of the triple's value: b + c is rounded to odd (its last
// bit set where something lies below it, so that no tie is seen where there is none), then a
// added (S. Boldo, G. Melquiond, Emulation of FMA and correctly rounded sums: proved
// algorithms using rounding to odd, 2008).
__device__ __forceinline__ float ts_round(float a, float b, float c) {
    two_sum(a, b);
    two_sum(b, c);
    int i = __float_as_int(b);
    if (c != 0.f && !(i & 1)) i += (i ^ __float_as_int(c)) < 0 ? -1 : 1;
    return __fadd_rn(a, __int_as_float(i));
}

// (a + b) + c rounded once for |c| far below ulp(a + b): TwoSum gives a + b = t + e
// exactly, then t + (e + c)
__device__ __forceinline__ float two_sum_plus(float a, float b, float c) {
    const float t = __fadd_rn(a, b);
    const float z = __fsub_rn(t, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(t, z)), __fsub_rn(b, z));
    return __fadd_rn(t, __fadd_rn(e, c));
}

}  // namespace elhl
