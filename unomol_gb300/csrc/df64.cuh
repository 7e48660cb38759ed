// Unevaluated sums of two floats: a value h + l with |l| about 2^-24 |h| carries about 48 bits.  GB300's
// FP64 pipe runs at 1/64 of the FP32 rate, so a product (4 FP32 instructions) or a fused multiply-add (12)
// in this form costs a small part of one FP64 instruction.  The error-free transformations are the
// published ones (T. J. Dekker, Numer. Math. 18, 224 (1971); D. E. Knuth, TAOCP 2, 4.2.2), with products
// through FMA.  Every operation is a rounding intrinsic, so that the compiler contracts none of them.
//
// The sums are left unnormalised: l may grow past half an ulp of h after a cancellation.  Errors stay below
// a few 2^-48 of the largest operand that entered, which is the bound that the callers rely on.
#pragma once
#include <cuda_runtime.h>

namespace ugb {

struct df {
    float h, l;
};

__device__ __forceinline__ df df_neg(df a) { return {-a.h, -a.l}; }
__device__ __forceinline__ df df_half(df a) { return {__fmul_rn(0.5f, a.h), __fmul_rn(0.5f, a.l)}; }

// the same sum with h its rounded value and l the exact rest (|a.h| >= |a.l|)
__device__ __forceinline__ df df_norm(df a) {
    const float s = __fadd_rn(a.h, a.l);
    return {s, __fsub_rn(a.l, __fsub_rn(s, a.h))};
}

// a b
__device__ __forceinline__ df df_mul(df a, df b) {
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return {p, e};
}
// a b, normalised, for the factors that many others are multiplied with: three additions more, and the next product
// leaves out the square of half an ulp and not of a few
__device__ __forceinline__ df df_muln(df a, df b) { return df_norm(df_mul(a, b)); }
// a^2.  l^2 counts although it lies below the last bit: it is never negative, so leaving it out, or adding it to a
// value that is rounded already, would make every square too small, by 2^-50 of it on average, and sums over many
// quartets keep such a bias where they average rounding away
__device__ __forceinline__ df df_sqr(df a) {
    const float p = __fmul_rn(a.h, a.h);
    const float t = __fmaf_rn(__fadd_rn(a.h, a.h), a.l, __fmul_rn(a.l, a.l));
    return {p, __fadd_rn(__fmaf_rn(a.h, a.h, -p), t)};
}
// a f with a single float f
__device__ __forceinline__ df df_mulf(df a, float f) {
    const float p = __fmul_rn(a.h, f);
    float e = __fmaf_rn(a.h, f, -p);
    e = __fmaf_rn(a.l, f, e);
    return {p, e};
}
// a + b, any magnitudes
__device__ __forceinline__ df df_add(df a, df b) {
    const float s = __fadd_rn(a.h, b.h);
    const float t = __fsub_rn(s, a.h);
    const float e = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, t)), __fsub_rn(b.h, t));
    return {s, __fadd_rn(e, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ df df_sub(df a, df b) { return df_add(a, df_neg(b)); }
// a - c of two sums of three floats on common steps (PairCentre): the differences of the first and of the second parts
// are exact, and the first is zero or at least as large as the second
__device__ __forceinline__ df df_triple_diff(float ah, float am, float al, float ch, float cm, float cl) {
    const float h = __fsub_rn(ah, ch), m = __fsub_rn(am, cm), s = __fadd_rn(h, m);
    return {s, __fadd_rn(__fsub_rn(m, __fsub_rn(s, h)), __fsub_rn(al, cl))};
}
// a - b, normalised: of two close values what is left of l is up to half an ulp of a and not of the difference, and
// the products, which leave out l l, would then be off by its square
__device__ __forceinline__ df df_diff(df a, df b) { return df_norm(df_sub(a, b)); }
// a b + c, any magnitudes
__device__ __forceinline__ df df_fma(df a, df b, df c) { return df_add(c, df_mul(a, b)); }
// f - a for |f| >= |a|
__device__ __forceinline__ df df_rsubf(float f, df a) {
    const float s = __fsub_rn(f, a.h);
    return {s, __fsub_rn(__fsub_rn(__fsub_rn(f, s), a.h), a.l)};
}
// 1 / sqrt(a), a > 0, normalised (its square is taken): the hardware approximation r and the series of
// (1 - e)^(-1/2) with e = 1 - a r^2 to second order (|e| is about 2^-21, so what is left out is below 2^-60)
__device__ __forceinline__ df df_rsqrt(df a) {
    const float r = rsqrtf(a.h);
    const float q = __fmul_rn(r, r), ql = __fmaf_rn(r, r, -q);
    const float p = __fmul_rn(a.h, q);
    float t = __fmaf_rn(a.h, q, -p);
    t = __fmaf_rn(a.h, ql, t);
    t = __fmaf_rn(a.l, q, t);
    const float e = __fsub_rn(__fsub_rn(1.0f, p), t);
    const float c = __fmul_rn(__fmul_rn(r, e), __fmaf_rn(0.375f, e, 0.5f));
    return df_norm({r, c});
}

}  // namespace ugb
