// ofx_num.cuh -- the two arithmetic types of the wide-state crystal pass
// (ofx_passx.cuh): native FP64, and float-float ("ff"), an unevaluated sum
// hi + lo of two FP32 values carrying about 48 significant bits.
//
// Why float-float on GB300: its FP64 rate is about 1/64 of its FP32 rate, so a
// complex multiply-add in float-float (~30 FP32 operations) costs less issue
// time than the same operation in FP64 (6 FP64 operations), while giving
// ~1e-14 relative precision -- enough for the high-gain cases in which the FP32
// field's rounding, amplified by the parametric gain, dominates the result.
//
// The float-float operations are the classical error-free transformations:
// TwoSum (Knuth, TAOCP vol. 2, 4.2.2), QuickTwoSum (Dekker 1971) and the exact
// product through a fused multiply-add (a*b - p = fma(a, b, -p)), combined as in
// the double-double literature (Hida, Li and Bailey, "Algorithms for quad-double
// precision floating point arithmetic", ARITH 2001), here one level down on FP32.
// Additions use the "sloppy" form: its error is bounded by a few units of 2^-48
// of max(|a|, |b|), which is the bound the FFT and the stage sums need (errors
// relative to the field's magnitude, not to a cancelled result).
//
// The translation unit that instantiates the float-float kernel is compiled with
// -fmad=false so that no a*b+c of an error-free transformation is contracted;
// every intended fused multiply-add is written as fmaf().
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

namespace ofx {

// ---------------------------------------------------------------------------
// float-float scalar
// ---------------------------------------------------------------------------
struct ff { float hi, lo; };

__device__ __forceinline__ ff ff_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    const float e = (a - (s - bb)) + (b - bb);
    return ff{s, e};
}
__device__ __forceinline__ ff ff_quick(float a, float b) {   // |a| >= |b|
    const float s = a + b;
    return ff{s, b - (s - a)};
}
__device__ __forceinline__ ff ff_add(ff a, ff b) {
    const ff s = ff_two_sum(a.hi, b.hi);
    return ff_quick(s.hi, s.lo + (a.lo + b.lo));
}
// scaling by an exact power of two (0.5, 2): exact
__device__ __forceinline__ ff ff_pow2(ff a, float s) { return ff{a.hi * s, a.lo * s}; }
__device__ __forceinline__ ff ff_from(double x) {
    const float h = (float)x;
    return ff{h, (float)(x - (double)h)};
}
__device__ __forceinline__ double ff_d(ff a) { return (double)a.hi + (double)a.lo; }

// ---------------------------------------------------------------------------
// complex types and the operations the kernel uses, per arithmetic type
// ---------------------------------------------------------------------------
// float-float complex, stored as {re.hi, im.hi, re.lo, im.lo}: the two parts' operations
// run as packed FP32 pairs
struct __align__(16) cff { float rh, ih, rl, il; };

template <typename R> struct Num;

template <> struct Num<double> {
    using cplx = double2;
    using real = double;
    static __device__ __forceinline__ cplx make(real re, real im) { return make_double2(re, im); }
    static __device__ __forceinline__ cplx zero() { return make_double2(0.0, 0.0); }
    static __device__ __forceinline__ real re(cplx a) { return a.x; }
    static __device__ __forceinline__ real im(cplx a) { return a.y; }
    static __device__ __forceinline__ cplx add(cplx a, cplx b) { return make_double2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ cplx sub(cplx a, cplx b) { return make_double2(a.x - b.x, a.y - b.y); }
    static __device__ __forceinline__ cplx mul(cplx a, cplx b) {
        return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    }
    static __device__ __forceinline__ cplx mulc(cplx a, cplx b) {   // a * conj(b)
        return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
    }
    static __device__ __forceinline__ cplx scale(cplx a, real s) { return make_double2(a.x * s, a.y * s); }
    static __device__ __forceinline__ cplx pow2(cplx a, double s) { return make_double2(a.x * s, a.y * s); }
    static __device__ __forceinline__ cplx mul_i(cplx a) { return make_double2(-a.y, a.x); }       // i a
    static __device__ __forceinline__ cplx mul_mi(cplx a) { return make_double2(a.y, -a.x); }      // -i a
    static __device__ __forceinline__ real rfrom(double x) { return x; }
    static __device__ __forceinline__ cplx from(double2 v) { return v; }
    static __device__ __forceinline__ double2 to_d(cplx v) { return v; }
    static __device__ __forceinline__ bool finite(cplx a) { return isfinite(a.x) && isfinite(a.y); }
    static __device__ __forceinline__ real triple(real a) { return 3.0 * a; }
    // n - i c d
    static __device__ __forceinline__ cplx sub_i(cplx n, cplx d, real c) {
        return make_double2(fma(c, d.y, n.x), fma(-c, d.x, n.y));
    }
    // a + b / 2
    static __device__ __forceinline__ cplx add_half(cplx a, cplx b) {
        return make_double2(fma(0.5, b.x, a.x), fma(0.5, b.y, a.y));
    }
    // |re|, |im| in FP32 from the bits (truncated; zero below FP32's range, infinite
    // above): GB300 converts FP64 at the rate of its narrow FP64 pipe
    static __device__ __forceinline__ float mag32(double x) {
        const unsigned h = __double2hiint(x) & 0x7fffffffu;
        const unsigned f = ((h - (896u << 20)) << 3) | ((unsigned)__double2loint(x) >> 29);
        return h < (897u << 20) ? 0.f : (h >= (1151u << 20) ? INFINITY : __uint_as_float(f));
    }
    static __device__ __forceinline__ float2 abs32(cplx a) { return make_float2(mag32(a.x), mag32(a.y)); }
};

// Packed pairs: the error-free transformations above on (re, im) at once.  The packed
// instructions name their rounding, so none is contracted.
__device__ __forceinline__ float2 pk_sub(float2 a, float2 b) {
    unsigned long long x, y, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
}
struct ff2 { float2 h, l; };                   // two float-float values
__device__ __forceinline__ ff2 ff2_quick(float2 a, float2 b) {
    const float2 s = __fadd2_rn(a, b);
    return ff2{s, pk_sub(b, pk_sub(s, a))};
}
__device__ __forceinline__ ff2 ff2_two_sum(float2 a, float2 b) {
    const float2 s = __fadd2_rn(a, b), bb = pk_sub(s, a);
    return ff2{s, __fadd2_rn(pk_sub(a, pk_sub(s, bb)), pk_sub(b, bb))};
}
__device__ __forceinline__ ff2 ff2_add(ff2 a, ff2 b) {
    const ff2 s = ff2_two_sum(a.h, b.h);
    return ff2_quick(s.h, __fadd2_rn(s.l, __fadd2_rn(a.l, b.l)));
}
__device__ __forceinline__ float2 pk_neg(float2 a) { return make_float2(-a.x, -a.y); }
// a*b + c*d per component, one final normalisation
__device__ __forceinline__ ff2 ff2_dot2(ff2 a, ff2 b, ff2 c, ff2 d) {
    const float2 p = __fmul2_rn(a.h, b.h), q = __fmul2_rn(c.h, d.h);
    const float2 ep = __ffma2_rn(a.h, b.h, pk_neg(p)), eq = __ffma2_rn(c.h, d.h, pk_neg(q));
    const ff2 s = ff2_two_sum(p, q);
    float2 t = __fadd2_rn(s.l, __fadd2_rn(ep, eq));
    t = __ffma2_rn(a.h, b.l, __ffma2_rn(a.l, b.h, t));
    t = __ffma2_rn(c.h, d.l, __ffma2_rn(c.l, d.h, t));
    return ff2_quick(s.h, t);
}
__device__ __forceinline__ ff2 ff2_mul(ff2 a, ff2 b) {
    const float2 p = __fmul2_rn(a.h, b.h);
    const float2 e = __ffma2_rn(a.h, b.h, pk_neg(p));
    return ff2_quick(p, __ffma2_rn(a.h, b.l, __ffma2_rn(a.l, b.h, e)));
}

template <> struct Num<ff> {
    using cplx = cff;
    using real = ff;
    static __device__ __forceinline__ cplx make(real re, real im) { return cff{re.hi, im.hi, re.lo, im.lo}; }
    static __device__ __forceinline__ cplx zero() { return cff{0.f, 0.f, 0.f, 0.f}; }
    static __device__ __forceinline__ real re(cplx a) { return ff{a.rh, a.rl}; }
    static __device__ __forceinline__ real im(cplx a) { return ff{a.ih, a.il}; }
    static __device__ __forceinline__ ff2 pk(cplx a) { return ff2{make_float2(a.rh, a.ih), make_float2(a.rl, a.il)}; }
    static __device__ __forceinline__ cplx un(ff2 a) { return cff{a.h.x, a.h.y, a.l.x, a.l.y}; }
    static __device__ __forceinline__ ff2 dup(real a) { return ff2{make_float2(a.hi, a.hi), make_float2(a.lo, a.lo)}; }
    static __device__ __forceinline__ ff2 swap(cplx a) { return ff2{make_float2(a.ih, a.rh), make_float2(a.il, a.rl)}; }
    static __device__ __forceinline__ cplx add(cplx a, cplx b) { return un(ff2_add(pk(a), pk(b))); }
    static __device__ __forceinline__ cplx sub(cplx a, cplx b) {
        return un(ff2_add(pk(a), ff2{make_float2(-b.rh, -b.ih), make_float2(-b.rl, -b.il)}));
    }
    // (ar br - ai bi, ar bi + ai br)
    static __device__ __forceinline__ cplx mul(cplx a, cplx b) {
        const ff2 ai{make_float2(-a.ih, a.ih), make_float2(-a.il, a.il)};
        return un(ff2_dot2(dup(re(a)), pk(b), ai, swap(b)));
    }
    // a conj(b) = (ar br + ai bi, ai br - ar bi)
    static __device__ __forceinline__ cplx mulc(cplx a, cplx b) {
        const ff2 bi{make_float2(b.ih, -b.ih), make_float2(b.il, -b.il)};
        return un(ff2_dot2(pk(a), dup(re(b)), swap(a), bi));
    }
    static __device__ __forceinline__ cplx scale(cplx a, real s) { return un(ff2_mul(pk(a), dup(s))); }
    static __device__ __forceinline__ cplx pow2(cplx a, double s) {
        const float f = (float)s;
        return cff{a.rh * f, a.ih * f, a.rl * f, a.il * f};
    }
    static __device__ __forceinline__ cplx mul_i(cplx a) { return cff{-a.ih, a.rh, -a.il, a.rl}; }
    static __device__ __forceinline__ cplx mul_mi(cplx a) { return cff{a.ih, -a.rh, a.il, -a.rl}; }
    static __device__ __forceinline__ real rfrom(double x) { return ff_from(x); }
    static __device__ __forceinline__ cplx from(double2 v) { return make(ff_from(v.x), ff_from(v.y)); }
    static __device__ __forceinline__ double2 to_d(cplx v) { return make_double2(ff_d(re(v)), ff_d(im(v))); }
    static __device__ __forceinline__ bool finite(cplx a) { return isfinite(a.rh) && isfinite(a.ih); }
    static __device__ __forceinline__ real triple(real a) { return ff_add(a, ff_pow2(a, 2.f)); }
    static __device__ __forceinline__ cplx sub_i(cplx n, cplx d, real c) { return sub(n, mul_i(scale(d, c))); }
    static __device__ __forceinline__ cplx add_half(cplx a, cplx b) { return add(a, pow2(b, 0.5)); }
    static __device__ __forceinline__ float2 abs32(cplx a) { return make_float2(a.rh, a.ih); }
};

}  // namespace ofx
