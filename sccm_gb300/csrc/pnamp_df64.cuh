// Double-float arithmetic: a value is the unevaluated sum hi + lo of two
// floats (|lo| <= ulp(hi)/2), about 48 significant bits. GB300 issues FP32
// FMAs at ~60x its FP64 rate, so the O(n^3) per-point algebra in this form
// runs on the FP32 pipes. Algorithms: Knuth's TwoSum, Dekker's FastTwoSum and
// the FMA-based TwoProduct (exact product error), combined as in the
// double-double literature (Hida, Li, Bailey, "Algorithms for quad-double
// precision floating point arithmetic", 2001) one level down.
// The _rn intrinsics keep the compiler from contracting or reassociating the
// error-free transformations.
#pragma once
#include <cuda_runtime.h>

#include "pnamp_device.cuh"

namespace pnamp {

struct dd {
    float hi, lo;
};

__device__ __forceinline__ dd dd_make(float h, float l) {
    dd r;
    r.hi = h;
    r.lo = l;
    return r;
}
__device__ __forceinline__ dd two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float v = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v));
    return dd_make(s, e);
}
// requires |a| >= |b| (or a == 0)
__device__ __forceinline__ dd quick_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return dd_make(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
    const dd s = two_sum(a.hi, b.hi);
    return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ dd dd_neg(dd a) { return dd_make(-a.hi, -a.lo); }
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return quick_two_sum(p, e);
}
// a * b + c
__device__ __forceinline__ dd dd_fma(dd a, dd b, dd c) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    const dd s = two_sum(p, c.hi);
    return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(e, c.lo)));
}
// 1 / b: float reciprocal refined by one Newton step with a double-float residual
__device__ __forceinline__ dd dd_recip(dd b) {
    const float q = __frcp_rn(b.hi);
    const dd r = dd_fma(dd_neg(b), dd_make(q, 0.0f), dd_make(1.0f, 0.0f));
    return quick_two_sum(q, __fmul_rn(r.hi, q));
}
__device__ __forceinline__ dd dd_from(double x) {
    const float h = __double2float_rn(x);
    return dd_make(h, __double2float_rn(x - (double)h));
}
__device__ __forceinline__ double dd_to(dd a) { return (double)a.hi + (double)a.lo; }

// ------------------------------------------------------------------ packed pairs
// Two floats in one 64-bit register pair, one add / mul / fma.f32x2 for both. The FP32 pipe
// does the same 128 lane operations per cycle and SM either way (measured: 113-121 per cycle
// scalar and packed), but a packed instruction takes one issue slot for two of them, and the
// double-float kernels are issue-bound (an error-free sum is six operations around one load).
struct f2 {
    unsigned long long u;
};
__device__ __forceinline__ f2 f2_make(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 f2_dup(float a) { return f2_make(a, a); }
__device__ __forceinline__ float f2_a(f2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v.u));
    return a;
}
__device__ __forceinline__ float f2_b(f2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v.u));
    return b;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
    return r;
}
__device__ __forceinline__ f2 f2_neg(f2 a) { return f2_make(-f2_a(a), -f2_b(a)); }
__device__ __forceinline__ f2 f2_swap(f2 a) { return f2_make(f2_b(a), f2_a(a)); }

// A pair of double-floats and the operations above on both at once.
struct dd2 {
    f2 hi, lo;
};
__device__ __forceinline__ dd2 two_sum(f2 a, f2 b) {
    const f2 s = f2_add(a, b);
    const f2 v = f2_sub(s, a);
    return {s, f2_add(f2_sub(a, f2_sub(s, v)), f2_sub(b, v))};
}
__device__ __forceinline__ dd2 quick_two_sum(f2 a, f2 b) {
    const f2 s = f2_add(a, b);
    return {s, f2_sub(b, f2_sub(s, a))};
}
__device__ __forceinline__ dd2 dd2_add(dd2 a, dd2 b) {
    const dd2 s = two_sum(a.hi, b.hi);
    return quick_two_sum(s.hi, f2_add(s.lo, f2_add(a.lo, b.lo)));
}
__device__ __forceinline__ dd2 dd2_mul(dd2 a, dd2 b) {
    const f2 p = f2_mul(a.hi, b.hi);
    f2 e = f2_fma(a.hi, b.hi, f2_neg(p));
    e = f2_fma(a.hi, b.lo, e);
    e = f2_fma(a.lo, b.hi, e);
    return quick_two_sum(p, e);
}
__device__ __forceinline__ dd2 dd2_fma(dd2 a, dd2 b, dd2 c) {
    const f2 p = f2_mul(a.hi, b.hi);
    f2 e = f2_fma(a.hi, b.hi, f2_neg(p));
    e = f2_fma(a.hi, b.lo, e);
    e = f2_fma(a.lo, b.hi, e);
    const dd2 s = two_sum(p, c.hi);
    return quick_two_sum(s.hi, f2_add(s.lo, f2_add(e, c.lo)));
}

// ------------------------------------------------------------------ complex
// real and imaginary part side by side: (re, im) high words, then (re, im) low words
struct __align__(16) zd {
    f2 hi, lo;
};
__device__ __forceinline__ dd re(zd a) { return dd_make(f2_a(a.hi), f2_a(a.lo)); }
__device__ __forceinline__ dd im(zd a) { return dd_make(f2_b(a.hi), f2_b(a.lo)); }
__device__ __forceinline__ double re(zc a) { return a.x; }
__device__ __forceinline__ double im(zc a) { return a.y; }
__device__ __forceinline__ zd mkd(dd a, dd b) { return {f2_make(a.hi, b.hi), f2_make(a.lo, b.lo)}; }
__device__ __forceinline__ zd as_zd(dd2 a) { return {a.hi, a.lo}; }
__device__ __forceinline__ dd2 pair_of(zd a) { return {a.hi, a.lo}; }
__device__ __forceinline__ dd2 dup(dd a) { return {f2_dup(a.hi), f2_dup(a.lo)}; }
__device__ __forceinline__ dd2 alt(dd a) { return {f2_make(-a.hi, a.hi), f2_make(-a.lo, a.lo)}; }      // (-a, a)
__device__ __forceinline__ dd2 alt_neg(dd a) { return {f2_make(a.hi, -a.hi), f2_make(a.lo, -a.lo)}; }  // (a, -a)
__device__ __forceinline__ dd2 swapped(zd a) { return {f2_swap(a.hi), f2_swap(a.lo)}; }                // (im, re)
__device__ __forceinline__ zd operator+(zd a, zd b) { return as_zd(dd2_add(pair_of(a), pair_of(b))); }
__device__ __forceinline__ zd operator-(zd a) { return {f2_neg(a.hi), f2_neg(a.lo)}; }
__device__ __forceinline__ zd operator-(zd a, zd b) { return a + (-b); }
// (a.x b.x - a.y b.y, a.x b.y + a.y b.x)
__device__ __forceinline__ zd operator*(zd a, zd b) {
    const dd2 t = dd2_mul(alt(im(a)), swapped(b));
    return as_zd(dd2_fma(dup(re(a)), pair_of(b), t));
}
__device__ __forceinline__ zd operator*(dd s, zd a) { return as_zd(dd2_mul(dup(s), pair_of(a))); }
__device__ __forceinline__ zd zconj(zd a) { return mkd(re(a), dd_neg(im(a))); }
// c + a*b
__device__ __forceinline__ zd zfma(zd a, zd b, zd c) {
    const dd2 t = dd2_fma(alt(im(a)), swapped(b), pair_of(c));
    return as_zd(dd2_fma(dup(re(a)), pair_of(b), t));
}
// c - a*b
__device__ __forceinline__ zd zfms(zd a, zd b, zd c) {
    const dd2 t = dd2_fma(alt_neg(im(a)), swapped(b), pair_of(c));
    return as_zd(dd2_fma(dup(dd_neg(re(a))), pair_of(b), t));
}
// c + r*a, r real
__device__ __forceinline__ zd rfma(dd r, zd a, zd c) { return as_zd(dd2_fma(dup(r), pair_of(a), pair_of(c))); }
__device__ __forceinline__ zd zrecip(zd b) {
    const dd bx = re(b), by = im(b);
    const dd n2 = dd_fma(bx, bx, dd_mul(by, by));
    const dd inv = dd_recip(n2);
    return mkd(dd_mul(bx, inv), dd_neg(dd_mul(by, inv)));
}
__device__ __forceinline__ bool zfinite(zd a) { return isfinite(f2_a(a.hi)) && isfinite(f2_b(a.hi)); }
__device__ __forceinline__ zd zd_from(zc a) { return mkd(dd_from(a.x), dd_from(a.y)); }
__device__ __forceinline__ zc zd_to(zd a) { return mk(dd_to(re(a)), dd_to(im(a))); }

}  // namespace pnamp
