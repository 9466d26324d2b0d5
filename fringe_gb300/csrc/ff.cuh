// ff.cuh -- float-float arithmetic: an unevaluated sum of two floats, about 46
// significant bits, on the FP32 pipe.
//
// FP64 issues two operations per SM and clock on this part; a float-float
// multiply-add is 15 FP32 instructions, of which an SM issues 128 lanes per
// clock: four to six times the rate.  The operations are Dekker's and Knuth's
// error-free sums and products with the low parts added in (relative errors of
// a few 2^-47 of the larger operand); every step is an explicit intrinsic, so that no
// contraction changes it.  The type takes double's place in the pixel solver's templates;
// its functions are found by argument-dependent lookup.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace fpl_ff {

struct ff {
    float h, l;
    __device__ __forceinline__ ff() {}
    __device__ __forceinline__ explicit ff(float a) : h(a), l(0.f) {}
    __device__ __forceinline__ explicit ff(int a) : h((float)a), l(0.f) {}      // |a| < 2^24
    __device__ __forceinline__ explicit ff(double a) : h((float)a), l((float)(a - (double)(float)a)) {}
    __device__ __forceinline__ ff(float a, float b) : h(a), l(b) {}
    __device__ __forceinline__ explicit operator float() const { return h; }
};

// (s, e) with |e| small against s, renormalised
__device__ __forceinline__ ff quick(float s, float e)
{
    const float h = __fadd_rn(s, e);
    return ff(h, __fsub_rn(e, __fsub_rn(h, s)));
}
// s = a + b and its rounding error
__device__ __forceinline__ float two_sum(float a, float b, float &e)
{
    const float s = __fadd_rn(a, b), v = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v));
    return s;
}
__device__ __forceinline__ float rcp1(float a)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

__device__ __forceinline__ ff operator-(ff a) { return ff(-a.h, -a.l); }
__device__ __forceinline__ ff operator+(ff a, ff b)
{
    float e;
    const float s = two_sum(a.h, b.h, e);
    return quick(s, __fadd_rn(e, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ ff operator-(ff a, ff b) { return a + (-b); }
__device__ __forceinline__ ff operator*(ff a, ff b)
{
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return quick(p, e);
}
__device__ __forceinline__ ff fma(ff a, ff b, ff c)
{
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p), t;
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    const float s = two_sum(p, c.h, t);
    return quick(s, __fadd_rn(t, __fadd_rn(e, c.l)));
}
__device__ __forceinline__ ff operator/(ff a, ff b)
{
    const float r = rcp1(b.h), q = __fmul_rn(a.h, r);
    const ff d = fma(ff(-q), b, a);                     // a - q b
    const float q2 = __fmul_rn(d.h, r);
    const ff d2 = fma(ff(-q2), b, d);
    const ff s = quick(q, q2);
    return s + ff(__fmul_rn(d2.h, r));
}
__device__ __forceinline__ ff &operator+=(ff &a, ff b) { return a = a + b; }
__device__ __forceinline__ ff &operator-=(ff &a, ff b) { return a = a - b; }
__device__ __forceinline__ ff &operator*=(ff &a, ff b) { return a = a * b; }

__device__ __forceinline__ bool operator<(ff a, ff b) { return a.h < b.h || (a.h == b.h && a.l < b.l); }
__device__ __forceinline__ bool operator>(ff a, ff b) { return b < a; }
__device__ __forceinline__ bool operator<=(ff a, ff b) { return a.h < b.h || (a.h == b.h && a.l <= b.l); }
__device__ __forceinline__ bool operator>=(ff a, ff b) { return b <= a; }
__device__ __forceinline__ bool operator==(ff a, ff b) { return a.h == b.h && a.l == b.l; }
__device__ __forceinline__ bool operator!=(ff a, ff b) { return !(a == b); }

__device__ __forceinline__ ff abs(ff a) { return a.h < 0.f ? -a : a; }
__device__ __forceinline__ ff max(ff a, ff b) { return a < b ? b : a; }
__device__ __forceinline__ ff min(ff a, ff b) { return b < a ? b : a; }
__device__ __forceinline__ bool isfinite(ff a) { return ::isfinite(a.h); }
__device__ __forceinline__ ff sqrt(ff a)
{
    if (!(a.h > 0.f)) return ff(sqrtf(a.h));            // 0, negative, NaN as sqrtf
    const float x = rsqrtf(a.h), s = __fmul_rn(a.h, x);
    const ff d = fma(ff(-s), ff(s), a);                 // a - s^2
    const ff r = quick(s, __fmul_rn(d.h, __fmul_rn(0.5f, x)));
    const ff d2 = fma(-r, r, a);
    return r + ff(__fmul_rn(d2.h, __fmul_rn(0.5f, x)));
}
// 1 / sqrt(a), a > 0: one Newton step on the FP32 value
__device__ __forceinline__ ff rsqrt_t(ff a)
{
    const float y = rsqrtf(a.h);
    const ff d = fma(a * ff(y), ff(-y), ff(1.f));       // 1 - a y^2
    return ff(y) + d * ff(__fmul_rn(0.5f, y)) + ff(__fmul_rn(__fmul_rn(0.375f, y), __fmul_rn(d.h, d.h)));
}
__device__ __forceinline__ ff fdiv_fast(ff a, ff b) { return a / b; }

__device__ __forceinline__ ff __shfl_sync(unsigned m, ff v, int src)
{
    return ff(::__shfl_sync(m, v.h, src), ::__shfl_sync(m, v.l, src));
}
__device__ __forceinline__ ff __shfl_xor_sync(unsigned m, ff v, int o)
{
    return ff(::__shfl_xor_sync(m, v.h, o), ::__shfl_xor_sync(m, v.l, o));
}

}  // namespace fpl_ff
