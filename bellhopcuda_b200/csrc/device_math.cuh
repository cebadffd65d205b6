// Small device math helpers: 2-vectors and complex numbers in the bulk real
// type R (float in the mixed-precision tracer, double in the FP64 tracer).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace bhcb {

template<typename T> struct V2 {
    T x, y;
};
template<typename T> __device__ __forceinline__ V2<T> mk2(T x, T y) { return V2<T>{x, y}; }
template<typename T> __device__ __forceinline__ V2<T> add2(V2<T> a, V2<T> b) { return {a.x + b.x, a.y + b.y}; }
template<typename T> __device__ __forceinline__ V2<T> sub2(V2<T> a, V2<T> b) { return {a.x - b.x, a.y - b.y}; }
template<typename T> __device__ __forceinline__ V2<T> scl2(T s, V2<T> a) { return {s * a.x, s * a.y}; }
template<typename T> __device__ __forceinline__ V2<T> div2(V2<T> a, T s) { return {a.x / s, a.y / s}; }
template<typename T> __device__ __forceinline__ T dot2(V2<T> a, V2<T> b) { return a.x * b.x + a.y * b.y; }
template<typename T, typename U> __device__ __forceinline__ V2<T> cvt2(V2<U> a)
{
    return {(T)a.x, (T)a.y};
}

template<typename T> struct Cx {
    T r, i;
};
template<typename T> __device__ __forceinline__ Cx<T> cx(T r, T i) { return Cx<T>{r, i}; }
template<typename T> __device__ __forceinline__ Cx<T> cadd(Cx<T> a, Cx<T> b) { return {a.r + b.r, a.i + b.i}; }
template<typename T> __device__ __forceinline__ Cx<T> csub(Cx<T> a, Cx<T> b) { return {a.r - b.r, a.i - b.i}; }
template<typename T> __device__ __forceinline__ Cx<T> cmul(Cx<T> a, Cx<T> b)
{
    return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r};
}
template<typename T> __device__ __forceinline__ Cx<T> cscl(T s, Cx<T> a) { return {s * a.r, s * a.i}; }
// complex division by Smith's method (scales by the larger component, exact
// for a purely real divisor)
template<typename T> __device__ __forceinline__ Cx<T> cdiv(Cx<T> a, Cx<T> b)
{
    if(fabs(b.r) >= fabs(b.i)) {
        T rat = b.i / b.r, den = b.r + b.i * rat;
        return {(a.r + a.i * rat) / den, (a.i - a.r * rat) / den};
    } else {
        T rat = b.r / b.i, den = b.r * rat + b.i;
        return {(a.r * rat + a.i) / den, (a.i * rat - a.r) / den};
    }
}
template<typename T> __device__ __forceinline__ Cx<T> rdivc(T a, Cx<T> b)
{
    return cdiv(Cx<T>{a, (T)0}, b);
}
template<typename T> __device__ __forceinline__ T cabs_(Cx<T> a) { return hypot(a.r, a.i); }
// principal square root
template<typename T> __device__ __forceinline__ Cx<T> csqrt_(Cx<T> z)
{
    T m = hypot(z.r, z.i);
    if(m == (T)0) return {(T)0, z.i};
    if(z.r >= (T)0) {
        T t = sqrt((m + z.r) * (T)0.5);
        return {t, z.i / (t + t)};
    }
    T t = sqrt((m - z.r) * (T)0.5);
    return {fabs(z.i) / (t + t), copysign(t, z.i)};
}

// Hardware approximations (PTX .approx.ftz forms) for the mixed-precision
// contribution math; arguments of sin/cos are range-reduced by the caller.
__device__ __forceinline__ float ex2_ftz(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_ftz(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sin_ftz(float x)
{
    float y;
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float cos_ftz(float x)
{
    float y;
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Correctly rounded FP64 reciprocal, quotient and square root without the branch to
// a slow path that `/` and sqrt() carry, so that independent ones overlap and one
// reciprocal serves several quotients (a dependent `/` takes 115 cycles on B200, a
// sqrt 80, a DFMA 8; the tracers are one dependent chain per ray). Newton's iteration
// on the hardware estimate, then Markstein's residual correction with fused
// multiply-adds (P. Markstein, IBM J. Res. Dev. 34, 1990; Cornea, Harrison and Tang,
// IEEE Trans. Comput. 2002): the last correction rounds the exact residual once. For
// finite operands with |b|, |a| and the result between 2^-900 and 2^900 (a = 0
// allowed, infinities and NaN not); the callers' divisors are sound speeds, step
// lengths and direction components that they have checked.
//
// The correction of a quotient needs the correctly rounded reciprocal: with one an ulp
// off, four in ten of the quotients nearest to a midpoint between doubles come out
// wrong. A last Newton step yields (1 - e^2) / b, e the error before it: below 1 / b,
// and so wrong if 1 / b lies above a midpoint by less than e^2 and y is the double
// below (b all ones, where the rounding has a tie). The step before rounds up, so y is
// then the double above, half an ulp off, and 1 / b, at least 2^-106 of itself above
// the midpoint, is rounded to it.
//
// For b > 0. Of a negative b all ones (1.99... to the last bit) the reciprocal, and with
// it one of the quotients next to a midpoint, is the double beside: taking the sign
// aside, as rcp_signed does, would lengthen the tracers' chain by 2 %.
__device__ __forceinline__ double rcp_est(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
}
__device__ __forceinline__ double rcp_rn(double b)
{
    double y = rcp_est(b);
    double e = fma(-b, y, 1.0);
    y = __fma_ru(y, fma(e, e, e), y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}
__device__ __forceinline__ double rcp_signed(double b) { return copysign(rcp_rn(fabs(b)), b); }
// 1 / bsq, bsq = b * b rounded and y = rcp_rn(b). y * y is up to two ulps off, after
// which one step alone misses six mantissas of b (those whose bsq times an odd 54-bit
// integer is next to a power of two).
__device__ __forceinline__ double rcp_square(double bsq, double y)
{
    double z = y * y;
    z = __fma_ru(z, fma(-bsq, z, 1.0), z);
    return fma(z, fma(-bsq, z, 1.0), z);
}
// a / b given y, the correctly rounded 1 / b
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ double div_rn(double a, double b) { return quot_rn(a, b, rcp_rn(b)); }
// a >= 2^-900 (0 is the caller's to exclude)
__device__ __forceinline__ double sqrt_rn(double a)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double g = a * y, h = 0.5 * y;
    double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    return fma(fma(-g, g, a), h, g);
}

// sqrt(a) of any a; the square of a spreading that has grown without bound is infinite
__device__ __forceinline__ double sqrt_any(double a) { return a > 1.0e-270 && a < 1.0e270 ? sqrt_rn(a) : sqrt(a); }

// The exponents of a ray's p (2^961 or more) or q (infinite, NaN) are so large that the
// terms 0 q of an ocean without depth curvature, nothing in all other steps, are not
// numbers. p and q are of the step's start; q at half the step, q + h c p, can only
// overflow with such a p.
__device__ __forceinline__ int exponent_bits(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ bool past_numbers(int p_bits, int q_bits)
{
    return p_bits >= 0x7c000000 || q_bits >= 0x7ff00000;
}

// |nextafter(v, 0) - v| of a finite v: the bit pattern below v's magnitude
__device__ __forceinline__ double spacing_d(double v)
{
    const double a = fabs(v);
    return a > 0.0 ? a - __longlong_as_double(__double_as_longlong(a) - 1) : 0.0;
}

} // namespace bhcb
