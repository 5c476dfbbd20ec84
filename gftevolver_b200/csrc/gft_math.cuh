// gft_math.cuh -- elementary functions for the throughput kernels.
//
// Written with a two/three-term Cody-Waite reduction by pi (W. J. Cody,
// W. Waite, "Software Manual for the Elementary Functions", 1980):
// r = x - k*pi with k = rint(x/pi), |r| <= pi/2, then sin(x) = (-1)^k sin(r),
// cos(x) = (-1)^k cos(r).  On the reduced range:
//   float : minimax polynomials fitted for this library by the Remez exchange
//           (gft_math_fit.py regenerates them): sin r = r + r^3 P(r^2), degree 9,
//           relative error <= 6.1e-9; cos r = 1 + r^2 Q(r^2), degree 10, absolute
//           error <= 2.5e-10 -- both below float's rounding, and two multiply-adds
//           shorter each than the Taylor series of equal accuracy (degree 13 / 14);
//   double: the same forms by the same fit in extended precision, sin of degree 17
//           (relative error <= 2.8e-19), cos of degree 18 (absolute error <= 6.8e-21; one
//           degree less leaves no room for -1/2 to be exact, and its rounding counts at every
//           angle): three multiply-adds shorter each than the Taylor series of equal use.
// The reduction uses the 1.5*2^p rounding constant (no conversion to integer):
// it holds for |x| < 1.3e7 (float) / 1.4e15 (double); phases that large do not
// occur in the evolution (the step kernels flag |theta| > 1e4).
// asin: x + x^3 A(x^2), minimax for |x| <= 1/4 (float, relative error <= 5.5e-11)
// or 1/8 (double, <= 4.5e-19) -- the link update's argument is dt * E ~ 1e-3 to
// 1e-1 -- and CUDA's asin otherwise.
#pragma once

#include <cuda_runtime.h>

namespace gft {

// Double minimax coefficients on |r| <= pi/2 (gft_math_fit.py), sin r = r + r^3 P(r^2), cos r = 1 + r^2 Q(r^2).
#define GFT_S3 (-1.66666666666666656e-1)
#define GFT_S5 (8.33333333333319431e-3)
#define GFT_S7 (-1.98412698412092192e-4)
#define GFT_S9 (2.75573192111372807e-6)
#define GFT_S11 (-2.5052106872802643e-8)
#define GFT_S13 (1.6058939705911306e-10)
#define GFT_S15 (-7.64299148958033802e-13)
#define GFT_S17 (2.72117496446829863e-15)
#define GFT_C2 (-0.5)
#define GFT_C4 (4.1666666666666661e-2)
#define GFT_C6 (-1.38888888888885709e-3)
#define GFT_C8 (2.48015873014999769e-5)
#define GFT_C10 (-2.75573192104185647e-7)
#define GFT_C12 (2.08767557145721576e-9)
#define GFT_C14 (-1.14706719540102727e-11)
#define GFT_C16 (4.77690866610973073e-14)
#define GFT_C18 (-1.51229471791906704e-16)

// Float minimax coefficients on |r| <= pi/2 (gft_math_fit.py): sin r = r + r^3 P(r^2), cos r = 1 + r^2 Q(r^2).
#define GFT_FS3 (-0.16666659712791443f)
#define GFT_FS5 (0.00833306647837162f)
#define GFT_FS7 (-0.00019809602235909551f)
#define GFT_FS9 (2.605780537123792e-06f)
#define GFT_FC2 (-0.5f)
#define GFT_FC4 (0.04166664183139801f)
#define GFT_FC6 (-0.00138884037733078f)
#define GFT_FC8 (2.4761886379565112e-05f)
#define GFT_FC10 (-2.607710598567792e-07f)

__device__ __forceinline__ void sincos_poly(float r, float& s, float& c)
{
    const float r2 = r * r;
    float ps = GFT_FS9;
    ps = fmaf(ps, r2, GFT_FS7);
    ps = fmaf(ps, r2, GFT_FS5);
    ps = fmaf(ps, r2, GFT_FS3);
    s = fmaf(ps * r2, r, r);
    float pc = GFT_FC10;
    pc = fmaf(pc, r2, GFT_FC8);
    pc = fmaf(pc, r2, GFT_FC6);
    pc = fmaf(pc, r2, GFT_FC4);
    pc = fmaf(pc, r2, GFT_FC2);
    c = fmaf(pc, r2, 1.0f);
}

__device__ __forceinline__ float sin_poly(float r)
{
    const float r2 = r * r;
    float ps = GFT_FS9;
    ps = fmaf(ps, r2, GFT_FS7);
    ps = fmaf(ps, r2, GFT_FS5);
    ps = fmaf(ps, r2, GFT_FS3);
    return fmaf(ps * r2, r, r);
}

// x = k*pi + r: t = x/pi + 1.5*2^23 rounds x/pi to the integer k held in the
// low mantissa bits of t (valid while |x/pi| < 2^22, i.e. |x| < 1.3e7; the
// step kernels flag phases beyond 1e4 with GFT_W_RANGE); then
// r = x - k*PI_A - k*PI_B with PI_A = float(pi), PI_B = float(pi - PI_A).
// Returns r and the sign bit (-1)^k as an integer mask.
__device__ __forceinline__ float reduce_pi(float x, unsigned& sign)
{
    const float t = fmaf(x, 0.3183098861837907f, 12582912.0f);
    const float kf = t - 12582912.0f;
    sign = __float_as_uint(t) << 31;
    const float r = fmaf(-kf, 3.1415927410125732f, x);
    return fmaf(-kf, -8.742277657347586e-08f, r);
}

__device__ __forceinline__ float gsin(float x)
{
    unsigned sg;
    const float r = reduce_pi(x, sg);
    return __uint_as_float(__float_as_uint(sin_poly(r)) ^ sg);
}

__device__ __forceinline__ void gsincos(float x, float& s, float& c)
{
    unsigned sg;
    const float r = reduce_pi(x, sg);
    sincos_poly(r, s, c);
    s = __uint_as_float(__float_as_uint(s) ^ sg);
    c = __uint_as_float(__float_as_uint(c) ^ sg);
}

// Out-of-line wide-argument paths: taken only when |x| > 1/4 (asin) or c >= 1/64
// (sqrt), which the link update's small increments never reach; keeping them out
// of the inlined step body shortens the hot loop's code (measured 1-1.5 % faster).
static __device__ __noinline__ float gasin_wide(float x) { return asinf(x); }
static __device__ __noinline__ double gasin_wide(double x) { return asin(x); }
static __device__ __noinline__ float sqrt1m_wide(float c) { return -c / (1.0f + sqrtf(1.0f - c)); }
static __device__ __noinline__ double sqrt1m_wide(double c) { return -c / (1.0 + sqrt(1.0 - c)); }

// Where the series below serve, per compute type.
template <class C>
struct AsinSeries;
template <>
struct AsinSeries<float> {
    static constexpr float limit = 0.25f;
};
template <>
struct AsinSeries<double> {
    static constexpr double limit = 0.125;
};
template <class C>
struct Sqrt1mSeries;
template <>
struct Sqrt1mSeries<float> {
    static constexpr float limit = 0.015625f;
};
template <>
struct Sqrt1mSeries<double> {
    static constexpr double limit = 0.015625;
};

__device__ __forceinline__ float asin_series(float x)
{
    const float x2 = x * x;
    float p = 3.40801214445308396e-2f;
    p = fmaf(p, x2, 4.4443265213162178e-2f);
    p = fmaf(p, x2, 7.50041907289998445e-2f);
    p = fmaf(p, x2, 1.6666663944730844e-1f);
    return fmaf(p * x2, x, x);
}
__device__ __forceinline__ float gasin(float x)
{
    return fabsf(x) > AsinSeries<float>::limit ? gasin_wide(x) : asin_series(x);
}

// ---- double ----------------------------------------------------------------
__device__ __forceinline__ void sincos_poly(double r, double& s, double& c)
{
    const double r2 = r * r;
    double ps = GFT_S17;
    ps = fma(ps, r2, GFT_S15);
    ps = fma(ps, r2, GFT_S13);
    ps = fma(ps, r2, GFT_S11);
    ps = fma(ps, r2, GFT_S9);
    ps = fma(ps, r2, GFT_S7);
    ps = fma(ps, r2, GFT_S5);
    ps = fma(ps, r2, GFT_S3);
    s = fma(ps * r2, r, r);
    double pc = GFT_C18;
    pc = fma(pc, r2, GFT_C16);
    pc = fma(pc, r2, GFT_C14);
    pc = fma(pc, r2, GFT_C12);
    pc = fma(pc, r2, GFT_C10);
    pc = fma(pc, r2, GFT_C8);
    pc = fma(pc, r2, GFT_C6);
    pc = fma(pc, r2, GFT_C4);
    pc = fma(pc, r2, GFT_C2);
    c = fma(pc, r2, 1.0);
}

__device__ __forceinline__ double sin_poly(double r)
{
    const double r2 = r * r;
    double ps = GFT_S17;
    ps = fma(ps, r2, GFT_S15);
    ps = fma(ps, r2, GFT_S13);
    ps = fma(ps, r2, GFT_S11);
    ps = fma(ps, r2, GFT_S9);
    ps = fma(ps, r2, GFT_S7);
    ps = fma(ps, r2, GFT_S5);
    ps = fma(ps, r2, GFT_S3);
    return fma(ps * r2, r, r);
}

// As for float, with t = x/pi + 1.5*2^52 (valid while |x| < 1.4e15) and
// pi = PI_A + PI_B + PI_C, each the double nearest to the remainder; with FMA
// each step rounds once, so r carries a relative error of ~1 ulp, next to a multiple
// of pi too: there r is as small as 1e-18 and without PI_C off by 7e-14 of itself.
__device__ __forceinline__ double reduce_pi(double x, unsigned long long& sign)
{
    const double t = fma(x, 0.3183098861837907, 6755399441055744.0);
    const double kd = t - 6755399441055744.0;
    sign = (unsigned long long)__double_as_longlong(t) << 63;
    double r = fma(-kd, 3.141592653589793, x);
    r = fma(-kd, 1.2246467991473532e-16, r);
    return fma(-kd, -2.9947698097183397e-33, r);
}

__device__ __forceinline__ double gsin(double x)
{
    unsigned long long sg;
    const double r = reduce_pi(x, sg);
    return __longlong_as_double(__double_as_longlong(sin_poly(r)) ^ (long long)sg);
}

__device__ __forceinline__ void gsincos(double x, double& s, double& c)
{
    unsigned long long sg;
    const double r = reduce_pi(x, sg);
    sincos_poly(r, s, c);
    s = __longlong_as_double(__double_as_longlong(s) ^ (long long)sg);
    c = __longlong_as_double(__double_as_longlong(c) ^ (long long)sg);
}

__device__ __forceinline__ double asin_series(double x)
{
    const double x2 = x * x;
    double p = 1.81280312314050132e-2;
    p = fma(p, x2, 2.23556390763832123e-2);
    p = fma(p, x2, 3.03821168203033322e-2);
    p = fma(p, x2, 4.4642856235161617e-2);
    p = fma(p, x2, 7.50000000021955577e-2);
    p = fma(p, x2, 1.66666666666664899e-1);
    return fma(p * x2, x, x);
}
__device__ __forceinline__ double gasin(double x)
{
    return fabs(x) > AsinSeries<double>::limit ? gasin_wide(x) : asin_series(x);
}

// sqrt(1 - c) - 1 for the link update's |c|^2 = c (tiny in practice): -c/2 + c^2 G(c), minimax for c
// <= 1/64 (relative error <= 1.2e-8 float, 8.4e-19 double), else the exact -c / (1 + sqrt(1 - c)).
// The sum rounds once, so float's 7.2e-8 and double's 1.14e-16 in all are below those of c times a
// rounded factor (1.2e-7, 2.2e-16).  The limit covers links that turn by up to 0.125 a step; a double
// series to 1/8192 sent fields at equilibrium (dt E ~ 0.015 per component) to the square root and division.
__device__ __forceinline__ float sqrt1m_series(float c)
{
    return fmaf(c * c, fmaf(c, -6.33604442620192054e-2f, -1.24995822362758278e-1f), -0.5f * c);
}
__device__ __forceinline__ double sqrt1m_series(double c)
{
    double g = -1.68402103550365345e-2;
    g = fma(g, c, -2.04923222794776193e-2);
    g = fma(g, c, -2.7343911625824167e-2);
    g = fma(g, c, -3.90624991489605221e-2);
    g = fma(g, c, -6.25000000020583453e-2);
    g = fma(g, c, -1.24999999999998343e-1);
    return fma(c * c, g, -0.5 * c);
}
template <class C>
__device__ __forceinline__ C sqrt1m_minus1(C c)
{
    return c < Sqrt1mSeries<C>::limit ? sqrt1m_series(c) : sqrt1m_wide(c);
}

// The largest magnitude of several values against a limit.  In FP64 by the words that hold the
// exponents, as integers: a comparison of doubles takes the FP64 pipe.  A NaN does not exceed
// (float; the series pass it on) or does (double).
template <class C>
struct MaxAbs;
template <>
struct MaxAbs<float> {
    float m = 0.0f;
    __device__ __forceinline__ void add(float x) { m = fmaxf(m, fabsf(x)); }
    __device__ __forceinline__ bool exceeds(float limit) const { return m > limit; }
};
template <>
struct MaxAbs<double> {
    unsigned m = 0u;
    __device__ __forceinline__ void add(double x) { m = max(m, (unsigned)__double2hiint(x) & 0x7fffffffu); }
    // true from the first value with the high word of `limit` on
    __device__ __forceinline__ bool exceeds(double limit) const { return m >= (unsigned)__double2hiint(limit); }
};

// 1/sqrt(s) and 1/d for arguments of order one: the hardware approximations
// (rsqrt.approx, rcp.approx; relative error below 2^-22) refined by one
// Newton-Raphson step each, r <- r (3 - s r^2) / 2 and q <- q (2 - d q), which
// squares that error; the results are within about one ulp of the rounded
// quotients.
__device__ __forceinline__ float rsqrt_nr(float s)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    return r * fmaf(-0.5f * s * r, r, 1.5f);
}
__device__ __forceinline__ float rcp_nr(float d)
{
    float q;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(d));
    return q * fmaf(-d, q, 2.0f);
}

// 1 - a0/|a| of a quaternion with scalar part w and |vector part|^2 = v2,
// without cancellation: v2 / (|a| (|a| + w)) = v2 r^2 / (1 + w r) when w >= 0
// (r = 1/|a|), else 1 - w r.  Float form of the energy terms' plaquette and
// electric traces; a few ulp of the same expression evaluated with IEEE
// square root and division (checked by gft_selftest_math).
__device__ __forceinline__ float one_minus_cos_nr(float w, float v2)
{
    const float r = rsqrt_nr(fmaf(w, w, v2));
    const float c = w * r;
    return (w >= 0.0f) ? v2 * r * r * rcp_nr(1.0f + c) : 1.0f - c;
}

}  // namespace gft
