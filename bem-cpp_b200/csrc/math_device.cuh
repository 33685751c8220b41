// Elementary functions of the quadrature kernels without the branches of
// CUDA's: those, for large arguments and special values, keep the compiler
// from interleaving the independent evaluations of a quadrature loop, and the
// kernels are bound by the latency of these chains at 8 to 16 warps per SM.
// bem_selftest_math evaluates each beside CUDA's function; the tests hold
// their errors against exact values and against CUDA's.
#pragma once
#include <cuda_runtime.h>

namespace bem {

// sin and cos for |x| below SINCOS_MAX.  Argument reduction in the two parts
// of Cody and Waite: n = round(2 x / pi), x - n pi/2 in two fused steps, the
// first of them exact (both operands are multiples of the remainder's last
// place), the second with its rounding kept, r + rl.  On [-pi/4, pi/4] the
// polynomials sin r = r + r^3 p(r^2) and cos r = 1 - r^2/2 + r^4 q(r^2), p and q
// of degree 5 with the least largest error (Remez exchange, in 60 digits):
// 1.6e-18 and 5e-20; rl enters to first order.  Then the quadrant's exchange
// and signs.  Largest error measured 1.12 (sin) and 1.10 (cos) of 2^-53,
// CUDA's functions 1.15 on the same arguments; without rl, which is three
// of the 24 operations, 1.29.
constexpr double SINCOS_MAX = 1048576.0;
__device__ __forceinline__ void sincos_bounded(double x, double* sn, double* cs) {
    const double shift = 6755399441055744.0;  // 1.5 * 2^52: the sum's low bits are the rounded integer
    const double t = __fma_rn(x, 0.63661977236758134308, shift);
    const int n = __double2loint(t);
    const double fn = t - shift;
    const double r1 = __fma_rn(-fn, 1.5707963267948965580, x);
    const double r = __fma_rn(-fn, 6.1232339957367660359e-17, r1);
    const double rl = __fma_rn(-fn, 6.1232339957367660359e-17, r1 - r);
    const double z = r * r;
    double p = __fma_rn(z, 1.5888585349551085e-10, -2.5050600226854755e-08);
    p = __fma_rn(z, p, 2.7557312544683082e-06);
    p = __fma_rn(z, p, -0.00019841269825933777);
    p = __fma_rn(z, p, 0.00833333333331648);
    p = __fma_rn(z, p, -0.166666666666666);
    const double s = r + __fma_rn(r * z, p, rl);
    double q = __fma_rn(z, -1.1359669571037437e-11, 2.087572367861325e-09);
    q = __fma_rn(z, q, -2.7557314355197716e-07);
    q = __fma_rn(z, q, 2.4801587289491668e-05);
    q = __fma_rn(z, q, -0.0013888888888874138);
    q = __fma_rn(z, q, 0.0416666666666666);
    const double c = 1.0 + __fma_rn(z, __fma_rn(z, q, -0.5), -(r * rl));
    const double a = (n & 1) ? c : s, b = (n & 1) ? s : c;
    *sn = __hiloint2double(__double2hiint(a) ^ (int)((unsigned)(n & 2) << 30), __double2loint(a));
    *cs = __hiloint2double(__double2hiint(b) ^ (int)((unsigned)((n + 1) & 2) << 30), __double2loint(b));
}

// e^-x without a branch, x clamped to [-708, 708] (e^-0 = 1 exactly; below
// e^-708 the value does not count, above e^708 the callers do not come): x = -(n ln 2 + r), |r| <= ln 2 / 2, in two fused
// steps (Cody and Waite's reduction), the Taylor polynomial of degree 13 (first
// omitted term below 5e-18) and 2^n added to the exponent.  Largest relative
// error measured 1.24 of 2^-53, CUDA's exp 1.24 on the same arguments.
__device__ __forceinline__ double exp_decay_bounded(double x) {
    x = fmin(fmax(x, -708.0), 708.0);
    const double shift = 6755399441055744.0;
    const double t = __fma_rn(x, -1.4426950408889634074, shift);
    const double fn = t - shift;
    double r = __fma_rn(fn, -0.69314718055994530942, -x);
    r = __fma_rn(fn, -2.3190468138462995585e-17, r);
    double p = __fma_rn(r, 1.0 / 6227020800.0, 1.0 / 479001600.0);
    p = __fma_rn(r, p, 1.0 / 39916800.0);
    p = __fma_rn(r, p, 1.0 / 3628800.0);
    p = __fma_rn(r, p, 1.0 / 362880.0);
    p = __fma_rn(r, p, 1.0 / 40320.0);
    p = __fma_rn(r, p, 1.0 / 5040.0);
    p = __fma_rn(r, p, 1.0 / 720.0);
    p = __fma_rn(r, p, 1.0 / 120.0);
    p = __fma_rn(r, p, 1.0 / 24.0);
    p = __fma_rn(r, p, 1.0 / 6.0);
    p = __fma_rn(r, p, 0.5);
    p = __fma_rn(r, p, 1.0);
    p = __fma_rn(r, p, 1.0);
    return __hiloint2double(__double2hiint(p) + (int)((unsigned)__double2loint(t) << 20), __double2loint(p));
}

// 1 / sqrt(x) for a normal x > 0: the hardware's approximation y (about 2^-20,
// its lower 32 bits zero, so y^2 is exact) and one step of third order, y (1 +
// e / 2 + 3 e^2 / 8) with e = 1 - x y^2, the binomial series of (1 - e)^(-1/2).
// Largest relative error measured 1.01 of 2^-53, CUDA's rsqrt the same;
// 1.24 with x y rounded before the second product.
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x, y * y, 1.0);
    return __fma_rn(y * e, __fma_rn(e, 0.375, 0.5), y);
}

// 1 / p of a pivot, conj(p) / |p|^2, without the divisions' branches (~100
// cycles of every panel column): the hardware's approximation of 1 / |p|^2 (about
// 2^-20), two Newton steps, and each quotient corrected once by its remainder
// (Markstein), which rounds it as a division does: no difference in 2e6
// random pivots, against one in four without the correction.  Divisions where |p|^2 leaves the approximation's range.
__device__ __forceinline__ double2 pivot_recip(double2 p) {
    const double den = p.x * p.x + p.y * p.y;
    if (!(den > 1e-290 && den < 1e290)) return make_double2(p.x / den, -p.y / den);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
    y = __fma_rn(y, __fma_rn(-den, y, 1.0), y);
    y = __fma_rn(y, __fma_rn(-den, y, 1.0), y);
    double re = p.x * y, im = p.y * y;
    re = __fma_rn(__fma_rn(-den, re, p.x), y, re);
    im = __fma_rn(__fma_rn(-den, im, p.y), y, im);
    return make_double2(re, -im);
}

}  // namespace bem
