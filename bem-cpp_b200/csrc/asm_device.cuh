// Device helpers shared by the assembly kernels (assembly.cu) and the
// shape-gradient kernels (grad_geom.cu): complex arithmetic, the Green's
// function pieces and the Graglia singular integrals.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

namespace bem {

#define INV4PI_D 0.079577471545947667884

// ------------------------------------------------------------ complex helpers
struct cplx {
    double re, im;
};
__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

struct Medium {
    double kr, ki;  // k = kr + i ki
};

// sin and cos without a branch, for |x| below SINCOS_MAX: n = round(2 x / pi),
// the remainder x - n pi/2 in two fused steps (the first is exact: both
// operands are multiples of the remainder's last place), the Taylor
// polynomials of degree 15 and 16 on [-pi/4, pi/4] (their first omitted terms
// are below 5e-17 and 3e-18) and the quadrant's exchange and signs.  Within
// 2e-16 of the exact values (tests).  The library's function takes a branch
// for large arguments at every call, which keeps the compiler from
// interleaving the independent evaluations of a quadrature loop: the kernels
// here are bound by the latency of these chains at 8 to 16 warps per SM.
constexpr double SINCOS_MAX = 1048576.0;
__device__ __forceinline__ void sincos_bounded(double x, double* sn, double* cs) {
    const double shift = 6755399441055744.0;  // 1.5 * 2^52: the sum's low bits are the rounded integer
    const double t = __fma_rn(x, 0.63661977236758134308, shift);
    const int n = __double2loint(t);
    const double fn = t - shift;
    double r = __fma_rn(-fn, 1.5707963267948965580, x);
    r = __fma_rn(-fn, 6.1232339957367660359e-17, r);
    const double z = r * r;
    double p = __fma_rn(z, -1.0 / 1307674368000.0, 1.0 / 6227020800.0);
    p = __fma_rn(z, p, -1.0 / 39916800.0);
    p = __fma_rn(z, p, 1.0 / 362880.0);
    p = __fma_rn(z, p, -1.0 / 5040.0);
    p = __fma_rn(z, p, 1.0 / 120.0);
    p = __fma_rn(z, p, -1.0 / 6.0);
    const double s = __fma_rn(r * z, p, r);
    double q = __fma_rn(z, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
    q = __fma_rn(z, q, 1.0 / 479001600.0);
    q = __fma_rn(z, q, -1.0 / 3628800.0);
    q = __fma_rn(z, q, 1.0 / 40320.0);
    q = __fma_rn(z, q, -1.0 / 720.0);
    q = __fma_rn(z, q, 1.0 / 24.0);
    q = __fma_rn(z, q, -0.5);
    const double c = __fma_rn(z, q, 1.0);
    const double a = (n & 1) ? c : s, b = (n & 1) ? s : c;
    *sn = __hiloint2double(__double2hiint(a) ^ (int)((unsigned)(n & 2) << 30), __double2loint(a));
    *cs = __hiloint2double(__double2hiint(b) ^ (int)((unsigned)((n + 1) & 2) << 30), __double2loint(b));
}

// e^-x for x >= 0.  Below 2^-54 the correctly rounded value is exactly 1;
// the literal G_smooth at coincident points (R_s = 1e-15) subtracts
// 1/(4 pi R_s) from e^-x cos(k R_s)/(4 pi R_s), so one unit in the last
// place of e^-x there would become 0.0156 in G.
__device__ __forceinline__ double exp_decay(double x) { return x < 5.551115123125783e-17 ? 1.0 : exp(-x); }

// e^-x without a branch, x clamped to [0, 708] (e^-0 = 1 exactly; below e^-708
// the value does not count): x = -(n ln 2 + r), |r| <= ln 2 / 2, in two fused
// steps, the Taylor polynomial of degree 13 (first omitted term below 5e-18)
// and 2^n added to the exponent.
__device__ __forceinline__ double exp_decay_bounded(double x) {
    x = fmin(fmax(x, 0.0), 708.0);
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

// 1 / sqrt(x) for a normal x > 0: the hardware's approximation (about 2^-20)
// and one cubically convergent step, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - x y^2.
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x * y, y, 1.0);
    return __fma_rn(y * e, __fma_rn(e, 0.375, 0.5), y);
}

// G_smooth = (exp(ikR) - 1)/(4 pi R) without cancellation (limit ik/(4 pi)).
__device__ __forceinline__ cplx g_smooth_exact(Medium k, double R) {
    if (R == 0.0) return {-k.ki * INV4PI_D, k.kr * INV4PI_D};
    double s, c, sh, ch;
    sincos(k.kr * R, &s, &c);
    sincos(0.5 * k.kr * R, &sh, &ch);
    double re = expm1(-k.ki * R) * c - 2.0 * sh * sh;
    double im = exp(-k.ki * R) * s;
    double f = INV4PI_D / R;
    return {re * f, im * f};
}

// ------------------------------------------------------------ Graglia (FP64)
struct TriQ {
    int n;
    double l1[25], l2[25], w[25];
};

// int_T 1/|r - r'| dS' (Graglia 1993) -- graglia.h:11-66, same guards.
__device__ inline double potential_integral(double rx, double ry, double rz, const double* v) {
    const double ax = v[0], ay = v[1], az = v[2], bx = v[3], by = v[4], bz = v[5],
                 cx = v[6], cy = v[7], cz = v[8];
    double e1x = bx - ax, e1y = by - ay, e1z = bz - az;
    double e2x = cx - ax, e2y = cy - ay, e2z = cz - az;
    double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
    double nn = sqrt(nx * nx + ny * ny + nz * nz);
    if (nn < 1e-15) return 0.0;
    nx /= nn, ny /= nn, nz /= nn;
    double res = 0.0;
    for (int i = 0; i < 3; i++) {
        const double* vi = v + 3 * i;
        const double* vj = v + 3 * ((i + 1) % 3);
        double ex = vj[0] - vi[0], ey = vj[1] - vi[1], ez = vj[2] - vi[2];
        double le = sqrt(ex * ex + ey * ey + ez * ez);
        if (le < 1e-15) continue;
        double tx = ex / le, ty = ey / le, tz = ez / le;
        double mx = ny * tz - nz * ty, my = nz * tx - nx * tz, mz = nx * ty - ny * tx;
        double dix = rx - vi[0], diy = ry - vi[1], diz = rz - vi[2];
        double d = dix * mx + diy * my + diz * mz;
        double h = dix * nx + diy * ny + diz * nz;
        double djx = vj[0] - rx, djy = vj[1] - ry, djz = vj[2] - rz;
        double dkx = vi[0] - rx, dky = vi[1] - ry, dkz = vi[2] - rz;
        double sp = djx * tx + djy * ty + djz * tz;
        double sm = dkx * tx + dky * ty + dkz * tz;
        double Rp = sqrt(djx * djx + djy * djy + djz * djz);
        double Rm = sqrt(dkx * dkx + dky * dky + dkz * dkz);
        if (Rp + sp > 1e-15 && Rm + sm > 1e-15) {
            double arg = (Rp + sp) / (Rm + sm);
            if (arg > 0) res += d * log(arg);
        }
        double ah = fabs(h);
        if (ah > 1e-15) {
            double R0 = d * d + h * h;
            double t1 = atan2(d * sp, R0 + ah * Rp);
            double t2 = atan2(d * sm, R0 + ah * Rm);
            res -= ah * (t1 - t2);
        }
    }
    return res;
}

// int_T |r - r'| dS' by the triangle rule -- graglia.h:69-85.  Evaluated with
// explicitly rounded operations (no FMA contraction) in the reference's
// order: the central difference below divides by 2e-6, so W must round the
// way the reference rounds it.
__device__ inline double integral_R(double rx, double ry, double rz, const double* v, const TriQ& q) {
    double e1x = __dsub_rn(v[3], v[0]), e1y = __dsub_rn(v[4], v[1]), e1z = __dsub_rn(v[5], v[2]);
    double e2x = __dsub_rn(v[6], v[0]), e2y = __dsub_rn(v[7], v[1]), e2z = __dsub_rn(v[8], v[2]);
    double nx = __dsub_rn(__dmul_rn(e1y, e2z), __dmul_rn(e1z, e2y));
    double ny = __dsub_rn(__dmul_rn(e1z, e2x), __dmul_rn(e1x, e2z));
    double nz = __dsub_rn(__dmul_rn(e1x, e2y), __dmul_rn(e1y, e2x));
    double area = __dmul_rn(0.5, __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(nx, nx), __dmul_rn(ny, ny)),
                                                      __dmul_rn(nz, nz))));
    double acc = 0.0;
    for (int k = 0; k < q.n; k++) {
        double l0 = __dsub_rn(__dsub_rn(1.0, q.l1[k]), q.l2[k]);
        double px = __dadd_rn(__dadd_rn(__dmul_rn(l0, v[0]), __dmul_rn(q.l1[k], v[3])), __dmul_rn(q.l2[k], v[6]));
        double py = __dadd_rn(__dadd_rn(__dmul_rn(l0, v[1]), __dmul_rn(q.l1[k], v[4])), __dmul_rn(q.l2[k], v[7]));
        double pz = __dadd_rn(__dadd_rn(__dmul_rn(l0, v[2]), __dmul_rn(q.l1[k], v[5])), __dmul_rn(q.l2[k], v[8]));
        double dx = __dsub_rn(px, rx), dy = __dsub_rn(py, ry), dz = __dsub_rn(pz, rz);
        double R = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
        acc = __dadd_rn(acc, __dmul_rn(q.w[k], R));
    }
    return __dmul_rn(area, acc);
}

// P = int_T 1/|r - r'| dS' and V = r P - grad_r W (W = int_T |r - r'| dS',
// central differences with eps = 1e-6) at the point of barycentric
// coordinates (l1, l2) of triangle v -- graglia.h:90-112.
__device__ inline void graglia_point(const double* v, double l1, double l2, const TriQ& q, double* P, double* V) {
    double l0 = __dsub_rn(__dsub_rn(1.0, l1), l2);
    double r[3];
    for (int d = 0; d < 3; d++)
        r[d] = __dadd_rn(__dadd_rn(__dmul_rn(v[d], l0), __dmul_rn(v[3 + d], l1)), __dmul_rn(v[6 + d], l2));
    double p = potential_integral(r[0], r[1], r[2], v);
    const double eps = 1e-6;
    double g[3];
    for (int d = 0; d < 3; d++) {
        double rp[3] = {r[0], r[1], r[2]}, rm[3] = {r[0], r[1], r[2]};
        rp[d] = __dadd_rn(rp[d], eps);
        rm[d] = __dsub_rn(rm[d], eps);
        double wp = integral_R(rp[0], rp[1], rp[2], v, q);
        double wm = integral_R(rm[0], rm[1], rm[2], v, q);
        g[d] = __ddiv_rn(__dsub_rn(wp, wm), 2.0 * eps);
    }
    *P = p;
    for (int d = 0; d < 3; d++) V[d] = __dsub_rn(__dmul_rn(r[d], p), g[d]);
}

}  // namespace bem
