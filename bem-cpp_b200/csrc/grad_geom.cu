// Adjoint contraction of the derivatives of the PMCHWT operator, the
// plane-wave right-hand sides and the far field with respect to the vertex
// coordinates and the interior wavenumber, without forming dZ.
//
// With the forward solutions x_c, the adjoint vectors lambda_c and
// D = diag(I, -I), the operator term of the gradient is
//   -Re sum_c lambda_c^T (dZ/dp) x_c = -Re sum_ij S_ij (dZ D)_ij / dp,
//   S = sym(P D), P = sum_c lambda_c x_c^T,
// because Z D is symmetric (its blocks are the symmetric Galerkin L and K).
// In terms of the N x N blocks of S:
//   Psi = Re sum_mn [WLe L_e + WLi L_i + WK (K_e + K_i)]_mn,
//   WLe = eta_e S11 - S22 / eta_e,  WLi = eta_i S11 - S22 / eta_i,
//   WK = S12 + S21  (all symmetric),
// and dPsi/dp is the operator term up to its sign.  L and K are sums over
// triangle pairs (a, b) of half-pair integrals; with the RWG basis
// f jw = alpha w (r - v_free), alpha = sign l / 2, the area cancels:
//   L_ts = alpha_t alpha_s sum_pq w_p w_q G(R) [ik (r_p - v_Ft).(r_q - v_Fs) - 4i/k]
//   K_ts = alpha_t alpha_s sum_pq w_p w_q g(R) (r_p - v_Ft).((r_p - r_q) x (r_q - v_Fs))
// with G = exp(ikR)/(4 pi R), g = G'(R)/R (the forms of assemble_LK_kernel,
// assembly.cu:14-135, and of this library's assembly).  Psi_ab = Psi_ba for
// symmetric weights, so the derivative with respect to the vertices of a is
// twice the derivative of sum_b Psi_ab through a's points, free vertices and
// edge lengths: grad_pair_kernel, one block per triangle a, analytic.  The
// same-triangle terms (the G_smooth quadrature and the Graglia singular
// correction, apply_singular_corrections, assembly.cu:208-321) are
// differentiated by central differences of the triangle's own term in its 9
// coordinates (grad_self_kernel); their k derivative is analytic.
// grad_rhs_kernel and grad_ff_kernel differentiate the right-hand sides
// (rhs.cpp:6-64) and the far field at fixed coefficients (farfield.cu:100-262)
// per RWG half.  Each kernel writes per-triangle or per-half gradients in the
// triangle's own vertex slots; the host adds them into the vertices.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "asm_device.cuh"
#include "bem_internal.h"
#include "lu_internal.h"

namespace bem {
namespace {

constexpr int GQ = 13;  // largest quadrature

__device__ __forceinline__ cplx cadd(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cplx csub(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ cplx cscale(cplx a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
    const double d = b.re * b.re + b.im * b.im;
    return {(a.re * b.re + a.im * b.im) / d, (a.im * b.re - a.re * b.im) / d};
}
__device__ __forceinline__ cplx c2(double2 v) { return {v.x, v.y}; }

// Per-triangle RWG halves: (RWG n or -1, sign, local index of the free vertex)
struct HalfInfo {
    int n[3], sign[3], jf[3];
};

__device__ __forceinline__ HalfInfo load_halves(const int* hinfo, int t) {
    HalfInfo h;
    for (int k = 0; k < 3; k++) {
        h.n[k] = hinfo[(t * 3 + k) * 3];
        h.sign[k] = hinfo[(t * 3 + k) * 3 + 1];
        h.jf[k] = hinfo[(t * 3 + k) * 3 + 2];
    }
    return h;
}

// alpha = sign |v_e1 - v_e2| / 2 with e1, e2 the vertices other than jf
__device__ __forceinline__ double half_alpha(const double* v, int sign, int jf) {
    const int e1 = (jf + 1) % 3, e2 = (jf + 2) % 3;
    const double dx = v[3 * e1] - v[3 * e2], dy = v[3 * e1 + 1] - v[3 * e2 + 1], dz = v[3 * e1 + 2] - v[3 * e2 + 2];
    return 0.5 * sign * sqrt(dx * dx + dy * dy + dz * dz);
}

// adds g * d alpha / d v into gv (9: the triangle's vertices)
__device__ __forceinline__ void alpha_to_vertices(const double* v, int sign, int jf, double g, double* gv) {
    const int e1 = (jf + 1) % 3, e2 = (jf + 2) % 3;
    double d[3];
    for (int c = 0; c < 3; c++) d[c] = v[3 * e1 + c] - v[3 * e2 + c];
    const double l = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    const double f = g * 0.5 * sign / l;
    for (int c = 0; c < 3; c++) {
        gv[3 * e1 + c] += f * d[c];
        gv[3 * e2 + c] -= f * d[c];
    }
}

__device__ __forceinline__ void bary_point(const double* v, double l1, double l2, double* r) {
    const double l0 = 1.0 - l1 - l2;
    for (int c = 0; c < 3; c++) r[c] = (v[c] * l0 + v[3 + c] * l1) + v[6 + c] * l2;
}

struct GradWeights {
    const double2 *WLe, *WLi, *WK, *Weta;  // N x N, row-major, symmetric
    int N;
};

struct PairArgs {
    const double* tv;   // nt x 9
    const int* hinfo;   // nt x 3 x 3
    int nt, Nq;
    TriQ q;
    Medium ke, ki;
    GradWeights W;
    double* gtri;       // nt x 9: d Psi / d (vertices of the triangle), pair terms
    double* sk;         // nt x 2: sum of WLi dL_i/dk_i + WK dK_i/dk_i over the triangle's pairs
    double* seta;       // nt x 2: sum of Weta L_i
};

// Block reduction of `cnt` doubles per thread into out (thread 0 writes).
template <int CNT>
__device__ void block_sum(double* vals, double* smem, double* out) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    for (int i = 0; i < CNT; i++) {
        double v = vals[i];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) smem[wid * CNT + i] = v;
    }
    __syncthreads();
    if (tid < CNT) {
        double s = 0.0;
        for (int w = 0; w < nw; w++) s += smem[w * CNT + tid];
        out[tid] = s;
    }
}

// One block per triangle a; its threads take the triangles b != a.
// In b's frame, r_q = v0 + l1 e1 + l2 e2 and rho = r_p - v0, the halves of b
// enter through three weights per matrix, c = sum_s c_s, c1 and c2 (those of
// the halves whose free vertex is v1, v2):
//   sum_s c_s (r_q - v_Fs) = (l1 c - c1) e1 + (l2 c - c2) e2,
// and d x W, W the same sum with the K weights, is linear in (l1, l2) as well.
// So a point p needs of its point pairs the moments of G and G'/R in
// (1, l1, l2) and of g = G'/R and g'/R in (1, l1, l2, l1^2, l1 l2, l2^2) (for
// the derivatives along d = rho - l1 e1 - l2 e2), and the three halves of a
// are contracted with these moments instead of with each point pair.
// Bound by the FP64 pipe: ~10 k operations of point pairs and ~8 k of
// contractions a triangle pair (~100 k with three evaluations of both
// Green's functions and six complex cross products per point pair).
// 1280 triangles, 7 points, an absorbing interior: 8.94 -> 3.17 ms, the pipe 56 %
// busy.
// DAMP: bit e, Im k_e != 0; BOUNDED: a real exterior k, Im k >= 0 inside and
// phases below SINCOS_MAX, the range of the branch-free functions (else the
// library's functions).
constexpr int GP_THREADS = 128, GP_W = 24;  // weights per half of a: (c, c1, c2) of WLe, WLi, WK, Weta

// c m_1 - c_1 m_0 and the like: Re(x y - z w)
__device__ __forceinline__ double re_msub(cplx x, cplx y, cplx z, cplx w) {
    return x.re * y.re - x.im * y.im - z.re * w.re + z.im * w.im;
}
__device__ __forceinline__ cplx cmsub(cplx x, cplx y, cplx z, cplx w) {
    return {x.re * y.re - x.im * y.im - z.re * w.re + z.im * w.im, x.re * y.im + x.im * y.re - z.re * w.im - z.im * w.re};
}
__device__ __forceinline__ void cfma(cplx& a, cplx b, double f) { a.re += b.re * f, a.im += b.im * f; }
__device__ __forceinline__ double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
    c[0] = a[1] * b[2] - a[2] * b[1], c[1] = a[2] * b[0] - a[0] * b[2], c[2] = a[0] * b[1] - a[1] * b[0];
}

template <int DAMP, bool BOUNDED> __global__ void __launch_bounds__(GP_THREADS, 2) grad_pair_kernel(PairArgs a) {
    extern __shared__ double s_w[];  // [3 GP_W][GP_THREADS]: each thread's weights
    const int ta = blockIdx.x, tid = threadIdx.x, Nq = a.Nq, N = a.W.N;
    __shared__ double s_va[9], s_rp[GQ][3], s_alpha[3];
    __shared__ double s_red[4 * 13];
    if (tid < 9) s_va[tid] = a.tv[9 * ta + tid];
    __syncthreads();
    const HalfInfo ha = load_halves(a.hinfo, ta);
    if (tid < Nq) bary_point(s_va, a.q.l1[tid], a.q.l2[tid], s_rp[tid]);
    if (tid < 3) s_alpha[tid] = ha.n[tid] >= 0 ? half_alpha(s_va, ha.sign[tid], ha.jf[tid]) : 0.0;
    __syncthreads();

    double gv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double gF[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, gal[3] = {0, 0, 0};
    cplx Sk = {0, 0}, Se = {0, 0};
    const Medium med[2] = {a.ke, a.ki};

    for (int tb = tid; tb < a.nt; tb += GP_THREADS) {
        if (tb == ta) continue;
        double v0[3], e1[3], e2[3], nv[3];
        {
            double vb[9], as[3];
            for (int j = 0; j < 9; j++) vb[j] = a.tv[9 * tb + j];
            const HalfInfo hb = load_halves(a.hinfo, tb);
#pragma unroll
            for (int s = 0; s < 3; s++) as[s] = hb.n[s] >= 0 ? half_alpha(vb, hb.sign[s], hb.jf[s]) : 0.0;
            for (int c = 0; c < 3; c++) v0[c] = vb[c], e1[c] = vb[3 + c] - vb[c], e2[c] = vb[6 + c] - vb[c];
            cross3(e1, e2, nv);
            const double2* const mats[4] = {a.W.WLe, a.W.WLi, a.W.WK, a.W.Weta};
#pragma unroll
            for (int t = 0; t < 3; t++) {
                if (ha.n[t] < 0) continue;
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    cplx w[3] = {{0, 0}, {0, 0}, {0, 0}};
#pragma unroll
                    for (int s = 0; s < 3; s++) {
                        if (hb.n[s] < 0) continue;
                        const cplx c = cscale(c2(mats[m][(size_t)ha.n[t] * N + hb.n[s]]), s_alpha[t] * as[s]);
                        const double f1 = hb.jf[s] == 1 ? 1.0 : 0.0, f2 = hb.jf[s] == 2 ? 1.0 : 0.0;
                        w[0] = cadd(w[0], c);
                        cfma(w[1], c, f1);
                        cfma(w[2], c, f2);
                    }
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        s_w[(t * GP_W + m * 6 + 2 * j) * GP_THREADS + tid] = w[j].re;
                        s_w[(t * GP_W + m * 6 + 2 * j + 1) * GP_THREADS + tid] = w[j].im;
                    }
                }
            }
        }
#pragma unroll 1
        for (int p = 0; p < Nq; p++) {
            double rho[3];
            for (int c = 0; c < 3; c++) rho[c] = s_rp[p][c] - v0[c];
            // moments: G and g of each medium, g'/R of both, R G of the interior
            cplx G[2][3], g[2][6], h[6], rg[3];
#pragma unroll
            for (int j = 0; j < 6; j++) {
                g[0][j] = g[1][j] = h[j] = {0, 0};
                if (j < 3) G[0][j] = G[1][j] = rg[j] = {0, 0};
            }
#pragma unroll 1
            for (int q = 0; q < Nq; q++) {
                const double l1 = a.q.l1[q], l2 = a.q.l2[q];
                const double m[6] = {1.0, l1, l2, l1 * l1, l1 * l2, l2 * l2};
                double d[3];
                for (int c = 0; c < 3; c++) d[c] = rho[c] - l1 * e1[c] - l2 * e2[c];
                const double R2 = dot3(d, d);
                const double invR = BOUNDED ? rsqrt_normal(R2) : rsqrt(R2), R = R2 * invR, invR2 = invR * invR;
                const double f = a.q.w[p] * a.q.w[q] * INV4PI_D * invR;
                cplx hs = {0, 0};
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const Medium k = med[e];
                    double sn, cs, ea = f;
                    if (BOUNDED)
                        sincos_bounded(k.kr * R, &sn, &cs);
                    else
                        sincos(k.kr * R, &sn, &cs);
                    if ((DAMP >> e) & 1) ea *= BOUNDED ? exp_decay_bounded(k.ki * R) : exp(-k.ki * R);
                    const cplx Gq = {ea * cs, ea * sn};
                    // g = G (ik - 1/R) / R, g' = -G (k^2 R^2 + 3 i k R - 3) / R^3
                    const cplx gq = cscale(cmul(Gq, cplx{-k.ki - invR, k.kr}), invR);
                    const cplx kk = cmul(cplx{k.kr, k.ki}, cplx{k.kr, k.ki});
                    const cplx pg = {kk.re * R2 - 3.0 * k.ki * R - 3.0, kk.im * R2 + 3.0 * k.kr * R};
                    hs = cadd(hs, cmul(Gq, pg));
#pragma unroll
                    for (int j = 0; j < 6; j++) {
                        cfma(g[e][j], gq, m[j]);
                        if (j < 3) cfma(G[e][j], Gq, m[j]);
                        if (j < 3 && e == 1) cfma(rg[j], Gq, R * m[j]);
                    }
                }
                hs = cscale(hs, -invR2 * invR2);
#pragma unroll
                for (int j = 0; j < 6; j++) cfma(h[j], hs, m[j]);
            }
            // moments times i k (the L form's scalar product) and 4 i / k (its charge term)
            cplx gs[3], Gf[2], gf[2][3], kG[3], nu[3], ns;
            {
                const Medium k = med[1];
                const cplx ik = {-k.ki, k.kr}, kc = {k.kr, k.ki};
                const double kn = k.kr * k.kr + k.ki * k.ki;
                const cplx fik = {4.0 * k.ki / kn, 4.0 * k.kr / kn}, f4k2 = cdiv(cplx{0.0, 4.0}, cmul(kc, kc));
                // d/dk: dG/dk = i R G, dg/dk = -k G, and the factors i k and 4 i / k
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    gs[j] = cadd(g[0][j], g[1][j]);
                    kG[j] = cmul(kc, G[1][j]);
                    const cplx x = cadd(cmul(ik, rg[j]), G[1][j]);
                    nu[j] = {-x.im, x.re};
                }
                const cplx y = cmul(fik, rg[0]);
                ns = cadd(cmul(f4k2, G[1][0]), cplx{y.im, -y.re});
            }
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const Medium k = med[e];
                const cplx ik = {-k.ki, k.kr};
                const double kn = k.kr * k.kr + k.ki * k.ki;
                const cplx fik = {4.0 * k.ki / kn, 4.0 * k.kr / kn};
                Gf[e] = cmul(fik, G[e][0]);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    gf[e][j] = cmul(fik, g[e][j]);
                    G[e][j] = cmul(ik, G[e][j]);
                }
#pragma unroll
                for (int j = 0; j < 6; j++) g[e][j] = cmul(ik, g[e][j]);
            }
            double re1[3], re2[3], grp[3] = {0, 0, 0}, z[3] = {0, 0, 0};
            cross3(rho, e1, re1);
            cross3(rho, e2, re2);
            constexpr int MI[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};  // moments of (1, l1, l2) times l_i
#pragma unroll
            for (int t = 0; t < 3; t++) {
                if (ha.n[t] < 0) continue;
                auto wt = [&](int i) -> cplx {
                    const double* w = s_w + (t * GP_W + 2 * i) * GP_THREADS + tid;
                    return {w[0], w[GP_THREADS]};
                };
                double u[3], e1u[3], e2u[3];
                for (int c = 0; c < 3; c++) u[c] = s_rp[p][c] - s_va[3 * ha.jf[t] + c];
                cross3(e1, u, e1u);
                cross3(e2, u, e2u);
                const double p1 = dot3(u, e1), p2 = dot3(u, e2), b1 = dot3(u, re1), b2 = dot3(u, re2), bn = dot3(u, nv);
                double x1 = 0, x2 = 0, x3 = 0;
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const cplx w0 = wt(3 * e), w1 = wt(3 * e + 1), w2 = wt(3 * e + 2);
                    x1 += re_msub(w0, G[e][1], w1, G[e][0]);
                    x2 += re_msub(w0, G[e][2], w2, G[e][0]);
                    x3 += w0.re * Gf[e].re - w0.im * Gf[e].im;
#pragma unroll
                    for (int i = 0; i < 3; i++)
                        z[i] += p1 * re_msub(w0, g[e][MI[i][1]], w1, g[e][MI[i][0]]) +
                                p2 * re_msub(w0, g[e][MI[i][2]], w2, g[e][MI[i][0]]) -
                                (w0.re * gf[e][i].re - w0.im * gf[e][i].im);
                    if (e == 1) {
                        const cplx s1 = cmsub(w0, nu[1], w1, nu[0]), s2 = cmsub(w0, nu[2], w2, nu[0]);
                        Sk = cadd(Sk, cmul(w0, ns));
                        cfma(Sk, s1, p1);
                        cfma(Sk, s2, p2);
                    }
                }
                const cplx k0 = wt(6), k1 = wt(7), k2 = wt(8);
                const double y1 = re_msub(k0, gs[1], k1, gs[0]), y2 = re_msub(k0, gs[2], k2, gs[0]),
                             y3 = re_msub(k2, gs[1], k1, gs[2]);
#pragma unroll
                for (int i = 0; i < 3; i++)
                    z[i] += b1 * re_msub(k0, h[MI[i][1]], k1, h[MI[i][0]]) +
                            b2 * re_msub(k0, h[MI[i][2]], k2, h[MI[i][0]]) + bn * re_msub(k2, h[MI[i][1]], k1, h[MI[i][2]]);
                cfma(Sk, cmsub(k0, kG[1], k1, kG[0]), -b1);
                cfma(Sk, cmsub(k0, kG[2], k2, kG[0]), -b2);
                cfma(Sk, cmsub(k2, kG[1], k1, kG[2]), -bn);
                const cplx n0 = wt(9), n1 = wt(10), n2 = wt(11);
                cfma(Se, cmsub(n0, G[1][1], n1, G[1][0]), p1);
                cfma(Se, cmsub(n0, G[1][2], n2, G[1][0]), p2);
                Se = csub(Se, cmul(n0, Gf[1]));
                gal[t] += p1 * x1 + p2 * x2 - x3 + b1 * y1 + b2 * y2 + bn * y3;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double m = x1 * e1[c] + x2 * e2[c] + y1 * re1[c] + y2 * re2[c] + y3 * nv[c];
                    gF[t][c] -= m;
                    grp[c] += m + y1 * e1u[c] + y2 * e2u[c];
                }
            }
            const double l1 = a.q.l1[p], l2 = a.q.l2[p], l0 = 1.0 - l1 - l2;
            for (int c = 0; c < 3; c++) {
                grp[c] += rho[c] * z[0] - e1[c] * z[1] - e2[c] * z[2];
                gv[c] += l0 * grp[c];
                gv[3 + c] += l1 * grp[c];
                gv[6 + c] += l2 * grp[c];
            }
        }
    }
    for (int t = 0; t < 3; t++) {
        if (ha.n[t] < 0) continue;
        for (int c = 0; c < 3; c++) gv[3 * ha.jf[t] + c] += gF[t][c];
        alpha_to_vertices(s_va, ha.sign[t], ha.jf[t], gal[t] / s_alpha[t], gv);
    }
    // Psi_ab = Psi_ba: the b-side derivatives are the a-side ones of (b, a)
    double vals[13];
    for (int i = 0; i < 9; i++) vals[i] = 2.0 * gv[i];
    vals[9] = Sk.re, vals[10] = Sk.im, vals[11] = Se.re, vals[12] = Se.im;
    __shared__ double s_out[13];
    block_sum<13>(vals, s_red, s_out);
    __syncthreads();
    if (tid < 9) a.gtri[9 * ta + tid] = s_out[tid];
    if (tid == 0) {
        a.sk[2 * ta] = s_out[9], a.sk[2 * ta + 1] = s_out[10];
        a.seta[2 * ta] = s_out[11], a.seta[2 * ta + 1] = s_out[12];
    }
}

struct SelfArgs {
    const double* tv;
    const int* hinfo;
    int nt, Nq;
    TriQ q;
    Medium ke, ki;
    unsigned flags;
    GradWeights W;
    double* gtri;   // nt x 9 (central differences of the triangle's own term)
    double* sk;     // nt x 4: the k contraction for Re k, then for Im k (complex each)
    double* seta;   // nt x 2
};

// The triangle's own term: Re sum over its ordered half pairs (t, s) and both
// media of W_e(n_t, n_s) times the same-triangle part of L_e(n_t, n_s) -- the
// G_smooth quadrature (assembly kernels with sing = true) plus the Graglia
// correction (singular_fixup_kernel); with want_k / eta also the interior
// medium's k derivative and the Weta contraction.
// The interior wavenumber enters holomorphically everywhere except at the
// coincident points of the literal G_smooth, exp(ik R_s)/(4 pi R_s) -
// 1/(4 pi R_s) at R_s = 1e-15: there the real part is the rounding of
// exp(-Im k R_s) cos(Re k R_s) to 1 (zero, or a step of one unit in the last
// place) and does not follow Im k, while the imaginary part follows Re k.  So
// the k derivative is returned for Re k (skr) and Im k (ski) separately.
template <bool EXTRA>
__device__ double self_term(const double* v, const HalfInfo& h, const SelfArgs& a, cplx* skr, cplx* ski, cplx* se) {
    const int Nq = a.Nq, N = a.W.N;
    double rp[GQ][3];
    for (int p = 0; p < Nq; p++) bary_point(v, a.q.l1[p], a.q.l2[p], rp[p]);
    double al[3], vF[3][3];
    for (int t = 0; t < 3; t++) {
        al[t] = h.n[t] >= 0 ? half_alpha(v, h.sign[t], h.jf[t]) : 0.0;
        for (int c = 0; c < 3; c++) vF[t][c] = h.n[t] >= 0 ? v[3 * h.jf[t] + c] : 0.0;
    }
    const double e1x = v[3] - v[0], e1y = v[4] - v[1], e1z = v[5] - v[2];
    const double e2x = v[6] - v[0], e2y = v[7] - v[1], e2z = v[8] - v[2];
    const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
    const double area = 0.5 * sqrt(nx * nx + ny * ny + nz * nz);
    // Graglia P and V at the triangle's points
    double P[GQ], V[GQ][3];
    for (int p = 0; p < Nq; p++) graglia_point(v, a.q.l1[p], a.q.l2[p], a.q, &P[p], V[p]);
    const bool exact = (a.flags & BEM_ASM_GSMOOTH_EXACT) != 0;
    const Medium med[2] = {a.ke, a.ki};
    double psi = 0.0;
    if (EXTRA) *skr = *ski = *se = {0, 0};
    for (int e = 0; e < 2; e++) {
        const Medium k = med[e];
        const cplx ik = {-k.ki, k.kr};
        const double kn = k.kr * k.kr + k.ki * k.ki;
        const cplx iok = {k.ki / kn, k.kr / kn};  // i/k
        // the 3 x 3 half pairs share the Green's function of a point pair
        cplx Ls[3][3], Lkr[EXTRA ? 3 : 1][3], Lki[EXTRA ? 3 : 1][3];
#pragma unroll
        for (int t = 0; t < 3; t++)
#pragma unroll
            for (int s = 0; s < 3; s++) {
                Ls[t][s] = {0, 0};
                if (EXTRA) Lkr[t][s] = Lki[t][s] = {0, 0};
            }
        for (int p = 0; p < Nq; p++)
            for (int q = 0; q < Nq; q++) {
                const double d0 = rp[p][0] - rp[q][0], d1 = rp[p][1] - rp[q][1], d2 = rp[p][2] - rp[q][2];
                const double R2 = fmax(d0 * d0 + d1 * d1 + d2 * d2, 1e-30);
                const double invR = rsqrt(R2), Rs = R2 * invR;
                const double i4R = __dmul_rn(INV4PI_D, invR);
                double sn, cs;
                sincos(k.kr * Rs, &sn, &cs);
                const double ea = k.ki != 0.0 ? exp_decay(k.ki * Rs) : 1.0;
                cplx Gs = {ea * cs * i4R - i4R, ea * sn * i4R};
                if (exact) Gs = g_smooth_exact(k, p == q ? 0.0 : Rs);
                const double ww = a.q.w[p] * a.q.w[q];
#pragma unroll
                for (int t = 0; t < 3; t++)
#pragma unroll
                    for (int s = 0; s < 3; s++) {
                        double uu = 0.0;
                        for (int c = 0; c < 3; c++) uu += (rp[p][c] - vF[t][c]) * (rp[q][c] - vF[s][c]);
                        // G_s (ik u.u' - 4i/k)
                        const cplx Q = {ik.re * uu - 4.0 * iok.re, ik.im * uu - 4.0 * iok.im};
                        const cplx term = cmul(Gs, Q);
                        Ls[t][s].re += ww * term.re, Ls[t][s].im += ww * term.im;
                        if (EXTRA && e == 1) {
                            // dG_s/dk = i exp(ikR)/(4 pi); d Q/dk = i u.u' + 4i/k^2
                            const cplx dGs = {-ea * sn * INV4PI_D, ea * cs * INV4PI_D};
                            const cplx f4k2 = cdiv(cplx{0.0, 4.0}, cmul(cplx{k.kr, k.ki}, cplx{k.kr, k.ki}));
                            const cplx dQ = {f4k2.re, uu + f4k2.im};
                            const cplx dt = cadd(cmul(dGs, Q), cmul(Gs, dQ));
                            Lkr[t][s].re += ww * dt.re, Lkr[t][s].im += ww * dt.im;
                            // d/dIm k = i d/dk, except the literal G_s at a coincident point
                            const cplx di = (p == q && !exact) ? cmul(Gs, cmul(cplx{0.0, 1.0}, dQ))
                                                               : cmul(cplx{0.0, 1.0}, dt);
                            Lki[t][s].re += ww * di.re, Lki[t][s].im += ww * di.im;
                        }
                    }
            }
#pragma unroll
        for (int t = 0; t < 3; t++) {
            if (h.n[t] < 0) continue;
#pragma unroll
            for (int s = 0; s < 3; s++) {
                if (h.n[s] < 0) continue;
                const double aa = al[t] * al[s];
                const size_t ix = (size_t)h.n[t] * N + h.n[s];
                // Graglia sums (without the alpha alpha / A factor)
                double sA = 0.0, sB = 0.0;
                for (int p = 0; p < Nq; p++) {
                    sA += a.q.w[p] * P[p];
                    double dot = 0.0;
                    for (int c = 0; c < 3; c++) dot += (rp[p][c] - vF[t][c]) * (V[p][c] - vF[s][c] * P[p]);
                    sB += a.q.w[p] * dot;
                }
                const double SA = 4.0 * aa / area * sA * INV4PI_D, SB = aa / area * sB * INV4PI_D;
                // L_e(self) = alpha alpha sum + (-(i/k) SA + ik SB)
                const cplx corr = {-iok.re * SA + ik.re * SB, -iok.im * SA + ik.im * SB};
                const cplx Lself = {aa * Ls[t][s].re + corr.re, aa * Ls[t][s].im + corr.im};
                const cplx W = c2((e ? a.W.WLi : a.W.WLe)[ix]);
                psi += W.re * Lself.re - W.im * Lself.im;
                if (EXTRA && e == 1) {
                    // d/dk of the correction: (i/k^2) SA + i SB (holomorphic)
                    const cplx ik2 = cdiv(cplx{0.0, 1.0}, cmul(cplx{k.kr, k.ki}, cplx{k.kr, k.ki}));
                    const cplx dcorr = {ik2.re * SA, ik2.im * SA + SB};
                    const cplx dLr = {aa * Lkr[t][s].re + dcorr.re, aa * Lkr[t][s].im + dcorr.im};
                    const cplx dci = cmul(cplx{0.0, 1.0}, dcorr);
                    const cplx dLi = {aa * Lki[t][s].re + dci.re, aa * Lki[t][s].im + dci.im};
                    *skr = cadd(*skr, cmul(W, dLr));
                    *ski = cadd(*ski, cmul(W, dLi));
                    *se = cadd(*se, cmul(c2(a.W.Weta[ix]), Lself));
                }
            }
        }
    }
    return psi;
}

// Central differences of a triangle's own term in its 9 coordinates (step
// 1e-4 of its longest edge), and the k / eta contractions: SELF_EVALS = 19
// evaluations per triangle, a thread each (18 displaced ones and the
// undisplaced one with its k derivatives, which sits in a warp of its own
// kind only by chance: one in 19).  C5: 6.4 ms with one thread per triangle
// making all 19 in turn (20 blocks) and the Green's function taken per half pair.
constexpr int SELF_EVALS = 19, SELF_TRI = 6;
__global__ void __launch_bounds__(SELF_EVALS * SELF_TRI) grad_self_kernel(SelfArgs a) {
    __shared__ double s_psi[SELF_TRI][SELF_EVALS];
    const int tl = threadIdx.x % SELF_TRI, ev = threadIdx.x / SELF_TRI, t = blockIdx.x * SELF_TRI + tl;
    double hstep = 0.0;
    if (t < a.nt) {
        double v[9];
        for (int j = 0; j < 9; j++) v[j] = a.tv[9 * (size_t)t + j];
        const HalfInfo h = load_halves(a.hinfo, t);
        double lmax = 0.0;
        for (int j = 0; j < 3; j++) {
            const int j1 = (j + 1) % 3;
            const double dx = v[3 * j] - v[3 * j1], dy = v[3 * j + 1] - v[3 * j1 + 1],
                         dz = v[3 * j + 2] - v[3 * j1 + 2];
            lmax = fmax(lmax, sqrt(dx * dx + dy * dy + dz * dz));
        }
        hstep = 1e-4 * lmax;
        if (ev < SELF_EVALS - 1) {
            const int j = ev >> 1;
            const double step = (ev & 1) ? -hstep : hstep;
            for (int i = 0; i < 9; i++) v[i] = i == j ? v[i] + step : v[i];
            s_psi[tl][ev] = self_term<false>(v, h, a, nullptr, nullptr, nullptr);
        } else {
            cplx skr, ski, se;
            self_term<true>(v, h, a, &skr, &ski, &se);
            a.sk[4 * t] = skr.re, a.sk[4 * t + 1] = skr.im, a.sk[4 * t + 2] = ski.re, a.sk[4 * t + 3] = ski.im;
            a.seta[2 * t] = se.re, a.seta[2 * t + 1] = se.im;
        }
    }
    __syncthreads();
    if (t < a.nt && ev < 9) a.gtri[9 * (size_t)t + ev] = (s_psi[tl][2 * ev] - s_psi[tl][2 * ev + 1]) / (2.0 * hstep);
}

struct HalfArgs {
    const double* tv;
    const int* htri;  // (2N) triangle of half h*N+n
    const int* hjf;   // (2N) local free vertex of the half
    int N, Nq;
    TriQ q;
    double kr, ki, eta;
    const double* RT;         // n_orient x 9
    int n_orient;
    const double2* Lam;       // adjoint vectors, column-major n x 2 n_orient
    int64_t ldl;
    double* ghalf;            // 2N x 9
};

// Right-hand sides: Re sum_c lambda_c^T dB_c, per RWG half (thread), with
// B_c[n] = sum_t alpha_t sum_p w_p (r_p - v_Ft).E0_c exp(ik khat_c.r_p) and
// H0_c = khat_c x E0_c / eta in the rows N + n (rhs.cpp:6-64).
__global__ void grad_rhs_kernel(HalfArgs a) {
    const int hn = blockIdx.x * blockDim.x + threadIdx.x;
    if (hn >= 2 * a.N) return;
    const int n = hn % a.N, sign = hn < a.N ? 1 : -1, t = a.htri[hn], jf = a.hjf[hn], Nq = a.Nq;
    double v[9];
    for (int j = 0; j < 9; j++) v[j] = a.tv[9 * t + j];
    const double al = half_alpha(v, sign, jf);
    const double* vF = v + 3 * jf;
    double gv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, gF[3] = {0, 0, 0}, gal = 0.0;
    double rp[GQ][3];
    for (int p = 0; p < Nq; p++) bary_point(v, a.q.l1[p], a.q.l2[p], rp[p]);
    double grp[GQ][3];
    for (int p = 0; p < Nq; p++) grp[p][0] = grp[p][1] = grp[p][2] = 0.0;
    for (int o = 0; o < a.n_orient; o++) {
        const double* R = a.RT + 9 * o;
        double kh[3], ep[2][3], H[2][3];
        for (int i = 0; i < 3; i++) kh[i] = R[3 * i + 2], ep[0][i] = R[3 * i], ep[1][i] = R[3 * i + 1];
        for (int pl = 0; pl < 2; pl++) {
            H[pl][0] = (kh[1] * ep[pl][2] - kh[2] * ep[pl][1]) / a.eta;
            H[pl][1] = (kh[2] * ep[pl][0] - kh[0] * ep[pl][2]) / a.eta;
            H[pl][2] = (kh[0] * ep[pl][1] - kh[1] * ep[pl][0]) / a.eta;
        }
        cplx Q[3] = {{0, 0}, {0, 0}, {0, 0}};
        for (int pl = 0; pl < 2; pl++) {
            const int c = 2 * o + pl;
            const cplx lj = c2(a.Lam[(int64_t)c * a.ldl + n]), lm = c2(a.Lam[(int64_t)c * a.ldl + a.N + n]);
            for (int i = 0; i < 3; i++) Q[i] = cadd(Q[i], cadd(cscale(lj, ep[pl][i]), cscale(lm, H[pl][i])));
        }
        for (int p = 0; p < Nq; p++) {
            const double s = kh[0] * rp[p][0] + kh[1] * rp[p][1] + kh[2] * rp[p][2];
            double sn, cs;
            sincos(a.kr * s, &sn, &cs);
            const double ea = exp(-a.ki * s);
            const cplx ph = {ea * cs, ea * sn};  // exp(ik s)
            const double u[3] = {rp[p][0] - vF[0], rp[p][1] - vF[1], rp[p][2] - vF[2]};
            const cplx uQ = cadd(cadd(cscale(Q[0], u[0]), cscale(Q[1], u[1])), cscale(Q[2], u[2]));
            const cplx pQ = cmul(ph, uQ);
            const cplx ikp = cmul(cplx{-a.ki, a.kr}, pQ);  // ik phase (u.Q)
            const double w = a.q.w[p];
            for (int i = 0; i < 3; i++) {
                const cplx pq = cmul(ph, Q[i]);
                grp[p][i] += al * w * (pq.re + ikp.re * kh[i]);
                gF[i] -= al * w * pq.re;
            }
            gal += w * pQ.re;
        }
    }
    for (int p = 0; p < Nq; p++) {
        const double l1 = a.q.l1[p], l2 = a.q.l2[p], l0 = 1.0 - l1 - l2;
        for (int c = 0; c < 3; c++) {
            gv[c] += l0 * grp[p][c];
            gv[3 + c] += l1 * grp[p][c];
            gv[6 + c] += l2 * grp[p][c];
        }
    }
    for (int c = 0; c < 3; c++) gv[3 * jf + c] += gF[c];
    alpha_to_vertices(v, sign, jf, gal, gv);
    for (int j = 0; j < 9; j++) a.ghalf[9 * (size_t)hn + j] = gv[j];
}

struct FFArgs2 {
    const double* tv;      // nt x 9
    const int* hinfo;      // nt x 3 x 3
    int nt, N, Nq;
    TriQ q;
    double kr, ki, eta;
    const double* RT;      // n_orient x 9
    int n_orient, ntheta;
    const double2* ab;     // [c][theta][2]: components A, B of the adjoint weight of the far field
    const double2* X;      // forward solutions, column-major 2N x 2 n_orient
    int64_t ldx;
    double* gpart;         // gridDim.y x nt x 9
};

// Far field at fixed coefficients: Re sum_c sum_theta h . dF_c(theta) in the
// vertices of every triangle, F = -ik/(4 pi) [eta J_perp - rhat x M] with
// J = sum_n x_n sum_t alpha_t sum_p w_p (r_p - v_Ft) exp(-ik rhat.r_p)
// (farfield.cu:100-262).  With ph = exp(-ik rhat.r_p), Y = eta x_J h +
// x_M rhat x h and u = r_p - v_Ft a point needs sum ph Y and
// sum ph (u.Y) rhat.  h = A e_par + B e_perp, rhat x h = A e3 - B e_par,
// e_par = e1 cos t - e2 sin t, rhat = e1 sin t + e2 cos t (the frame of
// farfield_adjoint_kernel), so all of it is linear in ten complex sums over
// the directions that depend on the point and the column alone,
//   sum ph A (1, cos, sin, cos sin, cos^2) and the same with B.
// Thread: one quadrature point of a triangle; it takes the phase once for
// both polarisations and the three RWG halves, and applies coefficients and
// free vertices after the sum.  Block (x, y): 128 / Nq triangles, every
// gridDim.y-th orientation.  C5 (2N = 3840, 64 orientations, 181 angles):
// 45.3 ms with a thread per RWG half that formed Y and u.Y per direction
// (120 warps on the chip, 3 x the exponentials, 3 x the multiply-adds).
constexpr int GFF_THREADS = 128, GFF_SPLIT = 32;
__global__ void __launch_bounds__(GFF_THREADS) grad_ff_kernel(FFArgs2 a) {
    extern __shared__ __align__(16) double sm2[];
    double2* s_t = (double2*)sm2;          // ntheta: sin, cos
    double2* s_ab = s_t + a.ntheta;        // ntheta x 4: A0 B0 A1 B1
    double* s_red = sm2;                   // GFF_THREADS x 13, after the sums
    const int tid = threadIdx.x, Nq = a.Nq, per = GFF_THREADS / Nq;
    const int tl = tid / Nq, p = tid % Nq, tri = blockIdx.x * per + tl;
    const bool act = tl < per && tri < a.nt;
    double v[9], r[3] = {0, 0, 0};
    HalfInfo h;
    if (act) {
        for (int j = 0; j < 9; j++) v[j] = a.tv[9 * (size_t)tri + j];
        h = load_halves(a.hinfo, tri);
        bary_point(v, a.q.l1[p], a.q.l2[p], r);
    }
    for (int t = tid; t < a.ntheta; t += blockDim.x) {
        double st, ct;
        sincos(a.ntheta > 1 ? M_PI * t / (a.ntheta - 1) : 0.0, &st, &ct);
        s_t[t] = make_double2(st, ct);
    }
    double grp[3] = {0, 0, 0}, gF[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, gal[3] = {0, 0, 0};
    const cplx pk = {a.ki * INV4PI_D, -a.kr * INV4PI_D};  // -ik/(4 pi)
    const cplx mik = {a.ki, -a.kr};                        // -ik
    for (int o = blockIdx.y; o < a.n_orient; o += gridDim.y) {
        __syncthreads();
        for (int e = tid; e < 4 * a.ntheta; e += blockDim.x)
            s_ab[e] = a.ab[((size_t)(2 * o + (e & 3) / 2) * a.ntheta + e / 4) * 2 + (e & 1)];
        __syncthreads();
        if (!act) continue;
        double e1[3], e2[3], e3[3], x1 = 0.0, x2 = 0.0;
        const double* R = a.RT + 9 * (size_t)o;
        for (int i = 0; i < 3; i++) {
            e1[i] = R[3 * i], e3[i] = R[3 * i + 1], e2[i] = R[3 * i + 2];
            x1 += e1[i] * r[i], x2 += e2[i] * r[i];
        }
        cplx sA[2][5], sB[2][5];  // weights 1, cos, sin, cos sin, cos^2
#pragma unroll
        for (int pol = 0; pol < 2; pol++)
#pragma unroll
            for (int k = 0; k < 5; k++) sA[pol][k] = sB[pol][k] = {0, 0};
        for (int t = 0; t < a.ntheta; t++) {
            const double st = s_t[t].x, ct = s_t[t].y, rd = st * x1 + ct * x2;
            double sn, cs;
            sincos(a.kr * rd, &sn, &cs);
            const double ea = a.ki != 0.0 ? exp(a.ki * rd) : 1.0;
            const cplx ph = {ea * cs, -ea * sn};
            const double w[5] = {1.0, ct, st, ct * st, ct * ct};
#pragma unroll
            for (int pol = 0; pol < 2; pol++) {
                const cplx pa = cmul(ph, c2(s_ab[4 * t + 2 * pol])), pb = cmul(ph, c2(s_ab[4 * t + 2 * pol + 1]));
#pragma unroll
                for (int k = 0; k < 5; k++) {
                    sA[pol][k].re += w[k] * pa.re, sA[pol][k].im += w[k] * pa.im;
                    sB[pol][k].re += w[k] * pb.re, sB[pol][k].im += w[k] * pb.im;
                }
            }
        }
        const double wp = a.q.w[p];
#pragma unroll
        for (int pol = 0; pol < 2; pol++) {
            const cplx *A = sA[pol], *B = sB[pol];
            const cplx Ass = csub(A[0], A[4]), Bss = csub(B[0], B[4]);  // sin^2 = 1 - cos^2
            const int64_t col = (int64_t)(2 * o + pol) * a.ldx;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                if (h.n[k] < 0) continue;
                const cplx xJ = cscale(c2(a.X[col + h.n[k]]), a.eta), xM = c2(a.X[col + a.N + h.n[k]]);
                const double al = half_alpha(v, h.sign[k], h.jf[k]);
                double u[3], u1 = 0.0, u2 = 0.0, u3 = 0.0;
                for (int i = 0; i < 3; i++) {
                    u[i] = r[i] - v[3 * h.jf[k] + i];
                    u1 += u[i] * e1[i], u2 += u[i] * e2[i], u3 += u[i] * e3[i];
                }
                // sum ph Y in the frame (e1, e2, e3)
                const cplx y1 = csub(cmul(xJ, A[1]), cmul(xM, B[1])), y2 = csub(cmul(xM, B[2]), cmul(xJ, A[2])),
                           y3 = cadd(cmul(xJ, B[0]), cmul(xM, A[0]));
                // sum ph (u.Y) sin t and sum ph (u.Y) cos t
                const cplx js = cadd(csub(cscale(A[3], u1), cscale(Ass, u2)), cscale(B[2], u3)),
                           ms = cadd(csub(cscale(A[2], u3), cscale(B[3], u1)), cscale(Bss, u2)),
                           jc = cadd(csub(cscale(A[4], u1), cscale(A[3], u2)), cscale(B[1], u3)),
                           mc = cadd(csub(cscale(A[1], u3), cscale(B[4], u1)), cscale(B[3], u2));
                const cplx S = cmul(mik, cadd(cmul(xJ, js), cmul(xM, ms))), Cc = cmul(mik, cadd(cmul(xJ, jc), cmul(xM, mc)));
                const double f1 = cmul(pk, y1).re, f2 = cmul(pk, y2).re, f3 = cmul(pk, y3).re;
                const double gs = cmul(pk, S).re, gc = cmul(pk, Cc).re;
                for (int i = 0; i < 3; i++) {
                    const double F = al * wp * (e1[i] * f1 + e2[i] * f2 + e3[i] * f3);
                    gF[k][i] -= F;
                    grp[i] += F + al * wp * (e1[i] * gs + e2[i] * gc);
                }
                gal[k] += wp * (u1 * f1 + u2 * f2 + u3 * f3);
            }
        }
    }
    __syncthreads();
    if (act) {
        const double l1 = a.q.l1[p], l2 = a.q.l2[p], l0 = 1.0 - l1 - l2;
        double* out = s_red + (size_t)tid * 13;
        for (int i = 0; i < 3; i++) {
            out[i] = l0 * grp[i];
            out[3 + i] = l1 * grp[i];
            out[6 + i] = l2 * grp[i];
        }
        for (int k = 0; k < 3; k++) {
            if (h.n[k] >= 0)
                for (int i = 0; i < 3; i++) out[3 * h.jf[k] + i] += gF[k][i];
            out[9 + k] = gal[k];
        }
    }
    __syncthreads();
    if (act && p == 0) {
        double gv[12];
        for (int j = 0; j < 12; j++) gv[j] = 0.0;
        for (int q = 0; q < Nq; q++)
            for (int j = 0; j < 12; j++) gv[j] += s_red[(size_t)(tid + q) * 13 + j];
        for (int k = 0; k < 3; k++)
            if (h.n[k] >= 0) alpha_to_vertices(v, h.sign[k], h.jf[k], gv[9 + k], gv);
        for (int j = 0; j < 9; j++) a.gpart[((size_t)blockIdx.y * a.nt + tri) * 9 + j] = gv[j];
    }
}

// out[i] = sum over the parts in order
__global__ void part_sum_kernel(const double* __restrict__ part, int parts, int count, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    double s = 0.0;
    for (int k = 0; k < parts; k++) s += part[(size_t)k * count + i];
    out[i] = s;
}

// S = (Lam Xd^T + Xd Lam^T) / 2 -> the four N x N weight matrices
__global__ void weights_kernel(const double2* __restrict__ S, int N, double eta_e, double eta_i,
                               double2* __restrict__ WLe, double2* __restrict__ WLi, double2* __restrict__ WK,
                               double2* __restrict__ Weta) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)N * N) return;
    const int m = (int)(i / N), n = (int)(i % N);
    const int64_t ld = 2 * (int64_t)N;
    const double2 s11 = S[m * ld + n], s22 = S[(N + m) * ld + N + n], s12 = S[m * ld + N + n],
                  s21 = S[(N + m) * ld + n];
    WLe[i] = make_double2(eta_e * s11.x - s22.x / eta_e, eta_e * s11.y - s22.y / eta_e);
    WLi[i] = make_double2(eta_i * s11.x - s22.x / eta_i, eta_i * s11.y - s22.y / eta_i);
    WK[i] = make_double2(s12.x + s21.x, s12.y + s21.y);
    const double ie2 = 1.0 / (eta_i * eta_i);
    Weta[i] = make_double2(s11.x + s22.x * ie2, s11.y + s22.y * ie2);
}

// Y[i][c] = s(i) X[c][i]: column-major n x nc -> row-major n x nc, rows >= flip negated
__global__ void transpose_flip_kernel(const double2* __restrict__ X, int64_t ldx, int n, int nc, int flip_from,
                                      double2* __restrict__ Y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * nc) return;
    const int r = (int)(i / nc), c = (int)(i % nc);
    double2 v = X[(int64_t)c * ldx + r];
    if (r >= flip_from) v = make_double2(-v.x, -v.y);
    Y[i] = v;
}

struct DevBuf {
    void* p = nullptr;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    int alloc(bem_ctx* ctx, size_t bytes) {
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            return fail(ctx, BEM_ERR_OOM, "gradient buffer of %zu bytes", bytes);
        }
        return BEM_OK;
    }
};

unsigned nblocks(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

int adjoint_geometry(bem_ctx* ctx, const bem_geom* g, std::complex<double> kext, std::complex<double> kint,
                     double eta_e, double eta_i, unsigned flags, const void* X, const void* Lam, int ncols,
                     const double* RT_dev, int n_orient, const void* ab_dev, int ntheta,
                     double* grad_v, double* dpsi_dk, double* dpsi_deta) {
    const int N = g->N, n = 2 * N, nt = g->nt, Nq = g->Nq, nv = g->nv;
    cudaStream_t st = ctx->stream;
    // per-triangle halves and per-half (triangle, local free vertex)
    std::vector<int> hinfo((size_t)nt * 9, -1), htri(2 * (size_t)N), hjf(2 * (size_t)N);
    std::vector<int> cnt(nt, 0);
    const HostMesh& M = g->mesh;
    const HostRWG& r = g->rwg;
    for (int h = 0; h < 2; h++)
        for (int m = 0; m < N; m++) {
            const int t = h == 0 ? r.tri_p[m] : r.tri_m[m];
            const int vf = h == 0 ? r.vfree_p[m] : r.vfree_m[m];
            int jf = -1;
            for (int j = 0; j < 3; j++)
                if (M.tris[3 * t + j] == vf) jf = j;
            if (jf < 0 || cnt[t] >= 3) return fail(ctx, BEM_ERR_INVALID, "RWG %d: free vertex not on triangle %d", m, t);
            const int k = cnt[t]++;
            hinfo[((size_t)t * 3 + k) * 3] = m;
            hinfo[((size_t)t * 3 + k) * 3 + 1] = h == 0 ? 1 : -1;
            hinfo[((size_t)t * 3 + k) * 3 + 2] = jf;
            htri[(size_t)h * N + m] = t;
            hjf[(size_t)h * N + m] = jf;
        }
    TriQ tq;
    tq.n = g->quad.n;
    for (int i = 0; i < 25; i++) tq.l1[i] = g->quad.l1[i], tq.l2[i] = g->quad.l2[i], tq.w[i] = g->quad.w[i];
    const size_t NN = (size_t)N * N;
    DevBuf dS, dW, dT, dInfo, dOut;
    BEM_TRY(dS.alloc(ctx, (size_t)n * n * sizeof(double2)));
    BEM_TRY(dW.alloc(ctx, 4 * NN * sizeof(double2)));
    BEM_TRY(dT.alloc(ctx, 2 * (size_t)n * ncols * sizeof(double2)));
    BEM_TRY(dInfo.alloc(ctx, (hinfo.size() + 4 * (size_t)N) * sizeof(int)));
    // far field: the orientations in up to GFF_SPLIT parts, summed in order
    const int ff_parts = std::min(n_orient, GFF_SPLIT);
    const size_t out_dbl = 3 * (size_t)nt * 9 + 10 * (size_t)nt + (size_t)n * 9;
    BEM_TRY(dOut.alloc(ctx, (out_dbl + (size_t)ff_parts * nt * 9) * sizeof(double)));
    int* d_hinfo = (int*)dInfo.p;
    int* d_htri = d_hinfo + hinfo.size();
    int* d_hjf = d_htri + 2 * N;
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(d_hinfo, hinfo.data(), hinfo.size() * 4, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(d_htri, htri.data(), htri.size() * 4, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(d_hjf, hjf.data(), hjf.size() * 4, cudaMemcpyHostToDevice, st));
    // S = (Lam Xd^T + Xd Lam^T) / 2, Xd = D X
    double2* LT = (double2*)dT.p;
    double2* XT = LT + (size_t)n * ncols;
    const int64_t nx = (int64_t)n * ncols;
    transpose_flip_kernel<<<nblocks(nx, 256), 256, 0, st>>>((const double2*)Lam, n, n, ncols, n, LT);
    BEM_LAUNCHED(ctx);
    transpose_flip_kernel<<<nblocks(nx, 256), 256, 0, st>>>((const double2*)X, n, n, ncols, N, XT);
    BEM_LAUNCHED(ctx);
    double2* S = (double2*)dS.p;
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(S, 0, (size_t)n * n * sizeof(double2), st));
    BEM_TRY(cgemm<double>(ctx, n, n, ncols, LT, ncols, XT, ncols, true, S, n, false, make_double2(0.5, 0),
                          make_double2(1, 0)));
    BEM_TRY(cgemm<double>(ctx, n, n, ncols, XT, ncols, LT, ncols, true, S, n, false, make_double2(0.5, 0),
                          make_double2(1, 0)));
    double2* W = (double2*)dW.p;
    weights_kernel<<<nblocks((int64_t)NN, 256), 256, 0, st>>>(S, N, eta_e, eta_i, W, W + NN, W + 2 * NN, W + 3 * NN);
    BEM_LAUNCHED(ctx);
    GradWeights gw{W, W + NN, W + 2 * NN, W + 3 * NN, N};
    double* o_pair = (double*)dOut.p;
    double* o_self = o_pair + (size_t)nt * 9;
    double* o_skp = o_self + (size_t)nt * 9;
    double* o_sep = o_skp + 2 * (size_t)nt;
    double* o_sks = o_sep + 2 * (size_t)nt;
    double* o_ses = o_sks + 4 * (size_t)nt;
    double* o_rhs = o_ses + 2 * (size_t)nt;
    double* o_ff = o_rhs + (size_t)n * 9;
    const Medium ke{kext.real(), kext.imag()}, ki{kint.real(), kint.imag()};
    PairArgs pa{g->sing.tv, d_hinfo, nt, Nq, tq, ke, ki, gw, o_pair, o_skp, o_sep};
    // the branch-free functions where no phase can leave their range
    const bool bounded = std::max(std::abs(ke.kr), std::abs(ki.kr)) * g->extent < SINCOS_MAX && ke.ki == 0 && ki.ki >= 0;
    auto pair = !bounded ? grad_pair_kernel<3, false> : ki.ki != 0 ? grad_pair_kernel<2, true> : grad_pair_kernel<0, true>;
    const size_t pair_smem = (size_t)3 * GP_W * GP_THREADS * sizeof(double);
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(pair, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pair_smem));
    pair<<<nt, GP_THREADS, pair_smem, st>>>(pa);
    BEM_LAUNCHED(ctx);
    SelfArgs sa{g->sing.tv, d_hinfo, nt, Nq, tq, ke, ki, flags, gw, o_self, o_sks, o_ses};
    grad_self_kernel<<<nblocks(nt, SELF_TRI), SELF_EVALS * SELF_TRI, 0, st>>>(sa);
    BEM_LAUNCHED(ctx);
    HalfArgs ha{g->sing.tv, d_htri, d_hjf, N, Nq, tq, kext.real(), kext.imag(), eta_e, RT_dev, n_orient,
                (const double2*)Lam, n, o_rhs};
    grad_rhs_kernel<<<nblocks(n, 64), 64, 0, st>>>(ha);
    BEM_LAUNCHED(ctx);
    double* d_part = (double*)dOut.p + out_dbl;
    FFArgs2 fa{g->sing.tv, d_hinfo, nt, N, Nq, tq, kext.real(), kext.imag(), eta_e, RT_dev, n_orient, ntheta,
               (const double2*)ab_dev, (const double2*)X, n, d_part};
    const size_t smem = std::max((size_t)ntheta * 5 * 16, (size_t)GFF_THREADS * 13 * 8);
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(grad_ff_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           ADJ_MAX_ANGLES * 5 * 16));  // the largest size: the limit is the device's
    grad_ff_kernel<<<dim3(nblocks(nt, GFF_THREADS / Nq), ff_parts), GFF_THREADS, smem, st>>>(fa);
    BEM_LAUNCHED(ctx);
    part_sum_kernel<<<nblocks(9 * (int64_t)nt, 256), 256, 0, st>>>(d_part, ff_parts, 9 * nt, o_ff);
    BEM_LAUNCHED(ctx);
    std::vector<double> out(out_dbl);
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(out.data(), dOut.p, out_dbl * 8, cudaMemcpyDeviceToHost, st));
    BEM_TRY_CUDA(ctx, cudaStreamSynchronize(st));
    const double* h_pair = out.data();
    const double* h_self = h_pair + (size_t)nt * 9;
    const double* h_skp = h_self + (size_t)nt * 9;
    const double* h_sep = h_skp + 2 * (size_t)nt;
    const double* h_sks = h_sep + 2 * (size_t)nt;
    const double* h_ses = h_sks + 4 * (size_t)nt;
    const double* h_rhs = h_ses + 2 * (size_t)nt;
    const double* h_ff = h_rhs + (size_t)n * 9;
    if (grad_v) {
        std::fill(grad_v, grad_v + 3 * (size_t)nv, 0.0);
        for (int t = 0; t < nt; t++)
            for (int j = 0; j < 3; j++)
                for (int c = 0; c < 3; c++)
                    grad_v[3 * (size_t)M.tris[3 * t + j] + c] +=
                        h_ff[9 * t + 3 * j + c] - (h_pair[9 * t + 3 * j + c] + h_self[9 * t + 3 * j + c]);
        for (int hn = 0; hn < n; hn++) {
            const int t = htri[hn];
            for (int j = 0; j < 3; j++)
                for (int c = 0; c < 3; c++)
                    grad_v[3 * (size_t)M.tris[3 * t + j] + c] += h_rhs[9 * (size_t)hn + 3 * j + c];
        }
    }
    // pair terms are holomorphic in k: d/dIm k = i d/dRe k
    double skr[2] = {0, 0}, ski[2] = {0, 0}, se[2] = {0, 0};
    for (int t = 0; t < nt; t++) {
        skr[0] += h_skp[2 * t] + h_sks[4 * t], skr[1] += h_skp[2 * t + 1] + h_sks[4 * t + 1];
        ski[0] += -h_skp[2 * t + 1] + h_sks[4 * t + 2], ski[1] += h_skp[2 * t] + h_sks[4 * t + 3];
        se[0] += h_sep[2 * t] + h_ses[2 * t], se[1] += h_sep[2 * t + 1] + h_ses[2 * t + 1];
    }
    if (dpsi_dk) dpsi_dk[0] = skr[0], dpsi_dk[1] = skr[1], dpsi_dk[2] = ski[0], dpsi_dk[3] = ski[1];
    if (dpsi_deta) dpsi_deta[0] = se[0], dpsi_deta[1] = se[1];
    return BEM_OK;
}

}  // namespace bem
