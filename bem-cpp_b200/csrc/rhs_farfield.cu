// Plane-wave right-hand sides, far field and Mueller reduction on the device.
//
// rhs_kernel       -- compute_rhs_planewave (rhs.cpp:6-64) for a batch of
//                     orientations; par and perp share the phase.
// farfield_kernel  -- farfield_batch_kernel (farfield.cu:100-262) for both
//                     polarisations of an orientation at once, with the
//                     S-matrix / Mueller epilogue of main.cpp:811-845 and
//                     amplitude_to_mueller (farfield.cu:464-508) fused.
// mueller_sum      -- deterministic weighted sum over orientations.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "asm_device.cuh"
#include "bem_internal.h"

namespace bem {

#define INV4PI_FF 0.079577471545947667884

// The dynamic shared-memory limit of a kernel belongs to the device, not to a
// context, and contexts of other host threads launch the same kernels: every
// launch here sets the largest size that the kernel can need, never its own.
constexpr int FF_MAXQ = 13;

struct RhsArgs {
    DevTriAsm ta;
    const double* coef;  // 2N: sign l / (2A) of a half
    int N, Nq, n_orient;
    double kr, ki, eta;
    const double* RT;  // n_orient * 9, row-major R^T
    const double* E0;  // optional explicit (E0, k_hat) for one wave
    double2* B;
    int64_t ldb;
};

// a . b = h + l: the products with their roundings (fused multiply-add), their
// sums with theirs (Knuth's two-sum).
__device__ __forceinline__ void dot_two(const double* a, const double* b, double* h, double* l) {
    double s = __dmul_rn(a[0], b[0]), e = __fma_rn(a[0], b[0], -s);
#pragma unroll
    for (int i = 1; i < 3; i++) {
        const double p = __dmul_rn(a[i], b[i]), t = __dadd_rn(s, p), bb = t - s;  // no contraction
        e += __fma_rn(a[i], b[i], -p) + ((s - (t - bb)) + (p - bb));
        s = t;
    }
    *h = s, *l = e;
}

// Sums and products in two doubles h + l (Knuth's two-sum, Dekker's product by a
// fused multiply-add), good to about 2^-100 of the largest term.
struct Two {
    double h, l;
};
__device__ __forceinline__ Two two_sum(double a, double b) {
    const double s = __dadd_rn(a, b), v = s - a;
    return {s, (a - (s - v)) + (b - v)};
}
__device__ __forceinline__ Two two_add(Two a, Two b) {
    const Two s = two_sum(a.h, b.h);
    return two_sum(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ Two two_mul(Two a, Two b) {
    const double p = __dmul_rn(a.h, b.h);
    return two_sum(p, __fma_rn(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}

// sin and cos of pi num / den, |num| <= 2 den, to about 2^-63: the nearest multiple
// of pi / 2 off as an integer, then the Taylor polynomials of degree 19 and 18
// with their first two terms in two doubles.
__device__ void sincospi_two(int num, int den, Two* sn, Two* cs) {
    const long long q = (4LL * num + (num >= 0 ? den : -den)) / (2LL * den);  // 2 num / den, rounded
    const double rem = (double)(2LL * num - q * den), dd = (double)den, a = rem / dd;
    const Two r = two_mul(Two{a, __fma_rn(-a, dd, rem) / dd}, Two{1.5707963267948965580, 6.1232339957367660359e-17});
    const Two z = two_mul(r, r);
    const double x = z.h;
    double p = 1.0 / 120.0 + x * (-1.0 / 5040.0 + x * (1.0 / 362880.0 + x * (-1.0 / 39916800.0 + x * (1.0 / 6227020800.0 +
               x * (-1.0 / 1307674368000.0 + x * (1.0 / 355687428096000.0 + x * (-1.0 / 121645100408832000.0)))))));
    double c = -1.0 / 720.0 + x * (1.0 / 40320.0 + x * (-1.0 / 3628800.0 + x * (1.0 / 479001600.0 +
               x * (-1.0 / 87178291200.0 + x * (1.0 / 20922789888000.0 + x * (-1.0 / 6402373705728000.0))))));
    // 1/6 and 1/24 in two doubles: 1/3 is 0.333.. + 1.85e-17
    const Two sixth = {-1.0 / 6.0, -9.2518585385429706566e-18}, t24 = {1.0 / 24.0, 2.3129646346357426642e-18};
    const Two s = two_add(r, two_mul(two_mul(r, z), two_add(sixth, Two{x * p, 0.0})));
    const Two u = two_add(two_add(Two{1.0, 0.0}, Two{-0.5 * z.h, -0.5 * z.l}),
                          two_mul(two_mul(z, z), two_add(t24, Two{x * c, 0.0})));
    const bool odd = q & 1;
    const double fs = ((q & 2) != 0) ? -1.0 : 1.0, fc = (((q + 1) & 2) != 0) ? -1.0 : 1.0;
    const Two vs = odd ? u : s, vc = odd ? s : u;
    *sn = {fs * vs.h, fs * vs.l};
    *cs = {fc * vc.h, fc * vc.l};
}

// Both polarisations of RHS_ORI orientations at a time for the 16 RWGs of an
// assembly tile, by triangles: the phase at a quadrature point is shared by
// the RWG halves of its triangle, f_h = s_h (u - pi_h), so the tile's ~16
// triangles are taken once per orientation (thread: triangle and
// orientation; E0 = sum ph w, Eu = sum ph w u into shared memory) and each RWG
// then adds s_h (Eu.e - (pi_h.e) E0) of its two halves for the four field
// vectors e (thread: RWG and orientation).  2 x fewer exponentials than per
// RWG half, and the fields are dotted once per half instead of per point.
// Bound by the FP64 pipe; the output is 4 x 16 B per (RWG, orientation).
// The phase k k_hat.r takes the triangle's centroid in two doubles and adds what
// lies between it and the point, which is short, so k_hat.r is rounded once at
// its own size: error against 64 bits 1.004 of that of the sums per RWG half at
// 2N = 15360, k rmax = 10 (1.10 with the centroids dotted plainly), for 19 of
// ~330 operations a triangle and orientation (510 -> 519 us).
// GENERAL: complex k or arguments beyond sincos_bounded (library functions).
constexpr int RHS_ORI = 16, RHS_THREADS = 288;  // 18 triangles x 16 orientations a pass
constexpr int RHS_FLD = 15;                     // k_hat and (E, H) of two polarisations
constexpr int RHS_E = 9;                        // E0, Eu of an orientation: 8, padded to an odd pitch
constexpr int RHS_TRI = RHS_ORI * RHS_E + 1;    // a triangle's, odd as well: the RWGs of a warp read without conflicts
template <bool GENERAL, int NQ>
__global__ void __launch_bounds__(RHS_THREADS, 3) rhs_kernel(RhsArgs a) {
    extern __shared__ __align__(16) double sm[];
    const int tile = blockIdx.x, tid = threadIdx.x, Nq = NQ > 0 ? NQ : a.Nq, N = a.N;
    const int ntri = a.ta.tile_ntri[tile], npol = a.E0 ? 1 : 2;
    double* s_pt = sm;                                  // ntri x Nq x 4: u, w
    double* s_c = s_pt + ASM_TRI_MAX * Nq * 4;          // ntri x 3
    double* s_f = s_c + ASM_TRI_MAX * 3;                // RHS_ORI x RHS_FLD
    double* s_E = s_f + RHS_ORI * RHS_FLD;              // ntri x RHS_TRI
    __shared__ int s_loc[ASM_TILE * 2];
    for (int e = tid; e < ntri * Nq; e += RHS_THREADS) {
        const size_t src = (size_t)a.ta.tile_tri[(size_t)tile * ASM_TRI_MAX + e / Nq] * Nq + e % Nq;
        for (int x = 0; x < 3; x++) s_pt[4 * e + x] = a.ta.u[src * 3 + x];
        s_pt[4 * e + 3] = a.ta.jw[src];
    }
    for (int e = tid; e < ntri * 3; e += RHS_THREADS) {
        s_c[e] = a.ta.c[(size_t)a.ta.tile_tri[(size_t)tile * ASM_TRI_MAX + e / 3] * 3 + e % 3];
        const int ent = a.ta.tile_ent[(size_t)tile * ASM_TRI_MAX * 3 + e];
        if (ent != 0xff) s_loc[ent] = e / 3;
    }
    // the RWG of this thread in the second phase (RHS_THREADS is a multiple of ASM_TILE)
    static_assert(RHS_THREADS % ASM_TILE == 0, "a thread keeps its RWG");
    const int sl = tid % ASM_TILE, n = a.ta.tile_rwg[(size_t)tile * ASM_TILE + sl];
    double sg[2] = {0, 0}, pi[2][3] = {{0, 0, 0}, {0, 0, 0}};
    if (n >= 0)
        for (int h = 0; h < 2; h++) {
            sg[h] = a.coef[h * N + n];
            for (int i = 0; i < 3; i++) pi[h][i] = a.ta.pi[3 * (size_t)(h * N + n) + i];
        }
    const double ieta = 1.0 / a.eta;
    for (int g0 = blockIdx.y * RHS_ORI; g0 < a.n_orient; g0 += gridDim.y * RHS_ORI) {
        const int go = min(RHS_ORI, a.n_orient - g0);
        __syncthreads();
        if (tid < go) {
            double* f = s_f + tid * RHS_FLD;
            const double* R = a.E0 ? nullptr : a.RT + 9 * (size_t)(g0 + tid);
            double kh[3];
            for (int i = 0; i < 3; i++) f[i] = kh[i] = a.E0 ? a.E0[3 + i] : R[3 * i + 2];
            for (int p = 0; p < 2; p++) {
                double* e = f + 3 + 6 * p;
                for (int i = 0; i < 3; i++) e[i] = a.E0 ? a.E0[i] : R[3 * i + p];  // R^T x, R^T y
                // H0 = k_hat x E0 / eta
                e[3] = (kh[1] * e[2] - kh[2] * e[1]) * ieta;
                e[4] = (kh[2] * e[0] - kh[0] * e[2]) * ieta;
                e[5] = (kh[0] * e[1] - kh[1] * e[0]) * ieta;
            }
        }
        __syncthreads();
        for (int it = tid; it < ntri * RHS_ORI; it += RHS_THREADS) {
            const int li = it / RHS_ORI, ol = it % RHS_ORI;
            if (ol >= go) continue;
            const double* kh = s_f + ol * RHS_FLD;
            const double kx = kh[0], ky = kh[1], kz = kh[2];
            const double* c = s_c + 3 * li;
            double s0, sc;
            dot_two(kh, c, &s0, &sc);
            double E[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int q = 0; q < Nq; q++) {
                const double2 uxy = *(const double2*)(s_pt + 4 * (li * Nq + q)),
                              uzw = *(const double2*)(s_pt + 4 * (li * Nq + q) + 2);
                const double sq = s0 + __fma_rn(kx, uxy.x, __fma_rn(ky, uxy.y, __fma_rn(kz, uzw.x, sc)));
                double sn, cs;
                if constexpr (GENERAL) {
                    sincos(a.kr * sq, &sn, &cs);
                    const double ea = exp(-a.ki * sq);
                    sn *= ea, cs *= ea;
                } else {
                    sincos_bounded(a.kr * sq, &sn, &cs);
                }
                const double pr = cs * uzw.y, pm = sn * uzw.y;
                E[0] += pr, E[1] += pm;
                E[2] += pr * uxy.x, E[3] += pm * uxy.x;
                E[4] += pr * uxy.y, E[5] += pm * uxy.y;
                E[6] += pr * uzw.x, E[7] += pm * uzw.x;
            }
            for (int i = 0; i < 8; i++) s_E[li * RHS_TRI + ol * RHS_E + i] = E[i];
        }
        __syncthreads();
        if (n < 0) continue;
        for (int ol = tid / ASM_TILE; ol < go; ol += RHS_THREADS / ASM_TILE) {
            const double* f = s_f + ol * RHS_FLD + 3;
            const double *Ep = s_E + s_loc[2 * sl] * RHS_TRI + ol * RHS_E,
                         *Em = s_E + s_loc[2 * sl + 1] * RHS_TRI + ol * RHS_E;
#pragma unroll
            for (int p = 0; p < 2; p++) {
                if (p >= npol) break;
                double2* col = a.B + (int64_t)(npol * (g0 + ol) + p) * a.ldb;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const double* v = f + 6 * p + 3 * k;
                    const double pp = pi[0][0] * v[0] + pi[0][1] * v[1] + pi[0][2] * v[2];
                    const double pm = pi[1][0] * v[0] + pi[1][1] * v[1] + pi[1][2] * v[2];
                    double2 out;
                    out.x = sg[0] * ((Ep[2] * v[0] + Ep[4] * v[1] + Ep[6] * v[2]) - pp * Ep[0]) +
                            sg[1] * ((Em[2] * v[0] + Em[4] * v[1] + Em[6] * v[2]) - pm * Em[0]);
                    out.y = sg[0] * ((Ep[3] * v[0] + Ep[5] * v[1] + Ep[7] * v[2]) - pp * Ep[1]) +
                            sg[1] * ((Em[3] * v[0] + Em[5] * v[1] + Em[7] * v[2]) - pm * Em[1]);
                    col[(int64_t)k * N + n] = out;
                }
            }
        }
    }
}

int rhs_dev(bem_ctx* ctx, const bem_geom* g, double k_re, double k_im, double eta,
            const double* RT_host, const double* E0_host, const double* khat_host, int n_orient,
            void* B, int64_t ldb) {
    if (!g || !B || ldb < 2 * g->N || n_orient < 1 || !(eta > 0))
        return fail(ctx, BEM_ERR_INVALID, "bad rhs arguments");
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    size_t bytes = RT_host ? (size_t)n_orient * 9 * 8 : 6 * 8;
    BEM_TRY(ctx->ensure_ws(bytes));
    std::vector<double> tmp(6);
    const double* src = RT_host;
    if (!RT_host) {
        for (int i = 0; i < 3; i++) tmp[i] = E0_host[i], tmp[3 + i] = khat_host[i];
        src = tmp.data();
    }
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->ws, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    RhsArgs a;
    a.ta = g->tri;
    a.coef = g->sing_coef;
    a.N = g->N;
    a.Nq = g->Nq;
    a.n_orient = RT_host ? n_orient : 1;
    a.kr = k_re;
    a.ki = k_im;
    a.eta = eta;
    a.RT = RT_host ? (const double*)ctx->ws : nullptr;
    a.E0 = RT_host ? nullptr : (const double*)ctx->ws;
    a.B = (double2*)B;
    a.ldb = ldb;
    // the largest |k_hat| of the call bounds the phases k k_hat.r
    double kh2 = 0.0;
    for (int o = 0; o < a.n_orient; o++) {
        double h2 = 0.0;
        for (int i = 0; i < 3; i++) {
            const double v = RT_host ? RT_host[9 * (size_t)o + 3 * i + 2] : khat_host[i];
            h2 += v * v;
        }
        kh2 = std::max(kh2, h2);
    }
    const bool general = k_im != 0.0 || !(std::fabs(k_re) * g->rmax * std::sqrt(kh2) < SINCOS_MAX);
    // about four waves of blocks (two a SM), each taking several groups of orientations
    const int groups = (a.n_orient + RHS_ORI - 1) / RHS_ORI;
    const int gy = std::max(1, std::min(groups, (int)((8LL * ctx->sm_count + g->tri.ntile - 1) / g->tri.ntile)));
    auto smem_bytes = [](int nq) {
        return ((size_t)ASM_TRI_MAX * (nq * 4 + 3) + RHS_ORI * RHS_FLD + (size_t)ASM_TRI_MAX * RHS_TRI) * 8;
    };
    const size_t smem = smem_bytes(g->Nq);
    auto kern = general ? rhs_kernel<true, 0> : g->Nq == 7 ? rhs_kernel<false, 7> : g->Nq == 4 ? rhs_kernel<false, 4> : rhs_kernel<false, 0>;
    if (g->Nq > FF_MAXQ) return fail(ctx, BEM_ERR_INVALID, "quadrature of %d points (at most %d)", g->Nq, FF_MAXQ);
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(FF_MAXQ)));
    kern<<<dim3(g->tri.ntile, gy), RHS_THREADS, smem, ctx->stream>>>(a);
    BEM_LAUNCHED(ctx);
    // the workspace is reused by later calls: finish before returning
    BEM_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BEM_OK;
}

// ------------------------------------------------------------- far field
struct FFArgs {
    DevHalf h;
    int N, Nq, n_orient, ndir, n_calls;
    double kr, ki, eta;
    // coefficients of call c: J at cJ + c*cs, M at cM + c*cs
    const double2* cJ;
    const double2* cM;
    int64_t cs;
    // directions: rhat (n_orient*ndir*3) or generated from RT and theta
    const double* rhat;
    const double* RT;     // n_orient*9
    const double* theta;  // ndir
    // outputs
    double2* Fv;          // n_calls*ndir*3 (optional)
    double* Mo;           // n_orient*16*ndir: w_o M_o / |k|^2 (optional)
    const double* w;      // n_orient
    int gamma_mirror;
};

// theta_d = pi d / (ndir - 1) (main.cpp:331-333) unless an array is given
__device__ __forceinline__ double theta_of(const FFArgs& a, int d) {
    return a.theta ? a.theta[d] : (a.ndir > 1 ? M_PI * d / (a.ndir - 1) : 0.0);
}

// Far-field vectors of both polarisations from the accumulated J and M
// sums, then the S matrix and the weighted Mueller matrix of the direction
// (main.cpp:785-845, amplitude_to_mueller farfield.cu:464-508).
__device__ void ff_epilogue(const FFArgs& a, int o, int d, const double* r, double (*acc)[2]) {
    // F = -ik/(4 pi) (eta (J - r (r.J)) - r x M)   (sM = -1)
    const double pfr = a.ki * INV4PI_FF, pfi = -a.kr * INV4PI_FF;
    double F[2][3][2];
    for (int pol = 0; pol < 2; pol++) {
        double (*J)[2] = &acc[6 * pol];
        double (*M)[2] = &acc[6 * pol + 3];
        double rdJ[2] = {r[0] * J[0][0] + r[1] * J[1][0] + r[2] * J[2][0],
                         r[0] * J[0][1] + r[1] * J[1][1] + r[2] * J[2][1]};
        double mc[3][2];
        for (int c = 0; c < 2; c++) {
            mc[0][c] = r[1] * M[2][c] - r[2] * M[1][c];
            mc[1][c] = r[2] * M[0][c] - r[0] * M[2][c];
            mc[2][c] = r[0] * M[1][c] - r[1] * M[0][c];
        }
        for (int x = 0; x < 3; x++) {
            double vr = a.eta * (J[x][0] - r[x] * rdJ[0]) - mc[x][0];
            double vi = a.eta * (J[x][1] - r[x] * rdJ[1]) - mc[x][1];
            F[pol][x][0] = pfr * vr - pfi * vi;
            F[pol][x][1] = pfr * vi + pfi * vr;
        }
    }
    if (a.Fv) {
        for (int pol = 0; pol < 2; pol++) {
            int c = 2 * o + pol;
            if (c >= a.n_calls) break;
            double2* out = a.Fv + ((size_t)c * a.ndir + d) * 3;
            for (int x = 0; x < 3; x++) out[x] = make_double2(F[pol][x][0], F[pol][x][1]);
        }
    }
    if (a.Mo) {
        // e_par = R^T e_theta_lab, e_perp = R^T y (main.cpp:785-799, 817-831)
        double st, ct;
        sincos(theta_of(a, d), &st, &ct);
        const double* R = a.RT + 9 * o;
        double epa[3], epe[3];
        for (int i = 0; i < 3; i++) {
            epa[i] = R[3 * i] * ct - R[3 * i + 2] * st;
            epe[i] = R[3 * i + 1];
        }
        double S[5][2];  // S1..S4 at index 1..4
        auto proj = [&](int pol, const double* e, double* out) {
            out[0] = F[pol][0][0] * e[0] + F[pol][1][0] * e[1] + F[pol][2][0] * e[2];
            out[1] = F[pol][0][1] * e[0] + F[pol][1][1] * e[1] + F[pol][2][1] * e[2];
        };
        double fp[2];
        // S = -ik F
        const double ikr = a.ki, iki = -a.kr;
        auto mulik = [&](const double* f, double* s) {
            s[0] = ikr * f[0] - iki * f[1];
            s[1] = ikr * f[1] + iki * f[0];
        };
        proj(0, epa, fp); mulik(fp, S[2]);
        proj(0, epe, fp); mulik(fp, S[4]);
        proj(1, epa, fp); mulik(fp, S[3]);
        proj(1, epe, fp); mulik(fp, S[1]);
        auto nrm = [&](int i) { return S[i][0] * S[i][0] + S[i][1] * S[i][1]; };
        // z_ij = S_i conj(S_j)
        auto zr = [&](int i, int j) { return S[i][0] * S[j][0] + S[i][1] * S[j][1]; };
        auto zi = [&](int i, int j) { return S[i][1] * S[j][0] - S[i][0] * S[j][1]; };
        double a1 = nrm(1), a2 = nrm(2), a3 = nrm(3), a4 = nrm(4);
        double M[16];
        M[0] = 0.5 * (a1 + a2 + a3 + a4);
        M[1] = 0.5 * (a2 - a1 + a4 - a3);
        M[2] = zr(2, 3) + zr(1, 4);
        M[3] = zi(2, 3) - zi(1, 4);
        M[4] = 0.5 * (a2 - a1 - a4 + a3);
        M[5] = 0.5 * (a2 + a1 - a4 - a3);
        M[6] = zr(2, 3) - zr(1, 4);
        M[7] = zi(2, 3) + zi(1, 4);
        M[8] = zr(2, 4) + zr(1, 3);
        M[9] = zr(2, 4) - zr(1, 3);
        M[10] = zr(1, 2) + zr(3, 4);
        M[11] = zi(2, 1) + zi(4, 3);
        M[12] = zi(4, 2) + zi(1, 3);
        M[13] = zi(4, 2) - zi(1, 3);
        M[14] = zi(1, 2) - zi(3, 4);
        M[15] = zr(1, 2) - zr(3, 4);
        if (a.gamma_mirror) {
            const int odd[8] = {2, 3, 6, 7, 8, 9, 12, 13};
            for (int i = 0; i < 8; i++) M[odd[i]] = 0.0;
        }
        double k2 = a.kr * a.kr + a.ki * a.ki;
        double wk = a.w[o] / k2;
        for (int i = 0; i < 16; i++) a.Mo[((size_t)o * 16 + i) * a.ndir + d] = wk * M[i];
    }
}

constexpr int FF_LANES = 4;
constexpr int FF_CHUNK = 256;  // points staged per step

// Block: dpb directions x FF_LANES point lanes; grid (direction chunks, orientations).
__global__ void __launch_bounds__(256) farfield_kernel(FFArgs a, int dpb) {
    extern __shared__ double sm[];
    double* s_p = sm;                   // FF_CHUNK * 6 : x y z wfx wfy wfz
    double2* s_c = (double2*)(sm + FF_CHUNK * 6);  // FF_CHUNK * 4 : cJ0 cM0 cJ1 cM1
    const int o = blockIdx.y;
    const int dl = threadIdx.x / FF_LANES, lane = threadIdx.x % FF_LANES;
    const int d = blockIdx.x * dpb + dl;
    const bool active = dl < dpb && d < a.ndir;
    const int c0 = 2 * o, c1 = 2 * o + 1;
    const bool has1 = c1 < a.n_calls;
    double r[3] = {0, 0, 1};
    if (active) {
        if (a.rhat) {
            const double* rr = a.rhat + ((size_t)o * a.ndir + d) * 3;
            r[0] = rr[0], r[1] = rr[1], r[2] = rr[2];
        } else {
            double st, ct;
            sincos(theta_of(a, d), &st, &ct);
            const double* R = a.RT + 9 * o;
            for (int i = 0; i < 3; i++) r[i] = R[3 * i] * st + R[3 * i + 2] * ct;
        }
    }
    double acc[12][2];
    for (int i = 0; i < 12; i++) acc[i][0] = acc[i][1] = 0.0;
    const int P = 2 * a.N * a.Nq;
    for (int base = 0; base < P; base += FF_CHUNK) {
        __syncthreads();
        for (int e = threadIdx.x; e < FF_CHUNK; e += blockDim.x) {
            int p = base + e;
            if (p < P) {
                double w = a.h.jw[p];
                s_p[e * 6 + 0] = a.h.px[p];
                s_p[e * 6 + 1] = a.h.py[p];
                s_p[e * 6 + 2] = a.h.pz[p];
                s_p[e * 6 + 3] = a.h.fx[p] * w;
                s_p[e * 6 + 4] = a.h.fy[p] * w;
                s_p[e * 6 + 5] = a.h.fz[p] * w;
                int n = (p / a.Nq) % a.N;
                s_c[e * 4 + 0] = a.cJ[(int64_t)c0 * a.cs + n];
                s_c[e * 4 + 1] = a.cM[(int64_t)c0 * a.cs + n];
                s_c[e * 4 + 2] = has1 ? a.cJ[(int64_t)c1 * a.cs + n] : make_double2(0, 0);
                s_c[e * 4 + 3] = has1 ? a.cM[(int64_t)c1 * a.cs + n] : make_double2(0, 0);
            } else {
                for (int k = 0; k < 6; k++) s_p[e * 6 + k] = 0.0;
                for (int k = 0; k < 4; k++) s_c[e * 4 + k] = make_double2(0, 0);
            }
        }
        __syncthreads();
        if (!active) continue;
        const int lim = min(FF_CHUNK, P - base);
        for (int e = lane; e < lim; e += FF_LANES) {
            const double* q = s_p + e * 6;
            double rd = r[0] * q[0] + r[1] * q[1] + r[2] * q[2];
            double sn, cs;
            sincos(a.kr * rd, &sn, &cs);
            double ea = a.ki != 0.0 ? exp(a.ki * rd) : 1.0;
            double phr = cs * ea, phi = -sn * ea;  // exp(-i k r.r')
            const double2* cc = s_c + e * 4;
            // u_k = c_k exp(-i k r.r') once per coefficient, then the real
            // weighted basis vector: 40 FP64 operations per point instead of 54
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double ur = cc[k].x * phr - cc[k].y * phi, ui = cc[k].x * phi + cc[k].y * phr;
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    acc[3 * k + x][0] += q[3 + x] * ur;
                    acc[3 * k + x][1] += q[3 + x] * ui;
                }
            }
        }
    }
    // reduce the FF_LANES lanes of each direction
    __syncthreads();
    double* red = sm;  // blockDim.x * 24
    for (int i = 0; i < 12; i++) {
        red[threadIdx.x * 24 + 2 * i] = acc[i][0];
        red[threadIdx.x * 24 + 2 * i + 1] = acc[i][1];
    }
    __syncthreads();
    if (!active || lane != 0) return;
    for (int l = 1; l < FF_LANES; l++)
        for (int i = 0; i < 24; i++) (&acc[0][0])[i] += red[(threadIdx.x + l) * 24 + i];
    ff_epilogue(a, o, d, r, acc);
}


// The same far field by triangles: the phase exp(-ik rhat.r_q) at a
// triangle's quadrature point is shared by the (up to three) RWG halves on
// it, whose basis is f_h = s_h (u - pi_h) with u = r - c_t.  Per (direction,
// triangle): E0 = sum_q ph_q w_q and Eu = sum_q ph_q w_q u_q, then for each
// coefficient column k the triangle adds alpha_k Eu + gamma_k E0 with
// alpha_k = sum_h c_kh s_h and gamma_k = -sum_h c_kh s_h pi_h (direction
// independent, formed once per block and staged chunk).  One sincos per
// triangle point instead of per RWG-half point, ~4x fewer operations.
constexpr int FT_CHUNK = 64;  // triangles staged per step

__global__ void __launch_bounds__(256) farfield_tri_kernel(FFArgs a, DevTriAsm ta, int nt, const double* coef,
                                                           int dpb) {
    extern __shared__ double sm[];
    double* s_c = sm;                                     // FT_CHUNK * 3 centroids
    double* s_u = s_c + FT_CHUNK * 3;                     // FT_CHUNK * FF_MAXQ * 3
    double* s_w = s_u + FT_CHUNK * FF_MAXQ * 3;           // FT_CHUNK * FF_MAXQ
    double2* s_al = (double2*)(s_w + FT_CHUNK * FF_MAXQ);  // FT_CHUNK * 4
    double2* s_ga = s_al + FT_CHUNK * 4;                  // FT_CHUNK * 4 * 3
    const int o = blockIdx.y, tid = threadIdx.x;
    const int dl = tid / FF_LANES, lane = tid % FF_LANES;
    const int d = blockIdx.x * dpb + dl;
    const bool active = dl < dpb && d < a.ndir;
    const int c0 = 2 * o, c1 = 2 * o + 1;
    const bool has1 = c1 < a.n_calls;
    const int N = a.N, Nq = a.Nq;
    double r[3] = {0, 0, 1};
    if (active) {
        if (a.rhat) {
            const double* rr = a.rhat + ((size_t)o * a.ndir + d) * 3;
            r[0] = rr[0], r[1] = rr[1], r[2] = rr[2];
        } else {
            double st, ct;
            sincos(theta_of(a, d), &st, &ct);
            const double* R = a.RT + 9 * o;
            for (int i = 0; i < 3; i++) r[i] = R[3 * i] * st + R[3 * i + 2] * ct;
        }
    }
    double acc[12][2];
    for (int i = 0; i < 12; i++) acc[i][0] = acc[i][1] = 0.0;
    for (int t0 = 0; t0 < nt; t0 += FT_CHUNK) {
        const int cnt = min(FT_CHUNK, nt - t0);
        __syncthreads();
        for (int e = tid; e < cnt * 3; e += blockDim.x) s_c[e] = ta.c[(size_t)t0 * 3 + e];
        for (int e = tid; e < cnt * Nq; e += blockDim.x) {
            const int tt = e / Nq, q = e % Nq;
            const size_t src = (size_t)(t0 + tt) * Nq + q;
            s_w[tt * FF_MAXQ + q] = ta.jw[src];
            for (int x = 0; x < 3; x++) s_u[(tt * FF_MAXQ + q) * 3 + x] = ta.u[src * 3 + x];
        }
        for (int e = tid; e < cnt * 4; e += blockDim.x) {
            const int tt = e / 4, k = e % 4;  // k: J0 M0 J1 M1
            const double2* src = (k & 1) ? a.cM : a.cJ;
            const int col = k < 2 ? c0 : c1;
            double2 al = make_double2(0, 0), ga[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
            if (k < 2 || has1) {
                for (int j = 0; j < 3; j++) {
                    const int hn = ta.tri_half[(size_t)(t0 + tt) * 3 + j];
                    if (hn < 0) break;
                    const double2 cc = src[(int64_t)col * a.cs + hn % N];
                    const double sg = coef[hn];
                    al.x += cc.x * sg, al.y += cc.y * sg;
                    for (int x = 0; x < 3; x++) {
                        const double sp = sg * ta.pi[(size_t)hn * 3 + x];
                        ga[x].x -= cc.x * sp, ga[x].y -= cc.y * sp;
                    }
                }
            }
            s_al[tt * 4 + k] = al;
            for (int x = 0; x < 3; x++) s_ga[(tt * 4 + k) * 3 + x] = ga[x];
        }
        __syncthreads();
        if (!active) continue;
        for (int tt = lane; tt < cnt; tt += FF_LANES) {
            const double rdc = r[0] * s_c[tt * 3] + r[1] * s_c[tt * 3 + 1] + r[2] * s_c[tt * 3 + 2];
            double E0r = 0, E0i = 0, Eu[3][2] = {{0, 0}, {0, 0}, {0, 0}};
            for (int q = 0; q < Nq; q++) {
                const double* u = &s_u[(tt * FF_MAXQ + q) * 3];
                const double rd = rdc + (r[0] * u[0] + r[1] * u[1] + r[2] * u[2]);
                double sn, cs;
                sincos(a.kr * rd, &sn, &cs);
                const double ea = a.ki != 0.0 ? exp(a.ki * rd) : 1.0;
                const double w = s_w[tt * FF_MAXQ + q];
                const double pr = cs * ea * w, pim = -sn * ea * w;  // exp(-i k rhat.r) w
                E0r += pr, E0i += pim;
#pragma unroll
                for (int x = 0; x < 3; x++) Eu[x][0] += pr * u[x], Eu[x][1] += pim * u[x];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double2 al = s_al[tt * 4 + k];
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    const double2 ga = s_ga[(tt * 4 + k) * 3 + x];
                    acc[3 * k + x][0] += al.x * Eu[x][0] - al.y * Eu[x][1] + ga.x * E0r - ga.y * E0i;
                    acc[3 * k + x][1] += al.x * Eu[x][1] + al.y * Eu[x][0] + ga.x * E0i + ga.y * E0r;
                }
            }
        }
    }
    __syncthreads();
    double* red = sm;  // blockDim.x * 24
    for (int i = 0; i < 12; i++) {
        red[tid * 24 + 2 * i] = acc[i][0];
        red[tid * 24 + 2 * i + 1] = acc[i][1];
    }
    __syncthreads();
    if (!active || lane != 0) return;
    for (int l = 1; l < FF_LANES; l++)
        for (int i = 0; i < 24; i++) (&acc[0][0])[i] += red[(tid + l) * 24 + i];
    ff_epilogue(a, o, d, r, acc);
}

// ------------------------------------------- far field from a band limit
// On the circle rhat(t) = R^T x sin t + R^T z cos t of an orientation the
// coefficient sums J(t), M(t) of a particle within rmax of the origin are
// trigonometric polynomials to rounding: exp(-ik rhat.r) =
// sum_n (-i)^n J_n(k rho) e^(in(t - phi)) with rho <= rmax (Jacobi-Anger), and
// J_n(x) falls below 1e-17 a few tens of orders past n = x.  So the sums are
// taken at 2 H equally spaced nodes of the whole circle, H that order, and
// the ntheta directions of the Mueller matrix interpolate them exactly
// (trigonometric interpolation at equispaced nodes: condition ~ log H).  For
// a real k the node t + pi costs nothing: the phase is the conjugate one and
// everything it multiplies is real or a coefficient, so E(t + pi) = conj E(t)
// per triangle, and with P = sum alpha Re Eu + gamma Re E0, Q the same with
// Im, the two nodes are P + iQ and P - iQ.  H phases per point instead of
// ntheta: 47 instead of 181 at k rmax = 16, 18 at k rmax = 1.
//
// An error of a node's angle is the same for every triangle and orientation and
// does not average out, so the node's sine and cosine and a centroid's
// projections are held in two doubles and the centroid's phase is summed in
// two.  With the weights rounded once and the nodes taken from far to near, the
// Mueller matrices are 2.7e-16 to 3.2e-16 off 80-bit sums (k rmax = 1 to 15), the
// kernel per direction 3.5e-16 to 4.3e-16.
//
// farfield_nodes_kernel is bound by the FP64 pipe (66 % busy): per (node pair,
// triangle) Nq (24 for the sine and cosine, 11) + 18 for the centroid + 96
// operations.  512 orientations at 2N = 15360: 4.37 ms, 3.90 ms with plain sums
// of the phases.  Block: FN_PAIRS node pairs x FN_LANES triangle lanes of one
// orientation, and every gridDim.z-th chunk of FN_CHUNK triangles; the parts are
// added in order by farfield_interp_kernel.
constexpr int FN_PAIRS = 16, FN_LANES = 8, FN_CHUNK = 64;
constexpr int FN_REC = 19;  // a triangle's 4 alpha and 12 gamma and its centroid's two projections, padded: odd, so the lanes' records do not conflict

template <int NQ>
__global__ void __launch_bounds__(FN_PAIRS* FN_LANES, 3)
farfield_nodes_kernel(FFArgs a, DevTriAsm ta, int nt, const double* __restrict__ coef, int H,
                      double* __restrict__ nodes) {
    extern __shared__ __align__(16) double sm[];
    const int Nq = NQ > 0 ? NQ : a.Nq;
    double2* s_p = (double2*)sm;                      // FN_CHUNK * Nq * 3: (x1, x2) of u, (w, w u_x) (w u_y, w u_z)
    double2* s_ag = s_p + FN_CHUNK * Nq * 3;          // FN_CHUNK * FN_REC: per column k alpha, gamma; the centroid's x1, x2
    const int o = blockIdx.y, tid = threadIdx.x, lane = tid % FN_LANES;
    const int j = blockIdx.x * FN_PAIRS + tid / FN_LANES;  // node pair: t_j = pi j / H and t_j + pi
    const int c0 = 2 * o, c1 = 2 * o + 1, N = a.N;
    const double* R = a.RT + 9 * (size_t)o;
    Two kst, kct;  // k times the node's sine and cosine
    sincospi_two(j, H, &kst, &kct);
    kst = two_mul(kst, Two{a.kr, 0.0}), kct = two_mul(kct, Two{a.kr, 0.0});
    const double st = kst.h, ct = kct.h;
    double P[12][2], Q[12][2];
#pragma unroll
    for (int i = 0; i < 12; i++) P[i][0] = P[i][1] = Q[i][0] = Q[i][1] = 0.0;
    for (int t0 = blockIdx.z * FN_CHUNK; t0 < nt; t0 += gridDim.z * FN_CHUNK) {
        const int cnt = min(FN_CHUNK, nt - t0);
        __syncthreads();
        for (int e = tid; e < cnt * Nq; e += FN_PAIRS * FN_LANES) {
            const size_t src = (size_t)t0 * Nq + e;
            const double ux = ta.u[src * 3], uy = ta.u[src * 3 + 1], uz = ta.u[src * 3 + 2], w = ta.jw[src];
            // R^T x . u and R^T z . u
            s_p[3 * e] = make_double2(R[0] * ux + R[3] * uy + R[6] * uz, R[2] * ux + R[5] * uy + R[8] * uz);
            s_p[3 * e + 1] = make_double2(w, w * ux);
            s_p[3 * e + 2] = make_double2(w * uy, w * uz);
        }
        for (int e = tid; e < cnt * 2; e += FN_PAIRS * FN_LANES) {
            const int k = e % 2 * 2;  // R^T x . c and R^T z . c
            const double ax[3] = {R[k], R[3 + k], R[6 + k]};
            double h, l;
            dot_two(ax, ta.c + 3 * (size_t)(t0 + e / 2), &h, &l);
            s_ag[e / 2 * FN_REC + 16 + e % 2] = make_double2(h, l);
        }
        for (int e = tid; e < cnt * 4; e += FN_PAIRS * FN_LANES) {
            const int tt = e / 4, k = e % 4;  // k: J0 M0 J1 M1
            const double2* src = ((k & 1) ? a.cM : a.cJ) + (int64_t)(k < 2 ? c0 : c1) * a.cs;
            double2 al = make_double2(0, 0), ga[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
            for (int h = 0; h < 3; h++) {
                const int hn = ta.tri_half[(size_t)(t0 + tt) * 3 + h];
                if (hn < 0) break;
                const double2 cc = src[hn >= N ? hn - N : hn];
                const double sg = coef[hn];
                al.x += cc.x * sg, al.y += cc.y * sg;
                for (int x = 0; x < 3; x++) {
                    const double sp = sg * ta.pi[(size_t)hn * 3 + x];
                    ga[x].x -= cc.x * sp, ga[x].y -= cc.y * sp;
                }
            }
            double2* rec = s_ag + tt * FN_REC + 4 * k;
            rec[0] = al;
            for (int x = 0; x < 3; x++) rec[1 + x] = ga[x];
        }
        __syncthreads();
        for (int tt = lane; tt < cnt; tt += FN_LANES) {
            double E0r = 0, E0i = 0, Eu[3][2] = {{0, 0}, {0, 0}, {0, 0}};
            const double2* pt = s_p + (size_t)tt * Nq * 3;
            // the centroid's phase x0 + x0l
            const double2 c1 = s_ag[tt * FN_REC + 16], c2 = s_ag[tt * FN_REC + 17];
            const double p1 = __dmul_rn(st, c1.x), p2 = __dmul_rn(ct, c2.x);
            const Two ph = two_sum(p1, p2);
            const double x0 = ph.h, x0l = ph.l + ((__fma_rn(st, c1.x, -p1) + __fma_rn(ct, c2.x, -p2)) +
                                                  (st * c1.y + ct * c2.y + kst.l * c1.x + kct.l * c2.x));
#pragma unroll
            for (int q = 0; q < Nq; q++) {
                const double2 x = pt[3 * q], wx = pt[3 * q + 1], yz = pt[3 * q + 2];
                double sn, cs;
                sincos_bounded(x0 + __fma_rn(st, x.x, __fma_rn(ct, x.y, x0l)), &sn, &cs);
                // exp(-i k rhat.r) = cs - i sn
                E0r += cs * wx.x, E0i -= sn * wx.x;
                Eu[0][0] += cs * wx.y, Eu[0][1] -= sn * wx.y;
                Eu[1][0] += cs * yz.x, Eu[1][1] -= sn * yz.x;
                Eu[2][0] += cs * yz.y, Eu[2][1] -= sn * yz.y;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double2 *rec = s_ag + tt * FN_REC + 4 * k, al = rec[0];
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    const double2 ga = rec[1 + x];
                    P[3 * k + x][0] += al.x * Eu[x][0] + ga.x * E0r;
                    P[3 * k + x][1] += al.y * Eu[x][0] + ga.y * E0r;
                    Q[3 * k + x][0] += al.x * Eu[x][1] + ga.x * E0i;
                    Q[3 * k + x][1] += al.y * Eu[x][1] + ga.y * E0i;
                }
            }
        }
    }
    // the lanes of a node pair are neighbours in a warp
#pragma unroll
    for (int i = 0; i < 12; i++)
#pragma unroll
        for (int c = 0; c < 2; c++)
            for (int off = FN_LANES / 2; off > 0; off >>= 1) {
                P[i][c] += __shfl_down_sync(0xffffffffu, P[i][c], off);
                Q[i][c] += __shfl_down_sync(0xffffffffu, Q[i][c], off);
            }
    if (lane != 0 || j >= H) return;
    double* out = nodes + (((size_t)blockIdx.z * a.n_orient + o) * 2 * H + j) * 24;
#pragma unroll
    for (int i = 0; i < 12; i++) {
        out[2 * i] = P[i][0] - Q[i][1];
        out[2 * i + 1] = P[i][1] + Q[i][0];
        out[(size_t)H * 24 + 2 * i] = P[i][0] + Q[i][1];
        out[(size_t)H * 24 + 2 * i + 1] = P[i][1] - Q[i][0];
    }
}

// The nodes in the order in which a direction's sums take them, from the
// farthest to the nearest: e = 0 .. 2 H - 1 -> node jc + H, then jc +- (H - 1)
// and so on to jc, the node nearest to t_d.  The weights fall off as the
// cotangent of the distance, so the partial sums stay small until the last few
// terms, and those alone round at the result's size: 0.72 of 2^-53 in the 2-norm
// against 2 (H = 17) to 3.6 (H = 48) in the order of the nodes (restated in NumPy).
__device__ __forceinline__ int ff_node(int e, int jc, int H) {
    const int k = e == 0 ? H : H - (e + 1) / 2;
    int j = (e & 1) ? jc + k : jc - k;
    if (j < 0) j += 2 * H;
    if (j >= 2 * H) j -= 2 * H;
    return j;
}
__device__ __forceinline__ int ff_nearest(int d, int H, int nd) { return (2 * d * H + nd) / (2 * nd); }

// W[e][d] of the trigonometric interpolation from the 2 H nodes t_j = pi j / H
// to the call's theta_d, j = ff_node(e, ..): sin(H x) cot(x / 2) / (2 H), x =
// theta_d - t_j.  theta_d is pi d / (ndir - 1) rounded: the weight is formed for the
// exact fraction, where x = pi m / (H (ndir - 1)) with an integer m and sin(H x) =
// +-sin(pi m / (ndir - 1)) (2 H ndir <= FF_MAX_WEIGHTS, so the integers fit 32
// bits), and corrected to first order for the rounding of theta_d.  A weight's
// error is the same for every orientation, so it is rounded once.
constexpr int FF_MAX_WEIGHTS = 1 << 27;
__global__ void ff_weights_kernel(int H, int ndir, const double* __restrict__ theta, double* __restrict__ W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * H * ndir) return;
    const int d = i % ndir, nd = ndir - 1, j = ff_node(i / ndir, ff_nearest(d, H, nd), H);
    const int per = 2 * H * nd;
    int m = (int)(((long long)d * H - (long long)j * nd) % per);  // x modulo 2 pi in (-pi, pi]
    if (m > per / 2) m -= per;
    if (m <= -per / 2) m += per;
    double w = 1.0;
    if (m != 0) {
        Two s, c, sh, ch;
        sincospi_two(m, per, &s, &c);              // x / 2
        sincospi_two(m % (2 * nd), nd, &sh, &ch);  // H x
        const Two num = two_mul(sh, c), den = two_mul(s, Two{2.0 * H, 0.0});
        const double q = num.h / den.h;
        // theta_d - pi d / nd = -(pi d - theta_d nd) / nd, and the weight's slope there
        const double th = theta[d], pd = __dmul_rn(3.1415926535897931160, (double)d);
        const double off = -((__fma_rn(-th, (double)nd, pd) + __fma_rn(3.1415926535897931160, (double)d, -pd)) +
                             1.2246467991473532072e-16 * d) / nd;
        const double slope = (ch.h * c.h * H - sh.h / (2.0 * s.h)) / den.h;
        w = q + ((__fma_rn(-q, den.h, num.h) + (num.l - q * den.l)) / den.h + off * slope);
    }
    W[i] = w;
}

// Thread: one direction of the orientation blockIdx.x; the node sums (all
// parts, in order) in shared memory, an odd number of 16-byte units apart: the
// lanes of a warp are at up to 16 neighbouring nodes.
constexpr int FF_NODE = 26, FF_MAX_H = 533, FF_INTERP_SMEM = 2 * FF_MAX_H * FF_NODE * 8;
__global__ void __launch_bounds__(192) farfield_interp_kernel(FFArgs a, const double* __restrict__ nodes, int parts,
                                                              int H, const double* __restrict__ W) {
    extern __shared__ __align__(16) double sm[];  // 2 H x FF_NODE
    const int o = blockIdx.x, cnt = 2 * H * 24;
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
        double s = 0.0;
        for (int z = 0; z < parts; z++) s += nodes[((size_t)z * a.n_orient + o) * cnt + e];
        sm[e / 24 * FF_NODE + e % 24] = s;
    }
    __syncthreads();
    const int d = blockIdx.y * blockDim.x + threadIdx.x;
    if (d >= a.ndir) return;
    double acc[12][2];
#pragma unroll
    for (int i = 0; i < 12; i++) acc[i][0] = acc[i][1] = 0.0;
    const int jc = ff_nearest(d, H, a.ndir - 1);
    for (int e = 0; e < 2 * H; e++) {
        const double w = W[(size_t)e * a.ndir + d];
        const double2* v = (const double2*)(sm + (size_t)ff_node(e, jc, H) * FF_NODE);
#pragma unroll
        for (int i = 0; i < 12; i++) {
            const double2 x = v[i];
            acc[i][0] += w * x.x, acc[i][1] += w * x.y;
        }
    }
    double st, ct, r[3];
    sincos(theta_of(a, d), &st, &ct);
    const double* R = a.RT + 9 * (size_t)o;
    for (int i = 0; i < 3; i++) r[i] = R[3 * i] * st + R[3 * i + 2] * ct;
    ff_epilogue(a, o, d, r, acc);
}

// Node pairs for the band limit: one past the first order n > x at which
// J_n(x) <= exp(n (tanh b - b)) / sqrt(2 pi n tanh b), cosh b = n / x (Debye),
// is below 1e-17.  0: more than `limit`.
static int ff_node_pairs(double x, int limit) {
    x = std::max(x, 1e-3);
    for (int n = (int)x + 2; n < limit; n++) {
        const double b = std::acosh(n / x), t = std::tanh(b);
        if (std::exp(n * (t - b)) < 1e-17 * std::sqrt(2.0 * M_PI * n * t)) return n + 1;
    }
    return 0;
}

// Plan of the band-limited far field of a call, H = 0 where the direct kernel
// takes it: a complex k (no conjugate nodes), directions of the caller,
// arguments beyond the sine's range, so many directions that their weights
// would take more than 1 GB (and the indices 32 bits), or so few that H node
// pairs and the interpolation cost more (operations per direction: Nq 33 + 96 per
// triangle either way; per node pair and direction 48 of interpolation).
// RT (host) need not be orthonormal: |rhat(t).r| <= smax |r| with smax the
// largest singular value of (R^T x, R^T z).
struct FFPlan {
    int H = 0, parts = 1;
    size_t node_bytes = 0, weight_bytes = 0;
};
static FFPlan plan_ff(const bem_ctx* ctx, const bem_geom* g, const double* RT, int n_orient, int ndir, double k_re,
                      double k_im) {
    FFPlan p;
    if (ctx->ff_kernel != 0 || k_im != 0.0 || ndir < 8 || g->Nq > FF_MAXQ) return p;
    double s2 = 0.0;
    for (int o = 0; o < n_orient; o++) {
        const double* R = RT + 9 * (size_t)o;
        double aa = 0, bb = 0, ab = 0;
        for (int i = 0; i < 3; i++)
            aa += R[3 * i] * R[3 * i], bb += R[3 * i + 2] * R[3 * i + 2], ab += R[3 * i] * R[3 * i + 2];
        s2 = std::max(s2, 0.5 * (aa + bb) + std::sqrt(0.25 * (aa - bb) * (aa - bb) + ab * ab));
    }
    const double x = std::fabs(k_re) * g->rmax * std::sqrt(s2);
    if (!(x < SINCOS_MAX)) return p;
    const int H = ff_node_pairs(x, ndir);
    const double per_dir = (g->Nq * 33.0 + 96.0) * g->nt;
    if ((int64_t)2 * H * ndir > FF_MAX_WEIGHTS) return p;
    // the interpolation's shared memory bounds H as well
    if (H < 1 || H * (per_dir + 48.0 * ndir) > per_dir * ndir || H > FF_MAX_H) return p;
    p.H = H;
    const int chunks = (H + FN_PAIRS - 1) / FN_PAIRS, tchunks = (g->nt + FN_CHUNK - 1) / FN_CHUNK;
    // three blocks of 128 threads fit an SM: enough parts for about four waves
    const int64_t want = 12LL * ctx->sm_count, have = (int64_t)chunks * n_orient;
    p.parts = (int)std::max<int64_t>(1, std::min<int64_t>(std::min(tchunks, 64), (want + have - 1) / have));
    p.node_bytes = (size_t)p.parts * n_orient * 2 * H * 24 * 8;
    p.weight_bytes = (size_t)2 * H * ndir * 8;
    return p;
}

static int launch_ff_nodes(bem_ctx* ctx, const bem_geom* g, const FFArgs& a, const FFPlan& p, double* nodes,
                           double* weights) {
    cudaEvent_t ev = ctx->prof_begin(PROF_FARFIELD);
    ff_weights_kernel<<<(2 * p.H * a.ndir + 255) / 256, 256, 0, ctx->stream>>>(p.H, a.ndir, a.theta, weights);
    BEM_LAUNCHED(ctx);
    auto kern = g->Nq == 7 ? farfield_nodes_kernel<7> : g->Nq == 4 ? farfield_nodes_kernel<4> : farfield_nodes_kernel<0>;
    const size_t smem = (size_t)FN_CHUNK * (g->Nq * 3 + FN_REC) * 16;
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           FN_CHUNK * (FF_MAXQ * 3 + FN_REC) * 16));
    kern<<<dim3((p.H + FN_PAIRS - 1) / FN_PAIRS, a.n_orient, p.parts), FN_PAIRS * FN_LANES, smem, ctx->stream>>>(
        a, g->tri, g->nt, g->sing_coef, p.H, nodes);
    BEM_LAUNCHED(ctx);
    const size_t ismem = (size_t)2 * p.H * FF_NODE * 8;
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(farfield_interp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           FF_INTERP_SMEM));
    farfield_interp_kernel<<<dim3(a.n_orient, (a.ndir + 191) / 192), 192, ismem, ctx->stream>>>(a, nodes, p.parts, p.H,
                                                                                             weights);
    BEM_LAUNCHED(ctx);
    // the unit of launch_ff: (orientation, direction, point) terms
    if (ev)
        ctx->prof_end(PROF_FARFIELD, ev, 110.0 * a.n_orient * (double)a.ndir * 2.0 * a.N * a.Nq,
                      (double)a.n_orient * a.ndir * 16 * 8);
    return BEM_OK;
}

// M_avg[i*ndir + d] = sum over o in order of Mo[o][i][d]
__global__ void mueller_sum_kernel(const double* __restrict__ Mo, int n_orient, int nel,
                                   double* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nel) return;
    double s = 0.0;
#pragma unroll 8
    for (int o = 0; o < n_orient; o++) s += Mo[(size_t)o * nel + i];
    out[i] = s;
}

static int launch_ff(bem_ctx* ctx, const bem_geom* g, FFArgs& a) {
    int nchunk = (a.ndir + 63) / 64;
    int dpb = (a.ndir + nchunk - 1) / nchunk;
    int threads = dpb * FF_LANES;  // 256 at most: no kernel here takes more than 48 KB
    static_assert(64 * FF_LANES * 24 * 8 <= 48 * 1024 &&
                      FT_CHUNK * (3 + FF_MAXQ * 4) * 8 + FT_CHUNK * 16 * 16 <= 48 * 1024 &&
                      FF_CHUNK * (6 * 8 + 4 * 16) <= 48 * 1024,
                  "far field shared memory");
    dim3 grid(nchunk, a.n_orient);
    cudaEvent_t ev = ctx->prof_begin(PROF_FARFIELD);
    if (ctx->ff_kernel == 0) {
        if (g->Nq > FF_MAXQ) return fail(ctx, BEM_ERR_INVALID, "quadrature of %d points (at most %d)", g->Nq, FF_MAXQ);
        size_t smem = std::max((size_t)FT_CHUNK * (3 + FF_MAXQ * 4) * 8 + (size_t)FT_CHUNK * 16 * 16,
                               (size_t)threads * 24 * 8);
        farfield_tri_kernel<<<grid, threads, smem, ctx->stream>>>(a, g->tri, g->nt, g->sing_coef, dpb);
    } else {
        size_t smem = std::max((size_t)FF_CHUNK * (6 * 8 + 4 * 16), (size_t)threads * 24 * 8);
        farfield_kernel<<<grid, threads, smem, ctx->stream>>>(a, dpb);
    }
    BEM_LAUNCHED(ctx);
    // algorithmic unit: one (orientation, direction, point) term, ~110 flop
    if (ev)
        ctx->prof_end(PROF_FARFIELD, ev, 110.0 * a.n_orient * (double)a.ndir * 2.0 * a.N * a.Nq,
                      (double)a.n_orient * a.ndir * 16 * 8);
    return BEM_OK;
}

int farfield_dev(bem_ctx* ctx, const bem_geom* g, const void* X, int64_t ldx, int n_calls_x,
                 const double* coeffJ_host, const double* coeffM_host, const double* rhat_host,
                 int n_orient, int ndir, double k_re, double k_im, double eta, double* Fv_host) {
    (void)X;
    (void)ldx;
    (void)n_calls_x;
    const int N = g->N;
    int n_calls = 2 * n_orient;
    size_t cb = (size_t)n_calls * N * 16, rb = (size_t)n_orient * ndir * 3 * 8,
           fb = (size_t)n_calls * ndir * 3 * 16;
    size_t off = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 255) & ~(size_t)255; return o; };
    size_t oJ = take(cb), oM = take(cb), oR = take(rb), oF = take(fb);
    BEM_TRY(ctx->ensure_ws(off));
    char* ws = (char*)ctx->ws;
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ws + oJ, coeffJ_host, cb, cudaMemcpyHostToDevice, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ws + oM, coeffM_host, cb, cudaMemcpyHostToDevice, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ws + oR, rhat_host, rb, cudaMemcpyHostToDevice, ctx->stream));
    FFArgs a{};
    a.h = g->half;
    a.N = N;
    a.Nq = g->Nq;
    a.n_orient = n_orient;
    a.ndir = ndir;
    a.n_calls = n_calls;
    a.kr = k_re;
    a.ki = k_im;
    a.eta = eta;
    a.cJ = (const double2*)(ws + oJ);
    a.cM = (const double2*)(ws + oM);
    a.cs = N;
    a.rhat = (const double*)(ws + oR);
    a.Fv = (double2*)(ws + oF);
    BEM_TRY(launch_ff(ctx, g, a));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(Fv_host, ws + oF, fb, cudaMemcpyDeviceToHost, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BEM_OK;
}

int mueller_dev(bem_ctx* ctx, const bem_geom* g, const void* X, int64_t ldx, const double* RT,
                const double* w, int n_orient, double k_re, double k_im, double eta, int ntheta,
                int gamma_mirror, double* M_avg, double* M_orient_dev, double* Fv_host) {
    const int N = g->N;
    size_t rtb = (size_t)n_orient * 9 * 8, wb = (size_t)n_orient * 8, tb = (size_t)ntheta * 8,
           mob = M_orient_dev ? 0 : (size_t)n_orient * 16 * ntheta * 8, mab = (size_t)16 * ntheta * 8,
           fvb = Fv_host ? (size_t)2 * n_orient * ntheta * 3 * 16 : 0;
    size_t off = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 255) & ~(size_t)255; return o; };
    FFPlan plan = plan_ff(ctx, g, RT, n_orient, ntheta, k_re, k_im);
    size_t oRT = take(rtb), oW = take(wb), oT = take(tb), oMo = take(mob), oMa = take(mab), oFv = take(fvb);
    const size_t direct = off;
    size_t oNd = take(plan.node_bytes), oWt = take(plan.weight_bytes);
    if (ctx->ensure_ws(off) != BEM_OK) {
        if (plan.H == 0) return BEM_ERR_OOM;
        plan = FFPlan{};  // without room for the node sums: every direction on its own
        BEM_TRY(ctx->ensure_ws(direct));
    }
    char* ws = (char*)ctx->ws;
    std::vector<double> th(ntheta);
    for (int i = 0; i < ntheta; i++) th[i] = ntheta > 1 ? M_PI * i / (ntheta - 1) : 0.0;
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ws + oRT, RT, rtb, cudaMemcpyHostToDevice, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ws + oW, w, wb, cudaMemcpyHostToDevice, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(ws + oT, th.data(), tb, cudaMemcpyHostToDevice, ctx->stream));
    FFArgs a{};
    a.h = g->half;
    a.N = N;
    a.Nq = g->Nq;
    a.n_orient = n_orient;
    a.ndir = ntheta;
    a.n_calls = 2 * n_orient;
    a.kr = k_re;
    a.ki = k_im;
    a.eta = eta;
    a.cJ = (const double2*)X;
    a.cM = (const double2*)X + N;
    a.cs = ldx;
    a.RT = (const double*)(ws + oRT);
    a.theta = (const double*)(ws + oT);
    a.w = (const double*)(ws + oW);
    a.Mo = M_orient_dev ? M_orient_dev : (double*)(ws + oMo);
    a.gamma_mirror = gamma_mirror;
    a.Fv = Fv_host ? (double2*)(ws + oFv) : nullptr;
    if (plan.H > 0)
        BEM_TRY(launch_ff_nodes(ctx, g, a, plan, (double*)(ws + oNd), (double*)(ws + oWt)));
    else
        BEM_TRY(launch_ff(ctx, g, a));
    int nel = 16 * ntheta;
    mueller_sum_kernel<<<(nel + 63) / 64, 64, 0, ctx->stream>>>(a.Mo, n_orient, nel, (double*)(ws + oMa));
    BEM_LAUNCHED(ctx);
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(M_avg, ws + oMa, mab, cudaMemcpyDeviceToHost, ctx->stream));
    if (Fv_host) BEM_TRY_CUDA(ctx, cudaMemcpyAsync(Fv_host, ws + oFv, fvb, cudaMemcpyDeviceToHost, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BEM_OK;
}

// ---------------------------------------------------- allocation-free variant
// Scratch of bem_farfield_mueller_noalloc: a file-scope device array, so the
// entry point needs no cudaMalloc.  Host code must not use the symbol as an
// address: its device address is looked up per device with
// cudaGetSymbolAddress on the first call there, which should therefore come
// before any stream capture begins.
static __device__ __align__(256) unsigned char g_noalloc_scratch[BEM_NOALLOC_SCRATCH_BYTES];
static void* g_noalloc_dev_ptr[64];
static std::mutex g_noalloc_mu;

static int noalloc_scratch(bem_ctx* ctx, void** out) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (ctx->device < 0 || ctx->device >= 64) return fail(ctx, BEM_ERR_INVALID, "device ordinal %d", ctx->device);
    if (!g_noalloc_dev_ptr[ctx->device]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);  // device is current (cudaSetDevice)
        if (e != cudaSuccess || !p)
            return fail(ctx, BEM_ERR_CUDA, "cudaGetSymbolAddress of the scratch array: %s", cudaGetErrorString(e));
        g_noalloc_dev_ptr[ctx->device] = p;
    }
    *out = g_noalloc_dev_ptr[ctx->device];
    return BEM_OK;
}

int mueller_noalloc(bem_ctx* ctx, const bem_geom* g, const void* X, int64_t ldx, const double* RT,
                    const double* w, int n_orient, double k_re, double k_im, double eta, int ntheta,
                    int gamma_mirror, double* M_out_dev) {
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    size_t rtb = al((size_t)n_orient * 9 * 8), wb = al((size_t)n_orient * 8),
           mob = al((size_t)n_orient * 16 * ntheta * 8);
    if (rtb + wb + mob > (size_t)BEM_NOALLOC_SCRATCH_BYTES)
        return fail(ctx, BEM_ERR_INVALID,
                    "%d orientations x %d angles need %zu bytes of scratch, above the %d-byte maximum of "
                    "bem_farfield_mueller_noalloc; pass fewer orientations per call and add the results",
                    n_orient, ntheta, rtb + wb + mob, (int)BEM_NOALLOC_SCRATCH_BYTES);
    void* base = nullptr;
    BEM_TRY(noalloc_scratch(ctx, &base));
    char* sc = (char*)base;
    double* d_RT = (double*)sc;
    double* d_w = (double*)(sc + rtb);
    double* d_Mo = (double*)(sc + rtb + wb);
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(d_RT, RT, (size_t)n_orient * 9 * 8, cudaMemcpyHostToDevice, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(d_w, w, (size_t)n_orient * 8, cudaMemcpyHostToDevice, ctx->stream));
    FFArgs a{};
    a.h = g->half;
    a.N = g->N;
    a.Nq = g->Nq;
    a.n_orient = n_orient;
    a.ndir = ntheta;
    a.n_calls = 2 * n_orient;
    a.kr = k_re;
    a.ki = k_im;
    a.eta = eta;
    a.cJ = (const double2*)X;
    a.cM = (const double2*)X + g->N;
    a.cs = ldx;
    a.RT = d_RT;
    a.theta = nullptr;  // computed in the kernel
    a.w = d_w;
    a.Mo = d_Mo;  // every (o, i, d) entry is written: nothing to clear
    a.gamma_mirror = gamma_mirror;
    BEM_TRY(launch_ff(ctx, g, a));
    int nel = 16 * ntheta;
    mueller_sum_kernel<<<(nel + 63) / 64, 64, 0, ctx->stream>>>(d_Mo, n_orient, nel, M_out_dev);
    BEM_LAUNCHED(ctx);
    return BEM_OK;
}

}  // namespace bem

using namespace bem;

extern "C" {

int bem_farfield_mueller_noalloc(bem_ctx* ctx, const bem_geom* g, const void* X_dev, int64_t ldx,
                                 const double* RT, const double* w, int n_orient, double k_re, double k_im,
                                 double eta_ext, int ntheta, int gamma_mirror, double* M_avg_dev) {
    if (!ctx || !g || !X_dev || !RT || !w || !M_avg_dev || n_orient < 1 || ntheta < 2 || ldx < 2 * g->N)
        return ctx ? fail(ctx, BEM_ERR_INVALID, "bad bem_farfield_mueller_noalloc arguments") : BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    return mueller_noalloc(ctx, g, X_dev, ldx, RT, w, n_orient, k_re, k_im, eta_ext, ntheta, gamma_mirror,
                           M_avg_dev);
}

int bem_rhs_planewave_dev(bem_ctx* ctx, const bem_geom* g, double k_re, double k_im, double eta_ext,
                          const double* RT, int n_orient, void* B_dev, int64_t ldb) {
    if (!ctx || !g || !RT) return BEM_ERR_INVALID;
    return rhs_dev(ctx, g, k_re, k_im, eta_ext, RT, nullptr, nullptr, n_orient, B_dev, ldb);
}

int bem_rhs_planewave(bem_ctx* ctx, const bem_geom* g, double k_re, double k_im, double eta_ext,
                      const double* E0, const double* k_hat, double* b) {
    if (!ctx || !g || !E0 || !k_hat || !b) return BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    void* d = nullptr;
    size_t bytes = (size_t)2 * g->N * 16;
    BEM_TRY_CUDA(ctx, cudaMalloc(&d, bytes));
    int s = rhs_dev(ctx, g, k_re, k_im, eta_ext, nullptr, E0, k_hat, 1, d, 2 * g->N);
    if (s == BEM_OK) s = d2h(ctx, b, d, bytes);
    cudaFree(d);
    return s;
}

int bem_farfield_batch(bem_ctx* ctx, const bem_geom* g, const double* coeffs_J, const double* coeffs_M,
                       const double* r_hats, double k_re, double k_im, double eta_ext, int n_calls,
                       int n_orient, int ndir, double* Fv) {
    if (!ctx || !g || !coeffs_J || !coeffs_M || !r_hats || !Fv || n_orient < 1 || ndir < 1 ||
        n_calls != 2 * n_orient)
        return ctx ? fail(ctx, BEM_ERR_INVALID, "bem_farfield_batch: n_calls must be 2*n_orient")
                   : BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    return farfield_dev(ctx, g, nullptr, 0, n_calls, coeffs_J, coeffs_M, r_hats, n_orient, ndir, k_re,
                        k_im, eta_ext, Fv);
}

int bem_farfield_mueller_dev(bem_ctx* ctx, const bem_geom* g, const void* X_dev, int64_t ldx,
                             const double* RT, const double* w, int n_orient, double k_re, double k_im,
                             double eta_ext, int ntheta, int gamma_mirror, double* M_avg,
                             double* M_orient_dev) {
    if (!ctx || !g || !X_dev || !RT || !w || !M_avg || n_orient < 1 || ntheta < 2 || ldx < 2 * g->N)
        return ctx ? fail(ctx, BEM_ERR_INVALID, "bad bem_farfield_mueller_dev arguments") : BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    return mueller_dev(ctx, g, X_dev, ldx, RT, w, n_orient, k_re, k_im, eta_ext, ntheta, gamma_mirror,
                       M_avg, M_orient_dev);
}

// amplitude_to_mueller (farfield.cu:464-508), host.
int bem_amplitude_to_mueller(const double* S1, const double* S2, const double* S3, const double* S4,
                             int ntheta, double* M) {
    if (!S1 || !S2 || !S3 || !S4 || !M || ntheta < 1) return BEM_ERR_INVALID;
    for (int t = 0; t < ntheta; t++) {
        const double* S[5] = {nullptr, S1 + 2 * t, S2 + 2 * t, S3 + 2 * t, S4 + 2 * t};
        auto nrm = [&](int i) { return S[i][0] * S[i][0] + S[i][1] * S[i][1]; };
        auto zr = [&](int i, int j) { return S[i][0] * S[j][0] + S[i][1] * S[j][1]; };
        auto zi = [&](int i, int j) { return S[i][1] * S[j][0] - S[i][0] * S[j][1]; };
        double a1 = nrm(1), a2 = nrm(2), a3 = nrm(3), a4 = nrm(4);
        double m[16] = {0.5 * (a1 + a2 + a3 + a4), 0.5 * (a2 - a1 + a4 - a3), zr(2, 3) + zr(1, 4),
                        zi(2, 3) - zi(1, 4),       0.5 * (a2 - a1 - a4 + a3), 0.5 * (a2 + a1 - a4 - a3),
                        zr(2, 3) - zr(1, 4),       zi(2, 3) + zi(1, 4),       zr(2, 4) + zr(1, 3),
                        zr(2, 4) - zr(1, 3),       zr(1, 2) + zr(3, 4),       zi(2, 1) + zi(4, 3),
                        zi(4, 2) + zi(1, 3),       zi(4, 2) - zi(1, 3),       zi(1, 2) - zi(3, 4),
                        zr(1, 2) - zr(3, 4)};
        for (int i = 0; i < 16; i++) M[i * ntheta + t] = m[i];
    }
    return BEM_OK;
}

}  // extern "C"
