// Adjoint gradient of an orientation-averaged M11 misfit with respect to the
// relative refractive index m = m_re + i m_im.
//
//   loss = sum_t wt_t (M11(theta_t) - target_t)^2
//
// One FP64 forward solve X = Z^-1 B, the far field F of every column, the
// adjoint right-hand sides g_c = dloss/dx_c (an adjoint far-field kernel),
// one adjoint solve with the same factors (the PMCHWT Z satisfies
// Z^T = D Z D, D = diag(I, -I), so Z^-T g = D Z^-1 D g), and the operator
// derivatives dZ/dm_re, dZ/dm_im from central differences of the assembled Z
// in m (the exterior blocks cancel exactly):
//   dloss/dp = -Re sum_c lambda_c^T (dZ/dp) x_c,   lambda = Z^-T g.
// The reference has no gradient code; this follows its forward path (the
// dense branch of main.cpp:660-854) and is checked against central
// differences of that forward path.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "bem_internal.h"
#include "lu_internal.h"

namespace bem {

constexpr double INV4PI_G = 0.07957747154594767;  // 1 / (4 pi)

struct AdjFFArgs {
    int nt, N, Nq, ntheta;
    double kr, ki, eta;
    const double *c, *u, *jw, *pi;  // triangle data of the assembly (DevTriAsm)
    const int* tri_half;            // nt x 3 halves h N + n, -1 padded
    const double* coef;             // 2N: sign l / (2A) of a half
    const double* RT;               // n_orient * 9
    const double2* ab;              // [c][theta][2]: the adjoint weight's components A, B
    double2* G;                     // column-major n x ncols, zeroed before the launch
    int64_t ldg;
};

// Adjoint far field by triangles.  The weight of a direction is transverse,
// h = A e_par + B e_perp, with e_par = e1 cos t - e2 sin t, e_perp = e3 and
// rhat = e1 sin t + e2 cos t in the orientation's frame (e1 = R^T x,
// e2 = R^T z, e3 = R^T y), so rhat x h = A e3 - B e_par and six complex sums
// over the directions,
//   sum ph A (1, cos t, sin t) and sum ph B (1, cos t, sin t),
// ph = exp(-ik rhat.r), give both sum ph h and sum ph rhat x h at a point.
// Thread: one quadrature point of a triangle, both polarisations of the
// orientation blockIdx.y; the phase is taken once for them and for the three
// RWG halves of the triangle, 6 x fewer exponentials than per RWG half and
// column.  An RWG's entry is the sum of its two halves' terms, added to a
// zeroed G: 0 + x + y, the same in either order.  C5 (2N = 3840, 64
// orientations, 181 angles): 2.77 ms per half and column before.
constexpr int AFF_THREADS = 128;
__global__ void __launch_bounds__(AFF_THREADS) farfield_adjoint_kernel(AdjFFArgs a) {
    extern __shared__ __align__(16) double sm[];
    double2* s_t = (double2*)sm;           // ntheta: sin, cos
    double2* s_ab = s_t + a.ntheta;        // ntheta x 4: A0 B0 A1 B1
    double* s_red = sm;                    // AFF_THREADS x 25, after the sums
    const int o = blockIdx.y, tid = threadIdx.x, Nq = a.Nq, per = AFF_THREADS / Nq;
    for (int t = tid; t < a.ntheta; t += blockDim.x) {
        double st, ct;
        sincos(a.ntheta > 1 ? M_PI * t / (a.ntheta - 1) : 0.0, &st, &ct);
        s_t[t] = make_double2(st, ct);
        for (int pol = 0; pol < 2; pol++)
            for (int k = 0; k < 2; k++) s_ab[4 * t + 2 * pol + k] = a.ab[((size_t)(2 * o + pol) * a.ntheta + t) * 2 + k];
    }
    __syncthreads();
    const int tl = tid / Nq, q = tid % Nq, tri = blockIdx.x * per + tl;
    const bool act = tl < per && tri < a.nt;
    double e1[3], e2[3], e3[3];
    const double* R = a.RT + 9 * o;
    for (int i = 0; i < 3; i++) e1[i] = R[3 * i], e3[i] = R[3 * i + 1], e2[i] = R[3 * i + 2];
    double u[3] = {0, 0, 0};
    double sA[2][3][2], sB[2][3][2];
#pragma unroll
    for (int pol = 0; pol < 2; pol++)
#pragma unroll
        for (int k = 0; k < 3; k++) sA[pol][k][0] = sA[pol][k][1] = sB[pol][k][0] = sB[pol][k][1] = 0.0;
    if (act) {
        double x1 = 0.0, x2 = 0.0;
        for (int i = 0; i < 3; i++) {
            u[i] = a.u[((size_t)tri * Nq + q) * 3 + i];
            const double r = a.c[3 * (size_t)tri + i] + u[i];
            x1 += e1[i] * r, x2 += e2[i] * r;
        }
        for (int t = 0; t < a.ntheta; t++) {
            const double st = s_t[t].x, ct = s_t[t].y, rd = st * x1 + ct * x2;
            double sn, cs;
            sincos(a.kr * rd, &sn, &cs);
            const double ea = a.ki != 0.0 ? exp(a.ki * rd) : 1.0;
            const double er = cs * ea, ei = -sn * ea;
#pragma unroll
            for (int pol = 0; pol < 2; pol++) {
                const double2 A = s_ab[4 * t + 2 * pol], B = s_ab[4 * t + 2 * pol + 1];
                const double ar = er * A.x - ei * A.y, ai = er * A.y + ei * A.x;
                const double br = er * B.x - ei * B.y, bi = er * B.y + ei * B.x;
                sA[pol][0][0] += ar, sA[pol][0][1] += ai;
                sA[pol][1][0] += ct * ar, sA[pol][1][1] += ct * ai;
                sA[pol][2][0] += st * ar, sA[pol][2][1] += st * ai;
                sB[pol][0][0] += br, sB[pol][0][1] += bi;
                sB[pol][1][0] += ct * br, sB[pol][1][1] += ct * bi;
                sB[pol][2][0] += st * br, sB[pol][2][1] += st * bi;
            }
        }
    }
    __syncthreads();
    // the point's term of every (half, polarisation, J / M): f w . sum ph h and f w . sum ph (rhat x h)
    if (act) {
        const double w = a.jw[(size_t)tri * Nq + q];
        for (int k = 0; k < 3; k++) {
            const int hn = a.tri_half[3 * (size_t)tri + k];
            double f1 = 0, f2 = 0, f3 = 0;
            if (hn >= 0) {
                const double s = a.coef[hn] * w;
                for (int i = 0; i < 3; i++) {
                    const double f = s * (u[i] - a.pi[3 * (size_t)hn + i]);
                    f1 += f * e1[i], f2 += f * e2[i], f3 += f * e3[i];
                }
            }
#pragma unroll
            for (int pol = 0; pol < 2; pol++)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    double* out = s_red + (size_t)tid * 25 + (k * 2 + pol) * 4 + c;
                    out[0] = f1 * sA[pol][1][c] - f2 * sA[pol][2][c] + f3 * sB[pol][0][c];
                    out[2] = f3 * sA[pol][0][c] - f1 * sB[pol][1][c] + f2 * sB[pol][2][c];
                }
        }
    }
    __syncthreads();
    // -ik/(4 pi) = (k_im - i k_re)/(4 pi); the J part also carries eta
    const double pr = a.ki * INV4PI_G, pim = -a.kr * INV4PI_G;
    for (int e = tid; e < per * 12; e += blockDim.x) {
        const int t = blockIdx.x * per + e / 12, v = e % 12, k = v / 4, pol = (v / 2) % 2, jm = v % 2;
        if (t >= a.nt) break;
        const int hn = a.tri_half[3 * (size_t)t + k];
        if (hn < 0) continue;
        double gr = 0.0, gi = 0.0;
        for (int p = 0; p < Nq; p++) {
            const double* in = s_red + (size_t)((e / 12) * Nq + p) * 25 + (k * 2 + pol) * 4 + 2 * jm;
            gr += in[0], gi += in[1];
        }
        const double sc = jm == 0 ? a.eta : 1.0;
        double2* out = &a.G[(int64_t)(2 * o + pol) * a.ldg + (int64_t)jm * a.N + hn % a.N];
        atomicAdd(&out->x, sc * (pr * gr - pim * gi));
        atomicAdd(&out->y, sc * (pr * gi + pim * gr));
    }
}

// partial[b] = sum over this block's entries of L[i] R[i] (complex, no conjugate)
__global__ void cdot_kernel(const double2* __restrict__ L, const double2* __restrict__ R, int64_t count,
                            double2* __restrict__ partial) {
    __shared__ double sr[256], si[256];
    double ar = 0, ai = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 l = L[i], r = R[i];
        ar += l.x * r.x - l.y * r.y;
        ai += l.x * r.y + l.y * r.x;
    }
    sr[threadIdx.x] = ar;
    si[threadIdx.x] = ai;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sr[threadIdx.x] += sr[threadIdx.x + o];
            si[threadIdx.x] += si[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(sr[0], si[0]);
}

// rows [r0, n) of every column negated (D = diag(I, -I) applied to a block)
__global__ void flip_rows_kernel(double2* __restrict__ X, int64_t ldx, int r0, int n, int ncols) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int m = n - r0;
    if (t >= (int64_t)m * ncols) return;
    const int r = r0 + (int)(t % m), c = (int)(t / m);
    double2 v = X[(int64_t)c * ldx + r];
    X[(int64_t)c * ldx + r] = make_double2(-v.x, -v.y);
}

// Y = A - B elementwise, scaled by s
__global__ void diff_scale_kernel(const double2* __restrict__ A, const double2* __restrict__ B, double s,
                                  double2* __restrict__ Y, int64_t count) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    Y[i] = make_double2((A[i].x - B[i].x) * s, (A[i].y - B[i].y) * s);
}

namespace {
struct DevMem {
    void* p = nullptr;
    ~DevMem() {
        if (p) cudaFree(p);
    }
};
unsigned blocks_for(int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, 1 << 30); }
}  // namespace

}  // namespace bem

using namespace bem;

// Forward solve, adjoint solve, then the requested gradients: with respect to
// (Re m, Im m) (grad_m, 2 values) and/or the vertex coordinates (grad_v, 3 nv
// values).  The vertex derivatives use, per coordinate, the operator, the
// right-hand sides and the far field (at fixed coefficients) assembled on
// the geometry moved by +-h:
//   dloss/dv = Re sum_c lambda_c^T (dB_c/dv - dZ/dv x_c) + dloss/dv|_x
static int adjoint_core(bem_ctx* ctx, const bem_problem* p, const double* target, const double* wt,
                        double* loss_out, double* grad_out, double* grad_v, double* mueller_out) {
    if (!ctx || !p || !target || !loss_out || (!grad_out && !grad_v)) return BEM_ERR_INVALID;
    if (!(p->ka > 0) || p->ntheta < 2) return fail(ctx, BEM_ERR_INVALID, "ka must be > 0, ntheta >= 2");
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    const std::complex<double> m(p->m_re, p->m_im), kext(p->ka, 0.0);
    const double eta_e = 1.0;
    bem_geom* g = nullptr;
    int N = 0;
    BEM_TRY(bem_geom_create(ctx, p->verts, p->nv, p->tris, p->nt, p->quad_order, &g, &N));
    struct GeomGuard {
        bem_geom* g;
        ~GeomGuard() { bem_geom_free(g); }
    } gg{g};
    const int n = 2 * N;
    std::vector<double> RT, w;
    if (p->single) {
        RT = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        w = {1.0};
    } else {
        orientations(p->n_alpha, p->n_beta, p->n_gamma, p->beta_sym < 1 ? 1 : p->beta_sym,
                     p->gamma_sym < 1 ? 1 : p->gamma_sym, p->gamma_mirror != 0, true, RT, w);
    }
    const int no = (int)w.size(), nc = 2 * no, nt = p->ntheta;
    const size_t zb = (size_t)n * n * 16, xb = (size_t)n * nc * 16;
    const bool fd = ctx->grad_method == 1;  // derivatives of reassembled operators (else the contraction kernels)
    DevMem dZ, dZp, dX, dB, dL, dY;
    if (cudaMalloc(&dZ.p, zb) != cudaSuccess || (fd && cudaMalloc(&dZp.p, zb) != cudaSuccess) ||
        cudaMalloc(&dX.p, xb) != cudaSuccess || cudaMalloc(&dB.p, xb) != cudaSuccess ||
        cudaMalloc(&dL.p, xb) != cudaSuccess || cudaMalloc(&dY.p, xb) != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, BEM_ERR_OOM, "gradient buffers for n=%d, %d columns", n, nc);
    }
    auto assemble_m = [&](std::complex<double> mm, void* Zout) {
        const std::complex<double> ki = kext * mm;
        return assemble_dev(ctx, g, kext.real(), kext.imag(), ki.real(), ki.imag(), eta_e, 1.0 / std::abs(mm),
                            p->asm_flags, 2, Zout, n, nullptr, nullptr);
    };
    // forward solve (FP64)
    BEM_TRY(assemble_m(m, dZ.p));
    BEM_TRY(rhs_dev(ctx, g, kext.real(), kext.imag(), eta_e, RT.data(), nullptr, nullptr, no, dB.p, n));
    // the vertex derivatives reassemble only the tiles around a moved vertex
    // into a copy of the unperturbed operator
    DevMem dZbase;
    if (grad_v && fd) {
        if (cudaMalloc(&dZbase.p, zb) != cudaSuccess) {
            cudaGetLastError();
            return fail(ctx, BEM_ERR_OOM, "gradient buffers for n=%d", n);
        }
        BEM_TRY_CUDA(ctx, cudaMemcpyAsync(dZbase.p, dZ.p, zb, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    bem_lu* lu = nullptr;
    int info = 0;
    BEM_TRY(bem_lu_factor_dev(ctx, dZ.p, n, n, BEM_PREC_FP64, &lu, &info));
    struct LuGuard {
        bem_lu* lu;
        ~LuGuard() { bem_lu_free(lu); }
    } lg{lu};
    if (info > 0) return fail(ctx, BEM_ERR_SINGULAR, "zero pivot at %d", info);
    BEM_TRY(bem_lu_solve_dev(ctx, lu, dB.p, n, dX.p, n, nc, 0.0, 0, nullptr));
    // far field of every column and the averaged Mueller matrix
    std::vector<double> M(16 * (size_t)nt), Fv((size_t)nc * nt * 3 * 2);
    BEM_TRY(mueller_dev(ctx, g, dX.p, n, RT.data(), w.data(), no, kext.real(), kext.imag(), eta_e, nt,
                        p->gamma_mirror, M.data(), nullptr, Fv.data()));
    auto misfit = [&](const double* MM) {
        double l = 0.0;
        for (int t = 0; t < nt; t++) {
            const double wtt = wt ? wt[t] : 1.0, r = MM[t] - target[t];
            l += wtt * r * r;
        }
        return l;
    };
    const double loss = misfit(M.data());
    std::vector<double> coef(nt);
    for (int t = 0; t < nt; t++) coef[t] = 2.0 * (wt ? wt[t] : 1.0) * (M[t] - target[t]);
    // adjoint weights h_c(theta) = coef w_o sum_{e in (e_par, e_perp)} conj(F.e) e: their two components
    std::vector<double> ab((size_t)nc * nt * 2 * 2);
    for (int c = 0; c < nc; c++) {
        const int o = c / 2;
        const double* R = RT.data() + 9 * o;
        for (int t = 0; t < nt; t++) {
            const double th = M_PI * t / (nt - 1), st = std::sin(th), ct = std::cos(th);
            const double* F = Fv.data() + ((size_t)c * nt + t) * 6;
            const double s = coef[t] * w[o];
            double ar = 0, ai = 0, br = 0, bi = 0;
            for (int i = 0; i < 3; i++) {
                const double ep = R[3 * i] * ct - R[3 * i + 2] * st, ee = R[3 * i + 1];
                ar += F[2 * i] * ep, ai += F[2 * i + 1] * ep;
                br += F[2 * i] * ee, bi += F[2 * i + 1] * ee;
            }
            double* q = ab.data() + ((size_t)c * nt + t) * 4;
            q[0] = s * ar, q[1] = -s * ai, q[2] = s * br, q[3] = -s * bi;
        }
    }
    DevMem dAB, dRT, dPart;
    const size_t hb = ab.size() * 8;
    if (cudaMalloc(&dAB.p, hb) != cudaSuccess || cudaMalloc(&dRT.p, RT.size() * 8) != cudaSuccess ||
        cudaMalloc(&dPart.p, 1024 * 16) != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, BEM_ERR_OOM, "gradient weights");
    }
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(dAB.p, ab.data(), hb, cudaMemcpyHostToDevice, ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(dRT.p, RT.data(), RT.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
    AdjFFArgs aa{};
    aa.nt = g->nt;
    aa.N = N;
    aa.Nq = g->Nq;
    aa.ntheta = nt;
    aa.kr = kext.real();
    aa.ki = kext.imag();
    aa.eta = eta_e;
    aa.c = g->tri.c;
    aa.u = g->tri.u;
    aa.jw = g->tri.jw;
    aa.pi = g->tri.pi;
    aa.tri_half = g->tri.tri_half;
    aa.coef = g->sing_coef;
    aa.RT = (const double*)dRT.p;
    aa.ab = (const double2*)dAB.p;
    aa.G = (double2*)dY.p;  // g
    aa.ldg = n;
    // ntheta x (1 + 4) complex, reused by the 25 values of a thread
    if (nt > ADJ_MAX_ANGLES) return fail(ctx, BEM_ERR_INVALID, "ntheta %d too large for the adjoint far field", nt);
    const size_t smem = std::max((size_t)nt * 5 * 16, (size_t)AFF_THREADS * 25 * 8);
    // the limit is the device's, shared with other host threads' contexts: always the largest size
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(farfield_adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           ADJ_MAX_ANGLES * 5 * 16));
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(dY.p, 0, xb, ctx->stream));
    const int per = AFF_THREADS / g->Nq;
    farfield_adjoint_kernel<<<dim3((g->nt + per - 1) / per, no), AFF_THREADS, smem, ctx->stream>>>(aa);
    BEM_LAUNCHED(ctx);
    // lambda = D Z^-1 D g
    const int64_t half = (int64_t)(n - N) * nc;
    flip_rows_kernel<<<blocks_for(half), 256, 0, ctx->stream>>>((double2*)dY.p, n, N, n, nc);
    BEM_LAUNCHED(ctx);
    BEM_TRY(bem_lu_solve_dev(ctx, lu, dY.p, n, dL.p, n, nc, 0.0, 0, nullptr));
    flip_rows_kernel<<<blocks_for(half), 256, 0, ctx->stream>>>((double2*)dL.p, n, N, n, nc);
    BEM_LAUNCHED(ctx);
    // sum over all entries of lambda . Y (complex, no conjugate)
    std::vector<double> part(2048);
    auto dot_lambda = [&](const void* Y, double* re) {
        cdot_kernel<<<1024, 256, 0, ctx->stream>>>((const double2*)dL.p, (const double2*)Y, (int64_t)n * nc,
                                                  (double2*)dPart.p);
        BEM_LAUNCHED(ctx);
        BEM_TRY_CUDA(ctx, cudaMemcpyAsync(part.data(), dPart.p, 1024 * 16, cudaMemcpyDeviceToHost, ctx->stream));
        BEM_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        double tr = 0;
        for (int i = 0; i < 1024; i++) tr += part[2 * i];
        *re = tr;
        return (int)BEM_OK;
    };
    if (!fd) {
        // the contraction kernels (grad_geom.cu): vertex gradient, and the
        // interior wavenumber / impedance contractions for m
        const double am = std::abs(m), am3 = am * am * am;
        double dk[4] = {0, 0, 0, 0}, deta[2] = {0, 0};
        BEM_TRY(adjoint_geometry(ctx, g, kext, kext * m, eta_e, 1.0 / am, p->asm_flags, dX.p, dL.p, nc,
                                 (const double*)dRT.p, no, dAB.p, nt, grad_v, dk, deta));
        if (grad_out) {
            // k_i = k_e m with k_e real: d/dRe m = k_e d/dRe k_i, d/dIm m = k_e d/dIm k_i;
            // eta_i = 1/|m|
            grad_out[0] = -(kext.real() * dk[0] + (-m.real() / am3) * deta[0]);
            grad_out[1] = -(kext.real() * dk[2] + (-m.imag() / am3) * deta[0]);
        }
        *loss_out = loss;
        if (mueller_out) std::memcpy(mueller_out, M.data(), M.size() * 8);
        return BEM_OK;
    }
    // dZ/dp by central differences in m, contracted with lambda and x
    const double delta = 1e-5;
    for (int comp = 0; grad_out && comp < 2; comp++) {
        const std::complex<double> dm = comp == 0 ? std::complex<double>(delta, 0) : std::complex<double>(0, delta);
        BEM_TRY(assemble_m(m + dm, dZ.p));
        BEM_TRY(assemble_m(m - dm, dZp.p));
        const int64_t nn = (int64_t)n * n;
        diff_scale_kernel<<<blocks_for(nn), 256, 0, ctx->stream>>>((const double2*)dZ.p, (const double2*)dZp.p,
                                                                  0.5 / delta, (double2*)dZ.p, nn);
        BEM_LAUNCHED(ctx);
        // Y = -dZ X, then t = sum lambda . Y = -sum lambda^T dZ x
        BEM_TRY_CUDA(ctx, cudaMemsetAsync(dY.p, 0, xb, ctx->stream));
        BEM_TRY(cgemm<double>(ctx, n, nc, n, (const double2*)dZ.p, n, (const double2*)dX.p, n, true, (double2*)dY.p,
                              n, true, make_double2(-1, 0), make_double2(1, 0)));
        double tr = 0;
        BEM_TRY(dot_lambda(dY.p, &tr));
        grad_out[comp] = tr;  // Re(-sum lambda^T dZ x)
    }
    if (grad_v) {
        // per vertex coordinate: Z, B and the far field on the geometry moved by +-h
        const double h = 1e-6;
        std::vector<double> vp(p->verts, p->verts + 3 * (size_t)p->nv);
        std::vector<double> Mp(16 * (size_t)nt), Mm(16 * (size_t)nt);
        DevMem dBm;
        if (cudaMalloc(&dBm.p, xb) != cudaSuccess) {
            cudaGetLastError();
            return fail(ctx, BEM_ERR_OOM, "gradient buffers");
        }
        const std::complex<double> ki = kext * m;
        // RWGs around each vertex (the RWGs with a triangle on it): the
        // entries the vertex moves; assembly recomputes only their tiles
        std::vector<std::vector<int>> vrwg(p->nv);
        for (int mm = 0; mm < N; mm++)
            for (int tri : {g->rwg.tri_p[mm], g->rwg.tri_m[mm]})
                for (int k = 0; k < 3; k++) {
                    auto& vr = vrwg[p->tris[3 * tri + k]];
                    if (vr.empty() || vr.back() != mm) vr.push_back(mm);
                }
        DevMem dMask;
        if (cudaMalloc(&dMask.p, N) != cudaSuccess) {
            cudaGetLastError();
            return fail(ctx, BEM_ERR_OOM, "gradient buffers");
        }
        std::vector<unsigned char> mask(N);
        // one working geometry, moved in place per evaluation (same topology,
        // tiles and device arrays as a geometry created from the moved mesh)
        struct GeomGuard {
            bem_geom* g = nullptr;
            ~GeomGuard() {
                if (g) bem_geom_free(g);
            }
        } gw;
        {
            int Nw = 0;
            BEM_TRY(bem_geom_create(ctx, vp.data(), p->nv, p->tris, p->nt, p->quad_order, &gw.g, &Nw));
            if (Nw != N) return fail(ctx, BEM_ERR_INVALID, "working geometry has %d RWGs, not %d", Nw, N);
        }
        for (int iv = 0; iv < p->nv; iv++) {
            std::fill(mask.begin(), mask.end(), 0);
            for (int mm : vrwg[iv]) mask[mm] = 1;
            BEM_TRY_CUDA(ctx, cudaMemcpyAsync(dMask.p, mask.data(), N, cudaMemcpyHostToDevice, ctx->stream));
            for (int comp = 0; comp < 3; comp++) {
                const double v0 = vp[3 * iv + comp];
                double lpm[2] = {0, 0};
                void* Zs[2] = {dZ.p, dZp.p};
                void* Bs[2] = {dB.p, dBm.p};
                double* Ms[2] = {Mp.data(), Mm.data()};
                for (int sgn = 0; sgn < 2; sgn++) {
                    vp[3 * iv + comp] = v0 + (sgn == 0 ? h : -h);
                    bem_geom* gs = gw.g;
                    int st = geom_set_vertices(ctx, gs, vp.data());
                    if (st == BEM_OK && cudaMemcpyAsync(Zs[sgn], dZbase.p, zb, cudaMemcpyDeviceToDevice,
                                                        ctx->stream) != cudaSuccess)
                        st = fail(ctx, BEM_ERR_CUDA, "operator copy");
                    if (st == BEM_OK)
                        st = assemble_dev(ctx, gs, kext.real(), kext.imag(), ki.real(), ki.imag(), eta_e,
                                          1.0 / std::abs(m), p->asm_flags, 2, Zs[sgn], n, nullptr, nullptr,
                                          (const unsigned char*)dMask.p);
                    if (st == BEM_OK)
                        st = rhs_dev(ctx, gs, kext.real(), kext.imag(), eta_e, RT.data(), nullptr, nullptr, no,
                                     Bs[sgn], n);
                    if (st == BEM_OK)
                        st = mueller_dev(ctx, gs, dX.p, n, RT.data(), w.data(), no, kext.real(), kext.imag(), eta_e,
                                         nt, p->gamma_mirror, Ms[sgn], nullptr);
                    if (st != BEM_OK) {
                        vp[3 * iv + comp] = v0;
                        return st;
                    }
                    lpm[sgn] = misfit(Ms[sgn]);
                }
                vp[3 * iv + comp] = v0;
                const double inv2h = 0.5 / h;
                const int64_t nn = (int64_t)n * n, nx = (int64_t)n * nc;
                // -dZ/dv x
                diff_scale_kernel<<<blocks_for(nn), 256, 0, ctx->stream>>>((const double2*)dZ.p, (const double2*)dZp.p,
                                                                          inv2h, (double2*)dZ.p, nn);
                BEM_LAUNCHED(ctx);
                BEM_TRY_CUDA(ctx, cudaMemsetAsync(dY.p, 0, xb, ctx->stream));
                BEM_TRY(cgemm<double>(ctx, n, nc, n, (const double2*)dZ.p, n, (const double2*)dX.p, n, true,
                                      (double2*)dY.p, n, true, make_double2(-1, 0), make_double2(1, 0)));
                double t_z = 0, t_b = 0;
                BEM_TRY(dot_lambda(dY.p, &t_z));
                // dB/dv
                diff_scale_kernel<<<blocks_for(nx), 256, 0, ctx->stream>>>((const double2*)dB.p, (const double2*)dBm.p,
                                                                          inv2h, (double2*)dY.p, nx);
                BEM_LAUNCHED(ctx);
                BEM_TRY(dot_lambda(dY.p, &t_b));
                grad_v[3 * iv + comp] = t_z + t_b + (lpm[0] - lpm[1]) * inv2h;
            }
        }
    }
    *loss_out = loss;
    if (mueller_out) std::memcpy(mueller_out, M.data(), M.size() * 8);
    return BEM_OK;
}

extern "C" int bem_adjoint_grad(bem_ctx* ctx, const bem_problem* p, const double* target, const double* wt,
                                double* loss, double* grad, double* mueller) {
    if (!grad) return BEM_ERR_INVALID;
    return adjoint_core(ctx, p, target, wt, loss, grad, nullptr, mueller);
}

extern "C" int bem_adjoint_grad_vertices(bem_ctx* ctx, const bem_problem* p, const double* target, const double* wt,
                                         double* loss, double* grad_verts, double* mueller) {
    if (!grad_verts) return BEM_ERR_INVALID;
    return adjoint_core(ctx, p, target, wt, loss, nullptr, grad_verts, mueller);
}
