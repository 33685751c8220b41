// Complex LU with partial pivoting and multi-RHS solves, FP64 and FP32.
//
// Replaces cusolverDnZgetrf / cusolverDnZgetrs (solver.cu:7-142) with a
// blocked right-looking factorisation of the row-major matrix (P Z = L U,
// unit L, LAPACK-style 0-based row pivots kept on the device):
//
//   for each block column of width NB:
//     for each sub-panel of width W inside it:
//       panel_kernel  -- cooperative kernel, whole sub-panel held in shared
//                        memory across all SMs, one grid barrier per column
//                        (pivot search, swap, scale, rank-1 update); panels
//                        of up to 8192 rows run panel_reg_kernel instead,
//                        rows in registers, on one cluster of at most 16
//                        CTAs with one exchange of candidates per column
//       interchanges + U12 + thin GEMM for the rest of the block column
//     interchanges of the block's pivots on the other columns
//     U12 = L11^-1 A12  (blocked TRSM)
//     A22 -= L21 U12    (the trailing update: FP64 on the FP64 tensor path,
//                        mma.sync f64, three real products per complex
//                        one; FP32 on tcgen05 with FP16 (or TF32) parts)
//
// The pivot rule is the one of LAPACK izamax: largest |re| + |im|, first
// index on ties.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "bem_internal.h"
#include "cgemm_simt.cuh"
#include "lu_internal.h"
#include "math_device.cuh"
#include "zgemm_dmma.cuh"

namespace bem {

// ------------------------------------------------------------------- GEMM
template <typename R>
int cgemm(bem_ctx* ctx, int M, int N, int K, const typename C2T<R>::type* A, int64_t lda,
          const typename C2T<R>::type* B, int64_t ldb, bool b_kmajor,
          typename C2T<R>::type* C, int64_t ldc, bool c_colmajor,
          typename C2T<R>::type alpha, typename C2T<R>::type beta, int prof_cls, int batch, int64_t sA,
          int64_t sB, int64_t sC) {
    if (M <= 0 || N <= 0 || batch <= 0) return BEM_OK;
    if (K <= 0) {
        // C = beta*C only; our callers never need it with beta != 1
        return BEM_OK;
    }
    if (batch > 1 && sizeof(R) != 8) return fail(ctx, BEM_ERR_INVALID, "batched GEMM is FP64 only");
    dim3 grid((N + 63) / 64, (M + 63) / 64, batch);
    // the 3M kernel's tile: the least time of the SM with the most tiles.  Per
    // K = 256 and SM, measured (us): 64 x 64 34 alone, 32 each of more; 32 x 32
    // 10.7 and 9; 32 x 8 4.1 and 2.75 (3.5 with an N-major B).
    int tile = 0;
    if (sizeof(R) == 8 && ctx->dmma_3m) {
        const int bm[3] = {64, 32, 32}, bn[3] = {64, 32, 8};
        const double one[3] = {34.0, 10.7, 4.1}, each[3] = {32.0, 9.0, b_kmajor ? 2.75 : 3.5};
        double best = 0.0;
        for (int t = 0; t < 3; t++) {
            const int64_t tiles = (int64_t)((M + bm[t] - 1) / bm[t]) * ((N + bn[t] - 1) / bn[t]) * batch;
            const int64_t per_sm = (tiles + ctx->sm_count - 1) / ctx->sm_count;
            const double cost = std::max(one[t], each[t] * (double)per_sm);
            if (t == 0 || (cost < best && (M + 31) / 32 <= 65535)) best = cost, tile = t;
        }
        grid = dim3((N + bn[tile] - 1) / bn[tile], (M + bm[tile] - 1) / bm[tile], batch);
    }
    if (grid.y > 65535) return fail(ctx, BEM_ERR_INVALID, "gemm M too large");
    cudaEvent_t ev = prof_cls >= 0 ? ctx->prof_begin(prof_cls) : nullptr;
    if (sizeof(R) == 8) {
        // FP64: the m8n8k4 f64 tensor path (zgemm_dmma.cuh)
        // the attribute is per device: one bit per (kernel variant, device id)
        // (three real products per complex one unless the context asks for four)
        static std::atomic<unsigned long long> attr[16];
        const double2* Ad = reinterpret_cast<const double2*>(A);
        const double2* Bd = reinterpret_cast<const double2*>(B);
        double2* Cd = reinterpret_cast<double2*>(C);
        double2 al = make_double2(alpha.x, alpha.y), be = make_double2(beta.x, beta.y);
        auto go = [&](auto kern, int slot, int threads, int smem, int smem_max) -> int {
            const unsigned long long bit = 1ull << (ctx->device & 63);
            if (!(attr[slot].load() & bit)) {
                BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
                attr[slot].fetch_or(bit);
            }
            kern<<<grid, threads, smem, ctx->stream>>>(M, N, K, Ad, lda, Bd, ldb, Cd, ldc, al, be, sA, sB, sC);
            return BEM_OK;
        };
        const int nst = (K + dmma::BKC - 1) / dmma::BKC;
        auto go3 = [&](auto tl, int slot) -> int {
            using T = decltype(tl);
            if (b_kmajor)
                return c_colmajor ? go(dmma::zgemm3m_kernel<T, true, true>, slot, T::THREADS, T::smem_bytes(true, nst), T::smem_bytes(true, 1 << 20))
                                  : go(dmma::zgemm3m_kernel<T, true, false>, slot + 1, T::THREADS, T::smem_bytes(true, nst), T::smem_bytes(true, 1 << 20));
            return c_colmajor ? go(dmma::zgemm3m_kernel<T, false, true>, slot + 2, T::THREADS, T::smem_bytes(false, nst), T::smem_bytes(false, 1 << 20))
                              : go(dmma::zgemm3m_kernel<T, false, false>, slot + 3, T::THREADS, T::smem_bytes(false, nst), T::smem_bytes(false, 1 << 20));
        };
        const int t4 = 128, s4 = dmma::SMEM_BYTES;
        int s;
        if (ctx->dmma_3m) {
            s = tile == 0 ? go3(dmma::M3Big{}, 4) : tile == 1 ? go3(dmma::M3Small{}, 8) : go3(dmma::M3Thin{}, 12);
        } else if (b_kmajor) {
            s = c_colmajor ? go(dmma::zgemm_kernel<true, true>, 0, t4, s4, s4) : go(dmma::zgemm_kernel<true, false>, 1, t4, s4, s4);
        } else {
            s = c_colmajor ? go(dmma::zgemm_kernel<false, true>, 2, t4, s4, s4)
                           : go(dmma::zgemm_kernel<false, false>, 3, t4, s4, s4);
        }
        BEM_TRY(s);
    } else if (b_kmajor) {
        if (c_colmajor)
            cgemm_simt_kernel<R, true, true><<<grid, 256, 0, ctx->stream>>>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta);
        else
            cgemm_simt_kernel<R, true, false><<<grid, 256, 0, ctx->stream>>>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta);
    } else {
        if (c_colmajor)
            cgemm_simt_kernel<R, false, true><<<grid, 256, 0, ctx->stream>>>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta);
        else
            cgemm_simt_kernel<R, false, false><<<grid, 256, 0, ctx->stream>>>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta);
    }
    BEM_LAUNCHED(ctx);
    if (ev)
        ctx->prof_end(prof_cls, ev, 8.0 * M * N * K * batch,
                      (double)sizeof(typename C2T<R>::type) * ((double)M * K + (double)K * N + 2.0 * M * N) * batch);
    return BEM_OK;
}

template <typename C2> static C2 mk(double re, double im) {
    C2 c;
    c.x = re;
    c.y = im;
    return c;
}

// ------------------------------------------------------------- grid barrier
// Monotonic arrival counter, reset to 0 before the launch.  Thread 0 of each
// CTA arrives and waits for `target` arrivals, giving up after ~2 s of clock
// cycles (status word := BEM_ERR_TIMEOUT); the kernel then returns.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, int* status,
                                             int* s_flag) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(bar, 1u);
        long long t0 = clock64();
        int ok = 1;
        while (true) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if (*(volatile int*)status != 0 || clock64() - t0 > 4000000000LL) {
                atomicCAS(status, 0, (int)BEM_ERR_TIMEOUT);
                ok = 0;
                break;
            }
            __nanosleep(20);
        }
        __threadfence();
        *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
}

template <typename R> __device__ __forceinline__ R cabs1(typename C2T<R>::type v) {
    return fabs(v.x) + fabs(v.y);
}

// ------------------------------------------------------------ panel kernel
__device__ __forceinline__ float2 pivot_recip(float2 p) {
    const float den = p.x * p.x + p.y * p.y;
    return make_float2(p.x / den, -p.y / den);
}

// The two per-element operations of a panel column, with explicit fused
// multiply-adds so that every panel kernel rounds them alike:
// l = a inv and x - l u (complex).
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename C2> __device__ __forceinline__ C2 panel_mul(C2 a, C2 inv) {
    C2 l;
    l.x = fma_rn(a.x, inv.x, -(a.y * inv.y));
    l.y = fma_rn(a.x, inv.y, a.y * inv.x);
    return l;
}
template <typename C2> __device__ __forceinline__ C2 panel_msub(C2 x, C2 l, C2 u) {
    x.x = fma_rn(-l.x, u.x, fma_rn(l.y, u.y, x.x));
    x.y = fma_rn(-l.x, u.y, fma_rn(-l.y, u.x, x.y));
    return x;
}
// x -= a b of the substitutions: the product first, so that x is rounded once.
// Their sums run over up to 256 products that are mostly smaller than x, and
// two roundings of x for each (panel_msub) made the FP64 solution's error 7.6 %
// larger (24 systems of 2N = 960 to 4608).
template <typename C2> __device__ __forceinline__ void csub_mul(C2& x, C2 a, C2 b) {
    x.x -= fma_rn(a.x, b.x, -(a.y * b.y));
    x.y -= fma_rn(a.x, b.y, a.y * b.x);
}

// Column jj of a panel tile after the interchange: rows below the pivot row
// are scaled by 1/pivot (l = a inv) and the columns right of jj take the
// rank-1 update x -= l u (u: the pivot row).  tpr = w rounded up to a power
// of two threads per row, so a row's threads sit in one warp: they read
// a[i][jj] before the thread of column jj overwrites it with l (__syncwarp),
// with no integer division per element.  Every thread runs the same number
// of passes.
template <typename R>
__device__ __forceinline__ void panel_eliminate(typename C2T<R>::type* tile, int w, int nloc, int lo, int jj,
                                                const typename C2T<R>::type* s_piv, typename C2T<R>::type inv) {
    using C2 = typename C2T<R>::type;
    int tpr = 1;
    while (tpr < w) tpr <<= 1;
    const int rpp = (int)blockDim.x / tpr, cc = (int)threadIdx.x % tpr, i0 = (int)threadIdx.x / tpr;
    const int passes = (nloc + rpp - 1) / rpp;
    C2 u;
    u.x = 0;
    u.y = 0;
    if (cc < w) u = s_piv[cc];
    for (int ps = 0; ps < passes; ps++) {
        const int i = i0 + ps * rpp;
        const bool act = i < nloc && lo + i > jj && cc >= jj && cc < w;
        C2 a;
        a.x = 0;
        a.y = 0;
        if (act) a = tile[i * w + jj];
        const C2 l = panel_mul(a, inv);
        __syncwarp();
        if (act) {
            if (cc == jj)
                tile[i * w + jj] = l;
            else
                tile[i * w + cc] = panel_msub(tile[i * w + cc], l, u);
        }
    }
}

// Dynamic shared memory that panel_kernel may take, always set as its limit:
// the limit is the device's, and other host threads' contexts launch it too.
constexpr int PANEL_SMEM = 220 * 1024;

// Factors the sub-panel rows [r0, n), columns [r0, r0+w) of the row-major
// matrix A.  CTA b owns panel rows [b*Rp, min((b+1)*Rp, nrows)) (relative
// to r0) in shared memory; Rp >= w so the w pivot rows live in CTA 0.
// Batched: CTAs [i Gm, (i+1) Gm) factor matrix i (A + i sA, pivots ipiv +
// i sPiv, info + i); every CTA of the grid meets at the one barrier.
template <typename R>
__global__ void __launch_bounds__(256)
panel_kernel(typename C2T<R>::type* __restrict__ A, int64_t lda, int r0, int nrows, int w, int Rp,
             int* __restrict__ ipiv, int* __restrict__ info, PanelWS ws, int Gm, int64_t sA, int sPiv) {
    using C2 = typename C2T<R>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C2* tile = (C2*)smem_raw;                   // Rp * w
    C2* s_piv = tile + (size_t)Rp * w;          // w
    __shared__ R s_val[8];
    __shared__ int s_row[8];
    __shared__ int s_flag;
    __shared__ R s_best;
    __shared__ int s_brow;

    const int G = Gm, mi = blockIdx.x / Gm, b = blockIdx.x % Gm, tid = threadIdx.x;
    const unsigned Gall = gridDim.x;
    A += mi * sA;
    ipiv += mi * sPiv;
    info += mi;
    const int lane = tid & 31, warp = tid >> 5;
    const int lo = b * Rp;
    const int nloc = max(0, min(Rp, nrows - lo));
    R* cval = (R*)ws.cval + (size_t)mi * 2 * Gm;
    int* crow = ws.crow + (size_t)mi * 2 * Gm;
    C2* cdata = (C2*)ws.cdata + (size_t)mi * 2 * Gm * w;
    C2* disp = (C2*)ws.disp + (size_t)mi * 2 * w;

    for (int e = tid; e < nloc * w; e += blockDim.x) {
        int i = e / w, c = e % w;
        tile[e] = A[(int64_t)(r0 + lo + i) * lda + r0 + c];
    }
    __syncthreads();

    for (int jj = 0; jj < w; jj++) {
        const int par = jj & 1;
        // 1. local pivot candidate among rows >= jj
        R bv = (R)-1;
        int br = 0x7fffffff;
        for (int i = tid; i < nloc; i += blockDim.x) {
            int gr = lo + i;
            if (gr < jj) continue;
            R v = cabs1<R>(tile[i * w + jj]);
            if (v > bv || (v == bv && gr < br)) bv = v, br = gr;
        }
        for (int o = 16; o > 0; o >>= 1) {
            R ov = __shfl_down_sync(0xffffffffu, bv, o);
            int orw = __shfl_down_sync(0xffffffffu, br, o);
            if (ov > bv || (ov == bv && orw < br)) bv = ov, br = orw;
        }
        if (lane == 0) s_val[warp] = bv, s_row[warp] = br;
        __syncthreads();
        if (tid == 0) {
            for (int k = 1; k < (int)(blockDim.x >> 5); k++)
                if (s_val[k] > bv || (s_val[k] == bv && s_row[k] < br)) bv = s_val[k], br = s_row[k];
            s_best = bv;
            s_brow = br;
            __stcg(&cval[par * G + b], bv);
            __stcg(&crow[par * G + b], br);
        }
        __syncthreads();
        br = s_brow;
        if (br != 0x7fffffff)
            for (int c = tid; c < w; c += blockDim.x) __stcg(&cdata[((size_t)par * G + b) * w + c], tile[(br - lo) * w + c]);
        if (b == 0)
            for (int c = tid; c < w; c += blockDim.x) __stcg(&disp[par * w + c], tile[jj * w + c]);
        // 2. all candidates published
        if (!grid_barrier(ws.bar, (unsigned)(jj + 1) * Gall, ws.status, &s_flag)) return;
        // 3. global argmax (|re|+|im| max, smallest row on ties); warp 0 also
        // fetches the pivot row
        if (warp == 0) {
            bv = (R)-1;
            br = 0x7fffffff;
            int bo = -1;
            for (int k = lane; k < G; k += 32) {
                R v = __ldcg(&cval[par * G + k]);
                int r = __ldcg(&crow[par * G + k]);
                if (r == 0x7fffffff) continue;
                if (v > bv || (v == bv && r < br)) bv = v, br = r, bo = k;
            }
            for (int o = 16; o > 0; o >>= 1) {
                R ov = __shfl_down_sync(0xffffffffu, bv, o);
                int orw = __shfl_down_sync(0xffffffffu, br, o);
                int oo = __shfl_down_sync(0xffffffffu, bo, o);
                if (ov > bv || (ov == bv && orw < br)) bv = ov, br = orw, bo = oo;
            }
            bv = __shfl_sync(0xffffffffu, bv, 0);
            br = __shfl_sync(0xffffffffu, br, 0);
            bo = __shfl_sync(0xffffffffu, bo, 0);
            const bool zero = !(bv > (R)0);
            if (zero) {
                br = jj;  // no interchange; LAPACK records info and skips the scaling
                bo = -1;
            }
            if (lane < w)
                s_piv[lane] = bo >= 0 ? __ldcg(&cdata[((size_t)par * G + bo) * w + lane]) : __ldcg(&disp[par * w + lane]);
            if (lane == 0) {
                if (zero) atomicCAS(info, 0, r0 + jj + 1);
                s_brow = br;
                s_best = bv;
                if (b == 0) ipiv[r0 + jj] = r0 + br;
            }
        }
        __syncthreads();
        const int piv = s_brow;
        const bool zero = !(s_best > (R)0);
        // 4. interchange rows jj and piv
        if (piv != jj) {
            if (b == 0)
                for (int c = tid; c < w; c += blockDim.x) tile[jj * w + c] = s_piv[c];
            if (piv >= lo && piv < lo + nloc)
                for (int c = tid; c < w; c += blockDim.x) tile[(piv - lo) * w + c] = __ldcg(&disp[par * w + c]);
        }
        __syncthreads();
        // 5. scale column jj below the diagonal, rank-1 update of the rest
        if (!zero) {
            panel_eliminate<R>(tile, w, nloc, lo, jj, s_piv, pivot_recip(s_piv[jj]));
        }
        __syncthreads();
    }
    for (int e = tid; e < nloc * w; e += blockDim.x) {
        int i = e / w, c = e % w;
        A[(int64_t)(r0 + lo + i) * lda + r0 + c] = tile[e];
    }
}

// ---------------------------------------------------- register panel kernel
// The sub-panel of panel_kernel with every row in the registers of one
// thread, on one thread-block cluster per matrix: thread t of CTA b owns
// panel row b T + t.  No row is moved while the columns are eliminated:
// interchanging rows jj and p only exchanges their positions (one integer per
// thread, which is also the tie break), and each row is written to its final
// position at the end.  Per column jj:
//   1. every warp has its largest |re| + |im| of column jj among rows not yet
//      taken (smallest position on ties), searched with the row's reciprocal
//      while the columns after jj were updated; the winning lane leaves both
//      and its columns jj.. in shared memory; block barrier;
//   2. every warp k < C reduces the CTA's candidates and sends the best one to
//      CTA k's shared memory (st.async, counted on an mbarrier there);
//   3. every thread waits for its CTA's C messages, every warp reduces the C
//      candidates from its own shared memory, and every row still active is
//      scaled and takes the rank-1 update x -= l u, u read as a broadcast,
//      column jj + 1 first.
// So a column costs one block barrier and one message's way to another SM.
// 16 columns, us, now and with stores, a cluster barrier and the reciprocal
// after it: 256 rows (1 CTA) 18.7 and 18.7, 2048 (8) 26.7 and 28.9, 4096 (16)
// 28.3 and 37.0 (on 8 CTAs), 4608 (16) 30.1 and 39.0; 1 to 1.5 us of them are the
// bound of the waits and the corrected reciprocal.  Of ~2600 cycles a
// column on 8 CTAs the row's way into shared memory takes 430, the message 820,
// the reductions 250 to 300 each and the updates 650.
// Buffers alternate between two parities: a CTA sending to a peer in column
// jj + 2 has that peer's message of jj + 1, sent after the block barrier that
// follows the peer's reads of column jj.
// Same pivot rule and per-element arithmetic (panel_mul, panel_msub) as
// panel_kernel, so the same pivots and factors.
// A wait that runs out (wait_cycles: ~1 s of a peer that does not send) ends
// the columns: the warp takes nothing from the messages it lacks, so every
// position stays one of the panel, and its CTA leaves at the next block barrier
// (s_stop, by column parity: a column writes the next one's word) before it
// sends again, stores no row and records BEM_ERR_TIMEOUT.  The kernels queued
// behind it read that word before they follow `moves`.
// moves (2 n integers per matrix): for the w top positions k of the panel,
// moves[r0 + k] is the row now at position k and moves[n + r0 + k] the
// position of the row formerly there: the interchanges as one gather.
template <typename R> struct PanelW { static constexpr int v = 64 / (2 * (int)sizeof(R) / 4); };  // 64 registers a row
constexpr int PR_THREADS = 512, PR_WARPS = PR_THREADS / 32, PR_CLUSTER = 16, PG = 4;
constexpr int PR_PITCH = 256 + 16;  // bytes of a row in shared memory

// A pivot candidate: |v| as its bit pattern (v >= 0, 0 for none: the bits of
// non-negative floating-point numbers order like unsigned integers, so integer
// warp reductions compare them) and its row's position.
__device__ __forceinline__ uint4 cand_bits(double v, int pos) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return make_uint4((unsigned)(b >> 32), (unsigned)b, (unsigned)pos, 0u);
}
__device__ __forceinline__ uint4 cand_bits(float v, int pos) { return make_uint4(__float_as_uint(v), 0u, (unsigned)pos, 0u); }
// The lane with the warp's largest candidate, the smallest position on ties,
// -1 where there is none; mhi is the largest upper word of all lanes.
__device__ __forceinline__ int cand_lane(uint4 c, unsigned mhi) {
    unsigned win = __ballot_sync(0xffffffffu, c.x == mhi);
    if (win & (win - 1)) {  // several lanes share the upper word: the lower one and the row decide
        const unsigned mlo = __reduce_max_sync(0xffffffffu, c.x == mhi ? c.y : 0u);
        if ((mhi | mlo) == 0u) return -1;
        const bool top = c.x == mhi && c.y == mlo;
        const unsigned mrow = __reduce_min_sync(0xffffffffu, top ? c.z : 0xffffffffu);
        win = __ballot_sync(0xffffffffu, top && c.z == mrow);
    }
    return __ffs(win) - 1;
}

// A value into a peer's shared memory, counted on the peer's mbarrier.
__device__ __forceinline__ void st_async(uint32_t dst, uint32_t bar, uint4 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t dst, uint32_t bar, double2 v) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(v.x), y = (unsigned long long)__double_as_longlong(v.y);
    st_async(dst, bar, make_uint4((unsigned)x, (unsigned)(x >> 32), (unsigned)y, (unsigned)(y >> 32)));
}
__device__ __forceinline__ void st_async(uint32_t dst, uint32_t bar, float2 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t smem, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(rank));
    return r;
}
// Waits until the phase of this parity is complete, `limit` clock cycles at most (0: gives up at once).
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, long long limit) {
    if (limit <= 0) return false;
    long long t0 = 0;
    for (int i = 0;; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (i == 0) t0 = clock64();
        if (clock64() - t0 > limit) return false;
    }
}

template <typename R>
__global__ void __launch_bounds__(PR_THREADS, 1)
panel_reg_kernel(typename C2T<R>::type* __restrict__ A, int64_t lda, int n, int r0, int nrows, int w,
                 int* __restrict__ ipiv, int* __restrict__ info, int* __restrict__ moves, int64_t sA,
                 int* __restrict__ status, long long wait_cycles) {
    using C2 = typename C2T<R>::type;
    namespace cg = cooperative_groups;
    constexpr int W = PanelW<R>::v;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ __align__(16) C2 s_row[2][PR_WARPS][W];    // a warp's candidate row
    __shared__ __align__(16) C2 r_row[2][PR_CLUSTER][W];  // a CTA's candidate row (written by the peers)
    __shared__ __align__(16) C2 s_inv[2][PR_WARPS], r_inv[2][PR_CLUSTER];
    __shared__ __align__(16) uint4 s_cand[2][PR_WARPS], r_cand[2][PR_CLUSTER];
    __shared__ __align__(8) unsigned long long r_bar[2];
    __shared__ int s_at[PR_THREADS], s_stop[2];
    // the rows on their way in and out, 256 B each: 16 lanes a row in global
    // memory, a thread a row here (an odd number of 16-byte units apart)
    extern __shared__ __align__(16) unsigned char pr_smem[];

    const int C = (int)cluster.num_blocks(), b = (int)cluster.block_rank(), tid = threadIdx.x, T = blockDim.x;
    const int mi = blockIdx.x / C, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    A += mi * sA;
    ipiv += (int64_t)mi * n;
    info += mi;
    moves += (int64_t)mi * 2 * n;
    const uint32_t bar0 = static_cast<uint32_t>(__cvta_generic_to_shared(&r_bar[0]));
    if (C > 1 && tid == 0) {
        for (int k = 0; k < 2; k++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * k) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 2) s_stop[tid] = 0;
    const int gr = b * T + tid;
    const bool valid = gr < nrows;
    bool act = valid;
    int pos = gr;
    C2 x[W];
    C2* mine = reinterpret_cast<C2*>(pr_smem + (size_t)tid * PR_PITCH);
    C2* base = A + (int64_t)(r0 + b * T) * lda + r0;  // the CTA's first row
    const int rows = max(0, min(T, nrows - b * T));
    // whole 16-byte units (FP32: even lda and r0), else element by element
    const bool wide = w == W && ((reinterpret_cast<uintptr_t>(base) | ((uintptr_t)lda * sizeof(C2))) & 15) == 0;
    if (wide) {
        for (int e = tid; e < rows * 16; e += T)
            dmma::cp16(pr_smem + (size_t)(e >> 4) * PR_PITCH + 16 * (e & 15),
                       reinterpret_cast<const unsigned char*>(base + (int64_t)(e >> 4) * lda) + 16 * (e & 15), true);
        dmma::cp_commit();
        dmma::cp_wait<0>();
    } else {
        for (int e = tid; e < rows * w; e += T)
            reinterpret_cast<C2*>(pr_smem + (size_t)(e / w) * PR_PITCH)[e % w] = base[(int64_t)(e / w) * lda + e % w];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < W; c++) {
        x[c].x = x[c].y = 0;
        if (valid && c < w) x[c] = mine[c];
    }
    if (C > 1) cluster.sync();  // every CTA runs before its shared memory is written
    // PG columns at a time: x[0 .. PG) are the current ones, x[rem .. W) the
    // finished ones; the row rotates left by PG after each group, so W / PG
    // groups bring it back.  One loop over the groups instead of W unrolled
    // columns: those were 13 k instructions that every launch fetched anew.
    // this thread's candidate of a column, the warp's largest upper word and
    // the reciprocal that the row needs if it wins: all under the update of
    // the columns after it
    uint4 cand;
    unsigned mhi;
    C2 rinv;
    auto search = [&](C2 xv) {
        R v = act ? cabs1<R>(xv) : (R)0;
        if (!(v > (R)0)) {  // a NaN is no candidate either
            v = (R)0;
            xv.x = 1, xv.y = 0;
        }
        cand = cand_bits(v, pos);
        mhi = __reduce_max_sync(0xffffffffu, cand.x);
        rinv = pivot_recip(xv);
    };
    const uint4 none = make_uint4(0u, 0u, 0x7fffffffu, 0u);
    search(x[0]);
    bool stop = false;
    for (int g0 = 0; g0 < W && !stop; g0 += PG) {
      const int rem = W - g0;
#pragma unroll
      for (int q = 0; q < PG; q++) {
        const int jj = g0 + q;
        if (jj >= w) break;
        const int par = q & 1;  // PG is even: the parity of jj
        // 1. this warp's candidate
        const int wl = cand_lane(cand, mhi);
        if (lane == max(wl, 0)) {
            s_cand[par][warp] = wl < 0 ? none : cand;
            s_inv[par][warp] = rinv;
#pragma unroll
            for (int c0 = 0; c0 < W; c0 += PG)
                if (c0 < rem) {
#pragma unroll
                    for (int c = c0; c < c0 + PG; c++)
                        if (c >= q) s_row[par][warp][c] = x[c];
                }
        }
        __syncthreads();
        uint4 rec = lane < nw ? s_cand[par][lane] : none;
        if (C > 1 && s_stop[par]) {  // a warp's wait of the column before ran out
            stop = true;
            break;
        }
        bool late = false;
        const C2* u;
        C2 inv;
        if (C > 1) {
            // 2. the CTA's candidate into every CTA of the cluster
            const uint32_t bar = bar0 + 8 * par;
            if (tid == 0) {
                const int bytes = C * ((rem - q + 1) * (int)sizeof(C2) + (int)sizeof(uint4));
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            }
            if (warp < C) {
                const int ck = cand_lane(rec, __reduce_max_sync(0xffffffffu, rec.x)), cw = max(ck, 0);
                const C2 e = s_row[par][cw][lane < W ? lane : 0], iv = s_inv[par][cw];
                const uint4 cc = ck < 0 ? none : s_cand[par][cw];
                const uint32_t row = static_cast<uint32_t>(__cvta_generic_to_shared(&r_row[par][b][lane < W ? lane : 0])),
                               to = static_cast<uint32_t>(__cvta_generic_to_shared(&r_cand[par][b])),
                               rcp = static_cast<uint32_t>(__cvta_generic_to_shared(&r_inv[par][b]));
                for (int k = warp; k < C; k += nw) {
                    const uint32_t kb = map_rank(bar, k);
                    if (lane >= q && lane < rem) st_async(map_rank(row, k), kb, e);
                    if (lane == 0) {
                        st_async(map_rank(to, k), kb, cc);
                        st_async(map_rank(rcp, k), kb, iv);
                    }
                }
            }
            late = __any_sync(0xffffffffu, !mbar_wait_cluster(bar, (uint32_t)(jj >> 1) & 1u, wait_cycles));
            if (late && lane == 0) s_stop[par ^ 1] = 1;
            rec = lane < C && !late ? r_cand[par][lane] : none;
        }
        const int bk = cand_lane(rec, __reduce_max_sync(0xffffffffu, rec.x)), bw = max(bk, 0);
        int piv;
        if (C > 1) {
            u = r_row[par][bw];
            inv = r_inv[par][bw];
            piv = (int)r_cand[par][bw].z;
        } else {
            u = s_row[par][bw];
            inv = s_inv[par][bw];
            piv = (int)s_cand[par][bw].z;
        }
        // 3. no candidate: a zero column, no interchange and no scaling (LAPACK records it)
        const bool zp = bk < 0;
        if (zp) piv = jj;
        if (b == 0 && tid == 0) {
            ipiv[r0 + jj] = r0 + piv;
            if (zp && !late) atomicCAS(info, 0, r0 + jj + 1);
        }
        if (pos == piv) {
            pos = jj;
            act = false;
        } else if (pos == jj) {
            pos = piv;
        }
        const bool on = act && !zp;
        const C2 l = panel_mul(x[q], inv);
        if (on) x[q] = l;
        // the next column first: its candidates are searched under the others' update
        if (q + 1 < W && q + 1 < rem) {
            if (on) x[q + 1] = panel_msub(x[q + 1], l, u[q + 1]);
            search(x[q + 1]);
        }
        if (on) {
#pragma unroll
            for (int c0 = 0; c0 < W; c0 += PG)
                if (c0 < rem) {
#pragma unroll
                    for (int c = c0; c < c0 + PG; c++)
                        if (c > q + 1) x[c] = panel_msub(x[c], l, u[c]);
                }
        }
      }
      C2 done[PG];
#pragma unroll
      for (int c = 0; c < PG; c++) done[c] = x[c];
#pragma unroll
      for (int c = 0; c + PG < W; c++) x[c] = x[c + PG];
#pragma unroll
      for (int c = 0; c < PG; c++) x[W - PG + c] = done[c];
    }
    __syncthreads();  // a late warp of the last column
    const bool lost = C > 1 && (s_stop[0] | s_stop[1]) != 0;
    if (lost && tid == 0) *status = BEM_ERR_TIMEOUT;
    __syncwarp();
    // no CTA ends while a peer may still write to it (the wait is at the end)
    if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (lost) {
        // messages sent before the peers arrived may still be on their way: ~0.1 ms, a hundred times what one takes
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        for (const long long t0 = clock64(); clock64() - t0 < 200000;) __nanosleep(1000);
        return;
    }
    // rows to their positions (every row of the panel was read before the first barrier)
    if (valid) {
#pragma unroll
        for (int c = 0; c < W; c++)
            if (c < w) mine[c] = x[c];
        s_at[tid] = pos;
    }
    __syncthreads();
    C2* top = A + (int64_t)r0 * lda + r0;
    if (wide) {
        for (int e = tid; e < rows * 16; e += T)
            *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(top + (int64_t)s_at[e >> 4] * lda) + 16 * (e & 15)) =
                *reinterpret_cast<const uint4*>(pr_smem + (size_t)(e >> 4) * PR_PITCH + 16 * (e & 15));
    } else {
        for (int e = tid; e < rows * w; e += T)
            top[(int64_t)s_at[e / w] * lda + e % w] = reinterpret_cast<const C2*>(pr_smem + (size_t)(e / w) * PR_PITCH)[e % w];
    }
    if (valid) {
        if (pos < w) moves[r0 + pos] = r0 + gr;
        if (gr < w) moves[n + r0 + gr] = r0 + pos;
    }
    __syncwarp();
    if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// CTAs per cluster (`most` at most) and threads per CTA for a sub-panel of
// nrows rows, 0 when it does not fit: 256 rows a CTA up to `most` CTAs, then up
// to 512 rows a CTA -- 8192 rows on 16 CTAs, 4096 on 8.  Few rows a CTA keep the
// rank-1 update short (64 registers a row, the FP64 pipe of one SM).
struct PanelShape {
    int C = 0, T = 0;
};
static PanelShape panel_reg_shape(int nrows, int most) {
    PanelShape p;
    if (nrows > most * PR_THREADS) return p;
    p.C = std::min(most, (nrows + 255) / 256);
    p.T = ((nrows + p.C - 1) / p.C + 31) / 32 * 32;
    return p;
}

// Clusters of a shape that this device holds at a time (asked once per shape
// and remembered).
template <typename R> static int panel_resident(bem_ctx* ctx, PanelShape p) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, int>, int> known;
    const auto key = std::make_tuple(ctx->device, p.C, p.T);
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(key);
    if (it == known.end()) {
        auto kern = panel_reg_kernel<R>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)p.C);
        cfg.blockDim = dim3((unsigned)p.T);
        cfg.dynamicSmemBytes = (size_t)p.T * PR_PITCH;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)p.C;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int ncl = 0;
        const bool fits =
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_THREADS * PR_PITCH) == cudaSuccess &&
            (p.C <= 8 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
            cudaOccupancyMaxActiveClusters(&ncl, (const void*)kern, &cfg) == cudaSuccess && ncl >= 1;
        if (!fits) cudaGetLastError();
        it = known.emplace(key, fits ? ncl : 0).first;
    }
    return it->second;
}

// The shape for a sub-panel of `batch` matrices: up to 16 CTAs, or up to 8
// where the rows fit 8 and fewer such clusters than matrices can be resident
// (the rest would wait for a second round; none on a device that holds no
// cluster of more than 8).  C = 0: panel_kernel takes it.
template <typename R>
static PanelShape panel_reg_choice(bem_ctx* ctx, int nrows, int iw, int batch) {
    if (!ctx->panel_clusters || iw > PanelW<R>::v) return PanelShape{};
    const int most = ctx->panel_clusters == 1 ? PR_CLUSTER : std::min(ctx->panel_clusters, PR_CLUSTER);
    const PanelShape wide = panel_reg_shape(nrows, most), narrow = panel_reg_shape(nrows, std::min(most, 8));
    const int nw = wide.C > 0 ? panel_resident<R>(ctx, wide) : 0;
    if (narrow.C > 0 && narrow.C < wide.C && nw < batch && panel_resident<R>(ctx, narrow) > 0) return narrow;
    return nw > 0 ? wide : PanelShape{};
}

// One launch of panel_reg_kernel: `batch` matrices (A + i sA, pivots
// ipiv + i n, info + i, moves + 2 i n), one cluster each.
template <typename R>
static int launch_panel_reg(bem_ctx* ctx, typename C2T<R>::type* A, int64_t lda, int n, int i0, int nrows, int iw,
                            int* d_ipiv, int* d_info, int* d_moves, int batch, int64_t sA, PanelShape p) {
    using C2 = typename C2T<R>::type;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.C * batch));
    cfg.blockDim = dim3((unsigned)p.T);
    cfg.dynamicSmemBytes = (size_t)p.T * PR_PITCH;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)p.C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaEvent_t ev = ctx->prof_begin(PROF_PANEL);
    BEM_TRY_CUDA(ctx, cudaLaunchKernelEx(&cfg, panel_reg_kernel<R>, A, lda, n, i0, nrows, iw, d_ipiv, d_info, d_moves, sA,
                                         ctx->d_status, ctx->panel_wait));
    BEM_LAUNCHED(ctx);
    if (ev)
        ctx->prof_end(PROF_PANEL, ev, 8.0 * (double)nrows * iw * iw / 2 * batch,
                      (double)nrows * iw * 2 * sizeof(C2) * batch);
    return BEM_OK;
}

// moves of a sub-panel (see panel_reg_kernel) from its interchanges, for the
// panels of panel_kernel.  One thread per matrix: w <= 32 steps.  A panel whose
// barrier gave up (status) has left no pivots to follow.
__global__ void moves_kernel(const int* __restrict__ ipiv, int n, int r0, int w, int* __restrict__ moves, int batch,
                             const int* __restrict__ status) {
    const int mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi >= batch || *status != 0) return;
    ipiv += (int64_t)mi * n;
    moves += (int64_t)mi * 2 * n;
    // a position below the top is only ever exchanged with a top row, and only top rows go there
    int top[32], out_row[32], out_of[32], cnt = 0;
    for (int k = 0; k < w; k++) top[k] = r0 + k;
    for (int k = 0; k < w; k++) {
        const int p = ipiv[r0 + k];
        if (p < r0 + w) {
            const int t = top[k];
            top[k] = top[p - r0];
            top[p - r0] = t;
            continue;
        }
        int e = 0;
        while (e < cnt && out_row[e] != p) e++;
        if (e == cnt) out_row[cnt] = p, out_of[cnt] = p, cnt++;
        const int t = top[k];
        top[k] = out_of[e];
        out_of[e] = t;
    }
    for (int k = 0; k < w; k++) {
        moves[r0 + k] = top[k];
        if (top[k] < r0 + w) moves[n + top[k]] = r0 + k;
    }
    for (int e = 0; e < cnt; e++)
        if (out_of[e] < r0 + w) moves[n + out_of[e]] = out_row[e];
}

// ------------------------------------------------------------------ laswp
// The interchanges of the sub-panels [k0, k1) (w rows each, in order) on the
// columns of up to two ranges, one thread per column: a sub-panel's rows are
// all loaded before any is stored (moves names each top position's new row
// and each displaced row's new position), so its latency is one load instead
// of one per interchange -- 16 of them per sub-panel, 60 us for the 256 of a
// block column before.  SOLVE (one sub-panel): the columns of the second
// range are then solved with the panel's unit lower triangle (U12 of the
// sub-panel), saving that kernel's launch and its pass over the rows.
// A non-zero status word (a panel's wait ran out) leaves the rows where they
// are: `moves` is then not all written.
template <typename R, bool SOLVE>
__global__ void __launch_bounds__(64)
move_rows_kernel(typename C2T<R>::type* __restrict__ A, int64_t lda, const int* __restrict__ moves, int n, int k0,
                 int k1, int w, int c0a, int c1a, int c0b, int c1b, const int* __restrict__ status, int64_t sA = 0) {
    using C2 = typename C2T<R>::type;
    constexpr int W = PanelW<R>::v;
    A += blockIdx.y * sA;  // batched: blockIdx.y selects the matrix
    moves += (int64_t)blockIdx.y * 2 * n;
    __shared__ C2 sT[SOLVE ? W : 1][W + 1];
    __shared__ int s_src[W], s_dst[W];
    const int t = blockIdx.x * blockDim.x + threadIdx.x, na = c1a - c0a;
    const bool in = t < na + (c1b - c0b), second = t >= na;
    const int c = second ? c0b + (t - na) : c0a + t;
    const int gave_up = *status;  // used after the first loads of `moves`
    for (int r0 = k0; r0 < k1; r0 += w) {
        const int iw = min(w, k1 - r0);
        __syncthreads();
        if (threadIdx.x < iw) {
            s_src[threadIdx.x] = moves[r0 + threadIdx.x];
            s_dst[threadIdx.x] = moves[n + r0 + threadIdx.x];
        }
        if (SOLVE)
            for (int e = threadIdx.x; e < iw * iw; e += blockDim.x)
                sT[e / iw][e % iw] = A[(int64_t)(r0 + e / iw) * lda + r0 + e % iw];
        __syncthreads();
        if (gave_up != 0) return;
        if (!in) continue;
        C2 x[W], y[W];
#pragma unroll
        for (int k = 0; k < W; k++) {
            x[k].x = x[k].y = y[k].x = y[k].y = 0;
            if (k >= iw) continue;
            if (SOLVE || s_src[k] != r0 + k) x[k] = A[(int64_t)s_src[k] * lda + c];
            if (s_dst[k] >= r0 + iw) y[k] = A[(int64_t)(r0 + k) * lda + c];
        }
        if (SOLVE && second) {
#pragma unroll
            for (int k = 0; k < W; k++) {
                if (k >= iw) break;
#pragma unroll
                for (int i = k + 1; i < W; i++) {
                    if (i >= iw) break;
                    csub_mul(x[i], sT[i][k], x[k]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < W; k++) {
            if (k >= iw) continue;
            if (s_dst[k] >= r0 + iw) A[(int64_t)s_dst[k] * lda + c] = y[k];
            if (s_src[k] != r0 + k || (SOLVE && second)) A[(int64_t)(r0 + k) * lda + c] = x[k];
        }
    }
}

// Row gather for the solve: X[k] = B[perm[k]] for every column (column-major).
template <typename R>
__global__ void permute_rows_kernel(const typename C2T<R>::type* __restrict__ B, int64_t ldb,
                                    typename C2T<R>::type* __restrict__ X, int64_t ldx, const int* __restrict__ perm,
                                    int n, int nrhs, int64_t sB = 0, int64_t sX = 0, int sPerm = 0) {
    B += blockIdx.y * sB;  // batched: blockIdx.y selects the system
    X += blockIdx.y * sX;
    if (perm) perm += blockIdx.y * sPerm;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * nrhs) return;
    int r = (int)(i % n), c = (int)(i / n);
    X[(int64_t)c * ldx + r] = B[(int64_t)c * ldb + (perm ? perm[r] : r)];
}

// ------------------------------------------------------------ block TRSM
// Solves T X = X for a whole diagonal block T = A[r0.., r0..] (kb <= 256 rows;
// UPPER: non-unit upper, backward substitution; else unit lower, forward) in
// one launch, for the columns [c0, c1) of a right-hand side held row-major in
// the factor itself (B_ROWMAJOR, the U12 step) or column-major (the solves).
// One CTA owns RB columns; thread r holds row r of them in registers, so
// warp s holds the 32-row sub-block s, and its 32 x 32 diagonal block of T as
// well.  Step s: warp s substitutes through that block, x_k going to the other
// lanes by shuffles, and leaves the solved rows in shared memory; after the
// one block barrier every later warp subtracts T's segment of its rows times
// them.  The segment comes by cp.async into the warp's 32 x 33 buffer while
// warp s works, lanes along a row of T (a lane per row reads 32 lines per
// load: 7 k cycles a step, twice the substitution).  Bound by 256 dependent
// steps of a shuffle, a product and a subtraction.  FP64, 32 columns: 19.8 us a
// lower and 21.3 us an upper block; 32.7 and 30.1 us with the segments of T in
// registers, loaded by a lane per row, the diagonal blocks in shared memory
// and two columns a CTA.
// An upper block's rows are scaled by their diagonal's reciprocal beforehand,
// which takes the division out of the chain of steps.
//
// MODE bits: TRSM_TRANS reads T transposed (T[i][j] = A[r0+j][r0+i], the L^T
// of an L D L^T factor), TRSM_UNIT makes an upper T unit-diagonal, and
// TRSM_DIVDIAG divides the solution of a unit-lower T by T's diagonal (the D
// of L D L^T) when it is stored.
constexpr int TRSM_KB = 256, TRSM_TS = 32, TRSM_PITCH = TRSM_TS + 1;
static_assert(TRSM_KB == TRSM_BLOCK, "diagonal block rows");
constexpr int TRSM_TRANS = 1, TRSM_UNIT = 2, TRSM_DIVDIAG = 4;

template <typename C2> __device__ __forceinline__ C2 cdiv(C2 a, C2 d) {
    const auto den = d.x * d.x + d.y * d.y;
    C2 q;
    q.x = (a.x * d.x + a.y * d.y) / den;
    q.y = (a.y * d.x - a.x * d.y) / den;
    return q;
}

__device__ __forceinline__ float2 shfl_c(float2 v, int k) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, k), __shfl_sync(0xffffffffu, v.y, k));
}
__device__ __forceinline__ double2 shfl_c(double2 v, int k) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, k), __shfl_sync(0xffffffffu, v.y, k));
}

__device__ __forceinline__ void cp_elem(double2* smem, const double2* gmem, bool valid) { dmma::cp16(smem, gmem, valid); }
__device__ __forceinline__ void cp_elem(float2* smem, const float2* gmem, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int n = valid ? 8 : 0;  // 0: fill with zeros
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(gmem), "r"(n) : "memory");
}

template <typename R, bool UPPER, bool B_ROWMAJOR, int RB, int MODE = 0>
__global__ void __launch_bounds__(TRSM_KB)
trsm_block_kernel(const typename C2T<R>::type* __restrict__ T, int64_t ldt, int r0, int kb,
                  typename C2T<R>::type* __restrict__ B, int64_t ldb, int br0, int c0, int c1, int64_t strideT = 0,
                  int64_t strideB = 0) {
    T += blockIdx.y * strideT;  // batched: blockIdx.y selects the system
    B += blockIdx.y * strideB;
    constexpr bool TRANS = (MODE & TRSM_TRANS) != 0, UNIT = (MODE & TRSM_UNIT) != 0,
                   DIVDIAG = (MODE & TRSM_DIVDIAG) != 0;
    using C2 = typename C2T<R>::type;
    constexpr int TS = TRSM_TS;
    extern __shared__ __align__(16) unsigned char trsm_smem[];
    __shared__ __align__(16) C2 xs[2][TS][RB];
    const int r = threadIdx.x, lane = r & 31, warp = r >> 5, nsb = (int)blockDim.x >> 5;
    const int cb = c0 + blockIdx.x * RB, nc = min(RB, c1 - cb);
    const bool row = r < kb;
    C2 zero;
    zero.x = 0;
    zero.y = 0;
    C2* buf = reinterpret_cast<C2*>(trsm_smem) + (size_t)warp * TS * TRSM_PITCH;  // [row][k] of one segment
    // segment (warp, s) of T: rows of this warp, columns of sub-block s
    auto fetch = [&](int s) {
#pragma unroll 8
        for (int e = lane; e < TS * TS; e += 32) {
            const int i = TRANS ? e % TS : e / TS, k = TRANS ? e / TS : e % TS;
            const int ti = warp * TS + i, tk = s * TS + k;
            const bool ok = ti < kb && tk < kb;
            const C2* src = TRANS ? T + (int64_t)(r0 + tk) * ldt + r0 + ti : T + (int64_t)(r0 + ti) * ldt + r0 + tk;
            cp_elem(buf + i * TRSM_PITCH + k, ok ? src : T, ok);
        }
        dmma::cp_commit();
    };
    fetch(warp);
    C2 x[RB], inv = zero, D[TS];
#pragma unroll
    for (int c = 0; c < RB; c++) {
        x[c] = zero;
        if (row && c < nc) x[c] = B_ROWMAJOR ? B[(int64_t)(br0 + r) * ldb + cb + c] : B[(int64_t)(cb + c) * ldb + br0 + r];
    }
    dmma::cp_wait<0>();
    __syncwarp();
    if (UPPER && !UNIT && row) {
        C2 one = zero;
        one.x = 1;
        inv = cdiv(one, buf[lane * TRSM_PITCH + lane]);
    }
#pragma unroll
    for (int k = 0; k < TS; k++) {
        D[k] = zero;
        if (UPPER ? k > lane : k < lane) D[k] = buf[lane * TRSM_PITCH + k];
        if (UPPER && !UNIT) D[k] = panel_mul(D[k], inv);
    }
    __syncwarp();
    if (UPPER ? warp < nsb - 1 : warp > 0) fetch(UPPER ? nsb - 1 : 0);
    for (int step = 0; step < nsb; step++) {
        const int s = UPPER ? nsb - 1 - step : step, par = step & 1;
        if (warp == s) {
            if (UPPER && !UNIT) {
#pragma unroll
                for (int c = 0; c < RB; c++) x[c] = panel_mul(x[c], inv);
            }
#pragma unroll
            for (int kk = 0; kk < TS; kk++) {
                const int k = UPPER ? TS - 1 - kk : kk;
                const bool open = UPPER ? lane < k : lane > k;
#pragma unroll
                for (int c = 0; c < RB; c++) {
                    const C2 xk = shfl_c(x[c], k);
                    if (open) csub_mul(x[c], D[k], xk);
                }
            }
#pragma unroll
            for (int c = 0; c < RB; c++) xs[par][lane][c] = x[c];
        }
        const bool later = UPPER ? warp < s : warp > s;
        if (later) dmma::cp_wait<0>();
        __syncthreads();
        if (later) {
            const C2* t = buf + lane * TRSM_PITCH;
#pragma unroll 8
            for (int k = 0; k < TS; k++) {
                const C2 tk = t[k];
#pragma unroll
                for (int c = 0; c < RB; c++) csub_mul(x[c], tk, xs[par][k][c]);
            }
            __syncwarp();
            const int next = UPPER ? s - 1 : s + 1;
            if (UPPER ? warp < next : warp > next) fetch(next);
        }
    }
    if (!row) return;
    C2 dd = zero;
    if (DIVDIAG) dd = T[(int64_t)(r0 + r) * ldt + r0 + r];
#pragma unroll
    for (int c = 0; c < RB; c++) {
        if (c >= nc) break;
        const C2 v = DIVDIAG ? cdiv(x[c], dd) : x[c];
        if (B_ROWMAJOR) B[(int64_t)(br0 + r) * ldb + cb + c] = v;
        else B[(int64_t)(cb + c) * ldb + br0 + r] = v;
    }
}

template <typename R, bool UPPER, bool B_ROWMAJOR, int RB, int MODE>
static int launch_trsm_block(bem_ctx* ctx, const typename C2T<R>::type* T, int64_t ldt, int r0, int kb,
                             typename C2T<R>::type* B, int64_t ldb, int c0, int c1, int br0, int batch, int64_t sT,
                             int64_t sB) {
    using C2 = typename C2T<R>::type;
    // the attribute is per device: one bit per device id, set once
    static std::atomic<unsigned long long> attr_set{0};
    const unsigned long long bit = 1ull << (ctx->device & 63);
    if (!(attr_set.load() & bit)) {
        BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(trsm_block_kernel<R, UPPER, B_ROWMAJOR, RB, MODE>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(TRSM_KB * TRSM_PITCH * sizeof(C2))));
        attr_set.fetch_or(bit);
    }
    const int threads = (kb + TRSM_TS - 1) / TRSM_TS * TRSM_TS;
    const dim3 grid((c1 - c0 + RB - 1) / RB, batch);
    trsm_block_kernel<R, UPPER, B_ROWMAJOR, RB, MODE><<<grid, threads, (size_t)threads * TRSM_PITCH * sizeof(C2), ctx->stream>>>(
        T, ldt, r0, kb, B, ldb, br0, c0, c1, sT, sB);
    return BEM_OK;
}

// B's rows of the block start at br0 (at r0, the block's own rows, when br0 < 0).
// Columns per CTA: one while that gives no more CTAs than SMs, then two (the
// substitution's chain is the time: 20, 22 to 24 us), else eight, whose
// registers still hold the rows of T.
template <typename R, bool UPPER, bool B_ROWMAJOR, int MODE = 0>
int trsm_block(bem_ctx* ctx, const typename C2T<R>::type* T, int64_t ldt, int r0, int kb,
               typename C2T<R>::type* B, int64_t ldb, int c0, int c1, int br0 = -1, int batch = 1, int64_t sT = 0,
               int64_t sB = 0) {
    if (br0 < 0) br0 = r0;
    using C2 = typename C2T<R>::type;
    if (c1 <= c0 || kb <= 0) return BEM_OK;
    if (kb > TRSM_KB) return fail(ctx, BEM_ERR_INVALID, "block TRSM: %d rows > %d", kb, TRSM_KB);
    cudaEvent_t ev = ctx->prof_begin(PROF_TRSM);
    if ((int64_t)(c1 - c0) * batch <= ctx->sm_count)
        BEM_TRY((launch_trsm_block<R, UPPER, B_ROWMAJOR, 1, MODE>(ctx, T, ldt, r0, kb, B, ldb, c0, c1, br0, batch, sT, sB)));
    else if ((int64_t)(c1 - c0 + 1) / 2 * batch <= ctx->sm_count)
        BEM_TRY((launch_trsm_block<R, UPPER, B_ROWMAJOR, 2, MODE>(ctx, T, ldt, r0, kb, B, ldb, c0, c1, br0, batch, sT, sB)));
    else
        BEM_TRY((launch_trsm_block<R, UPPER, B_ROWMAJOR, 8, MODE>(ctx, T, ldt, r0, kb, B, ldb, c0, c1, br0, batch, sT, sB)));
    BEM_LAUNCHED(ctx);
    if (ev)
        ctx->prof_end(PROF_TRSM, ev, 4.0 * kb * (double)kb * (c1 - c0) * batch,
                      (double)sizeof(C2) * ((double)kb * kb / 2 + 2.0 * kb * (c1 - c0)) * batch);
    return BEM_OK;
}

// Unit-lower TRSM on rows [r0, r0+kb) of the row-major matrix itself, for
// columns [c0, c1): the U12 step of the factorisation.
template <typename R>
int trsm_rows_lower_unit(bem_ctx* ctx, typename C2T<R>::type* A, int64_t lda, int r0, int kb,
                         int c0, int c1, int batch = 1, int64_t sA = 0) {
    return trsm_block<R, false, true>(ctx, A, lda, r0, kb, A, lda, c0, c1, -1, batch, sA, sA);
}

// U12 = L11^-1 A12 for the jb x jb unit lower block at (j0, j0), columns
// [c0, n), as a blocked forward substitution: 64-row slabs solved by the
// block triangular solve, each followed by the GEMM update of the slabs
// below (on the FP64 tensor path).  The same arithmetic as the block solve
// of all jb rows, regrouped: three quarters of its flops move to the GEMM.
constexpr int U12_SLAB = 64;
template <typename R>
static int u12_blocked(bem_ctx* ctx, typename C2T<R>::type* A, int64_t lda, int j0, int jb, int c0, int n, int batch,
                       int64_t sA) {
    using C2 = typename C2T<R>::type;
    const int nc = n - c0;
    for (int s0 = 0; s0 < jb; s0 += U12_SLAB) {
        const int sb = std::min(U12_SLAB, jb - s0), below = jb - s0 - sb;
        BEM_TRY(trsm_rows_lower_unit<R>(ctx, A, lda, j0 + s0, sb, c0, n, batch, sA));
        if (below > 0)
            BEM_TRY(cgemm<R>(ctx, below, nc, sb, A + (int64_t)(j0 + s0 + sb) * lda + j0 + s0, lda,
                             A + (int64_t)(j0 + s0) * lda + c0, lda, false, A + (int64_t)(j0 + s0 + sb) * lda + c0, lda,
                             false, mk<C2>(-1, 0), mk<C2>(1, 0), PROF_TRSM, batch, sA, sA, sA));
    }
    return BEM_OK;
}

// ------------------------------------------------------------------ getrf
template <typename R>
int getrf(bem_ctx* ctx, typename C2T<R>::type* A, int64_t lda, int n, int* d_ipiv, int* d_info,
          const TrailingUpdate<R>* tc) {
    using C2 = typename C2T<R>::type;
    const int NB = 256;
    const int W = sizeof(R) == 8 ? 16 : 32;
    // panel workspace
    int occ = 0;
    const int Gmax_sm = ctx->sm_count;
    // rows per CTA for the first (largest) panel decides the shared memory
    // Rows per CTA: ceil(nrows / G) with G = min(SMs, nrows / w); it is at
    // most ceil(n / SMs) while G is capped by the SM count and below 2w
    // once G is nrows / w, so this bounds every panel launch.
    int G0 = std::min(Gmax_sm, std::max(1, n / W));
    int Rp0 = std::max((n + G0 - 1) / G0, 2 * W);
    size_t smem0 = ((size_t)Rp0 * W + W) * sizeof(C2);
    if (smem0 > PANEL_SMEM)
        return fail(ctx, BEM_ERR_INVALID, "n=%d too large for the panel kernel (%zu B smem)", n, smem0);
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(panel_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, PANEL_SMEM));
    BEM_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, panel_kernel<R>, 256, smem0));
    if (occ < 1) return fail(ctx, BEM_ERR_INVALID, "panel kernel does not fit on an SM");
    const int Gcap = occ * ctx->sm_count;
    // workspace: cval[2G] (R), crow[2G], cdata[2G*W], disp[2W], bar, status
    size_t ws_bytes = 0;
    auto take = [&](size_t b) { size_t o = ws_bytes; ws_bytes += (b + 255) & ~(size_t)255; return o; };
    size_t o_cval = take(2 * (size_t)Gcap * sizeof(R)), o_crow = take(2 * (size_t)Gcap * 4),
           o_cdata = take(2 * (size_t)Gcap * W * sizeof(C2)), o_disp = take(2 * W * sizeof(C2)),
           o_bar = take(256), o_mv = take(2 * (size_t)n * sizeof(int));
    BEM_TRY(ctx->ensure_ws(ws_bytes));
    char* ws = (char*)ctx->ws;
    PanelWS pw;
    pw.cval = ws + o_cval;
    pw.crow = (int*)(ws + o_crow);
    pw.cdata = ws + o_cdata;
    pw.disp = ws + o_disp;
    pw.bar = (unsigned*)(ws + o_bar);
    pw.status = ctx->d_status;
    int* d_moves = (int*)(ws + o_mv);
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(d_info, 0, sizeof(int), ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream));
    // FP64: U12 = L11^-1 A12 by 64-row slabs with GEMM updates between them
    // (u12_blocked) instead of one block triangular solve of 256 rows
    const bool u12b = sizeof(R) == 8 && ctx->lu_u12_slabs;
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = std::min(NB, n - j0);
        for (int i0 = j0; i0 < j0 + jb; i0 += W) {
            const int iw = std::min(W, j0 + jb - i0);
            const int nrows = n - i0;
            const PanelShape ps = panel_reg_choice<R>(ctx, nrows, iw, 1);
            if (ps.C > 0) {
                BEM_TRY(launch_panel_reg<R>(ctx, A, lda, n, i0, nrows, iw, d_ipiv, d_info, d_moves, 1, 0, ps));
            } else {
                int G = std::min(Gcap, std::max(1, nrows / iw));
                G = std::min(G, Gmax_sm);
                int Rp = (nrows + G - 1) / G;
                G = (nrows + Rp - 1) / Rp;
                size_t smem = ((size_t)Rp * iw + iw) * sizeof(C2);
                if (smem > smem0) return fail(ctx, BEM_ERR_INVALID, "panel smem bound violated");
                BEM_TRY_CUDA(ctx, cudaMemsetAsync(pw.bar, 0, sizeof(unsigned), ctx->stream));
                int64_t s0 = 0;
                int p0 = 0;
                void* args[] = {&A, (void*)&lda, (void*)&i0, (void*)&nrows, (void*)&iw, (void*)&Rp,
                                &d_ipiv, &d_info, &pw, &G, &s0, &p0};
                cudaEvent_t ev = ctx->prof_begin(PROF_PANEL);
                BEM_TRY_CUDA(ctx, cudaLaunchCooperativeKernel((void*)panel_kernel<R>, dim3(G), dim3(256),
                                                              args, smem, ctx->stream));
                BEM_LAUNCHED(ctx);
                if (ev)
                    ctx->prof_end(PROF_PANEL, ev, 8.0 * (double)nrows * iw * iw / 2,
                                  (double)nrows * iw * 2 * sizeof(C2));
                moves_kernel<<<1, 32, 0, ctx->stream>>>(d_ipiv, n, i0, iw, d_moves, 1, ctx->d_status);
                BEM_LAUNCHED(ctx);
            }
            // interchanges on the rest of this block column, and the sub-panel's U12
            int ca0 = j0, ca1 = i0, cb0 = i0 + iw, cb1 = j0 + jb;
            int ncol = (ca1 - ca0) + (cb1 - cb0);
            if (ncol > 0) {
                cudaEvent_t ev = ctx->prof_begin(PROF_PIVOT);
                move_rows_kernel<R, true><<<(ncol + 63) / 64, 64, 0, ctx->stream>>>(A, lda, d_moves, n, i0, i0 + iw, iw,
                                                                                  ca0, ca1, cb0, cb1, ctx->d_status);
                BEM_LAUNCHED(ctx);
                if (ev) ctx->prof_end(PROF_PIVOT, ev, 0.0, 4.0 * sizeof(C2) * iw * (double)ncol);
            }
            if (cb1 > cb0) {
                BEM_TRY(cgemm<R>(ctx, n - i0 - iw, cb1 - cb0, iw, A + (int64_t)(i0 + iw) * lda + i0, lda,
                                 A + (int64_t)i0 * lda + cb0, lda, false,
                                 A + (int64_t)(i0 + iw) * lda + cb0, lda, false, mk<C2>(-1, 0),
                                 mk<C2>(1, 0), PROF_PANEL_UPDATE));
            }
        }
        // interchanges on the columns outside the block column
        int ncol = j0 + (n - j0 - jb);
        if (ncol > 0) {
            cudaEvent_t ev = ctx->prof_begin(PROF_PIVOT);
            move_rows_kernel<R, false><<<(ncol + 63) / 64, 64, 0, ctx->stream>>>(A, lda, d_moves, n, j0, j0 + jb, W, 0, j0,
                                                                               j0 + jb, n, ctx->d_status);
            BEM_LAUNCHED(ctx);
            if (ev) ctx->prof_end(PROF_PIVOT, ev, 0.0, 4.0 * sizeof(C2) * jb * (double)ncol);
        }
        const int c0 = j0 + jb;
        if (c0 < n) {
            if (u12b) {
                BEM_TRY(u12_blocked<R>(ctx, A, lda, j0, jb, c0, n, 1, 0));
            } else {
                BEM_TRY(trsm_rows_lower_unit<R>(ctx, A, lda, j0, jb, c0, n));
            }
            const int Mt = n - c0;
            if (tc && tc->fn)
                BEM_TRY(tc->fn(ctx, tc->state, Mt, Mt, jb, A + (int64_t)c0 * lda + j0, lda,
                               A + (int64_t)j0 * lda + c0, lda, A + (int64_t)c0 * lda + c0, lda));
            else
                BEM_TRY(cgemm<R>(ctx, Mt, Mt, jb, A + (int64_t)c0 * lda + j0, lda, A + (int64_t)j0 * lda + c0,
                                 lda, false, A + (int64_t)c0 * lda + c0, lda, false, mk<C2>(-1, 0),
                                 mk<C2>(1, 0), PROF_LU_UPDATE));
        }
    }
    return BEM_OK;
}

// ------------------------------------------------------------------ getrs
// X = (P^T L U)^-1 B, column-major n x nrhs; X may alias B only if perm is
// applied through the workspace (the caller passes distinct buffers).
template <typename R>
int getrs(bem_ctx* ctx, const typename C2T<R>::type* LU, int64_t lda, int n, const int* d_perm,
          const typename C2T<R>::type* B, int64_t ldb, typename C2T<R>::type* X, int64_t ldx,
          int nrhs, const TrailingUpdate<R>* tc) {
    using C2 = typename C2T<R>::type;
    const int NB = 256;
    if (nrhs <= 0) return BEM_OK;
    int64_t tot = (int64_t)n * nrhs;
    permute_rows_kernel<R><<<(unsigned)((tot + 255) / 256), 256, 0, ctx->stream>>>(B, ldb, X, ldx, d_perm,
                                                                                  n, nrhs);
    BEM_LAUNCHED(ctx);
    // forward: L Y = P B
    for (int j0 = 0; j0 < n; j0 += NB) {
        int jb = std::min(NB, n - j0);
        BEM_TRY((trsm_block<R, false, false>(ctx, LU, lda, j0, jb, X, ldx, 0, nrhs)));
        int below = n - j0 - jb;
        if (below > 0) {
            if (tc && tc->fn_solve)
                BEM_TRY(tc->fn_solve(ctx, tc->state, below, nrhs, jb, LU + (int64_t)(j0 + jb) * lda + j0, lda,
                                     X + j0, ldx, X + j0 + jb, ldx));
            else
                BEM_TRY(cgemm<R>(ctx, below, nrhs, jb, LU + (int64_t)(j0 + jb) * lda + j0, lda, X + j0, ldx,
                                 true, X + j0 + jb, ldx, true, mk<C2>(-1, 0), mk<C2>(1, 0), PROF_SOLVE_UPDATE));
        }
    }
    // backward: U X = Y
    int nblk = (n + NB - 1) / NB;
    for (int bi = nblk - 1; bi >= 0; bi--) {
        int j0 = bi * NB, jb = std::min(NB, n - j0);
        BEM_TRY((trsm_block<R, true, false>(ctx, LU, lda, j0, jb, X, ldx, 0, nrhs)));
        if (j0 > 0) {
            if (tc && tc->fn_solve)
                BEM_TRY(tc->fn_solve(ctx, tc->state, j0, nrhs, jb, LU + j0, lda, X + j0, ldx, X, ldx));
            else
                BEM_TRY(cgemm<R>(ctx, j0, nrhs, jb, LU + j0, lda, X + j0, ldx, true, X, ldx, true,
                                 mk<C2>(-1, 0), mk<C2>(1, 0), PROF_SOLVE_UPDATE));
        }
    }
    return BEM_OK;
}

// ------------------------------------------------------------- batched FP64
// The blocked LU of getrf for a batch of equally sized matrices, one launch
// per step for the whole batch.  The panel's CTAs per matrix (Gm) are as many
// as fit co-resident next to the other matrices' (one cooperative grid);
// batches larger than that are factored in chunks.
int getrf_batched(bem_ctx* ctx, double2* A, int64_t lda, int64_t sA, int n, int batch, int* d_ipiv, int* d_info,
                  LuShape shape, bool clear_status) {
    using R = double;
    using C2 = double2;
    const int NB = shape.NB, W = shape.W;
    if (n < 1 || batch < 1) return fail(ctx, BEM_ERR_INVALID, "batched LU: n=%d batch=%d", n, batch);
    if (W < 1 || W > PanelW<R>::v || NB < W || NB > TRSM_KB || NB % W != 0)
        return fail(ctx, BEM_ERR_INVALID, "batched LU shape NB=%d W=%d", NB, W);
    const size_t smem_max = PANEL_SMEM;
    // every sub-panel fits one cluster (the first is the tallest): no
    // cooperative grid, no chunking of the batch
    const bool all_clusters = panel_reg_choice<R>(ctx, n, W, batch).C > 0;
    const int Rp_max = (int)std::min<int64_t>(n, ((int64_t)smem_max / (int64_t)sizeof(C2) - W) / W);
    if (Rp_max < 2 * W) return fail(ctx, BEM_ERR_INVALID, "batched LU: panel does not fit");
    const int Gm_min = (n + Rp_max - 1) / Rp_max;
    // CTAs per matrix for the first panel, and the batch chunk that fits
    int Gm = std::max(Gm_min, std::min(std::max(1, n / W), ctx->sm_count));
    int Rp0 = 0, occ = 0;
    size_t smem0 = 0;
    int chunk = 0;
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(panel_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem_max));
    for (;;) {
        Rp0 = std::max((n + Gm - 1) / Gm, 2 * W);
        smem0 = ((size_t)Rp0 * W + W) * sizeof(C2);
        BEM_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, panel_kernel<R>, 256, smem0));
        if (occ < 1) return fail(ctx, BEM_ERR_INVALID, "batched LU: panel kernel does not fit on an SM");
        chunk = std::min(batch, occ * ctx->sm_count / Gm);
        if (chunk >= batch || Gm == Gm_min) break;
        Gm = std::max(Gm_min, std::min(Gm - 1, occ * ctx->sm_count / batch));
    }
    if (all_clusters) chunk = batch;
    if (chunk < 1) return fail(ctx, BEM_ERR_INVALID, "batched LU: no co-resident panel grid");
    if (chunk < batch) {
        for (int b0 = 0; b0 < batch; b0 += chunk) {
            const int nb = std::min(chunk, batch - b0);
            BEM_TRY(getrf_batched(ctx, A + (int64_t)b0 * sA, lda, sA, n, nb, d_ipiv + (int64_t)b0 * n, d_info + b0,
                                  shape, clear_status && b0 == 0));
        }
        return BEM_OK;
    }
    size_t ws_bytes = 0;
    auto take = [&](size_t b) { size_t o = ws_bytes; ws_bytes += (b + 255) & ~(size_t)255; return o; };
    const size_t per = (size_t)batch * 2 * Gm;
    size_t o_cval = take(per * sizeof(R)), o_crow = take(per * 4), o_cdata = take(per * W * sizeof(C2)),
           o_disp = take((size_t)batch * 2 * W * sizeof(C2)), o_bar = take(256),
           o_mv = take((size_t)batch * 2 * n * sizeof(int));
    BEM_TRY(ctx->ensure_ws(ws_bytes));
    char* ws = (char*)ctx->ws;
    PanelWS pw;
    pw.cval = ws + o_cval;
    pw.crow = (int*)(ws + o_crow);
    pw.cdata = ws + o_cdata;
    pw.disp = ws + o_disp;
    pw.bar = (unsigned*)(ws + o_bar);
    pw.status = ctx->d_status;
    int* d_moves = (int*)(ws + o_mv);
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(d_info, 0, batch * sizeof(int), ctx->stream));
    // the chunks of a batch keep one status word: a wait that ran out in an earlier one is not forgotten
    if (clear_status) BEM_TRY_CUDA(ctx, cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream));
    const C2 m1 = mk<C2>(-1, 0), p1 = mk<C2>(1, 0);
    // U12 by 64-row slabs, as in getrf (the same arithmetic per matrix)
    const bool u12b = ctx->lu_u12_slabs;
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = std::min(NB, n - j0);
        for (int i0 = j0; i0 < j0 + jb; i0 += W) {
            const int iw = std::min(W, j0 + jb - i0);
            const int nrows = n - i0;
            const PanelShape ps = panel_reg_choice<R>(ctx, nrows, iw, batch);
            if (ps.C > 0) {
                BEM_TRY(launch_panel_reg<R>(ctx, A, lda, n, i0, nrows, iw, d_ipiv, d_info, d_moves, batch, sA, ps));
            } else {
                int G = std::min(Gm, std::max(1, nrows / iw));
                const int Rp = (nrows + G - 1) / G;
                G = (nrows + Rp - 1) / Rp;
                const size_t smem = ((size_t)Rp * iw + iw) * sizeof(C2);
                if (smem > smem0 || Rp < iw) return fail(ctx, BEM_ERR_INVALID, "batched LU: panel bound violated");
                BEM_TRY_CUDA(ctx, cudaMemsetAsync(pw.bar, 0, sizeof(unsigned), ctx->stream));
                int spiv = n;
                void* args[] = {&A, (void*)&lda, (void*)&i0, (void*)&nrows, (void*)&iw, (void*)&Rp,
                                &d_ipiv, &d_info, &pw, &G, &sA, &spiv};
                cudaEvent_t ev = ctx->prof_begin(PROF_PANEL);
                BEM_TRY_CUDA(ctx, cudaLaunchCooperativeKernel((void*)panel_kernel<R>, dim3(G * batch), dim3(256),
                                                              args, smem, ctx->stream));
                BEM_LAUNCHED(ctx);
                if (ev)
                    ctx->prof_end(PROF_PANEL, ev, 8.0 * (double)nrows * iw * iw / 2 * batch,
                                  (double)nrows * iw * 2 * sizeof(C2) * batch);
                moves_kernel<<<(batch + 31) / 32, 32, 0, ctx->stream>>>(d_ipiv, n, i0, iw, d_moves, batch, ctx->d_status);
                BEM_LAUNCHED(ctx);
            }
            const int ca0 = j0, ca1 = i0, cb0 = i0 + iw, cb1 = j0 + jb;
            const int ncol = (ca1 - ca0) + (cb1 - cb0);
            if (ncol > 0) {
                cudaEvent_t ev = ctx->prof_begin(PROF_PIVOT);
                move_rows_kernel<R, true><<<dim3((ncol + 63) / 64, batch), 64, 0, ctx->stream>>>(
                    A, lda, d_moves, n, i0, i0 + iw, iw, ca0, ca1, cb0, cb1, ctx->d_status, sA);
                BEM_LAUNCHED(ctx);
                if (ev) ctx->prof_end(PROF_PIVOT, ev, 0.0, 4.0 * sizeof(C2) * iw * (double)ncol * batch);
            }
            if (cb1 > cb0) {
                BEM_TRY(cgemm<R>(ctx, n - i0 - iw, cb1 - cb0, iw, A + (int64_t)(i0 + iw) * lda + i0, lda,
                                 A + (int64_t)i0 * lda + cb0, lda, false, A + (int64_t)(i0 + iw) * lda + cb0, lda,
                                 false, m1, p1, PROF_PANEL_UPDATE, batch, sA, sA, sA));
            }
        }
        const int ncol = j0 + (n - j0 - jb);
        if (ncol > 0) {
            cudaEvent_t ev = ctx->prof_begin(PROF_PIVOT);
            move_rows_kernel<R, false><<<dim3((ncol + 63) / 64, batch), 64, 0, ctx->stream>>>(A, lda, d_moves, n, j0, j0 + jb,
                                                                                            W, 0, j0, j0 + jb, n, ctx->d_status, sA);
            BEM_LAUNCHED(ctx);
            if (ev) ctx->prof_end(PROF_PIVOT, ev, 0.0, 4.0 * sizeof(C2) * jb * (double)ncol * batch);
        }
        const int c0 = j0 + jb;
        if (c0 < n) {
            if (u12b)
                BEM_TRY(u12_blocked<R>(ctx, A, lda, j0, jb, c0, n, batch, sA));
            else
                BEM_TRY(trsm_rows_lower_unit<R>(ctx, A, lda, j0, jb, c0, n, batch, sA));
            const int Mt = n - c0;
            BEM_TRY(cgemm<R>(ctx, Mt, Mt, jb, A + (int64_t)c0 * lda + j0, lda, A + (int64_t)j0 * lda + c0, lda, false,
                             A + (int64_t)c0 * lda + c0, lda, false, m1, p1, PROF_LU_UPDATE, batch, sA, sA, sA));
        }
    }
    return BEM_OK;
}

int getrs_batched(bem_ctx* ctx, const double2* LU, int64_t lda, int64_t sA, int n, int batch, const int* d_perm,
                  const double2* B, int64_t ldb, int64_t sB, double2* X, int64_t ldx, int64_t sX, int nrhs, int NB) {
    using R = double;
    using C2 = double2;
    if (nrhs <= 0 || batch <= 0) return BEM_OK;
    if (NB < 1 || NB > TRSM_KB) return fail(ctx, BEM_ERR_INVALID, "batched solve block %d", NB);
    const int64_t tot = (int64_t)n * nrhs;
    permute_rows_kernel<R><<<dim3((unsigned)((tot + 255) / 256), batch), 256, 0, ctx->stream>>>(
        B, ldb, X, ldx, d_perm, n, nrhs, sB, sX, n);
    BEM_LAUNCHED(ctx);
    const C2 m1 = mk<C2>(-1, 0), p1 = mk<C2>(1, 0);
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = std::min(NB, n - j0);
        BEM_TRY((trsm_block<R, false, false>(ctx, LU, lda, j0, jb, X, ldx, 0, nrhs, -1, batch, sA, sX)));
        const int below = n - j0 - jb;
        if (below > 0)
            BEM_TRY(cgemm<R>(ctx, below, nrhs, jb, LU + (int64_t)(j0 + jb) * lda + j0, lda, X + j0, ldx, true,
                             X + j0 + jb, ldx, true, m1, p1, PROF_SOLVE_UPDATE, batch, sA, sX, sX));
    }
    const int nblk = (n + NB - 1) / NB;
    for (int bi = nblk - 1; bi >= 0; bi--) {
        const int j0 = bi * NB, jb = std::min(NB, n - j0);
        BEM_TRY((trsm_block<R, true, false>(ctx, LU, lda, j0, jb, X, ldx, 0, nrhs, -1, batch, sA, sX)));
        if (j0 > 0)
            BEM_TRY(cgemm<R>(ctx, j0, nrhs, jb, LU + j0, lda, X + j0, ldx, true, X, ldx, true, m1, p1,
                             PROF_SOLVE_UPDATE, batch, sA, sX, sX));
    }
    return BEM_OK;
}

// Deterministic fill of a batch of test matrices for the autotuner: entries
// in [-1, 1) from an integer hash, plus n on the diagonal.
static __global__ void tune_fill_kernel(double2* A, int n, int64_t total) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    uint64_t h = (uint64_t)i * 0x9E3779B97F4A7C15ull;
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 29;
    const double re = (double)(h & 0xFFFFFF) / 8388608.0 - 1.0, im = (double)((h >> 24) & 0xFFFFFF) / 8388608.0 - 1.0;
    const int64_t e = i % ((int64_t)n * n);
    const bool diag = e / n == e % n;
    A[i] = make_double2(re + (diag ? n : 0.0), im);
}

// Shape of the batched FP64 LU for (n, batch): every candidate block / panel
// width is timed once (after one warm-up) on min(batch, 8) test matrices of
// order n, and the fastest kept for the context's later batches of that
// shape.
int tune_lu_shape(bem_ctx* ctx, int n, int batch, LuShape* out) {
    static std::map<std::pair<int, int>, LuShape> cache;  // per process: (n, batch) -> shape
    const int tb = std::min(batch, 8);
    const auto key = std::make_pair(n, tb);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return BEM_OK;
    }
    const LuShape cands[] = {{256, 16}, {128, 16}, {256, 8}, {128, 8}, {64, 16}};
    const size_t nn = (size_t)n * n;
    void* A = devmem_alloc(ctx->device, nn * tb * sizeof(double2), ctx);
    void* ip = devmem_alloc(ctx->device, (size_t)n * tb * sizeof(int) + (size_t)tb * sizeof(int), ctx);
    if (!A || !ip) {
        if (A) devmem_free(ctx->device, A, nn * tb * sizeof(double2), ctx);
        if (ip) devmem_free(ctx->device, ip, (size_t)n * tb * sizeof(int) + (size_t)tb * sizeof(int), ctx);
        *out = LuShape{};
        return BEM_OK;  // no room to tune: the default shape
    }
    int* d_ipiv = (int*)ip;
    int* d_info = d_ipiv + (size_t)n * tb;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float best = 1e30f;
    LuShape pick{};
    int s = BEM_OK;
    for (const LuShape& c : cands) {
        if (c.NB > n && c.NB != 256) continue;
        float ms = 0.f;
        for (int rep = 0; rep < 2 && s == BEM_OK; rep++) {
            const int64_t tot = (int64_t)nn * tb;
            tune_fill_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, ctx->stream>>>((double2*)A, n, tot);
            ctx->launches++;
            cudaEventRecord(e0, ctx->stream);
            s = getrf_batched(ctx, (double2*)A, n, (int64_t)nn, n, tb, d_ipiv, d_info, c);
            cudaEventRecord(e1, ctx->stream);
            if (cudaEventSynchronize(e1) != cudaSuccess) s = fail(ctx, BEM_ERR_CUDA, "LU autotuner");
            cudaEventElapsedTime(&ms, e0, e1);
        }
        if (s != BEM_OK) break;
        if (ms < best) best = ms, pick = c;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    devmem_free(ctx->device, A, nn * tb * sizeof(double2), ctx);
    devmem_free(ctx->device, ip, (size_t)n * tb * sizeof(int) + (size_t)tb * sizeof(int), ctx);
    if (s != BEM_OK) return s;
    cache[key] = pick;
    *out = pick;
    return BEM_OK;
}

template int getrf<double>(bem_ctx*, double2*, int64_t, int, int*, int*, const TrailingUpdate<double>*);
template int getrf<float>(bem_ctx*, float2*, int64_t, int, int*, int*, const TrailingUpdate<float>*);
template int getrs<double>(bem_ctx*, const double2*, int64_t, int, const int*, const double2*, int64_t,
                           double2*, int64_t, int, const TrailingUpdate<double>*);
template int getrs<float>(bem_ctx*, const float2*, int64_t, int, const int*, const float2*, int64_t,
                          float2*, int64_t, int, const TrailingUpdate<float>*);
template int cgemm<double>(bem_ctx*, int, int, int, const double2*, int64_t, const double2*, int64_t, bool,
                           double2*, int64_t, bool, double2, double2, int, int, int64_t, int64_t, int64_t);
template int cgemm<float>(bem_ctx*, int, int, int, const float2*, int64_t, const float2*, int64_t, bool,
                          float2*, int64_t, bool, float2, float2, int, int, int64_t, int64_t, int64_t);

// ============================================================ L D L^T
// Complex-symmetric factorisation without pivoting, S = L D L^T, for the
// FP32 + refinement solve of matrices with S = Z diag(s) symmetric: the
// PMCHWT matrix is [[A, -K], [K, C]] with A, C and K symmetric (the Galerkin
// L and K operators are), so Z diag(I, -I) = [[A, K], [K, -C]] is symmetric.
// Its diagonal blocks dominate enough that elimination without pivoting
// stays as accurate as partial pivoting on these systems (pivot growth below
// 5 at 2N = 960..3840); the refinement residual uses the original FP64 Z, and
// a factorisation that hits a zero pivot or does not let the refinement
// converge is redone with partial pivoting by the caller.  Half the flops of
// LU (the trailing update touches only the lower triangle) and no pivot
// search, so no grid-wide barrier per column.

// Exact (bitwise) symmetry tests of Z and of Z diag(I, -I), 32 x 32 tiles of
// the lower triangle (tile t, row by row) against the mirrored tiles.  flags
// bit 0: Z is not symmetric; bit 1: Z diag(I, -I) is not (n odd counts as
// not).  Both tiles' loads are issued together, 8 in flight per thread; Z is
// read once, bound by HBM (2N = 15360: 1.31 -> 1.19 ms).
__global__ void __launch_bounds__(256) sym_check_kernel(const double2* __restrict__ Z, int64_t ldz, int n,
                                                        unsigned* __restrict__ flags) {
    const int64_t t = blockIdx.x;
    int bi = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((int64_t)(bi + 1) * (bi + 2) / 2 <= t) bi++;
    while ((int64_t)bi * (bi + 1) / 2 > t) bi--;
    const int bj = (int)(t - (int64_t)bi * (bi + 1) / 2);
    __shared__ double2 tt[32][33];
    __shared__ int done;
    if (threadIdx.x == 0) done = *(volatile unsigned*)flags == 3u;  // both tests already failed
    __syncthreads();
    if (done) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 256 threads
    const int half = (n % 2 == 0) ? n / 2 : -1;
    double2 up[4], low[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int r = ty + 8 * k;
        const int iu = bj * 32 + r, ju = bi * 32 + tx, il = bi * 32 + r, jl = bj * 32 + tx;
        up[k] = (iu < n && ju < n) ? Z[(int64_t)iu * ldz + ju] : make_double2(0.0, 0.0);
        low[k] = (il < n && jl < n) ? Z[(int64_t)il * ldz + jl] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) tt[ty + 8 * k][tx] = up[k];
    __syncthreads();
    unsigned bad = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int r = ty + 8 * k, i = bi * 32 + r, j = bj * 32 + tx;
        if (i >= n || j >= n || j >= i) continue;
        const double2 a = low[k];      // Z[i][j]
        const double2 b = tt[tx][r];   // Z[j][i]
        if (a.x != b.x || a.y != b.y) bad |= 1u;
        // (Z D)[i][j] = Z[i][j] s_j  vs  (Z D)[j][i] = Z[j][i] s_i
        const double si = (half >= 0 && i >= half) ? -1.0 : 1.0, sj = (half >= 0 && j >= half) ? -1.0 : 1.0;
        if (half < 0 || a.x * sj != b.x * si || a.y * sj != b.y * si) bad |= 2u;
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && bad) atomicOr(flags, bad);
}

// Factors the jb x jb diagonal block at (j0, j0) in place: the strict lower
// triangle receives L, the diagonal D (the upper triangle is not touched).
// One CTA of 256 threads, thread i owning row i of the block.  The block is
// taken in 32-column sub-panels: each thread keeps its row's 32 sub-panel
// entries in registers and the columns are eliminated one at a time, with
// one block barrier per column (the pivot and the unscaled pivot column are
// published in shared memory, double-buffered by column parity); every row
// then scales by the pivot's reciprocal and applies the rank-1 update to
// its own registers.  The rest of the block's lower triangle is updated
// with the sub-panel: T = D L^T of the sub-panel is formed once in shared
// memory, and each thread accumulates an 8 x 4 set of outputs of a
// 128 x 64 block (rows ty + 16 r, columns tx + 16 c).  *info: first zero
// pivot (1-based).
constexpr int LDLT_SP = 32, LDLT_PITCH = LDLT_SP + 1, LDLT_TP = 256, LDLT_THREADS = 256;
constexpr size_t ldlt_smem_bytes(size_t esz) {
    return ((size_t)256 * LDLT_PITCH + (size_t)LDLT_SP * LDLT_TP) * esz;
}

template <typename R>
__global__ void __launch_bounds__(LDLT_THREADS, 1)
ldlt_diag_kernel(typename C2T<R>::type* __restrict__ A, int64_t lda, int j0, int jb, int* __restrict__ info) {
    using C2 = typename C2T<R>::type;
    extern __shared__ __align__(16) unsigned char ldlt_smem[];
    C2* P = reinterpret_cast<C2*>(ldlt_smem);  // [jb][LDLT_PITCH]: the eliminated sub-panel, rows c0..
    __shared__ C2 s_piv[2];                    // the pivot d of the column, by column parity
    __shared__ C2 s_col[2][LDLT_SP];           // unscaled column entries a[c][jj] of the sub-panel rows
    const int tid = threadIdx.x;
    C2 zero;
    zero.x = 0;
    zero.y = 0;
    for (int c0 = 0; c0 < jb; c0 += LDLT_SP) {
        const int w = min(LDLT_SP, jb - c0), rows = jb - c0;
        const int i = tid;  // this thread's row of the sub-panel
        const bool act = i < rows;
        // x[c] holds a[i][jj + c]: column jj is always x[0], the row shifting
        // left as columns retire (static register indices)
        C2 x[LDLT_SP];
#pragma unroll
        for (int c = 0; c < LDLT_SP; c++)
            x[c] = (act && c < w) ? A[(int64_t)(j0 + c0 + i) * lda + j0 + c0 + c] : zero;
        for (int jj = 0; jj < w; jj++) {
            const int par = jj & 1;
            if (i == jj) s_piv[par] = x[0];
            if (i > jj && i < w) s_col[par][i] = x[0];
            __syncthreads();
            const C2 d = s_piv[par];
            const bool zp = (d.x == 0 && d.y == 0);
            if (zp && i == jj) atomicCAS(info, 0, j0 + c0 + jj + 1);
            if (act && i > jj) {
                C2 one;
                one.x = 1;
                one.y = 0;
                const C2 inv = zp ? zero : cdiv(one, d);
                const C2 l = panel_mul(x[0], inv);
                // a[i][c] -= l_i (d l_c), d l_c being the unscaled a[c][jj]
#pragma unroll
                for (int c = 1; c < LDLT_SP; c++) {
                    if (jj + c < w) {
                        x[c] = panel_msub(x[c], l, s_col[par][jj + c]);
                    }
                }
                x[0] = l;
            }
            // column jj is final for this row: to shared memory, and its lower part to global
            if (act) {
                P[i * LDLT_PITCH + jj] = x[0];
                if (jj <= i) A[(int64_t)(j0 + c0 + i) * lda + j0 + c0 + jj] = x[0];
            }
#pragma unroll
            for (int c = 0; c + 1 < LDLT_SP; c++) x[c] = x[c + 1];
            x[LDLT_SP - 1] = zero;
        }
        __syncthreads();
        // the block's remaining lower triangle: A[i][c] -= sum_k L[i][k] d_k L[c][k]
        const int rest = rows - w;
        if (rest > 0) {
            C2* T = P + (size_t)256 * LDLT_PITCH;  // [k][c] = d_k L[w + c][k]
            for (int e = tid; e < w * rest; e += LDLT_THREADS) {
                const int k = e / rest, c = e % rest;
                const C2 dk = P[k * LDLT_PITCH + k], lc = P[(w + c) * LDLT_PITCH + k];
                T[k * LDLT_TP + c] = panel_mul(dk, lc);
            }
            __syncthreads();
            // 128 x 64 output blocks of the lower triangle, 8 x 4 per thread
            const int ty = tid >> 4, tx = tid & 15, nbr = (rest + 127) / 128;
            for (int bi = 0; bi < nbr; bi++)
                for (int bc = 0; bc * 64 < min(rest, bi * 128 + 128); bc++) {
                    C2 acc[8][4];
                    int ii[8], cc[4];
#pragma unroll
                    for (int r = 0; r < 8; r++) ii[r] = bi * 128 + ty + 16 * r;
#pragma unroll
                    for (int c = 0; c < 4; c++) cc[c] = bc * 64 + tx + 16 * c;
#pragma unroll
                    for (int r = 0; r < 8; r++)
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            acc[r][c] = (ii[r] < rest && cc[c] <= ii[r])
                                            ? A[(int64_t)(j0 + c0 + w + ii[r]) * lda + j0 + c0 + w + cc[c]]
                                            : zero;
#pragma unroll 2
                    for (int k = 0; k < w; k++) {
                        C2 a[8], b[4];
#pragma unroll
                        for (int r = 0; r < 8; r++) a[r] = ii[r] < rest ? P[(w + ii[r]) * LDLT_PITCH + k] : zero;
#pragma unroll
                        for (int c = 0; c < 4; c++) b[c] = T[k * LDLT_TP + cc[c]];
#pragma unroll
                        for (int r = 0; r < 8; r++)
#pragma unroll
                            for (int c = 0; c < 4; c++) acc[r][c] = panel_msub(acc[r][c], a[r], b[c]);
                    }
#pragma unroll
                    for (int r = 0; r < 8; r++)
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (ii[r] < rest && cc[c] <= ii[r])
                                A[(int64_t)(j0 + c0 + w + ii[r]) * lda + j0 + c0 + w + cc[c]] = acc[r][c];
                }
        }
        __syncthreads();
    }
}

// ------------------------------------- cluster L D L^T diagonal-block kernel
// The block of ldlt_diag_kernel (complex64) on one cluster of 8 CTAs, the
// block kept in distributed shared memory: CTA q holds block rows
// 32q..32q+31, columns 0..32q+31, so no entry makes a round trip through
// L2 between sub-panels.  Per 32-column sub-panel p:
//   A. CTA p factors the 32 x 32 diagonal sub-block, column by column with
//      a block barrier each: a lane per row, its 8 warps hold four columns
//      each; the warp of a column leaves its unscaled entries in U, one store
//      and one load a lane, and the scaling waits for the end;
//   cluster barrier;
//   B. every CTA q > p copies U and the pivots from CTA p and eliminates
//      the sub-panel columns of its own rows (four rows per warp, a lane per
//      column);
//   cluster barrier;
//   C. every CTA q > p updates its rows' lower triangle right of the
//      sub-panel: T = D L^T of block rows 32(p+1)..32q+31 is gathered from
//      CTAs p+1..q, 14 loads in flight per thread, then each thread
//      accumulates 4 rows of one column group after the other: CTA p + 1, on
//      which the next sub-panel waits, has one group.
// Every entry goes through the same operations, in the same order, as in
// ldlt_diag_kernel (the same pivot reciprocal, rank-1 updates in column
// order, T = d_k l_c, the trailing sums in k order).  2 np + 1 cluster
// barriers for np sub-panels, each at the top level of the kernel so that
// every thread of the cluster reaches it; no spin loop.  *info: first zero
// pivot (1-based).
// Bound by the chain A, C of CTA p + 1, B: 108 us per block alone (ncu, 1.9 GHz),
// 123 to 148 us in factorisations of 2N = 15360 and 29040, between tensor-core
// GEMMs at the power cap.  Alone as well: 148 us with four
// rows a warp and a lane per column in A (480 cycles a column, U stored and
// scaled on the way), four gathers in flight and all column groups at once in
// C; 277 us with one warp and a lane per row.
constexpr int LDC_CTAS = 8, LDC_ROWS = 32, LDC_PITCH = 8 * LDC_ROWS + 1, LDC_UP = LDC_ROWS + 1,
              LDC_TP = 7 * LDC_ROWS + 1;
constexpr size_t ldlt_cluster_smem_bytes() {
    return ((size_t)LDC_ROWS * LDC_PITCH + 2 * (size_t)LDC_ROWS * LDC_UP + (size_t)LDC_ROWS * LDC_TP + 2 * LDC_ROWS) *
           sizeof(float2);
}

__global__ void __launch_bounds__(LDLT_THREADS, 1)
ldlt_diag_cluster_kernel(float2* __restrict__ A, int64_t lda, int j0, int jb, int* __restrict__ info) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char ldc_smem[];
    float2* S = reinterpret_cast<float2*>(ldc_smem);  // [32][LDC_PITCH]: this CTA's block rows
    float2* U = S + LDC_ROWS * LDC_PITCH;              // [column][LDC_UP rows]: unscaled sub-block entries (phase A)
    float2* UL = U + LDC_ROWS * LDC_UP;                // the same, CTA p's U (phase B)
    float2* T = UL + LDC_ROWS * LDC_UP;                // [32][LDC_TP]: d_k L[c][k] (phase C)
    float2* dk = T + LDC_ROWS * LDC_TP;                // [32]: the sub-panel's pivots
    float2* dinv = dk + LDC_ROWS;                      // [32]: their reciprocals (0 for a zero pivot)
    const int q = (int)cluster.block_rank(), tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int r0 = q * LDC_ROWS;                       // this CTA's first block row
    const int nr = max(0, min(LDC_ROWS, jb - r0));     // its rows inside the block
    const int ncol = min(r0 + LDC_ROWS, jb);           // columns kept: 0..ncol-1
    const float2 zero = make_float2(0.f, 0.f), one = make_float2(1.f, 0.f);
    // this CTA's rows, columns 0..ncol-1, eight independent loads in flight per thread
    const int nload = nr * ncol;
    for (int e0 = 0; e0 < nload; e0 += 8 * LDLT_THREADS) {
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int e = e0 + u * LDLT_THREADS + tid;
            if (e < nload) v[u] = A[(int64_t)(j0 + r0 + e / ncol) * lda + j0 + e % ncol];
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int e = e0 + u * LDLT_THREADS + tid;
            if (e < nload) S[(e / ncol) * LDC_PITCH + e % ncol] = v[u];
        }
    }
    __syncthreads();
    const int np = (jb + LDC_ROWS - 1) / LDC_ROWS;
    for (int p = 0; p < np; p++) {
        const int c0 = p * LDC_ROWS, w = min(LDC_ROWS, jb - c0);
        // A. the diagonal sub-block (rows c0.. of the block are this CTA's rows 0..w-1):
        // lane: row, warp: four columns (the lower triangle counts); the warp that
        // holds a column publishes its unscaled entries
        if (q == p) {
            float2 x[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int c = wid * 4 + r;
                x[r] = (lane < w && c <= lane) ? S[lane * LDC_PITCH + c0 + c] : zero;
            }
            for (int j4 = 0; j4 < w; j4 += 4) {
#pragma unroll
                for (int r4 = 0; r4 < 4; r4++) {
                    const int jj = j4 + r4;
                    if (jj >= w) break;
                    float2* col = U + jj * LDC_UP;
                    if (wid * 4 == j4) col[lane] = x[r4];
                    __syncthreads();
                    if (wid * 4 + 3 > jj || wid == 0) {  // else this warp's columns are done
                        const float2 d = col[jj];
                        const bool zp = (d.x == 0 && d.y == 0);
                        const float2 inv = zp ? zero : cdiv(one, d);
                        if (tid == 0) {
                            dinv[jj] = inv;
                            if (zp) atomicCAS(info, 0, j0 + c0 + jj + 1);
                        }
                        // rows above the column take part in what lies above the diagonal, which nothing reads
                        const float2 l = panel_mul(col[lane], inv);
#pragma unroll
                        for (int r = 0; r < 4; r++)
                            if (wid * 4 + r > jj) x[r] = panel_msub(x[r], l, col[wid * 4 + r]);
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int c = wid * 4 + r;
                if (lane < w && c <= lane) S[lane * LDC_PITCH + c0 + c] = c < lane ? panel_mul(x[r], dinv[c]) : x[r];
            }
        }
        cluster.sync();
        // B. this CTA's rows below the sub-block
        if (q > p && nr > 0) {
            const float2* Up = cluster.map_shared_rank(U, p);
            const float2* Sp = cluster.map_shared_rank(S, p);
            // rows below: the sub-panel is whole, w = 32
#pragma unroll
            for (int e = tid; e < LDC_ROWS * LDC_ROWS; e += LDLT_THREADS)
                UL[(e >> 5) * LDC_UP + (e & 31)] = Up[(e >> 5) * LDC_UP + (e & 31)];
            if (tid < w) {
                const float2 d = Sp[tid * LDC_PITCH + c0 + tid];
                dk[tid] = d;
                dinv[tid] = (d.x == 0 && d.y == 0) ? zero : cdiv(one, d);
            }
            __syncthreads();
            // warp: four rows, lane: column
            float2 x[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int i = wid * 4 + r;
                x[r] = (i < nr && lane < w) ? S[i * LDC_PITCH + c0 + lane] : zero;
            }
#pragma unroll 4
            for (int jj = 0; jj < w; jj++) {
                const float2 inv = dinv[jj], u = UL[jj * LDC_UP + lane];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float2 l = panel_mul(shfl_c(x[r], jj), inv);
                    if (lane > jj) x[r] = panel_msub(x[r], l, u);
                }
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int i = wid * 4 + r;
                if (i < nr && lane < w) S[i * LDC_PITCH + c0 + lane] = panel_mul(x[r], dinv[lane]);
            }
        }
        cluster.sync();
        // C. this CTA's rows, columns cs..r0+31 of the lower triangle
        if (q > p && nr > 0) {
            const int cs = c0 + w, nc = r0 + LDC_ROWS - cs, ng = nc / 32;  // ng = q - p <= 7
            // 14 independent remote loads in flight per thread (w = 32 here)
            for (int e0 = 0; e0 < LDC_ROWS * nc; e0 += 14 * LDLT_THREADS) {
                float2 lc[14];
#pragma unroll
                for (int u = 0; u < 14; u++) {
                    const int e = e0 + u * LDLT_THREADS + tid, row = cs + (e >> 5);
                    lc[u] = zero;
                    if (e < LDC_ROWS * nc && row < jb)
                        lc[u] = cluster.map_shared_rank(S, row / LDC_ROWS)[(row % LDC_ROWS) * LDC_PITCH + c0 + (e & 31)];
                }
#pragma unroll
                for (int u = 0; u < 14; u++) {
                    const int e = e0 + u * LDLT_THREADS + tid;
                    if (e < LDC_ROWS * nc) T[(e & 31) * LDC_TP + (e >> 5)] = panel_mul(dk[e & 31], lc[u]);
                }
            }
            __syncthreads();
            // a column group at a time: the next sub-panel waits for the CTA with one group
            for (int g = 0; g < ng; g++) {
                const int col = cs + lane + 32 * g;
                float2 acc[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int i = wid * 4 + r;
                    acc[r] = (i < nr && col <= r0 + i) ? S[i * LDC_PITCH + col] : zero;
                }
#pragma unroll 8
                for (int k = 0; k < LDC_ROWS; k++) {
                    const float2 b = T[k * LDC_TP + lane + 32 * g];
#pragma unroll
                    for (int r = 0; r < 4; r++) acc[r] = panel_msub(acc[r], S[(wid * 4 + r) * LDC_PITCH + c0 + k], b);
                }
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int i = wid * 4 + r;
                    if (i < nr && col <= r0 + i) S[i * LDC_PITCH + col] = acc[r];
                }
            }
            __syncthreads();
        }
    }
    __syncthreads();
    for (int r = wid; r < nr; r += LDLT_THREADS / 32)
        for (int c = lane; c <= r0 + r; c += 32) A[(int64_t)(j0 + r0 + r) * lda + j0 + c] = S[r * LDC_PITCH + c];
    // no CTA leaves while another may still read its shared memory
    cluster.sync();
}

// Whether the cluster diagonal-block kernel can be resident on this device
// (8 CTAs with its shared memory; asked once per device and remembered).
static bool ldlt_cluster_fits(bem_ctx* ctx) {
    static std::mutex mu;
    static std::map<int, bool> ok;
    std::lock_guard<std::mutex> lk(mu);
    auto it = ok.find(ctx->device);
    if (it != ok.end()) return it->second;
    bool fits = cudaFuncSetAttribute(ldlt_diag_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)ldlt_cluster_smem_bytes()) == cudaSuccess;
    if (fits) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(LDC_CTAS);
        cfg.blockDim = dim3(LDLT_THREADS);
        cfg.dynamicSmemBytes = ldlt_cluster_smem_bytes();
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = LDC_CTAS;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int ncl = 0;
        fits = cudaOccupancyMaxActiveClusters(&ncl, (const void*)ldlt_diag_cluster_kernel, &cfg) == cudaSuccess &&
               ncl >= 1;
    }
    if (!fits) cudaGetLastError();
    ok[ctx->device] = fits;
    return fits;
}

static int launch_ldlt_diag_cluster(bem_ctx* ctx, float2* A, int64_t lda, int j0, int jb, int* d_info) {
    if (jb < 1 || jb > LDC_CTAS * LDC_ROWS) return fail(ctx, BEM_ERR_INVALID, "cluster diagonal block: jb out of range");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(LDC_CTAS);
    cfg.blockDim = dim3(LDLT_THREADS);
    cfg.dynamicSmemBytes = ldlt_cluster_smem_bytes();
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = LDC_CTAS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    BEM_TRY_CUDA(ctx, cudaLaunchKernelEx(&cfg, ldlt_diag_cluster_kernel, A, lda, j0, jb, d_info));
    BEM_LAUNCHED(ctx);
    return BEM_OK;
}

int sym_structure(bem_ctx* ctx, const double2* Z, int64_t ldz, int n, bool* sym, bool* sym_half) {
    unsigned* d_flags = nullptr;
    BEM_TRY_CUDA(ctx, cudaMalloc(&d_flags, sizeof(unsigned)));
    int s = BEM_OK;
    unsigned h = 3;
    do {
        if (cudaMemsetAsync(d_flags, 0, sizeof(unsigned), ctx->stream) != cudaSuccess) {
            s = fail(ctx, BEM_ERR_CUDA, "symmetry check");
            break;
        }
        const int64_t T = (n + 31) / 32, tiles = T * (T + 1) / 2;
        if (tiles > 0x7fffffff) {
            s = fail(ctx, BEM_ERR_INVALID, "symmetry check: n too large");
            break;
        }
        sym_check_kernel<<<(unsigned)tiles, 256, 0, ctx->stream>>>(Z, ldz, n, d_flags);
        ctx->launches++;
        if (cudaMemcpyAsync(&h, d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
            cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
            s = fail(ctx, BEM_ERR_CUDA, "symmetry check: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
    } while (0);
    cudaFree(d_flags);
    *sym = s == BEM_OK && !(h & 1u);
    *sym_half = s == BEM_OK && !(h & 2u);
    return s;
}

// W[c][r] (column-major, ld 256) = -1 on the diagonal, 0 elsewhere.
__global__ void neg_eye_kernel(float2* __restrict__ W, int jb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= jb * TRSM_KB) return;
    const int c = t / TRSM_KB, r = t % TRSM_KB;
    W[t] = make_float2(r == c ? -1.f : 0.f, 0.f);
}

// L[c * ldl + r] = W[c * 256 + r] d_r for c <= r < jb (W = -L11^-1 D^-1 of the
// diagonal block at j0, d_r its pivots): -L11^-1 itself.  The rest of L is zero already.
__global__ void linv_from_w_kernel(const float2* __restrict__ W, const float2* __restrict__ A, int64_t lda, int j0,
                                   int jb, float2* __restrict__ L, int ldl) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= TRSM_KB * TRSM_KB) return;
    const int c = t / TRSM_KB, r = t % TRSM_KB;
    if (c <= r && r < jb) {
        const float2 w = W[t], d = A[(int64_t)(j0 + r) * lda + j0 + r];
        const float2 v = make_float2(w.x * d.x - w.y * d.y, w.x * d.y + w.y * d.x);
        L[(size_t)c * ldl + r] = v;
    }
}

// Blocked right-looking L D L^T of the row-major complex64 S (lower triangle).
// Per 256-column block: the diagonal block is factored on one cluster of 8 CTAs
// (or, where that cannot be resident, in one CTA); its inverse factor W = L11^-T
// D^-1 comes from a block TRSM on -I; the panel below becomes L21 = S21 W in one
// tensor-core GEMM (in place: the operands are packed before the product is
// written); then the lower-triangle update.  With Linv the inverse blocks of
// linv_sb diagonal blocks are put together from W on the way.
int sytrf_nopiv(bem_ctx* ctx, float2* A, int64_t lda, int n, int* d_info, float2* Linv, int linv_sb) {
    using C2 = float2;
    const int NB = TRSM_KB;
    const size_t smem = ldlt_smem_bytes(sizeof(C2));
    static_assert(ldlt_smem_bytes(sizeof(float2)) <= 227 * 1024, "L D L^T diagonal block shared memory");
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(ldlt_diag_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
    // the diagonal blocks on one 8-CTA cluster where it fits, else on one CTA
    const bool diag_cluster = ctx->ldlt_cluster && ldlt_cluster_fits(ctx);
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(d_info, 0, sizeof(int), ctx->stream));
    BEM_TRY_CUDA(ctx, cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream));
    struct Buf {
        float2* p = nullptr;
        ~Buf() {
            if (p) cudaFree(p);
        }
    } W;
    const int SI = NB * linv_sb;  // rows of an inverse block
    BEM_TRY_CUDA(ctx, cudaMalloc(&W.p, (size_t)NB * (NB + SI) * sizeof(float2)));
    float2* T = W.p + (size_t)NB * NB;  // 256 x SI, column-major
    if (Linv) BEM_TRY_CUDA(ctx, cudaMemsetAsync(Linv, 0, linv_count(n, linv_sb) * sizeof(float2), ctx->stream));
    // the diagonal block at j0 and its panel below: L D L^T of the block,
    // then L21 = S21 L11^-T D^-1 for the rows [j0 + jb, n)
    auto factor_block = [&](int j0, int jb) -> int {
        const int below = n - j0 - jb;
        cudaEvent_t ev = ctx->prof_begin(PROF_PANEL);
        if (diag_cluster) {
            BEM_TRY(launch_ldlt_diag_cluster(ctx, A, lda, j0, jb, d_info));
        } else {
            ldlt_diag_kernel<float><<<1, LDLT_THREADS, smem, ctx->stream>>>(A, lda, j0, jb, d_info);
            BEM_LAUNCHED(ctx);
        }
        if (ev) ctx->prof_end(PROF_PANEL, ev, 8.0 * jb * (double)jb * jb / 3, 16.0 * (double)jb * jb);
        if (below > 0 || Linv) {
            // column c of W.p solves L11 x = -e_c, then x_r /= d_r:
            // W.p[c * 256 + r] = -L11^-1[r][c] / d_r
            neg_eye_kernel<<<(jb * NB + 255) / 256, 256, 0, ctx->stream>>>(W.p, jb);
            BEM_LAUNCHED(ctx);
            BEM_TRY((trsm_block<float, false, false, TRSM_DIVDIAG>(ctx, A, lda, j0, jb, W.p, NB, 0, jb, 0)));
        }
        if (Linv) {
            // into its place in the SI x SI inverse block at I0, then the rows left of it:
            // -[[A, 0], [C, B]]^-1 = [[Ma, 0], [Mb C Ma, Mb]] with Ma = -A^-1, Mb = -B^-1
            const int I0 = j0 / SI * SI, k = j0 - I0;
            float2* Mi = Linv + (size_t)(I0 / SI) * SI * SI;
            float2* Mb = Mi + (size_t)k * SI + k;
            linv_from_w_kernel<<<NB * NB / 256, 256, 0, ctx->stream>>>(W.p, A, lda, j0, jb, Mb, SI);
            BEM_LAUNCHED(ctx);
            if (k > 0) {
                TcOpts o;
                o.c_colmajor = true;
                o.store = true;
                o.prof_cls = PROF_PANEL_UPDATE;
                BEM_TRY(tc_gemm_ex(ctx, jb, k, k, A + (int64_t)j0 * lda + I0, lda, Mi, SI, T, NB, o));  // T = -C Ma
                o.a_trans = true;
                BEM_TRY(tc_gemm_ex(ctx, jb, k, jb, Mb, SI, T, NB, Mi + k, SI, o));                      // -Mb T
            }
        }
        if (below > 0) {
            // L21 = S21 L11^-T D^-1: B given row-major (K x N) is
            // B[k][j] = W.p[k * 256 + j] = -(L11^-T D^-1)[k][j]; the store mode writes C = -A B
            TcOpts o;
            o.b_rowmajor = true;
            o.store = true;
            o.prof_cls = PROF_PANEL_UPDATE;
            float2* S21 = A + (int64_t)(j0 + jb) * lda + j0;
            BEM_TRY(tc_gemm_ex(ctx, below, jb, jb, S21, lda, W.p, NB, S21, lda, o));
        }
        return (int)BEM_OK;
    };
    // Super-blocks of factor_sb 256-column blocks: each block is factored and
    // updates the super-block's later block columns alone (thin GEMMs), and
    // the lower-triangle update of the rest takes the whole super-block
    // (K = 256 factor_sb: fewer launches and fewer read-modify-writes of the
    // trailing matrix).
    const int SB = std::max(1, std::min(4, ctx->factor_sb)) * NB;
    for (int J0 = 0; J0 < n; J0 += SB) {
        const int JB = std::min(SB, n - J0);
        for (int j = J0; j < J0 + JB; j += NB) {
            const int jb = std::min(NB, J0 + JB - j);
            BEM_TRY(factor_block(j, jb));
            const int nc = J0 + JB - j - jb;  // the super-block's columns after this block
            if (nc > 0) {
                // S[j+jb:, j+jb:J0+JB] -= L21 D L21^T (rows j+jb.. of this block's L21)
                TcOpts o;
                o.bscale = A + (int64_t)j * lda + j;
                o.bscale_stride = lda + 1;
                o.prof_cls = PROF_LU_UPDATE;
                const float2* L21 = A + (int64_t)(j + jb) * lda + j;
                BEM_TRY(tc_gemm_ex(ctx, n - j - jb, nc, jb, L21, lda, L21, lda, A + (int64_t)(j + jb) * lda + j + jb,
                                   lda, o));
            }
        }
        const int below = n - J0 - JB;
        if (below > 0) {
            // S22 -= L21 D L21^T over the super-block, lower triangle
            TcOpts o;
            o.lower = true;
            o.bscale = A + (int64_t)J0 * lda + J0;
            o.bscale_stride = lda + 1;
            o.prof_cls = PROF_LU_UPDATE;
            const float2* L21 = A + (int64_t)(J0 + JB) * lda + J0;
            BEM_TRY(tc_gemm_ex(ctx, below, below, JB, L21, lda, L21, lda, A + (int64_t)(J0 + JB) * lda + J0 + JB, lda,
                               o));
        }
    }
    return BEM_OK;
}

// X[i][c] /= D_i
__global__ void diag_div_kernel(const float2* __restrict__ A, int64_t lda, float2* __restrict__ X, int64_t ldx, int n,
                                int nrhs) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * nrhs) return;
    const int r = (int)(t % n), c = (int)(t / n);
    X[(int64_t)c * ldx + r] = cdiv(X[(int64_t)c * ldx + r], A[(int64_t)r * lda + r]);
}

// X = S^-1 B with S = L D L^T (B, X column-major complex64; X may alias B).
int sytrs_nopiv(bem_ctx* ctx, const float2* A, int64_t lda, int n, const float2* B, int64_t ldb, float2* X,
                int64_t ldx, int nrhs, const float2* Linv, int linv_sb) {
    const int NB = TRSM_KB;
    if (nrhs <= 0) return BEM_OK;
    int64_t tot = (int64_t)n * nrhs;
    if (B != X || ldb != ldx) {
        permute_rows_kernel<float><<<(unsigned)((tot + 255) / 256), 256, 0, ctx->stream>>>(B, ldb, X, ldx, nullptr, n,
                                                                                         nrhs);
        BEM_LAUNCHED(ctx);
    }
    // Super-blocks of solve_sb 256-row diagonal blocks: the blocks of a
    // super-block update one another with thin GEMMs, so the update of all
    // rows beyond runs with K = 256 solve_sb (fewer launches and fewer
    // read-modify-writes of X).  With the inverses of whole super-blocks a
    // super-block's own part is one product of M = K = 1024 over its
    // non-zero blocks: 20 ms -> 10 ms of a 161 ms solve (2N = 15360, 2790
    // columns) against products with 256-row inverses and K = 256 updates
    // between them, whose 22 tiles left two thirds of the SMs idle.
    const int SB = Linv ? linv_sb * NB : std::max(1, std::min(4, ctx->solve_sb)) * NB;
    const int DB = Linv ? SB : NB;  // rows of a diagonal block
    auto update = [&](int M, int K, const float2* Ablk, bool trans, float2* Bx, float2* Cx) {
        TcOpts o;
        o.c_colmajor = true;
        o.a_trans = trans;
        o.prof_cls = PROF_SOLVE_UPDATE;
        return tc_gemm_ex(ctx, M, nrhs, K, Ablk, lda, Bx, ldx, Cx, ldx, o);
    };
    // the diagonal block at J0 (jb rows): X_blk = L11^-1 X_blk (back: L11^-T),
    // as -(-L11^-1) X_blk (in place: the product packs X_blk before it writes), or a block triangular solve
    auto diag = [&](int J0, int jb, bool back) -> int {
        if (!Linv) {
            if (back)
                return trsm_block<float, true, false, TRSM_TRANS | TRSM_UNIT>(ctx, A, lda, J0, jb, X, ldx, 0, nrhs);
            return trsm_block<float, false, false>(ctx, A, lda, J0, jb, X, ldx, 0, nrhs);
        }
        TcOpts o;
        o.c_colmajor = true;
        o.store = true;
        o.a_trans = !back;  // forward: A[r][c] = Li[c * SB + r]; back: A[r][c] = Li[r * SB + c]
        o.a_tri = back ? 2 : 1;
        o.prof_cls = PROF_TRSM;
        const float2* Li = Linv + (size_t)(J0 / SB) * SB * SB;
        return tc_gemm_ex(ctx, jb, nrhs, jb, Li, SB, X + J0, ldx, X + J0, ldx, o);
    };
    // L z = b
    for (int J0 = 0; J0 < n; J0 += SB) {
        const int JB = std::min(SB, n - J0);
        for (int j = J0; j < J0 + JB; j += DB) {
            const int jb = std::min(DB, J0 + JB - j), nc = J0 + JB - j - jb;
            BEM_TRY(diag(j, jb, false));
            // the super-block's later rows: X[j+jb:J0+JB] -= L[j+jb:J0+JB, j:j+jb] X[j:j+jb]
            if (nc > 0) BEM_TRY(update(nc, jb, A + (int64_t)(j + jb) * lda + j, false, X + j, X + j + jb));
        }
        const int below = n - J0 - JB;
        if (below > 0) BEM_TRY(update(below, JB, A + (int64_t)(J0 + JB) * lda + J0, false, X + J0, X + J0 + JB));
    }
    // y = D^-1 z
    diag_div_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, ctx->stream>>>(A, lda, X, ldx, n, nrhs);
    BEM_LAUNCHED(ctx);
    // L^T x = y, super-blocks from the last
    const int nsb = (n + SB - 1) / SB;
    for (int bi = nsb - 1; bi >= 0; bi--) {
        const int J0 = bi * SB, JB = std::min(SB, n - J0);
        for (int j = J0 + ((JB - 1) / DB) * DB; j >= J0; j -= DB) {
            const int jb = std::min(DB, J0 + JB - j);
            BEM_TRY(diag(j, jb, true));
            // the super-block's earlier rows: X[J0:j] -= (L[j:j+jb, J0:j])^T X[j:j+jb]
            if (j > J0) BEM_TRY(update(j - J0, jb, A + (int64_t)j * lda + J0, true, X + j, X + J0));
        }
        // X[0:J0] -= (L[J0:J0+JB, 0:J0])^T X[J0:J0+JB]
        if (J0 > 0) BEM_TRY(update(J0, JB, A + (int64_t)J0 * lda, true, X + J0, X));
    }
    return BEM_OK;
}

// Row pivots (LAPACK interchange sequence, 0-based) -> gather permutation.
void pivots_to_perm(const std::vector<int>& ipiv, std::vector<int>& perm) {
    int n = (int)ipiv.size();
    perm.resize(n);
    for (int i = 0; i < n; i++) perm[i] = i;
    for (int k = 0; k < n; k++) std::swap(perm[k], perm[ipiv[k]]);
}

}  // namespace bem
