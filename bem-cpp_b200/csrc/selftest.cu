// Entry points that the tests use to see parts of the library on their own.
//
// The failure path of a bounded device-side wait, exercised without a fault.
//
// Every wait in this library's kernels (the tensor-core pipelines' mbarriers,
// the int8 residual's pacing) gives up after a fixed number of SM clock
// cycles, records BEM_ERR_TIMEOUT in a status word and returns, so a stuck
// producer surfaces as an error status while the context stays usable.  This
// entry point runs that pattern alone: one thread waits on a device flag for
// at most `cycles` clock cycles.  With the flag left at 0 nothing ever sets it
// and the wait runs out; with the flag set the wait ends at once.
#include <cuda_runtime.h>

#include <cstdint>

#include "bem_internal.h"
#include "math_device.cuh"

namespace bem {
namespace {

// own[i], ref[i] (two values a point for fn 0 and 3): the branch-free function
// of math_device.cuh and CUDA's at x[i] (fn 3: x[2i] + i x[2i + 1], by divisions).
__global__ void math_kernel(int fn, const double* __restrict__ x, int n, double* __restrict__ own,
                            double* __restrict__ ref) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (fn == 0) {
        sincos_bounded(x[i], &own[2 * i], &own[2 * i + 1]);
        sincos(x[i], &ref[2 * i], &ref[2 * i + 1]);
    } else if (fn == 1) {
        own[i] = exp_decay_bounded(x[i]);
        ref[i] = exp(-x[i]);
    } else if (fn == 2) {
        own[i] = rsqrt_normal(x[i]);
        ref[i] = rsqrt(x[i]);
    } else {
        const double2 p = make_double2(x[2 * i], x[2 * i + 1]), r = pivot_recip(p);
        const double den = p.x * p.x + p.y * p.y;
        own[2 * i] = r.x, own[2 * i + 1] = r.y;
        ref[2 * i] = p.x / den, ref[2 * i + 1] = -p.y / den;
    }
}

__global__ void bounded_wait_kernel(const volatile int* flag, long long cycles, int* status) {
    const long long t0 = clock64();
    while (*flag == 0) {
        if (clock64() - t0 > cycles) {
            *status = (int)BEM_ERR_TIMEOUT;
            return;
        }
    }
    *status = (int)BEM_OK;
}

}  // namespace
}  // namespace bem

extern "C" int bem_selftest_math(bem_ctx* ctx, int fn, const double* x, int n, double* own, double* ref) {
    if (!ctx || !x || !own || !ref || n < 1 || n > (1 << 26) || fn < 0 || fn > 3) return BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t in = (size_t)n * (fn == 3 ? 2 : 1), out = (size_t)n * (fn == 0 || fn == 3 ? 2 : 1);
    double* d = nullptr;
    BEM_TRY_CUDA(ctx, cudaMalloc(&d, (in + 2 * out) * sizeof(double)));
    cudaError_t e = cudaMemcpyAsync(d, x, in * sizeof(double), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        bem::math_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(fn, d, n, d + in, d + in + out);
        ctx->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(own, d + in, out * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ref, d + in + out, out * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d);
    return e == cudaSuccess ? BEM_OK : bem::fail(ctx, BEM_ERR_CUDA, "elementary functions: %s", cudaGetErrorString(e));
}

extern "C" int bem_selftest_bounded_wait(bem_ctx* ctx, int64_t cycles, int set_flag) {
    if (!ctx || cycles < 0 || cycles > 4000000000LL) return BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    int* d = nullptr;
    BEM_TRY_CUDA(ctx, cudaMalloc(&d, 2 * sizeof(int)));
    const int h[2] = {set_flag ? 1 : 0, -1};  // flag, status
    int st = -1;
    cudaError_t e = cudaMemcpyAsync(d, h, sizeof(h), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        bem::bounded_wait_kernel<<<1, 1, 0, ctx->stream>>>(d, (long long)cycles, d + 1);
        ctx->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&st, d + 1, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d);
    if (e != cudaSuccess) return bem::fail(ctx, BEM_ERR_CUDA, "bounded wait: %s", cudaGetErrorString(e));
    if (st == BEM_ERR_TIMEOUT)
        return bem::fail(ctx, BEM_ERR_TIMEOUT, "bounded wait ran out after %lld clock cycles", (long long)cycles);
    if (st != BEM_OK) return bem::fail(ctx, BEM_ERR_CUDA, "bounded wait: status %d", st);
    return BEM_OK;
}
