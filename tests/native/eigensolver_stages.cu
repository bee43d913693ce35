// The FP64 path's eigensolver stages on matrices of a test's choosing, in the order given (the library
// runs them on interpolated Hamiltonians only): stage 1 as chains of warm-started points, stage 2 from
// stage 1's vectors or from the caller's.  Host arrays, column-major matrices of np = nw rounded up to
// even (vectors of stage 1) or nw (the rest).
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "eigh.cuh"
#include "onesided.cuh"

namespace {

template <typename T> struct Buffer {
    T *p = nullptr;
    explicit Buffer(size_t n) { if (cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) p = nullptr; }
    ~Buffer() { cudaFree(p); }
};

cudaError_t allow(const void *fn) {
    int optin = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, fn);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes);
}

cudaError_t stage1(const double2 *h, int64_t n, int nw, int64_t chains, int warm, float2 *v) {
    const int np = nw + (nw & 1);
    int64_t stride = (int64_t)nw * nw;
    cudaError_t e;
    if (nw <= 32) {
        const RegKernel rk = onesided_kernel(np);
        if ((e = allow(rk.fn)) != cudaSuccess) return e;
        void *args[] = {&h, &stride, &n, &nw, &v, &chains, &warm};
        return cudaLaunchKernel(rk.fn, dim3((unsigned)((chains + 3) / 4)), dim3(128), args, 4 * rk.group_smem, 0);
    }
    const void *fn = onesided_cta_fn(np);
    if ((e = allow(fn)) != cudaSuccess) return e;
    void *args[] = {&h, &stride, &n, &nw, &v, &warm};
    return cudaLaunchKernel(fn, dim3((unsigned)chains), dim3(OsCtaSmem::threads(np)), args, OsCtaSmem::bytes(np), 0);
}

cudaError_t stage2(const double2 *h, int64_t n, int nw, const float2 *v, double *E, double2 *U) {
    const int np = nw + (nw & 1);
    int64_t stride = (int64_t)nw * nw;
    int converge = 1;
    if (nw <= 32) {
        unsigned char off[120][2] = {};
        for (int k2 = 1, w = 0; k2 < np / 2; ++k2)
            for (int k1 = 0; k1 < k2; ++k1, ++w) { off[w][0] = (unsigned char)k1; off[w][1] = (unsigned char)k2; }
        cudaError_t e = cudaMemcpyToSymbol(c_jacobi_offdiag, off, sizeof(off));
        const void *fn = (const void *)eigh_refine_f64_team_kernel<128>;
        if (e == cudaSuccess) e = allow(fn);
        if (e != cudaSuccess) return e;
        void *args[] = {&h, &stride, &v, &n, &nw, &E, &U, &converge};
        return cudaLaunchKernel(fn, dim3((unsigned)n), dim3(128), args, WarpRefineSmem::per_team(nw), 0);
    }
    const size_t bytes = (RefineCtaSmem::bytes(nw) + 255) & ~(size_t)255;
    Buffer<unsigned char> scratch(bytes * (size_t)n);
    if (!scratch.p) return cudaErrorMemoryAllocation;
    eigh_refine_f64_cta_kernel<true><<<(unsigned)n, 512>>>(h, stride, v, n, nw, E, U, converge, scratch.p, (int64_t)bytes);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : cudaDeviceSynchronize();
}

}  // namespace

// V: stage 1's vectors out, or stage 2's in when start = 1.  E, U: stage 2's results.  Returns the CUDA error code.
extern "C" __attribute__((visibility("default"))) int eigensolver_stages(const double *H, int64_t n, int nw, int64_t chains,
                                                                         int warm, int start, float *V, double *E, double *U) {
    if (n < 1 || nw < 17 || nw > 128 || chains < 1 || chains > n) return (int)cudaErrorInvalidValue;
    const int np = nw + (nw & 1);
    const size_t nn = (size_t)nw * nw, mm = (size_t)np * np;
    Buffer<double2> h(n * nn), u(n * nn);
    Buffer<float2> v(n * mm);
    Buffer<double> en((size_t)n * nw);
    if (!h.p || !u.p || !v.p || !en.p) return (int)cudaErrorMemoryAllocation;
    cudaError_t e = cudaMemcpy(h.p, H, n * nn * sizeof(double2), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && start) e = cudaMemcpy(v.p, V, n * mm * sizeof(float2), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !start) e = stage1(h.p, n, nw, chains, warm, v.p);
    if (e == cudaSuccess) e = stage2(h.p, n, nw, v.p, en.p, u.p);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess && !start) e = cudaMemcpy(V, v.p, n * mm * sizeof(float2), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(E, en.p, (size_t)n * nw * sizeof(double), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(U, u.p, n * nn * sizeof(double2), cudaMemcpyDeviceToHost);
    return (int)e;
}
