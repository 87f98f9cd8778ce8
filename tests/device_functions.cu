// Device functions by themselves, for test_gpu_device_functions.py: one thread an argument.
#include "../include/kerrsplat_b200.h"
#include "ks_gradient.cuh"

using namespace ks;

static __device__ MomentCoeffs d_moments;

static __global__ void k_sincos(long long n, const double* x, double* s, double* c) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) fsincos(x[i], s[i], c[i]);
}

// method 0: FP32 as the reverse pass takes it; 1: the seven FP64 duals through the step operator
static __global__ void k_step_adjoint(long long n, const double* in, const double* Dl, const double* w, const double* R, int method, double* cb) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (method == 0) {
        float fi[11], fw[4], fR[4], O[16], E[4], out[11];
        for (int q = 0; q < 11; ++q) fi[q] = float(in[11 * i + q]);
        for (int q = 0; q < 4; ++q) { fw[q] = float(w[4 * i + q]); fR[q] = float(R[4 * i + q]); }
        sample_adjoint_structured(d_moments, fi, float(Dl[i]), fw, fR, O, E, out);
        for (int q = 0; q < 11; ++q) cb[11 * i + q] = out[q];
    } else {
        double O[16], E[4];
        sample_adjoint(d_moments, in + 11 * i, Dl[i], w + 4 * i, R + 4 * i, O, E, cb + 11 * i);
    }
}

template <class F>
static int on_device(long long n, int nin, const double* const* in, const int* width, double* out, int wout, F launch) {
    double *d[5] = {}, *o = nullptr;
    cudaError_t e = cudaMalloc(&o, n * wout * sizeof(double));
    for (int q = 0; q < nin && e == cudaSuccess; ++q) {
        e = cudaMalloc(&d[q], n * width[q] * sizeof(double));
        if (e == cudaSuccess) e = cudaMemcpy(d[q], in[q], n * width[q] * sizeof(double), cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) {
        launch(d, o);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, o, n * wout * sizeof(double), cudaMemcpyDeviceToHost);
    for (double* p : d) cudaFree(p);
    cudaFree(o);
    return int(e);
}

extern "C" int probe_sincos(long long n, const double* x, double* out) {
    const int width[1] = {1};
    return on_device(n, 1, &x, width, out, 2, [&](double** d, double* o) { k_sincos<<<unsigned((n + 127) / 128), 128>>>(n, d[0], o, o + n); });
}

extern "C" int probe_step_adjoint(long long n, const double* in, const double* Dl, const double* w, const double* R, int method, double* cb) {
    MomentCoeffs mc;   // M_n(a) = sum_m (-a)^m / (m! (n + m + 1))
    for (int k = 0; k < 11; ++k) {
        double f = 1.0;
        for (int m = 0; m < 24; ++m) {
            if (m > 0) f *= m;
            mc.c[k][m] = ((m % 2) ? -1.0 : 1.0) / (f * (k + m + 1));
            mc.cf[k][m] = float(mc.c[k][m]);
        }
    }
    if (cudaMemcpyToSymbol(d_moments, &mc, sizeof mc) != cudaSuccess) return -1;
    const double* a[4] = {in, Dl, w, R};
    const int width[4] = {11, 1, 4, 4};
    return on_device(n, 4, a, width, cb, 11,
                     [&](double** d, double* o) { k_step_adjoint<<<unsigned((n + 63) / 64), 64>>>(n, d[0], d[1], d[2], d[3], method, o); });
}
