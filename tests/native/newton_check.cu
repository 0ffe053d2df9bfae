// Largest errors of sqrt_newton and rcp_newton, in units of the last place of the 64-bit result
// rounded to 32 bits, over every mantissa step of 2^7 and the exponents that squared distances,
// supports and densities take; and sqrt_newton(0).  Prints "sqrt <ulp> rcp <ulp> zero <value>".
#include <cstdio>
#include <cmath>
#include "sph_common.cuh"

__global__ void k_check(double* worst) {
    const unsigned int step = 128;
    double ws = 0.0, wr = 0.0;
    for (int e = 127 - 96 + (int)blockIdx.x; e <= 127 + 96; e += gridDim.x)
        for (unsigned int m = threadIdx.x * step; m < (1u << 23); m += blockDim.x * step) {
            const float x = __uint_as_float(((unsigned int)e << 23) | m);
            const double s = sqrt((double)x), r = 1.0 / (double)x;
            const double us = (double)(nextafterf((float)s, 3e38f) - (float)s), ur = (double)(nextafterf((float)r, 3e38f) - (float)r);
            ws = fmax(ws, fabs((double)wsph::sqrt_newton(x) - s) / us);
            wr = fmax(wr, fabs((double)wsph::rcp_newton(x) - r) / ur);
        }
    // positive doubles order as their bit patterns
    atomicMax(reinterpret_cast<unsigned long long*>(worst), (unsigned long long)__double_as_longlong(ws));
    atomicMax(reinterpret_cast<unsigned long long*>(worst + 1), (unsigned long long)__double_as_longlong(wr));
    if (blockIdx.x == 0 && threadIdx.x == 0) worst[2] = wsph::sqrt_newton(0.f);
}

int main() {
    double* d;
    double h[3];
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
    k_check<<<193, 256>>>(d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("sqrt %.4f rcp %.4f zero %g\n", h[0], h[1], h[2]);
    return 0;
}
