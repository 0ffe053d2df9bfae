// sqrt_newton and rcp_newton over every exponent, both signs of the reciprocal's argument, and the special
// values: counts the results outside the bounds that sph_common.cuh states.  A NaN fails every bound.
// Prints "sqrt <n> rcp <n> special <n>".
#include <cstdio>
#include <cmath>
#include "sph_common.cuh"

__device__ __forceinline__ double ulp_of(double v) {
    const float f = (float)v;
    return (double)(nextafterf(f, 3.4e38f) - f);
}
__global__ void k_check(unsigned int* bad) {
    unsigned int s = 0, r = 0;
    for (int e = (int)blockIdx.x; e < 255; e += gridDim.x)
        for (unsigned int m = threadIdx.x * 61; m < (1u << 23) + 61; m += blockDim.x * 61) {
            const float x = __uint_as_float(((unsigned int)e << 23) | (m < (1u << 23) ? m : (1u << 23) - 1));
            if (x == 0.f) continue;
            const double root = sqrt((double)x), inv = 1.0 / (double)x;
            const double y = (double)wsph::sqrt_newton(x);
            if (x >= 7.8886091e-31f) s += !(fabs(y - root) <= ulp_of(root));                    // 2^-100
            else if (e > 0) s += !(fabs(y - root) <= 2.0 * ulp_of(root));
            else s += !(y >= 0.0 && y <= root * 1.00001);
            #pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double sg = q ? -1.0 : 1.0, z = sg * (double)wsph::rcp_newton(q ? -x : x);
                if (e == 0) r += !(z == INFINITY);
                else if ((double)x <= 8.5070591730234616e37) r += !(fabs(z - inv) <= ulp_of(inv));     // 2^126
                else r += !(fabs(z - inv) <= 1.1754943508222875e-38);
            }
        }
    atomicAdd(bad, s);
    atomicAdd(bad + 1, r);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const float inf = INFINITY, nan = __int_as_float(0x7fc00000), z = wsph::rcp_newton(-inf);
        bad[2] = !(wsph::sqrt_newton(0.f) == 0.f) + (wsph::sqrt_newton(inf) < inf) + !isnan(wsph::sqrt_newton(nan)) + !(wsph::rcp_newton(0.f) == inf) +
                 !(wsph::rcp_newton(-0.f) == -inf) + !(wsph::rcp_newton(inf) == 0.f) + !(z == 0.f && signbit(z)) + !isnan(wsph::rcp_newton(nan));
    }
}

int main() {
    unsigned int *d, h[3];
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
    k_check<<<255, 256>>>(d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("sqrt %u rcp %u special %u\n", h[0], h[1], h[2]);
    return 0;
}
