// div_markstein and rcp_markstein against the rounded quotients: the reciprocal over every significand
// and several exponents, the quotient over pseudo-random operands, with the precomputed (rounded)
// reciprocal and with rcp_markstein's.  Prints the numbers of results that differ:
// "rcp <n> div <n> div2 <n>"; a significand of all ones may be one of them in rcp.
#include <cstdio>
#include "sph_common.cuh"

__device__ __forceinline__ unsigned int mix(unsigned int h) {
    h ^= h >> 16; h *= 0x7feb352du; h ^= h >> 15; h *= 0x846ca68bu; return h ^ (h >> 16);
}
__global__ void k_check(unsigned long long* bad) {
    const unsigned int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    unsigned long long r = 0, d = 0, d2 = 0;
    for (int e = 127 - 60; e <= 127 + 60; e += 15)
        for (unsigned int m = t; m < (1u << 23); m += nt) {
            const float b = __uint_as_float(((unsigned int)e << 23) | m), y = __fdiv_rn(1.f, b);
            if (m != (1u << 23) - 1) r += wsph::rcp_markstein(b) != y;
            const unsigned int u = mix(m * 9u + (unsigned int)e);
            const float a = __uint_as_float((((u >> 23) % 60u + 97u) << 23) | (u & 0x7fffffu)) * ((u & 1u) ? 1.f : -1.f), q = __fdiv_rn(a, b);
            d += wsph::div_markstein(a, b, y) != q;
            d2 += wsph::div_markstein(a, b, wsph::rcp_markstein(b)) != q;
        }
    atomicAdd(bad, r); atomicAdd(bad + 1, d); atomicAdd(bad + 2, d2);
}

int main() {
    unsigned long long *dev, h[3];
    if (cudaMalloc(&dev, sizeof(h)) != cudaSuccess || cudaMemset(dev, 0, sizeof(h)) != cudaSuccess) return 1;
    k_check<<<1184, 256>>>(dev);
    if (cudaMemcpy(h, dev, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("rcp %llu div %llu div2 %llu\n", h[0], h[1], h[2]);
    return 0;
}
