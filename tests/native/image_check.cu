// pair_vec against dist_vec, bit for bit: differences within 64 floats of L / 2 on both sides, and pseudo-random
// ones up to 1.5 L, for a range of box lengths; and an open axis.  The library's own parameter packing fills
// the domain.  Prints "differ <n> of <n>".
#include <cstdio>
#include <cmath>
#include "sph_common.cuh"

namespace wsph { int params_to_dev(const SphParams* p, DevParams* o); }

__device__ __forceinline__ unsigned int mix(unsigned int h) {
    h ^= h >> 16; h *= 0x7feb352du; h ^= h >> 15; h *= 0x846ca68bu; return h ^ (h >> 16);
}
__global__ void k_check(wsph::DomainF dom, int open, unsigned int* out) {
    const unsigned int t = blockIdx.x * blockDim.x + threadIdx.x;
    const float h = dom.L[0] * 0.5f;
    float d = t < 129 ? __int_as_float(__float_as_int(h) + (int)t - 64) : dom.L[0] * 1.5f * ((float)(mix(t) >> 8) / 16777216.f);
    if (open && t == 200) d = INFINITY;
    unsigned int bad = 0;
    for (int q = 0; q < 2; ++q) {
        const wsph::Vec<1> a{{q ? -d : d}}, z{{0.f}};
        bad += __float_as_uint(wsph::pair_vec<1>(a, z, dom).v[0]) != __float_as_uint(wsph::dist_vec<1>(a, z, dom).v[0]);
    }
    atomicAdd(out, bad);
    atomicAdd(out + 1, 2u);
}

int main() {
    unsigned int *d, h[2];
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
    const double lengths[] = {1.0, 2.0, 3.0, 0.37, 1.2, 7.0, 10.0, 1e-3, 1.9999999, 4.7e4, 6.02e23, 1.6e-19, 0.1, 1.0 / 3.0, 255.0, 2e-30};
    for (double L : lengths)
        for (int periodic = 0; periodic < 2; ++periodic) {
            SphParams p{};
            wsph::DevParams P;
            p.dim = 1; p.kernel = SPH_KERNEL_WENDLAND2; p.verlet_scale = 1.0;
            for (int a = 0; a < 3; ++a) { p.domain_min[a] = -L / 2; p.domain_max[a] = L / 2; p.periodic[a] = periodic; }
            if (wsph::params_to_dev(&p, &P)) return 2;
            k_check<<<64, 256>>>(P.dom, !periodic, d);
        }
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("differ %u of %u\n", h[0], h[1]);
    return 0;
}
