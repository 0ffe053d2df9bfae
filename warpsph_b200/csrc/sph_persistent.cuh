// Bounded grid-wide barrier for cooperative persistent kernels (the DFSPH Jacobi solves
// and the batched delta-SPH step).  The launch must be cooperative (every block
// co-resident).  A wait gives up after limit_ns nanoseconds of the global timer (2 s by
// default; the Jacobi solves take the limit from their launch arguments) or 2^26 polls,
// sets SPH_STATUS_TIMEOUT in the control block and makes every block return, so a
// failure ends the kernel instead of hanging the GPU.
//
// The arrival counter only ever grows: block b's k-th wait ends when it has reached
// k * gridDim.x, so no block resets it and no second word is published (at most
// 2^21 waits x 2^11 blocks in a solve, compared modulo 2^32).  One thread arrives with a
// release and polls with an acquire; the block barriers on both sides extend that order to
// the whole block, so plain loads after the barrier see every write made before it.
#pragma once
#include <cuda_runtime.h>
#include "sph_common.cuh"

namespace wsph {

struct BarrierCtl {
    unsigned int count;        // arrivals since the control block was zeroed
    unsigned int pad0;
    int status;                // SPH_STATUS_* bits
    int pad;
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr unsigned long long kBarrierLimitNs = 2000000000ull;

static __device__ __noinline__ bool grid_wait(BarrierCtl* c, unsigned int arrived, unsigned long long limit_ns) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->count) : "memory");
        const unsigned long long t0 = global_ns();
        unsigned int spins = 0, now;
        int good = 1;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(&c->count) : "memory");
            if (static_cast<int>(now - arrived) >= 0) break;
            if (*reinterpret_cast<volatile int*>(&c->status) & SPH_STATUS_TIMEOUT) { good = 0; break; }
            if (++spins > (1u << 26) || global_ns() - t0 > limit_ns) {
                atomicOr(&c->status, SPH_STATUS_TIMEOUT);
                good = 0;
                break;
            }
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}
// `arrived` counts the arrivals this block waits for; it starts at 0 with the zeroed control
// block and is the same in every thread.  Returns false when any block gave up
// (SPH_STATUS_TIMEOUT); the caller then returns.
__device__ __forceinline__ bool grid_barrier(BarrierCtl* c, unsigned int& arrived, unsigned long long limit_ns = kBarrierLimitNs) {
    arrived += gridDim.x;
    return grid_wait(c, arrived, limit_ns);
}

// Blocks of a persistent launch over n particles with ppb of them per block and round: what n needs, at most
// the co-resident blocks and `limit` (slots of per-block results).  With one_round, for a kernel whose groups keep
// one particle each for the whole launch, 0 when that many blocks cannot hold the particles in one round.
constexpr int persistent_grid(int64_t n, int ppb, int64_t resident, int64_t limit, bool one_round) {
    const int64_t need = (n + ppb - 1) / ppb, cap = resident < limit ? resident : limit;
    if (one_round && need > cap) return 0;
    return (int)(need < cap ? need : cap);
}

}  // namespace wsph
