// Incompressible (DFSPH) pressure solves of the warpSPH hot path.
//
//   sph_dfsph_alpha                modules/incompressible/wp_alpha.py:35-118, :294-313
//   sph_incompressible_divergence  modules/momentum/incompressible.py:9-34
//   sph_pressure_accel_iisph       modules/pressure/iisph.py:7-24
//   sph_pressure_shift_iisph       modules/incompressible/drift.py:38-57
//   sph_dfsph_div_solve            modules/incompressible/divergenceFree.py:23-139
//   sph_dfsph_density_solve        modules/incompressible/incompressible.py:21-143
//
// The reference runs each Jacobi iteration as two Warp launches plus torch
// reductions and reads the residual back to the host every iteration.  Here a
// whole solve is one cooperative persistent kernel: every iteration is
//   phase A  a_i = -sum_j m_j (p_i/rho_i^2 + p_j/rho_j^2) gradW_ij   (pressure gauge
//            of the previous iteration applied on the fly), writes p_i and a_i
//   barrier
//   phase B  s_i = -sum_j V_j (a_j - a_i).gradW_ij, r_i = src_i - dt_f s_i,
//            p_i += omega r_i / diag_i, block partial sums of p and of the error
//            term folded into FP64 accumulators
//   barrier
//   decide   every block reads the same sums, so all take the same branch
// with a final phase A for the returned acceleration.  The grid barrier is a
// counter + generation pair in the caller's workspace; its waits are bounded
// (SPH_STATUS_TIMEOUT after ~2 s) so a failure returns instead of hanging.
//
// Data written in one phase and read by other blocks in the next (p, a) is
// loaded with ld.global.cg (L2), never through the non-coherent L1.
#include <cuda_runtime.h>
#include <mutex>
#include "sph_pair_common.cuh"
#include "sph_persistent.cuh"

namespace wsph {

constexpr int JAC_BLOCK = 256;
constexpr int JAC_G = 8;
constexpr int JAC_PPB = JAC_BLOCK / JAC_G;   // particles per block and round

struct JacobiCtl {
    BarrierCtl bar;            // grid barrier and SPH_STATUS_* bits
    double sum[3][2];          // [slot][0] = sum p, [slot][1] = sum of the error term
    unsigned int mm[3][2];     // [slot][0] = min p, [slot][1] = max p (ordered encoding)
};

__device__ __forceinline__ unsigned int f2o(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(unsigned int o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// ---------------------------------------------------------------- per-lane partial sums
// Pressure acceleration, modules/pressure/iisph.py:7-24 with the symmetric gradient
// rho_i sum_j m_j (q_i/rho_i^2 + q_j/rho_j^2) gradW(x_ij, H_j).  p_j = praw_j - mu.
template <int KF, int D, int G, bool CG>
__device__ __forceinline__ Vec<D> accel_partial(int i, int lane, const DevParams& P, const float* __restrict__ x,
                                                const float* __restrict__ H, const float* __restrict__ m,
                                                const float* __restrict__ rho, const float* praw, float mu, float qi,
                                                const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt,
                                                const int32_t* __restrict__ list) {
    Vec<D> s = vzero<D>();
    const Vec<D> xi = load_vec<D>(x, i);
    const int b = offs[i], e = b + cnt[i];
    for (int q = b + lane; q < e; q += G) {
        int j, k; entry(list, q, j, k);
        const Vec<D> xij = dist_vec<D>(xi, load_vec<D>(x, j), P.dom);
        const float r = safe_sqrt(dot<D>(xij, xij));
        float W; Vec<D> g;
        kernelWG<KF, D>(xij, r, __ldg(H + j), W, g);
        const float rj = __ldg(rho + j);
        const float pj = (CG ? __ldcg(praw + j) : __ldg(praw + j)) - mu;
        const float c = __ldg(m + j) * (qi + pj / (rj * rj));
        #pragma unroll
        for (int a = 0; a < D; ++a) s.v[a] += c * g.v[a];
    }
    return s;
}

// Pressure shift, modules/incompressible/drift.py:38-57: -sum_j V_j (a_j - a_i).gradW(x_ij, H_j).
template <int KF, int D, int G, bool CG>
__device__ __forceinline__ float shift_partial(int i, int lane, const DevParams& P, const float* __restrict__ x,
                                               const float* __restrict__ H, const float* __restrict__ m,
                                               const float* __restrict__ rho, const float* acc, const Vec<D>& ai,
                                               const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt,
                                               const int32_t* __restrict__ list) {
    float s = 0.f;
    const Vec<D> xi = load_vec<D>(x, i);
    const int b = offs[i], e = b + cnt[i];
    for (int q = b + lane; q < e; q += G) {
        int j, k; entry(list, q, j, k);
        const Vec<D> xij = dist_vec<D>(xi, load_vec<D>(x, j), P.dom);
        const float r = safe_sqrt(dot<D>(xij, xij));
        float W; Vec<D> g;
        kernelWG<KF, D>(xij, r, __ldg(H + j), W, g);
        const Vec<D> aj = CG ? load_vec_cg<D>(acc, j) : load_vec<D>(acc, j);
        float t = 0.f;
        #pragma unroll
        for (int a = 0; a < D; ++a) t += (aj.v[a] - ai.v[a]) * g.v[a];
        s += __ldg(m + j) / __ldg(rho + j) * t;
    }
    return s;
}

// ---------------------------------------------------------------- cached pair gradients
// A solve evaluates the same pair gradients m_j gradW(x_ij, H_j) twice per iteration.  The
// prep pass, which forms them anyway, stores them by row entry and the iterations stream them
// back: in 3D with the neighbour's index in the fourth word, one 16-byte load per entry.
// They are read once per phase, so they bypass L1, which is left to the gathers.
template <int D> constexpr int pair_grad_floats() { return D == 3 ? 4 : D; }
template <int D> __device__ __forceinline__ void put_pair_grad(float* __restrict__ grads, int k, int j, float mj, const Vec<D>& g) {
    if constexpr (D == 3)
        reinterpret_cast<float4*>(grads)[k] = make_float4(mj * g.v[0], mj * g.v[1], mj * g.v[2], __int_as_float(j));
    else if constexpr (D == 2)
        reinterpret_cast<float2*>(grads)[k] = make_float2(mj * g.v[0], mj * g.v[1]);
    else
        grads[k] = mj * g.v[0];
}
template <int D> __device__ __forceinline__ void get_pair_grad(const float* __restrict__ grads, const int32_t* __restrict__ list, int k,
                                                               int& j, Vec<D>& g) {
    if constexpr (D == 3) {
        float4 t;
        asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
            : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w) : "l"(reinterpret_cast<const float4*>(grads) + k));
        g.v[0] = t.x; g.v[1] = t.y; g.v[2] = t.z;
        j = __float_as_int(t.w);
    } else {
        j = __ldg(list + k);
        if constexpr (D == 2) {
            asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];"
                : "=f"(g.v[0]), "=f"(g.v[1]) : "l"(reinterpret_cast<const float2*>(grads) + k));
        } else {
            g.v[0] = __ldg(grads + k);
        }
    }
}

// ---------------------------------------------------------------- prep: divergence, alpha, source, diagonal
// mode -1: standalone (div_out and/or alpha_out); 0: divergence-free solve; 1: density solve.
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_dfsph_prep(int n, DevParams P, int mode, float rho0, const float* __restrict__ x, const float* __restrict__ H,
             const float* __restrict__ m, const float* __restrict__ rho, const float* __restrict__ v,
             const float* __restrict__ dvdt, const float* __restrict__ dtp, const int32_t* __restrict__ offs,
             const int32_t* __restrict__ cnt, const int32_t* __restrict__ list, float* __restrict__ div_out,
             float* __restrict__ alpha_out, const float* __restrict__ p_init, int init_mode, float* __restrict__ src,
             float* __restrict__ diag, float* __restrict__ p0, float* __restrict__ grads = nullptr,
             float2* __restrict__ pq = nullptr) {
    Grp<G> g(n);
    const bool want_div = div_out || src, want_alpha = alpha_out || diag;
    const float dt = dtp ? *dtp : 0.f;
    float sdiv = 0.f, sB = 0.f;
    Vec<D> sA = vzero<D>();
    if (g.valid) {
        const int i = g.i;
        const Vec<D> xi = load_vec<D>(x, i);
        const float Hi = H[i];
        Vec<D> vi = load_vec<D>(v, i);
        if (dvdt) {
            const Vec<D> ai = load_vec<D>(dvdt, i);
            #pragma unroll
            for (int a = 0; a < D; ++a) vi.v[a] = __fadd_rn(vi.v[a], __fmul_rn(dt, ai.v[a]));
        }
        const int b = offs[i], e = b + cnt[i];
        for (int q = b + g.lane; q < e; q += G) {
            int j, k; entry(list, q, j, k);
            const Vec<D> xij = dist_vec<D>(xi, load_vec<D>(x, j), P.dom);
            const float r = safe_sqrt(dot<D>(xij, xij));
            const float Hj = __ldg(H + j), mj = __ldg(m + j);
            const float Vj = mj / __ldg(rho + j);
            float W;
            Vec<D> gS, gG;
            kernelWG<KF, D>(xij, r, Hj, W, gS);
            if (grads) put_pair_grad<D>(grads, k, j, mj, gS);
            if (Hj == Hi) gG = gS; else kernelWG<KF, D>(xij, r, Hi, W, gG);
            if (want_div) {
                Vec<D> vj = load_vec<D>(v, j);
                if (dvdt) {
                    const Vec<D> aj = load_vec<D>(dvdt, j);
                    #pragma unroll
                    for (int a = 0; a < D; ++a) vj.v[a] = __fadd_rn(vj.v[a], __fmul_rn(dt, aj.v[a]));
                }
                float t = 0.f;
                #pragma unroll
                for (int a = 0; a < D; ++a) t += (vj.v[a] - vi.v[a]) * gS.v[a];
                sdiv += Vj * t;
            }
            if (want_alpha) {
                #pragma unroll
                for (int a = 0; a < D; ++a) sA.v[a] += Vj * gG.v[a];
                sB += Vj * Vj / mj * dot<D>(gG, gG);
            }
        }
    }
    sdiv = gsum<G>(sdiv);
    sB = gsum<G>(sB);
    #pragma unroll
    for (int a = 0; a < D; ++a) sA.v[a] = gsum<G>(sA.v[a]);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    const float div = -rho0 * sdiv;                       // momentum/incompressible.py:22
    const float Ai = m[i] / rho[i];
    const float alpha = -(Ai / m[i] * dot<D>(sA, sA) + Ai * sB);   // wp_alpha.py:115, :313
    if (div_out) div_out[i] = div;
    if (alpha_out) alpha_out[i] = alpha;
    if (mode == 0) {                                      // divergenceFree.py:54, :62, :72
        src[i] = -div;
        diag[i] = dt * alpha;
        p0[i] = init_mode ? p_init[i] : p_init[i] * 0.75f;
    } else if (mode == 1) {                               // incompressible.py:54-79
        float rs = __fadd_rn(rho[i], __fmul_rn(dt, div));
        rs = rs < 0.9f ? 0.9f : rs;
        src[i] = rho0 - rs;
        const float a = (dt * dt) * alpha;
        diag[i] = a > -1e-6f ? -1e-6f : a;
        p0[i] = init_mode ? p_init[i] : 0.f;
    }
    if (pq) pq[i] = make_float2(p0[i], 1.f / (rho[i] * rho[i]));
}

// ---------------------------------------------------------------- standalone accel / shift passes
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_iisph_accel(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
              const float* __restrict__ rho, const float* __restrict__ pr, const int32_t* __restrict__ offs,
              const int32_t* __restrict__ cnt, const int32_t* __restrict__ list, float* __restrict__ acc) {
    Grp<G> g(n);
    Vec<D> s = vzero<D>();
    float rhoi = 1.f;
    if (g.valid) {
        rhoi = rho[g.i];
        s = accel_partial<KF, D, G, false>(g.i, g.lane, P, x, H, m, rho, pr, 0.f, pr[g.i] / (rhoi * rhoi), offs, cnt, list);
    }
    #pragma unroll
    for (int a = 0; a < D; ++a) s.v[a] = gsum<G>(s.v[a]);
    if (!g.valid || g.lane != 0) return;
    #pragma unroll
    for (int a = 0; a < D; ++a) s.v[a] = -(rhoi * s.v[a]) / rhoi;
    store_vec<D>(acc, g.i, s);
}

template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_iisph_shift(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
              const float* __restrict__ rho, const float* __restrict__ acc, const int32_t* __restrict__ offs,
              const int32_t* __restrict__ cnt, const int32_t* __restrict__ list, float* __restrict__ shift) {
    Grp<G> g(n);
    float s = 0.f;
    if (g.valid) s = shift_partial<KF, D, G, false>(g.i, g.lane, P, x, H, m, rho, acc, load_vec<D>(acc, g.i), offs, cnt, list);
    s = gsum<G>(s);
    if (g.valid && g.lane == 0) shift[g.i] = -s;
}

// ---------------------------------------------------------------- persistent Jacobi solve
struct JacobiArgs {
    int n, mode, min_it, max_it;
    float omega, tol;
    DevParams P;
    const float *x, *H, *m, *rho, *src, *diag, *dtp;
    const int32_t *offs, *cnt, *list;
    float* praw;       // un-gauged pressure of the last update (p0 before the first)
    float* p_out;      // gauged pressure (the iteration's pressureA; the result at the end)
    float* acc;        // pressure acceleration [n*D]
    float* hist;       // [max_it*4]
    int32_t* iters_out;
    int32_t* status_out;
    JacobiCtl* ctl;
    unsigned long long barrier_ns;   // grid-barrier wait limit
};

template <typename T> __device__ __forceinline__ T warp_sum(T v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ unsigned int warp_min_u(unsigned int v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ unsigned int warp_max_u(unsigned int v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// A grid barrier ran out: the block records the timeout (block 0 also the iteration it
// had reached) and returns.  p_out and acc hold the last completed phase A.
__device__ __forceinline__ void jacobi_gave_up(const JacobiArgs& a, int it) {
    if (threadIdx.x == 0) {
        atomicOr(a.status_out, SPH_STATUS_TIMEOUT);
        if (blockIdx.x == 0) *a.iters_out = it;
    }
}

template <int KF, int D>
__global__ void __launch_bounds__(JAC_BLOCK)
k_jacobi(JacobiArgs a) {
    constexpr int G = JAC_G;
    __shared__ double sh_sum[JAC_BLOCK / 32][2];
    __shared__ unsigned int sh_mm[JAC_BLOCK / 32][2];
    const int lane = threadIdx.x & (G - 1);
    const int warp = threadIdx.x >> 5;
    const int n = a.n;
    const int rounds = (n + (int)gridDim.x * JAC_PPB - 1) / ((int)gridDim.x * JAC_PPB);
    const float dt = *a.dtp;
    const float dtf = a.mode == 0 ? dt : dt * dt;
    JacobiCtl* c = a.ctl;
    float mu = 0.f;
    unsigned int arrived = 0;
    int it = 0;
    bool converged = false;

    for (;;) {
        // ------------------------------------------------ phase A: pressure acceleration
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const int s1 = (it + 1) % 3;
            c->sum[s1][0] = 0.0; c->sum[s1][1] = 0.0;
            c->mm[s1][0] = 0xffffffffu; c->mm[s1][1] = 0u;
            if (it == 0) { c->sum[0][0] = 0.0; c->sum[0][1] = 0.0; c->mm[0][0] = 0xffffffffu; c->mm[0][1] = 0u; }
        }
        for (int rd = 0; rd < rounds; ++rd) {
            const int i = (rd * (int)gridDim.x + (int)blockIdx.x) * JAC_PPB + (int)threadIdx.x / G;
            const bool valid = i < n;
            Vec<D> s = vzero<D>();
            float pi = 0.f, rhoi = 1.f;
            if (valid) {
                pi = __ldcg(a.praw + i) - mu;
                rhoi = __ldg(a.rho + i);
                s = accel_partial<KF, D, G, true>(i, lane, a.P, a.x, a.H, a.m, a.rho, a.praw, mu, pi / (rhoi * rhoi),
                                                      a.offs, a.cnt, a.list);
            }
            #pragma unroll
            for (int d = 0; d < D; ++d) s.v[d] = gsum<G>(s.v[d]);
            if (valid && lane == 0) {
                #pragma unroll
                for (int d = 0; d < D; ++d) s.v[d] = -(rhoi * s.v[d]) / rhoi;
                store_vec<D>(a.acc, i, s);
                a.p_out[i] = pi;
            }
        }
        if (converged || it >= a.max_it) break;
        if (!grid_barrier(&c->bar, arrived, a.barrier_ns)) { jacobi_gave_up(a, it); return; }

        // ------------------------------------------------ phase B: shift, residual, update
        double psum = 0.0, esum = 0.0;
        unsigned int pmin = 0xffffffffu, pmax = 0u;
        for (int rd = 0; rd < rounds; ++rd) {
            const int i = (rd * (int)gridDim.x + (int)blockIdx.x) * JAC_PPB + (int)threadIdx.x / G;
            const bool valid = i < n;
            float s = 0.f;
            if (valid) s = shift_partial<KF, D, G, true>(i, lane, a.P, a.x, a.H, a.m, a.rho, a.acc, load_vec_cg<D>(a.acc, i),
                                                             a.offs, a.cnt, a.list);
            s = gsum<G>(s);
            if (valid && lane == 0) {
                const float r = a.src[i] - dtf * (-s);
                float pb = __ldcg(a.p_out + i) + a.omega * r / a.diag[i];
                float e;
                if (a.mode == 1) {
                    pb = pb < 0.f ? 0.f : pb;                       // incompressible.py:108
                    e = -r < -a.tol ? -a.tol : -r;                  // :111
                } else {
                    e = fabsf(r);                                   // divergenceFree.py:112
                }
                a.praw[i] = pb;
                psum += (double)pb;
                esum += (double)e;
                const unsigned int o = f2o(pb);
                pmin = min(pmin, o);
                pmax = max(pmax, o);
            }
        }
        psum = warp_sum(psum); esum = warp_sum(esum);
        pmin = warp_min_u(pmin); pmax = warp_max_u(pmax);
        if ((threadIdx.x & 31) == 0) { sh_sum[warp][0] = psum; sh_sum[warp][1] = esum; sh_mm[warp][0] = pmin; sh_mm[warp][1] = pmax; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double ps = 0.0, es = 0.0;
            unsigned int lo = 0xffffffffu, hi = 0u;
            for (int w = 0; w < JAC_BLOCK / 32; ++w) { ps += sh_sum[w][0]; es += sh_sum[w][1]; lo = min(lo, sh_mm[w][0]); hi = max(hi, sh_mm[w][1]); }
            const int sl = it % 3;
            atomicAdd(&c->sum[sl][0], ps);
            atomicAdd(&c->sum[sl][1], es);
            atomicMin(&c->mm[sl][0], lo);
            atomicMax(&c->mm[sl][1], hi);
        }
        if (!grid_barrier(&c->bar, arrived, a.barrier_ns)) { jacobi_gave_up(a, it); return; }

        // ------------------------------------------------ decide (identical in every block)
        const int sl = it % 3;
        const double ps = *(volatile double*)&c->sum[sl][0];
        const double es = *(volatile double*)&c->sum[sl][1];
        const float lo = o2f(*(volatile unsigned int*)&c->mm[sl][0]);
        const float hi = o2f(*(volatile unsigned int*)&c->mm[sl][1]);
        const double mean = ps / (double)n;
        const double err = es / (double)n;
        mu = a.mode == 0 ? (float)mean : 0.f;                       // divergenceFree.py:104
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.hist[it * 4 + 0] = (float)err;
            a.hist[it * 4 + 1] = lo - mu;
            a.hist[it * 4 + 2] = hi - mu;
            a.hist[it * 4 + 3] = (float)(mean - (double)mu);
        }
        const bool finite = isfinite(err);
        if (!finite) { if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(&c->bar.status, SPH_STATUS_NONFINITE); }
        converged = (it >= a.min_it && err < (double)a.tol) || !finite;
        ++it;
    }
    if (threadIdx.x == 0) {
        int st = *(volatile int*)&c->bar.status;
        if (blockIdx.x == 0) {
            if (!converged && a.max_it > 0) st |= SPH_STATUS_NOT_CONVERGED;
            *a.iters_out = it;
        }
        if (st) atomicOr(a.status_out, st);
    }
}

// The same solve over cached pair gradients g_ij = m_j gradW(x_ij, H_j):
//   phase A   a_i = -sum_j (p_i / rho_i^2 + p_j / rho_j^2) g_ij
//   phase B   s_i = -sum_j (1 / rho_j) (a_j - a_i) . g_ij
// An entry is one streamed load and one gather of the neighbour's (p, 1 / rho^2) or (a, 1 / rho),
// packed in one word pair or quad, instead of five gathers, a minimum image and a kernel
// gradient with its divisions.  U entries per lane are loaded together.  The gathered arrays
// are rewritten by other blocks between the phases: they are read with plain loads, which the
// acquire of the grid barrier makes current, and so may hit L1.
//
// Large solves are bound by the stream of gradients from HBM (16 bytes per entry and phase in
// 3D): 1,000,000 particles with 40 neighbours take 128 us per phase, 5.2 TB/s of stream, where
// k_jacobi took 353 us; 4 lanes per particle with 5 entries in flight beat 8 x 4 (149 us) and
// 16 x 3 (168 us).  Small solves are bound by the latency of a phase and its barrier.  With
// HOLD a group keeps one particle for the whole solve, its first G * U entries in registers, so
// a phase is one gather, one reduction and one barrier; more entries are loaded each time.
// 9,216 particles: 3.1 us per phase and barrier, 10.8 us in k_jacobi (3.7 against 4.5 us streaming when the two
// were compared, before the blocks' slots);
// 4,096 particles in 3D: 160 us a solve of 33 phases with 8 lanes against 182 us with 4 and 197 us
// streaming.  The blocks' partial sums go to one slot each, which every block adds up after
// the barrier: four atomics per block on one line cost 144 blocks 1 us per iteration more.
struct JacobiGradArgs {
    int n, mode, min_it, max_it;
    float omega, tol;
    const float *rho, *src, *diag, *dtp, *grads;
    const int32_t *offs, *cnt, *list;
    float2* pq;        // (un-gauged pressure of the last update, 1 / rho^2)
    float4* a4;        // (pressure acceleration, 1 / rho)
    struct JacobiSums* sums;   // per block
    float* p_out;
    float* acc;
    float* hist;
    int32_t* iters_out;
    int32_t* status_out;
    JacobiCtl* ctl;
    unsigned long long barrier_ns;
};
template <int D> __device__ __forceinline__ Vec<D> vec_of(const float4& t) {
    Vec<D> r;
    r.v[0] = t.x;
    if constexpr (D > 1) r.v[1] = t.y;
    if constexpr (D > 2) r.v[2] = t.z;
    return r;
}

// Partial sums of one block: sum p, sum of the error term, min p and max p (ordered encoding).
struct JacobiSums { double p, e; unsigned int lo, hi; };
// Sums over the block, in a fixed order, returned to every thread.
template <int BLOCK> __device__ __forceinline__ JacobiSums block_sums(JacobiSums t, JacobiSums* sh) {
    t.p = warp_sum(t.p); t.e = warp_sum(t.e);
    t.lo = warp_min_u(t.lo); t.hi = warp_max_u(t.hi);
    __syncthreads();                              // earlier readers of sh are done
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    t = sh[0];
    #pragma unroll
    for (int w = 1; w < BLOCK / 32; ++w) { t.p += sh[w].p; t.e += sh[w].e; t.lo = min(t.lo, sh[w].lo); t.hi = max(t.hi, sh[w].hi); }
    return t;
}

template <int D, int G, int U, int BLOCK, int MINB, bool HOLD>
__global__ void __launch_bounds__(BLOCK, MINB)
k_jacobi_grad(JacobiGradArgs a) {
    constexpr int PPB = BLOCK / G;
    __shared__ JacobiSums sh[BLOCK / 32];
    const int lane = threadIdx.x & (G - 1);
    const int n = a.n;
    const int rounds = (n + (int)gridDim.x * PPB - 1) / ((int)gridDim.x * PPB);
    const float dt = *a.dtp;
    const float dtf = a.mode == 0 ? dt : dt * dt;
    JacobiCtl* c = a.ctl;
    float mu = 0.f;
    unsigned int arrived = 0;
    int it = 0;
    bool converged = false, gave_up = false;

    // U entries of the row of particle i from entry q on (past the row's end: no gradient)
    int j[U];
    Vec<D> g[U];
    auto load_entries = [&](int i, int q, int e) {
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            j[u] = i; g[u] = vzero<D>();
            if (q + u * G < e) get_pair_grad<D>(a.grads, a.list, q + u * G, j[u], g[u]);
        }
    };
    // HOLD: one particle per group for the whole solve, its first G * U entries in registers
    int hb = 0, he = 0;
    if (HOLD) {
        const int i = (int)blockIdx.x * PPB + (int)threadIdx.x / G;
        if (i < n) { hb = a.offs[i]; he = hb + a.cnt[i]; }
        load_entries(i < n ? i : 0, hb + lane, he);
    }

    for (;;) {
        // ------------------------------------------------ phase A: pressure acceleration
        for (int rd = 0; rd < rounds; ++rd) {
            const int i = (rd * (int)gridDim.x + (int)blockIdx.x) * PPB + (int)threadIdx.x / G;
            const bool valid = i < n;
            Vec<D> s = vzero<D>();
            if (valid) {
                const float2 ti = a.pq[i];
                const float qi = (ti.x - mu) * ti.y;
                const int b = HOLD ? hb : a.offs[i], e = HOLD ? he : b + a.cnt[i];
                bool reload = false;
                for (int q = b + lane; q < e; q += G * U) {
                    if (!HOLD || q != b + lane) { load_entries(i, q, e); reload = HOLD; }
                    float2 t[U];
                    #pragma unroll
                    for (int u = 0; u < U; ++u) t[u] = a.pq[j[u]];
                    #pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float w = qi + (t[u].x - mu) * t[u].y;
                        #pragma unroll
                        for (int d = 0; d < D; ++d) s.v[d] += w * g[u].v[d];
                    }
                }
                if (HOLD && reload) load_entries(i, b + lane, e);
            }
            #pragma unroll
            for (int d = 0; d < D; ++d) s.v[d] = gsum<G>(s.v[d]);
            if (valid && lane == 0)
                a.a4[i] = make_float4(-s.v[0], D > 1 ? -s.v[D > 1 ? 1 : 0] : 0.f, D > 2 ? -s.v[D > 2 ? 2 : 0] : 0.f, 1.f / a.rho[i]);
        }
        if (converged || it >= a.max_it) break;
        if (!grid_barrier(&c->bar, arrived, a.barrier_ns)) { gave_up = true; break; }

        // ------------------------------------------------ phase B: shift, residual, update
        double psum = 0.0, esum = 0.0;
        unsigned int pmin = 0xffffffffu, pmax = 0u;
        for (int rd = 0; rd < rounds; ++rd) {
            const int i = (rd * (int)gridDim.x + (int)blockIdx.x) * PPB + (int)threadIdx.x / G;
            const bool valid = i < n;
            float s = 0.f;
            if (valid) {
                const Vec<D> ai = vec_of<D>(a.a4[i]);
                const int b = HOLD ? hb : a.offs[i], e = HOLD ? he : b + a.cnt[i];
                bool reload = false;
                for (int q = b + lane; q < e; q += G * U) {
                    if (!HOLD || q != b + lane) { load_entries(i, q, e); reload = HOLD; }
                    float4 t[U];
                    #pragma unroll
                    for (int u = 0; u < U; ++u) t[u] = a.a4[j[u]];
                    #pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const Vec<D> aj = vec_of<D>(t[u]);
                        float w = 0.f;
                        #pragma unroll
                        for (int d = 0; d < D; ++d) w += (aj.v[d] - ai.v[d]) * g[u].v[d];
                        s += t[u].w * w;
                    }
                }
                if (HOLD && reload) load_entries(i, b + lane, e);
            }
            s = gsum<G>(s);
            if (valid && lane == 0) {
                const float r = a.src[i] - dtf * (-s);
                float pb = (a.pq[i].x - mu) + a.omega * r / a.diag[i];
                float e;
                if (a.mode == 1) {
                    pb = pb < 0.f ? 0.f : pb;                       // incompressible.py:108
                    e = -r < -a.tol ? -a.tol : -r;                  // :111
                } else {
                    e = fabsf(r);                                   // divergenceFree.py:112
                }
                a.pq[i].x = pb;
                psum += (double)pb;
                esum += (double)e;
                const unsigned int o = f2o(pb);
                pmin = min(pmin, o);
                pmax = max(pmax, o);
            }
        }
        JacobiSums t = block_sums<BLOCK>(JacobiSums{psum, esum, pmin, pmax}, sh);
        if (threadIdx.x == 0) a.sums[blockIdx.x] = t;
        if (!grid_barrier(&c->bar, arrived, a.barrier_ns)) { gave_up = true; break; }

        // ------------------------------------------------ decide (identical in every block: each sums
        // every block's partial sums in the same order)
        t = JacobiSums{0.0, 0.0, 0xffffffffu, 0u};
        for (int q = threadIdx.x; q < (int)gridDim.x; q += BLOCK) {
            const JacobiSums o = a.sums[q];
            t.p += o.p; t.e += o.e; t.lo = min(t.lo, o.lo); t.hi = max(t.hi, o.hi);
        }
        t = block_sums<BLOCK>(t, sh);
        const double ps = t.p, es = t.e;
        const float lo = o2f(t.lo), hi = o2f(t.hi);
        const double mean = ps / (double)n;
        const double err = es / (double)n;
        mu = a.mode == 0 ? (float)mean : 0.f;                       // divergenceFree.py:104
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.hist[it * 4 + 0] = (float)err;
            a.hist[it * 4 + 1] = lo - mu;
            a.hist[it * 4 + 2] = hi - mu;
            a.hist[it * 4 + 3] = (float)(mean - (double)mu);
        }
        const bool finite = isfinite(err);
        if (!finite) { if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(&c->bar.status, SPH_STATUS_NONFINITE); }
        converged = (it >= a.min_it && err < (double)a.tol) || !finite;
        ++it;
    }
    // the results of this block's particles, which its own lead lanes wrote: the last phase A
    for (int rd = 0; rd < rounds; ++rd) {
        const int i = (rd * (int)gridDim.x + (int)blockIdx.x) * PPB + (int)threadIdx.x / G;
        if (i >= n || lane != 0) continue;
        store_vec<D>(a.acc, i, vec_of<D>(a.a4[i]));
        a.p_out[i] = a.pq[i].x - mu;
    }
    if (threadIdx.x == 0) {
        int st = gave_up ? SPH_STATUS_TIMEOUT : *(volatile int*)&c->bar.status;
        if (blockIdx.x == 0) {
            if (!gave_up && !converged && a.max_it > 0) st |= SPH_STATUS_NOT_CONVERGED;
            *a.iters_out = it;
        }
        if (st) atomicOr(a.status_out, st);
    }
}

// ---------------------------------------------------------------- host side
constexpr size_t kCtlBytes = 256;
static_assert(sizeof(JacobiCtl) <= kCtlBytes, "control block");

static size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

static int64_t dfsph_ws_bytes(int64_t n) { return (int64_t)(kCtlBytes + 3 * align256((size_t)n * sizeof(float))); }

// SMs of the current device (a B200's 148 where the query fails: the launch then reports why).
static int device_sms() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return sms;
}

// One cooperative launch of a persistent solve kernel over n particles (KERN names the kernel, so
// that each instantiation keeps its own occupancy), of at most LIMIT blocks.  ONE_ROUND: the kernel needs all
// particles in one round; where they do not fit, nothing is launched and *launched stays false.
template <auto KERN, int BLOCK, int PPB, bool ONE_ROUND, int64_t LIMIT, typename Args>
static int launch_persistent(Args& a, cudaStream_t s, bool* launched) {
    static std::mutex mu;
    static int cached_dev = -1, blocks_per_sm = 0, num_sms = 0;
    int64_t resident = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "jacobi: cudaGetDevice: %s", cudaGetErrorString(e));
    {
        std::lock_guard<std::mutex> lock(mu);
        if (cached_dev != dev) {
            int coop = 0;
            e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
            if (e != cudaSuccess || !coop) return set_error(SPH_ERR_UNSUPPORTED, "jacobi: device %d has no cooperative launch", dev);
            e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "jacobi: SM count: %s", cudaGetErrorString(e));
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, KERN, BLOCK, 0);
            if (e != cudaSuccess || blocks_per_sm < 1) return set_error(SPH_ERR_CUDA, "jacobi: occupancy query failed");
            cached_dev = dev;
        }
        resident = (int64_t)blocks_per_sm * num_sms;
    }
    const int grid = persistent_grid(a.n, PPB, resident, LIMIT, ONE_ROUND);
    if (grid == 0) return SPH_OK;
    *launched = true;
    void* args[] = {&a};
    count_launch();
    e = cudaLaunchCooperativeKernel((const void*)KERN, dim3(grid), dim3(BLOCK), args, 0, s);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "jacobi: cooperative launch: %s", cudaGetErrorString(e));
    return SPH_OK;
}

// Bytes per row entry and in all of the buffer of cached pair gradients: the particles' (p, 1 / rho^2)
// and (a, 1 / rho), then one gradient per entry.
constexpr int64_t kSumSlots = 2048;                          // one per block of a solve
constexpr size_t kSumsBytes = kSumSlots * sizeof(JacobiSums);
static int64_t dfsph_grad_bytes(int64_t n, int64_t entries, int dim) {
    return (int64_t)(kSumsBytes + align256((size_t)n * sizeof(float2)) + align256((size_t)n * sizeof(float4)) +
                     align256((size_t)entries * (dim == 3 ? 4 : dim) * sizeof(float)));
}

static int dfsph_solve(int mode, const SphParams* p, const SphJacobiConfig* cfg, int64_t n, const float* x, const float* H,
                       const float* m, const float* rho, const float* v, const float* dvdt, const float* p_init,
                       const float* dt, const int32_t* offs, const int32_t* cnt, const int32_t* list, void* ws,
                       int64_t ws_bytes, float* p_out, float* accel_out, float* history, int32_t* iterations, int32_t* status,
                       void* stream, int64_t entries = 0, void* gradients = nullptr, int64_t gradient_bytes = 0) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(cfg); WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(v);
    WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(ws); WSPH_CHECK_PTR(p_out); WSPH_CHECK_PTR(accel_out); WSPH_CHECK_PTR(history);
    WSPH_CHECK_PTR(iterations); WSPH_CHECK_PTR(status); CHECK_CSR();
    if (cfg->init_mode != 0 && cfg->init_mode != 1) return set_error(SPH_ERR_BAD_ARG, "jacobi: init_mode must be 0 or 1");
    if ((mode == 0 || cfg->init_mode == 1) && !p_init) return set_error(SPH_ERR_BAD_ARG, "jacobi: p_init is required");
    if (cfg->max_iterations < 0 || cfg->min_iterations < 0 || cfg->max_iterations > (1 << 20))
        return set_error(SPH_ERR_BAD_ARG, "jacobi: iteration counts out of range");
    if (!(cfg->relaxation == cfg->relaxation) || !(cfg->tolerance == cfg->tolerance))
        return set_error(SPH_ERR_BAD_ARG, "jacobi: NaN relaxation or tolerance");
    if (cfg->barrier_timeout_us < 0) return set_error(SPH_ERR_BAD_ARG, "jacobi: barrier_timeout_us must be >= 0");
    if (ws_bytes < dfsph_ws_bytes(n)) return set_error(SPH_ERR_WORKSPACE, "jacobi: workspace %lld < %lld bytes", (long long)ws_bytes,
                                                       (long long)dfsph_ws_bytes(n));
    if (reinterpret_cast<uintptr_t>(ws) & 255) return set_error(SPH_ERR_BAD_ARG, "jacobi: workspace must be 256-byte aligned");
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, dvdt, "dvdt")) ||
        (rc = check_align_vec(P, accel_out, "accel_out")))
        return rc;
    if (gradients) {
        if (entries < 0 || entries > 0x7fffffff) return set_error(SPH_ERR_BAD_ARG, "jacobi: entries out of range");
        if (gradient_bytes < dfsph_grad_bytes(n, entries, P.dim))
            return set_error(SPH_ERR_WORKSPACE, "jacobi: gradient buffer %lld < %lld bytes", (long long)gradient_bytes,
                             (long long)dfsph_grad_bytes(n, entries, P.dim));
        if (reinterpret_cast<uintptr_t>(gradients) & 255) return set_error(SPH_ERR_BAD_ARG, "jacobi: the gradient buffer must be 256-byte aligned");
    }
    char* w = static_cast<char*>(ws);
    JacobiCtl* ctl = reinterpret_cast<JacobiCtl*>(w);
    const size_t nb = align256((size_t)n * sizeof(float));
    float* praw = reinterpret_cast<float*>(w + kCtlBytes);
    float* src = reinterpret_cast<float*>(w + kCtlBytes + nb);
    float* diag = reinterpret_cast<float*>(w + kCtlBytes + 2 * nb);
    cudaError_t e = cudaMemsetAsync(ctl, 0, kCtlBytes, s);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "jacobi: memset: %s", cudaGetErrorString(e));
    const float rho0 = (float)cfg->rest_density;
    float2* pq = nullptr;
    float4* a4 = nullptr;
    float* grads = nullptr;
    if (gradients) {
        char* gb = static_cast<char*>(gradients) + kSumsBytes;
        pq = reinterpret_cast<float2*>(gb);
        gb += align256((size_t)n * sizeof(float2));
        a4 = reinterpret_cast<float4*>(gb);
        grads = reinterpret_cast<float*>(gb + align256((size_t)n * sizeof(float4)));
    }
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_dfsph_prep<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, mode, rho0, x, H, m, rho, v, dvdt, dt, offs, cnt, list, nullptr, nullptr, p_init, cfg->init_mode, src, diag, praw, grads, pq)));
    if ((rc = check_launch("jacobi prep"))) return rc;
    const unsigned long long barrier_ns = cfg->barrier_timeout_us > 0 ? 1000ull * (unsigned long long)cfg->barrier_timeout_us : kBarrierLimitNs;
    if (gradients) {
        JacobiGradArgs a;
        a.n = (int)n; a.mode = mode; a.min_it = cfg->min_iterations; a.max_it = cfg->max_iterations;
        a.omega = (float)cfg->relaxation; a.tol = (float)cfg->tolerance;
        a.rho = rho; a.src = src; a.diag = diag; a.dtp = dt; a.grads = grads;
        a.offs = offs; a.cnt = cnt; a.list = list; a.pq = pq; a.a4 = a4; a.sums = static_cast<JacobiSums*>(gradients);
        a.p_out = p_out; a.acc = accel_out; a.hist = history; a.iters_out = iterations; a.status_out = status; a.ctl = ctl;
        a.barrier_ns = barrier_ns;
#define JACOBI_GRAD(G, U, MINB, HOLD) WSPH_DISPATCH_DIM(P.dim, \
        (rc = launch_persistent<k_jacobi_grad<D, G, U, JAC_BLOCK, MINB, HOLD>, JAC_BLOCK, JAC_BLOCK / G, HOLD, kSumSlots>(a, s, &launched)))
        // The split by size (see k_jacobi_grad): one block of 8 lanes per particle on each SM, two
        // blocks of 4 lanes, or a loop over particles, which also takes what the first two cannot hold (fewer
        // resident blocks than their launch bounds ask for).
        const int sms = device_sms();
        bool launched = false;
        if (n <= (int64_t)sms * (JAC_BLOCK / 8)) { JACOBI_GRAD(8, 6, 2, true); }
        else if (n <= (int64_t)sms * 2 * (JAC_BLOCK / 4)) { JACOBI_GRAD(4, 10, 2, true); }
        if (rc == SPH_OK && !launched) { rc = SPH_ERR_UNSUPPORTED; JACOBI_GRAD(4, 5, 4, false); }
#undef JACOBI_GRAD
        return rc;
    }
    JacobiArgs a;
    a.n = (int)n; a.mode = mode; a.min_it = cfg->min_iterations; a.max_it = cfg->max_iterations;
    a.omega = (float)cfg->relaxation; a.tol = (float)cfg->tolerance; a.P = P;
    a.x = x; a.H = H; a.m = m; a.rho = rho; a.src = src; a.diag = diag; a.dtp = dt;
    a.offs = offs; a.cnt = cnt; a.list = list;
    a.praw = praw; a.p_out = p_out; a.acc = accel_out; a.hist = history;
    a.iters_out = iterations; a.status_out = status; a.ctl = ctl;
    a.barrier_ns = barrier_ns;
    bool launched = false;
    rc = SPH_ERR_UNSUPPORTED;
    WSPH_DISPATCH_KD(P.kernel, P.dim, (rc = launch_persistent<k_jacobi<KF, D>, JAC_BLOCK, JAC_PPB, false, INT64_MAX>(a, s, &launched)));
    return rc;
}

// ---------------------------------------------------------------- learned warm start: input features
// Sums over particles of |src/diag|, the row count and diag (FP64, into the control block).
__global__ void k_feature_sums(int n, const float* __restrict__ src, const float* __restrict__ diag, const int32_t* __restrict__ cnt,
                               double* __restrict__ sums3) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        a += fabs((double)src[i] / (double)diag[i]);
        b += (double)cnt[i];
        c += (double)diag[i];
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0) { atomicAdd(sums3, a); atomicAdd(sums3 + 1, b); atomicAdd(sums3 + 2, c); }
}

// Eight per-particle features (gather support W(r, H_i), V_j = m_j / rho_j):
//   0  p_jac_i / P           p_jac = src / diag, the diagonal (one-iteration) Jacobi estimate
//   1  sum_j V_j W_ij p_jac_j / P
//   2  p_prev_i / P
//   3  sum_j V_j W_ij p_prev_j / P
//   4  100 (rho_i / rho0 - 1)
//   5  sum_j V_j W_ij - 1    (Shepard deficit: free surface)
//   6  cnt_i / mean(cnt) - 1
//   7  diag_i / mean(diag) - 1
// with P = mean_i |p_jac_i| (written to scale_out[0]); a network output y maps to p = y P.
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_features(int n, DevParams P, float rho0, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
           const float* __restrict__ rho, const float* __restrict__ src, const float* __restrict__ diag,
           const float* __restrict__ p_prev, const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt,
           const int32_t* __restrict__ list, const double* __restrict__ sums3, float* __restrict__ feats,
           float* __restrict__ scale_out) {
    Grp<G> g(n);
    const float Pref = (float)(sums3[0] / (double)n);
    const float inv_P = Pref > 0.f ? 1.f / Pref : 0.f;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
    if (g.valid) {
        const int i = g.i;
        const Vec<D> xi = load_vec<D>(x, i);
        const float Hi = H[i];
        const int b = offs[i], e = b + cnt[i];
        for (int q = b + g.lane; q < e; q += G) {
            int j, k; entry(list, q, j, k);
            const Vec<D> xij = dist_vec<D>(xi, load_vec<D>(x, j), P.dom);
            const float w = __ldg(m + j) / __ldg(rho + j) * kernelW<KF, D>(safe_sqrt(dot<D>(xij, xij)), Hi);
            s0 += w;
            s1 += w * (__ldg(src + j) / __ldg(diag + j));
            s2 += w * __ldg(p_prev + j);
        }
    }
    s0 = gsum<G>(s0); s1 = gsum<G>(s1); s2 = gsum<G>(s2);
    if (blockIdx.x == 0 && threadIdx.x == 0 && scale_out) scale_out[0] = Pref;
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    const float mean_cnt = (float)(sums3[1] / (double)n), mean_diag = (float)(sums3[2] / (double)n);
    float f[8];
    f[0] = src[i] / diag[i] * inv_P;
    f[1] = s1 * inv_P;
    f[2] = p_prev[i] * inv_P;
    f[3] = s2 * inv_P;
    f[4] = 100.f * (rho[i] / rho0 - 1.f);
    f[5] = s0 - 1.f;
    f[6] = mean_cnt > 0.f ? (float)cnt[i] / mean_cnt - 1.f : 0.f;
    f[7] = mean_diag != 0.f ? diag[i] / mean_diag - 1.f : 0.f;
    float4* o = reinterpret_cast<float4*>(feats + (size_t)i * 8);
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
}

}  // namespace wsph

using namespace wsph;

extern "C" {

int sph_dfsph_alpha(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                    const int32_t* offs, const int32_t* cnt, const int32_t* list, float* alpha_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(alpha_out); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    // v is only read for the divergence; x stands in as a valid vector array
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_dfsph_prep<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, -1, 0.f, x, H, m, rho, x, nullptr, nullptr, offs, cnt, list, nullptr, alpha_out, nullptr, 0, nullptr, nullptr, nullptr)));
    return check_launch("sph_dfsph_alpha");
}

int sph_incompressible_divergence(const SphParams* p, int64_t n, double rest_density, const float* x, const float* H,
                                  const float* m, const float* rho, const float* v, const float* dvdt, const float* dt,
                                  const int32_t* offs, const int32_t* cnt, const int32_t* list, float* div_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(div_out); CHECK_CSR();
    if (dvdt && !dt) return set_error(SPH_ERR_BAD_ARG, "sph_incompressible_divergence: dvdt given without dt");
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, dvdt, "dvdt"))) return rc;
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_dfsph_prep<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, -1, (float)rest_density, x, H, m, rho, v, dvdt, dt, offs, cnt, list, div_out, nullptr, nullptr, 0, nullptr, nullptr,
        nullptr)));
    return check_launch("sph_incompressible_divergence");
}

int sph_pressure_accel_iisph(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                             const float* pressure, const int32_t* offs, const int32_t* cnt, const int32_t* list, float* accel_out,
                             void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(pressure); WSPH_CHECK_PTR(accel_out);
    CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, accel_out, "accel_out"))) return rc;
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_iisph_accel<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, x, H, m, rho, pressure, offs, cnt, list, accel_out)));
    return check_launch("sph_pressure_accel_iisph");
}

int sph_pressure_shift_iisph(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                             const float* accel, const int32_t* offs, const int32_t* cnt, const int32_t* list, float* shift_out,
                             void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(accel); WSPH_CHECK_PTR(shift_out);
    CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, accel, "accel"))) return rc;
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_iisph_shift<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, x, H, m, rho, accel, offs, cnt, list, shift_out)));
    return check_launch("sph_pressure_shift_iisph");
}

int sph_dfsph_features(const SphParams* p, const SphJacobiConfig* cfg, int32_t mode, int64_t n, const float* x, const float* H,
                       const float* m, const float* rho, const float* v, const float* dvdt, const float* p_prev, const float* dt,
                       const int32_t* offs, const int32_t* cnt, const int32_t* list, void* workspace, int64_t workspace_bytes,
                       float* feats_out, float* scale_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(cfg); WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(v);
    WSPH_CHECK_PTR(p_prev); WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(workspace); WSPH_CHECK_PTR(feats_out); WSPH_CHECK_PTR(scale_out);
    CHECK_CSR();
    if (mode != 0 && mode != 1) return set_error(SPH_ERR_BAD_ARG, "sph_dfsph_features: mode must be 0 or 1");
    if (workspace_bytes < dfsph_ws_bytes(n)) return set_error(SPH_ERR_WORKSPACE, "sph_dfsph_features: workspace too small");
    if (reinterpret_cast<uintptr_t>(workspace) & 255) return set_error(SPH_ERR_BAD_ARG, "sph_dfsph_features: workspace must be 256-byte aligned");
    if (reinterpret_cast<uintptr_t>(feats_out) & 15) return set_error(SPH_ERR_BAD_ARG, "sph_dfsph_features: feats_out must be 16-byte aligned");
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, dvdt, "dvdt"))) return rc;
    char* w = static_cast<char*>(workspace);
    const size_t nb = align256((size_t)n * sizeof(float));
    double* sums3 = reinterpret_cast<double*>(w);
    float* p0 = reinterpret_cast<float*>(w + kCtlBytes);
    float* src = reinterpret_cast<float*>(w + kCtlBytes + nb);
    float* diag = reinterpret_cast<float*>(w + kCtlBytes + 2 * nb);
    cudaError_t e = cudaMemsetAsync(sums3, 0, 3 * sizeof(double), s);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "sph_dfsph_features: memset: %s", cudaGetErrorString(e));
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_dfsph_prep<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, mode, (float)cfg->rest_density, x, H, m, rho, v, dvdt, dt, offs, cnt, list, nullptr, nullptr, p_prev, 1, src, diag, p0)));
    int rb = grid_for(n, 256);
    if (rb > 148 * 4) rb = 148 * 4;
    count_launch();
    k_feature_sums<<<rb, 256, 0, s>>>((int)n, src, diag, cnt, sums3);
    count_launch();
    WSPH_DISPATCH_KDS(*p, (k_features<KF, D, G_LIGHT><<<grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s>>>(
        (int)n, P, (float)cfg->rest_density, x, H, m, rho, src, diag, p_prev, offs, cnt, list, sums3, feats_out, scale_out)));
    return check_launch("sph_dfsph_features");
}

int64_t sph_dfsph_workspace_size(int64_t n, int32_t dim) {
    (void)dim;
    return n < 0 ? -1 : dfsph_ws_bytes(n);
}

int sph_dfsph_div_solve(const SphParams* p, const SphJacobiConfig* cfg, int64_t n, const float* x, const float* H, const float* m,
                        const float* rho, const float* v, const float* dvdt, const float* p_init, const float* dt,
                        const int32_t* offs, const int32_t* cnt, const int32_t* list, void* workspace, int64_t workspace_bytes,
                        float* p_out, float* accel_out, float* history, int32_t* iterations, int32_t* status, void* stream) {
    return dfsph_solve(0, p, cfg, n, x, H, m, rho, v, dvdt, p_init, dt, offs, cnt, list, workspace, workspace_bytes, p_out,
                       accel_out, history, iterations, status, stream);
}

int64_t sph_dfsph_gradient_bytes(int64_t n, int64_t entries, int32_t dim) {
    return n < 0 || entries < 0 || dim < 1 || dim > 3 ? -1 : dfsph_grad_bytes(n, entries, dim);
}

int sph_dfsph_solve_cached(int32_t mode, const SphParams* p, const SphJacobiConfig* cfg, int64_t n, int64_t entries, const float* x,
                           const float* H, const float* m, const float* rho, const float* v, const float* dvdt, const float* p_init,
                           const float* dt, const int32_t* offs, const int32_t* cnt, const int32_t* list, void* workspace,
                           int64_t workspace_bytes, void* gradients, int64_t gradient_bytes, float* p_out, float* accel_out,
                           float* history, int32_t* iterations, int32_t* status, void* stream) {
    if (mode != 0 && mode != 1) return set_error(SPH_ERR_BAD_ARG, "sph_dfsph_solve_cached: mode must be 0 or 1");
    if (n > 0) WSPH_CHECK_PTR(gradients);
    return dfsph_solve(mode, p, cfg, n, x, H, m, rho, v, dvdt, p_init, dt, offs, cnt, list, workspace, workspace_bytes, p_out,
                       accel_out, history, iterations, status, stream, entries, gradients, gradient_bytes);
}

int sph_dfsph_density_solve(const SphParams* p, const SphJacobiConfig* cfg, int64_t n, const float* x, const float* H,
                            const float* m, const float* rho, const float* v, const float* dvdt, const float* p_init,
                            const float* dt, const int32_t* offs, const int32_t* cnt, const int32_t* list, void* workspace,
                            int64_t workspace_bytes, float* p_out, float* accel_out, float* history, int32_t* iterations,
                            int32_t* status, void* stream) {
    return dfsph_solve(1, p, cfg, n, x, H, m, rho, v, dvdt, p_init, dt, offs, cnt, list, workspace, workspace_bytes, p_out,
                       accel_out, history, iterations, status, stream);
}

}  // extern "C"
