// SPH pair-interaction kernels of the compressible (CRKSPH / CompSPH) hot path.
//
// Layout: G lanes of a warp cooperate on one particle i.  Lane l walks the entries
// b+l, b+l+G, ... of i's neighbour row, so the G lanes read G consecutive entries
// (coalesced index loads and pair-array stores), accumulate per-lane partial sums,
// and reduce them with warp shuffles inside the group.  A row is either a whole Verlet
// row or its interacting prefix (the list builder stores the entries with
// r < max(H_i, H_j) first), which removes the beyond-support entries -- about half of
// a Verlet row -- from every pass that only needs W != 0.  The entry index of a pair
// is its position in the Verlet list in both cases.
//
// Arithmetic restates the reference (file:line at each kernel); divisions by the
// same quantity are replaced by multiplications with a reciprocal, so results
// differ from the CPU oracle by rounding only.
//
// In 2D the passes are bound by issue slots, in 3D by L1.  Taking the minimum image with
// one comparison (pair_vec), square roots and reciprocals as approximation plus Newton step
// (sqrt_newton, rcp_newton), the factors of H_i out of the sums and skipping entries outside
// the support took, per launch at 262,144 particles in 2D, the adaptive support from 76 to
// 52 us, the CRK factors from 75 to 60 us, the velocity gradient from 93 to 78 us, the row
// rewrite from 98 to 82 us and the Cullen switch from 104 to 94 us; errors against 64 bits
// are those of before within 2 per cent (5 in single sums; geometric mean of 120 random sets).
#include <cuda.h>
#include <cuda_runtime.h>
#include <cfloat>
#include <atomic>
#include <mutex>
#include "sph_pair_common.cuh"
#include "sph_pinv.cuh"

namespace wsph {

// ---------------------------------------------------------------- density (modules/density/density.py:16-28)
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_density(int n, int mode, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
          const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
          float* __restrict__ rho) {
    pdl_entry();
    Grp<G> g(n);
    float s = 0.f;
    if (g.valid) {
        Vec<D> xi = load_vec<D>(x, g.i);
        float Hi = H[g.i];
        int b = offs[g.i], e = b + cnt[g.i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            Vec<D> xij = dist_vec<D>(xi, xj, P.dom);
            float r = safe_sqrt(dot<D>(xij, xij));
            s += __ldg(m + j) * kernelW_mode<KF, D>(r, Hi, __ldg(H + j), mode);
        }
    }
    s = gsum<G>(s);
    if (g.valid && g.lane == 0) rho[g.i] = s;
}

// ---------------------------------------------------------------- adaptive support
// h(V) of utils/support.py:24-44 (volumeToSupportHelper)
template <int D> __device__ __forceinline__ float volume_to_support(float V, float nH) {
    if constexpr (D == 1) return nH * V / 2.f;
    else if constexpr (D == 2) return sqrtf(nH * V / 3.14159265358979f);
    else return powf(nH * V / 3.14159265358979f * 3.f / 4.f, 1.f / 3.f);
}

// One Newton iteration of modules/adaptiveSupport/optimalSupportMonaghan.py:87-125
// with Omega of modules/adaptiveSupport/wp_omega.py:40-60 (gather support).
// The neighbours' positions and masses come packed in one 16-byte word each (xm: sph_pack_xh of
// the masses) or, with PK false, from x and m.
template <int KF, int D, int G, bool PK>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_adaptive_h(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
             const float4* __restrict__ xm,
             const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
             const float* __restrict__ hb, float* __restrict__ rho_out, float* __restrict__ H_out, float* __restrict__ ratio) {
    pdl_entry();
    Grp<G> g(n);
    float rs = 0.f, ds = 0.f, Hi = 1.f, invHi = 1.f;
    if (g.valid) {
        Vec<D> xi = load_vec<D>(x, g.i);
        Hi = H[g.i];
        invHi = 1.f / Hi;
        int b = offs[g.i], e = b + cnt[g.i];
        typename PairPipe<D, PK>::T rp(list, PairPipe<D, PK>::src(x, xm), b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j;
            Vec<D> xj;
            float mj_ahead = 0.f;
            if constexpr (PK) {
                float4 t;
                rp.take(q, j, t);
                xj = vec_of_word<D>(t);
                mj_ahead = support_of<D>(t);
            } else {
                rp.take(q, j, xj);
                // the mass ahead of the kernel evaluation in 1D and 2D; in 3D most Verlet entries
                // lie outside the support (the load is skipped for them)
                if (D < 3) mj_ahead = __ldg(m + j);
            }
            // W = C / H^d k(q), dW/dH = -C / H^(d+1) (d k - q^2 p): the factors of H_i are taken out of
            // the sums
            const Vec<D> xij = pair_vec<D>(xi, xj, P.dom);
            const float q1 = sqrt_newton(dot<D>(xij, xij)) * invHi;
            if (!(q1 < 1.f)) continue;
            float k, p;
            kernel_kp<KF, D>(q1, k, p);
            const float mj = PK || D < 3 ? mj_ahead : __ldg(m + j);
            rs += mj * k;
            ds += mj * ((float)D * k - q1 * q1 * p);
        }
    }
    const float cH = KernelTraits<KF, D>::C * ipow<D>(invHi);
    rs = cH * gsum<G>(rs);
    ds = -cH * invHi * gsum<G>(ds);
    if (!g.valid || g.lane != 0) return;
    float rho = rs;
    float safe_rho = isfinite(rho) ? fmaxf(rho, 1e-12f) : 1.f;
    float Fv = Hi - volume_to_support<D>(m[g.i] / safe_rho, P.target_neighbors);
    float dh_drho = -Hi / (rho * (float)D);
    float omega = 1.f - dh_drho * ds;
    if (!isfinite(omega)) omega = 0.f;
    float step = Fv / (omega + 1e-6f);
    if (!isfinite(step)) step = 0.f;
    float hn = Hi - step;
    if (!isfinite(hn)) hn = Hi;
    hn = fminf(fmaxf(hn, hb[0] * 0.25f), hb[1] * 4.f);
    rho_out[g.i] = rho;
    H_out[g.i] = hn;
    if (ratio) ratio[g.i] = hn / (Hi + 1e-6f);
}

// ---------------------------------------------------------------- Owen adaptive support
// One iteration of modules/adaptiveSupport/optimalSupportOwen.py:70-108 for every particle:
//   psi0_i  = (sum_j h_i^d W(r_ij, h_i))^(1/d), psi0H_i = (sum_j h_i^(d+1) |grad W(r_ij, h_i)|)^(1/d)
//             (wp_psi0.py:46-98, gather support; h^k taken as 1 / h^-k as there),
//   n_h_i   = the (psiH -> n_h) table linearly interpolated at psi0H_i in FP64 (owenLUT.py:6-12,
//             64-67: index of the last entry <= psi0H, clamped to the table, weight clamped to [0, 1]),
//   s = target / n_h_i, a = 0.4 (1 + s^-3) if s >= 1 else 0.4 (1 + s^2), h_new = (1 - a + a s) h
//             (optimalSupportOwen.py:27-33), clamped to [hbounds[0] / 4, 4 hbounds[1]] (:96);
//   ratio   = h_new / h (:100).
__device__ __forceinline__ float owen_nh(const double* __restrict__ lut_nh, const double* __restrict__ lut_psiH, int nlut, float psiH) {
    const double x = (double)psiH;
    int lo = 0, hi = nlut;                       // first index with lut_psiH[idx] > x
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(lut_psiH + mid) <= x) lo = mid + 1; else hi = mid;
    }
    int il = lo - 1;
    il = il < 0 ? 0 : (il > nlut - 2 ? nlut - 2 : il);
    const double xl = __ldg(lut_psiH + il), xr = __ldg(lut_psiH + il + 1);
    double alpha = (x - xl) / (xr - xl);
    alpha = alpha < 0.0 ? 0.0 : (alpha > 1.0 ? 1.0 : alpha);
    return (float)(__ldg(lut_nh + il) * (1.0 - alpha) + __ldg(lut_nh + il + 1) * alpha);
}

template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_owen(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H,
       const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
       const double* __restrict__ lut_nh, const double* __restrict__ lut_psiH, int nlut, float target,
       const float* __restrict__ hb, float* __restrict__ psi0_out, float* __restrict__ psiH_out,
       float* __restrict__ H_out, float* __restrict__ ratio) {
    pdl_entry();
    Grp<G> g(n);
    float sW = 0.f, sG = 0.f, Hi = 1.f;
    if (g.valid) {
        const int i = g.i;
        Vec<D> xi = load_vec<D>(x, i);
        Hi = H[i];
        const float invHi = 1.f / Hi;
        const float hsW = 1.f / powf(Hi, -(float)D), hsG = 1.f / powf(Hi, -(float)(D + 1));
        int b = offs[i], e = b + cnt[i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            Vec<D> xij = dist_vec<D>(xi, xj, P.dom);
            float r = safe_sqrt(dot<D>(xij, xij));
            float W; Vec<D> gW;
            kWG_inv<KF, D>(xij, r, invHi, W, gW);
            sW += hsW * W;
            sG += hsG * safe_sqrt(dot<D>(gW, gW));
        }
    }
    sW = gsum<G>(sW);
    sG = gsum<G>(sG);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    const float psi0 = powf(sW, 1.f / (float)D), psiH = powf(sG, 1.f / (float)D);
    const float nh = owen_nh(lut_nh, lut_psiH, nlut, psiH);
    const float s = target / nh;
    const float a = s >= 1.f ? 0.4f * (1.f + powf(s, -3.f)) : 0.4f * (1.f + powf(s, 2.f));
    float hn = (1.f - a + a * s) * Hi;
    hn = fminf(fmaxf(hn, hb[0] * 0.25f), hb[1] * 4.f);
    if (psi0_out) psi0_out[i] = psi0;
    if (psiH_out) psiH_out[i] = psiH;
    H_out[i] = hn;
    if (ratio) ratio[i] = hn / Hi;
}

// ---------------------------------------------------------------- CRK volume (scatter support)
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_crk_volume(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H,
             const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
             float* __restrict__ V) {
    pdl_entry();
    Grp<G> g(n);
    float s = 0.f;
    if (g.valid) {
        Vec<D> xi = load_vec<D>(x, g.i);
        int b = offs[g.i], e = b + cnt[g.i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            Vec<D> xij = pair_vec<D>(xi, xj, P.dom);
            s += kW_inv<KF, D>(sqrt_newton(dot<D>(xij, xij)), rcp_newton(__ldg(H + j)));
        }
    }
    s = gsum<G>(s);
    if (g.valid && g.lane == 0) V[g.i] = 1.f / s;
}

// Inverse of a symmetric DxD matrix in double; returns the determinant.
template <int D> __device__ __forceinline__ double inv_sym(const double (&a)[D][D], double (&r)[D][D]) {
    if constexpr (D == 1) {
        r[0][0] = 1.0 / a[0][0];
        return a[0][0];
    } else if constexpr (D == 2) {
        double det = a[0][0] * a[1][1] - a[0][1] * a[1][0];
        double id = 1.0 / det;
        r[0][0] = a[1][1] * id; r[1][1] = a[0][0] * id;
        r[0][1] = -a[0][1] * id; r[1][0] = -a[1][0] * id;
        return det;
    } else {
        double c00 = a[1][1] * a[2][2] - a[1][2] * a[2][1];
        double c01 = a[1][2] * a[2][0] - a[1][0] * a[2][2];
        double c02 = a[1][0] * a[2][1] - a[1][1] * a[2][0];
        double det = a[0][0] * c00 + a[0][1] * c01 + a[0][2] * c02;
        double id = 1.0 / det;
        r[0][0] = c00 * id;
        r[0][1] = (a[0][2] * a[2][1] - a[0][1] * a[2][2]) * id;
        r[0][2] = (a[0][1] * a[1][2] - a[0][2] * a[1][1]) * id;
        r[1][0] = c01 * id;
        r[1][1] = (a[0][0] * a[2][2] - a[0][2] * a[2][0]) * id;
        r[1][2] = (a[0][2] * a[1][0] - a[0][0] * a[1][2]) * id;
        r[2][0] = c02 * id;
        r[2][1] = (a[0][1] * a[2][0] - a[0][0] * a[2][1]) * id;
        r[2][2] = (a[0][0] * a[1][1] - a[0][1] * a[1][0]) * id;
        return det;
    }
}

// CRK moments (FP32 sums, W_ij = W(r_ij, H_j); the derivatives' moments through the symmetric sums
// of s x, s x x and s x x x with gradW = s x_ij: 18 sums instead of 21 in 2D, 33 instead of 44
// in 3D, where the pass went from 1.11 to 0.81 ms at 884,736 particles), FP64 solve for A, B, gradA, gradB
// (Frontiere, Raskin & Owen 2017: linear reproducing conditions) and the CRK density
// sum_j m_j W^R_ij.  A singular second moment (fewer than D+1 effective neighbours)
// falls back to the zeroth-order correction.
template <int D> struct CrkAcc {
    static constexpr int N2 = D * (D + 1) / 2, N3 = D * (D + 1) * (D + 2) / 6;
    // place of the pair u <= c and of the triple u <= c <= w
    static __device__ __forceinline__ constexpr int at2(int u, int c) { return u + c + (D == 3 && u > 0 ? 1 : 0); }
    static __device__ __forceinline__ constexpr int at3(int u, int c, int w) { return u == 0 ? at2(c, w) : u + c + w + (D == 3 ? 3 : 0); }
    float m0, s0, m1[D], s1[D], g1[D], m2[N2], g2[N2], g3[N3];
};
// The ideal-gas EOS of one particle (modules/eos/idealGas.py:16-36), as k_eos computes it:
// fused into the epilogue of the pass that produces the density.
struct EosOut { const float* u; float* A; float* P; float* c; float gamma; };
// Packed gathers of the factors pass: positions with supports in, velocities (v) packed with V and
// m / rho out (fv, and vol in 3D).
struct FactorWords { const float4* xh; const float* v; float4* fv; float* vol; };
__device__ __forceinline__ void eos_ideal_gas_at(int i, const EosOut& eo, float r) {
    const float gamma = eo.gamma, ui = eo.u[i];
    if (eo.c) eo.c[i] = sqrtf(fabsf(ui) * gamma * (gamma - 1.f));
    if (eo.P) eo.P[i] = (gamma - 1.f) * r * ui;
    if (eo.A) eo.A[i] = ui * (gamma - 1.f) * powf(r, 1.f - gamma);
}

template <int KF, int D, int G, bool PK>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_crk_factors(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
              const float* __restrict__ V, const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt,
              const int32_t* __restrict__ list, float* __restrict__ Aout, float* __restrict__ Bout,
              float* __restrict__ gAout, float* __restrict__ gBout, float* __restrict__ rho_out, EosOut eo, FactorWords fw) {
    pdl_entry();
    Grp<G> g(n);
    CrkAcc<D> a;
    {
        float* f = reinterpret_cast<float*>(&a);
        #pragma unroll
        for (int q = 0; q < (int)(sizeof(CrkAcc<D>) / 4); ++q) f[q] = 0.f;
    }
    if (g.valid) {
        const Vec<D> xi = PK ? vec_of_word<D>(__ldg(fw.xh + g.i)) : load_vec<D>(x, g.i);
        int b = offs[g.i], e = b + cnt[g.i];
        typename PairPipe<D, PK>::T rp(list, PairPipe<D, PK>::src(x, fw.xh), b + g.lane, e, G);
        float Vn = __ldg(V + rp.j1), mn = __ldg(m + rp.j1);
        for (int q = b + g.lane; q < e; q += G) {
            int j;
            Vec<D> xj;
            float invHj;
            if constexpr (PK) {
                float4 t; rp.take(q, j, t);
                xj = vec_of_word<D>(t);
                invHj = inv_support_of<D>(t);
            } else {
                rp.take(q, j, xj);
                invHj = rcp_newton(__ldg(H + j));
            }
            const float Vj = Vn, mj = mn;
            Vn = __ldg(V + rp.j1);
            mn = __ldg(m + rp.j1);
            const Vec<D> xij = pair_vec<D>(xi, xj, P.dom);
            const float q1 = sqrt_newton(dot<D>(xij, xij)) * invHj;
            if (!(q1 < 1.f)) continue;
            float k, p;
            kernel_kp<KF, D>(q1, k, p);
            const float cH = KernelTraits<KF, D>::C * ipow<D>(invHj);
            const float W = cH * k, VW = Vj * W, mW = mj * W, Vs = -Vj * (cH * p * (invHj * invHj));   // V_j gradW = Vs x_ij
            a.m0 += VW;
            a.s0 += mW;
            #pragma unroll
            for (int u = 0; u < D; ++u) {
                const float Wx = VW * xij.v[u], gx = Vs * xij.v[u];
                a.m1[u] += Wx;
                a.s1[u] += mW * xij.v[u];
                a.g1[u] += gx;
                #pragma unroll
                for (int c = u; c < D; ++c) {
                    const float gxx = gx * xij.v[c];
                    a.m2[a.at2(u, c)] += Wx * xij.v[c];
                    a.g2[a.at2(u, c)] += u == c ? gxx + VW : gxx;
                    #pragma unroll
                    for (int w = c; w < D; ++w) a.g3[a.at3(u, c, w)] += gxx * xij.v[w];
                }
            }
        }
    }
    {
        float* f = reinterpret_cast<float*>(&a);
        #pragma unroll
        for (int q = 0; q < (int)(sizeof(CrkAcc<D>) / 4); ++q) f[q] = gsum<G>(f[q]);
    }
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    // The moments of the derivatives from the symmetric sums g1 = sum Vs x, g2 = sum (Vs x x + delta VW) and
    // g3 = sum Vs x x x (gradW = s x_ij): with m1,
    //   dm0_w = g1_w,  dm1 = g2,  dm2_ucw = g3_ucw + delta_uw m1_c + delta_cw m1_u
    // The diagonal's two parts almost cancel: added up apart they cost gradB 12 % more error.
    double M2[D][D], Mi[D][D], G2[D][D], G3[D][D][D], tr = 0.0;
    #pragma unroll
    for (int u = 0; u < D; ++u) {
        #pragma unroll
        for (int c = u; c < D; ++c) {
            M2[u][c] = M2[c][u] = (double)a.m2[a.at2(u, c)];
            G2[u][c] = G2[c][u] = (double)a.g2[a.at2(u, c)];
            #pragma unroll
            for (int w = c; w < D; ++w) {
                const double t = (double)a.g3[a.at3(u, c, w)];
                G3[u][c][w] = t; G3[u][w][c] = t; G3[c][u][w] = t; G3[c][w][u] = t; G3[w][u][c] = t; G3[w][c][u] = t;
            }
        }
        tr += (double)a.m2[a.at2(u, u)];
    }
    auto dm2 = [&](int u, int c, int w) { return G3[u][c][w] + (u == w ? (double)a.m1[c] : 0.0) + (c == w ? (double)a.m1[u] : 0.0); };
    double det = inv_sym<D>(M2, Mi);
    double sc = tr / D, sD = sc;
    #pragma unroll
    for (int u = 1; u < D; ++u) sD *= sc;
    bool ok = isfinite(det) && fabs(det) > 1e-10 * fabs(sD) && a.m0 > 0.f;
    double A, Bv[D], gA[D], gB[D][D];
    if (ok) {
        double mb = a.m0;
        #pragma unroll
        for (int u = 0; u < D; ++u) {
            double t = 0.0;
            #pragma unroll
            for (int c = 0; c < D; ++c) t -= Mi[u][c] * (double)a.m1[c];
            Bv[u] = t;
        }
        #pragma unroll
        for (int u = 0; u < D; ++u) mb += (double)a.m1[u] * Bv[u];
        A = 1.0 / mb;
        #pragma unroll
        for (int w = 0; w < D; ++w) {
            double rhs[D];
            #pragma unroll
            for (int u = 0; u < D; ++u) {
                double t = G2[u][w];
                #pragma unroll
                for (int c = 0; c < D; ++c) t += dm2(u, c, w) * Bv[c];
                rhs[u] = t;
            }
            #pragma unroll
            for (int u = 0; u < D; ++u) {
                double t = 0.0;
                #pragma unroll
                for (int c = 0; c < D; ++c) t -= Mi[u][c] * rhs[c];
                gB[u][w] = t;
            }
        }
        #pragma unroll
        for (int w = 0; w < D; ++w) {
            double t = (double)a.g1[w];
            #pragma unroll
            for (int u = 0; u < D; ++u) t += G2[u][w] * Bv[u] + (double)a.m1[u] * gB[u][w];
            gA[w] = -A * A * t;
        }
    } else {
        double m0d = (double)a.m0;
        A = 1.0 / m0d;
        #pragma unroll
        for (int u = 0; u < D; ++u) {
            Bv[u] = 0.0;
            gA[u] = -(double)a.g1[u] / (m0d * m0d);
            #pragma unroll
            for (int c = 0; c < D; ++c) gB[u][c] = 0.0;
        }
    }
    double rho = (double)a.s0;
    #pragma unroll
    for (int u = 0; u < D; ++u) rho += Bv[u] * (double)a.s1[u];
    rho *= A;
    Aout[i] = (float)A;
    #pragma unroll
    for (int u = 0; u < D; ++u) {
        Bout[(size_t)i * D + u] = (float)Bv[u];
        gAout[(size_t)i * D + u] = (float)gA[u];
        #pragma unroll
        for (int c = 0; c < D; ++c) gBout[(size_t)i * D * D + u * D + c] = (float)gB[u][c];
    }
    if (rho_out) rho_out[i] = (float)rho;
    if (eo.u) eos_ideal_gas_at(i, eo, (float)rho);
    if constexpr (PK) {
        const float vol = m[i] / (float)rho;
        fw.fv[i] = make_flow<D>(load_vec<D>(fw.v, i), V[i], vol);
        if (D == 3) fw.vol[i] = vol;
    }
}

// ---------------------------------------------------------------- EOS (modules/eos/idealGas.py:16-36)
__global__ void k_eos(int n, float gamma, const float* __restrict__ u, const float* __restrict__ rho,
                      float* __restrict__ Aout, float* __restrict__ Pout, float* __restrict__ cout) {
    pdl_entry();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float ui = u[i], r = rho[i];
    if (cout) cout[i] = sqrtf(fabsf(ui) * gamma * (gamma - 1.f));
    if (Pout) Pout[i] = (gamma - 1.f) * r * ui;
    if (Aout) Aout[i] = ui * (gamma - 1.f) * powf(r, 1.f - gamma);
}

// ---------------------------------------------------------------- CRK velocity gradient (+ Cullen div, v_sig)
// schemes/crkSPH.py:158-172 (difference form, scatter support, CRK kernel, .mT),
// CullenDehnen2010.py:246-257 (super-symmetric divergence), wp_vsig.py:55-90.
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_grad_v(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
         const float* __restrict__ rho, const float* __restrict__ V, const float* __restrict__ A, const float* __restrict__ B,
         const float* __restrict__ gA, const float* __restrict__ gB, const float* __restrict__ v, const float* __restrict__ c,
         const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
         float* __restrict__ DvDx, float* __restrict__ drhodt, float* __restrict__ div_out, float* __restrict__ vsig_out) {
    pdl_entry();
    Grp<G> g(n);
    const bool want_div = div_out != nullptr, want_vs = vsig_out != nullptr;
    Mat<D> Gm = mzero<D>();
    float div = 0.f, vsig = 0.f;
    if (g.valid) {
        const int i = g.i;
        Vec<D> xi = load_vec<D>(x, i), vi = load_vec<D>(v, i);
        float Hi = H[i], Ai = A[i];
        const float invHi = rcp_newton(Hi);
        Vec<D> Bi = load_vec<D>(B, i), gAi = load_vec<D>(gA, i);
        Mat<D> gBi = load_mat<D>(gB, i);
        float ci = want_vs ? c[i] : 0.f;
        int b = offs[i], e = b + cnt[i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            const float Hj = __ldg(H + j), Vj = __ldg(V + j);   // gathers issued together
            const float mj = want_div ? __ldg(m + j) : 0.f, rhoj = want_div ? __ldg(rho + j) : 1.f;
            const Vec<D> vj = load_vec<D>(v, j);
            Vec<D> xij = pair_vec<D>(xi, xj, P.dom);
            const float r = sqrt_newton(dot<D>(xij, xij)), invHj = rcp_newton(Hj);
            float W, sW;
            if (kWS_inv<KF, D>(r, invHj, W, sW)) {
                Vec<D> gR = crk_grad_s<D>(xij, W, sW, Ai, Bi, gAi, gBi);
                #pragma unroll
                for (int a = 0; a < D; ++a) {
                    float dv = Vj * (vj.v[a] - vi.v[a]);
                    #pragma unroll
                    for (int w = 0; w < D; ++w) Gm.m[a][w] += dv * gR.v[w];
                }
            }
            float Hs = wmax(Hi, Hj);
            float W2, s2;
            if (want_div && kWS_inv<KF, D>(r, fminf(invHi, invHj), W2, s2)) {
                float s = 0.f;
                #pragma unroll
                for (int a = 0; a < D; ++a) s += (vj.v[a] - vi.v[a]) * xij.v[a];
                div += mj * rcp_newton(rhoj) * (s2 * s);
            }
            if (want_vs && r < P.verlet_scale * Hs) {
                float mu = 0.f;
                #pragma unroll
                for (int a = 0; a < D; ++a) mu += (vi.v[a] - vj.v[a]) * xij.v[a];
                mu = mu / (r + 1e-14f * Hi);
                float vsv = 0.5f * (ci + __ldg(c + j)) - mu;
                if (mu > 0.f) vsv = 0.f;
                vsig = wmax(vsig, vsv);
            }
        }
    }
    #pragma unroll
    for (int a = 0; a < D; ++a)
        #pragma unroll
        for (int w = 0; w < D; ++w) Gm.m[a][w] = gsum<G>(Gm.m[a][w]);
    if (want_div) div = gsum<G>(div);
    if (want_vs) vsig = gmaxw<G>(vsig);
    if (!g.valid || g.lane != 0) return;
    store_mat<D>(DvDx, g.i, Gm);
    if (drhodt) {
        float tr = Gm.m[0][0];
        #pragma unroll
        for (int a = 1; a < D; ++a) tr += Gm.m[a][a];
        drhodt[g.i] = -tr * rho[g.i];
    }
    if (want_div) div_out[g.i] = div;
    if (want_vs) vsig_out[g.i] = fabsf(vsig);
}

// ---------------------------------------------------------------- Cullen-Dehnen switch
// R (CullenDehnen2010.py:121-164, gather interpolation of rho_j sgn(div_j) / rho_j * m_j),
// v_sig over the Verlet set when not supplied (wp_vsig.py:55-90), Xi (:166-191) and the
// alpha / alpha0 update (:281-314).
__device__ __forceinline__ float cullen_alpha(const DevParams& P, float Hi, float R, float vs, float dv, float dv_prev, float a0, float dt) {
    float omr = 1.f - R;
    float omr2 = omr * omr;
    float nom = P.beta_xi * (omr2 * omr2) * dv;
    float Xi = P.limit_xi ? (nom * nom + 1e-14f * Hi) / (nom * nom + 0.f + 1e-14f * Hi)
                          : (nom * nom) / (nom * nom + 0.f + 1e-14f * Hi);
    float ddiv = (dv - dv_prev) / dt;
    float Ai = Xi * fmaxf(-ddiv, 0.f);
    float scaling = Hi * Hi * Ai / (vs * vs + Hi * Hi * Ai + 1e-14f * Hi);
    float alphas = fminf(fmaxf(P.alpha_max * scaling, P.alpha_min), P.alpha_max);
    float tau = Hi * (1.f / P.kxi) / (2.f * 0.05f * vs);
    float adot = (alphas - a0) / tau;
    a0 = alphas > a0 ? alphas : a0;
    a0 = alphas < a0 ? a0 + adot * dt : a0;
    return fminf(fmaxf(a0, P.alpha_min), P.alpha_max);
}

template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_cullen(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
         const float* __restrict__ rho, const float* __restrict__ div, const float* __restrict__ div_prev,
         const float* __restrict__ vsig_in, const float* __restrict__ v, const float* __restrict__ c,
         const float* __restrict__ alpha0_prev, const float* __restrict__ dtp,
         const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
         float* __restrict__ alpha_out, float* __restrict__ R_out, float* __restrict__ vsig_out) {
    pdl_entry();
    Grp<G> g(n);
    const bool want_vs = vsig_in == nullptr;
    float s = 0.f, vsig = 0.f;
    float Hi = 1.f;
    if (g.valid) {
        const int i = g.i;
        Vec<D> xi = load_vec<D>(x, i);
        Hi = H[i];
        const float invHi = 1.f / Hi;
        Vec<D> vi = want_vs ? load_vec<D>(v, i) : vzero<D>();
        float ci = want_vs ? c[i] : 0.f;
        int b = offs[i], e = b + cnt[i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            // every gather of the entry issued together, ahead of the tests that select them;
            // in 3D, where about two thirds of a Verlet row lie outside the support, the
            // divergence and the mass are loaded only for the entries inside it (measured:
            // 11.3 against 12.8 ms per step at 128^3; in 2D loading them ahead wins)
            const float dj_ahead = D < 3 ? __ldg(div + j) : 0.f, mj_ahead = D < 3 ? __ldg(m + j) : 0.f;
            const float Hj = want_vs ? __ldg(H + j) : 0.f, cj = want_vs ? __ldg(c + j) : 0.f;
            const Vec<D> vj = want_vs ? load_vec<D>(v, j) : vzero<D>();
            Vec<D> xij = pair_vec<D>(xi, xj, P.dom);
            float r = sqrt_newton(dot<D>(xij, xij));
            float W = kW_inv<KF, D>(r, invHi);   // gather support
            if (W != 0.f) {
                const float dj = D < 3 ? dj_ahead : __ldg(div + j), mj = D < 3 ? mj_ahead : __ldg(m + j);
                float sg = dj > 0.f ? 1.f : (dj < 0.f ? -1.f : 0.f);
                s += mj * sg * W;
            }
            if (want_vs) {
                float Hs = wmax(Hi, Hj);
                if (r < P.verlet_scale * Hs) {
                    float mu = 0.f;
                    #pragma unroll
                    for (int a = 0; a < D; ++a) mu += (vi.v[a] - vj.v[a]) * xij.v[a];
                    mu = mu * rcp_newton(r + 1e-14f * Hi);
                    float vsv = 0.5f * (ci + cj) - mu;
                    if (mu > 0.f) vsv = 0.f;
                    vsig = wmax(vsig, vsv);
                }
            }
        }
    }
    s = gsum<G>(s);
    if (want_vs) vsig = gmaxw<G>(vsig);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    float vs = want_vs ? fabsf(vsig) : vsig_in[i];
    if (want_vs && vsig_out) vsig_out[i] = vs;
    float rhoi = rho[i];
    float R = 1.f / rhoi * s;
    alpha_out[i] = cullen_alpha(P, Hi, R, vs, div[i], div_prev[i], alpha0_prev[i], *dtp);
    if (R_out) R_out[i] = R;
}

// ---------------------------------------------------------------- packed velocity gradient and Cullen switch
// k_grad_v and k_cullen over packed words: two 16-byte gathers per entry (a scalar more in 3D)
// instead of 7 to 10 scalar ones, which in 3D is what L1 is spent on: at 884,736 particles with
// 128 neighbours the gradient went from 1.36 to 0.69 ms, the switch from 2.56 to 1.13 ms and the
// row rewrite from 1.32 to 0.85 ms; at 262,144 in 2D from 78, 94 and 82 to 63, 77 and 79 us.
template <int D>
__global__ void k_pack_xh(int n, const float* __restrict__ x, const float* __restrict__ H, float4* __restrict__ xh) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) xh[i] = make_xh<D>(load_vec<D>(x, i), H[i]);
}

template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_grad_v_packed(int n, DevParams P, const float4* __restrict__ xh, const float4* __restrict__ fv, const float* __restrict__ volume,
                const float* __restrict__ m, const float* __restrict__ rho, const float* __restrict__ c, const float* __restrict__ A,
                const float* __restrict__ B, const float* __restrict__ gA, const float* __restrict__ gB,
                const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
                float* __restrict__ DvDx, float* __restrict__ drhodt, float* __restrict__ divergence_out, float* __restrict__ div_out,
                float4* __restrict__ fc, float* __restrict__ msgn) {
    pdl_entry();
    Grp<G> g(n);
    const bool want_div = div_out != nullptr;
    Mat<D> Gm = mzero<D>();
    float div = 0.f;
    if (g.valid) {
        const int i = g.i;
        const float4 ti = __ldg(xh + i);
        const Vec<D> xi = vec_of_word<D>(ti), vi = vec_of_word<D>(__ldg(fv + i));
        const float invHi = inv_support_of<D>(ti), Ai = A[i];
        const Vec<D> Bi = load_vec<D>(B, i), gAi = load_vec<D>(gA, i);
        const Mat<D> gBi = load_mat<D>(gB, i);
        const int b = offs[i], e = b + cnt[i];
        WordPipe rp(list, xh, b + g.lane, e, G);
        float4 fn = __ldg(fv + rp.j1);         // 3D: a second word ahead (0.68 -> 0.67 ms; 2D: 65 -> 67 us)
        for (int q = b + g.lane; q < e; q += G) {
            int j;
            float4 t;
            rp.take(q, j, t);
            const float4 f = D == 3 ? fn : __ldg(fv + j);
            if (D == 3) fn = __ldg(fv + rp.j1);
            const float vol3 = D == 3 && want_div ? __ldg(volume + j) : 0.f;
            const Vec<D> xij = pair_vec<D>(xi, vec_of_word<D>(t), P.dom), vj = vec_of_word<D>(f);
            const float r = sqrt_newton(dot<D>(xij, xij)), invHj = inv_support_of<D>(t);
            Vec<D> dv;
            #pragma unroll
            for (int a = 0; a < D; ++a) dv.v[a] = vj.v[a] - vi.v[a];
            float W, s;
            if (kWS_inv<KF, D>(r, invHj, W, s)) {
                const Vec<D> gR = crk_grad_s<D>(xij, W, s, Ai, Bi, gAi, gBi);
                const float Vj = D == 3 ? f.w : f.z;
                #pragma unroll
                for (int a = 0; a < D; ++a) {
                    const float dVv = Vj * dv.v[a];
                    #pragma unroll
                    for (int w = 0; w < D; ++w) Gm.m[a][w] += dVv * gR.v[w];
                }
            }
            float W2, s2;
            if (want_div && kWS_inv<KF, D>(r, fminf(invHi, invHj), W2, s2)) div += (D == 3 ? vol3 : f.w) * (s2 * dot<D>(dv, xij));
        }
    }
    #pragma unroll
    for (int a = 0; a < D; ++a)
        #pragma unroll
        for (int w = 0; w < D; ++w) Gm.m[a][w] = gsum<G>(Gm.m[a][w]);
    if (want_div) div = gsum<G>(div);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    store_mat<D>(DvDx, i, Gm);
    float tr = Gm.m[0][0];
    #pragma unroll
    for (int a = 1; a < D; ++a) tr += Gm.m[a][a];
    const float rhoi = rho[i], dr = -tr * rhoi;
    drhodt[i] = dr;
    if (divergence_out) divergence_out[i] = -dr / rhoi;
    if (want_div) {
        div_out[i] = div;
        const float ms = m[i] * (div > 0.f ? 1.f : (div < 0.f ? -1.f : 0.f));
        fc[i] = make_flow<D>(vec_of_word<D>(__ldg(fv + i)), c[i], ms);
        if (D == 3) msgn[i] = ms;
    }
}

template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_cullen_packed(int n, DevParams P, const float4* __restrict__ xh, const float4* __restrict__ fc, const float* __restrict__ msgn,
                const float* __restrict__ rho, const float* __restrict__ div, const float* __restrict__ div_prev,
                const float* __restrict__ alpha0_prev, const float* __restrict__ dtp, const int32_t* __restrict__ offs,
                const int32_t* __restrict__ cnt, const int32_t* __restrict__ list, float* __restrict__ alpha_out) {
    pdl_entry();
    Grp<G> g(n);
    float s = 0.f, vsig = 0.f, Hi = 1.f;
    if (g.valid) {
        const int i = g.i;
        const float4 ti = __ldg(xh + i), fi = __ldg(fc + i);
        const Vec<D> xi = vec_of_word<D>(ti), vi = vec_of_word<D>(fi);
        Hi = support_of<D>(ti);
        const float invHi = inv_support_of<D>(ti), ci = D == 3 ? fi.w : fi.z;
        const int b = offs[i], e = b + cnt[i];
        WordPipe rp(list, xh, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j;
            float4 t;
            rp.take(q, j, t);
            const float4 f = __ldg(fc + j);
            const Vec<D> xij = pair_vec<D>(xi, vec_of_word<D>(t), P.dom), vj = vec_of_word<D>(f);
            const float r = sqrt_newton(dot<D>(xij, xij)), q1 = r * invHi;
            if (q1 < 1.f) {
                float k, p;
                kernel_kp<KF, D>(q1, k, p);
                s += (D == 3 ? __ldg(msgn + j) : f.w) * k;
            }
            if (r < P.verlet_scale * wmax(Hi, support_of<D>(t))) {
                float mu = 0.f;
                #pragma unroll
                for (int a = 0; a < D; ++a) mu += (vi.v[a] - vj.v[a]) * xij.v[a];
                mu = mu * rcp_newton(r + 1e-14f * Hi);
                float vsv = 0.5f * (ci + (D == 3 ? f.w : f.z)) - mu;
                if (mu > 0.f) vsv = 0.f;
                vsig = wmax(vsig, vsv);
            }
        }
        s *= KernelTraits<KF, D>::C * ipow<D>(invHi);
    }
    s = gsum<G>(s);
    vsig = gmaxw<G>(vsig);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    alpha_out[i] = cullen_alpha(P, Hi, 1.f / rho[i] * s, fabsf(vsig), div[i], div_prev[i], alpha0_prev[i], *dtp);
}

// ---------------------------------------------------------------- Cullen-Hopkins switch
// modules/shockCapturing/CullenHopkins.py:7-45 (computeHopkinsTerms): the gather difference
// gradient V_i = sum_j m_j/rho_j (v_j - v_i) (x) grad W(r_ij, H_i) (computeShearTensor,
// common.py:41-85), its trace (the divergence) and |S|^2 = tr(S S^T) of the traceless
// symmetric part S.  With correctVelocityGradient the same pass accumulates the moment
// matrix M_i = -sum_j m_j x_ij (x) grad W(r_ij, H_i) (common.py:10-25, wp_computeM.py:55-86)
// and the gradient becomes pinv(M_i) V_i (common.py:76-78).
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_hopkins_grad(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
               const float* __restrict__ rho, const float* __restrict__ v,
               const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
               float* __restrict__ div_out, float* __restrict__ shear2_out) {
    pdl_entry();
    Grp<G> g(n);
    Mat<D> Gm = mzero<D>(), Mm = mzero<D>();
    const bool corr = P.correct_grad_v != 0;
    if (g.valid) {
        const int i = g.i;
        Vec<D> xi = load_vec<D>(x, i), vi = load_vec<D>(v, i);
        const float invHi = 1.f / H[i];
        int b = offs[i], e = b + cnt[i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            Vec<D> xij = dist_vec<D>(xi, xj, P.dom);
            float r = safe_sqrt(dot<D>(xij, xij));
            float W; Vec<D> gW;
            kWG_inv<KF, D>(xij, r, invHi, W, gW);
            if (W == 0.f) continue;
            const float mj = __ldg(m + j);
            const float Vj = mj / __ldg(rho + j);
            Vec<D> vj = load_vec<D>(v, j);
            #pragma unroll
            for (int a = 0; a < D; ++a) {
                const float dv = Vj * (vj.v[a] - vi.v[a]);
                #pragma unroll
                for (int w = 0; w < D; ++w) Gm.m[a][w] += dv * gW.v[w];
            }
            if (corr) {
                #pragma unroll
                for (int a = 0; a < D; ++a)
                    #pragma unroll
                    for (int w = 0; w < D; ++w) Mm.m[a][w] -= mj * xij.v[a] * gW.v[w];
            }
        }
    }
    #pragma unroll
    for (int a = 0; a < D; ++a)
        #pragma unroll
        for (int w = 0; w < D; ++w) Gm.m[a][w] = gsum<G>(Gm.m[a][w]);
    if (corr) {
        #pragma unroll
        for (int a = 0; a < D; ++a)
            #pragma unroll
            for (int w = 0; w < D; ++w) Mm.m[a][w] = gsum<G>(Mm.m[a][w]);
    }
    if (!g.valid || g.lane != 0) return;
    if (corr) {
        double Md[D][D], Pd[D][D];
        #pragma unroll
        for (int a = 0; a < D; ++a)
            #pragma unroll
            for (int w = 0; w < D; ++w) Md[a][w] = (double)Mm.m[a][w];
        pinv_jacobi<D>(Md, Pd, (double)D * (double)FLT_EPSILON);
        Mat<D> C;
        #pragma unroll
        for (int a = 0; a < D; ++a)
            #pragma unroll
            for (int w = 0; w < D; ++w) {
                double acc = 0.0;
                #pragma unroll
                for (int c = 0; c < D; ++c) acc += Pd[a][c] * (double)Gm.m[c][w];
                C.m[a][w] = (float)acc;
            }
        Gm = C;
    }
    float tr = Gm.m[0][0];
    #pragma unroll
    for (int a = 1; a < D; ++a) tr += Gm.m[a][a];
    float s2 = 0.f;
    #pragma unroll
    for (int a = 0; a < D; ++a)
        #pragma unroll
        for (int w = 0; w < D; ++w) {
            float sv = (Gm.m[a][w] + Gm.m[w][a]) / 2.f - (a == w ? tr / (float)D : 0.f);
            s2 += sv * sv;
        }
    div_out[g.i] = tr;
    shear2_out[g.i] = s2;
}

// R (CullenDehnen2010.py:121-164, gather), Xi with the shear term (:166-191) and
// alpha = max(Xi alpha0, alpha_min) (CullenHopkins.py:25).
template <int KF, int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_hopkins_alpha(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
                const float* __restrict__ rho, const float* __restrict__ div, const float* __restrict__ shear2,
                const float* __restrict__ alpha0, const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt,
                const int32_t* __restrict__ list, float* __restrict__ alpha_out, float* __restrict__ R_out) {
    pdl_entry();
    Grp<G> g(n);
    float s = 0.f;
    if (g.valid) {
        const int i = g.i;
        Vec<D> xi = load_vec<D>(x, i);
        const float invHi = 1.f / H[i];
        int b = offs[i], e = b + cnt[i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            Vec<D> xij = dist_vec<D>(xi, xj, P.dom);
            float W = kW_inv<KF, D>(safe_sqrt(dot<D>(xij, xij)), invHi);
            if (W == 0.f) continue;
            float dj = __ldg(div + j);
            float sg = dj > 0.f ? 1.f : (dj < 0.f ? -1.f : 0.f);
            s += __ldg(m + j) * sg * W;
        }
    }
    s = gsum<G>(s);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    const float Hi = H[i];
    const float R = 1.f / rho[i] * s;
    const float omr = 1.f - R, omr2 = omr * omr;
    const float nom = P.beta_xi * (omr2 * omr2) * div[i];
    const float Xi = P.limit_xi ? (nom * nom + 1e-14f * Hi) / (nom * nom + shear2[i] + 1e-14f * Hi)
                                : (nom * nom) / (nom * nom + shear2[i] + 1e-14f * Hi);
    alpha_out[i] = fmaxf(Xi * alpha0[i], P.alpha_min);
    if (R_out) R_out[i] = R;
}

// computeHopkinsUpdate (CullenHopkins.py:48-149): v_sig over the Verlet rows
// (wp_vsig.py:55-90), d(div)/dt = (div - div_prev) / dt, the local alpha_tmp and the
// relaxation of alpha0 towards it.
template <int D, int G>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_hopkins_update(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ v,
                 const float* __restrict__ c, const float* __restrict__ div, const float* __restrict__ div_prev,
                 const float* __restrict__ alpha0, const float* __restrict__ dtp,
                 const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
                 float* __restrict__ alpha0_out, float* __restrict__ vsig_out) {
    pdl_entry();
    Grp<G> g(n);
    float vsig = 0.f;
    if (g.valid) {
        const int i = g.i;
        Vec<D> xi = load_vec<D>(x, i), vi = load_vec<D>(v, i);
        const float Hi = H[i], ci = c[i];
        int b = offs[i], e = b + cnt[i];
        RowPipe<D> rp(list, x, b + g.lane, e, G);
        for (int q = b + g.lane; q < e; q += G) {
            int j; Vec<D> xj; rp.take(q, j, xj);
            Vec<D> xij = dist_vec<D>(xi, xj, P.dom);
            float r = safe_sqrt(dot<D>(xij, xij));
            if (!(r < P.verlet_scale * wmax(Hi, __ldg(H + j)))) continue;
            Vec<D> vj = load_vec<D>(v, j);
            float mu = 0.f;
            #pragma unroll
            for (int a = 0; a < D; ++a) mu += (vi.v[a] - vj.v[a]) * xij.v[a];
            mu = mu / (r + 1e-14f * Hi);
            float vsv = 0.5f * (ci + __ldg(c + j)) - mu;
            if (mu > 0.f) vsv = 0.f;
            vsig = wmax(vsig, vsv);
        }
    }
    vsig = gmaxw<G>(vsig);
    if (!g.valid || g.lane != 0) return;
    const int i = g.i;
    const float vs = fabsf(vsig);
    const float dt = *dtp;
    const float Hi = H[i], ci = c[i], dv = div[i];
    const float f_kern = 1.f / P.kxi;
    const float ddiv = (dv - div_prev[i]) / dt;
    const float ad = fabsf(ddiv);
    const float fh = f_kern * Hi;
    float at = P.alpha_max * ad / (ad + P.beta_c * (ci * ci) / (fh * fh) + 1e-14f);
    if (ddiv > 0.f || dv > 0.f) at = 0.f;
    const float a0 = alpha0[i];
    const float next = at + (a0 - at) * expf(-P.beta_d * dt * vs / (2.f * f_kern * Hi));
    alpha0_out[i] = at >= a0 ? at : next;
    if (vsig_out) vsig_out[i] = vs;
}

// Balsara switch from the velocity gradient (schemes/crkSPH.py:132-133 comment).
template <int D>
__global__ void k_balsara(int n, const float* __restrict__ DvDx, const float* __restrict__ c, float* __restrict__ alpha) {
    pdl_entry();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Mat<D> Gm = load_mat<D>(DvDx, i);
    float dv = Gm.m[0][0];
    for (int a = 1; a < D; ++a) dv += Gm.m[a][a];
    float curl2 = 0.f;
    if constexpr (D == 2) { float w = Gm.m[1][0] - Gm.m[0][1]; curl2 = w * w; }
    if constexpr (D == 3) {
        float w0 = Gm.m[2][1] - Gm.m[1][2], w1 = Gm.m[0][2] - Gm.m[2][0], w2 = Gm.m[1][0] - Gm.m[0][1];
        curl2 = w0 * w0 + w1 * w1 + w2 * w2;
    }
    float ad = fabsf(dv);
    float bal = ad / (ad + sqrtf(curl2) + 1e-4f * c[i]);
    alpha[i] = fminf(fmaxf(bal, 0.f), 1.f);
}

// ---------------------------------------------------------------- CRK accel + dudt
// modules/crk/limiter.py:10-16
__device__ __forceinline__ float limiter_vl(float x) {
    if (x <= 0.f) return 0.f;
    float vL = __fdividef(2.f, 1.f + x);
    return x * vL * vL;
}

// modules/crk/limiter.py:27-86 (quadratic-form Van Leer) from g_i = x_ij.(G_i x_ij) and g_j, whose
// quarters are the reference's (G h).h, h = x_ij / 2.  The limiter's argument min(g_i / g_j, g_j / g_i)
// is the quotient of the smaller by the larger where their signs agree, and not positive where they differ.
__device__ __forceinline__ float van_leer(float gi, float gj) {
    const bool less = fabsf(gi) < fabsf(gj);
    float x = __fdividef(less ? gi : gj, less ? gj : gi);
    if (x != x) x = 1.f;
    return limiter_vl(x);
}

// Zero pairwise outputs of the entries [offs + cnt, offs + vcnt) of a row: the Verlet
// entries after the interacting prefix, which carry no interaction (contiguous stores).
template <int D, int G>
__device__ __forceinline__ void zero_row_tail(int lane, int e, int te, float* __restrict__ ap, float* __restrict__ av) {
    for (int q = e + lane; q < te; q += G) {
        if (ap) store_vec<D>(ap, q, vzero<D>());
        if (av) store_vec<D>(av, q, vzero<D>());
    }
}

// Packed per-particle record of the CRK accel pass: every field a pair reads from
// particle j (and the pass reads from particle i) in one block of R floats, R a multiple
// of 4, so a pair's neighbour gather is R/4 128-bit loads from adjacent sectors instead
// of 2D^2+4D+6 scalar loads from as many arrays (D = 2: 6 loads and 3 sectors instead of
// 22 loads and 22 sectors).  The fields are in the order the pair body first uses them,
// and the body loads them in three groups of 16-byte granules: position and support
// (before the distance test), velocity, gradient, sound speed and pressure (the limiter
// and Q), and the rest (the corrected gradient of W_ji), which keeps fewer of them live.
template <int D> struct CrkRec {
    static constexpr int NS = D * (D + 1) / 2;
    static constexpr int X = 0, H = D, QQ = D + 1, V = D + 2, S = 2 * D + 2, QL = S + NS, P = QL + 1, VOL = P + 1, A = P + 2,
                         C = P + 3, E = C + D, F = E + D, END = F + D * D, R = (END + 3) / 4 * 4;
    static constexpr int K1 = (H + 1 + 3) / 4;      // granules of the first group
    static constexpr int K2 = (P + 1 + 3) / 4;      // ... of the first two groups
    static constexpr int K3 = R / 4;
};
template <int D, int K0, int K1>
__device__ __forceinline__ void rec_granules(const float4* __restrict__ rec, int n, int j, float (&r)[CrkRec<D>::R]) {
    #pragma unroll
    for (int k = K0; k < K1; ++k) {
        float4 t = __ldg(rec + (size_t)k * n + j);
        r[4 * k] = t.x; r[4 * k + 1] = t.y; r[4 * k + 2] = t.z; r[4 * k + 3] = t.w;
    }
}

// The fields of one particle as the accel pass uses them, with what depends on it alone formed once:
//   grad W^R = A (1 + B.x) s x + W (gA (1 + B.x) + A (B + gB^T x)) = s (A + C.x) x + W (E + F x),
//              C = A B, E = gA + A B, F = gA B^T + A gB^T (x = x_ij, grad W = s x)
//   x.(G x)  = S over the products x_a x_b, a <= b (the velocity gradient enters the pass through it alone)
//   rho (-C_l c mu + C_q mu^2) = mu (qq mu - ql), qq = rho C_q, ql = rho C_l c
template <int D> struct CrkPart {
    Vec<D> x, v, C, E;
    Mat<D> F;
    float S[D * (D + 1) / 2];
    float H, V, P, A, qq, ql;
};
template <int D>
__device__ __forceinline__ void crk_part(const DevParams& P, float rho, float c, float A, const Vec<D>& B, const Vec<D>& gA, const Mat<D>& gB,
                                         const Mat<D>& G, CrkPart<D>& o) {
    o.A = A;
    #pragma unroll
    for (int a = 0; a < D; ++a) {
        o.C.v[a] = A * B.v[a];
        o.E.v[a] = gA.v[a] + o.C.v[a];
        #pragma unroll
        for (int b = 0; b < D; ++b) o.F.m[a][b] = gA.v[a] * B.v[b] + A * gB.m[b][a];
    }
    int k = 0;
    #pragma unroll
    for (int a = 0; a < D; ++a)
        #pragma unroll
        for (int b = a; b < D; ++b) o.S[k++] = a == b ? G.m[a][a] : G.m[a][b] + G.m[b][a];
    o.qq = rho * P.C_q;
    o.ql = rho * P.C_l * c;
}
// s (A + C.x) x + W (E + F x)
template <int D> __device__ __forceinline__ Vec<D> crk_part_grad(const CrkPart<D>& p, const Vec<D>& x, float W, float s) {
    const float cx = s * (p.A + dot<D>(p.C, x));
    Vec<D> r;
    #pragma unroll
    for (int g = 0; g < D; ++g) {
        float t = p.E.v[g];
        #pragma unroll
        for (int a = 0; a < D; ++a) t += p.F.m[g][a] * x.v[a];
        r.v[g] = cx * x.v[g] + W * t;
    }
    return r;
}
// Group 1: position and support; group 2: velocity, velocity gradient, viscosity factors and
// pressure; group 3: volume and the corrections.
template <int D> __device__ __forceinline__ void crk_unpack1(const float (&r)[CrkRec<D>::R], CrkPart<D>& o) {
    using L = CrkRec<D>;
    #pragma unroll
    for (int a = 0; a < D; ++a) o.x.v[a] = r[L::X + a];
    o.H = r[L::H];
}
template <int D> __device__ __forceinline__ void crk_unpack2(const float (&r)[CrkRec<D>::R], CrkPart<D>& o) {
    using L = CrkRec<D>;
    #pragma unroll
    for (int a = 0; a < D; ++a) o.v.v[a] = r[L::V + a];
    #pragma unroll
    for (int a = 0; a < L::NS; ++a) o.S[a] = r[L::S + a];
    o.qq = r[L::QQ]; o.ql = r[L::QL]; o.P = r[L::P];
}
template <int D> __device__ __forceinline__ void crk_unpack3(const float (&r)[CrkRec<D>::R], CrkPart<D>& o) {
    using L = CrkRec<D>;
    #pragma unroll
    for (int a = 0; a < D; ++a) { o.C.v[a] = r[L::C + a]; o.E.v[a] = r[L::E + a]; }
    #pragma unroll
    for (int a = 0; a < D * D; ++a) o.F.m[a / D][a % D] = r[L::F + a];
    o.V = r[L::VOL]; o.A = r[L::A];
}

template <int D>
__global__ void k_crk_pack(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ rho,
                           const float* __restrict__ V, const float* __restrict__ A, const float* __restrict__ B,
                           const float* __restrict__ gA, const float* __restrict__ gB, const float* __restrict__ v,
                           const float* __restrict__ c, const float* __restrict__ Pr, const float* __restrict__ DvDx,
                           float* __restrict__ rec) {
    pdl_entry();
    using L = CrkRec<D>;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    CrkPart<D> o;
    o.x = load_vec<D>(x, i);
    o.v = load_vec<D>(v, i);
    o.H = H[i]; o.V = V[i]; o.P = Pr[i];
    crk_part<D>(P, rho[i], c[i], A[i], load_vec<D>(B, i), load_vec<D>(gA, i), load_mat<D>(gB, i), load_mat<D>(DvDx, i), o);
    float r[L::R];
    #pragma unroll
    for (int a = 0; a < D; ++a) { r[L::X + a] = o.x.v[a]; r[L::V + a] = o.v.v[a]; r[L::C + a] = o.C.v[a]; r[L::E + a] = o.E.v[a]; }
    #pragma unroll
    for (int a = 0; a < L::NS; ++a) r[L::S + a] = o.S[a];
    #pragma unroll
    for (int a = 0; a < D * D; ++a) r[L::F + a] = o.F.m[a / D][a % D];
    r[L::H] = o.H; r[L::QQ] = o.qq; r[L::QL] = o.ql; r[L::P] = o.P; r[L::VOL] = o.V; r[L::A] = o.A;
    #pragma unroll
    for (int a = L::END; a < L::R; ++a) r[a] = 0.f;
    float4* dst = reinterpret_cast<float4*>(rec) + i;
    #pragma unroll
    for (int k = 0; k < L::R / 4; ++k) dst[(size_t)k * n] = make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
}

// modules/crk/accel.py:65-250 and modules/crk/dudt.py:62-229 in one pass.  The pair
// body's quotients (Van Leer ratios, 1/H_j, the mu_ij denominators) use the fast FP32
// divide (about 2 ulp): about a tenth of the pass's time, well inside the pass's parity
// tolerance against the oracle's IEEE quotients.  The
// unused computePi_actual calls of the reference (accel.py:143-168, dudt.py:128-153)
// have no effect on the outputs and are not evaluated.  dE/dt = m v.dv/dt + m du/dt
// (schemes/crkSPH.py:330) is written per particle.  Walking the interacting prefix of
// each Verlet row (cnt = interacting counts) with vcnt = the Verlet counts, the
// ap_ij / av_ij entries of the rest of the row are written as zeros.
#ifndef CRK_REC_BLOCKS
#define CRK_REC_BLOCKS 7
#endif
template <int KF, int D, int G, bool REC>
__global__ void __launch_bounds__(PAIR_BLOCK, (D == 3 ? 5 : (REC ? CRK_REC_BLOCKS : 8)))
k_crk_accel_dudt(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const float* __restrict__ m,
                 const float* __restrict__ rho, const float* __restrict__ V, const float* __restrict__ A,
                 const float* __restrict__ B, const float* __restrict__ gA, const float* __restrict__ gB,
                 const float* __restrict__ v, const float* __restrict__ c, const float* __restrict__ Pr,
                 const float* __restrict__ DvDx, const float* __restrict__ rec, const int32_t* __restrict__ offs,
                 const int32_t* __restrict__ cnt, const int32_t* __restrict__ list, const int32_t* __restrict__ vcnt,
                 float* __restrict__ dvdt, float* __restrict__ dudt, float* __restrict__ dEdt, float* __restrict__ ap,
                 float* __restrict__ av) {
    pdl_entry();
    Grp<G> g(n);
    const bool comp = P.kahan != 0;
    KSum acc[D], du;
    #pragma unroll
    for (int a = 0; a < D; ++a) acc[a].init();
    du.init();
    if (g.valid) {
        const int i = g.i;
        CrkPart<D> pi;
        if constexpr (REC) {
            float r[CrkRec<D>::R];
            rec_granules<D, 0, CrkRec<D>::K3>(reinterpret_cast<const float4*>(rec), n, i, r);
            crk_unpack1<D>(r, pi); crk_unpack2<D>(r, pi); crk_unpack3<D>(r, pi);
        } else {
            pi.x = load_vec<D>(x, i); pi.v = load_vec<D>(v, i);
            pi.H = H[i]; pi.V = V[i]; pi.P = Pr[i];
            crk_part<D>(P, rho[i], c[i], A[i], load_vec<D>(B, i), load_vec<D>(gA, i), load_mat<D>(gB, i), load_mat<D>(DvDx, i), pi);
        }
        const float Hi = pi.H, Pi = pi.P;
        const float invHi = 1.f / Hi;
        const float hVi_m = 0.5f * (pi.V / m[i]);
        const float ks = P.kscale;
        const float inv_smooth_i = ks * invHi;   // 1 / (H_i / ks)
        const float sm_i = Hi / ks;
        const float eps_i = 1.0e-7f * sm_i * sm_i;
        int b = offs[i], e = b + cnt[i];
        for (int q = b + g.lane; q < e; q += G) {
            int j, k; entry(list, q, j, k);
            CrkPart<D> pj;
            float rj[CrkRec<D>::R];
            const float4* sj = reinterpret_cast<const float4*>(rec);
            if constexpr (REC) {
                // the first two groups issued together (walked rows are interacting prefixes, so
                // the range test below almost never discards the second)
                rec_granules<D, 0, CrkRec<D>::K2>(sj, n, j, rj);
                crk_unpack1<D>(rj, pj);
            }
            else { pj.x = load_vec<D>(x, j); pj.H = __ldg(H + j); }
            Vec<D> xij = pair_vec<D>(pi.x, pj.x, P.dom);
            float r2 = dot<D>(xij, xij);
            const float Hj = pj.H;
            float Hm = wmax(Hi, Hj);
            if (!(r2 < Hm * Hm)) {
                if (ap) store_vec<D>(ap, k, vzero<D>());
                if (av) store_vec<D>(av, k, vzero<D>());
                continue;
            }
            if constexpr (REC) {
                crk_unpack2<D>(rj, pj);
            } else {
                pj.v = load_vec<D>(v, j);
                pj.P = __ldg(Pr + j);
                pj.V = __ldg(V + j);
                crk_part<D>(P, __ldg(rho + j), __ldg(c + j), __ldg(A + j), load_vec<D>(B, j), load_vec<D>(gA, j), load_mat<D>(gB, j),
                            load_mat<D>(DvDx, j), pj);
            }
            float r = sqrt_newton(r2);
            const float invHj = rcp_newton(Hj);
            const float Pj = pj.P;
            // CRK limiter (limiter.py:89-128), eta measured in supports
            float factor = 1.f;
            if (P.enable_crk_limiter) {
                float eta = r * wmin(invHi, invHj);
                if (eta < P.eta_crit) { float t = (eta - P.eta_crit) / P.eta_fold; factor = expf(-(t * t)); }
            }
            float gi = 0.f, gj = 0.f;
            {
                int u = 0;
                #pragma unroll
                for (int a = 0; a < D; ++a)
                    #pragma unroll
                    for (int b = a; b < D; ++b) {
                        const float xx = xij.v[a] * xij.v[b];
                        gi += pi.S[u] * xx;
                        gj += pj.S[u] * xx;
                        ++u;
                    }
            }
            float phi = 0.f;
            if (P.enable_vanleer) phi = van_leer(gi, gj) * factor;
            if (P.force_vl_off) phi = 0.f;
            if (P.force_vl_on) phi = 1.f;
            phi = wmax(wmin(phi, 1.f), 0.f);
            const float hp = 0.5f * phi;
            // corrected gradients (accel.py:170-187, dudt.py:155-170)
            float Wi, si;
            kWS_inv<KF, D>(r, invHj, Wi, si);
            const Vec<D> gradw_i = crk_part_grad<D>(pi, xij, Wi, si);
            if constexpr (REC) {
                rec_granules<D, CrkRec<D>::K2, CrkRec<D>::K3>(sj, n, j, rj); crk_unpack3<D>(rj, pj);
            }
            Vec<D> xji;
            #pragma unroll
            for (int a = 0; a < D; ++a) xji.v[a] = -xij.v[a];
            float Wj, sj_;
            kWS_inv<KF, D>(r, invHi, Wj, sj_);
            const Vec<D> gradw_j = crk_part_grad<D>(pj, xji, Wj, sj_);
            Vec<D> gij;                            // twice the mean gradient; the half is in w
            #pragma unroll
            for (int a = 0; a < D; ++a) gij.v[a] = gradw_i.v[a] - gradw_j.v[a];
            // mu_ij, mu_ji and Q (accel.py:189-206): eta = x_ij / smoothing length
            const float inv_smooth_j = ks * invHj;
            const float sm_j = Hj / ks;
            const float eps_j = 1.0e-7f * sm_j * sm_j;
            float den_i = r2 * (inv_smooth_i * inv_smooth_i) + eps_i;
            float den_j = r2 * (inv_smooth_j * inv_smooth_j) + eps_j;
            // (v_dot_i - v_dot_j).x_ij with the half gradients taken off (accel.py:137-141; dudt.py:122-126 uses
            // gradV_j . (-x_ij))
            float vx = 0.f;
            #pragma unroll
            for (int a = 0; a < D; ++a) vx += (pi.v.v[a] - pj.v.v[a]) * xij.v[a];
            const float xa = vx - hp * (gi + gj), xd = vx - hp * (gi - gj);
            float idi = __fdividef(inv_smooth_i, den_i), idj = __fdividef(inv_smooth_j, den_j);
            float mia = wmin(0.f, xa * idi), mja = wmin(0.f, xa * idj);
            float mid = wmin(0.f, xd * idi), mjd = wmin(0.f, xd * idj);
            const float Qa = mia * (pi.qq * mia - pi.ql) + mja * (pj.qq * mja - pj.ql);
            const float Qd = mid * (pi.qq * mid - pi.ql) + mjd * (pj.qq * mjd - pj.ql);
            // accel.py:228-249 (mu_ij = 1 there)
            const float w = pj.V * hVi_m, cp = -(Pi + Pj) * w, cv = -Qa * w;   // V_i V_j / (2 m_i)
            Vec<D> pt, vt;
            float dotu = 0.f;
            #pragma unroll
            for (int a = 0; a < D; ++a) {
                pt.v[a] = cp * gij.v[a];
                vt.v[a] = cv * gij.v[a];
                acc[a].add(pt.v[a] + vt.v[a], comp);
                dotu += (pi.v.v[a] - pj.v.v[a]) * gij.v[a];
            }
            if (ap) store_vec<D>(ap, k, pt);
            if (av) store_vec<D>(av, k, vt);
            // dudt.py:208-226
            du.add((Pj + 0.5f * Qd) * dotu * w, comp);
        }
        if (vcnt && (ap || av)) zero_row_tail<D, G>(g.lane, e, b + __ldg(vcnt + i), ap, av);
    }
    float o[D], od;
    #pragma unroll
    for (int a = 0; a < D; ++a) o[a] = gsum<G>(acc[a].s) + gsum<G>(acc[a].c);
    od = gsum<G>(du.s) + gsum<G>(du.c);
    if (!g.valid || g.lane != 0) return;
    Vec<D> ov;
    #pragma unroll
    for (int a = 0; a < D; ++a) ov.v[a] = o[a];
    if (dvdt) store_vec<D>(dvdt, g.i, ov);
    if (dudt) dudt[g.i] = od;
    if (dEdt) {
        const float mi = m[g.i];
        Vec<D> vi;
        if constexpr (REC) {
            #pragma unroll
            for (int a = 0; a < D; ++a) {
                constexpr int V = CrkRec<D>::V;
                vi.v[a] = __ldg(rec + 4 * ((size_t)((V + a) / 4) * n + g.i) + (V + a) % 4);
            }
        } else {
            vi = load_vec<D>(v, g.i);
        }
        dEdt[g.i] = mi * dot<D>(vi, ov) + mi * od;
    }
}

// ---------------------------------------------------------------- energy partition f_ij (modules/compSPH/balance.py:62-154)
__device__ __forceinline__ float sgn0(float x) { return x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f); }

// (v, s) of one particle in a 16-byte word.
template <int D> __device__ __forceinline__ float4 make_vs(const Vec<D>& v, float s) {
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    #pragma unroll
    for (int a = 0; a < D; ++a) w[a] = v.v[a];
    w[D] = s;
    return make_float4(w[0], w[1], w[2], w[3]);
}
// Per-particle prologue: half-step velocity v + dt/2 dv/dt (schemes/crkSPH.py:341) and
// the CRK entropy P / rho^gamma (balance.py:126-127).
template <int D>
__global__ void k_balance_prep(int n, DevParams P, const float* __restrict__ rho, const float* __restrict__ Pr,
                               const float* __restrict__ v, const float* __restrict__ dvdt, const float* __restrict__ dtp,
                               float* __restrict__ vh, float* __restrict__ sarr, float4* __restrict__ words) {
    pdl_entry();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float hdt = 0.5f * (*dtp);
    Vec<D> vi = load_vec<D>(v, i), ai = load_vec<D>(dvdt, i);
    #pragma unroll
    for (int a = 0; a < D; ++a) vi.v[a] = vi.v[a] + hdt * ai.v[a];
    const float s = Pr[i] / powf(rho[i], P.gamma);
    if (words) { words[i] = make_vs<D>(vi, s); return; }
    store_vec<D>(vh, i, vi);
    sarr[i] = s;
}

template <int D, int G, bool PK>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_balance(int n, DevParams P, const float* __restrict__ m, const float* __restrict__ rho, const float* __restrict__ Pr,
          const float* __restrict__ u, const float* __restrict__ vh, const float* __restrict__ sarr, const float* __restrict__ dtp,
          const int32_t* __restrict__ offs, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
          const int32_t* __restrict__ icnt, const float* __restrict__ ap, const float* __restrict__ av, float* __restrict__ fout,
          const float4* __restrict__ words) {
    pdl_entry();
    Grp<G> g(n);
    if (!g.valid) return;
    const int i = g.i;
    const float dt = *dtp;
    const float4 wi = PK ? __ldg(words + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    const Vec<D> vi = PK ? vec_of_word<D>(wi) : load_vec<D>(vh, i);
    const float mi = m[i], rhoi = rho[i], Pi = Pr[i], ui = u[i], si = PK ? word_of(wi, D) : sarr[i];
    const int scheme = P.energy_scheme;
    int b = offs[i], e = b + cnt[i];
    // entries past the interacting prefix carry ap = av = 0, so their dE is 0 (the same
    // value the loads would give) and their pair arrays and half-step velocities are not read
    const int ie = icnt ? b + icnt[i] : e;
    for (int q = b + g.lane; q < e; q += G) {
        int j, k; entry(list, q, j, k);
        // issued with the entry's other gathers
        const float4 wj = PK ? __ldg(words + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float sj_crk = PK ? word_of(wj, D) : (scheme == SPH_ENERGY_CRK ? __ldg(sarr + j) : 0.f);
        float dE = 0.f;
        if (q < ie) {
            const Vec<D> vj = PK ? vec_of_word<D>(wj) : load_vec<D>(vh, j);
            Vec<D> apk = load_vec<D>(ap, k), avk = load_vec<D>(av, k);
            #pragma unroll
            for (int a = 0; a < D; ++a) dE += (vj.v[a] - vi.v[a]) * (apk.v[a] + avk.v[a]);
        }
        dE = mi * dE * dt;
        float f = 0.5f;
        if (scheme == SPH_ENERGY_CRK) {
            const float sj = sj_crk;
            const float smin = wmin(fabsf(si), fabsf(sj)), smax = wmax(fabsf(si), fabsf(sj));
            const bool mB = (dE >= 0.f && si >= sj) || (dE < 0.f && si < sj);
            const bool mC = (dE >= 0.f && si < sj) || (dE < 0.f && si >= sj);
            if (fabsf(si - sj) != 0.f && (mB || mC)) f = (mB ? smin : smax) * rcp_newton(smin + smax + 1.0e-14f);
            f = wmax(0.f, wmin(1.f, f));
        } else if (scheme == SPH_ENERGY_PDV) {
            float rhoj = __ldg(rho + j), Pj = __ldg(Pr + j);
            f = (Pi / (rhoi * rhoi)) / (Pi / (rhoi * rhoi) + Pj / (rhoj * rhoj));
        } else if (scheme == SPH_ENERGY_DIMINISHING) {
            float uji = __ldg(u + j) - ui, un = fabsf(uji);
            f = 0.5f * (1.f + (uji * sgn0(dE)) / (un + 1.f / (1.f + un)));
        } else if (scheme == SPH_ENERGY_MONOTONIC || scheme == SPH_ENERGY_HYBRID) {
            float mj = __ldg(m + j), uj = __ldg(u + j), uji = uj - ui;
            float Aq = dE / (uji + 1.0e-14f);
            float Bq = Aq >= 0.f ? Aq / mi : Aq / mj;
            float t1 = wmax(0.f, sgn0(Bq));
            float t2 = mi / (dE + 1.0e-14f) * ((dE + mi * ui + mj * uj) / (mi + mj) - ui);
            float fm = fabsf(Bq) <= 1.f ? t1 : t2;
            if (scheme == SPH_ENERGY_MONOTONIC) f = fm;
            else {
                float un = fabsf(uji);
                float fsm = 0.5f * (1.f + (uji * sgn0(dE)) / (un + 1.f / (1.f + un)));
                float chi = fabsf(uji) / (fabsf(ui) + fabsf(uj) + 1.0e-14f);
                f = chi * fm + (1.f - chi) * fsm;
            }
        }
        fout[k] = f;
    }
}

// ---------------------------------------------------------------- CFL dt (modules/timestep/compressible.py:18-61)
__global__ void k_cfl_reduce(int n, float gamma, const float* __restrict__ H, const float* __restrict__ u,
                             float* __restrict__ red /* [0]=min H, [1]=max c */) {
    pdl_entry();
    float hmin = __int_as_float(0x7f800000), cmax = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        hmin = fminf(hmin, H[i]);
        cmax = fmaxf(cmax, sqrtf(fabsf(u[i]) * gamma * (gamma - 1.f)));
    }
    hmin = block_reduce(hmin, __int_as_float(0x7f800000), OpMinF());
    cmax = block_reduce(cmax, 0.f, OpMaxF());
    if (threadIdx.x == 0) {
        atomicMin(reinterpret_cast<int*>(red), __float_as_int(hmin));
        atomicMax(reinterpret_cast<int*>(red + 1), __float_as_int(cmax));
    }
}
__global__ void k_cfl_init(float* red) {
    pdl_entry(); red[0] = __int_as_float(0x7f800000); red[1] = 0.f; }
__global__ void k_cfl_final(DevParams P, const float* __restrict__ red, const float* __restrict__ dt_prev, float* __restrict__ dt_out) {
    pdl_entry();
    // min_i cfl*h/(c_i*xi) is attained at max_i c_i (the map c -> cfl*h/(c*xi) is monotone)
    float dt = P.cfl * red[0] / (red[1] * P.kxi);
    dt = fminf(fmaxf(dt, P.min_dt), P.max_dt);
    if (dt_prev) {
        float prev = *dt_prev;
        if (dt > prev) dt = fminf(dt, P.dt_growth * prev);
    }
    *dt_out = dt;
}

// ---------------------------------------------------------------- RK stage combination
struct KPtrs { const float* k[8]; float w[8]; };
__global__ void k_rk_combine(int64_t count, const float* __restrict__ y0, int nk, KPtrs K, const float* __restrict__ dtp,
                             int wrap_dim, DomainF dom, float* __restrict__ y) {
    pdl_entry();
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    float dt = *dtp;
    // explicitly rounded (no FMA) so the CPU oracle reproduces the stage states bit for bit
    float s = 0.f;
    for (int q = 0; q < nk; ++q) s = __fadd_rn(s, __fmul_rn(K.w[q], K.k[q][idx]));
    float val = __fadd_rn(y0[idx], __fmul_rn(dt, s));
    if (wrap_dim > 0) {
        int a = (int)(idx % wrap_dim);
        if (dom.periodic[a]) {
            if (val >= dom.max[a]) val = __fsub_rn(val, dom.L[a]);
            else if (val < dom.min[a]) val = __fadd_rn(val, dom.L[a]);
        }
    }
    y[idx] = val;
}

// Several fields combined in one launch (the integrator's positions, velocities and
// energies of one stage): the same arithmetic as k_rk_combine per element.
constexpr int RKF_MAX = 4;
struct FieldPtrs {
    const float* y0[RKF_MAX];
    float* y[RKF_MAX];
    const float* k[RKF_MAX][8];
    int64_t end[RKF_MAX];        // cumulative element counts
    int wrap[RKF_MAX];
    float w[8];
};
// One row of blocks per field, ITEMS elements per thread with their loads together: with the field found per
// element and the domain indexed through local memory a launch of 1.3 M elements took 25 us against 13 now.
// Below 303,104 elements (8 blocks of 256 per SM) one element per thread fills the chip better.
template <int ITEMS>
__global__ void __launch_bounds__(256)
k_rk_combine_fields(int nk, const __grid_constant__ FieldPtrs F, const float* __restrict__ dtp, const __grid_constant__ DomainF dom) {
    pdl_entry();
    const int f = blockIdx.y;
    const int64_t count = F.end[f] - (f > 0 ? F.end[f - 1] : 0), base = (int64_t)blockIdx.x * (256 * ITEMS) + threadIdx.x;
    if (base >= count) return;
    const float* y0 = F.y0[f];
    const float dt = *dtp;
    float s[ITEMS], y[ITEMS];
    #pragma unroll
    for (int u = 0; u < ITEMS; ++u) { s[u] = 0.f; y[u] = base + 256 * u < count ? y0[base + 256 * u] : 0.f; }
    for (int q = 0; q < nk; ++q) {
        const float* k = F.k[f][q];
        const float w = F.w[q];
        #pragma unroll
        for (int u = 0; u < ITEMS; ++u)
            if (base + 256 * u < count) s[u] = __fadd_rn(s[u], __fmul_rn(w, k[base + 256 * u]));
    }
    const int wd = F.wrap[f];
    #pragma unroll
    for (int u = 0; u < ITEMS; ++u) {
        const int64_t idx = base + 256 * u;
        if (idx >= count) break;
        float val = __fadd_rn(y[u], __fmul_rn(dt, s[u]));
        if (wd > 0) {
            const int a = wd == 1 ? 0 : (wd == 2 ? (int)(idx & 1) : (int)(idx % 3));
            if (dom.periodic[a]) {
                if (val >= dom.max[a]) val = __fsub_rn(val, dom.L[a]);
                else if (val < dom.min[a]) val = __fadd_rn(val, dom.L[a]);
            }
        }
        F.y[f][idx] = val;
    }
}

// ---------------------------------------------------------------- compatible energy
// modules/compSPH/multistep.py:52-94 and systems/compSPH.py:100-111
struct StagePtrs {
    const float* dvdt[8];
    const int32_t* offs[8];
    const int32_t* cnt[8];
    const int32_t* list[8];
    const float* f[8];
    const float* ap[8];
    const float* av[8];
    float w[8];
};
template <int D>
__global__ void k_vhalf(int n, int ns, StagePtrs S, const float* __restrict__ dtp, const float* __restrict__ v0, float* __restrict__ vh) {
    pdl_entry();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float dt = *dtp;
    #pragma unroll
    for (int a = 0; a < D; ++a) {
        float fa = 0.f;
        for (int s = 0; s < ns; ++s) fa += S.w[s] * S.dvdt[s][(size_t)i * D + a];
        vh[(size_t)i * D + a] = v0[(size_t)i * D + a] + 0.5f * fa * dt;
    }
}
// PAIRS: the half-step velocities may be read as float2 (2D).  They follow n floats of du_out, so
// in 2D an odd n leaves them 4 bytes off an 8-byte boundary, and they are read word by word.
// Latency bound: four entries per lane in flight in 1D and 2D (131 -> 122 us at 512^2 with 32 neighbours);
// in 3D, where an entry is seven scalar loads, the compiler's own choice (128 neighbours, 884,736 particles:
// 1.65 ms against 1.79 with four entries and 1.98 with eight).
template <int D, int G, bool PAIRS>
__global__ void __launch_bounds__(PAIR_BLOCK)
k_finalize(int n, int ns, StagePtrs S, int pdv, const float* __restrict__ dtp, const float* __restrict__ vh,
           const float* __restrict__ u0, float* __restrict__ u_out, float* __restrict__ du_out) {
    pdl_entry();
    Grp<G> g(n);
    float du = 0.f;
    if (g.valid) {
        auto half = [&](int i) {
            if constexpr (PAIRS) {
                return load_vec<D>(vh, i);
            } else {
                Vec<D> r;
                #pragma unroll
                for (int a = 0; a < D; ++a) r.v[a] = __ldg(vh + (size_t)i * D + a);
                return r;
            }
        };
        Vec<D> vi = half(g.i);
        for (int s = 0; s < ns; ++s) {
            const int32_t* __restrict__ lst = S.list[s];
            const float* __restrict__ f = S.f[s];
            const float* __restrict__ ap = S.ap[s];
            const float* __restrict__ av = S.av[s];
            const float w = S.w[s];
            int b = S.offs[s][g.i], e = b + S.cnt[s][g.i];
            float acc = 0.f;
            auto add = [&](int q) {
                int j, k; entry(lst, q, j, k);
                Vec<D> vj = half(j);
                Vec<D> a1 = load_vec<D>(ap, k), a2 = load_vec<D>(av, k);
                float fk = __ldg(f + k);
                float d1 = 0.f, d2 = 0.f;
                #pragma unroll
                for (int a = 0; a < D; ++a) { float vji = vj.v[a] - vi.v[a]; d1 += vji * a1.v[a]; d2 += vji * a2.v[a]; }
                acc += pdv ? (w * fk * d1 + w * 0.5f * d2) : (w * fk * (d1 + d2));
            };
            if constexpr (D == 3) {
                for (int q = b + g.lane; q < e; q += G) add(q);
            } else {
                #pragma unroll 4
                for (int q = b + g.lane; q < e; q += G) add(q);
            }
            du += acc;
        }
    }
    du = gsum<G>(du);
    if (!g.valid || g.lane != 0) return;
    float dt = *dtp;
    if (du_out) du_out[g.i] = du;
    u_out[g.i] = u0[g.i] + du * dt;
}

// ---------------------------------------------------------------- conservation sums (FP64)
template <int D>
__global__ void k_cons(int n, const float* __restrict__ m, const float* __restrict__ v, const float* __restrict__ u, double* out) {
    pdl_entry();
    double M = 0, KE = 0, IE = 0, p[3] = {0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double mi = m[i];
        double v2 = 0;
        for (int a = 0; a < D; ++a) { double va = v[(size_t)i * D + a]; v2 += va * va; p[a] += mi * va; }
        M += mi; KE += 0.5 * mi * v2; IE += mi * (double)u[i];
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        M += __shfl_xor_sync(0xffffffffu, M, o); KE += __shfl_xor_sync(0xffffffffu, KE, o); IE += __shfl_xor_sync(0xffffffffu, IE, o);
        for (int a = 0; a < 3; ++a) p[a] += __shfl_xor_sync(0xffffffffu, p[a], o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out + 0, M); atomicAdd(out + 1, KE); atomicAdd(out + 2, IE); atomicAdd(out + 3, KE + IE);
        for (int a = 0; a < D; ++a) atomicAdd(out + 4 + a, p[a]);
    }
}

}  // namespace wsph

using namespace wsph;

// Fixed scratch for sph_compsph_balance_noalloc: n*(dim+1) floats (half-step
// velocities, then P/rho^gamma).  One copy per device, placed by the module loader,
// so the entry point that uses it never calls an allocator.  Every element the
// balance kernel reads is written first by the prep kernel of the same call, so
// nothing in it has to start at zero.
static __device__ __align__(256) float g_balance_scratch[SPH_BALANCE_NOALLOC_MAX_FLOATS];

constexpr int kMaxDevices = 64;

// The scratch address is a property of the context that loaded this module: a
// cudaDeviceReset (or another context made current on the same device) loads the module
// again and may place the array elsewhere.  So the address is cached per device together
// with the unique id of the context it was resolved in (cuCtxGetId, reached through
// cudaGetDriverEntryPoint, so the library does not link the driver API), and resolved
// again with cudaGetSymbolAddress whenever the current context's id differs.
struct ScratchSlot {
    unsigned long long ctx_id;
    float* ptr;
};
static ScratchSlot g_balance_scratch_slot[kMaxDevices];
static std::mutex g_balance_scratch_mu;

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// The unique id of the context current on this thread; 0 when none is current yet.
static int current_context_id(unsigned long long* id) {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void* f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<CtxGetIdFn>(f);
    });
    if (!get_current || !get_id)
        return set_error(SPH_ERR_CUDA, "sph_compsph_balance_noalloc: the driver does not provide cuCtxGetCurrent/cuCtxGetId");
    CUcontext ctx = nullptr;
    if (get_current(&ctx) != CUDA_SUCCESS) return set_error(SPH_ERR_CUDA, "sph_compsph_balance_noalloc: cuCtxGetCurrent failed");
    *id = 0;
    if (ctx && get_id(ctx, id) != CUDA_SUCCESS) return set_error(SPH_ERR_CUDA, "sph_compsph_balance_noalloc: cuCtxGetId failed");
    return SPH_OK;
}

// Address of g_balance_scratch in the current context, resolved once per device and
// context with cudaGetSymbolAddress while that device is current.
static int balance_scratch_on_current_device(float** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "sph_compsph_balance_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return set_error(SPH_ERR_BAD_ARG, "sph_compsph_balance_noalloc: device %d >= %d", dev, kMaxDevices);
    unsigned long long id = 0;
    int rc = current_context_id(&id);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_balance_scratch_mu);
    ScratchSlot& slot = g_balance_scratch_slot[dev];
    if (id == 0 || !slot.ptr || slot.ctx_id != id) {
        // cudaGetSymbolAddress also initialises the device's primary context when no
        // context was current yet; the id is read again after it
        void* sym = nullptr;
        e = cudaGetSymbolAddress(&sym, g_balance_scratch);
        if (e != cudaSuccess || !sym)
            return set_error(SPH_ERR_CUDA, "sph_compsph_balance_noalloc: cudaGetSymbolAddress on device %d: %s", dev,
                             cudaGetErrorString(e));
        if (id == 0 && (rc = current_context_id(&id))) return rc;
        slot.ptr = static_cast<float*>(sym);
        slot.ctx_id = id;
    }
    *out = slot.ptr;
    return SPH_OK;
}

extern "C" {

int sph_density_gather(const SphParams* p, int64_t n, int32_t support_mode, const float* x, const float* H, const float* m,
                       const int32_t* offs, const int32_t* cnt, const int32_t* list, float* rho_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho_out); CHECK_CSR();
    if (support_mode < 0 || support_mode > 4) return set_error(SPH_ERR_BAD_ARG, "bad support mode %d", support_mode);
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_density<KF, D, G_LIGHT>, grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s, (int)n, support_mode, P, x, H, m, offs, cnt, list, rho_out)));
    return check_launch("sph_density_gather");
}

int sph_adaptive_h_iter(const SphParams* p, int64_t n, int32_t support_mode, const float* x, const float* H, const float* m,
                        const int32_t* offs, const int32_t* cnt, const int32_t* list, const float* hbounds,
                        float* rho_out, float* H_out, float* ratio_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(hbounds); WSPH_CHECK_PTR(rho_out); WSPH_CHECK_PTR(H_out); CHECK_CSR();
    if (support_mode != SPH_SUPPORT_GATHER) return set_error(SPH_ERR_UNSUPPORTED, "adaptive support: only the gather scheme is implemented");
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_adaptive_h<KF, D, G_SCAN(D), false>, grid_g<G_SCAN(D)>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, (const float4*)nullptr, offs, cnt, list, hbounds, rho_out, H_out, ratio_out)));
    return check_launch("sph_adaptive_h_iter");
}

int sph_adaptive_h_iter_packed(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* xm,
                               const int32_t* offs, const int32_t* cnt, const int32_t* list, const float* hbounds, float* rho_out,
                               float* H_out, float* ratio_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(xm); WSPH_CHECK_PTR(hbounds); WSPH_CHECK_PTR(rho_out);
    WSPH_CHECK_PTR(H_out); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    if (reinterpret_cast<uintptr_t>(xm) & 15) return set_error(SPH_ERR_BAD_ARG, "sph_adaptive_h_iter_packed: xm must be 16-byte aligned");
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_ADAPT(D), G_WIDE, launch_pdl(k_adaptive_h<KF, D, LG, true>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m,
                                                                        reinterpret_cast<const float4*>(xm), offs, cnt, list, hbounds,
                                                                        rho_out, H_out, ratio_out)));
    return check_launch("sph_adaptive_h_iter_packed");
}

int sph_owen_iter(const SphParams* p, int64_t n, const float* x, const float* H, const int32_t* offs, const int32_t* cnt,
                  const int32_t* list, const double* lut_nh, const double* lut_psiH, int32_t nlut, double target_nh,
                  const float* hbounds, float* psi0_out, float* psiH_out, float* H_out, float* ratio_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(lut_nh); WSPH_CHECK_PTR(lut_psiH); WSPH_CHECK_PTR(hbounds);
    WSPH_CHECK_PTR(H_out); CHECK_CSR();
    if (nlut < 2) return set_error(SPH_ERR_BAD_ARG, "sph_owen_iter: the table needs at least 2 entries");
    if (!(target_nh > 0.0)) return set_error(SPH_ERR_BAD_ARG, "sph_owen_iter: target n_h must be positive");
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_owen<KF, D, G_LIGHT>, grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, offs, cnt, list, lut_nh, lut_psiH,
                                                                                             (int)nlut, (float)target_nh, hbounds, psi0_out,
                                                                                             psiH_out, H_out, ratio_out)));
    return check_launch("sph_owen_iter");
}

int sph_crk_volume(const SphParams* p, int64_t n, const float* x, const float* H, const int32_t* offs, const int32_t* cnt,
                   const int32_t* list, float* V_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(V_out); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_crk_volume<KF, D, G_SCAN(D)>, grid_g<G_SCAN(D)>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, offs, cnt, list, V_out)));
    return check_launch("sph_crk_volume");
}

int sph_crk_factors(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* V,
                    const int32_t* offs, const int32_t* cnt, const int32_t* list, float* A, float* B, float* gradA,
                    float* gradB, float* rho_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(V);
    WSPH_CHECK_PTR(A); WSPH_CHECK_PTR(B); WSPH_CHECK_PTR(gradA); WSPH_CHECK_PTR(gradB); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_CRK, G_WIDE, launch_pdl(k_crk_factors<KF, D, LG, false>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, V, offs, cnt, list, A, B, gradA, gradB, rho_out,
                                                                                                   EosOut{nullptr, nullptr, nullptr, nullptr, 0.f}, FactorWords{})));
    return check_launch("sph_crk_factors");
}

int sph_crk_factors_eos(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* V,
                        const int32_t* offs, const int32_t* cnt, const int32_t* list, float* A, float* B, float* gradA,
                        float* gradB, float* rho_out, const float* u, float* entropy_out, float* P_out, float* c_out,
                        void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(V);
    WSPH_CHECK_PTR(A); WSPH_CHECK_PTR(B); WSPH_CHECK_PTR(gradA); WSPH_CHECK_PTR(gradB); WSPH_CHECK_PTR(rho_out); WSPH_CHECK_PTR(u);
    CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_CRK, G_WIDE, launch_pdl(k_crk_factors<KF, D, LG, false>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, V, offs, cnt, list, A, B, gradA, gradB, rho_out,
                                                                                                   EosOut{u, entropy_out, P_out, c_out, P.gamma}, FactorWords{})));
    return check_launch("sph_crk_factors_eos");
}

int sph_pack_xh(const SphParams* p, int64_t n, const float* x, const float* H, float* xh, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(xh);
    if ((rc = check_align_vec(P, x, "x"))) return rc;
    if (reinterpret_cast<uintptr_t>(xh) & 15) return set_error(SPH_ERR_BAD_ARG, "sph_pack_xh: xh must be 16-byte aligned");
    wsph::count_launch();
    WSPH_DISPATCH_DS(*p, (launch_pdl(k_pack_xh<D>, (unsigned)((n + 255) / 256), 256, 0, s, (int)n, x, H, reinterpret_cast<float4*>(xh))));
    return check_launch("sph_pack_xh");
}

int sph_crk_factors_packed(const SphParams* p, int64_t n, const float* xh, const float* m, const float* V, const float* v,
                           const int32_t* offs, const int32_t* cnt, const int32_t* list, float* A, float* B, float* gradA,
                           float* gradB, float* rho_out, const float* u, float* entropy_out, float* P_out, float* c_out, float* fv,
                           float* vol, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(xh); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(V); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(fv);
    WSPH_CHECK_PTR(A); WSPH_CHECK_PTR(B); WSPH_CHECK_PTR(gradA); WSPH_CHECK_PTR(gradB); WSPH_CHECK_PTR(rho_out); WSPH_CHECK_PTR(u);
    CHECK_CSR();
    if (P.dim == 3) WSPH_CHECK_PTR(vol);
    if ((rc = check_align_vec(P, v, "v"))) return rc;
    if ((reinterpret_cast<uintptr_t>(xh) | reinterpret_cast<uintptr_t>(fv)) & 15)
        return set_error(SPH_ERR_BAD_ARG, "sph_crk_factors_packed: packed words must be 16-byte aligned");
    const FactorWords fw{reinterpret_cast<const float4*>(xh), v, reinterpret_cast<float4*>(fv), vol};
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_CRK, G_WIDE, launch_pdl(k_crk_factors<KF, D, LG, true>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, (const float*)nullptr,
                                      (const float*)nullptr, m, V, offs, cnt, list, A, B, gradA, gradB, rho_out,
                                      EosOut{u, entropy_out, P_out, c_out, P.gamma}, fw)));
    return check_launch("sph_crk_factors_packed");
}

int sph_grad_v_packed(const SphParams* p, int64_t n, const float* xh, const float* fv, const float* vol, const float* m, const float* rho,
                      const float* c, const float* A, const float* B, const float* gradA, const float* gradB, const int32_t* offs,
                      const int32_t* cnt, const int32_t* list, float* DvDx_out, float* drhodt_out, float* divergence_out,
                      float* div_out, float* fc, float* msgn, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(xh); WSPH_CHECK_PTR(fv); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(A); WSPH_CHECK_PTR(B); WSPH_CHECK_PTR(gradA);
    WSPH_CHECK_PTR(gradB); WSPH_CHECK_PTR(DvDx_out); WSPH_CHECK_PTR(drhodt_out); CHECK_CSR();
    if (div_out) { WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(c); WSPH_CHECK_PTR(fc); }
    if (div_out && P.dim == 3) { WSPH_CHECK_PTR(vol); WSPH_CHECK_PTR(msgn); }
    if ((rc = check_align_vec(P, B, "B")) || (rc = check_align_vec(P, gradA, "gradA"))) return rc;
    if ((reinterpret_cast<uintptr_t>(xh) | reinterpret_cast<uintptr_t>(fv) | reinterpret_cast<uintptr_t>(fc)) & 15)
        return set_error(SPH_ERR_BAD_ARG, "sph_grad_v_packed: packed words must be 16-byte aligned");
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_GRADV(D), G_WIDE, launch_pdl(k_grad_v_packed<KF, D, LG>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P,
                                      reinterpret_cast<const float4*>(xh), reinterpret_cast<const float4*>(fv), vol, m, rho, c, A, B, gradA,
                                      gradB, offs, cnt, list, DvDx_out, drhodt_out, divergence_out, div_out, reinterpret_cast<float4*>(fc), msgn)));
    return check_launch("sph_grad_v_packed");
}

int sph_switch_cullen_packed(const SphParams* p, int64_t n, const float* xh, const float* fc, const float* msgn, const float* rho,
                             const float* div, const float* div_prev, const float* alpha0_prev, const float* dt, const int32_t* offs,
                             const int32_t* cnt, const int32_t* list, float* alpha_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(xh); WSPH_CHECK_PTR(fc); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(div); WSPH_CHECK_PTR(div_prev);
    WSPH_CHECK_PTR(alpha0_prev); WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(alpha_out); CHECK_CSR();
    if (P.dim == 3) WSPH_CHECK_PTR(msgn);
    if ((reinterpret_cast<uintptr_t>(xh) | reinterpret_cast<uintptr_t>(fc)) & 15)
        return set_error(SPH_ERR_BAD_ARG, "sph_switch_cullen_packed: packed words must be 16-byte aligned");
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_CULLEN(D), G_WIDE, launch_pdl(k_cullen_packed<KF, D, LG>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P,
                                      reinterpret_cast<const float4*>(xh), reinterpret_cast<const float4*>(fc), msgn, rho, div, div_prev,
                                      alpha0_prev, dt, offs, cnt, list, alpha_out)));
    return check_launch("sph_switch_cullen_packed");
}

int sph_eos_ideal_gas(const SphParams* p, int64_t n, const float* u, const float* rho, float* A_out, float* P_out,
                      float* c_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(u); WSPH_CHECK_PTR(rho);
    wsph::count_launch(); launch_pdl(k_eos, grid_for(n, 256), 256, 0, s, (int)n, P.gamma, u, rho, A_out, P_out, c_out);
    return check_launch("sph_eos_ideal_gas");
}

int sph_grad_v(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
               const float* V, const float* A, const float* B, const float* gradA, const float* gradB, const float* v,
               const float* c, const int32_t* offs, const int32_t* cnt, const int32_t* list, float* DvDx_out,
               float* drhodt_out, float* div_out, float* vsig_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(V); WSPH_CHECK_PTR(A); WSPH_CHECK_PTR(B);
    WSPH_CHECK_PTR(gradA); WSPH_CHECK_PTR(gradB); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(DvDx_out); CHECK_CSR();
    if (div_out) WSPH_CHECK_PTR(m);
    if (vsig_out) WSPH_CHECK_PTR(c);
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, B, "B")) ||
        (rc = check_align_vec(P, gradA, "gradA")))
        return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_grad_v<KF, D, G_SCAN(D)>, grid_g<G_SCAN(D)>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, rho, V, A, B, gradA, gradB, v, c,
                                                                                                  offs, cnt, list, DvDx_out, drhodt_out, div_out, vsig_out)));
    return check_launch("sph_grad_v");
}

int sph_switch_cullen(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                      const float* div, const float* div_prev, const float* vsig, const float* v, const float* c,
                      const float* alpha0_prev, const float* dt, const int32_t* offs, const int32_t* cnt, const int32_t* list,
                      float* alpha_out, float* R_out, float* vsig_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(div); WSPH_CHECK_PTR(div_prev);
    WSPH_CHECK_PTR(alpha0_prev); WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(alpha_out); CHECK_CSR();
    if (!vsig) { WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(c); }   // v_sig needs the whole Verlet rows
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_cullen<KF, D, G_SCAN(D)>, grid_g<G_SCAN(D)>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, rho, div, div_prev, vsig, v, c,
                                                                                                  alpha0_prev, dt, offs, cnt, list, alpha_out, R_out, vsig_out)));
    return check_launch("sph_switch_cullen");
}

int sph_switch_hopkins_terms(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                             const float* v, const float* alpha0, const int32_t* offs, const int32_t* cnt, const int32_t* list,
                             float* div_out, float* shear2_out, float* alpha_out, float* R_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(alpha0);
    WSPH_CHECK_PTR(div_out); WSPH_CHECK_PTR(shear2_out); WSPH_CHECK_PTR(alpha_out); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_hopkins_grad<KF, D, G_LIGHT>, grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, rho, v, offs, cnt, list,
                                                                                                       div_out, shear2_out)));
    if ((rc = check_launch("sph_switch_hopkins_terms"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_KDS(*p, (launch_pdl(k_hopkins_alpha<KF, D, G_LIGHT>, grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, rho, div_out, shear2_out,
                                                                                                        alpha0, offs, cnt, list, alpha_out, R_out)));
    return check_launch("sph_switch_hopkins_terms");
}

int sph_switch_hopkins_update(const SphParams* p, int64_t n, const float* x, const float* H, const float* v, const float* c,
                              const float* div, const float* div_prev, const float* alpha0, const float* dt,
                              const int32_t* offs, const int32_t* cnt, const int32_t* list, float* alpha0_out, float* vsig_out,
                              void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(c); WSPH_CHECK_PTR(div); WSPH_CHECK_PTR(div_prev);
    WSPH_CHECK_PTR(alpha0); WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(alpha0_out); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v"))) return rc;
    wsph::count_launch();
    WSPH_DISPATCH_DS(*p, (launch_pdl(k_hopkins_update<D, G_LIGHT>, grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, v, c, div, div_prev, alpha0, dt,
                                                                                                  offs, cnt, list, alpha0_out, vsig_out)));
    return check_launch("sph_switch_hopkins_update");
}

int sph_switch_balsara(const SphParams* p, int64_t n, const float* DvDx, const float* c, float* alpha_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(DvDx); WSPH_CHECK_PTR(c); WSPH_CHECK_PTR(alpha_out);
    wsph::count_launch(); WSPH_DISPATCH_DIM(P.dim, (launch_pdl(k_balsara<D>, grid_for(n, 256), 256, 0, s, (int)n, DvDx, c, alpha_out)));
    return check_launch("sph_switch_balsara");
}

static int crk_accel_dudt_impl(const SphParams* p, int64_t n, const float* x, const float* H, const float* m,
                               const float* rho, const float* V, const float* A, const float* B, const float* gradA,
                               const float* gradB, const float* v, const float* c, const float* Pr, const float* DvDx,
                               const int32_t* offs, const int32_t* cnt, const int32_t* list, const int32_t* verlet_cnt,
                               float* dvdt_out, float* dudt_out, float* dEdt_out, float* ap_ij, float* av_ij, float* records,
                               void* stream, const char* name) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(V); WSPH_CHECK_PTR(A);
    WSPH_CHECK_PTR(B); WSPH_CHECK_PTR(gradA); WSPH_CHECK_PTR(gradB); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(c); WSPH_CHECK_PTR(Pr);
    WSPH_CHECK_PTR(DvDx); CHECK_CSR();
    if ((rc = check_align_vec(P, x, "x")) || (rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, B, "B")) ||
        (rc = check_align_vec(P, gradA, "gradA")) || (rc = check_align_vec(P, dvdt_out, "dvdt")) ||
        (rc = check_align_vec(P, ap_ij, "ap_ij")) || (rc = check_align_vec(P, av_ij, "av_ij")))
        return rc;
    if (records && (reinterpret_cast<uintptr_t>(records) & 15))
        return set_error(SPH_ERR_BAD_ARG, "%s: records must be 16-byte aligned", name);
    if (records) {
        wsph::count_launch();
        WSPH_DISPATCH_DS(*p, (launch_pdl(k_crk_pack<D>, (unsigned)((n + 255) / 256), 256, 0, s, (int)n, P, x, H, rho, V, A, B, gradA, gradB, v, c,
                                                                                       Pr, DvDx, records)));
        wsph::count_launch();
        WSPH_DISPATCH_KDS(*p, PAIR_LANES(n, G_ACCEL(D), G_WIDE, launch_pdl(k_crk_accel_dudt<KF, D, LG, true>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, rho, V, A, B, gradA, gradB, v, c, Pr, DvDx, records, offs, cnt, list,
                                  verlet_cnt, dvdt_out, dudt_out, dEdt_out, ap_ij, av_ij)));
    } else {
        wsph::count_launch();
        WSPH_DISPATCH_KDS(*p, (launch_pdl(k_crk_accel_dudt<KF, D, G_ACCEL(D), false>, grid_g<G_ACCEL(D)>(n), PAIR_BLOCK, 0, s, (int)n, P, x, H, m, rho, V, A, B, gradA, gradB, v, c, Pr, DvDx, nullptr, offs, cnt, list,
                                  verlet_cnt, dvdt_out, dudt_out, dEdt_out, ap_ij, av_ij)));
    }
    return check_launch(name);
}

int sph_crk_accel_dudt(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                       const float* V, const float* A, const float* B, const float* gradA, const float* gradB,
                       const float* v, const float* c, const float* Pr, const float* DvDx, const int32_t* offs,
                       const int32_t* cnt, const int32_t* list, const int32_t* verlet_cnt, float* dvdt_out, float* dudt_out,
                       float* dEdt_out, float* ap_ij, float* av_ij, void* stream) {
    return crk_accel_dudt_impl(p, n, x, H, m, rho, V, A, B, gradA, gradB, v, c, Pr, DvDx, offs, cnt, list, verlet_cnt, dvdt_out,
                               dudt_out, dEdt_out, ap_ij, av_ij, nullptr, stream, "sph_crk_accel_dudt");
}

int sph_crk_record_floats(int32_t dim) {
    return dim == 1 ? CrkRec<1>::R : dim == 2 ? CrkRec<2>::R : dim == 3 ? CrkRec<3>::R : 0;
}

int sph_crk_accel_dudt_packed(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                              const float* V, const float* A, const float* B, const float* gradA, const float* gradB,
                              const float* v, const float* c, const float* Pr, const float* DvDx, const int32_t* offs,
                              const int32_t* cnt, const int32_t* list, const int32_t* verlet_cnt, float* dvdt_out,
                              float* dudt_out, float* dEdt_out, float* ap_ij, float* av_ij, float* records, void* stream) {
    WSPH_CHECK_PTR(records);
    return crk_accel_dudt_impl(p, n, x, H, m, rho, V, A, B, gradA, gradB, v, c, Pr, DvDx, offs, cnt, list, verlet_cnt, dvdt_out,
                               dudt_out, dEdt_out, ap_ij, av_ij, records, stream, "sph_crk_accel_dudt_packed");
}

int sph_crk_accel(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                  const float* V, const float* A, const float* B, const float* gradA, const float* gradB, const float* v,
                  const float* c, const float* P, const float* DvDx, const int32_t* offs, const int32_t* cnt,
                  const int32_t* list, const int32_t* verlet_cnt, float* dvdt_out, float* ap_ij, float* av_ij, void* stream) {
    return sph_crk_accel_dudt(p, n, x, H, m, rho, V, A, B, gradA, gradB, v, c, P, DvDx, offs, cnt, list, verlet_cnt, dvdt_out,
                              nullptr, nullptr, ap_ij, av_ij, stream);
}

int sph_crk_dudt(const SphParams* p, int64_t n, const float* x, const float* H, const float* m, const float* rho,
                 const float* V, const float* A, const float* B, const float* gradA, const float* gradB, const float* v,
                 const float* c, const float* P, const float* DvDx, const int32_t* offs, const int32_t* cnt,
                 const int32_t* list, float* dudt_out, void* stream) {
    return sph_crk_accel_dudt(p, n, x, H, m, rho, V, A, B, gradA, gradB, v, c, P, DvDx, offs, cnt, list, nullptr, nullptr, dudt_out,
                              nullptr, nullptr, nullptr, stream);
}

int sph_compsph_balance(const SphParams* p, int64_t n, const float* m, const float* rho, const float* Pr, const float* u,
                        const float* v, const float* dvdt, const float* dt, const int32_t* offs, const int32_t* cnt,
                        const int32_t* list, const int32_t* inter_counts, const float* ap_ij, const float* av_ij, float* scratch,
                        float* f_ij_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(Pr); WSPH_CHECK_PTR(u); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(dvdt);
    WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(ap_ij); WSPH_CHECK_PTR(av_ij); WSPH_CHECK_PTR(scratch); WSPH_CHECK_PTR(f_ij_out); CHECK_CSR();
    if (P.energy_scheme < 0 || P.energy_scheme > 5) return set_error(SPH_ERR_BAD_ARG, "bad energy scheme %d", P.energy_scheme);
    if ((rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, dvdt, "dvdt")) || (rc = check_align_vec(P, ap_ij, "ap_ij")) ||
        (rc = check_align_vec(P, av_ij, "av_ij")) || (rc = check_align_vec(P, scratch, "scratch")))
        return rc;
    float* vh = scratch;
    float* sarr = scratch + n * P.dim;
    wsph::count_launch(); WSPH_DISPATCH_DIM(P.dim, (launch_pdl(k_balance_prep<D>, grid_for(n, 256), 256, 0, s, (int)n, P, rho, Pr, v, dvdt, dt, vh, sarr,
                                                               (float4*)nullptr)));
    wsph::count_launch();
    WSPH_DISPATCH_DS(*p, PAIR_LANES(n, G_BALANCE(D), G_WIDE, launch_pdl(k_balance<D, LG, false>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, m, rho, Pr, u, vh, sarr, dt, offs, cnt,
                                                                        list, inter_counts, ap_ij, av_ij, f_ij_out, (const float4*)nullptr)));
    return check_launch("sph_compsph_balance");
}

// sph_compsph_balance in 3D with the half-step velocity and entropy of each particle packed in one
// 16-byte word (words: n * 4 floats): 1.00 against 1.36 ms at 884,736 particles (with 16 lanes per
// particle, 1.21 with 16 lanes alone).  In 2D, where a pair's two gathers are 12 bytes, packing
// them gains nothing (92 against 89 us at 262,144).
int sph_compsph_balance_packed(const SphParams* p, int64_t n, const float* m, const float* rho, const float* Pr, const float* u,
                               const float* v, const float* dvdt, const float* dt, const int32_t* offs, const int32_t* cnt,
                               const int32_t* list, const int32_t* inter_counts, const float* ap_ij, const float* av_ij, float* words,
                               float* f_ij_out, void* stream) {
    PAIR_PRELUDE();
    WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(Pr); WSPH_CHECK_PTR(u); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(dvdt);
    WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(ap_ij); WSPH_CHECK_PTR(av_ij); WSPH_CHECK_PTR(words); WSPH_CHECK_PTR(f_ij_out); CHECK_CSR();
    if (P.energy_scheme < 0 || P.energy_scheme > 5) return set_error(SPH_ERR_BAD_ARG, "bad energy scheme %d", P.energy_scheme);
    if ((rc = check_align_vec(P, v, "v")) || (rc = check_align_vec(P, dvdt, "dvdt")) || (rc = check_align_vec(P, ap_ij, "ap_ij")) ||
        (rc = check_align_vec(P, av_ij, "av_ij")))
        return rc;
    if (reinterpret_cast<uintptr_t>(words) & 15) return set_error(SPH_ERR_BAD_ARG, "sph_compsph_balance_packed: words must be 16-byte aligned");
    if (P.dim != 3) return set_error(SPH_ERR_UNSUPPORTED, "sph_compsph_balance_packed: dim must be 3");
    float4* w = reinterpret_cast<float4*>(words);
    wsph::count_launch();
    launch_pdl(k_balance_prep<3>, grid_for(n, 256), 256, 0, s, (int)n, P, rho, Pr, v, dvdt, dt, (float*)nullptr, (float*)nullptr, w);
    wsph::count_launch();
    PAIR_LANES(n, G_BALANCE(3), G_WIDE, launch_pdl(k_balance<3, LG, true>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, P, m, rho, Pr, u, (const float*)nullptr,
                                                   (const float*)nullptr, dt, offs, cnt, list, inter_counts, ap_ij, av_ij, f_ij_out, (const float4*)w));
    return check_launch("sph_compsph_balance_packed");
}

// sph_compsph_balance with its scratch taken from g_balance_scratch instead of the
// caller.  For callers that cannot allocate device memory on the step path: a plain C
// or Fortran host code bound through the FFI with no caching allocator of its own, or
// a timed inner loop, where cudaMalloc/cudaFree would synchronise the whole device.
// The first call on each device (and the first after that device's context was replaced,
// e.g. by cudaDeviceReset) resolves the scratch address (cudaGetSymbolAddress); make that
// first call before any stream capture.  Every device that loads the library holds the
// 16 MiB array until the process exits.  Calls in flight at the same time on one device
// (different streams, or different host threads) share the scratch and race.
int sph_compsph_balance_noalloc(const SphParams* p, int64_t n, const float* m, const float* rho, const float* Pr,
                                const float* u, const float* v, const float* dvdt, const float* dt, const int32_t* offs,
                                const int32_t* cnt, const int32_t* list, const float* ap_ij, const float* av_ij,
                                float* f_ij_out, void* stream) {
    if (!p) return set_error(SPH_ERR_BAD_ARG, "sph_compsph_balance_noalloc: null params");
    if (p->dim < 1 || p->dim > 3) return set_error(SPH_ERR_BAD_ARG, "sph_compsph_balance_noalloc: dim must be 1, 2 or 3");
    if (n > 0 && n * (int64_t)(p->dim + 1) > (int64_t)SPH_BALANCE_NOALLOC_MAX_FLOATS)
        return set_error(SPH_ERR_BAD_ARG, "sph_compsph_balance_noalloc: n*(dim+1) = %lld exceeds the fixed scratch of %d floats",
                         (long long)(n * (p->dim + 1)), SPH_BALANCE_NOALLOC_MAX_FLOATS);
    if (n <= 0) return sph_compsph_balance(p, n, m, rho, Pr, u, v, dvdt, dt, offs, cnt, list, nullptr, ap_ij, av_ij, nullptr, f_ij_out, stream);
    float* scratch = nullptr;
    int rc = balance_scratch_on_current_device(&scratch);
    if (rc) return rc;
    return sph_compsph_balance(p, n, m, rho, Pr, u, v, dvdt, dt, offs, cnt, list, nullptr, ap_ij, av_ij, scratch, f_ij_out, stream);
}

int sph_cfl_dt(const SphParams* p, int64_t n, const float* H, const float* u, const float* rho, const float* dt_prev,
               float* dt_out, void* stream) {
    DevParams P;
    int rc = params_to_dev(p, &P);
    if (rc) return rc;
    if (n <= 0 || n > 0x7fffffff) return set_error(SPH_ERR_BAD_ARG, "sph_cfl_dt: n must be in [1, 2^31)");
    WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(u); WSPH_CHECK_PTR(dt_out);
    (void)rho;
    cudaStream_t s = WSPH_STREAM(stream);
    float* red = dt_out + 1;
    wsph::count_launch(); launch_pdl(k_cfl_init, 1, 1, 0, s, red);
    int blocks = (int)((n + 1023) / 1024);
    if (blocks > 148 * 4) blocks = 148 * 4;
    wsph::count_launch(); launch_pdl(k_cfl_reduce, blocks, 256, 0, s, (int)n, P.gamma, H, u, red);
    wsph::count_launch(); launch_pdl(k_cfl_final, 1, 1, 0, s, P, red, dt_prev, dt_out);
    return check_launch("sph_cfl_dt");
}

int sph_rk_combine(const SphParams* p, int64_t count, const float* y0, int32_t nk, const float* const* k_ptrs,
                   const double* weights, const float* dt, int32_t wrap_dim, float* y_out, void* stream) {
    DevParams P;
    int rc = params_to_dev(p, &P);
    if (rc) return rc;
    if (count < 0) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine: count < 0");
    if (count == 0) return SPH_OK;
    if (nk < 0 || nk > 8) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine: nk must be in [0, 8]");
    WSPH_CHECK_PTR(y0); WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(y_out);
    KPtrs K;
    for (int q = 0; q < 8; ++q) { K.k[q] = nullptr; K.w[q] = 0.f; }
    for (int q = 0; q < nk; ++q) {
        if (!k_ptrs || !k_ptrs[q] || !weights) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine: null derivative %d", q);
        K.k[q] = k_ptrs[q]; K.w[q] = (float)weights[q];
    }
    wsph::count_launch(); launch_pdl(k_rk_combine, grid_for(count, 256), 256, 0, WSPH_STREAM(stream), count, y0, nk, K, dt, wrap_dim, P.dom, y_out);
    return check_launch("sph_rk_combine");
}

int sph_rk_combine_fields(const SphParams* p, int32_t nfields, const int64_t* counts, const float* const* y0s,
                          float* const* y_outs, const int32_t* wrap_dims, int32_t nk, const float* const* k_ptrs,
                          const double* weights, const float* dt, void* stream) {
    DevParams P;
    int rc = params_to_dev(p, &P);
    if (rc) return rc;
    if (nfields < 1 || nfields > RKF_MAX) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine_fields: nfields must be in [1, %d]", RKF_MAX);
    if (nk < 0 || nk > 8) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine_fields: nk must be in [0, 8]");
    WSPH_CHECK_PTR(counts); WSPH_CHECK_PTR(y0s); WSPH_CHECK_PTR(y_outs); WSPH_CHECK_PTR(wrap_dims); WSPH_CHECK_PTR(dt);
    if (nk > 0) { WSPH_CHECK_PTR(k_ptrs); WSPH_CHECK_PTR(weights); }
    FieldPtrs F;
    memset(&F, 0, sizeof(F));
    int64_t total = 0, largest = 0;
    for (int f = 0; f < nfields; ++f) {
        if (counts[f] > largest) largest = counts[f];
        if (counts[f] < 0) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine_fields: count %d < 0", f);
        if (counts[f] > 0 && (!y0s[f] || !y_outs[f])) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine_fields: null field %d", f);
        if (wrap_dims[f] < 0 || wrap_dims[f] > 3) return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine_fields: wrap_dim %d out of range", f);
        F.y0[f] = y0s[f]; F.y[f] = y_outs[f]; F.wrap[f] = wrap_dims[f];
        for (int q = 0; q < nk; ++q) {
            if (counts[f] > 0 && !k_ptrs[f * nk + q])
                return set_error(SPH_ERR_BAD_ARG, "sph_rk_combine_fields: null derivative %d of field %d", q, f);
            F.k[f][q] = k_ptrs[f * nk + q];
        }
        total += counts[f];
        F.end[f] = total;
    }
    for (int q = 0; q < nk; ++q) F.w[q] = (float)weights[q];
    if (total == 0) return SPH_OK;
    wsph::count_launch();
    if (largest <= 148 * 2048) launch_pdl(k_rk_combine_fields<1>, dim3((unsigned)((largest + 255) / 256), (unsigned)nfields), 256, 0,
                                          WSPH_STREAM(stream), (int)nk, F, dt, P.dom);
    else launch_pdl(k_rk_combine_fields<4>, dim3((unsigned)((largest + 1023) / 1024), (unsigned)nfields), 256, 0, WSPH_STREAM(stream), (int)nk, F,
                    dt, P.dom);
    return check_launch("sph_rk_combine_fields");
}

int sph_finalize_compatible_energy(const SphParams* p, int64_t n, int32_t nstages, const double* weights, const float* dt,
                                   const float* v0, const float* u0, const float* const* dvdt_s,
                                   const int32_t* const* offs_s, const int32_t* const* cnt_s, const int32_t* const* list_s,
                                   const float* const* f_ij_s, const float* const* ap_ij_s, const float* const* av_ij_s,
                                   float* u_out, float* du_out, void* stream) {
    PAIR_PRELUDE();
    if (nstages < 1 || nstages > 8) return set_error(SPH_ERR_BAD_ARG, "nstages must be in [1, 8]");
    WSPH_CHECK_PTR(weights); WSPH_CHECK_PTR(dt); WSPH_CHECK_PTR(v0); WSPH_CHECK_PTR(u0); WSPH_CHECK_PTR(u_out);
    WSPH_CHECK_PTR(dvdt_s); WSPH_CHECK_PTR(offs_s); WSPH_CHECK_PTR(cnt_s); WSPH_CHECK_PTR(list_s);
    WSPH_CHECK_PTR(f_ij_s); WSPH_CHECK_PTR(ap_ij_s); WSPH_CHECK_PTR(av_ij_s);
    StagePtrs S;
    for (int q = 0; q < nstages; ++q) {
        if (!dvdt_s[q] || !offs_s[q] || !cnt_s[q] || !list_s[q] || !f_ij_s[q] || !ap_ij_s[q] || !av_ij_s[q])
            return set_error(SPH_ERR_BAD_ARG, "finalize: null array for stage %d", q);
        S.dvdt[q] = dvdt_s[q]; S.offs[q] = offs_s[q]; S.cnt[q] = cnt_s[q]; S.list[q] = list_s[q];
        S.f[q] = f_ij_s[q]; S.ap[q] = ap_ij_s[q]; S.av[q] = av_ij_s[q]; S.w[q] = (float)weights[q];
    }
    if (!du_out) return set_error(SPH_ERR_BAD_ARG, "finalize: du_out must hold n*(1+dim) floats (du and v_half scratch)");
    float* vh = du_out + n;
    int pdv = P.energy_scheme == SPH_ENERGY_PDV;
    wsph::count_launch(); WSPH_DISPATCH_DIM(P.dim, (launch_pdl(k_vhalf<D>, grid_for(n, 256), 256, 0, s, (int)n, nstages, S, dt, v0, vh)));
    wsph::count_launch();
    const bool pairs = P.dim != 2 || !(reinterpret_cast<uintptr_t>(vh) & 7);
    if (pairs) {
        WSPH_DISPATCH_DS(*p, PAIR_LANES(n, G_LIGHT, G_WIDE, launch_pdl(k_finalize<D, LG, true>, grid_g<LG>(n), PAIR_BLOCK, 0, s, (int)n, nstages, S, pdv, dt, vh, u0, u_out, du_out)));
    } else {
        launch_pdl(k_finalize<2, G_LIGHT, false>, grid_g<G_LIGHT>(n), PAIR_BLOCK, 0, s, (int)n, nstages, S, pdv, dt, vh, u0, u_out, du_out);
    }
    return check_launch("sph_finalize_compatible_energy");
}

int sph_conservation_sums(const SphParams* p, int64_t n, const float* m, const float* v, const float* u, double* out,
                          void* stream) {
    DevParams P;
    int rc = params_to_dev(p, &P);
    if (rc) return rc;
    WSPH_CHECK_PTR(out);
    cudaStream_t s = WSPH_STREAM(stream);
    cudaMemsetAsync(out, 0, sizeof(double) * 7, s);
    if (n <= 0) return check_launch("sph_conservation_sums");
    WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(u);
    int blocks = grid_for(n, 256);
    if (blocks > 148 * 4) blocks = 148 * 4;
    wsph::count_launch(); WSPH_DISPATCH_DIM(P.dim, (launch_pdl(k_cons<D>, blocks, 256, 0, s, (int)n, m, v, u, out)));
    return check_launch("sph_conservation_sums");
}

}  // extern "C"
