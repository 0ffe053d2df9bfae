// Batched ensemble of independent periodic delta-SPH boxes (no counterpart in the
// reference, which runs one simulation per process; the right-hand side per box is
// schemes/deltaSPH.py's, see sph_deltasph.cuh).
//
// All boxes share the periodic domain of SphParams but not their particles: box b has
// its own cell grid of G_b^dim cells (cell size L / G_b >= verlet_scale * max H in the
// box), and the cell keys of box b start at box_cell_base[b], so a neighbour search over
// every particle of every box in one set of launches (segment offsets into one cell
// table) never pairs particles of different boxes.
//
// One time step of every box is ONE cooperative persistent launch (k_ens_step): Heun
// RK2 with two right-hand sides, five phases separated by four bounded grid barriers:
//   pack y0 | A(y0) | B(y0), y1 = y0 + dt k1 | A(y1) | B(y1), y = y0 + dt/2 (k1 + k2)
// where A is the renormalised density gradient + EOS and B the delta-SPH right-hand side.
// dt is per box (box_dt).  The step also reduces the largest displacement since the list
// was built, so the caller can tell when the Verlet skin is used up.
#include <cuda_runtime.h>
#include <algorithm>
#include <mutex>
#include "sph_deltasph.cuh"
#include "sph_persistent.cuh"

namespace wsph {

// ---------------------------------------------------------------- neighbour search
template <int D> __device__ __forceinline__ void ens_cell(const Vec<D>& x, const DomainF& dom, int G, int* c) {
    #pragma unroll
    for (int a = 0; a < D; ++a) {
        int k = (int)floorf(__fdiv_rn(__fsub_rn(x.v[a], dom.min[a]), dom.L[a]) * (float)G);
        c[a] = k < 0 ? 0 : (k >= G ? G - 1 : k);
    }
}
template <int D> __device__ __forceinline__ int ens_key(const int* c, int G, int base) {
    int k = c[D - 1];
    #pragma unroll
    for (int a = D - 2; a >= 0; --a) k = k * G + c[a];
    return base + k;
}

template <int D>
__global__ void k_ens_keys(int n, DomainF dom, const float* __restrict__ x, const int32_t* __restrict__ box_of,
                           const int32_t* __restrict__ box_grid, const int32_t* __restrict__ box_base, int32_t* __restrict__ keys,
                           int32_t* __restrict__ slot, int32_t* __restrict__ counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = box_of[i];
    int c[D];
    ens_cell<D>(load_vec<D>(x, i), dom, box_grid[b], c);
    const int key = ens_key<D>(c, box_grid[b], box_base[b]);
    keys[i] = key;
    slot[i] = atomicAdd(counts + key, 1);
}

__global__ void k_ens_scatter(int n, const int32_t* __restrict__ keys, const int32_t* __restrict__ slot,
                              const int32_t* __restrict__ start, int32_t* __restrict__ sorted) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sorted[start[keys[i]] + slot[i]] = i;
}

// Ascending particle index inside each cell (deterministic rows).
__global__ void k_ens_sort_cells(int64_t ncells, const int32_t* __restrict__ start, const int32_t* __restrict__ counts,
                                 int32_t* __restrict__ sorted) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    int32_t* s = sorted + start[c];
    const int k = counts[c];
    for (int a = 1; a < k; ++a) {
        const int v = s[a];
        int b = a - 1;
        while (b >= 0 && s[b] > v) { s[b + 1] = s[b]; --b; }
        s[b + 1] = v;
    }
}

// Position and support of the particles in cell order: the search below reads candidates as
// consecutive 16-byte words instead of an index, a position and a support each.
template <int D>
__global__ void k_ens_pack_sorted(int n, const float* __restrict__ x, const float* __restrict__ H, const int32_t* __restrict__ sorted,
                                  float4* __restrict__ words) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int j = sorted[s];
    words[s] = make_xh<D>(load_vec<D>(x, j), H[j]);
}

// Count (FILL = false) or fill the Verlet rows: j in the 3^dim stencil cells of i's box
// grid (periodic wrap, x fastest), ascending index within a cell, kept when
// |x_i - x_j|^2 < (verlet_scale max(H_i, H_j))^2 with the minimum-image distance.
template <int D, int G, bool FILL>
__global__ void __launch_bounds__(128)
k_ens_verlet(int n, DevParams P, const float* __restrict__ x, const float* __restrict__ H, const int32_t* __restrict__ box_of,
             const int32_t* __restrict__ box_grid, const int32_t* __restrict__ box_base, const int32_t* __restrict__ start,
             const int32_t* __restrict__ counts, const int32_t* __restrict__ sorted, const float4* __restrict__ words,
             int32_t* __restrict__ num,
             const int32_t* __restrict__ offs, int32_t* __restrict__ list, const long long* __restrict__ nnz, int64_t cap) {
    Grp<G> g(n);
    if (FILL && *nnz > cap) return;            // uniform over the grid
    // every group (valid or not) walks the same stencil with a warp-uniform candidate
    // loop, so the ballots below always have the full warp
    const int i = g.valid ? g.i : 0;
    Vec<D> xi = vzero<D>();
    float Hi = 0.f;
    int Gb = 1, base = 0, c[D], row = 0;
    #pragma unroll
    for (int a = 0; a < D; ++a) c[a] = 0;
    if (g.valid) {
        xi = load_vec<D>(x, i);
        Hi = H[i];
        const int b = box_of[i];
        Gb = box_grid[b];
        base = box_base[b];
        ens_cell<D>(xi, P.dom, Gb, c);
        if (FILL) row = offs[i];
    }
    const unsigned int lanes = (1u << G) - 1u;
    const int gshift = threadIdx.x & 31 & ~(G - 1);
    int w = 0;
    constexpr int NS = D == 1 ? 3 : (D == 2 ? 9 : 27);
    for (int sidx = 0; sidx < NS; ++sidx) {
        int s0 = 0, cn = 0;
        if (g.valid) {
            int cc[D], t = sidx;
            #pragma unroll
            for (int a = 0; a < D; ++a) {
                cc[a] = c[a] + (t % 3) - 1;                       // periodic: one wrap at most
                cc[a] = cc[a] < 0 ? cc[a] + Gb : (cc[a] >= Gb ? cc[a] - Gb : cc[a]);
                t /= 3;
            }
            const int key = ens_key<D>(cc, Gb, base);
            s0 = start[key];
            cn = counts[key];
        }
        for (int q0 = 0; __any_sync(0xffffffffu, q0 < cn); q0 += G) {
            const int q = q0 + g.lane;
            bool keep = false;
            if (q < cn) {
                const float4 t = __ldg(words + s0 + q);
                const Vec<D> d = dist_vec<D>(xi, vec_of_word<D>(t), P.dom);
                const float R = __fmul_rn(P.verlet_scale, wmax(Hi, support_of<D>(t)));
                keep = dist2_rn<D>(d) < __fmul_rn(R, R);
            }
            const unsigned int bits = (__ballot_sync(0xffffffffu, keep) >> gshift) & lanes;
            if (FILL && keep) list[row + w + __popc(bits & ((1u << g.lane) - 1u))] = __ldg(sorted + s0 + q);
            w += __popc(bits);
        }
    }
    if (!FILL && g.valid && g.lane == 0) num[g.i] = w;
}

__global__ void k_ens_check(const long long* __restrict__ nnz, int64_t cap, int32_t* __restrict__ status) {
    if (*nnz > cap) atomicOr(status, SPH_STATUS_LIST_OVERFLOW);
}

struct EnsNbWs {
    int32_t *keys, *slot, *counts, *start, *sorted;
    float4* words;
    long long* total;
    char* scan;
    int64_t bytes;
};
static int64_t al256(int64_t b) { return (b + 255) / 256 * 256; }
static EnsNbWs ens_carve(char* base, int64_t n, int64_t ncells) {
    EnsNbWs w;
    int64_t o = 0;
    w.total = reinterpret_cast<long long*>(base + o); o += 256;
    w.keys = reinterpret_cast<int32_t*>(base + o); o += al256(n * 4);
    w.slot = reinterpret_cast<int32_t*>(base + o); o += al256(n * 4);
    w.sorted = reinterpret_cast<int32_t*>(base + o); o += al256(n * 4);
    // 16-byte aligned whatever the base's alignment
    w.words = reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(base) + o + 15) & ~static_cast<uintptr_t>(15));
    o += al256(n * 16 + 16);
    w.counts = reinterpret_cast<int32_t*>(base + o); o += al256(ncells * 4);
    w.start = reinterpret_cast<int32_t*>(base + o); o += al256(ncells * 4);
    w.scan = base + o;
    o += al256(scan_ws_bytes(ncells > n ? ncells : n));
    w.bytes = o;
    return w;
}

// ---------------------------------------------------------------- persistent step
// What the pair passes gather of a particle, in 16-byte words written by the phase that computes
// them.  Other blocks read them after a grid barrier, with plain loads (never the read-only path).
//   xv  position, then velocity (1D, 2D: one word; 3D: one word each)          one set per stage:
//   sv  density, V = m / rho, H                                                the first is still read
//   gp  renormalised density gradient, then the pressure                       while the second is written
struct EnsSet { float4 *xv, *sv; };
struct EnsArgs {
    int n;
    DevParams P;
    WcDev W;
    const int32_t *box_of;
    const float *box_dt, *H, *m, *x_build;
    float *x, *v, *rho;                    // state y0 (updated in place at the end of the step)
    float *dv1, *drho1;                    // first right-hand side
    EnsSet set[2];
    float4* gp;
    void* near;                            // ENS_NEAR bits per particle: see EnsWalk
    const int32_t *offs, *cnt, *list;
    BarrierCtl* ctl;
    int* work;                             // next particle of each pair pass
    unsigned int* disp;                    // max |x - x_build| / H since the list was built (ordered float)
    int32_t* status;
};

__device__ __forceinline__ unsigned int ens_ord(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
template <int D> __device__ __forceinline__ Vec<D> wrap_pos(Vec<D> x, const DomainF& dom) {
    #pragma unroll
    for (int a = 0; a < D; ++a)
        if (dom.periodic[a]) {
            if (x.v[a] >= dom.max[a]) x.v[a] -= dom.L[a];
            else if (x.v[a] < dom.min[a]) x.v[a] += dom.L[a];
        }
    return x;
}

template <int D> __device__ __forceinline__ void put_xv(const EnsSet& s, int i, const Vec<D>& x, const Vec<D>& v) {
    float w[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    constexpr int V0 = D == 3 ? 4 : D;
    #pragma unroll
    for (int a = 0; a < D; ++a) { w[a] = x.v[a]; w[V0 + a] = v.v[a]; }
    constexpr int NW = D == 3 ? 2 : 1;
    #pragma unroll
    for (int k = 0; k < NW; ++k) s.xv[(size_t)i * NW + k] = make_float4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
}
template <int D> __device__ __forceinline__ float4 get_x_word(const EnsSet& s, int i) { return s.xv[D == 3 ? 2 * (size_t)i : (size_t)i]; }
template <int D> __device__ __forceinline__ Vec<D> get_v(const EnsSet& s, int i, const float4& xw) {
    if constexpr (D == 3) {
        return vec_of_word<3>(s.xv[2 * (size_t)i + 1]);
    } else {
        Vec<D> v;
        #pragma unroll
        for (int a = 0; a < D; ++a) v.v[a] = word_of(xw, D + a);
        return v;
    }
}

// The entries of a row that are inside the support at y0 or at y1 = y0 + dt v0 are known before the
// first pair pass (y1 moves with the velocities of y0), so the four passes of a step walk
// those alone: half of a Verlet row.  ENS_NEAR bits per particle say which, each lane of the G
// holding the bits of its own entries (lane, lane + G, ...), in order: a lane adds the terms it
// would add without them in the same order, the others being exact zeros, so the sums are the
// same to the bit.  Entries behind the first ENS_NEAR of a row are always walked.
constexpr int ENS_NEAR = 256;
template <int G> struct NearWord;
template <> struct NearWord<4> { using T = unsigned long long; };
template <> struct NearWord<8> { using T = unsigned int; };
template <> struct NearWord<16> { using T = unsigned short; };

// One lane's walk: the entry index and the neighbour two entries ahead, its position word one ahead.
template <int D, int G> struct EnsWalk {
    static constexpr int KM = ENS_NEAR / G;
    const int32_t* __restrict__ row;       // this lane's first entry
    const EnsSet& st;
    unsigned int bits, more;               // near entries from `base` on; with 64 per lane, the second half
    int base, tail, nk, j1, j2;            // j < 0: no entry
    float4 w1;
    __device__ __forceinline__ int next() {
        int k;
        if (KM > 32 && !bits) { bits = more; more = 0; base += 32; }
        if (bits) {
            k = base + __ffs((int)bits) - 1;
            bits &= bits - 1;
        } else {
            k = tail++;
        }
        return k < nk ? __ldg(row + k * G) : -1;
    }
    __device__ __forceinline__ EnsWalk(const EnsArgs& a, const EnsSet& s, int i, int lane) : st(s) {
        row = a.list + a.offs[i] + lane;
        nk = (a.cnt[i] - lane + G - 1) / G;
        tail = KM;
        const auto near = static_cast<const typename NearWord<G>::T*>(a.near)[(size_t)i * G + lane];
        bits = (unsigned int)near;
        more = KM > 32 ? (unsigned int)((unsigned long long)near >> 32) : 0u;
        base = 0;
        j1 = next();
        j2 = next();
        w1 = get_x_word<D>(st, j1 < 0 ? 0 : j1);
    }
    __device__ __forceinline__ bool take(int& j, float4& w) {
        j = j1;
        w = w1;
        j1 = j2;
        if (j >= 0) {
            w1 = get_x_word<D>(st, j1 < 0 ? 0 : j1);
            j2 = j1 < 0 ? -1 : next();
        }
        return j >= 0;
    }
};

// The bits of this lane's entries.  x1_ij = x_ij + dt (v_i - v_j) up to the rounding of the positions,
// which the limit allows for.
template <int D, int G>
__device__ __forceinline__ void ens_near(int i, int lane, const EnsArgs& a, const EnsSet& st) {
    using T = typename NearWord<G>::T;
    const float4 wi = get_x_word<D>(st, i);
    const Vec<D> xi = vec_of_word<D>(wi), vi = get_v<D>(st, i, wi);
    const float Hi = a.H[i], dt = a.box_dt[a.box_of[i]];
    float scale = 0.f;
    #pragma unroll
    for (int c = 0; c < D; ++c) scale = fmaxf(scale, fabsf(xi.v[c]) + a.P.dom.L[c]);
    const float slack = 1e-6f * scale;
    const int nk = min((a.cnt[i] - lane + G - 1) / G, ENS_NEAR / G);
    const int32_t* row = a.list + a.offs[i] + lane;
    T bits = 0;
    int jn = nk > 0 ? __ldg(row) : 0;
    #pragma unroll 2
    for (int k = 0; k < nk; ++k) {
        const int j = jn;
        if (k + 1 < nk) jn = __ldg(row + (k + 1) * G);
        const float4 wj = get_x_word<D>(st, j);
        const Vec<D> vj = get_v<D>(st, j, wj);
        const float lim = fmaf(fmaxf(Hi, __ldg(a.H + j)), 1.0001f, slack), lim2 = lim * lim;
        const Vec<D> d0 = pair_vec<D>(xi, vec_of_word<D>(wj), a.P.dom);
        Vec<D> d1;
        #pragma unroll
        for (int c = 0; c < D; ++c) d1.v[c] = fmaf(dt, vi.v[c] - vj.v[c], d0.v[c]);
        const bool far = dot<D>(d0, d0) >= lim2 && dot<D>(d1, d1) >= lim2;       // NaN is near
        bits |= (T)((T)(!far) << k);
    }
    static_cast<T*>(a.near)[(size_t)i * G + lane] = bits;
}

// What a pair needs of the larger support.
template <int KF, int D> struct EnsSupport {
    float H, rH, HH, rHH, cH;
    __device__ __forceinline__ explicit EnsSupport(float h)
        : H(h), rH(1.f / h), HH(h * h), rHH(1.f / (h * h)), cH(KernelTraits<KF, D>::C / ipow<D>(h)) {}
};
// gradW(x_ij, max(H_i, H_j)) as kernelWG gives it; false outside the support.
template <int KF, int D>
__device__ __forceinline__ bool ens_grad(const Vec<D>& xij, float r, const EnsSupport<KF, D>& hi, float Hj, Vec<D>& gW) {
    EnsSupport<KF, D> h = hi;
    if (Hj > hi.H) h = EnsSupport<KF, D>(Hj);
    const float q = div_markstein(r, h.H, h.rH);
    if (q >= 1.f) return false;
    float k, p;
    kernel_kp<KF, D>(q, k, p);
    const float s = div_markstein(-h.cH * p, h.HH, h.rHH);
    #pragma unroll
    for (int a = 0; a < D; ++a) gW.v[a] = s * xij.v[a];
    return true;
}

// Pass A (passA_partial over the near entries).
template <int KF, int D, int G>
__device__ __forceinline__ void ens_passA(int i, int lane, const EnsArgs& a, const EnsSet& st, Mat<D>& M, Vec<D>& g) {
    const Vec<D> xi = vec_of_word<D>(get_x_word<D>(st, i));
    const float4 si = st.sv[i];
    const float rhoi = si.x;
    const EnsSupport<KF, D> hi(si.z);
    EnsWalk<D, G> walk(a, st, i, lane);
    int j;
    float4 w;
    while (walk.take(j, w)) {
        const float4 sj = st.sv[j];
        const Vec<D> xij = pair_vec<D>(xi, vec_of_word<D>(w), a.P.dom);
        const float r = safe_sqrt(dot<D>(xij, xij));
        Vec<D> gW;
        if (!ens_grad<KF, D>(xij, r, hi, sj.z, gW)) continue;
        const float Vj = sj.y;
        const float dr = sj.x - rhoi;
        #pragma unroll
        for (int c = 0; c < D; ++c) {
            g.v[c] += Vj * dr * gW.v[c];
            #pragma unroll
            for (int e = 0; e < D; ++e) M.m[c][e] += Vj * gW.v[c] * (-xij.v[e]);
        }
    }
}

// Pass B (passB_partial over the near entries, without a free-surface indicator).
template <int KF, int D, int G, bool USUAL>
__device__ __forceinline__ void ens_passB(int i, int lane, const EnsArgs& a, const EnsSet& st, float& cont, float& dd, Vec<D>& pf,
                                          Vec<D>& visc) {
    const WcDev& W = a.W;
    const float4 wi = get_x_word<D>(st, i), si = st.sv[i], gi = a.gp[i];
    const Vec<D> xi = vec_of_word<D>(wi), vi = get_v<D>(st, i, wi), gLi = vec_of_word<D>(gi);
    const float rhoi = si.x, Pi = word_of(gi, D), Hi = si.z;
    const EnsSupport<KF, D> hi(Hi);
    const float eps = 1.0e-14f * Hi;
    const float factor = W.inviscid ? W.alpha * W.c0 * Hi / W.xi : W.visc_nu;
    EnsWalk<D, G> walk(a, st, i, lane);
    int j;
    float4 w;
    while (walk.take(j, w)) {
        const float4 sj = st.sv[j], gj = a.gp[j];
        const Vec<D> xij = pair_vec<D>(xi, vec_of_word<D>(w), a.P.dom);
        const float r2 = dot<D>(xij, xij);
        const float r = safe_sqrt(r2);
        Vec<D> gW;
        if (!ens_grad<KF, D>(xij, r, hi, sj.z, gW)) continue;
        const float rj = sj.x, Vj = sj.y;
        const Vec<D> vj = get_v<D>(st, j, w), gLj = vec_of_word<D>(gj);
        // continuity (inconsistent.py:19-31): V_j (v_j - v_i).gW
        float t = 0.f;
        #pragma unroll
        for (int c = 0; c < D; ++c) t += (vj.v[c] - vi.v[c]) * gW.v[c];
        cont += Vj * t;
        // density diffusion (wp_densityDelta.py:88-117)
        {
            const float inv = rcp_markstein(r + eps);
            const float s = 2.f * (rj - rhoi) * inv * inv;      // 2 (rho_j - rho_i) n_ij / (r + eps), n_ij = x_ij / (r + eps)
            float pd = 0.f;
            #pragma unroll
            for (int c = 0; c < D; ++c) {
                float psi;
                if (USUAL || W.density_scheme == SPH_DENSITY_DIFFUSION_DELTA) psi = (gLi.v[c] + gLj.v[c]) - s * xij.v[c];
                else if (W.density_scheme == SPH_DENSITY_DIFFUSION_DENSITY_ONLY) psi = -(s * xij.v[c]);
                else psi = gLi.v[c] + gLj.v[c];
                pd += psi * gW.v[c];
            }
            dd += Vj * pd;
        }
        // pressure (wp_surfaceAware.py:48-102)
        {
            const float Pj = word_of(gj, D);
            float pij;
            if (USUAL) pij = (Pi >= 0.f || Pj >= 0.f) ? Pj + Pi : Pj - Pi;
            else switch (W.pressure_term) {
                case SPH_PRESSURE_CONSERVATIVE: pij = Pj - Pi; break;
                case SPH_PRESSURE_NONCONSERVATIVE: pij = Pj + Pi; break;
                case SPH_PRESSURE_ANTUONO: pij = (Pi >= 0.f || Pj >= 0.f) ? Pj + Pi : Pj - Pi; break;
                case SPH_PRESSURE_I: pij = Pi; break;
                case SPH_PRESSURE_J: pij = Pj; break;
                default: pij = (Pj / (rj * rj) + Pi / (rhoi * rhoi)) * rj; break;
            }
            #pragma unroll
            for (int c = 0; c < D; ++c) pf.v[c] += Vj * pij * gW.v[c];
        }
        // velocity diffusion (wp_viscosityDelta.py:86-106)
        {
            float vx = 0.f;
            #pragma unroll
            for (int c = 0; c < D; ++c) vx += (vi.v[c] - vj.v[c]) * xij.v[c];
            const float rr = fmaxf(r2 + eps * Hi, 1.2e-38f);
            float mu = div_markstein(vx, rr, rcp_markstein(rr));
            mu = mu > 0.f ? 0.f : mu;
            const float rho_bar = (rj + rhoi) / 2.f;
            const float ww = div_markstein(Vj * mu * factor, rho_bar, rcp_markstein(rho_bar));
            #pragma unroll
            for (int c = 0; c < D; ++c) visc.v[c] += ww * gW.v[c];
        }
    }
}

// Bound by issue slots (64 %) and the latency of the gathers.  1.3 M particles in 64 boxes, 99 entries
// per row of which 50 interact: 5.84 -> 2.81 ms per step; of that the walk of the near entries, packed
// words and quotients hoisted to the particle give 2.2 ms, divisions without the general case's
// branches 0.3, the usual terms as constants 0.1, particles handed to free warps (1, 2 or 4 warpfuls
// at a time: 0.27, 0.21, 0.21) and 9 blocks of 128 threads per SM (56 registers; 8: 0.1 more, 10: 0.06
// more) the rest.  Rows reordered by distance were faster still (2.14 ms with static shares) but change
// the order of the sums: the Antuono pressure switch jumps where P_j crosses 0, so a rounding there
// moves whole pair terms.
template <int KF, int D, int G, int BLOCK>
__global__ void __launch_bounds__(BLOCK, (D == 3 ? 1 : 1152 / BLOCK))
k_ens_step(const __grid_constant__ EnsArgs a) {
    constexpr int PPW = 32 / G;            // particles of a warp at a time
    const int lane = threadIdx.x & (G - 1), sub = (threadIdx.x & 31) / G;
    unsigned int dmax = 0u, arrived = 0;
    // The particles of a pass go to the warps as they become free (rows differ in length, and a grid
    // barrier waits for the last), PPW at a time.
    auto take = [&](int pass) {
        int base = 0;
        if ((threadIdx.x & 31) == 0) base = atomicAdd(a.work + pass, PPW);
        return __shfl_sync(0xffffffffu, base, 0);
    };
    const bool usual = a.W.density_scheme == SPH_DENSITY_DIFFUSION_DELTA && a.W.pressure_term == SPH_PRESSURE_ANTUONO;
    // ---- the first stage's words
    for (int i = blockIdx.x * BLOCK + threadIdx.x; i < a.n; i += gridDim.x * BLOCK) {
        const float r = a.rho[i];
        put_xv<D>(a.set[0], i, load_vec<D>(a.x, i), load_vec<D>(a.v, i));
        a.set[0].sv[i] = make_float4(r, a.m[i] / r, a.H[i], 0.f);
    }
    if (!grid_barrier(a.ctl, arrived)) { if (threadIdx.x == 0) atomicOr(a.status, SPH_STATUS_TIMEOUT); return; }
    for (int stage = 0; stage < 2; ++stage) {
        const EnsSet& st = a.set[stage];
        // ---- pass A: renormalised density gradient and EOS
        for (int base = take(2 * stage); base < a.n; base = take(2 * stage)) {
            const int i = base + sub;
            const bool valid = i < a.n;
            Mat<D> M = mzero<D>();
            Vec<D> s = vzero<D>();
            if (valid) {
                if (stage == 0) ens_near<D, G>(i, lane, a, st);
                ens_passA<KF, D, G>(i, lane, a, st, M, s);
            }
            passA_reduce<D, G>(M, s);
            if (valid && lane == 0) {
                const Vec<D> g = renormalise<D>(M, s);
                const float Pr = wc_eos(a.W, st.sv[i].x);
                float w[4] = {0.f, 0.f, 0.f, 0.f};
                #pragma unroll
                for (int c = 0; c < D; ++c) w[c] = g.v[c];
                w[D] = Pr;
                a.gp[i] = make_float4(w[0], w[1], w[2], w[3]);
            }
        }
        if (!grid_barrier(a.ctl, arrived)) { if (threadIdx.x == 0) atomicOr(a.status, SPH_STATUS_TIMEOUT); return; }
        // ---- pass B: right-hand side, stage update
        for (int base = take(2 * stage + 1); base < a.n; base = take(2 * stage + 1)) {
            const int i = base + sub;
            const bool valid = i < a.n;
            float cont = 0.f, dd = 0.f;
            Vec<D> pf = vzero<D>(), visc = vzero<D>();
            if (valid) {
                if (usual) ens_passB<KF, D, G, true>(i, lane, a, st, cont, dd, pf, visc);
                else ens_passB<KF, D, G, false>(i, lane, a, st, cont, dd, pf, visc);
            }
            cont = gsum<G>(cont); dd = gsum<G>(dd);
            #pragma unroll
            for (int c = 0; c < D; ++c) { pf.v[c] = gsum<G>(pf.v[c]); visc.v[c] = gsum<G>(visc.v[c]); }
            if (valid && lane == 0) {
                float dr; Vec<D> dv;
                passB_finish<D>(a.W, st.sv[i].x, a.H[i], cont, dd, pf, visc, dr, dv);
                const float dt = a.box_dt[a.box_of[i]];
                const float4 w0 = get_x_word<D>(a.set[0], i);
                const Vec<D> x0 = vec_of_word<D>(w0), v0 = get_v<D>(a.set[0], i, w0);
                const float r0 = a.set[0].sv[i].x;
                if (stage == 0) {
                    Vec<D> xn, vn;
                    #pragma unroll
                    for (int c = 0; c < D; ++c) { xn.v[c] = x0.v[c] + dt * v0.v[c]; vn.v[c] = v0.v[c] + dt * dv.v[c]; }
                    const float rn = r0 + dt * dr;
                    put_xv<D>(a.set[1], i, wrap_pos<D>(xn, a.P.dom), vn);
                    a.set[1].sv[i] = make_float4(rn, a.m[i] / rn, a.H[i], 0.f);
                    store_vec<D>(a.dv1, i, dv);
                    a.drho1[i] = dr;
                } else {
                    const Vec<D> v1 = get_v<D>(st, i, get_x_word<D>(st, i)), k1 = load_vec_cg<D>(a.dv1, i);
                    const float h = 0.5f * dt;
                    Vec<D> xn, vn;
                    #pragma unroll
                    for (int c = 0; c < D; ++c) { xn.v[c] = x0.v[c] + h * (v0.v[c] + v1.v[c]); vn.v[c] = v0.v[c] + h * (k1.v[c] + dv.v[c]); }
                    xn = wrap_pos<D>(xn, a.P.dom);
                    store_vec<D>(a.x, i, xn);
                    store_vec<D>(a.v, i, vn);
                    a.rho[i] = r0 + h * (__ldcg(a.drho1 + i) + dr);
                    const Vec<D> db = dist_vec<D>(xn, load_vec<D>(a.x_build, i), a.P.dom);
                    dmax = max(dmax, ens_ord(sqrtf(dot<D>(db, db)) / a.H[i]));   // in supports
                }
            }
        }
        if (stage == 0 && !grid_barrier(a.ctl, arrived)) { if (threadIdx.x == 0) atomicOr(a.status, SPH_STATUS_TIMEOUT); return; }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) dmax = max(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    if ((threadIdx.x & 31) == 0 && dmax) atomicMax(a.disp, dmax);
}

template <int KF, int D, int G, int BLOCK>
static int launch_ens(EnsArgs& a, cudaStream_t s) {
    static std::mutex mu;
    static int cached_dev = -1, bps = 0, sms = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "ensemble step: cudaGetDevice: %s", cudaGetErrorString(e));
    {
        std::lock_guard<std::mutex> lock(mu);
        if (cached_dev != dev) {
            int coop = 0;
            if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
                return set_error(SPH_ERR_UNSUPPORTED, "ensemble step: device %d has no cooperative launch", dev);
            if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
                return set_error(SPH_ERR_CUDA, "ensemble step: SM count");
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_ens_step<KF, D, G, BLOCK>, BLOCK, 0) != cudaSuccess || bps < 1)
                return set_error(SPH_ERR_CUDA, "ensemble step: occupancy query failed");
            cached_dev = dev;
        }
    }
    const int64_t need = (a.n + BLOCK / G - 1) / (BLOCK / G);
    const int grid = (int)std::min<int64_t>(need, (int64_t)bps * sms);
    void* args[] = {&a};
    count_launch();
    e = cudaLaunchCooperativeKernel((const void*)k_ens_step<KF, D, G, BLOCK>, dim3(grid), dim3(BLOCK), args, 0, s);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "ensemble step: cooperative launch: %s", cudaGetErrorString(e));
    return SPH_OK;
}

}  // namespace wsph

using namespace wsph;

extern "C" {

int64_t sph_ensemble_neighbors_workspace_size(int64_t n, int64_t total_cells) {
    if (n < 0 || total_cells < 1) return -1;
    return ens_carve(nullptr, n, total_cells).bytes;
}

int sph_ensemble_neighbors_build(const SphParams* p, int64_t n, int32_t nbox, const int32_t* box_of, const int32_t* box_grid,
                                 const int32_t* box_cell_base, int64_t total_cells, const float* x, const float* H, void* workspace,
                                 int64_t workspace_bytes, int32_t* offs, int32_t* cnt, int32_t* list, int64_t list_capacity,
                                 int64_t* nnz_out, int32_t* status, void* stream) {
    DevParams P;
    int rc = params_to_dev(p, &P);
    if (rc) return rc;
    if (n < 0 || n > 0x7fffffff || nbox < 1 || total_cells < 1 || total_cells > 0x7fffffff)
        return set_error(SPH_ERR_BAD_ARG, "sph_ensemble_neighbors_build: bad sizes");
    WSPH_CHECK_PTR(nnz_out); WSPH_CHECK_PTR(status);
    cudaStream_t s = WSPH_STREAM(stream);
    if (n == 0) { cudaMemsetAsync(nnz_out, 0, 8, s); return check_launch("sph_ensemble_neighbors_build"); }
    WSPH_CHECK_PTR(box_of); WSPH_CHECK_PTR(box_grid); WSPH_CHECK_PTR(box_cell_base); WSPH_CHECK_PTR(x); WSPH_CHECK_PTR(H);
    WSPH_CHECK_PTR(workspace); WSPH_CHECK_PTR(offs); WSPH_CHECK_PTR(cnt);
    if (list_capacity > 0) WSPH_CHECK_PTR(list);
    if (P.dim == 2 && (reinterpret_cast<uintptr_t>(x) & 7)) return set_error(SPH_ERR_BAD_ARG, "positions must be 8-byte aligned in 2D");
    EnsNbWs w = ens_carve(static_cast<char*>(workspace), n, total_cells);
    if (workspace_bytes < w.bytes) return set_error(SPH_ERR_WORKSPACE, "ensemble neighbour workspace %lld < %lld", (long long)workspace_bytes,
                                                    (long long)w.bytes);
    cudaMemsetAsync(w.counts, 0, total_cells * 4, s);
    count_launch();
    WSPH_DISPATCH_DIM(P.dim, (k_ens_keys<D><<<grid_for(n, 256), 256, 0, s>>>((int)n, P.dom, x, box_of, box_grid, box_cell_base, w.keys,
                                                                              w.slot, w.counts)));
    exclusive_scan_i32(w.counts, w.start, total_cells, w.scan, w.total, s);
    count_launch();
    k_ens_scatter<<<grid_for(n, 256), 256, 0, s>>>((int)n, w.keys, w.slot, w.start, w.sorted);
    count_launch();
    k_ens_sort_cells<<<grid_for(total_cells, 256), 256, 0, s>>>(total_cells, w.start, w.counts, w.sorted);
    count_launch();
    WSPH_DISPATCH_DIM(P.dim, (k_ens_pack_sorted<D><<<grid_for(n, 256), 256, 0, s>>>((int)n, x, H, w.sorted, w.words)));
    constexpr int GE = 8;
    count_launch();
    WSPH_DISPATCH_DIM(P.dim, (k_ens_verlet<D, GE, false><<<grid_for(n * GE, 128), 128, 0, s>>>(
        (int)n, P, x, H, box_of, box_grid, box_cell_base, w.start, w.counts, w.sorted, w.words, cnt, nullptr, nullptr, nullptr, 0)));
    exclusive_scan_i32(cnt, offs, n, w.scan, reinterpret_cast<long long*>(nnz_out), s);
    count_launch();
    k_ens_check<<<1, 1, 0, s>>>(reinterpret_cast<long long*>(nnz_out), list_capacity, status);
    count_launch();
    WSPH_DISPATCH_DIM(P.dim, (k_ens_verlet<D, GE, true><<<grid_for(n * GE, 128), 128, 0, s>>>(
        (int)n, P, x, H, box_of, box_grid, box_cell_base, w.start, w.counts, w.sorted, w.words, nullptr, offs, list,
        reinterpret_cast<long long*>(nnz_out), list_capacity)));
    return check_launch("sph_ensemble_neighbors_build");
}

int64_t sph_ensemble_step_workspace_size(int64_t n, int32_t dim) {
    if (n < 0 || dim < 1 || dim > 3) return -1;
    // control block, xv (twice in 3D) and sv of two stages, gp, the near bits, dv1 (n*dim), drho1 (n)
    return 256 + ((dim == 3 ? 4 : 2) + 2 + 1) * al256(n * 16) + al256(n * (ENS_NEAR / 8)) + al256(n * dim * 4) + al256(n * 4);
}

int sph_ensemble_step(const SphParams* p, const SphWcParams* wc, int64_t n, const int32_t* box_of, const float* box_dt,
                      const float* H, const float* m, float* x, float* v, float* rho, const float* x_build, const int32_t* offs,
                      const int32_t* cnt, const int32_t* list, void* workspace, int64_t workspace_bytes, int32_t lanes,
                      int32_t block, uint32_t* disp_max, int32_t* status, void* stream) {
    DevParams P;
    int rc = params_to_dev(p, &P);
    if (rc) return rc;
    if (n < 0 || n > 0x3fffffff) return set_error(SPH_ERR_BAD_ARG, "sph_ensemble_step: n out of range");
    if (n == 0) return SPH_OK;
    WSPH_CHECK_PTR(wc); WSPH_CHECK_PTR(box_of); WSPH_CHECK_PTR(box_dt); WSPH_CHECK_PTR(H); WSPH_CHECK_PTR(m); WSPH_CHECK_PTR(x);
    WSPH_CHECK_PTR(v); WSPH_CHECK_PTR(rho); WSPH_CHECK_PTR(x_build); WSPH_CHECK_PTR(offs); WSPH_CHECK_PTR(cnt); WSPH_CHECK_PTR(list);
    WSPH_CHECK_PTR(workspace); WSPH_CHECK_PTR(disp_max); WSPH_CHECK_PTR(status);
    WcDev W;
    if ((rc = wc_to_dev(wc, P, &W))) return rc;
    if (workspace_bytes < sph_ensemble_step_workspace_size(n, P.dim)) return set_error(SPH_ERR_WORKSPACE, "sph_ensemble_step: workspace too small");
    if (reinterpret_cast<uintptr_t>(workspace) & 255) return set_error(SPH_ERR_BAD_ARG, "sph_ensemble_step: workspace must be 256-byte aligned");
    if (P.dim == 2 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(x_build)) & 7))
        return set_error(SPH_ERR_BAD_ARG, "vectors must be 8-byte aligned in 2D");
    cudaStream_t s = WSPH_STREAM(stream);
    char* w = static_cast<char*>(workspace);
    EnsArgs a;
    a.n = (int)n; a.P = P; a.W = W; a.box_of = box_of; a.box_dt = box_dt; a.H = H; a.m = m; a.x_build = x_build;
    a.x = x; a.v = v; a.rho = rho;
    int64_t o = 256;
    const int64_t qb = al256(n * 16);
    for (EnsSet& q : a.set) {
        q.xv = reinterpret_cast<float4*>(w + o); o += P.dim == 3 ? 2 * qb : qb;
        q.sv = reinterpret_cast<float4*>(w + o); o += qb;
    }
    a.gp = reinterpret_cast<float4*>(w + o); o += qb;
    a.near = w + o; o += al256(n * (ENS_NEAR / 8));
    a.dv1 = reinterpret_cast<float*>(w + o); o += al256(n * P.dim * 4);
    a.drho1 = reinterpret_cast<float*>(w + o);
    a.offs = offs; a.cnt = cnt; a.list = list;
    a.ctl = reinterpret_cast<BarrierCtl*>(w);
    a.work = reinterpret_cast<int*>(w + 128);
    static_assert(sizeof(BarrierCtl) <= 128, "the control block's two halves");
    a.disp = disp_max; a.status = status;
    cudaError_t e = cudaMemsetAsync(a.ctl, 0, 128 + 4 * sizeof(int), s);
    if (e != cudaSuccess) return set_error(SPH_ERR_CUDA, "sph_ensemble_step: memset: %s", cudaGetErrorString(e));
    if (!(lanes == 4 || lanes == 8 || lanes == 16) || !(block == 128 || block == 256))
        return set_error(SPH_ERR_BAD_ARG, "sph_ensemble_step: lanes must be 4, 8 or 16 and block 128 or 256");
    rc = SPH_ERR_UNSUPPORTED;
#define ENS_LAUNCH(GL, BL) WSPH_DISPATCH_KD(P.kernel, P.dim, (rc = launch_ens<KF, D, GL, BL>(a, s)))
    if (lanes == 4 && block == 128) { ENS_LAUNCH(4, 128); }
    else if (lanes == 4) { ENS_LAUNCH(4, 256); }
    else if (lanes == 8 && block == 128) { ENS_LAUNCH(8, 128); }
    else if (lanes == 8) { ENS_LAUNCH(8, 256); }
    else if (block == 128) { ENS_LAUNCH(16, 128); }
    else { ENS_LAUNCH(16, 256); }
#undef ENS_LAUNCH
    return rc;
}

}  // extern "C"
