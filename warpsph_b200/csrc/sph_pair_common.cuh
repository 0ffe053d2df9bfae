// Shared pieces of the pair passes: G lanes of a warp per particle, row-entry
// decoding (Verlet rows or their interacting prefixes), kernel
// evaluation with a precomputed 1/H, group reductions, and the host-side argument
// checks and template dispatch of the pair entry points.
#pragma once
#include <cstring>
#include <cuda_runtime.h>
#include "sph_common.cuh"

namespace wsph {

constexpr int PAIR_BLOCK = 128;

// ---------------------------------------------------------------- group helpers
template <int G> struct Grp {
    int i, lane;
    bool valid;
    __device__ __forceinline__ explicit Grp(int n) {
        int t = blockIdx.x * blockDim.x + threadIdx.x;
        i = t / G;
        lane = threadIdx.x & (G - 1);
        valid = i < n;
    }
};
template <int G> __device__ __forceinline__ float gsum(float v) {
    #pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int G> __device__ __forceinline__ float gmaxw(float v) {
    #pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = wmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// Row entry q: neighbour j and the Verlet entry index k that pairwise arrays use (the
// rows a pass walks are Verlet rows or their interacting prefixes, so k = q).
__device__ __forceinline__ void entry(const int32_t* __restrict__ list, int q, int& j, int& k) {
    j = __ldg(list + q); k = q;
}
// One lane's walk over a row (entries q0, q0 + step, ... < e) with the neighbour index loaded
// two entries ahead and the neighbour's D-vector from `src` one entry ahead: the dependent
// global loads of an entry are in flight while the entry before it is computed.  Past the
// row's end the prefetches read index 0 (a valid particle whenever a row is walked).
template <int D> struct RowPipe {
    const int32_t* __restrict__ list;
    const float* __restrict__ src;
    int e, step, j1, j2;
    Vec<D> v1;
    __device__ __forceinline__ RowPipe(const int32_t* __restrict__ l, const float* __restrict__ s, int q0, int e_, int st)
        : list(l), src(s), e(e_), step(st) {
        j1 = q0 < e_ ? __ldg(l + q0) : 0;
        j2 = q0 + st < e_ ? __ldg(l + q0 + st) : 0;
        v1 = load_vec<D>(s, j1);
    }
    // the entry at q (the caller's loop index, q0 + k * step): its neighbour and vector
    __device__ __forceinline__ void take(int q, int& j, Vec<D>& vj) {
        j = j1;
        vj = v1;
        j1 = j2;
        v1 = load_vec<D>(src, j1);
        j2 = q + 2 * step < e ? __ldg(list + q + 2 * step) : 0;
    }
};

// The same walk over 16-byte words (positions packed with the support, k_pack_xh).
struct WordPipe {
    const int32_t* __restrict__ list;
    const float4* __restrict__ src;
    int e, step, j1, j2;
    float4 v1;
    __device__ __forceinline__ WordPipe(const int32_t* __restrict__ l, const float4* __restrict__ s, int q0, int e_, int st)
        : list(l), src(s), e(e_), step(st) {
        j1 = q0 < e_ ? __ldg(l + q0) : 0;
        j2 = q0 + st < e_ ? __ldg(l + q0 + st) : 0;
        v1 = __ldg(s + j1);
    }
    __device__ __forceinline__ void take(int q, int& j, float4& t) {
        j = j1;
        t = v1;
        j1 = j2;
        v1 = __ldg(src + j1);
        j2 = q + 2 * step < e ? __ldg(list + q + 2 * step) : 0;
    }
};

// The row walk of a pass over packed words or over separate arrays.
template <int D, bool PK> struct PairPipe {
    using T = RowPipe<D>;
    static __device__ __forceinline__ const float* src(const float* x, const float4*) { return x; }
};
template <int D> struct PairPipe<D, true> {
    using T = WordPipe;
    static __device__ __forceinline__ const float4* src(const float*, const float4* xh) { return xh; }
};

// Packed words of the CRK right-hand side, one 16-byte gather each:
//   xh   position and, behind it, the support; in 1D and 2D its reciprocal in the last word
//   fv   velocity, then (1D, 2D) V and m / rho in words 2 and 3; in 3D V in the last word and
//        m / rho in an array of its own
//   fc   velocity, then (1D, 2D) the sound speed and m sgn(div v) in words 2 and 3; in 3D the sound
//        speed in the last word and m sgn(div v) in an array of its own
__device__ __forceinline__ float word_of(const float4& t, int a) { return a == 0 ? t.x : (a == 1 ? t.y : (a == 2 ? t.z : t.w)); }
template <int D> __device__ __forceinline__ Vec<D> vec_of_word(const float4& t) {
    Vec<D> r;
    #pragma unroll
    for (int a = 0; a < D; ++a) r.v[a] = word_of(t, a);
    return r;
}
template <int D> __device__ __forceinline__ float support_of(const float4& xh) { return word_of(xh, D); }
template <int D> __device__ __forceinline__ float inv_support_of(const float4& xh) {
    if constexpr (D == 3) return rcp_newton(xh.w);
    else return xh.w;
}
template <int D> __device__ __forceinline__ float4 make_xh(const Vec<D>& x, float H) {
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    #pragma unroll
    for (int a = 0; a < D; ++a) w[a] = x.v[a];
    w[D] = H;
    if (D < 3) w[3] = 1.f / H;
    return make_float4(w[0], w[1], w[2], w[3]);
}
// (v, s, t) of fv and fc: word 2 and 3 below 3D, else the last word and `third`.
template <int D> __device__ __forceinline__ float4 make_flow(const Vec<D>& v, float s, float t) {
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    #pragma unroll
    for (int a = 0; a < D; ++a) w[a] = v.v[a];
    if (D < 3) { w[2] = s; w[3] = t; } else { w[3] = s; }
    return make_float4(w[0], w[1], w[2], w[3]);
}

template <int G> __host__ __forceinline__ int grid_g(int64_t n) { return (int)((n * G + PAIR_BLOCK - 1) / PAIR_BLOCK); }

// W and grad_i W with a precomputed 1/H.
template <int KF, int D> __device__ __forceinline__ float kW_inv(float r, float invH) {
    float q = r * invH;
    if (!(q < 1.f)) return 0.f;
    float k, p; kernel_kp<KF, D>(q, k, p);
    return KernelTraits<KF, D>::C * ipow<D>(invH) * k;
}
template <int KF, int D> __device__ __forceinline__ void kWG_inv(const Vec<D>& x, float r, float invH, float& W, Vec<D>& g) {
    float q = r * invH;
    if (!(q < 1.f)) { W = 0.f; g = vzero<D>(); return; }
    float k, p; kernel_kp<KF, D>(q, k, p);
    float cH = KernelTraits<KF, D>::C * ipow<D>(invH);
    W = cH * k;
    float s = -cH * p * (invH * invH);
    #pragma unroll
    for (int a = 0; a < D; ++a) g.v[a] = s * x.v[a];
}

// W and s with grad_i W = s x_ij; false (and zeros) outside the support.
template <int KF, int D> __device__ __forceinline__ bool kWS_inv(float r, float invH, float& W, float& s) {
    const float q = r * invH;
    if (!(q < 1.f)) { W = 0.f; s = 0.f; return false; }
    float k, p; kernel_kp<KF, D>(q, k, p);
    const float cH = KernelTraits<KF, D>::C * ipow<D>(invH);
    W = cH * k;
    s = -cH * p * (invH * invH);
    return true;
}
// CRK-corrected kernel gradient (Frontiere, Raskin & Owen 2017, eq. for d W^R_ij) of
// W^R = A (1 + B.x) W, x = x_ij, with grad W = s x and gB[a][g] = dB^a/dx^g:
//   A (1 + B.x) s x + W (gA (1 + B.x) + A (B + gB^T x))
template <int D> __device__ __forceinline__ Vec<D> crk_grad_s(const Vec<D>& x, float W, float s, float A, const Vec<D>& B,
                                                              const Vec<D>& gA, const Mat<D>& gB) {
    const float bx = 1.f + dot<D>(B, x), cx = A * bx * s, AW = A * W, bW = bx * W;
    Vec<D> r;
    #pragma unroll
    for (int g = 0; g < D; ++g) {
        float t = B.v[g];
        #pragma unroll
        for (int a = 0; a < D; ++a) t += gB.m[a][g] * x.v[a];
        r.v[g] = cx * x.v[g] + (gA.v[g] * bW + AW * t);
    }
    return r;
}

// Neumaier-compensated accumulator (DevParams::kahan).
struct KSum {
    float s, c;
    __device__ __forceinline__ void init() { s = 0.f; c = 0.f; }
    __device__ __forceinline__ void add(float x, bool comp) {
        if (!comp) { s += x; return; }
        float t = s + x;
        if (fabsf(s) >= fabsf(x)) c += (s - t) + x; else c += (x - t) + s;
        s = t;
    }
};

// Lanes per particle.  The sums of long rows want few lanes (no lane idles, few shuffles), streams
// of pair arrays more (contiguous rows), and a particle set that does not fill the chip wants many:
// below WIDE_LIMIT particles (64 per SM) a pass is a chain of dependent loads, shorter with 16 lanes.
// Microseconds per launch with 4 / 8 / 16 / 32 lanes (Wendland C4; 2D 32, 3D 128 neighbours):
//                        2D 262,144              3D 884,736                 2D 4,096
//   CRK accel            173 / 184 / 234 / 329   3189 / 2832 / 2911 / 3381  12.9 / 8.3 / 6.7 / 7.1
//   energy partition     103 /  88 /  94 / 114   1731 / 1366 / 1213 / 1255  10.8 / 6.9 / 4.9 / 4.0
//   velocity gradient     63 /  70 /  99 / 159    688 /  723 /  844 / 1126   6.0 / 4.7 / 4.3 / 4.6
//   Cullen switch         79 /  85 / 100 / 149   1291 / 1190 / 1135 / 1185   7.7 / 5.4 / 4.5 / 4.5
//   CRK factors           59 /  78 / 127 / 226    718 /  818 / 1072 / 1628   6.8 / 5.2 / 5.0 / 6.3
//   adaptive support      47 /  52 /  70 / 108   1014 / 1049 / 1101 / 1288   6.2 / 4.5 / 4.0 / 3.9
// Up to MID_LIMIT particles (112 per SM) the passes that take 4 lanes above it run with 8, for twice the
// warps.  Microseconds with 4 / 8 / 16 lanes (3D: 64 neighbours):
//                        2D 10,000            2D 16,384            2D 25,600            3D 10,648
//   CRK accel            13.5 /  9.7 / 11.7   14.9 / 11.6 / 14.7   17.1 / 18.2 / 21.8
//   velocity gradient     6.5 /  5.6 /  6.0    7.0 /  6.6 /  8.3    8.3 /  9.7 / 11.2    9.6 / 9.0 /  9.9
//   Cullen switch         8.2 /  6.0 /  6.1    8.4 /  7.3 /  9.7    9.7 / 10.3 / 12.4
//   CRK factors           7.1 /  6.1 /  7.6    7.8 /  7.6 / 10.6    8.8 / 11.3 / 15.2   10.9 / 9.8 / 12.7
//   adaptive support      6.5 /  4.7 /  4.9    6.8 /  5.6 /  6.5    7.0 /  7.3 /  9.2    9.7 / 6.9 /  7.4
//   CompSPH prep          6.6 /  4.9 /  5.0    6.6 /  5.6 /  7.4    7.1 /  7.3 /  9.1    9.4 / 7.2 /  7.2
// Six recorded steps in 2D, 4 against 8 lanes, with 20 / 32 / 50 neighbours: 14,400 particles 1209 / 1345 / 1653
// against 1214 / 1307 / 1547 us, 16,384 particles 1233 / 1512 / 1737 against 1237 / 1450 / 1564, 17,956 particles
// 1267 / 1550 / 1770 against 1286 / 1535 / 1635.
#ifndef G_LIGHT
#define G_LIGHT 8
#endif
#ifndef G_HEAVY
#define G_HEAVY 8
#endif
#ifndef G_CRK
#define G_CRK 4
#endif
// Light gather passes that walk long rows (CRK volume and the unpacked passes).
#define G_SCAN(D) ((D) == 3 ? 4 : G_LIGHT)
#define G_ACCEL(D) ((D) == 3 ? 8 : 4)
#define G_BALANCE(D) ((D) == 3 ? 16 : 8)
#define G_GRADV(D) 4
#define G_CULLEN(D) ((D) == 3 ? 16 : 4)
#define G_ADAPT(D) 4
constexpr int64_t WIDE_LIMIT = 148 * 64;
constexpr int64_t MID_LIMIT = 148 * 112;
#define G_WIDE 16
#define G_MID 8
// Runs the launch with LG lanes per particle: BASE, at least G_MID up to MID_LIMIT particles, or WIDE
// for small particle sets.
#define PAIR_LANES(n, BASE, WIDE, ...)                               \
    do {                                                             \
        if ((n) <= WIDE_LIMIT) { constexpr int LG = WIDE; __VA_ARGS__; } \
        else if ((n) <= MID_LIMIT) { constexpr int LG = (BASE) < G_MID ? G_MID : (BASE); __VA_ARGS__; } \
        else { constexpr int LG = BASE; __VA_ARGS__; }               \
    } while (0)

#define WSPH_DISPATCH_KDS(params, ...) WSPH_DISPATCH_KD(P.kernel, P.dim, __VA_ARGS__)
#define WSPH_DISPATCH_DS(params, ...) WSPH_DISPATCH_DIM(P.dim, __VA_ARGS__)

// Launch with programmatic stream serialization (the kernel must begin with pdl_entry()).
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    memset(at, 0, sizeof(at));
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kern, args...);
}

#define PAIR_PRELUDE()                                                        \
    DevParams P;                                                              \
    int rc = params_to_dev(p, &P);                                            \
    if (rc) return rc;                                                        \
    if (n < 0 || n > 0x3fffffff) return set_error(SPH_ERR_BAD_ARG, "%s: n out of range", __func__); \
    if (p->list_stride < 0 || p->list_stride > 1) return set_error(SPH_ERR_BAD_ARG, "%s: list_stride must be 1 (rows are Verlet rows or their interacting prefixes)", __func__); \
    if (n == 0) return SPH_OK;                                                \
    cudaStream_t s = WSPH_STREAM(stream);                                     \
    (void)s;

#define CHECK_CSR() do { WSPH_CHECK_PTR(offs); WSPH_CHECK_PTR(cnt); WSPH_CHECK_PTR(list); } while (0)

inline int check_align_vec(const DevParams& P, const void* ptr, const char* name) {
    if (P.dim == 2 && ptr && (reinterpret_cast<uintptr_t>(ptr) & 7))
        return set_error(SPH_ERR_BAD_ARG, "%s must be 8-byte aligned for dim 2", name);
    return SPH_OK;
}

}  // namespace wsph
