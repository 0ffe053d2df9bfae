// Learned warm start for the DFSPH pressure solves: a per-particle MLP
//   8 features -> 64 -> 64 -> 64 -> 1, ReLU hidden layers,
// with FP32 master parameters, BF16 weights and activations into the tensor cores and
// FP32 accumulation.  No counterpart in the reference: it replaces the initial pressure
// guess of modules/incompressible/divergenceFree.py:72 (0.75 p_prev) and
// modules/incompressible/incompressible.py:79 (0).
//
// Tensor-core tiles: mma.sync m16n8k16 (BF16 x BF16 -> FP32).  One warp owns 16 samples;
// a hidden layer is 8 n-tiles x (K/16) k-steps.  The FP32 accumulator fragment of one
// layer maps onto the BF16 A fragment of the next without leaving registers:
//   A(k-block kb) = { C(n-tile 2kb)[0:2], C(2kb)[2:4], C(2kb+1)[0:2], C(2kb+1)[2:4] }.
// The weight-gradient GEMMs dW_l = dZ_l^T H_{l-1} contract over the 16 samples of the warp;
// their operands are staged transposed in per-warp shared memory.
//
// Parameter vector (FP32, SPH_MLP_PARAM_COUNT floats):
//   W1[64][8] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] w4[64] b4[1]
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cstdint>
#include <mutex>
#include "sph_common.cuh"
#include "sph_tcgen05.cuh"

namespace wsph {

constexpr int MLP_IN = 8, MLP_H = 64;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + MLP_H * MLP_IN, OFF_W2 = OFF_B1 + MLP_H, OFF_B2 = OFF_W2 + MLP_H * MLP_H,
              OFF_W3 = OFF_B2 + MLP_H, OFF_B3 = OFF_W3 + MLP_H * MLP_H, OFF_W4 = OFF_B3 + MLP_H, OFF_B4 = OFF_W4 + MLP_H,
              MLP_NPARAM = OFF_B4 + 1;
static_assert(MLP_NPARAM == SPH_MLP_PARAM_COUNT, "parameter layout");
constexpr int MLP_WARPS = 4;
constexpr int MLP_THREADS = 32 * MLP_WARPS;
constexpr int K1 = 16;   // layer-1 K padded to one mma k-step

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t lds32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// Weights staged in shared memory as BF16.  W1s is [64][16] (K zero padded); WT are the
// transposes used by the backward data GEMMs.
struct MlpSmemW {
    __nv_bfloat16 W1[MLP_H * K1];
    __nv_bfloat16 W2[MLP_H * MLP_H];
    __nv_bfloat16 W3[MLP_H * MLP_H];
    float b1[MLP_H], b2[MLP_H], b3[MLP_H], w4[MLP_H];
    float b4;
};

__device__ void stage_weights(const float* __restrict__ prm, MlpSmemW& s, __nv_bfloat16* W2T, __nv_bfloat16* W3T) {
    for (int t = threadIdx.x; t < MLP_H * K1; t += blockDim.x) {
        const int nrow = t / K1, k = t % K1;
        s.W1[t] = __float2bfloat16_rn(k < MLP_IN ? prm[OFF_W1 + nrow * MLP_IN + k] : 0.f);
    }
    for (int t = threadIdx.x; t < MLP_H * MLP_H; t += blockDim.x) {
        const int r = t / MLP_H, c = t % MLP_H;
        const __nv_bfloat16 w2 = __float2bfloat16_rn(prm[OFF_W2 + t]), w3 = __float2bfloat16_rn(prm[OFF_W3 + t]);
        s.W2[t] = w2;
        s.W3[t] = w3;
        if (W2T) { W2T[c * MLP_H + r] = w2; W3T[c * MLP_H + r] = w3; }
    }
    for (int t = threadIdx.x; t < MLP_H; t += blockDim.x) {
        s.b1[t] = prm[OFF_B1 + t]; s.b2[t] = prm[OFF_B2 + t]; s.b3[t] = prm[OFF_B3 + t]; s.w4[t] = prm[OFF_W4 + t];
    }
    if (threadIdx.x == 0) s.b4 = prm[OFF_B4];
}

// One hidden layer with K = 64: C[nt] = A x W^T (W row-major [64 out][64 in]) + bias, ReLU.
__device__ __forceinline__ void hidden_layer(const uint32_t (&A)[4][4], const __nv_bfloat16* W, const float* bias, int g, int t,
                                             float (&h)[8][4]) {
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        const __nv_bfloat16* wr = W + (nt * 8 + g) * MLP_H + 2 * t;
        #pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_bf16(c, A[ks][0], A[ks][1], A[ks][2], A[ks][3], lds32(wr + ks * 16), lds32(wr + ks * 16 + 8));
        const float bb0 = bias[nt * 8 + 2 * t], bb1 = bias[nt * 8 + 2 * t + 1];
        h[nt][0] = fmaxf(c[0] + bb0, 0.f); h[nt][1] = fmaxf(c[1] + bb1, 0.f);
        h[nt][2] = fmaxf(c[2] + bb0, 0.f); h[nt][3] = fmaxf(c[3] + bb1, 0.f);
    }
}
__device__ __forceinline__ void c_to_a(const float (&h)[8][4], uint32_t (&A)[4][4]) {
    #pragma unroll
    for (int kb = 0; kb < 4; ++kb) {
        A[kb][0] = pack_bf16(h[2 * kb][0], h[2 * kb][1]);
        A[kb][1] = pack_bf16(h[2 * kb][2], h[2 * kb][3]);
        A[kb][2] = pack_bf16(h[2 * kb + 1][0], h[2 * kb + 1][1]);
        A[kb][3] = pack_bf16(h[2 * kb + 1][2], h[2 * kb + 1][3]);
    }
}
__device__ __forceinline__ void layer1(const float* __restrict__ feats, int64_t n, int64_t r0, int g, int t, const MlpSmemW& s,
                                       uint32_t (&A0)[4], float (&h1)[8][4]) {
    const int64_t ra = r0 + g, rb = r0 + g + 8;
    float x0 = 0.f, x1 = 0.f, x2 = 0.f, x3 = 0.f;
    if (ra < n) { x0 = feats[ra * MLP_IN + 2 * t]; x1 = feats[ra * MLP_IN + 2 * t + 1]; }
    if (rb < n) { x2 = feats[rb * MLP_IN + 2 * t]; x3 = feats[rb * MLP_IN + 2 * t + 1]; }
    A0[0] = pack_bf16(x0, x1); A0[1] = pack_bf16(x2, x3); A0[2] = 0u; A0[3] = 0u;
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        const __nv_bfloat16* wr = s.W1 + (nt * 8 + g) * K1 + 2 * t;
        mma_bf16(c, A0[0], A0[1], A0[2], A0[3], lds32(wr), lds32(wr + 8));
        const float bb0 = s.b1[nt * 8 + 2 * t], bb1 = s.b1[nt * 8 + 2 * t + 1];
        h1[nt][0] = fmaxf(c[0] + bb0, 0.f); h1[nt][1] = fmaxf(c[1] + bb1, 0.f);
        h1[nt][2] = fmaxf(c[2] + bb0, 0.f); h1[nt][3] = fmaxf(c[3] + bb1, 0.f);
    }
}
// y for rows g (out[0]) and g+8 (out[1]) of the warp tile, valid in lanes with t == 0.
__device__ __forceinline__ void output_layer(const float (&h3)[8][4], const MlpSmemW& s, int t, float& ya, float& yb) {
    float pa = 0.f, pb = 0.f;
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const float w0 = s.w4[nt * 8 + 2 * t], w1 = s.w4[nt * 8 + 2 * t + 1];
        pa += h3[nt][0] * w0 + h3[nt][1] * w1;
        pb += h3[nt][2] * w0 + h3[nt][3] * w1;
    }
    pa += __shfl_xor_sync(0xffffffffu, pa, 1); pa += __shfl_xor_sync(0xffffffffu, pa, 2);
    pb += __shfl_xor_sync(0xffffffffu, pb, 1); pb += __shfl_xor_sync(0xffffffffu, pb, 2);
    ya = pa + s.b4;
    yb = pb + s.b4;
}

// ---------------------------------------------------------------- inference
__global__ void __launch_bounds__(MLP_THREADS)
k_mlp_forward(const float* __restrict__ prm, int64_t n, const float* __restrict__ feats, const float* __restrict__ scale,
              float* __restrict__ out) {
    __shared__ MlpSmemW s;
    stage_weights(prm, s, nullptr, nullptr);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const float sc = scale ? *scale : 1.f;
    for (int64_t r0 = ((int64_t)blockIdx.x * MLP_WARPS + warp) * 16; r0 < n; r0 += (int64_t)gridDim.x * MLP_WARPS * 16) {
        uint32_t A0[4], A[4][4];
        float h[8][4];
        layer1(feats, n, r0, g, t, s, A0, h);
        c_to_a(h, A);
        hidden_layer(A, s.W2, s.b2, g, t, h);
        c_to_a(h, A);
        hidden_layer(A, s.W3, s.b3, g, t, h);
        float ya, yb;
        output_layer(h, s, t, ya, yb);
        if (t == 0) {
            if (r0 + g < n) out[r0 + g] = ya * sc;
            if (r0 + g + 8 < n) out[r0 + g + 8] = yb * sc;
        }
    }
}

// ---------------------------------------------------------------- training: forward + backward
// Per warp: transposed BF16 copies of the layer inputs and of dZ for the weight GEMMs.
struct MlpWarpScratch {
    __nv_bfloat16 xT[K1 * 16];        // [k][r]
    __nv_bfloat16 h1T[MLP_H * 16];    // [c][r]
    __nv_bfloat16 h2T[MLP_H * 16];
    __nv_bfloat16 dzT[MLP_H * 16];
};
struct MlpSmemTrain {
    MlpSmemW w;
    __nv_bfloat16 W2T[MLP_H * MLP_H];
    __nv_bfloat16 W3T[MLP_H * MLP_H];
    float grad[MLP_NPARAM];
    MlpWarpScratch ws[MLP_WARPS];
    double loss[MLP_WARPS];
};

// Writes the fragment h (rows g, g+8; cols nt*8+2t, +1) transposed into dstT[c][r] as BF16.
__device__ __forceinline__ void store_T(const float (&h)[8][4], __nv_bfloat16* dstT, int g, int t) {
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const int c = nt * 8 + 2 * t;
        dstT[c * 16 + g] = __float2bfloat16_rn(h[nt][0]);
        dstT[(c + 1) * 16 + g] = __float2bfloat16_rn(h[nt][1]);
        dstT[c * 16 + g + 8] = __float2bfloat16_rn(h[nt][2]);
        dstT[(c + 1) * 16 + g + 8] = __float2bfloat16_rn(h[nt][3]);
    }
}
// grad[off + c*K + k] += sum_r dZT[c][r] * HT[k][r] over the warp's 16 samples, c < 64, k < kdim
// (kdim multiple of 8; HT rows beyond kdim are not read).
__device__ __forceinline__ void weight_grad(const __nv_bfloat16* dzT, const __nv_bfloat16* HT, int kdim, float* grad, int g, int t) {
    #pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
        const __nv_bfloat16* ar = dzT + (mt * 16 + g) * 16 + 2 * t;
        const uint32_t a0 = lds32(ar), a1 = lds32(ar + 8 * 16), a2 = lds32(ar + 8), a3 = lds32(ar + 8 * 16 + 8);
        for (int nt = 0; nt < kdim / 8; ++nt) {
            const __nv_bfloat16* br = HT + (nt * 8 + g) * 16 + 2 * t;
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            mma_bf16(c, a0, a1, a2, a3, lds32(br), lds32(br + 8));
            const int row = mt * 16 + g, col = nt * 8 + 2 * t;
            atomicAdd(grad + row * kdim + col, c[0]);
            atomicAdd(grad + row * kdim + col + 1, c[1]);
            atomicAdd(grad + (row + 8) * kdim + col, c[2]);
            atomicAdd(grad + (row + 8) * kdim + col + 1, c[3]);
        }
    }
}
// Bias gradient: sum over the 16 rows of the dz fragment (rows g, g+8 in each lane).
__device__ __forceinline__ void bias_grad(const float (&dz)[8][4], float* gb, int g, int t) {
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        float s0 = dz[nt][0] + dz[nt][2], s1 = dz[nt][1] + dz[nt][3];
        #pragma unroll
        for (int o = 4; o < 32; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
        if (g == 0) { atomicAdd(gb + nt * 8 + 2 * t, s0); atomicAdd(gb + nt * 8 + 2 * t + 1, s1); }
    }
}
// dH = dZ x W (W row-major [out][in], WT = its transpose [in][out]): M = 16 samples, N = 64 in, K = 64 out.
__device__ __forceinline__ void data_grad(const uint32_t (&A)[4][4], const __nv_bfloat16* WT, int g, int t, float (&dh)[8][4]) {
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        const __nv_bfloat16* br = WT + (nt * 8 + g) * MLP_H + 2 * t;
        #pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_bf16(c, A[ks][0], A[ks][1], A[ks][2], A[ks][3], lds32(br + ks * 16), lds32(br + ks * 16 + 8));
        dh[nt][0] = c[0]; dh[nt][1] = c[1]; dh[nt][2] = c[2]; dh[nt][3] = c[3];
    }
}
// dz = dh * relu'(z), with z > 0 read back from the BF16 activation hT[c][r].
__device__ __forceinline__ void relu_mask(float (&dh)[8][4], const __nv_bfloat16* hT, int g, int t) {
    #pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const int c = nt * 8 + 2 * t;
        if (!(__bfloat162float(hT[c * 16 + g]) > 0.f)) dh[nt][0] = 0.f;
        if (!(__bfloat162float(hT[(c + 1) * 16 + g]) > 0.f)) dh[nt][1] = 0.f;
        if (!(__bfloat162float(hT[c * 16 + g + 8]) > 0.f)) dh[nt][2] = 0.f;
        if (!(__bfloat162float(hT[(c + 1) * 16 + g + 8]) > 0.f)) dh[nt][3] = 0.f;
    }
}

// Mean-squared-error gradient over n samples: grad (FP32, MLP_NPARAM) += d/dtheta of
// (1/n) sum_r (y_r - target_r)^2, and *loss += sum_r (y_r - target_r)^2 (FP64).
__global__ void __launch_bounds__(MLP_THREADS)
k_mlp_grad(const float* __restrict__ prm, int64_t n, const float* __restrict__ feats, const float* __restrict__ target,
           float* __restrict__ grad, double* __restrict__ loss) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MlpSmemTrain& S = *reinterpret_cast<MlpSmemTrain*>(smem_raw);
    stage_weights(prm, S.w, S.W2T, S.W3T);
    for (int q = threadIdx.x; q < MLP_NPARAM; q += blockDim.x) S.grad[q] = 0.f;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    MlpWarpScratch& W = S.ws[warp];
    const float inv_n = 1.f / (float)n;
    double lsum = 0.0;
    for (int64_t r0 = ((int64_t)blockIdx.x * MLP_WARPS + warp) * 16; r0 < n; r0 += (int64_t)gridDim.x * MLP_WARPS * 16) {
        const int64_t ra = r0 + g, rb = r0 + g + 8;
        // ---- forward (keeps h3 in FP32, h1/h2/x transposed in BF16)
        uint32_t A0[4], A[4][4];
        float h1[8][4], h2[8][4], h3[8][4];
        layer1(feats, n, r0, g, t, S.w, A0, h1);
        {   // x^T for dW1 (cols 0..7 real, 8..15 zero)
            float x0 = 0.f, x1 = 0.f, x2 = 0.f, x3 = 0.f;
            if (ra < n) { x0 = feats[ra * MLP_IN + 2 * t]; x1 = feats[ra * MLP_IN + 2 * t + 1]; }
            if (rb < n) { x2 = feats[rb * MLP_IN + 2 * t]; x3 = feats[rb * MLP_IN + 2 * t + 1]; }
            W.xT[(2 * t) * 16 + g] = __float2bfloat16_rn(x0);
            W.xT[(2 * t + 1) * 16 + g] = __float2bfloat16_rn(x1);
            W.xT[(2 * t) * 16 + g + 8] = __float2bfloat16_rn(x2);
            W.xT[(2 * t + 1) * 16 + g + 8] = __float2bfloat16_rn(x3);
        }
        store_T(h1, W.h1T, g, t);
        c_to_a(h1, A);
        hidden_layer(A, S.w.W2, S.w.b2, g, t, h2);
        store_T(h2, W.h2T, g, t);
        c_to_a(h2, A);
        hidden_layer(A, S.w.W3, S.w.b3, g, t, h3);
        float ya, yb;
        output_layer(h3, S.w, t, ya, yb);
        // ---- loss and dy (same value in the four lanes of a row group)
        const float ta = ra < n ? target[ra] : ya, tb = rb < n ? target[rb] : yb;
        const float ea = ra < n ? ya - ta : 0.f, eb = rb < n ? yb - tb : 0.f;
        if (t == 0) lsum += (double)ea * ea + (double)eb * eb;
        const float dya = 2.f * ea * inv_n, dyb = 2.f * eb * inv_n;
        // ---- layer 4: dW4 = sum dy h3, db4 = sum dy; dz3 = dy w4 * relu'(z3)
        float dz[8][4];
        #pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int c = nt * 8 + 2 * t;
            float s0 = dya * h3[nt][0] + dyb * h3[nt][2], s1 = dya * h3[nt][1] + dyb * h3[nt][3];
            #pragma unroll
            for (int o = 4; o < 32; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
            if (g == 0) { atomicAdd(S.grad + OFF_W4 + c, s0); atomicAdd(S.grad + OFF_W4 + c + 1, s1); }
            const float w0 = S.w.w4[c], w1 = S.w.w4[c + 1];
            dz[nt][0] = h3[nt][0] > 0.f ? dya * w0 : 0.f;
            dz[nt][1] = h3[nt][1] > 0.f ? dya * w1 : 0.f;
            dz[nt][2] = h3[nt][2] > 0.f ? dyb * w0 : 0.f;
            dz[nt][3] = h3[nt][3] > 0.f ? dyb * w1 : 0.f;
        }
        {
            float sd = dya + dyb;
            #pragma unroll
            for (int o = 4; o < 32; o <<= 1) sd += __shfl_xor_sync(0xffffffffu, sd, o);
            if (lane == 0) atomicAdd(S.grad + OFF_B4, sd);
        }
        // ---- layer 3
        bias_grad(dz, S.grad + OFF_B3, g, t);
        store_T(dz, W.dzT, g, t);
        __syncwarp();
        weight_grad(W.dzT, W.h2T, MLP_H, S.grad + OFF_W3, g, t);
        c_to_a(dz, A);
        data_grad(A, S.W3T, g, t, dz);       // dz <- dh2
        relu_mask(dz, W.h2T, g, t);          // dz2
        __syncwarp();
        // ---- layer 2
        bias_grad(dz, S.grad + OFF_B2, g, t);
        store_T(dz, W.dzT, g, t);
        __syncwarp();
        weight_grad(W.dzT, W.h1T, MLP_H, S.grad + OFF_W2, g, t);
        c_to_a(dz, A);
        data_grad(A, S.W2T, g, t, dz);       // dh1
        relu_mask(dz, W.h1T, g, t);          // dz1
        __syncwarp();
        // ---- layer 1 (K = 8 real inputs)
        bias_grad(dz, S.grad + OFF_B1, g, t);
        store_T(dz, W.dzT, g, t);
        __syncwarp();
        weight_grad(W.dzT, W.xT, MLP_IN, S.grad + OFF_W1, g, t);
        __syncwarp();
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (lane == 0) S.loss[warp] = lsum;
    __syncthreads();
    for (int q = threadIdx.x; q < MLP_NPARAM; q += blockDim.x) {
        const float v = S.grad[q];
        if (v != 0.f) atomicAdd(grad + q, v);
    }
    if (threadIdx.x == 0) {
        double l = 0.0;
        for (int w = 0; w < MLP_WARPS; ++w) l += S.loss[w];
        atomicAdd(loss, l);
    }
}

// Adam (Kingma & Ba 2015) with bias correction, elementwise over the parameter vector.
__global__ void k_mlp_adam(float* __restrict__ prm, const float* __restrict__ grad, float* __restrict__ m1, float* __restrict__ m2,
                           int64_t count, float lr, float beta1, float beta2, float eps, float c1, float c2) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x) {
        const float gq = grad[q];
        const float a = beta1 * m1[q] + (1.f - beta1) * gq;
        const float b = beta2 * m2[q] + (1.f - beta2) * gq * gq;
        m1[q] = a;
        m2[q] = b;
        prm[q] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
    }
}

// ---------------------------------------------------------------- inference on tcgen05
// One CTA per SM: five warpgroups with a 128-sample tile each in flight (one sample per thread and
// TMEM lane), each issuing its own MMAs from one warp.  Each layer is one chain of
//   D[128 x 64] (TMEM, FP32) = A[128 x K] (TMEM, BF16) x W[64 x K]^T (shared, BF16)
// of K/16 tcgen05.mma kind::f16 instructions with A read from tensor memory, completed
// through tcgen05.commit on the warpgroup's mbarrier.  Warp w then reads TMEM lanes
// 32 (w % 4)..+31 of D (tcgen05.ld 32x32b), applies ReLU while rounding to BF16 (cvt.rn.relu)
// and stores the packed pairs straight back into the A columns of the next layer
// (tcgen05.st 32x32b).  Activations never pass through shared memory, which holds only the
// weights: with A in shared memory every MMA re-read its activations from there (about 98 KB
// of shared-memory traffic per tile, the limit).  The 64 -> 1 output layer is an FP32 dot product
// in registers.
//
// The biases ride in the contraction: A carries two constant-one columns after its real K
// columns (X columns 8, 9; H columns 64, 65) and W the bias split into BF16 hi + lo parts
// in the matching columns, so the FP32 accumulator receives b_hi + b_lo, which equals the
// FP32 bias to about 2^-17 relative.  The hidden layers thus run K = 80 (five k-steps).
// Rounding points otherwise match k_mlp_forward: BF16 features, weights and hidden
// activations, FP32 accumulation, FP32 output layer.
//
// A tile is three MMA round trips, latency bound (no pipe above 55 %): the tiles in flight decide, and
// TMEM holds five, because X lies in the first columns of H (which layer 1 has read when H1 is
// written) and the ones of the hidden layers are one block that the last k-step of every warpgroup
// reads.  An MMA costs its issuing warp about 73 cycles against 32 in the tensor pipe, so one issuing
// warp for all tiles was the limit.  16,777,216 samples: 545 us with four CTAs of a tile each and a
// diverged issuing thread, 490 with five tiles and one issuing warp, 374 with two, 350 with one per
// warpgroup; four partial sums of y or an earlier second tcgen05.ld change nothing (353 to 356).
// Back to back for longer than 0.1 s the GPU reaches its power limit and 350 becomes 410.
//
// TMEM columns (512 allocated, 32-bit each):
//   0..319    D of each warpgroup, the FP32 accumulator
//   320..479  H of each warpgroup: 64 BF16 activations, or X: 8 BF16 features (4 columns), 1, 1, 0...
//   480..487  1, 1, 0...: the bias columns of the hidden layers
constexpr int TC_M = 128, FT_WGS = 5, FT_THREADS = FT_WGS * TC_M, FT_TMEM_COLS = 512;
constexpr int TC_K2 = MLP_H + 16;   // hidden-layer K with the bias columns
constexpr uint32_t FT_COL_D = 0, FT_COL_H = FT_WGS * MLP_H, FT_H_COLS = MLP_H / 2, FT_COL_ONES = FT_COL_H + FT_WGS * FT_H_COLS;
constexpr uint32_t TC_IDESC = umma_idesc_bf16_f32<TC_M, MLP_H>();
static_assert(TC_IDESC == 0x08100490u, "kind::f16 descriptor: BF16 x BF16 -> FP32, M = 128, N = 64, K-major");
static_assert(FT_COL_ONES + 8 <= FT_TMEM_COLS, "TMEM column plan");
constexpr long long TC_WAIT_CYCLES = 1ll << 31;   // about a second at B200 clocks

struct MlpTcSmem {
    __nv_bfloat16 W1[MLP_H * K1];      // [64 x 16]: W1 | b1 hi | b1 lo | 0
    __nv_bfloat16 W2[MLP_H * TC_K2];   // [64 x 80]: W2 | b2 hi | b2 lo | 0
    __nv_bfloat16 W3[MLP_H * TC_K2];
    float4 feats[FT_WGS][2][TC_M];     // the next tile's rows, copied while a tile is computed
    float4 w4[MLP_H / 4];
    unsigned long long chain[FT_WGS];  // the warpgroup's chain is complete
    float b4;
    uint32_t tmem_base;
};
static_assert((sizeof(__nv_bfloat16) * MLP_H * K1) % 128 == 0 && (sizeof(__nv_bfloat16) * MLP_H * TC_K2) % 128 == 0,
              "128 B aligned operands");

// A test's stand-in for a wait that runs out: the thread gives up on the last chain of tile k.
#ifndef FT_GIVE_UP
#define FT_GIVE_UP(k) false
#endif

// relu of (lo, hi) rounded to BF16 and packed, lo in the low half
__device__ __forceinline__ uint32_t relu_bf16x2(uint32_t lo, uint32_t hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
    return d;
}
// Column `part` of the bias block: 0 -> BF16 hi part of b, 1 -> BF16 lo part
// (hi + lo reproduces b to about 2^-17 relative), 2.. -> 0.
__device__ __forceinline__ __nv_bfloat16 bias_part(float b, int part) {
    const __nv_bfloat16 hi = __float2bfloat16_rn(b);
    return part == 0 ? hi : part == 1 ? __float2bfloat16_rn(b - __bfloat162float(hi)) : __float2bfloat16_rn(0.f);
}

__global__ void __launch_bounds__(FT_THREADS, 1)
k_mlp_forward_tc(const float* __restrict__ prm, int64_t n, const float* __restrict__ feats, const float* __restrict__ scale,
                 float* __restrict__ out, int32_t* __restrict__ status) {
    extern __shared__ unsigned char ft_dyn[];
    MlpTcSmem& s = *reinterpret_cast<MlpTcSmem*>((reinterpret_cast<uintptr_t>(ft_dyn) + 127) & ~static_cast<uintptr_t>(127));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (warp == 0) {
        tmem_alloc(smem_u32(&s.tmem_base), FT_TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int w = 0; w < FT_WGS; ++w) {
            mbar_init(smem_u32(&s.chain[w]), 1);
        }
        s.b4 = prm[OFF_B4];
        fence_mbar_init();
    }
    // weights in the K-major core-matrix layout (B operands: rows = output units)
    for (int t = tid; t < MLP_H * K1; t += FT_THREADS) {
        const int r = t / K1, k = t % K1;
        s.W1[umma_k_index(r, k, MLP_H)] = k < MLP_IN ? __float2bfloat16_rn(prm[OFF_W1 + r * MLP_IN + k])
                                                     : bias_part(prm[OFF_B1 + r], k - MLP_IN);
    }
    for (int t = tid; t < MLP_H * TC_K2; t += FT_THREADS) {
        const int r = t / TC_K2, k = t % TC_K2;
        const bool w = k < MLP_H;
        s.W2[umma_k_index(r, k, MLP_H)] = w ? __float2bfloat16_rn(prm[OFF_W2 + r * MLP_H + k]) : bias_part(prm[OFF_B2 + r], k - MLP_H);
        s.W3[umma_k_index(r, k, MLP_H)] = w ? __float2bfloat16_rn(prm[OFF_W3 + r * MLP_H + k]) : bias_part(prm[OFF_B3 + r], k - MLP_H);
    }
    if (tid < MLP_H) reinterpret_cast<float*>(s.w4)[tid] = prm[OFF_W4 + tid];
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    const uint32_t tbase = s.tmem_base;
    const int wg = warp >> 2, r = tid & (TC_M - 1);
    const uint32_t tlane = tbase + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t one2 = pack_bf16(1.f, 1.f);
    if (wg == 0) {
        const uint32_t hb[8] = {one2, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        tmem_st_32x32b_x8(tlane + FT_COL_ONES, hb);
        tmem_st_wait();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    // the CTA's tiles are blockIdx.x + k gridDim.x, k < ktiles; warpgroup w takes k = w, w + 5, ...
    const int64_t ntiles = (n + TC_M - 1) / TC_M;
    const int ktiles = static_cast<int>((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
    // the issuing warps of the warpgroups lie on different sub-cores
    const bool issuer = (warp & 3) == (wg & 3);
    const uint32_t tDw = tbase + FT_COL_D + wg * MLP_H, tHw = tbase + FT_COL_H + wg * FT_H_COLS;
    const uint32_t tD = tlane + FT_COL_D + wg * MLP_H, tH = tlane + FT_COL_H + wg * FT_H_COLS, chain = smem_u32(&s.chain[wg]);
    constexpr uint32_t LBO_W = MLP_H * 16, SBO = 128;
    const uint64_t dW1 = umma_desc_kmajor(smem_u32(s.W1), LBO_W, SBO), dW2 = umma_desc_kmajor(smem_u32(s.W2), LBO_W, SBO),
                   dW3 = umma_desc_kmajor(smem_u32(s.W3), LBO_W, SBO);
    const float sc = scale ? *scale : 1.f;
    {
        uint32_t phase = 0u;
        bool ok = true;
        auto row_of = [&](int k) { return (blockIdx.x + static_cast<int64_t>(k) * gridDim.x) * TC_M + r; };
        // The A operand is in place: issue the chain of a layer, unless a wait before ran out in some thread
        // (one that gave up still comes to this barrier, so the warpgroup decides as one).
        auto issue = [&](int layer) {
            tmem_st_wait();
            tc_fence_before_sync();
            ok = bar_and_named(wg + 1, TC_M, ok);
            if (issuer && ok) {
                tc_fence_after_sync();
                if (elect_one()) {
                    if (layer == 0) {
                        umma_bf16_ts(tDw, tHw, dW1, TC_IDESC, 0u);
                    } else {
                        const uint64_t dW = layer == 1 ? dW2 : dW3;
                        #pragma unroll
                        for (int ks = 0; ks < MLP_H / 16; ++ks)
                            umma_bf16_ts(tDw, tHw + ks * 8, dW + ks * (2 * LBO_W / 16), TC_IDESC, ks > 0 ? 1u : 0u);
                        umma_bf16_ts(tDw, tbase + FT_COL_ONES, dW + (MLP_H / 16) * (2 * LBO_W / 16), TC_IDESC, 1u);
                    }
                    umma_commit(chain);
                }
                __syncwarp();
            }
        };
        auto wait_chain = [&]() {
            ok = mbar_wait_bounded(chain, phase, TC_WAIT_CYCLES);
            phase ^= 1u;
            tc_fence_after_sync();
        };
        // this thread's row of tile k into shared memory, without a register held meanwhile
        auto fetch_row = [&](int k) {
            const int64_t row = row_of(k);
            const bool in = k < ktiles && row < n;
            const float* src = in ? feats + row * MLP_IN : feats;
            cp_async_16(smem_u32(&s.feats[wg][0][r]), src, in ? 16 : 0);
            cp_async_16(smem_u32(&s.feats[wg][1][r]), src + 4, in ? 16 : 0);
        };
        auto put_x = [&]() {
            cp_async_wait();
            const float4 f0 = s.feats[wg][0][r], f1 = s.feats[wg][1][r];
            const uint32_t xw[8] = {pack_bf16(f0.x, f0.y), pack_bf16(f0.z, f0.w), pack_bf16(f1.x, f1.y), pack_bf16(f1.z, f1.w), one2, 0u, 0u, 0u};
            tmem_st_32x32b_x8(tH, xw);
        };
        if (wg < ktiles) {
            fetch_row(wg);
            put_x();
            issue(0);
        }
        int k = wg;
        #pragma unroll 1
        for (; k < ktiles; k += FT_WGS) {
            fetch_row(k + FT_WGS);
            #pragma unroll 1
            for (int layer = 0; layer < 2; ++layer) {
                wait_chain();
                #pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t v[32], h[16];
                    tmem_ld_32x32b_x32(tD + 32 * half, v);
                    tmem_ld_wait(v);
                    #pragma unroll
                    for (int j = 0; j < 16; ++j) h[j] = relu_bf16x2(v[2 * j], v[2 * j + 1]);
                    const uint32_t (&h0)[8] = *reinterpret_cast<const uint32_t(*)[8]>(h);
                    const uint32_t (&h1)[8] = *reinterpret_cast<const uint32_t(*)[8]>(h + 8);
                    tmem_st_32x32b_x8(tH + 16 * half, h0);
                    tmem_st_32x32b_x8(tH + 16 * half + 8, h1);
                }
                issue(layer + 1);
                if (!ok) break;
            }
            if (!ok) break;
            wait_chain();
            ok = ok && !FT_GIVE_UP(k);
            // the next tile's first chain runs while the second half of the output layer is summed
            float y = 0.f;
            #pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(tD + 32 * half, v);
                tmem_ld_wait(v);
                if (half == 1 && k + FT_WGS < ktiles) {
                    put_x();
                    issue(0);
                }
                #pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 w = s.w4[8 * half + q];
                    y = fmaf(fmaxf(__uint_as_float(v[4 * q]), 0.f), w.x, y);
                    y = fmaf(fmaxf(__uint_as_float(v[4 * q + 1]), 0.f), w.y, y);
                    y = fmaf(fmaxf(__uint_as_float(v[4 * q + 2]), 0.f), w.z, y);
                    y = fmaf(fmaxf(__uint_as_float(v[4 * q + 3]), 0.f), w.w, y);
                }
            }
            if (!ok) break;
            const int64_t row = row_of(k);
            if (row < n) out[row] = (y + s.b4) * sc;
        }
        if (!ok) {
            // A chain did not complete in time: the samples of this and later tiles get NaN.  Its MMAs may
            // still be in flight, so the issuing warp waits once more (bounded) before the TMEM columns
            // are released; the status tells the host that the context is suspect, and the host stops
            // issuing work to this device's MLP after it.
            if (issuer) (void)mbar_wait_bounded(chain, phase ^ 1u, TC_WAIT_CYCLES);
            // (every thread that gave up says so: behind the last chain of the last tile no barrier of the
            // warpgroup follows that would tell the others)
            if (status) atomicOr(status, SPH_STATUS_TIMEOUT);
            for (; k < ktiles; k += FT_WGS)
                if (row_of(k) < n) out[row_of(k)] = __int_as_float(0x7fc00000);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tbase, FT_TMEM_COLS);
    }
}

// ---------------------------------------------------------------- training on tcgen05
// The gradient of the mean squared error with every GEMM on the tensor cores.  One CTA per
// SM: three warpgroups, each with a 128-sample tile of its own in flight (one sample per
// thread and TMEM lane), and one warp of a fourth that issues every MMA and gives its
// registers to the others.
//   forward   the three hidden layers as in k_mlp_forward_tc (TS form, biases in the
//             contraction), keeping each layer's BF16 input in shared memory (X, H1, H2) and
//             the ReLU masks in registers;
//   output    y = h3 . w4 + b4 in FP32, dy = 2 (y - t) / n; the w4 and b4 gradients and the loss
//             are sums in registers over the thread's samples, reduced once at the end;
//   backward  dZ3 = dy w4 * [z3 > 0]; then per layer l = 3, 2, 1
//               dH_{l-1} = dZ_l W_l          (TS form, A = dZ_l in TMEM)
//               G_l (+)= dZ_l^T H_{l-1}      (SS form, M = 64 outputs, N = the inputs and a ones
//                                           column for db_l, K = 128 samples; accumulated in TMEM
//                                           over all tiles of the CTA)
//             and dZ_{l-1} = dH_{l-1} * [z_{l-1} > 0] in the epilogue.
// At the end G_1..G_3 are added to the global gradient with FP32 atomics.  Rounding points: BF16 inputs, weights, activations and
// dZ, FP32 accumulation, as the oracle's BF16 gradient (oracle/mlp.py); the bias gradients
// come from the BF16 dZ, which the oracle sums unrounded.
//
// The samples are the contraction of G_l, and a thread holds all units of one sample, so the
// operands of G_l are MN-major: 8 units of a sample are 16 contiguous bytes, stored at once and
// without bank conflicts (a K-major operand took 64 two-byte stores per layer with four-way
// conflicts).  The same reading of W (stored once, K-major for the forward pass) gives the
// B operand of dH without a transposed copy.
//
// A tile is a chain of five MMA round trips (about 900 cycles of waiting and 1000 of epilogue each),
// so the chain and not the tensor pipe (a third busy) bounds a single tile: three tiles in flight are
// what TMEM (3 x 104 columns beside G) and shared memory (3 x 60 KB) hold.  The chains that the
// epilogues wait for are issued by one warp and the G_l by another; an epilogue waits for G_l only
// before it overwrites dZ.  Each warp takes the warpgroups in turn, so the additions into G keep
// the order of the tiles.  4,194,304 samples: 2.23 -> 0.37 ms (one tile in flight with two-byte
// transposed stores before; 0.80 with one diverged issuing thread, 0.46 with the w4 sums spilled
// at 128 registers).  Starting the second half's tcgen05.ld ahead of the first half's arithmetic
// changes nothing (0.37 to 0.38).
//
// TMEM columns (512, one CTA per SM):
//   0..15, 32..103, 104..175   G_1, G_2, G_3: column = input unit, the ones column behind the last;
//             output unit o in lane 32 (o / 16) + o % 16, as an accumulator of M = 64 lies
//   192..383  D of each warpgroup: layer outputs in the forward pass, dH in the backward pass (FP32)
//   384..503  H of each warpgroup (40 columns): the A operand; X and its ones use the first 8
//             columns before layer 1, dZ the first 32 in the backward pass, the last 8 hold the
//             constant ones of the bias columns
//
// Shared memory of a warpgroup: 2 KB chunks of 8 units x 128 samples,
//   H1 (8 chunks) ones X0 ones X1 ones H2 (8 chunks) ones dZ (8 chunks);
// X alternates between two chunks because G_1 of a tile is issued after the next tile's X is
// written.
constexpr int GT_WGS = 3, GT_THREADS = (GT_WGS + 1) * TC_M, GT_TMEM_COLS = 512;
constexpr int GT_SUMS_THREADS = GT_WGS * TC_M + 64;      // the warpgroups and the two issuing warps
// registers per thread after the launch with 128: the w4 sums do not fit in 128
constexpr int GT_REGS = 160, GT_REGS_MMA = 32;
static_assert(TC_M * (GT_WGS * GT_REGS + GT_REGS_MMA) <= GT_THREADS * 128, "the shares add up to the launch's registers");
constexpr uint32_t GT_COL_D = 192, GT_COL_H = 384, GT_H_COLS = TC_K2 / 2;
static_assert(GT_COL_D + GT_WGS * MLP_H <= GT_COL_H && GT_COL_H + GT_WGS * GT_H_COLS <= GT_TMEM_COLS, "TMEM column plan");
constexpr int GT_CHUNK = TC_M * 16;
constexpr int GT_H1 = 0, GT_X = 9, GT_X_STEP = 2, GT_H2 = 13, GT_DZ = 22, GT_CHUNKS = 30;
constexpr int GT_N = MLP_H + 8, GT_N1 = MLP_IN + 8;      // columns of G_2, G_3 and of G_1: inputs, then the ones chunk
constexpr uint32_t GT_COL_G1 = 0, GT_COL_G2 = 32, GT_COL_G3 = GT_COL_G2 + GT_N;
static_assert(GT_COL_G3 + GT_N <= GT_COL_D, "TMEM column plan");
constexpr uint32_t GT_IDESC_G = umma_idesc_bf16_f32<MLP_H, GT_N, true, true>(), GT_IDESC_G1 = umma_idesc_bf16_f32<MLP_H, GT_N1, true, true>();
constexpr uint32_t GT_IDESC_DH = umma_idesc_bf16_f32<TC_M, MLP_H, false, true>();    // A in TMEM, B MN-major
constexpr int GT_STAGE = 73;      // floats per output of G_l staged in shared memory (odd: no bank conflicts)

struct MlpGradTcSmem {
    __nv_bfloat16 W1[MLP_H * K1];      // B of layer 1 [64 x 16]: W1 | b1 hi | b1 lo | 0
    __nv_bfloat16 W2[MLP_H * TC_K2];   // B of layer 2 [64 x 80]
    __nv_bfloat16 W3[MLP_H * TC_K2];
    uint4 act[GT_WGS][GT_CHUNKS][TC_M];
    float4 feats[GT_WGS][TC_M][2];     // the next tile's rows, copied while a tile is computed
    float4 w4[MLP_H / 4];
    float gw4[MLP_H];
    double loss;
    unsigned long long ready[GT_WGS];  // the warpgroup's operands of the next chain are in place (128 arrivals)
    unsigned long long gready[GT_WGS]; // those of the next G_l
    unsigned long long chain[GT_WGS];  // the chain that its epilogue waits for is complete
    unsigned long long wgrad[GT_WGS];  // G_l of its tile is complete
    unsigned long long done;           // every MMA of the CTA is complete
    float gb4;
    float b4;
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(MlpGradTcSmem) + 128 <= 227 * 1024, "one CTA per SM");
// A test's stand-in for a wait that runs out: the weight-gradient warp gives up before G_l of tile k.
#ifndef GT_GIVE_UP
#define GT_GIVE_UP(l, k) false
#endif
static_assert(sizeof(__nv_bfloat16) * MLP_H * (K1 + 2 * TC_K2) % 128 == 0, "128 B aligned operands");

// 0xffff in the low and high half if bit j, j + 16 of m is set: prmt replicates the signs of bytes 1 and 3
__device__ __forceinline__ uint32_t mask_halves(uint32_t m, int j) {
    uint32_t d;
    asm("prmt.b32 %0, %1, 0, 0xbb99;" : "=r"(d) : "r"(m << (15 - j)));
    return d;
}

__global__ void __launch_bounds__(GT_THREADS, 1)
k_mlp_grad_tc(const float* __restrict__ prm, int64_t n, const float* __restrict__ feats, const float* __restrict__ target,
              float* __restrict__ grad, double* __restrict__ loss_out, int32_t* __restrict__ status) {
    extern __shared__ unsigned char gt_dyn[];
    MlpGradTcSmem& s = *reinterpret_cast<MlpGradTcSmem*>((reinterpret_cast<uintptr_t>(gt_dyn) + 127) & ~static_cast<uintptr_t>(127));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (warp == 0) {
        tmem_alloc(smem_u32(&s.tmem_base), GT_TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int w = 0; w < GT_WGS; ++w) {
            mbar_init(smem_u32(&s.ready[w]), TC_M);
            mbar_init(smem_u32(&s.gready[w]), TC_M);
            mbar_init(smem_u32(&s.chain[w]), 1);
            mbar_init(smem_u32(&s.wgrad[w]), 1);
        }
        mbar_init(smem_u32(&s.done), 2);
        s.abort = 0;
        s.gb4 = 0.f;
        s.loss = 0.0;
        s.b4 = prm[OFF_B4];
        fence_mbar_init();
    }
    for (int t = tid; t < MLP_H * K1; t += GT_THREADS) {
        const int r = t / K1, k = t % K1;
        s.W1[umma_k_index(r, k, MLP_H)] = k < MLP_IN ? __float2bfloat16_rn(prm[OFF_W1 + r * MLP_IN + k])
                                                     : bias_part(prm[OFF_B1 + r], k - MLP_IN);
    }
    for (int t = tid; t < MLP_H * TC_K2; t += GT_THREADS) {
        const int r = t / TC_K2, k = t % TC_K2;
        const bool w = k < MLP_H;
        s.W2[umma_k_index(r, k, MLP_H)] = w ? __float2bfloat16_rn(prm[OFF_W2 + r * MLP_H + k]) : bias_part(prm[OFF_B2 + r], k - MLP_H);
        s.W3[umma_k_index(r, k, MLP_H)] = w ? __float2bfloat16_rn(prm[OFF_W3 + r * MLP_H + k]) : bias_part(prm[OFF_B3 + r], k - MLP_H);
    }
    const uint4 one_chunk = make_uint4(pack_bf16(1.f, 0.f), 0u, 0u, 0u);
    for (int t = tid; t < GT_WGS * TC_M; t += GT_THREADS) {
        const int w = t / TC_M, r = t % TC_M;
        s.act[w][GT_H1 + 8][r] = one_chunk;
        s.act[w][GT_X + 1][r] = one_chunk;
        s.act[w][GT_X + GT_X_STEP + 1][r] = one_chunk;
        s.act[w][GT_H2 + 8][r] = one_chunk;
    }
    if (tid < MLP_H) { reinterpret_cast<float*>(s.w4)[tid] = prm[OFF_W4 + tid]; s.gw4[tid] = 0.f; }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    const uint32_t tbase = s.tmem_base;
    const float inv_n = 2.f / static_cast<float>(n);
    // the CTA's tiles are blockIdx.x + k gridDim.x, k < ktiles; warpgroup w takes k = w, w + 3, ...
    const int64_t ntiles = (n + TC_M - 1) / TC_M;
    const int ktiles = static_cast<int>((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);

    if (warp >= GT_WGS * 4) {
        setmaxnreg_dec<GT_REGS_MMA>();
        // The loops are uniform over the warp, so that descriptors and addresses stay in uniform registers
        // (one diverged thread spent 85 cycles on moving them per MMA); one elected lane issues.
        const uint32_t aAct = smem_u32(s.act);
        constexpr uint32_t CORE = 128, LBO_W = MLP_H * 16, WG_BYTES = GT_CHUNKS * GT_CHUNK;
        uint32_t rphase = 0u;          // parity of each ready barrier
        bool ok = true;
        auto wait_ready = [&](uint32_t bars, int w) -> bool {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(bars + 8 * w, (rphase >> w) & 1u, TC_WAIT_CYCLES));
            rphase ^= 1u << w;
            tc_fence_after_sync();
            return ok;
        };
        if (warp == GT_WGS * 4) {
            // the chains that the epilogues wait for: layers 1, 2, 3, dH2, dH1
            const uint32_t aW1 = smem_u32(s.W1), aW2 = smem_u32(s.W2), aW3 = smem_u32(s.W3), aReady = smem_u32(s.ready), aChain = smem_u32(s.chain);
            #pragma unroll 1
            for (int k0 = 0; ok && k0 < ktiles; k0 += GT_WGS) {
                #pragma unroll 1
                for (int phase = 0; ok && phase < 5; ++phase) {
                    #pragma unroll 1
                    for (int w = 0; w < GT_WGS && k0 + w < ktiles; ++w) {
                        if (!wait_ready(aReady, w)) break;
                        const uint32_t tD = tbase + GT_COL_D + w * MLP_H, tH = tbase + GT_COL_H + w * GT_H_COLS;
                        if (elect_one()) {
                            if (phase == 0) {
                                umma_bf16_ts(tD, tH, umma_desc_kmajor(aW1, LBO_W, CORE), TC_IDESC, 0u);
                            } else if (phase <= 2) {
                                const uint64_t dW = umma_desc_kmajor(phase == 1 ? aW2 : aW3, LBO_W, CORE);
                                #pragma unroll
                                for (int ks = 0; ks < TC_K2 / 16; ++ks)
                                    umma_bf16_ts(tD, tH + ks * 8, dW + ks * (2 * LBO_W / 16), TC_IDESC, ks > 0 ? 1u : 0u);
                            } else {
                                const uint64_t dW = umma_desc_mnmajor(phase == 3 ? aW3 : aW2, CORE, LBO_W);
                                #pragma unroll
                                for (int ks = 0; ks < MLP_H / 16; ++ks)
                                    umma_bf16_ts(tD, tH + ks * 8, dW + ks * (2 * CORE / 16), GT_IDESC_DH, ks > 0 ? 1u : 0u);
                            }
                            umma_commit(aChain + 8 * w);
                        }
                        __syncwarp();
                    }
                }
            }
        } else if (warp == GT_WGS * 4 + 1) {
            // G_3, G_2, G_1 of each tile, in the order of the tiles
            const uint32_t aReady = smem_u32(s.gready), aWgrad = smem_u32(s.wgrad);
            uint32_t x = GT_X;
            #pragma unroll 1
            for (int k0 = 0; ok && k0 < ktiles; k0 += GT_WGS) {
                #pragma unroll 1
                for (int l = 3; ok && l >= 1; --l) {
                    const uint32_t tG = tbase + (l == 3 ? GT_COL_G3 : (l == 2 ? GT_COL_G2 : GT_COL_G1));
                    const uint32_t idesc = l == 1 ? GT_IDESC_G1 : GT_IDESC_G;
                    #pragma unroll 1
                    for (int w = 0; w < GT_WGS && k0 + w < ktiles; ++w) {
                        if (!wait_ready(aReady, w)) break;
                        if (GT_GIVE_UP(l, k0 + w)) { ok = false; break; }
                        const uint32_t act = aAct + w * WG_BYTES;
                        const uint64_t dA = umma_desc_mnmajor(act + GT_DZ * GT_CHUNK, CORE, GT_CHUNK);
                        const uint64_t dB = umma_desc_mnmajor(act + (l == 3 ? GT_H2 : (l == 2 ? GT_H1 : x)) * GT_CHUNK, CORE, GT_CHUNK);
                        if (elect_one()) {
                            umma_bf16_ss(tG, dA, dB, idesc, k0 + w > 0);
                            #pragma unroll
                            for (int ks = 1; ks < TC_M / 16; ++ks) umma_bf16_ss(tG, dA + ks * (2 * CORE / 16), dB + ks * (2 * CORE / 16), idesc, 1u);
                            umma_commit(aWgrad + 8 * w);
                        }
                        __syncwarp();
                    }
                }
                x = 2 * GT_X + GT_X_STEP - x;
            }
        }
        if (warp <= GT_WGS * 4 + 1) {
            if (elect_one()) umma_commit(smem_u32(&s.done));
            // also after a timeout: nothing may be in flight when the TMEM columns are released
            if (!mbar_wait_bounded(smem_u32(&s.done), 0u, TC_WAIT_CYCLES) || !ok) s.abort = 1;
            __syncwarp();
            bar_sync_named(GT_WGS + 1, GT_SUMS_THREADS);
        }
    } else {
        setmaxnreg_inc<GT_REGS>();
        const int wg = warp >> 2, r = tid & (TC_M - 1);
        const uint32_t tlane = tbase + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const uint32_t tD = tlane + GT_COL_D + wg * MLP_H, tH = tlane + GT_COL_H + wg * GT_H_COLS;
        const uint32_t ready = smem_u32(&s.ready[wg]), gready = smem_u32(&s.gready[wg]), chain = smem_u32(&s.chain[wg]), wgrad = smem_u32(&s.wgrad[wg]);
        const uint32_t one2 = pack_bf16(1.f, 1.f);
        uint4 (*act)[TC_M] = s.act[wg];
        uint32_t cphase = 0u, gphase = 0u;
        bool ok = true;
        float gw[MLP_H];
        #pragma unroll
        for (int j = 0; j < MLP_H; ++j) gw[j] = 0.f;
        float gb = 0.f;
        double lsum = 0.0;
        // operands of a chain, of a G_l, or of both are in place
        auto signal = [&](bool to_chain, bool to_g) {
            tmem_st_wait();
            fence_proxy_async_smem();
            tc_fence_before_sync();
            if (to_chain) mbar_arrive(ready);
            if (to_g) mbar_arrive(gready);
        };
        // a warp gives up as one, so that it stays converged for the tensor-memory instructions
        auto wait_on = [&](uint32_t bar, uint32_t& phase) -> bool {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, phase, TC_WAIT_CYCLES));
            phase ^= 1u;
            tc_fence_after_sync();
            return ok;
        };
        // this thread's row of tile k into shared memory, without a register held meanwhile
        auto fetch_row = [&](int k) {
            const int64_t row = (blockIdx.x + static_cast<int64_t>(k) * gridDim.x) * TC_M + r;
            const bool in = k < ktiles && row < n;
            const float* src = in ? feats + row * MLP_IN : feats;
            cp_async_16(smem_u32(&s.feats[wg][r][0]), src, in ? 16 : 0);
            cp_async_16(smem_u32(&s.feats[wg][r][1]), src + 4, in ? 16 : 0);
        };
        auto put_x = [&](int parity) {
            cp_async_wait();
            const float4 f0 = s.feats[wg][r][0], f1 = s.feats[wg][r][1];
            const uint4 x = make_uint4(pack_bf16(f0.x, f0.y), pack_bf16(f0.z, f0.w), pack_bf16(f1.x, f1.y), pack_bf16(f1.z, f1.w));
            const uint32_t xw[8] = {x.x, x.y, x.z, x.w, one2, 0u, 0u, 0u};
            tmem_st_32x32b_x8(tH, xw);
            act[GT_X + GT_X_STEP * parity][r] = x;
        };
        // 32 units (a half) as BF16 pairs: into the A operand and, 8 units at a time, the chunks from c0
        auto put_tmem = [&](int half, const uint32_t (&h)[16]) {
            const uint32_t (&h0)[8] = *reinterpret_cast<const uint32_t(*)[8]>(h);
            const uint32_t (&h1)[8] = *reinterpret_cast<const uint32_t(*)[8]>(h + 8);
            tmem_st_32x32b_x8(tH + 16 * half, h0);
            tmem_st_32x32b_x8(tH + 16 * half + 8, h1);
        };
        auto put_chunks = [&](int c0, int half, const uint32_t (&h)[16]) {
            #pragma unroll
            for (int q = 0; q < 4; ++q) act[c0 + 4 * half + q][r] = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
        };
        {
            const uint32_t hb[8] = {one2, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            tmem_st_32x32b_x8(tH + MLP_H / 2, hb);
        }
        if (wg < ktiles) {
            fetch_row(wg);
            put_x(0);
            signal(true, false);
        }
        int parity = 0;
        #pragma unroll 1
        for (int k = wg; k < ktiles; k += GT_WGS) {
            const int64_t row = (blockIdx.x + static_cast<int64_t>(k) * gridDim.x) * TC_M + r;
            const bool valid = row < n;
            const float tgt = valid ? __ldg(target + row) : 0.f;
            fetch_row(k + GT_WGS);
            // ---- forward
            uint32_t mask[2][2];     // [layer][32-unit half]: z > 0, units 2 j and 2 j + 1 in bits j and j + 16
            #pragma unroll
            for (int layer = 0; layer < 2; ++layer) {
                if (!wait_on(chain, cphase)) break;
                #pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t v[32], h[16], m = 0u;
                    tmem_ld_32x32b_x32(tD + 32 * half, v);
                    tmem_ld_wait(v);
                    #pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        h[j] = relu_bf16x2(v[2 * j], v[2 * j + 1]);
                        m |= __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&h[j]), __float2bfloat162_rn(0.f)) & (0x00010001u << j);
                    }
                    mask[layer][half] = m;
                    put_tmem(half, h);
                    put_chunks(layer == 0 ? GT_H1 : GT_H2, half, h);
                }
                signal(true, false);
            }
            if (!ok || !wait_on(chain, cphase)) break;
            // ---- output layer and dZ3
            float dy;
            {
                float y = 0.f;
                #pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(tD + 32 * half, v);
                    tmem_ld_wait(v);
                    #pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 w = s.w4[8 * half + q];
                        y = fmaf(fmaxf(__uint_as_float(v[4 * q]), 0.f), w.x, y);
                        y = fmaf(fmaxf(__uint_as_float(v[4 * q + 1]), 0.f), w.y, y);
                        y = fmaf(fmaxf(__uint_as_float(v[4 * q + 2]), 0.f), w.z, y);
                        y = fmaf(fmaxf(__uint_as_float(v[4 * q + 3]), 0.f), w.w, y);
                    }
                }
                const float e = valid ? y + s.b4 - tgt : 0.f;
                dy = e * inv_n;
                lsum += static_cast<double>(e) * static_cast<double>(e);
                gb += dy;
            }
            if (k != wg && !wait_on(wgrad, gphase)) break;      // G_1 of the tile before has read dZ1
            #pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t v[32], p[16];      // z3 of this half, read again now that dy is known
                tmem_ld_32x32b_x32(tD + 32 * half, v);
                tmem_ld_wait(v);
                #pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 w = s.w4[8 * half + q];
                    const float z[4] = {__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]),
                                        __uint_as_float(v[4 * q + 3])};
                    #pragma unroll
                    for (int t = 0; t < 4; ++t) gw[32 * half + 4 * q + t] = fmaf(dy, fmaxf(z[t], 0.f), gw[32 * half + 4 * q + t]);
                    p[2 * q] = pack_bf16(z[0] > 0.f ? dy * w.x : 0.f, z[1] > 0.f ? dy * w.y : 0.f);
                    p[2 * q + 1] = pack_bf16(z[2] > 0.f ? dy * w.z : 0.f, z[3] > 0.f ? dy * w.w : 0.f);
                }
                put_tmem(half, p);
                put_chunks(GT_DZ, half, p);
            }
            signal(true, true);
            // ---- backward: dZ_{l-1} = dH_{l-1} * [z_{l-1} > 0] for l = 3, 2
            #pragma unroll
            for (int l = 3; l >= 2; --l) {
                if (!wait_on(chain, cphase)) break;
                const bool more = l == 3 || k + GT_WGS < ktiles;
                if (l == 2) {
                    parity ^= 1;
                    if (more) put_x(parity);
                }
                uint32_t p[2][16];
                #pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const uint32_t m = mask[l - 2][half];
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(tD + 32 * half, v);
                    tmem_ld_wait(v);
                    #pragma unroll
                    for (int j = 0; j < 16; ++j)
                        p[half][j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])) & mask_halves(m, j);
                    if (l == 3) put_tmem(half, p[half]);     // dZ2 is the A operand of dH1 = dZ2 W2
                }
                if (!wait_on(wgrad, gphase)) break;          // G_l has read dZ_l
                put_chunks(GT_DZ, 0, p[0]);
                put_chunks(GT_DZ, 1, p[1]);
                signal(more, true);
            }
            if (!ok) break;
        }
        if (ok) ok = mbar_wait_bounded(smem_u32(&s.done), 0u, TC_WAIT_CYCLES);
        if (!ok) s.abort = 1;
        tc_fence_after_sync();
        // the thread's sums over its samples: a butterfly that halves the values per lane each
        // round leaves lane l with column l
        #pragma unroll
        for (int half = 0; half < 2; ++half) {
            float g[32];
            #pragma unroll
            for (int j = 0; j < 32; ++j) g[j] = gw[32 * half + j];
            #pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
                const bool upper = (lane & off) != 0;
                #pragma unroll
                for (int t = 0; t < off; ++t) {
                    const float send = upper ? g[t] : g[t + off];
                    const float keep = upper ? g[t + off] : g[t];
                    g[t] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
            atomicAdd(&s.gw4[32 * half + lane], g[0]);
        }
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
            gb += __shfl_xor_sync(0xffffffffu, gb, o);
        }
        if (lane == 0) { atomicAdd(&s.loss, lsum); atomicAdd(&s.gb4, gb); }
        // every warpgroup's sums, and the abort flag of both issuing warps: `done` alone says that nothing is in
        // flight, also where a warp gave up before the last G_l
        bar_sync_named(GT_WGS + 1, GT_SUMS_THREADS);
        if (s.abort) {
            if (tid == 0 && status) atomicOr(status, SPH_STATUS_TIMEOUT);
        } else {
            // each warpgroup brings one G_l through shared memory, so that the atomics run along its rows
            const int l = wg + 1;
            const uint32_t tG = tlane + (l == 1 ? GT_COL_G1 : (l == 2 ? GT_COL_G2 : GT_COL_G3));
            const int nin = l == 1 ? MLP_IN : MLP_H;
            const int offW = l == 1 ? OFF_W1 : (l == 2 ? OFF_W2 : OFF_W3), offB = l == 1 ? OFF_B1 : (l == 2 ? OFF_B2 : OFF_B3);
            float* stage = reinterpret_cast<float*>(s.act[wg]);
            const int o = (warp & 3) * 16 + lane;
            #pragma unroll 1
            for (int c = 0; c <= nin; c += 8) {
                uint32_t v[8];
                tmem_ld_32x32b_x8(tG + c, v);
                if (lane < 16) {
                    #pragma unroll
                    for (int j = 0; j < 8; ++j) stage[o * GT_STAGE + c + j] = __uint_as_float(v[j]);
                }
            }
            bar_sync_named(wg + 1, TC_M);
            for (int t = r; t < MLP_H * nin; t += TC_M) atomicAdd(&grad[offW + t], stage[(t / nin) * GT_STAGE + t % nin]);
            for (int t = r; t < MLP_H; t += TC_M) atomicAdd(&grad[offB + t], stage[t * GT_STAGE + nin]);
            if (tid < MLP_H) atomicAdd(&grad[OFF_W4 + tid], s.gw4[tid]);
            if (tid == 0) {
                atomicAdd(&grad[OFF_B4], s.gb4);
                atomicAdd(loss_out, s.loss);
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tbase, GT_TMEM_COLS);
    }
}

static int forward_tc_smem_bytes() { return (int)sizeof(MlpTcSmem) + 128; }

static int grad_tc_smem_bytes() { return (int)sizeof(MlpGradTcSmem) + 128; }

static int train_smem_bytes() { return (int)sizeof(MlpSmemTrain); }

}  // namespace wsph

using namespace wsph;

extern "C" {

int64_t sph_mlp_param_count(void) { return MLP_NPARAM; }

int sph_mlp_forward(const float* params, int64_t n, const float* feats, const float* scale, float* out, void* stream) {
    if (n < 0) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_forward: n < 0");
    if (n == 0) return SPH_OK;
    WSPH_CHECK_PTR(params); WSPH_CHECK_PTR(feats); WSPH_CHECK_PTR(out);
    if (reinterpret_cast<uintptr_t>(feats) & 7) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_forward: feats must be 8-byte aligned");
    const int64_t tiles = (n + 16 * MLP_WARPS - 1) / (16 * MLP_WARPS);
    const int grid = (int)(tiles < 148 * 16 ? tiles : 148 * 16);
    count_launch();
    k_mlp_forward<<<grid, MLP_THREADS, 0, WSPH_STREAM(stream)>>>(params, n, feats, scale, out);
    return check_launch("sph_mlp_forward");
}

int sph_mlp_forward_tc(const float* params, int64_t n, const float* feats, const float* scale, float* out, int32_t* status,
                       void* stream) {
    if (n < 0) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_forward_tc: n < 0");
    if (n == 0) return SPH_OK;
    WSPH_CHECK_PTR(params); WSPH_CHECK_PTR(feats); WSPH_CHECK_PTR(out);
    if (reinterpret_cast<uintptr_t>(feats) & 15) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_forward_tc: feats must be 16-byte aligned");
    const int64_t tiles = (n + TC_M - 1) / TC_M;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        attr_err = cudaFuncSetAttribute(k_mlp_forward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, forward_tc_smem_bytes());
    });
    if (attr_err != cudaSuccess)
        return set_error(SPH_ERR_CUDA, "sph_mlp_forward_tc: shared memory opt-in: %s", cudaGetErrorString(attr_err));
    const int grid = (int)(tiles < 148 ? tiles : 148);
    count_launch();
    k_mlp_forward_tc<<<grid, FT_THREADS, forward_tc_smem_bytes(), WSPH_STREAM(stream)>>>(params, n, feats, scale, out, status);
    return check_launch("sph_mlp_forward_tc");
}

int sph_mlp_grad(const float* params, int64_t n, const float* feats, const float* target, float* grad, double* loss, void* stream) {
    if (n < 0) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_grad: n < 0");
    WSPH_CHECK_PTR(params); WSPH_CHECK_PTR(grad); WSPH_CHECK_PTR(loss);
    cudaStream_t s = WSPH_STREAM(stream);
    cudaMemsetAsync(grad, 0, sizeof(float) * MLP_NPARAM, s);
    cudaMemsetAsync(loss, 0, sizeof(double), s);
    if (n == 0) return check_launch("sph_mlp_grad");
    WSPH_CHECK_PTR(feats); WSPH_CHECK_PTR(target);
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        attr_err = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, train_smem_bytes());
    });
    if (attr_err != cudaSuccess) return set_error(SPH_ERR_CUDA, "sph_mlp_grad: shared memory opt-in: %s", cudaGetErrorString(attr_err));
    const int64_t tiles = (n + 16 * MLP_WARPS - 1) / (16 * MLP_WARPS);
    const int grid = (int)(tiles < 148 * 2 ? tiles : 148 * 2);
    count_launch();
    k_mlp_grad<<<grid, MLP_THREADS, train_smem_bytes(), s>>>(params, n, feats, target, grad, loss);
    return check_launch("sph_mlp_grad");
}

int sph_mlp_grad_tc(const float* params, int64_t n, const float* feats, const float* target, float* grad, double* loss,
                    int32_t* status, void* stream) {
    if (n < 0) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_grad_tc: n < 0");
    WSPH_CHECK_PTR(params); WSPH_CHECK_PTR(grad); WSPH_CHECK_PTR(loss);
    cudaStream_t s = WSPH_STREAM(stream);
    cudaMemsetAsync(grad, 0, sizeof(float) * MLP_NPARAM, s);
    cudaMemsetAsync(loss, 0, sizeof(double), s);
    if (n == 0) return check_launch("sph_mlp_grad_tc");
    WSPH_CHECK_PTR(feats); WSPH_CHECK_PTR(target);
    if (reinterpret_cast<uintptr_t>(feats) & 15) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_grad_tc: feats must be 16-byte aligned");
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        attr_err = cudaFuncSetAttribute(k_mlp_grad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, grad_tc_smem_bytes());
    });
    if (attr_err != cudaSuccess)
        return set_error(SPH_ERR_CUDA, "sph_mlp_grad_tc: shared memory opt-in: %s", cudaGetErrorString(attr_err));
    const int64_t tiles = (n + TC_M - 1) / TC_M;
    const int grid = (int)(tiles < 148 ? tiles : 148);
    count_launch();
    k_mlp_grad_tc<<<grid, GT_THREADS, grad_tc_smem_bytes(), s>>>(params, n, feats, target, grad, loss, status);
    return check_launch("sph_mlp_grad_tc");
}

int sph_mlp_adam(float* params, const float* grad, float* m1, float* m2, int64_t count, float lr, float beta1, float beta2, float eps,
                 int64_t step, void* stream) {
    if (count < 0 || step < 1) return set_error(SPH_ERR_BAD_ARG, "sph_mlp_adam: count < 0 or step < 1");
    if (count == 0) return SPH_OK;
    WSPH_CHECK_PTR(params); WSPH_CHECK_PTR(grad); WSPH_CHECK_PTR(m1); WSPH_CHECK_PTR(m2);
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    count_launch();
    k_mlp_adam<<<grid_for(count, 256), 256, 0, WSPH_STREAM(stream)>>>(params, grad, m1, m2, count, lr, beta1, beta2, eps, c1, c2);
    return check_launch("sph_mlp_adam");
}

}  // extern "C"
