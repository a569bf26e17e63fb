// Learned coarse-space correction: MLP training and inference kernels.
//
//   forward    one kernel: 32 rows of the batch per CTA through all three layers
//              (mma.sync.m16n8k16 BF16 x BF16 -> FP32, weights and activations in
//              shared memory). A batch is a few thousand rows of 37,000 products each:
//              the launch and the weights' trip from L2 bound it, not the tensor cores.
//   backward   one kernel for both input gradients and each CTA's share of the
//              parameter gradients (its rows), one that adds the shares in order;
//              from the loss gradient w.r.t. the outputs (the loss, the
//              eigenvector share outside the coarse space, is a global function
//              of all cameras' outputs; the training script forms its gradient).
//   Adam       FP32 masters, BF16 copies refreshed after each step.
//   inference  features of S_cc and the camera -> MLP -> coarse basis rows Z_c.
// No reference counterpart (the reference has no iterative solver).

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <random>
#include <stdexcept>
#include <vector>

#include "blocks.cuh"
#include "common.cuh"
#include "mlp.hpp"
#include "solver.hpp"

namespace gba {
namespace {

constexpr long long kW1 = 0, kB1 = kW1 + 1ll * kMlpH * kMlpIn, kW2 = kB1 + kMlpH, kB2 = kW2 + 1ll * kMlpH * kMlpH,
                    kW3 = kB2 + kMlpH, kB3 = kW3 + 1ll * kMlpOut * kMlpH;
constexpr long long kBf16Count = 1ll * kMlpH * kMlpIn + 1ll * kMlpH * kMlpH + 1ll * kMlpOut * kMlpH;

__device__ __forceinline__ __nv_bfloat16 to_bf16(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

constexpr int kRowsT = 32;    // rows of the batch per CTA
constexpr int kMT = 256;      // threads (8 warps)
constexpr int kLdIn = kMlpIn + 8, kLdH = kMlpH + 8, kLdOut = kMlpOut + 8;  // shared-memory strides (BF16 values)

__device__ __forceinline__ uint32_t pair_at(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint32_t pair_of(__nv_bfloat16 a, __nv_bfloat16 b) {
    return static_cast<uint32_t>(__bfloat16_as_ushort(a)) | (static_cast<uint32_t>(__bfloat16_as_ushort(b)) << 16);
}

// Rows x cols BF16 matrix (row-major, cols a multiple of 8) into shared memory of stride ld.
__device__ __forceinline__ void load_weights(const __nv_bfloat16* __restrict__ w, int rows, int cols,
                                             __nv_bfloat16* dst, int ld) {
    const int per = cols / 8;
    for (int i = threadIdx.x; i < rows * per; i += kMT)
        *reinterpret_cast<uint4*>(dst + (i / per) * ld + 8 * (i % per)) = reinterpret_cast<const uint4*>(w)[i];
}
// kRowsT rows of an FP32 matrix from row r0 (zeros from row B on) as BF16. The
// callers' matrices may start at any float: 16-byte loads where they start at 16 bytes.
__device__ __forceinline__ void load_rows(const float* __restrict__ x, int r0, int B, int cols, __nv_bfloat16* dst,
                                          int ld) {
    const int per = cols / 4;
    const bool wide = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    for (int i = threadIdx.x; i < kRowsT * per; i += kMT) {
        const int r = i / per, c = 4 * (i % per);
        const float* src = x + static_cast<long long>(r0 + r) * cols + c;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r0 + r < B) v = wide ? *reinterpret_cast<const float4*>(src) : make_float4(src[0], src[1], src[2], src[3]);
        __nv_bfloat16* d = dst + r * ld + c;
        d[0] = to_bf16(v.x);
        d[1] = to_bf16(v.y);
        d[2] = to_bf16(v.z);
        d[3] = to_bf16(v.w);
    }
}

// acc[mt] = A (kRowsT x K, row-major) times the n8 tile nt of B, K ascending. kTrans:
// B(k, n) = Bs[k][n], else Bs[n][k].
template <int K, bool kTrans>
__device__ __forceinline__ void rows_times(const __nv_bfloat16* As, int lda, const __nv_bfloat16* Bs, int ldb, int nt,
                                           float (&acc)[2][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[mt][q] = 0.f;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t b[2];
        const int n = 8 * nt + g, k = k0 + 2 * t;
        if (kTrans) {
            b[0] = pair_of(Bs[k * ldb + n], Bs[(k + 1) * ldb + n]);
            b[1] = pair_of(Bs[(k + 8) * ldb + n], Bs[(k + 9) * ldb + n]);
        } else {
            b[0] = pair_at(Bs + n * ldb + k);
            b[1] = pair_at(Bs + n * ldb + k + 8);
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const __nv_bfloat16* a0 = As + (16 * mt + g) * lda + k;
            const uint32_t a[4] = {pair_at(a0), pair_at(a0 + 8 * lda), pair_at(a0 + 8), pair_at(a0 + 8 * lda + 8)};
            mma_bf16(acc[mt], a, b);
        }
    }
}

struct ForwardSmem {
    __nv_bfloat16 w1[kMlpH * kLdIn], w2[kMlpH * kLdH], w3[kMlpOut * kLdH];
    __nv_bfloat16 x[kRowsT * kLdIn], h1[kRowsT * kLdH], h2[kRowsT * kLdH];
};

// The whole network for 32 rows per CTA. Bound by latency: 32 CTAs of 1000 rows
// each bring the 77 KB of weights from L2 and go through 16 K-steps. 1000 rows:
// 15 us, against 3 x 29 us for a GEMM per layer with the activations through
// memory. h1, h2 (FP32, for backward) may be null.
__global__ void __launch_bounds__(kMT) mlp_forward_kernel(const float* __restrict__ feat, int B,
                                                         const __nv_bfloat16* __restrict__ wb,
                                                         const float* __restrict__ params, float* __restrict__ h1,
                                                         float* __restrict__ h2, float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char mlp_smem[];
    ForwardSmem& sm = *reinterpret_cast<ForwardSmem*>(mlp_smem);
    const int r0 = blockIdx.x * kRowsT, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    load_rows(feat, r0, B, kMlpIn, sm.x, kLdIn);
    load_weights(wb, kMlpH, kMlpIn, sm.w1, kLdIn);
    load_weights(wb + 1ll * kMlpH * kMlpIn, kMlpH, kMlpH, sm.w2, kLdH);
    load_weights(wb + 1ll * kMlpH * kMlpIn + 1ll * kMlpH * kMlpH, kMlpOut, kMlpH, sm.w3, kLdH);
    __syncthreads();
    // a layer's output tile: + bias, ReLU, FP32 to global and BF16 for the next layer
    auto store = [&](float (&acc)[2][4], int nt, const float* bias, bool relu, float* dst, int ld, __nv_bfloat16* next) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = 16 * mt + g + (q >= 2 ? 8 : 0), n = 8 * nt + 2 * t + (q & 1);
                float v = acc[mt][q] + bias[n];
                if (relu) v = fmaxf(v, 0.f);
                if (dst && r0 + r < B) dst[static_cast<long long>(r0 + r) * ld + n] = v;
                if (next) next[r * kLdH + n] = to_bf16(v);
            }
    };
    float acc[2][4];
    for (int nt = warp; nt < kMlpH / 8; nt += kMT / 32) {
        rows_times<kMlpIn, false>(sm.x, kLdIn, sm.w1, kLdIn, nt, acc);
        store(acc, nt, params + kB1, true, h1, kMlpH, sm.h1);
    }
    __syncthreads();
    for (int nt = warp; nt < kMlpH / 8; nt += kMT / 32) {
        rows_times<kMlpH, false>(sm.h1, kLdH, sm.w2, kLdH, nt, acc);
        store(acc, nt, params + kB2, true, h2, kMlpH, sm.h2);
    }
    __syncthreads();
    for (int nt = warp; nt < kMlpOut / 8; nt += kMT / 32) {
        rows_times<kMlpH, false>(sm.h2, kLdH, sm.w3, kLdH, nt, acc);
        store(acc, nt, params + kB3, false, out, kMlpOut, nullptr);
    }
}

struct BackwardSmem {
    __nv_bfloat16 w3[kMlpOut * kLdH], w2[kMlpH * kLdH];
    __nv_bfloat16 x[kRowsT * kLdIn], h1[kRowsT * kLdH], h2[kRowsT * kLdH];
    __nv_bfloat16 d3[kRowsT * kLdOut], d2[kRowsT * kLdH], d1[kRowsT * kLdH];
    float f[kRowsT][kMlpH + 1];  // a layer's gradient in FP32, for its bias sums
};

// The rows' share of dW (n x k) = dY^T X: warp mt owns rows 16 mt .. of dW; added
// to what the CTA's earlier rows left when !first.
template <int NT>
__device__ __forceinline__ void weight_share(const __nv_bfloat16* dY, int ldy, const __nv_bfloat16* X, int ldx, int mt,
                                             float* __restrict__ dst, bool first) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    uint32_t a[2][4];
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        const __nv_bfloat16* y = dY + (16 * ks + 2 * t) * ldy + 16 * mt + g;
        a[ks][0] = pair_of(y[0], y[ldy]);
        a[ks][1] = pair_of(y[8], y[ldy + 8]);
        a[ks][2] = pair_of(y[8 * ldy], y[9 * ldy]);
        a[ks][3] = pair_of(y[8 * ldy + 8], y[9 * ldy + 8]);
    }
#pragma unroll 4
    for (int nt = 0; nt < NT; ++nt) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const __nv_bfloat16* x = X + (16 * ks + 2 * t) * ldx + 8 * nt + g;
            const uint32_t b[2] = {pair_of(x[0], x[ldx]), pair_of(x[8 * ldx], x[9 * ldx])};
            mma_bf16(acc, a[ks], b);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float2* d = reinterpret_cast<float2*>(dst + (16 * mt + g + 8 * q) * (8 * NT) + 8 * nt + 2 * t);
            float2 v = make_float2(acc[2 * q], acc[2 * q + 1]);
            if (!first) {
                const float2 o = *d;
                v.x += o.x;
                v.y += o.y;
            }
            *d = v;
        }
    }
}

// Each CTA takes the 32-row groups blockIdx.x, + gridDim.x, ...; its shares of
// the parameter gradients go to part (flat layout, kMlpParams per CTA) and, for
// the biases in FP64, to bpart (kH of b1, kH of b2, kOut of b3 per CTA).
// Bound by latency as the forward pass; the batch is the reduction axis of the
// weight gradients, so one GEMM per layer had 8 CTAs walk all rows in turn (290 us
// each at 1000 rows, 1.0 ms in all); split by rows and fused: 29 us + 5.5 us for
// the ordered sum of the shares. One CTA per SM at most keeps the shares at
// 150 KB x SMs; a CTA adds its later groups onto its own share.
constexpr int kBias = 2 * kMlpH + kMlpOut;
__global__ void __launch_bounds__(kMT) mlp_backward_kernel(const float* __restrict__ feat,
                                                          const float* __restrict__ dO, int B,
                                                          const __nv_bfloat16* __restrict__ wb,
                                                          const float* __restrict__ h1, const float* __restrict__ h2,
                                                          float* __restrict__ part, double* __restrict__ bpart) {
    extern __shared__ __align__(16) unsigned char mlp_smem[];
    BackwardSmem& sm = *reinterpret_cast<BackwardSmem*>(mlp_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    float* p = part + static_cast<long long>(blockIdx.x) * kMlpParams;
    double* bp = bpart + static_cast<long long>(blockIdx.x) * kBias;
    load_weights(wb + 1ll * kMlpH * kMlpIn, kMlpH, kMlpH, sm.w2, kLdH);
    load_weights(wb + 1ll * kMlpH * kMlpIn + 1ll * kMlpH * kMlpH, kMlpOut, kMlpH, sm.w3, kLdH);
    double b1 = 0.0, b2 = 0.0, b3 = 0.0;  // this thread's columns' bias sums
    for (int r0 = blockIdx.x * kRowsT; r0 < B; r0 += gridDim.x * kRowsT) {
        const bool first = r0 == static_cast<int>(blockIdx.x) * kRowsT;
        load_rows(feat, r0, B, kMlpIn, sm.x, kLdIn);
        load_rows(h1, r0, B, kMlpH, sm.h1, kLdH);
        load_rows(h2, r0, B, kMlpH, sm.h2, kLdH);
        load_rows(dO, r0, B, kMlpOut, sm.d3, kLdOut);
        const int rows = min(kRowsT, B - r0);
        if (threadIdx.x < kMlpOut)
#pragma unroll 8
            for (int r = 0; r < rows; ++r) b3 += dO[static_cast<long long>(r0 + r) * kMlpOut + threadIdx.x];
        __syncthreads();
        // dH = (dY W) where the layer's activation is positive
        auto masked = [&](float (&acc)[2][4], int nt, const float* h, __nv_bfloat16* d) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = 16 * mt + g + (q >= 2 ? 8 : 0), n = 8 * nt + 2 * t + (q & 1);
                    float v = 0.f;
                    if (r < rows && h[static_cast<long long>(r0 + r) * kMlpH + n] > 0.f) v = acc[mt][q];
                    d[r * kLdH + n] = to_bf16(v);
                    sm.f[r][n] = v;
                }
        };
        float acc[2][4];
        for (int nt = warp; nt < kMlpH / 8; nt += kMT / 32) {
            rows_times<kMlpOut, true>(sm.d3, kLdOut, sm.w3, kLdH, nt, acc);
            masked(acc, nt, h2, sm.d2);
        }
        __syncthreads();
        if (threadIdx.x < kMlpH)
            for (int r = 0; r < rows; ++r) b2 += sm.f[r][threadIdx.x];
        if (warp < kMlpOut / 16) weight_share<kMlpH / 8>(sm.d3, kLdOut, sm.h2, kLdH, warp, p + kW3, first);
        weight_share<kMlpH / 8>(sm.d2, kLdH, sm.h1, kLdH, warp, p + kW2, first);
        __syncthreads();
        for (int nt = warp; nt < kMlpH / 8; nt += kMT / 32) {
            rows_times<kMlpH, true>(sm.d2, kLdH, sm.w2, kLdH, nt, acc);
            masked(acc, nt, h1, sm.d1);
        }
        __syncthreads();
        if (threadIdx.x < kMlpH)
            for (int r = 0; r < rows; ++r) b1 += sm.f[r][threadIdx.x];
        weight_share<kMlpIn / 8>(sm.d1, kLdH, sm.x, kLdIn, warp, p + kW1, first);
        __syncthreads();
    }
    if (threadIdx.x < kMlpH) {
        bp[threadIdx.x] = b1;
        bp[kMlpH + threadIdx.x] = b2;
    }
    if (threadIdx.x < kMlpOut) bp[2 * kMlpH + threadIdx.x] = b3;
}

// The CTAs' shares added in order.
__global__ void __launch_bounds__(256) mlp_grad_sum_kernel(const float* __restrict__ part,
                                                          const double* __restrict__ bpart, int n,
                                                          float* __restrict__ grad) {
    const long long i = blockIdx.x * 256ll + threadIdx.x;
    if (i >= kMlpParams) return;
    const long long at = i >= kB3 ? i - kB3 + 2 * kMlpH : i >= kB2 && i < kW3 ? i - kB2 + kMlpH
                         : i >= kB1 && i < kW2 ? i - kB1 : -1;  // among the biases
    if (at >= 0) {
        double s = 0.0;
        for (int c = 0; c < n; ++c) s += bpart[static_cast<long long>(c) * kBias + at];
        grad[i] = static_cast<float>(s);
    } else {
        float s = 0.f;
#pragma unroll 8
        for (int c = 0; c < n; ++c) s += part[c * kMlpParams + i];
        grad[i] = s;
    }
}

__global__ void to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16_rn(src[i]);
}

// Adam on the FP32 masters, and the weights' BF16 copies.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float c1,
                            float c2, __nv_bfloat16* __restrict__ wb) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        const long long w = i < kB1 ? i : i >= kW2 && i < kB2 ? i - kMlpH : i >= kW3 && i < kB3 ? i - 2 * kMlpH : -1;
        if (w >= 0) wb[w] = to_bf16(pi);
    }
}

// ---- inference-side kernels

// Per-camera track statistics: observations, sum of (track length - 1), mean track length.
__global__ void camera_stats_kernel(const int* __restrict__ cam_off, const int* __restrict__ cam_slots,
                                    const int* __restrict__ s_pt, const int* __restrict__ pt_off, int C,
                                    float* __restrict__ stats) {
    const int c = blockIdx.x;
    __shared__ double sh[8];
    double s1 = 0.0;
    for (int i = cam_off[c] + threadIdx.x; i < cam_off[c + 1]; i += 256) {
        const int p = s_pt[cam_slots[i]];
        s1 += pt_off[p + 1] - pt_off[p];
    }
    const double sk = block_sum<256>(s1, sh);
    if (threadIdx.x == 0) {
        const double n = cam_off[c + 1] - cam_off[c];
        stats[3 * c] = static_cast<float>(log1p(n) / 10.0);
        stats[3 * c + 1] = static_cast<float>(log1p(sk - n) / 15.0);
        stats[3 * c + 2] = static_cast<float>(n > 0 ? sk / n / 10.0 : 0.0);
    }
}

// Per-camera FP64 kernels (features, factor correction): one camera per
// thread in warp-sized blocks, so that C cameras spread over all SMs' FP64
// pipes.
constexpr int kCamT = 32;

__global__ void features_kernel(const double* __restrict__ Sdiag, const double* __restrict__ U,
                                const float* __restrict__ stats, const double* __restrict__ cams, double lambda,
                                int C, float* __restrict__ feat) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const double* S = Sdiag + 81ll * c;
    const double* Uc = U + 81ll * c;
    double isd[9];
    float* f = feat + 64ll * c;
    for (int i = 0; i < 9; ++i) {
        const double d = S[10 * i];
        isd[i] = d > 1e-300 ? 1.0 / sqrt(d) : 0.0;
        const double u = Uc[10 * i];
        const double ud = u + lambda * (u > 0.0 ? u : 1e-12);
        f[36 + i] = static_cast<float>(ud > 0.0 ? d / ud : 0.0);
    }
    int k = 0;
    for (int i = 1; i < 9; ++i)
        for (int j = 0; j < i; ++j) f[k++] = static_cast<float>(S[9 * i + j] * isd[i] * isd[j]);
    f[45] = stats[3 * c];
    f[46] = stats[3 * c + 1];
    f[47] = stats[3 * c + 2];
    f[48] = static_cast<float>(log10(lambda > 1e-300 ? lambda : 1e-300) / 10.0);
    const double* cam = cams + 9ll * c;
    for (int i = 0; i < 3; ++i) f[49 + i] = static_cast<float>(3.0 * cam[i]);
    for (int i = 0; i < 3; ++i) f[52 + i] = static_cast<float>(0.5 * cam[3 + i]);
    f[55] = static_cast<float>((cam[6] - 500.0) / 100.0);
    f[56] = static_cast<float>(10.0 * cam[7]);
    f[57] = static_cast<float>(100.0 * cam[8]);
    for (int i = kMlpUsedIn; i < 64; ++i) f[i] = 0.f;
}

// Coarse basis rows of camera c from the network outputs:
// Z[j][9c + i] = o[9 i + j] * unit_i (unit 1, the focal-length row f_c). A camera
// without observations gets zero rows: its block of S is decoupled (only the
// damping's 1e-12 floor), its right-hand side zero, and its step must stay zero.
__global__ void basis_kernel(const float* __restrict__ O, const double* __restrict__ cams,
                             const int* __restrict__ cam_off, int C, double* __restrict__ Z) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const double f = cams[9ll * c + 6];
    const bool observed = cam_off[c + 1] > cam_off[c];
    const long long n = 9ll * C;
    for (int i = 0; i < 9; ++i) {
        const double unit = !observed ? 0.0 : i == 6 ? f : 1.0;
        for (int j = 0; j < kCoarse; ++j) Z[j * n + 9ll * c + i] = unit * O[static_cast<long long>(kMlpOut) * c + 9 * i + j];
    }
}

template <typename T>
T* dalloc(long long n) {
    T* p = nullptr;
    GBA_CUDA_CHECK(cudaMalloc(reinterpret_cast<void**>(&p), sizeof(T) * n));
    return p;
}

// Stream-ordered allocation from the device's memory pool (inference mode).
template <typename T>
T* palloc(long long n, cudaStream_t s) {
    T* p = nullptr;
    GBA_CUDA_CHECK(cudaMallocAsync(reinterpret_cast<void**>(&p), sizeof(T) * n, s));
    return p;
}

const char kMagic[8] = {'G', 'B', 'A', 'M', 'L', 'P', '0', '2'};

std::vector<float> read_model(const std::string& path) {
    std::ifstream f(path, std::ios::binary);
    if (!f) throw std::runtime_error("cannot open model " + path);
    char magic[8];
    int32_t dims[3];
    f.read(magic, 8);
    f.read(reinterpret_cast<char*>(dims), sizeof dims);
    if (!f || std::memcmp(magic, kMagic, 8) != 0 || dims[0] != kMlpIn || dims[1] != kMlpH || dims[2] != kMlpOut)
        throw std::runtime_error("not a gba MLP model: " + path);
    std::vector<float> h(kMlpParams);
    f.read(reinterpret_cast<char*>(h.data()), sizeof(float) * kMlpParams);
    if (!f) throw std::runtime_error("truncated model " + path);
    return h;
}

}  // namespace

// ------------------------------------------------------------------ Mlp

// CTAs of the backward kernel: one per 32 rows, at most one per SM (more rows: several groups each).
static int backward_ctas(int B) { return std::min(ceil_div(B, kRowsT), device_sm_count()); }

void Mlp::alloc() {
    p_ = dalloc<float>(kMlpParams);
    g_ = dalloc<float>(kMlpParams);
    m_ = dalloc<float>(kMlpParams);
    v_ = dalloc<float>(kMlpParams);
    wb_ = dalloc<__nv_bfloat16>(kBf16Count);
    GBA_CUDA_CHECK(cudaMemset(g_, 0, sizeof(float) * kMlpParams));
    GBA_CUDA_CHECK(cudaMemset(m_, 0, sizeof(float) * kMlpParams));
    GBA_CUDA_CHECK(cudaMemset(v_, 0, sizeof(float) * kMlpParams));
    ensure_capacity(cap_);
}

void Mlp::ensure_capacity(int B) {
    if (B <= cap_ && (h1_ || inference_)) return;
    cap_ = std::max(B, std::max(cap_, 1));
    if (inference_) return;  // the activations stay in shared memory
    for (void* q : {static_cast<void*>(h1_), static_cast<void*>(h2_), static_cast<void*>(part_),
                    static_cast<void*>(bpart_)})
        if (q) cudaFree(q);
    h1_ = dalloc<float>(1ll * cap_ * kMlpH);
    h2_ = dalloc<float>(1ll * cap_ * kMlpH);
    const int ctas = backward_ctas(cap_);
    part_ = dalloc<float>(ctas * kMlpParams);
    bpart_ = dalloc<double>(1ll * ctas * kBias);
}

Mlp::Mlp(int capacity, uint64_t seed) : cap_(capacity) {
    alloc();
    std::vector<float> h(kMlpParams, 0.f);
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    const float s1 = std::sqrt(2.f / kMlpUsedIn), s2 = std::sqrt(2.f / kMlpH);
    for (int r = 0; r < kMlpH; ++r)
        for (int c = 0; c < kMlpUsedIn; ++c) h[kW1 + 1ll * r * kMlpIn + c] = s1 * nd(rng);
    for (long long i = 0; i < 1ll * kMlpH * kMlpH; ++i) h[kW2 + i] = s2 * nd(rng);
    const float s3 = 0.1f * s2;  // a small random last layer: a full-rank basis to start from
    for (int r = 0; r < kMlpUsedOut; ++r)
        for (int c = 0; c < kMlpH; ++c) h[kW3 + 1ll * r * kMlpH + c] = s3 * nd(rng);
    set_params(h.data());
}

Mlp::Mlp(const std::string& path, int capacity) : cap_(capacity) {
    const std::vector<float> h = read_model(path);
    alloc();
    set_params(h.data());
}

Mlp::Mlp(const std::string& path, cudaStream_t stream)
    : pool_stream_(stream), inference_(true), host_params_(read_model(path)) {
    p_ = palloc<float>(kMlpParams, stream);
    wb_ = palloc<__nv_bfloat16>(kBf16Count, stream);
    GBA_CUDA_CHECK(cudaMemcpyAsync(p_, host_params_.data(), sizeof(float) * kMlpParams, cudaMemcpyHostToDevice,
                                   stream));
    refresh_bf16(stream);
}

void Mlp::require_training() const {
    if (inference_) throw std::logic_error("this MLP was loaded for inference only");
}

Mlp::~Mlp() {
    if (inference_) {
        for (void* q : {static_cast<void*>(p_), wb_})
            if (q) cudaFreeAsync(q, pool_stream_);
        return;
    }
    for (void* q : {static_cast<void*>(p_), static_cast<void*>(g_), static_cast<void*>(m_), static_cast<void*>(v_), wb_,
                    static_cast<void*>(h1_), static_cast<void*>(h2_), static_cast<void*>(part_),
                    static_cast<void*>(bpart_)})
        if (q) cudaFree(q);
}

void Mlp::save(const std::string& path) const {
    std::vector<float> h(kMlpParams);
    get_params(h.data());
    std::ofstream f(path, std::ios::binary);
    if (!f) throw std::runtime_error("cannot write model " + path);
    const int32_t dims[3] = {kMlpIn, kMlpH, kMlpOut};
    f.write(kMagic, 8);
    f.write(reinterpret_cast<const char*>(dims), sizeof dims);
    f.write(reinterpret_cast<const char*>(h.data()), sizeof(float) * kMlpParams);
    if (!f) throw std::runtime_error("write failed for " + path);
}

void Mlp::get_params(float* host) const {
    GBA_CUDA_CHECK(cudaMemcpy(host, p_, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
}

void Mlp::set_params(const float* host) {
    GBA_CUDA_CHECK(cudaMemcpy(p_, host, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
    refresh_bf16(nullptr);
    GBA_CUDA_CHECK(cudaStreamSynchronize(nullptr));
}

void Mlp::grads(float* host) const {
    require_training();
    GBA_CUDA_CHECK(cudaDeviceSynchronize());
    GBA_CUDA_CHECK(cudaMemcpy(host, g_, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
}

void Mlp::refresh_bf16(cudaStream_t s) {
    __nv_bfloat16* wb = static_cast<__nv_bfloat16*>(wb_);
    to_bf16_kernel<<<64, 256, 0, s>>>(p_ + kW1, wb, 1ll * kMlpH * kMlpIn);
    GBA_LAUNCH_CHECK();
    to_bf16_kernel<<<64, 256, 0, s>>>(p_ + kW2, wb + 1ll * kMlpH * kMlpIn, 1ll * kMlpH * kMlpH);
    GBA_LAUNCH_CHECK();
    to_bf16_kernel<<<64, 256, 0, s>>>(p_ + kW3, wb + 1ll * kMlpH * kMlpIn + 1ll * kMlpH * kMlpH, 1ll * kMlpOut * kMlpH);
    GBA_LAUNCH_CHECK();
}

void Mlp::forward(const float* feat, int B, float* out, cudaStream_t s) {
    ensure_capacity(B);
    GBA_CUDA_CHECK(cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        sizeof(ForwardSmem)));
    mlp_forward_kernel<<<ceil_div(B, kRowsT), kMT, sizeof(ForwardSmem), s>>>(
        feat, B, static_cast<const __nv_bfloat16*>(wb_), p_, h1_, h2_, out);
    GBA_LAUNCH_CHECK();
}

void Mlp::backward(const float* feat, const float* dO, int B, cudaStream_t s) {
    require_training();
    if (B <= 0 || B > cap_) throw std::invalid_argument("backward: batch must be the last forward's (<= capacity)");
    GBA_CUDA_CHECK(cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        sizeof(BackwardSmem)));
    const int ctas = backward_ctas(B);
    mlp_backward_kernel<<<ctas, kMT, sizeof(BackwardSmem), s>>>(
        feat, dO, B, static_cast<const __nv_bfloat16*>(wb_), h1_, h2_, part_, bpart_);
    GBA_LAUNCH_CHECK();
    mlp_grad_sum_kernel<<<ceil_div(kMlpParams, 256), 256, 0, s>>>(part_, bpart_, ctas, g_);
    GBA_LAUNCH_CHECK();
}

void Mlp::adam_step(float lr, float beta1, float beta2, float eps, cudaStream_t s) {
    require_training();
    ++step_;
    const float c1 = 1.f - std::pow(beta1, static_cast<float>(step_));
    const float c2 = 1.f - std::pow(beta2, static_cast<float>(step_));
    adam_kernel<<<120, 256, 0, s>>>(p_, g_, m_, v_, kMlpParams, lr, beta1, beta2, eps, c1, c2,
                                    static_cast<__nv_bfloat16*>(wb_));
    GBA_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ solver side

void mlp_features(Solver& s, double lambda, float* feat) {
    if (!s.mlp_stats_.get()) {
        StreamAllocScope scope(s.stream_);
        s.mlp_stats_.alloc(3ull * s.C_);
        camera_stats_kernel<<<s.C_, 256, 0, s.stream_>>>(s.cam_off_.get(), s.cam_slots_.get(), s.s_pt_.get(),
                                                          s.pt_off_.get(), s.C_, s.mlp_stats_.get());
        GBA_LAUNCH_CHECK();
    }
    features_kernel<<<ceil_div(s.C_, kCamT), kCamT, 0, s.stream_>>>(s.Sdiag_.get(), s.U_.get(), s.mlp_stats_.get(),
                                                                 s.cams_.get(), lambda, s.C_, feat);
    GBA_LAUNCH_CHECK();
}

LearnedPreconditioner::LearnedPreconditioner(const std::string& path, cudaStream_t stream)
    : mlp_(path, stream), stream_(stream) {}

LearnedPreconditioner::~LearnedPreconditioner() {
    if (feat_) cudaFreeAsync(feat_, stream_);
    if (out_) cudaFreeAsync(out_, stream_);
}

void LearnedPreconditioner::coarse_basis(Solver& s, double lambda, double* Z) {
    if (cap_ < s.C_) {
        if (feat_) GBA_CUDA_CHECK(cudaFreeAsync(feat_, stream_));
        if (out_) GBA_CUDA_CHECK(cudaFreeAsync(out_, stream_));
        feat_ = palloc<float>(64ll * s.C_, stream_);
        out_ = palloc<float>(1ll * kMlpOut * s.C_, stream_);
        cap_ = s.C_;
    }
    mlp_features(s, lambda, feat_);
    cudaEvent_t ev = s.prof_start();
    mlp_.forward(feat_, s.C_, out_, s.stream_);
    s.prof_stop("mlp_forward", ev);
    basis_kernel<<<ceil_div(s.C_, kCamT), kCamT, 0, s.stream_>>>(out_, s.cams_.get(), s.cam_off_.get(), s.C_, Z);
    GBA_LAUNCH_CHECK();
}

Solver::~Solver() {
    prof_reset();
    delete model_;
    if (sync_ev_) cudaEventDestroy(sync_ev_);
}

void Solver::load_model(const std::string& path) {
    if (form_ == SolverForm::Plain) throw std::invalid_argument("the learned preconditioner needs a mixed form");
    if (path.empty()) throw std::invalid_argument("learned form: empty model path");
    auto* m = new LearnedPreconditioner(path, stream_);
    delete model_;
    model_ = m;
}

}  // namespace gba
