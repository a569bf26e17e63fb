#pragma once
// Sums over the threads of a cluster of CTAs, for the kernel that ends a PCG iteration
// (pcg.cu): up to two scalars and nine coarse sums at a time. Every CTA sends its
// partials to every other through distributed shared memory, one cluster barrier, and
// all add them in the same order.
//
// Precision: a warp's 32 values of a scalar, and 256 of a coarse sum, are added in FP32;
// everything after that in FP64 or, where a thread has several values (kPairs), in
// float-float. FP64 instructions hold their warp's scheduler for 64 cycles on GB300, so
// only single warps take the FP64 sums.

#include "common.cuh"
#include "ff.cuh"

namespace gba {
namespace csum {

using ffa::ff;

constexpr int kNine = 9;       // coarse sums
constexpr int kMaxCtas = 16;
constexpr int kFoldRows = 8;   // values of a thread that may be added in FP32 before fold_nine

struct Shared {
    double slot[4][2 + kNine][kMaxCtas];  // partials of each CTA, for the four sums of an iteration
    double tot[kNine];
    float wp[2 + kNine][33];              // warp sums
    float wl[2 + kNine][33];              // their low parts (kPairs)
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Store v at `local`'s place in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ void cluster_store(double* local, int rank, double v) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(local))), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// a += t. kPairs: the rounding error is kept (a thread's one value otherwise).
template <bool kPairs>
__device__ __forceinline__ void add_term(ff& a, float t) {
    if constexpr (kPairs) {
        float s, e;
        ffa::two_sum(a.hi, t, s, e);
        a.hi = s;
        a.lo = __fadd_rn(a.lo, e);
    } else {
        a.hi += t;
    }
}

// The warp's sums of v[0 .. 9), to acc: lanes 2 j and 2 j + 1 hold sum j. The values and
// the lanes that hold them are halved in turn.
template <bool kPairs>
__device__ __forceinline__ void fold_nine(const float* v, ff& acc) {
    const int lane = threadIdx.x & 31;
    float a[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) a[j] = j < kNine ? v[j] : 0.f;
#pragma unroll
    for (int o = 16, h = 8; h >= 1; o >>= 1, h >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const float keep = up ? a[j + h] : a[j], send = up ? a[j] : a[j + h];
            a[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    add_term<kPairs>(acc, a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1));
}

__device__ __forceinline__ ff warp_total(ff a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = ffa::add(a, ffa::shfl_xor(a, o));
    return a;
}

// Totals over the cluster of NS <= 2 scalars (s[0 .. NS)) and, with kWithNine, of nine
// coarse sums (the warps' folded sums in nine; into sm.tot). fin(t0, t1) runs in thread
// 0 with the scalars' totals; what it writes to shared memory is visible to every
// thread on return. A scalar's warps are added by one warp (warp j for scalar j), the
// nine sums by four lanes each of warps 2 and 3 (eight warps a lane), then the CTAs'
// partials the same way. Each call of a kernel takes its own `which`.
template <int NS, bool kWithNine, bool kPairs, class Fin>
__device__ __forceinline__ void totals(const ff (&s)[2], ff nine_sum, Shared& sm, int which, int rank, int nctas, Fin fin) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    double(&slot)[2 + kNine][kMaxCtas] = sm.slot[which];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        if constexpr (kPairs) {
            const ff t = warp_total(s[j]);
            if (lane == 0) {
                sm.wp[j][warp] = t.hi;
                sm.wl[j][warp] = t.lo;
            }
        } else {
            const float t = warp_sum(s[j].hi);
            if (lane == 0) sm.wp[j][warp] = t;
        }
    }
    if constexpr (kWithNine) {
        if (!(lane & 1) && lane < 2 * kNine) {
            sm.wp[NS + (lane >> 1)][warp] = nine_sum.hi;
            if constexpr (kPairs) sm.wl[NS + (lane >> 1)][warp] = nine_sum.lo;
        }
    }
    __syncthreads();
    if (warp < NS) {
        double d;
        if constexpr (kPairs) {
            d = ffa::to_double(warp_total(lane < nw ? ff{sm.wp[warp][lane], sm.wl[warp][lane]} : ff{0.f, 0.f}));
        } else {
            d = lane < nw ? static_cast<double>(sm.wp[warp][lane]) : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        }
        if (lane < nctas) cluster_store(&slot[warp][rank], lane, d);
    }
    const int j9 = NS + ((tid - 64) >> 2), g = tid & 3;
    const bool nine = kWithNine && (warp == 2 || warp == 3);
    if (nine) {
        double d = 0.0;
        if (j9 < NS + kNine) {
            const int w1 = min(8 * g + 8, nw);
            if constexpr (kPairs) {
                ff f = {0.f, 0.f};
                for (int w = 8 * g; w < w1; ++w) f = ffa::add(f, ff{sm.wp[j9][w], sm.wl[j9][w]});
                d = ffa::to_double(f);
            } else {
                float f = 0.f;
                for (int w = 8 * g; w < w1; ++w) f += sm.wp[j9][w];
                d = static_cast<double>(f);
            }
        }
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        if (j9 < NS + kNine)
            for (int c = g; c < nctas; c += 4) cluster_store(&slot[j9][rank], c, d);
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (NS > 0 && warp == 0) {  // scalar 0 on the lower lanes, scalar 1 on the upper ones
        const int c = lane & 15;
        double d = c < nctas && (NS == 2 || lane < 16) ? slot[lane >> 4][c] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        const double d1 = NS == 2 ? __shfl_sync(0xffffffffu, d, 16) : 0.0;
        if (lane == 0) fin(d, d1);
    }
    if (nine) {
        double d = 0.0;
        if (j9 < NS + kNine)
            for (int c = g; c < nctas; c += 4) d += slot[j9][c];
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        if (g == 0 && j9 < NS + kNine) sm.tot[j9 - NS] = d;
    }
    __syncthreads();
}

}  // namespace csum
}  // namespace gba
