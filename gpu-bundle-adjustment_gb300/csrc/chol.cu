// Blocked Cholesky factorisation of dense and band SPD matrices in scaled
// 64-bit fixed point (fix64.cuh), with the trailing update on the 5th-generation
// tensor cores.
//
// Reference: the host Eigen LLT of the reduced camera system (src/lm.cu:598-604).
//
// GB300's FP64 pipe is the bound of an FP64 factorisation: 1.05 TFLOP/s for the
// chip, 64 cycles per warp FMA, whether by DFMA or DMMA. Here no FP64
// arithmetic is left on the path:
//   scale     row exponents e_i from the diagonal (A_ii 2^(-2 e_i) in [1/8, 1/2))
//   convert   the lower triangle, in place, to 64-bit integers (2^-62 units)
//   per 64-column panel
//     panel   the 64 x 64 diagonal tile and the rows below it (chol_panel): the
//             factor's columns as FP64 in place, and the rows' base-512 digits
//             as FP16 tiles for the update
//     update  C -= L L^T over the remaining lower tiles (chol_update): the
//             digit products by tcgen05.mma (FP16 in, FP32 accumulators in
//             TMEM, exact: small integers), recombined into the 64-bit entries;
//             or, where few tiles are left, by integer multiply-adds (chol_update_int)
// A band is eliminated from both of its ends at once (band_potrf_twisted).
// Every entry is a sum of products rounded at 2^-62 of sqrt(A_ii A_jj) once a panel (a
// factor's at 2^-60). Against long double the factor is closer to the exact one than
// that of the FP64 kernels (dense.cu): 192 rows 5.0e-17 against 2.4e-16 at condition 20,
// 9.2e-17 against 13.2e-16 at 4e3, 3.1e-16 against 4.4e-15 at 4e5, 1.1e-15 against
// 9.4e-15 at 4e7; so is the solution (4,096 rows 6.4e-16 against 1.45e-15).
//
// A row that cannot belong to an SPD matrix (a diagonal entry that is not
// positive, an entry that is not finite or larger than the diagonal allows, a
// row of the factor that outgrows its diagonal entry) is marked in bad[]: its
// entries count as zero, and the factorisation stops at its pivot, as FP64
// arithmetic does at the negative or NaN pivot it meets there. An infinite
// diagonal entry is a pivot of weight infinity: its row and column of the
// factor are zero (a row with an entry there that is not finite is marked, and a row of
// infinite weight with an entry whose factor's square FP64 does not hold).
//
// Tile addressing: element (i, j) at A[i + j lda] in both layouts (dense.cu).

#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "fix64.cuh"
#include "solver.hpp"

namespace gba {
namespace {

using fx::Acc29;
using fx::Limbs29;

constexpr int NB = 64;                        // panel width / tile size
constexpr int kTileB = NB * NB * 2;           // bytes of one FP16 digit tile
constexpr int kNS = fx::kSlices;

// Workspace: digit tiles (kNS per 64-row tile), which small updates replace by the
// panel's rows as integers (64 per row), row exponents, row flags, and a diagonal
// tile of the factor per chain on its way to the matrix.
constexpr int kMaxChains = 2;
struct Work {
    unsigned char* tiles;
    long long* rows;
    int* e;
    int* bad;  // 1: fails at this row's pivot; 2: infinite diagonal entry
    double* diag;
};
Work carve(void* ws, int n) {
    Work w;
    w.tiles = static_cast<unsigned char*>(ws);
    w.rows = static_cast<long long*>(ws);
    w.e = reinterpret_cast<int*>(w.tiles + static_cast<size_t>(n / NB) * kNS * kTileB);
    w.bad = w.e + n;
    w.diag = reinterpret_cast<double*>(w.bad + n);  // (n is a multiple of 64)
    return w;
}

__global__ void chol_scale(const double* __restrict__ A, int n, int lda, int* __restrict__ e, int* __restrict__ bad,
                           int* __restrict__ info) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *info = 0;
    if (i >= n) return;
    const double d = A[i + static_cast<long long>(i) * lda];
    const bool ok = fx::finite_positive(d);
    e[i] = ok ? fx::row_exponent(d) : 0;
    bad[i] = ok ? 0 : d > 0.0 ? 2 : 1;
}

// Entry v of a row and a column with exponents ei, ej in fixed point; inf_row, inf_col:
// their diagonal entries are infinite.
__device__ __forceinline__ long long convert_entry(double v, int ei, int ej, bool inf_row, bool inf_col, bool diagonal,
                                                   bool* bad) {
    if (!inf_row && !inf_col) return fx::to_fixed<fx::kFracC>(v, ei + ej, bad);
    if (!diagonal && v != 0.0) {
        int x;
        uint64_t m;
        fx::decompose(v, &x, &m);  // x = 1024: infinite or not a number
        *bad = x == 1024 || (!inf_col && x - ej >= 511);
    }
    return 0;
}

// One CTA per lower tile (ti, tj), ti - tj <= bt: FP64 -> fixed point in place.
// The strict upper triangle of a diagonal tile is not touched.
__global__ void __launch_bounds__(256) chol_convert(double* __restrict__ A, int nt, int lda, int bt,
                                                   const int* __restrict__ e, int* __restrict__ bad) {
    const int tj = blockIdx.x, ti = tj + blockIdx.y;
    if (ti >= nt) return;
    pdl_wait();
    pdl_trigger();
    const int r = threadIdx.x & 63, i = ti * NB + r;
    const int ei = e[i];
    const bool inf_row = bad[i] == 2;
    long long* F = reinterpret_cast<long long*>(A);
    bool mine = false;
    double v[16];
    int ec[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int j = tj * NB + (threadIdx.x >> 6) + 4 * k;
        v[k] = j <= i ? A[i + static_cast<long long>(j) * lda] : 0.0;
        ec[k] = e[j];
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int j = tj * NB + (threadIdx.x >> 6) + 4 * k;
        if (j > i) continue;
        bool b = false;
        const long long f = convert_entry(v[k], ei, ec[k], inf_row, bad[j] == 2, i == j, &b);
        F[i + static_cast<long long>(j) * lda] = f;
        mine = mine || b;
    }
    if (mine) bad[i] = 1;
}

// ---------------------------------------------------------------- panel
//
// One CTA factors the panel's diagonal tile (every CTA of the grid does, each
// for itself: the tile is the critical path, and the SMs would idle otherwise)
// together with 16 rows below it, then solves the further rows it was given. No CTA
// writes that tile of the matrix: beside other work on the GPU some CTAs start only
// when others have ended, and read it then. Its factor goes to the workspace, and the
// update that follows puts it in its place.
//
// What bounds it is the chain of 64 pivots, each a reciprocal square root and
// three dependent 64-bit products (some 400 cycles), so one warp does nothing
// else, alone on its SM sub-partition: the pivot warp holds a window of 32 rows,
// one per lane (rows 0 to 31 of the tile for its first 32 columns, then rows 32 to
// 63), and advances four columns a round without waiting for anybody: it
// applies the previous round's rank-4 update to the next four columns itself.
// On the other three sub-partitions ten warps hold all rows (a thread owns one
// row and the columns j = 4 m + q of it, as 64-bit accumulators that shift
// down by one slot a round) and apply the rounds' updates, the window's
// columns two rounds ahead first; two warps solve the rows outside the window, a
// row per lane, a round behind the pivot warp. The solving warps, whose chain
// the others wait for, share theirs with the two lightest updating warps.
constexpr int kWin = 32;                  // rows of the pivot warp's window
constexpr int kExtra = 16;                // rows below the tile in the first group
constexpr int kRows = NB + kExtra;
constexpr int kOut = kRows - kWin;        // rows outside the first window
constexpr int kUpdateWarps = kRows / 8;
constexpr int kWorkers = 32 * (kUpdateWarps + 2);  // threads of the updating and solving warps
constexpr int kPanelThreads = 512;        // warps 4, 8, 12 share the pivot warp's sub-partition and rest
constexpr int kRows2 = kPanelThreads / 4; // rows per pass of the further rows
constexpr int kLvS = NB + 1;              // stride of the row-major factor values
constexpr int kLS = NB + 2;               // stride of the limbs of a row (16-byte aligned)

struct PanelSmem {
    Limbs29 L[NB * kLS];         // [row][column] limbs of the diagonal tile's factor
    Limbs29 lx[kExtra * 4];      // [row][4] limbs of the current columns, rows below the tile
    long long xw[2][4][kWin];    // the window's columns of a round (by the round's parity), in quarter units
    long long xn[4][kOut];       // the current four columns of the other rows, in quarter units
    long long lv[kRows2 * kLvS]; // factor values by row, for the output
    fx::Rsqrt y[NB];             // reciprocal pivots (y0 = 0: a pivot of weight infinity)
    float rest[kWin];            // rows 32 to 63: what their squares leave of the diagonal entry
    int diag_bad[NB];
    int fail;                    // 1 + failed column of the tile
    int fail_round;              // 1 + the round it is in (the pivot warp runs ahead of the others' checks)
};

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
// Named barriers: the window's columns of round b are there; round b's pivots
// are, for the updating and for the solving warps (apart: the solving warps
// must not wait for the updating ones' last round); the solving warps are done;
// the next columns are published; rows 32 to 63 are solved for columns 28 to
// 31. The pivot warp is at most two rounds ahead of the updating warps (it waits for
// the window's columns) and three of the solving ones, hence the two and four
// barriers in turn.
__device__ __forceinline__ int bar_window(int b) { return 1 + (b & 1); }
__device__ __forceinline__ int bar_pivots(int b) { return 3 + (b & 1); }
__device__ __forceinline__ int bar_pivots_solving(int b) { return 8 + (b & 3); }
constexpr int kBarSolved = 5, kBarNext = 6, kBarHandover = 7;
constexpr int kWindowCount = 32 + 32 * kUpdateWarps, kPivotsCount = 32 + 32 * kUpdateWarps, kPivotsSolving = 32 + 64;

// Limbs of four consecutive columns.
__device__ __forceinline__ void load_limbs4(const Limbs29* p, Limbs29 (&l)[4]) {
    const int4 a = reinterpret_cast<const int4*>(p)[0], b = reinterpret_cast<const int4*>(p)[1];
    l[0] = {a.x, a.y};
    l[1] = {a.z, a.w};
    l[2] = {b.x, b.y};
    l[3] = {b.z, b.w};
}
__device__ __forceinline__ void store_limbs4(Limbs29* p, const Limbs29 (&l)[4]) {
    reinterpret_cast<int4*>(p)[0] = make_int4(l[0].hi, l[0].lo, l[1].hi, l[1].lo);
    reinterpret_cast<int4*>(p)[1] = make_int4(l[2].hi, l[2].lo, l[3].hi, l[3].lo);
}

// Squares of a row of the factor against its diagonal entry: a row that outgrows
// it is not of an SPD matrix.
__device__ __forceinline__ float square_of(long long x) {
    const float f = static_cast<float>(static_cast<int>(x >> 32)) * 0x1p-28f;
    return f * f;
}

// The pivot warp (rows 32 (b / 8) + lane in round b).
__device__ __forceinline__ void pivot_warp(PanelSmem& sm, float diag) {
    const int lane = threadIdx.x;
    float rest = diag;
    int state = sm.diag_bad[lane];  // 1: the row has failed, 2: a pivot of weight infinity
    Limbs29 prev[4];
#pragma unroll 1
    for (int b = 0; b < 16; ++b) {
        const int k0 = 4 * b, row = (b >> 3) * kWin + lane, p0 = k0 & (kWin - 1);
        bar_sync(bar_window(b), kWindowCount);
        if (b == 8) {  // the second window's rows come from the solving warp
            bar_sync(kBarHandover, 64);
            load_limbs4(sm.L + row * kLS + k0 - 4, prev);
            rest = sm.rest[lane];
            state = sm.diag_bad[row];
        }
        Acc29 t[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) t[c] = {sm.xw[b & 1][c][lane], 0};
        if (b > 0) {  // the previous round's update of these columns
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                Limbs29 l[4];
                load_limbs4(sm.L + (k0 + c) * kLS + k0 - 4, l);
#pragma unroll
                for (int k = 0; k < 4; ++k) fx::fms(t[c], prev[k], l[k]);
            }
        }
        long long x[4], dv = fx::value(t[0]);  // dv: the pivot, on its row's lane
        int fail = 0;
        float sq = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const long long v = fx::value(t[c]);
            const long long d = __shfl_sync(0xffffffffu, dv, p0 + c);
            const int st = __shfl_sync(0xffffffffu, state, p0 + c);
            if (!fail && (st == 1 || (st == 0 && d <= 0))) fail = k0 + c + 1;
            fx::Rsqrt y = fx::rsqrt_fixed(d);  // (of a failed pivot: not used)
            bool ob = false;
            const long long ax = fx::scale_abs(v, y, &ob);
            const Limbs29 al = fx::split29(ax);
            if (c < 3) {  // the next pivot, from its lane's own entry
                Acc29 dn = t[c + 1];
                if (st != 2) fx::fms(dn, al, al);
                dv = fx::value(dn);
            }
            const bool zero = st == 2 || row < k0 + c;  // (or above the diagonal of the tile)
            if (ob && !zero && state == 0) state = 1;
            x[c] = zero ? 0 : v < 0 ? -ax : ax;
            prev[c] = zero ? Limbs29{0, 0} : v < 0 ? Limbs29{-al.hi, -al.lo} : al;
            if (lane == p0 + c) {
                if (st == 2) y.y0 = 0;
                sm.y[k0 + c] = y;
            }
            if (!zero) sq += square_of(ax);
#pragma unroll
            for (int r = c + 1; r < 4; ++r) {
                Limbs29 l;
                l.hi = __shfl_sync(0xffffffffu, prev[c].hi, p0 + r);
                l.lo = __shfl_sync(0xffffffffu, prev[c].lo, p0 + r);
                fx::fms(t[r], prev[c], l);
            }
        }
        if (row >= k0 + 4) {  // below the pivot block: the squares stay within the diagonal entry
            rest -= sq;
            if (state == 0 && rest < -0.01f) state = 1;
            if (state == 1) {
#pragma unroll
                for (int c = 0; c < 4; ++c) x[c] = 0, prev[c] = {0, 0};
            }
        }
        store_limbs4(sm.L + row * kLS + k0, prev);
        if (fail && lane == 0) {
            sm.fail = fail;
            sm.fail_round = b + 1;
        }
        __syncwarp();
        bar_arrive(bar_pivots_solving(b), kPivotsSolving);
        bar_arrive(bar_pivots(b), kPivotsCount);
        if (fail) return;
#pragma unroll
        for (int c = 0; c < 4; ++c) sm.lv[row * kLvS + k0 + c] = x[c];
    }
}

// A solving warp: row g of the tile's rows (row >= 64: below it), a round behind the pivots.
__device__ __forceinline__ void solving_warp(PanelSmem& sm, int g, bool live, float rest, bool* rbad) {
    bar_sync(kBarNext, kWorkers);
    Limbs29* const mine = g < NB ? sm.L + g * kLS : sm.lx + 4 * (min(g, kRows - 1) - NB);
    const int gn = min(g, kRows - 1) - kWin;
#pragma unroll 1
    for (int b = 0; b < 16; ++b) {
        const int k0 = 4 * b;
        bar_sync(bar_pivots_solving(b), kPivotsSolving);
        if (sm.fail_round == b + 1) return;
        if (g >= NB || b < 8) {  // rows 32 to 63 are the pivot warp's from round 8 on
            Acc29 t[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) t[c] = {sm.xn[c][gn], 0};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int k = k0 + c;
                const fx::Rsqrt y = sm.y[k];
                bool ob = false;
                long long x = y.y0 ? fx::scale(fx::value(t[0]), y, &ob) : 0;
                rest -= square_of(x);
                if (ob || rest < -0.01f) *rbad = true;
                if (*rbad) x = 0;
                const Limbs29 xl = fx::split29(x);
                if (live) {
                    (g < NB ? mine + k : mine + c)[0] = xl;
                    sm.lv[g * kLvS + k] = x;
                }
#pragma unroll
                for (int r = 1; r < 4; ++r) {  // (past the round's columns: not used)
                    fx::fms(t[r], xl, sm.L[min(k + r, NB - 1) * kLS + k]);
                    t[r - 1] = t[r];
                }
            }
            if (live && g < NB) {
                sm.rest[g - kWin] = rest;
                if (*rbad) sm.diag_bad[g] = 1;
            }
            if (b == 7 && g < NB) {
                __syncwarp();
                bar_arrive(kBarHandover, 64);
            }
        }
        bar_arrive(kBarSolved, kWorkers);
        if (b < 15) bar_sync(kBarNext, kWorkers);
    }
}

// An updating warp: the thread's row g and columns 4 m + q.
__device__ __forceinline__ void updating_warp(PanelSmem& sm, Acc29 (&a)[16], int g, int q) {
    if (g < kWin) {
        sm.xw[0][q][g] = fx::quarters(a[0]);
        sm.xw[1][q][g] = fx::quarters(a[1]);
    } else {
        sm.xn[q][g - kWin] = fx::quarters(a[0]);
    }
    bar_arrive(bar_window(0), kWindowCount);
    bar_arrive(bar_window(1), kWindowCount);
    bar_arrive(kBarNext, kWorkers);
    const int gw = g & ~7;  // the warp's first row (its rows share a window)
#pragma unroll 1
    for (int b = 0; b < 16; ++b) {
        const int k0 = 4 * b, w0 = (b >> 3) * kWin, w1 = w0 + kWin;  // the window's rows
        const bool window = gw >= w0 && gw < w1, outside = gw >= w1;
        const Limbs29* const col = sm.L + (k0 + q) * kLS + k0;  // limbs of row k0 + q, columns k0 ..
        bar_sync(bar_pivots(b), kPivotsCount);
        if (sm.fail_round == b + 1) return;
        Limbs29 xr[4], l[4];
        // the window's columns two rounds ahead (those of the next round are the pivot warp's)
        if (window) {
            load_limbs4(sm.L + g * kLS + k0, xr);
            if (k0 + 8 < w1) {
                load_limbs4(col + 8 * kLS, l);
#pragma unroll
                for (int c = 0; c < 4; ++c) fx::fms(a[2], xr[c], l[c]);
                sm.xw[b & 1][q][g - w0] = fx::quarters(a[2]);
            }
        }
        if (b <= 13 && b != 6 && b != 7) bar_arrive(bar_window(b + 2), kWindowCount);
        bar_sync(kBarSolved, kWorkers);
        if (b == 15) break;
        // the rows outside the window: the next round's columns first, for the solving warps
        if (outside) {
            load_limbs4(g < NB ? sm.L + g * kLS + k0 : sm.lx + 4 * (g - NB), xr);
#pragma unroll
            for (int m = 1; m < 3; ++m) {
                if (m > 15 - b) break;
                load_limbs4(col + 4 * m * kLS, l);
#pragma unroll
                for (int c = 0; c < 4; ++c) fx::fms(a[m], xr[c], l[c]);
            }
            sm.xn[q][g - kWin] = fx::quarters(a[1]);
            if (g < NB && (b == 6 || b == 7)) sm.xw[b & 1][q][g - kWin] = fx::quarters(a[2]);
        }
        if (b == 6 || b == 7) bar_arrive(bar_window(b + 2), kWindowCount);
        bar_arrive(kBarNext, kWorkers);
        // the columns further right, up to the window's, the row's or the panel's last
        const int end = window ? min(w1, gw + 8) : outside ? min(NB, g < NB ? gw + 8 : NB) : 0;
#pragma unroll
        for (int m = 3; m < 16; ++m) {
            if (k0 + 4 * m >= end) break;
            load_limbs4(col + 4 * m * kLS, l);
#pragma unroll
            for (int c = 0; c < 4; ++c) fx::fms(a[m], xr[c], l[c]);
        }
#pragma unroll
        for (int m = 0; m < 15; ++m) a[m] = a[m + 1];
    }
}

// FP64 columns and FP16 digit tiles of the rows in sm.lv[first, first + count):
// row i of them is matrix row r0 + i.
__device__ void panel_output(const PanelSmem& sm, int first, int count, int r0, double* __restrict__ A, int j0,
                             int lda, const int* __restrict__ e, unsigned char* __restrict__ tiles,
                             long long* __restrict__ rows) {
    if (rows) {
        for (int t = threadIdx.x; t < count * NB; t += kPanelThreads)
            rows[static_cast<long long>(r0) * NB + t] = sm.lv[(first + (t >> 6)) * kLvS + (t & 63)];
    }
    // digits: one thread per row and run of eight columns, a 16-byte store per digit,
    // in the 128-byte-swizzled K-major layout that the update's MMA reads
    for (int t = threadIdx.x; !rows && t < count * 8; t += kPanelThreads) {
        const int i = t % count, kc = t / count;
        const int r = r0 + i, rt = r & 63;
        int q[8][kNS];
#pragma unroll
        for (int k = 0; k < 8; ++k) fx::digits(sm.lv[(first + i) * kLvS + 8 * kc + k], q[k]);
        unsigned char* dst =
            tiles + static_cast<size_t>(r >> 6) * kNS * kTileB + (rt >> 3) * 1024 + (rt & 7) * 128 + ((kc ^ (rt & 7)) << 4);
#pragma unroll
        for (int s = 0; s < kNS; ++s) {
            __half2 h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                h[k] = __halves2half2(__int2half_rn(q[2 * k][s]), __int2half_rn(q[2 * k + 1][s]));
            *reinterpret_cast<uint4*>(dst + s * kTileB) = *reinterpret_cast<uint4*>(h);
        }
    }
    for (int t = threadIdx.x; t < count * NB; t += kPanelThreads) {
        const int i = t % count, k = t / count;
        const int r = r0 + i;
        A[r + static_cast<long long>(j0 + k) * lda] = fx::to_double(sm.lv[(first + i) * kLvS + k], e[r]);
    }
}

// rows: where the panel's rows go as integers, for chol_update_int (null: as digit tiles).
// diag: where the diagonal tile's factor goes, column-major (null, with one CTA per
// chain: to its place).
// j0: first column of the panel; blockIdx.y = 1: of the second chain's, dj further on.
__global__ void __launch_bounds__(kPanelThreads, 1) chol_panel(double* __restrict__ A, int j0, int dj, int lda,
                                                              int nbelow, int rpc, const int* __restrict__ e,
                                                              int* __restrict__ bad,
                                                              unsigned char* __restrict__ tiles,
                                                              long long* __restrict__ rows,
                                                              double* __restrict__ diag, int* __restrict__ info) {
    extern __shared__ __align__(16) unsigned char panel_smem[];
    PanelSmem& sm = *reinterpret_cast<PanelSmem*>(panel_smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    j0 += blockIdx.y * dj;
    pdl_wait();
    pdl_trigger();
    // one read per block: block 0 of this grid may set the flag meanwhile
    if (tid == 0) {
        sm.fail = *info;
        sm.fail_round = 0;
    }
    __syncthreads();
    if (sm.fail) return;
    const long long* F = reinterpret_cast<const long long*>(A);
    const int b0 = blockIdx.x * rpc, b1 = min(nbelow, b0 + rpc);  // this CTA's rows below the tile
    const int nx = max(0, min(kExtra, b1 - b0));                  // of them in the first group
    if (tid < NB) sm.diag_bad[tid] = bad[j0 + tid];
    // what the squares of a row of the factor may add up to, and whether it has failed
    auto matrix_row = [&](int g) { return g < NB ? j0 + g : j0 + NB + b0 + (g - NB); };
    auto diagonal = [&](int g) {
        const int r = matrix_row(g);
        return bad[r] == 2 ? 1.f : static_cast<float>(F[r + static_cast<long long>(r) * lda]) * 0x1p-62f;
    };
    __syncthreads();
    // workers by sub-partition 1, 2, 3 (warp & 3) and slot (warp >> 2): updating
    // warps 0 to 9 hold rows 8 w .., of which 4 to 9 have the most work; 10 and 11 solve
    const int worker = (warp & 3) == 1 ? (warp >> 2 ? 2 + 2 * (warp >> 2) : 0)
                       : (warp & 3) == 2 ? (warp >> 2 ? 3 + 2 * (warp >> 2) : 1)
                                         : (warp >> 2 < 2 ? 2 + (warp >> 2) : 8 + (warp >> 2));
    bool rbad = false;
    int srow = -1;
    if (warp == 0) {
        pivot_warp(sm, diagonal(lane));
    } else if ((warp & 3) == 0) {
        // rests
    } else if (worker < kUpdateWarps) {
        const int g = 8 * worker + (lane >> 2), q = lane & 3;
        const bool live = g < NB || g - NB < nx;
        Acc29 a[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int j = 4 * m + q;
            a[m] = {live && (g >= NB || j <= g) ? F[matrix_row(g) + static_cast<long long>(j0 + j) * lda] : 0, 0};
        }
        updating_warp(sm, a, g, q);
    } else {
        const int g = worker == kUpdateWarps ? kWin + lane : NB + lane;
        const bool live = g < NB || g - NB < nx;
        if (live) {
            srow = g;
            rbad = bad[matrix_row(g)] == 1;
        }
        solving_warp(sm, g, live, live ? diagonal(g) : 0.f, &rbad);
    }
    __syncthreads();
    if (sm.fail) {
        if (blockIdx.x == 0 && tid == 0) atomicCAS(info, 0, j0 + sm.fail);  // (another chain's block may find one too)
        return;
    }
    if (srow >= NB && rbad) bad[matrix_row(srow)] = 1;
    if (nx > 0) panel_output(sm, NB, nx, j0 + NB + b0, A, j0, lda, e, tiles, rows);
    if (blockIdx.x == 0) {  // the diagonal tile's factor
        for (int t = tid; t < NB * NB; t += kPanelThreads) {
            const int i = t & 63, k = t >> 6;
            if (i < k) continue;
            double v = fx::to_double(sm.lv[i * kLvS + k], e[j0 + i]);
            if (i == k && sm.diag_bad[i] == 2) v = __longlong_as_double(0x7ff0000000000000ll);
            if (diag)
                diag[blockIdx.y * NB * NB + t] = v;
            else
                A[(j0 + i) + static_cast<long long>(j0 + k) * lda] = v;
        }
    }
    // further rows, kRows2 at a time: the factor is known, four threads of a
    // warp solve a row with shuffles
    for (int c0 = b0 + kExtra; c0 < b1; c0 += kRows2) {
        const int g = tid >> 2, q = tid & 3;
        const int n = min(kRows2, b1 - c0);
        const int r = j0 + NB + c0 + g;
        const bool lv = g < n;
        bool rb = lv ? bad[r] == 1 : true;
        float rs = lv ? static_cast<float>(F[r + static_cast<long long>(r) * lda]) * 0x1p-62f : 0.f;
        if (lv && bad[r] == 2) rs = 1.f;
        Acc29 a[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) a[m] = {lv ? F[r + static_cast<long long>(j0 + 4 * m + q) * lda] : 0, 0};
        __syncthreads();  // sm.lv of the previous rows has been written out
        if (8 * warp < n) {
            for (int b = 0; b < 16; ++b) {
                const int k0 = 4 * b;
                Limbs29 xl[4], l[4];
                load_limbs4(sm.L + (k0 + q) * kLS + k0, l);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    bool ob = false;
                    long long x = 0;
                    const fx::Rsqrt y = sm.y[k0 + c];
                    if (q == c) {
                        x = fx::scale(fx::value(a[0]), y, &ob);
                        if (ob || rb || y.y0 == 0) x = 0;
                    }
                    const Limbs29 mine = fx::split29(x);
                    xl[c].hi = __shfl_sync(0xffffffffu, mine.hi, c, 4);
                    xl[c].lo = __shfl_sync(0xffffffffu, mine.lo, c, 4);
                    rb = __shfl_sync(0xffffffffu, ob ? 1 : 0, c, 4) || rb;
                    const float xf = static_cast<float>(xl[c].hi) * 0x1p-31f;
                    rs = fmaf(-xf, xf, rs);
                    if (rs < -0.01f) rb = true;
                    if (q == c) sm.lv[g * kLvS + k0 + c] = x;
                    if (c < 3) fx::fms(a[0], xl[c], l[c]);  // columns left of q: not used again
                }
#pragma unroll
                for (int m = 1; m < 16; ++m) {
                    if (m > 15 - b) break;
                    load_limbs4(sm.L + (4 * (b + m) + q) * kLS + k0, l);
#pragma unroll
                    for (int c = 0; c < 4; ++c) fx::fms(a[m], xl[c], l[c]);
                }
#pragma unroll
                for (int m = 0; m < 15; ++m) a[m] = a[m + 1];
            }
            if (lv && rb && q == 0) bad[r] = 1;
        }
        __syncthreads();
        panel_output(sm, 0, n, j0 + NB + c0, A, j0, lda, e, tiles, rows);
    }
}

// The panel's diagonal tile from the workspace to its place at row and column j0, by
// threads t of nthreads.
__device__ __forceinline__ void place_diagonal(double* __restrict__ A, int j0, int lda, const double* __restrict__ diag,
                                               int t, int nthreads) {
    for (; t < NB * NB; t += nthreads) {
        const int i = t & 63, k = t >> 6;
        if (i >= k) A[(j0 + i) + static_cast<long long>(j0 + k) * lda] = diag[t];
    }
}

// ---------------------------------------------------------------- trailing update
//
// C(I, J) -= L(I) L(J)^T for the lower tiles: 128 rows (two 64-row tiles) by 64
// columns, K = 64 (the panel). With L = sum_s q_s 2^(52 - 9 s), the products of
// digits s and t weigh 2^(46 - 9 (s + t)) of C's units of 2^-62: group d = s + t is
// summed in one FP32 accumulator of 64 TMEM columns (8 groups: all 512 columns); 34
// digit products of 4 MMAs (K = 16). The sums of groups 0 to 4 stay below 2^24 and
// are exact; a rounding in group 5, whose bound is 2^24.4, would weigh two units, in
// groups 6 and 7 less than one. The products left out (d > 7) weigh a hundredth of a
// unit. With entries in units of 2^-60 and d = 7 left out, a third of such a unit, the
// update was less precise than FP64 arithmetic from some 2,000 rows on: error of the
// solution at 4,096 rows 3.0e-15, FP64 1.45e-15, so 6.4e-16 (and 23.5 ms for a trial
// of 1,000 cameras, 22.7 without).
//
// One CTA per SM walks a contiguous run of tiles (row block by row block, so the
// row block's digits are loaded once): warp 0 loads digit tiles (bulk copies,
// columns double-buffered), warp 1 issues the MMAs, sixteen warps recombine. The
// low groups (4 to 7) come first: the recombination of one part overlaps
// the MMAs of the other. What bounds it: 34 x 4 MMAs of 128 x 64 x 16 a tile, which
// read their operands from shared memory at 6 KB per MMA, and the 16 bytes of
// each entry per panel from and to HBM.
constexpr int kGroups = 8;
constexpr int kUpdWarps = 16;  // recombining warps: 32 rows x 16 columns each
constexpr int kUpdThreads = 64 + 32 * kUpdWarps;
constexpr int kABytes = kNS * 2 * kTileB, kBBytes = kNS * kTileB;
constexpr int kUpdSmem = kABytes + 2 * kBBytes + 1024;
constexpr int kWaitLimit = 1 << 18;  // polls of a barrier before a role gives up (then info = INT_MIN)

enum { B_FULLA = 0, B_EMPTYA, B_FULLB, B_EMPTYB = 4, B_LOFULL = 6, B_LOEMPTY, B_HIFULL, B_HIEMPTY, B_COUNT };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for the phase of the given parity; false when it gave up (or another role has).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* gave_up) {
    for (int i = 0; i < kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 1023) == 1023 && *gave_up) return false;
    }
    *gave_up = 1;
    return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// K-major operand, rows of 128 bytes in 8-row groups of 1024 bytes, 128-byte swizzle.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr & 0x3ffff) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_load8(uint32_t addr, float (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_load() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// An integer-valued FP32 accumulator as an integer: by the add of 1.5 2^23 for
// |v| < 2^22 (groups 0 and 1), else by conversion.
__device__ __forceinline__ int small_int(float v) { return __float_as_int(v + 12582912.f) - 0x4b400000; }

// Tile t of the trailing matrix of nt 64-row tiles: row block I (tiles 2 I, 2 I + 1), column tile J.
__device__ __forceinline__ void tile_of(long long t, int* I, int* J) {
    int i = static_cast<int>((sqrtf(4.f * static_cast<float>(t) + 1.f) - 1.f) * 0.5f);
    while (static_cast<long long>(i) * (i + 1) > t) --i;
    while (static_cast<long long>(i + 1) * (i + 2) <= t) ++i;
    *I = i;
    *J = static_cast<int>(t - static_cast<long long>(i) * (i + 1));
}

__global__ void __launch_bounds__(kUpdThreads, 1) chol_update(double* __restrict__ A, int j1, int dj, int nt,
                                                             long long ntiles, int lda, const unsigned char* __restrict__ tiles,
                                                             const double* __restrict__ diag, int* __restrict__ info) {
    extern __shared__ unsigned char upd_raw[];
    __shared__ __align__(8) unsigned long long bars[B_COUNT];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int gave_up;
    __shared__ int info_s;
    const uint32_t base = (smem_u32(upd_raw) + 1023u) & ~1023u;
    const uint32_t sA = base, sB = base + kABytes;
    j1 += blockIdx.y * dj;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8u * i; };
    if (tid == 0) {
        for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i == B_LOEMPTY || i == B_HIEMPTY ? kUpdWarps : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        gave_up = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_trigger();
    if (tid == 0) info_s = *info;  // one read per block
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    const int failed = info_s;
    const long long t0 = ntiles * blockIdx.x / gridDim.x, t1 = failed ? t0 : ntiles * (blockIdx.x + 1) / gridDim.x;
    const int tile0 = j1 / NB;  // first tile of the trailing matrix

    if (warp == 0 && lane == 0) {
        int lastI = -1, na = 0;
        for (long long t = t0; t < t1; ++t) {
            int I, J;
            tile_of(t, &I, &J);
            if (I != lastI) {
                if (na > 0 && !mbar_wait(bar(B_EMPTYA), (na - 1) & 1, &gave_up)) break;
                const bool two = 2 * I + 1 < nt;
                mbar_expect(bar(B_FULLA), two ? kABytes : kABytes / 2);
                const unsigned char* src = tiles + static_cast<size_t>(tile0 + 2 * I) * kNS * kTileB;
                for (int s = 0; s < kNS; ++s) {
                    bulk_load(sA + s * 2 * kTileB, src + s * kTileB, kTileB, bar(B_FULLA));
                    if (two)
                        bulk_load(sA + s * 2 * kTileB + kTileB, src + (kNS + s) * kTileB, kTileB, bar(B_FULLA));
                }
                lastI = I;
                ++na;
            }
            const int i = static_cast<int>(t - t0), st = i & 1;
            if (i >= 2 && !mbar_wait(bar(B_EMPTYB + st), ((i >> 1) - 1) & 1, &gave_up)) break;
            mbar_expect(bar(B_FULLB + st), kBBytes);
            bulk_load(sB + st * kBBytes, tiles + static_cast<size_t>(tile0 + J) * kNS * kTileB, kBBytes,
                      bar(B_FULLB + st));
        }
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = (1u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);  // FP16 x FP16 -> FP32, M 128, N 64
        int lastI = -1, na = 0;
        for (long long t = t0; t < t1; ++t) {
            int I, J;
            tile_of(t, &I, &J);
            const int i = static_cast<int>(t - t0), st = i & 1;
            if (I != lastI) {
                if (!mbar_wait(bar(B_FULLA), na & 1, &gave_up)) break;
                lastI = I;
                ++na;
            }
            if (!mbar_wait(bar(B_FULLB + st), (i >> 1) & 1, &gave_up)) break;
            const uint32_t b = sB + st * kBBytes;
            auto group = [&](int d) {
                bool acc = false;
                for (int s = max(0, d - kNS + 1); s <= min(d, kNS - 1); ++s) {
                    const uint64_t da = operand_desc(sA + s * 2 * kTileB), db = operand_desc(b + (d - s) * kTileB);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {  // K = 16: 32 bytes along the swizzled row
                        mma_f16(tmem + 64 * d, da + 2 * k, db + 2 * k, idesc, acc);
                        acc = true;
                    }
                }
            };
            if (i > 0 && !mbar_wait(bar(B_LOEMPTY), (i - 1) & 1, &gave_up)) break;
            tc_fence_after();
            for (int d = 4; d < kGroups; ++d) group(d);
            mma_commit(bar(B_LOFULL));
            if (i > 0 && !mbar_wait(bar(B_HIEMPTY), (i - 1) & 1, &gave_up)) break;
            tc_fence_after();
            for (int d = 0; d < 4; ++d) group(d);
            mma_commit(bar(B_HIFULL));
            mma_commit(bar(B_EMPTYB + st));
            int I2 = -1, J2;
            if (t + 1 < t1) tile_of(t + 1, &I2, &J2);
            if (I2 != I) mma_commit(bar(B_EMPTYA));
        }
    } else if (warp >= 2) {
        const int quarter = warp & 3, part = (warp - 2) >> 2;  // TMEM lanes 32 quarter .., columns 16 part ..
        const uint32_t tm = tmem + (static_cast<uint32_t>(32 * quarter) << 16) + 16 * part;
        long long* F = reinterpret_cast<long long*>(A);
        if (blockIdx.x == 0 && !failed)  // (these warps wait for the first products)
            place_diagonal(A, j1 - NB, lda, diag + blockIdx.y * NB * NB, tid - 64, 32 * kUpdWarps);
        for (long long t = t0; t < t1; ++t) {
            int I, J;
            tile_of(t, &I, &J);
            const int i = static_cast<int>(t - t0);
            const int rloc = 128 * I + 32 * quarter + lane, cloc = 64 * J + 16 * part;  // within the trailing matrix
            const bool in = rloc < 64 * nt;
            long long* p = F + (j1 + rloc) + static_cast<long long>(j1 + cloc) * lda;
            long long c[16];
            if (!mbar_wait(bar(B_LOFULL), i & 1, &gave_up)) break;
            tc_fence_after();
#pragma unroll
            for (int k0 = 0; k0 < 16; k0 += 8) {
                float g4[8], g5[8], g6[8], g7[8];
                tmem_load8(tm + 4 * 64 + k0, g4);
                tmem_load8(tm + 5 * 64 + k0, g5);
                tmem_load8(tm + 6 * 64 + k0, g6);
                tmem_load8(tm + 7 * 64 + k0, g7);
                tmem_wait_load();
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    c[k0 + k] = static_cast<long long>(__float2int_rn(g4[k])) * 1024 +
                                (2 * __float2int_rn(g5[k]) + __float2int_rn(0x1p-8f * fmaf(g7[k], 0x1p-9f, g6[k])));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_LOEMPTY));
            if (!mbar_wait(bar(B_HIFULL), i & 1, &gave_up)) break;
            tc_fence_after();
#pragma unroll
            for (int k0 = 0; k0 < 16; k0 += 8) {
                float g0[8], g1[8], g2[8], g3[8];
                tmem_load8(tm + k0, g0);
                tmem_load8(tm + 64 + k0, g1);
                tmem_load8(tm + 128 + k0, g2);
                tmem_load8(tm + 192 + k0, g3);
                tmem_wait_load();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int top = small_int(g0[k]) * 512 + small_int(g1[k]);  // 2^37
                    c[k0 + k] += (static_cast<long long>(top) << 37) +
                                 static_cast<long long>(__float2int_rn(g2[k])) * (1 << 28) +
                                 static_cast<long long>(__float2int_rn(g3[k])) * (1 << 19);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_HIEMPTY));
            // subtracted at L2: the entries are not waited for
#pragma unroll
            for (int k = 0; k < 16; ++k)
                if (in && rloc >= cloc + k)
                    atomicAdd(reinterpret_cast<unsigned long long*>(p + static_cast<long long>(k) * lda),
                              static_cast<unsigned long long>(-c[k]));
        }
    }
    __syncwarp();
    if (gave_up)
        for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies and MMAs in flight land before the block ends
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    if (tid == 0 && gave_up) *info = INT_MIN;
}

// The update of a few tiles with integer multiply-adds, 16 x 16 entries per block, one
// per thread: a tile of chol_update occupies one SM for the 136 MMAs of its 34 digit
// products (77 cycles each) and its operands' way to shared memory, 11.7 us with the
// launch, however few tiles there are; here they spread over all SMs. 576 rows
// (9 panels) 380 -> 338 us. One more block places the panel's diagonal tile.
constexpr int kIntB = 16;
__global__ void __launch_bounds__(kIntB * kIntB) chol_update_int(double* __restrict__ A, int j1, int dj, int lda,
                                                                const long long* __restrict__ rows,
                                                                const double* __restrict__ diag,
                                                                const int* __restrict__ info) {
    __shared__ __align__(16) Limbs29 L[2][kIntB][NB + 2];
    j1 += blockIdx.y * dj;
    if (blockIdx.x == gridDim.x - 1) {
        pdl_wait();
        pdl_trigger();
        if (!*info) place_diagonal(A, j1 - NB, lda, diag + blockIdx.y * NB * NB, threadIdx.x, kIntB * kIntB);
        return;
    }
    int rb = static_cast<int>((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
    while (rb * (rb + 1) / 2 > static_cast<int>(blockIdx.x)) --rb;
    while ((rb + 1) * (rb + 2) / 2 <= static_cast<int>(blockIdx.x)) ++rb;
    const int cb = blockIdx.x - rb * (rb + 1) / 2;
    const int i = threadIdx.x & (kIntB - 1), j = threadIdx.x / kIntB;  // row, column of the block
    const int row = j1 + kIntB * rb + i, col = j1 + kIntB * cb + j;
    pdl_wait();
    pdl_trigger();
    if (*info) return;
    long long* p = reinterpret_cast<long long*>(A) + row + static_cast<long long>(col) * lda;
    Acc29 acc = {row >= col ? *p : 0, 0};
#pragma unroll
    for (int t = threadIdx.x; t < 2 * kIntB * NB; t += kIntB * kIntB) {
        const int h = t / (kIntB * NB), r = (t / NB) % kIntB, k = t % NB;
        L[h][r][k] = fx::split29(rows[static_cast<long long>(j1 + kIntB * (h ? cb : rb) + r) * NB + k]);
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < NB; k += 4) {
        Limbs29 a[4], b[4];
        load_limbs4(&L[0][i][k], a);
        load_limbs4(&L[1][j][k], b);
#pragma unroll
        for (int q = 0; q < 4; ++q) fx::fms_full(acc, a[q], b[q]);
    }
    if (row >= col) *p = fx::quarters(acc);
}
// Most tiles below the diagonal tile that it serves: of a step (panel and update) of
// 42 us, 5 us less at up to 8 tiles, 3 at 12, none at 16, 10 more at 24.
constexpr int kIntTiles = 12;

}  // namespace

size_t dense_potrf_workspace(int n) {
    return static_cast<size_t>(n / NB) * kNS * kTileB + 2 * sizeof(int) * static_cast<size_t>(n) +
           kMaxChains * NB * NB * sizeof(double);
}

// One panel and its update for `chains` (1 or 2) chains, dj rows apart: `below` tiles below the diagonal tile of each.
static void factor_panel(double* A, int j0, int dj, int chains, int below, int lda, const Work& w, int* info,
                         cudaStream_t s) {
    const int rows = below * NB, sms = device_sm_count();
    // rows per CTA: kExtra are solved along with the diagonal tile; more only
    // where the panel has more than that for every SM
    const int rpc = kExtra * std::max(1, ceil_div(rows * chains, kExtra * sms));
    const bool ints = below <= kIntTiles;
    launch_pdl(chol_panel, dim3(std::max(1, ceil_div(rows, rpc)), chains), kPanelThreads, sizeof(PanelSmem), s, A, j0,
               dj, lda, rows, rpc, w.e, w.bad, w.tiles, ints ? w.rows : nullptr, below ? w.diag : nullptr, info);
    if (below == 0) return;
    if (ints) {
        const int blocks = rows / kIntB;
        launch_pdl(chol_update_int, dim3(blocks * (blocks + 1) / 2 + 1, chains), kIntB * kIntB, 0, s, A, j0 + NB, dj,
                   lda, w.rows, w.diag, info);
        return;
    }
    const long long pairs = below / 2;
    const long long tiles = pairs * (pairs + 1) + (below % 2 ? below : 0);
    launch_pdl(chol_update, dim3(static_cast<unsigned>(std::min<long long>(tiles, std::max(1, sms / chains))), chains),
               kUpdThreads, kUpdSmem, s, A, j0 + NB, dj, below, tiles, lda, w.tiles, w.diag, info);
}
static void allow_smem() {
    GBA_CUDA_CHECK(cudaFuncSetAttribute(chol_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(PanelSmem)));
    GBA_CUDA_CHECK(cudaFuncSetAttribute(chol_update, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpdSmem));
}

// bt: tiles below the diagonal tile that hold nonzeros (n / 64 - 1 for a
// dense matrix; lda = ldb - 1 with ldb >= (bt + 2) 64 for a band).
void dense_potrf(double* A, int n, int lda, int bt, int* info, void* workspace, cudaStream_t s) {
    if (n % NB != 0 || bt < 0 || (bt < n / NB - 1 ? lda + 1 < (bt + 2) * NB : lda < n))
        throw std::invalid_argument("dense_potrf: n must be a multiple of 64 and lda hold the band");
    allow_smem();
    const Work w = carve(workspace, n);
    const int nt = n / NB;
    launch_pdl(chol_scale, ceil_div(n, 256), 256, 0, s, A, n, lda, w.e, w.bad, info);
    launch_pdl(chol_convert, dim3(nt, std::min(bt, nt - 1) + 1), 256, 0, s, A, nt, lda, bt, w.e, w.bad);
    for (int jb = 0; jb < nt; ++jb) factor_panel(A, jb * NB, 0, 1, std::min(nt - jb - 1, bt), lda, w, info, s);
}

// ---------------------------------------------------------------- band, from both ends
//
// A band's panels are a chain of its own length: each is as long as its 64
// pivots take, and uses a few SMs. So the band is eliminated from both ends at once:
// rows [0, a) downwards and rows [a + s, n) upwards, s = 64 bt rows between them, which
// no row of one part shares with the other; then the s rows that are left. In
// storage: chain 0 is rows [0, a + s) of the band; chain 1, from row a + s on, is the
// trailing part [a, n) with its order reversed, so a band of the same width whose
// last s rows are the rows between once more. Those start with their diagonal
// entries alone in chain 1 (its rows' scale and the bound of a row's squares need
// them) and are added to chain 0's when both chains have reached them, without the
// diagonal counted twice. 5,504 rows, 3 tiles below the diagonal tile: 45 panels in
// turn instead of 86, a damped solve with its assembly 5.6 -> 3.4 ms.

struct Twist {
    int n, a, s, base, np;  // base: chain 1's first row; np: rows of both chains
    explicit Twist(int n_, int bt, int ta) : n(n_), a(ta * NB), s(bt * NB), base(a + s), np(n_ + s) {}
    __host__ __device__ int source(int i) const { return i < base ? i : n - 1 - (i - base); }  // row of the band
    __host__ __device__ int mirror(int i) const { return base + n - 1 - i; }                   // row i >= a in chain 1
    __host__ __device__ bool copy(int i) const { return i >= np - s; }                         // chain 1's rows between
};

__global__ void twist_scale(const double* __restrict__ S, Twist t, int lda, int* __restrict__ e, int* __restrict__ bad,
                            int* __restrict__ info) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *info = 0;
    if (i >= t.np) return;
    const int r = t.source(i);
    const double d = S[r + static_cast<long long>(r) * lda];
    const bool ok = fx::finite_positive(d);
    e[i] = ok ? fx::row_exponent(d) : 0;
    bad[i] = ok ? 0 : d > 0.0 ? 2 : 1;
}

// chol_convert of the band S to the two chains in F; one CTA per tile of a chain.
// Chain 1's tiles are transposed and reversed: through shared memory.
__global__ void __launch_bounds__(256) twist_convert(const double* __restrict__ S, Twist t, int lda,
                                                    const int* __restrict__ e, int* __restrict__ bad,
                                                    long long* __restrict__ F, long long* __restrict__ dsep) {
    __shared__ double tile[NB][NB + 1];  // [column][row]
    const int tj = blockIdx.x, ti = tj + blockIdx.y;
    if (ti * NB >= (tj * NB < t.base ? t.base : t.np)) return;
    const bool second = tj * NB >= t.base, sep = second && t.copy(tj * NB);
    const int lane_row = threadIdx.x & 63;
    pdl_wait();
    pdl_trigger();
#pragma unroll 4
    for (int k = threadIdx.x >> 6; k < NB; k += 4) {  // k: column of S, lane_row: row
        if (!second) {
            const int i = ti * NB + lane_row, j = tj * NB + k;
            tile[k][lane_row] = j <= i ? S[i + static_cast<long long>(j) * lda] : 0.0;
        } else {
            const int j = tj * NB + lane_row, i = ti * NB + k, r = t.source(j), c = t.source(i);  // S(r, c) = S(c, r)
            tile[lane_row][k] = j <= i && (!sep || j == i) ? S[r + static_cast<long long>(c) * lda] : 0.0;
        }
    }
    __syncthreads();
    const int i = ti * NB + lane_row, ei = e[i];
    const bool inf_row = bad[i] == 2;
    bool mine = false;
    for (int k = threadIdx.x >> 6; k < NB; k += 4) {
        const int j = tj * NB + k;
        if (j > i) continue;
        bool b = false;
        const long long f = convert_entry(tile[k][lane_row], ei, e[j], inf_row, bad[j] == 2, i == j, &b);
        F[i + static_cast<long long>(j) * lda] = f;
        if (sep && i == j) dsep[i - (t.np - t.s)] = f;
        mine = mine || b;
    }
    if (mine) bad[i] = 1;
}

// Chain 1's rows between, added to chain 0's.
__global__ void twist_merge(long long* __restrict__ F, Twist t, int lda, int* __restrict__ bad,
                            const long long* __restrict__ dsep) {
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (r >= t.s || c > r) return;
    const int i = t.a + r, j = t.a + c, mi = t.mirror(i), mj = t.mirror(j);
    const long long v = F[mj + static_cast<long long>(mi) * lda];
    F[i + static_cast<long long>(j) * lda] += i == j ? v - dsep[mi - (t.np - t.s)] : v;
    if (i == j && bad[mi] == 1) bad[i] = 1;
}

static Work carve_twist(void* ws, const Twist& t, long long** dsep) {
    *dsep = static_cast<long long*>(ws);
    return carve(*dsep + t.s, t.np);
}
size_t band_twist_workspace(int n, int bt) {
    return sizeof(long long) * NB * static_cast<size_t>(bt) + dense_potrf_workspace(n + NB * bt);
}

void band_potrf_twisted(const double* S, int n, int lda, int bt, int ta, double* F, int* info, void* workspace,
                        cudaStream_t s) {
    if (n % NB != 0 || bt < 1 || lda + 1 < (bt + 2) * NB || ta < 1 || ta + bt >= n / NB)
        throw std::invalid_argument("band_potrf_twisted: no rows for the two chains");
    allow_smem();
    const Twist t(n, bt, ta);
    long long* dsep = nullptr;
    const Work w = carve_twist(workspace, t, &dsep);
    const int tb = n / NB - ta - bt;
    long long* Fi = reinterpret_cast<long long*>(F);
    launch_pdl(twist_scale, ceil_div(t.np, 256), 256, 0, s, S, t, lda, w.e, w.bad, info);
    launch_pdl(twist_convert, dim3(t.np / NB, bt + 1), 256, 0, s, S, t, lda, w.e, w.bad, Fi, dsep);
    for (int k = 0; k < std::max(ta, tb); ++k) {
        if (k < ta && k < tb)
            factor_panel(F, k * NB, t.base, 2, bt, lda, w, info, s);
        else
            factor_panel(F, k * NB + (k < ta ? 0 : t.base), 0, 1, bt, lda, w, info, s);
    }
    launch_pdl(twist_merge, dim3(ceil_div(t.s, 64), t.s), 64, 0, s, Fi, t, lda, w.bad, dsep);
    for (int k = 0; k < bt; ++k) factor_panel(F, t.a + k * NB, 0, 1, bt - 1 - k, lda, w, info, s);
}

}  // namespace gba
