// Plain form: on-device assembly of the reduced camera system, the triangular
// solves with its Cholesky factor (chol.cu) and the FP64 factorisation of
// the explicitly dense layout.
//
// Reference: the host assembly src/lm.cu:488-594 (T_e = W_e V'^-1, privatised
// S -= T_e W_f^T over edge pairs of each point, merge, rhs, damped U blocks) and
// the host Eigen LLT src/lm.cu:598-604. Here:
//   * T_e is computed per slot on the device;
//   * S is assembled output-stationary: the edge pairs (e, f) of every point
//     with cam(e) >= cam(f) are sorted once by camera-pair block, and each
//     9x9 block is written once as the ordered sum of its pairs (no atomics,
//     deterministic), then the damped U blocks are added;
//   * the FP64 factorisation is right-looking blocked Cholesky (panel width 64):
//     diagonal-block potrf in shared memory, panel triangular solve, and the
//     trailing update C -= A B^T with mma.sync.m8n8k4 FP64 (DMMA).
// S is column-major, n_pad x n_pad (n_pad = 9C rounded up to 64, identity on
// the padding), lower triangle meaningful; the upper triangle is never read.
//
// Band layout (for camera graphs of local covisibility, where S is mostly
// zero): cameras are renumbered by reverse Cuthill-McKee so the nonzero blocks
// gather near the diagonal, and S keeps per column only the ldb rows from the
// diagonal down: element (i, j), 0 <= i - j < ldb, at S[i + j (ldb - 1)]. Every
// kernel below addresses S as A[i + j lda], so the same kernels run on the band
// with lda = ldb - 1; the panel loops stop bt tiles below the diagonal tile
// (Cholesky creates no fill outside the band). Writes to the strict upper
// triangle of a diagonal tile (i - j in [-63, -1]) land in rows ldb - 63 ..
// ldb - 1 of the previous column, which ldb = (bt + 2) 64 keeps outside the band.

#include "common.cuh"
#include "solver.hpp"

namespace gba {
namespace {

constexpr int NB = 64;       // panel width / tile size
constexpr int kSP = NB + 8;  // shared-memory stride (doubles) of K-major tiles: conflict-free DMMA fragments

// T_e = W_e V'^-1 (9 x 3, row by row) and T_e bp_p at the observation's
// camera-major position (tb, 9 values), for the right-hand side. One thread per
// row: 24 contiguous bytes in and out.
constexpr int kTT = 288;
__global__ void __launch_bounds__(kTT) compute_T_kernel(const double* __restrict__ W, const double* __restrict__ Vinv,
                                                       const double* __restrict__ bp, const int* __restrict__ s_pt,
                                                       const int* __restrict__ cam_pos, int E, double* __restrict__ T,
                                                       double* __restrict__ tb) {
    const long long t = blockIdx.x * static_cast<long long>(kTT) + threadIdx.x;
    if (t >= 9ll * E) return;
    const long long s = t / 9;
    const int i = static_cast<int>(t - 9 * s);
    const long long p = s_pt[s];
    const double* Vi = Vinv + 6 * p;
    const double* b = bp + 3 * p;
    const double w0 = W[3 * t], w1 = W[3 * t + 1], w2 = W[3 * t + 2];
    const double t0 = w0 * Vi[0] + w1 * Vi[1] + w2 * Vi[3];
    const double t1 = w0 * Vi[1] + w1 * Vi[2] + w2 * Vi[4];
    const double t2 = w0 * Vi[3] + w1 * Vi[4] + w2 * Vi[5];
    T[3 * t] = t0;
    T[3 * t + 1] = t1;
    T[3 * t + 2] = t2;
    tb[9ll * cam_pos[s] + i] = t0 * b[0] + t1 * b[1] + t2 * b[2];
}

// acc_j += T_e(i,:) . W_f(j,:) for row i of the pair (e, f).
__device__ __forceinline__ void add_pair(const double* __restrict__ T, const double* __restrict__ W, int e, int f, int i,
                                         double (&acc)[9]) {
    const double* Te = T + 27ll * e + 3 * i;
    const double t0 = Te[0], t1 = Te[1], t2 = Te[2];
    const double* Wf = W + 27ll * f;
#pragma unroll
    for (int j = 0; j < 9; ++j) acc[j] = fma(t0, Wf[3 * j], fma(t1, Wf[3 * j + 1], fma(t2, Wf[3 * j + 2], acc[j])));
}

// S(9ce + i, 9cf + j) = -v, or its transpose where the renumbering put the block above the diagonal.
__device__ __forceinline__ void store_block(double* __restrict__ S, int lda, const int* __restrict__ perm, int ce, int cf,
                                            int i, int j, double v) {
    const long long pe = perm ? perm[ce] : ce, pf = perm ? perm[cf] : cf;
    if (pe >= pf)
        S[9 * pe + i + (9 * pf + j) * lda] = -v;
    else
        S[9 * pf + j + (9 * pe + i) * lda] = -v;
}

// Assembly of the blocks of at most kShortPairs pairs: one thread per (block, row i),
// S(9ce+i, 9cf+j) = -sum_{(e,f) in block} T_e(i,:) . W_f(j,:). What bounds it: the
// FP64 pipe (243 FMA per pair, as nested FMAs: the plain sum costs a product and an
// add more per entry, 2.0 against 1.5 ms at 1000 cameras) and blocks of unlike
// length in a warp.
__global__ void __launch_bounds__(288) assemble_kernel(const int* __restrict__ block_off,
                                                      const int* __restrict__ block_ce,
                                                      const int* __restrict__ block_cf, const int* __restrict__ pe,
                                                      const int* __restrict__ pf, const double* __restrict__ T,
                                                      const double* __restrict__ W, int nblocks, int lda,
                                                      const int* __restrict__ perm, double* __restrict__ S) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long b = t / 9;
    const int i = static_cast<int>(t % 9);
    if (b >= nblocks) return;
    const int q0 = block_off[b], q1 = block_off[b + 1];
    if (q1 - q0 > Solver::kShortPairs) return;
    double acc[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) acc[j] = 0.0;
    for (int q = q0; q < q1; ++q) add_pair(T, W, pe[q], pf[q], i, acc);
#pragma unroll
    for (int j = 0; j < 9; ++j) store_block(S, lda, perm, block_ce[b], block_cf[b], i, j, acc[j]);
}

// The longer blocks (a camera's own block holds all its observations; with few
// cameras, every block holds thousands of pairs), in chunks of kChunkPairs: one CTA
// per chunk, thread (slice, row i) takes every kSlices-th pair, the slices added in
// order; a thread per block and row ran one pair after the other (13.7 ms for 136
// blocks of 84,000 observations; 0.12 ms by chunks).
constexpr int kSlices = 32;
__global__ void __launch_bounds__(9 * kSlices) assemble_chunks_kernel(const int4* __restrict__ chunks,
                                                                     const int* __restrict__ pe,
                                                                     const int* __restrict__ pf,
                                                                     const double* __restrict__ T,
                                                                     const double* __restrict__ W,
                                                                     double* __restrict__ part) {
    __shared__ double sh[kSlices][81];
    const int4 c = chunks[blockIdx.x];  // block, first pair, end pair
    const int slice = threadIdx.x / 9, i = threadIdx.x - 9 * slice;
    double acc[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) acc[j] = 0.0;
    for (int q = c.y + slice; q < c.z; q += kSlices) add_pair(T, W, pe[q], pf[q], i, acc);
#pragma unroll
    for (int j = 0; j < 9; ++j) sh[slice][9 * i + j] = acc[j];
    __syncthreads();
    // 81 sums of kSlices values, three threads each (a third of the slices in order)
    __shared__ double third[3][81];
    if (threadIdx.x < 243) {
        const int k = threadIdx.x % 81, g = threadIdx.x / 81;
        double v = 0.0;
        for (int sl = 11 * g; sl < min(kSlices, 11 * g + 11); ++sl) v += sh[sl][k];
        third[g][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 81)
        part[81ll * blockIdx.x + threadIdx.x] = (third[0][threadIdx.x] + third[1][threadIdx.x]) + third[2][threadIdx.x];
}

// S blocks from their chunks' sums, in order: long block l has chunks [off[l], off[l + 1]).
__global__ void __launch_bounds__(96) assemble_finalize_kernel(const int* __restrict__ off,
                                                              const int4* __restrict__ chunks,
                                                              const int* __restrict__ block_ce,
                                                              const int* __restrict__ block_cf,
                                                              const double* __restrict__ part, int lda,
                                                              const int* __restrict__ perm, double* __restrict__ S) {
    if (threadIdx.x >= 81) return;
    const int c0 = off[blockIdx.x], c1 = off[blockIdx.x + 1], b = chunks[c0].x;
    double v = 0.0;
    for (int c = c0; c < c1; ++c) v += part[81ll * c + threadIdx.x];
    store_block(S, lda, perm, block_ce[b], block_cf[b], threadIdx.x / 9, threadIdx.x % 9, v);
}

// Diagonal blocks += U_c + lambda * max(diag U_c, 1e-12); identity on padding.
__global__ void add_damped_u_kernel(const double* __restrict__ U, double lambda, int C, int n_pad, int lda,
                                    const int* __restrict__ perm, double* __restrict__ S) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 81 * C) {
        const int c = t / 81, i = (t % 81) / 9, j = t % 9;
        double v = U[t];
        if (i == j) v += lambda * (v > 0.0 ? v : 1e-12);
        const long long pc = perm ? perm[c] : c;
        S[(9 * pc + i) + (9 * pc + j) * lda] += v;
    } else if (t < 81 * C + (n_pad - 9 * C)) {
        const long long r = 9ll * C + (t - 81 * C);
        S[r + r * lda] = 1.0;
    }
}

// Copies the assembled diagonal blocks S_cc (lower triangle mirrored) to Sdiag.
__global__ void extract_diag_blocks(const double* __restrict__ S, int C, int lda, const int* __restrict__ perm,
                                    double* __restrict__ Sdiag) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 81 * C) return;
    const int c = t / 81, i = (t % 81) / 9, j = t % 9;
    const int r = i >= j ? i : j, q = i >= j ? j : i;
    const long long pc = perm ? perm[c] : c;
    Sdiag[t] = S[(9 * pc + r) + (9 * pc + q) * lda];
}

// x[9 perm(c) + k] = v[9c + k] (to_band) or v[9c + k] = x[9 perm(c) + k].
__global__ void permute_cameras(const int* __restrict__ perm, int C, bool to_band, const double* __restrict__ in,
                                double* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 9 * C) return;
    const int c = t / 9, k = t % 9;
    const long long pos = 9ll * perm[c] + k;
    if (to_band)
        out[pos] = in[t];
    else
        out[t] = in[pos];
}

// Right-hand side: per camera chunk the sum of its T_e bp (tb, camera-major:
// contiguous), thread (position, component), positions added in order; then
// rhs_c = bc_c - the chunk sums in order.
constexpr int kRhsPos = 28;
__global__ void __launch_bounds__(9 * kRhsPos) rhs_chunks_kernel(const int* __restrict__ cchunk_begin,
                                                                const int* __restrict__ cchunk_cam,
                                                                const int* __restrict__ cam_off, int chunk_slots,
                                                                const double* __restrict__ tb,
                                                                double* __restrict__ part) {
    __shared__ double sh[9 * kRhsPos];
    const int k = blockIdx.x, b = cchunk_begin[k], e = min(b + chunk_slots, cam_off[cchunk_cam[k] + 1]);
    double v0 = 0.0, v1 = 0.0;
    const double* p = tb + 9ll * b;
    const int n = 9 * (e - b);
    int i = threadIdx.x;
    for (; i + 9 * kRhsPos < n; i += 18 * kRhsPos) {
        v0 += p[i];
        v1 += p[i + 9 * kRhsPos];
    }
    if (i < n) v0 += p[i];
    sh[threadIdx.x] = v0 + v1;
    __syncthreads();
    if (threadIdx.x < 9) {
        double v = 0.0;
        for (int q = 0; q < kRhsPos; ++q) v += sh[9 * q + threadIdx.x];
        part[9ll * k + threadIdx.x] = v;
    }
}
__global__ void rhs_finalize_kernel(const int* __restrict__ cam_chunk_off, const double* __restrict__ part,
                                    const double* __restrict__ bc, int C, double* __restrict__ rhs) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 9 * C) return;
    const int c = t / 9, k = t - 9 * c;
    double v = 0.0;
    for (int q = cam_chunk_off[c]; q < cam_chunk_off[c + 1]; ++q) v += part[9ll * q + k];
    rhs[t] = bc[t] - v;
}

// ---------------------------------------------------------------- FP64 Cholesky
//
// The explicitly chosen layouts, dense and band, keep the reference's arithmetic: an
// FP64 factorisation (the trailing update by mma.sync m8n8k4, the FP64 pipe's rate), for
// callers that want it and to check the fixed-point one (chol.cu) against, which serves
// the automatic layout and the standalone calls.

// Factor the NB x NB diagonal block at (j0, j0) in shared memory.
// The pivot's square root and its reciprocal are taken once per column (by
// thread 0) and the column is scaled by multiplication: FP64 square roots and
// divisions expand into many instructions on GB300's narrow FP64 pipe, and the
// kernel runs on one SM, on the factorisation's critical path.
__global__ void __launch_bounds__(256) potrf_diag_kernel(double* __restrict__ A, int j0, int lda, int* __restrict__ info) {
    __shared__ double a[NB][NB + 1];  // a[col][row]
    __shared__ double lk[2];          // L_kk, 1 / L_kk
    __shared__ int failed;
    if (*info) return;
    const int tid = threadIdx.x;
    for (int idx = tid; idx < NB * NB; idx += 256) {
        const int r = idx % NB, c = idx / NB;
        a[c][r] = r >= c ? A[(j0 + r) + (long long)(j0 + c) * lda] : 0.0;
    }
    if (tid == 0) failed = 0;
    __syncthreads();
    for (int k = 0; k < NB; ++k) {
        const double piv = a[k][k];
        if (!(piv > 0.0)) {
            if (tid == 0) {
                failed = 1;
                *info = j0 + k + 1;
            }
            break;  // every thread read the same pivot
        }
        if (tid == 0) {
            const double lkk = sqrt(piv);
            lk[0] = lkk;
            lk[1] = 1.0 / lkk;
        }
        __syncthreads();
        const double inv = lk[1];
        for (int r = k + 1 + tid; r < NB; r += 256) a[k][r] *= inv;
        if (tid == 0) a[k][k] = lk[0];
        __syncthreads();
        for (int idx = tid; idx < NB * NB; idx += 256) {
            const int r = idx % NB, c = idx / NB;
            if (c > k && r >= c) a[c][r] -= a[k][r] * a[k][c];
        }
        __syncthreads();
    }
    __syncthreads();
    if (failed) return;
    for (int idx = tid; idx < NB * NB; idx += 256) {
        const int r = idx % NB, c = idx / NB;
        if (r >= c) A[(j0 + r) + (long long)(j0 + c) * lda] = a[c][r];
    }
}

// Panel solve: rows [j0+NB, n) of columns [j0, j0+NB) := B L_jj^{-T}.
// Rows are independent in X L^T = B: a CTA takes `rows` (a divisor of NB) rows
// of one panel tile, so that a narrow panel (a band's few tiles) still spreads
// over NB / rows CTAs per tile.
__global__ void __launch_bounds__(256) trsm_panel_kernel(double* __restrict__ A, int j0, int lda, int rows,
                                                        const int* __restrict__ info) {
    extern __shared__ double tsm[];
    double(*L)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(tsm);                  // L[col][row]
    double(*X)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(tsm + NB * (NB + 1));  // X[col][row < rows]
    if (*info) return;
    const int tid = threadIdx.x;
    const int parts = NB / rows;
    const long long r0 = j0 + NB + (long long)NB * (blockIdx.x / parts) + (long long)rows * (blockIdx.x % parts);
    __shared__ double rinv[NB];  // 1 / L_kk, one division per column
    for (int idx = tid; idx < NB * NB; idx += 256) {
        const int r = idx % NB, c = idx / NB;
        L[c][r] = r >= c ? A[(j0 + r) + (long long)(j0 + c) * lda] : 0.0;
    }
    for (int idx = tid; idx < rows * NB; idx += 256) {
        const int r = idx % rows, c = idx / rows;
        X[c][r] = A[(r0 + r) + (long long)(j0 + c) * lda];
    }
    if (tid < NB) rinv[tid] = 1.0 / A[(j0 + tid) + (long long)(j0 + tid) * lda];
    __syncthreads();
    for (int k = 0; k < NB; ++k) {
        const double d = rinv[k];
        for (int r = tid; r < rows; r += 256) X[k][r] *= d;
        __syncthreads();
        for (int idx = tid; idx < rows * NB; idx += 256) {
            const int r = idx % rows, c = idx / rows;
            if (c > k) X[c][r] -= X[k][r] * L[k][c];
        }
        __syncthreads();
    }
    for (int idx = tid; idx < rows * NB; idx += 256) {
        const int r = idx % rows, c = idx / rows;
        A[(r0 + r) + (long long)(j0 + c) * lda] = X[c][r];
    }
}

__device__ __forceinline__ void dmma_m8n8k4(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Trailing update of the lower tiles: C(ti,tj) -= A(ti) A(tj)^T, K = NB (the
// panel). 8 warps per 64x64 tile, each warp 32x16 = 4x2 DMMA tiles.
__global__ void __launch_bounds__(256) syrk_update_kernel(double* __restrict__ A, int j0, int ntiles, int lda,
                                                         const int* __restrict__ info) {
    extern __shared__ double smem[];
    double* As = smem;             // [k][row], stride kSP
    double* Bs = smem + NB * kSP;  // [k][col]
    if (*info) return;
    // lower-triangular tile index from the linear block index
    const long long bidx = blockIdx.x;
    int ti = static_cast<int>((sqrt(8.0 * (double)bidx + 1.0) - 1.0) * 0.5);
    while ((long long)(ti + 1) * (ti + 2) / 2 <= bidx) ++ti;
    while ((long long)ti * (ti + 1) / 2 > bidx) --ti;
    const int tj = static_cast<int>(bidx - (long long)ti * (ti + 1) / 2);
    if (ti >= ntiles) return;
    const long long R0 = j0 + NB + (long long)NB * ti, C0 = j0 + NB + (long long)NB * tj;
    const int tid = threadIdx.x;
    for (int idx = tid; idx < NB * NB; idx += 256) {
        const int r = idx % NB, k = idx / NB;
        As[k * kSP + r] = A[(R0 + r) + (long long)(j0 + k) * lda];
        Bs[k * kSP + r] = A[(C0 + r) + (long long)(j0 + k) * lda];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 16;
    const int fr = lane >> 2, fk = lane & 3;
    double acc[4][2][2];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
#pragma unroll 4
    for (int kk = 0; kk < NB; kk += 4) {
        const double* ak = As + (kk + fk) * kSP + wm + fr;
        const double* bk = Bs + (kk + fk) * kSP + wn + fr;
        double af[4], bf[2];
#pragma unroll
        for (int m = 0; m < 4; ++m) af[m] = ak[8 * m];
#pragma unroll
        for (int n = 0; n < 2; ++n) bf[n] = bk[8 * n];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n) dmma_m8n8k4(acc[m][n], af[m], bf[n]);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const long long row = R0 + wm + 8 * m + fr;
            const long long col = C0 + wn + 8 * n + 2 * fk;
            A[row + col * lda] -= acc[m][n][0];
            A[row + (col + 1) * lda] -= acc[m][n][1];
        }
}

// The trailing update by 32 x 32 quadrants (four CTAs per 64 x 64 tile, the
// upper quadrant of a diagonal tile skipped): for steps with few tiles (a
// band's bt(bt+1)/2), so that the update spreads over four times as many SMs.
// 8 warps per quadrant, each warp 8 x 16 = 1 x 2 DMMA tiles.
constexpr int kSPq = 32 + 8;  // shared-memory stride (doubles) of the quadrant's K-major operands
__global__ void __launch_bounds__(256) syrk_update_quad_kernel(double* __restrict__ A, int j0, int ntiles, int lda,
                                                              const int* __restrict__ info) {
    __shared__ double As[NB * kSPq];  // [k][row]
    __shared__ double Bs[NB * kSPq];  // [k][col]
    if (*info) return;
    const long long bidx = blockIdx.x >> 2;
    const int quad = blockIdx.x & 3, qr = quad >> 1, qc = quad & 1;
    int ti = static_cast<int>((sqrt(8.0 * (double)bidx + 1.0) - 1.0) * 0.5);
    while ((long long)(ti + 1) * (ti + 2) / 2 <= bidx) ++ti;
    while ((long long)ti * (ti + 1) / 2 > bidx) --ti;
    const int tj = static_cast<int>(bidx - (long long)ti * (ti + 1) / 2);
    if (ti >= ntiles || (ti == tj && qr < qc)) return;
    const long long R0 = j0 + NB + (long long)NB * ti + 32 * qr, C0 = j0 + NB + (long long)NB * tj + 32 * qc;
    const int tid = threadIdx.x;
    for (int idx = tid; idx < 32 * NB; idx += 256) {
        const int r = idx % 32, k = idx / 32;
        As[k * kSPq + r] = A[(R0 + r) + (long long)(j0 + k) * lda];
        Bs[k * kSPq + r] = A[(C0 + r) + (long long)(j0 + k) * lda];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    const int wm = (warp & 3) * 8, wn = (warp >> 2) * 16;
    const int fr = lane >> 2, fk = lane & 3;
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 4
    for (int kk = 0; kk < NB; kk += 4) {
        const double af = As[(kk + fk) * kSPq + wm + fr];
        const double* bk = Bs + (kk + fk) * kSPq + wn + fr;
        dmma_m8n8k4(acc[0], af, bk[0]);
        dmma_m8n8k4(acc[1], af, bk[8]);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const long long row = R0 + wm + fr;
        const long long col = C0 + wn + 8 * n + 2 * fk;
        A[row + col * lda] -= acc[n][0];
        A[row + (col + 1) * lda] -= acc[n][1];
    }
}

// ---------------------------------------------------------------- triangular solves
//
// The 64 dependent steps of a substitution through a diagonal tile take two
// FP64 instructions each, and GB300 issues one per warp every 64 cycles: 27 us a
// tile. So the diagonal tiles are inverted first, all at once (tile_inverse),
// and the substitution through the tiles is then one kernel per tile: x_j =
// L_jj^-1 b_j, refined once with the residual b_j - L_jj x_j (in every block, for
// itself), and the update of the block's own rows (forward) or columns (backward).
// Without the refinement a tile's backward error is four times that of the
// substitution (1.7 against 0.4 u |L||x|); with it, the same. What bounds a step: the
// launch, the three 64 x 64 products at 1.7 FMA per cycle, and the update; the
// operands (constant during the solve) are loaded before the previous step has ended.
// The first step is launched to start when the inversion has ended: waiting inside the
// kernel would order only the loads after the wait.

// A lower-triangular tile packed for its products with a vector: rows p and 63 - p have 65
// entries together, held in order (row p's first) by lane p, one per 32 places.
constexpr int kPacked = 65 * 32;
__device__ __forceinline__ int packed_at(int i, int k) {  // i >= k
    return i < 32 ? 32 * k + i : 32 * (k + 64 - i) + 63 - i;
}
// Per tile: its inverse and itself, and the same with rows and columns reversed and
// transposed (the upper triangle of the transpose as a lower one).
struct PackedTile {
    double inv[kPacked], tile[kPacked], inv_t[kPacked], tile_t[kPacked];
};

// L_jj^-1 and L_jj of every tile, packed: kInvCols columns X of the inverse per block,
// X_k = (e_k - sum_m L_km X_m) / L_kk as rank-1 updates of the rows below, one entry per
// thread. Bound by the 64 dependent steps (a product, a barrier and the update, whose
// FP64 instructions the warps of a sub-partition take in turn): one tile per block with
// its rows and columns in turn took 60 us, 12 us so.
constexpr int kInvCols = 8;
constexpr int kInvT = NB * kInvCols;
__global__ void __launch_bounds__(kInvT) tile_inverse(const double* __restrict__ L, int lda,
                                                     PackedTile* __restrict__ out, const int* __restrict__ info) {
    extern __shared__ double t[];         // t[column NB + row] of L
    __shared__ double x[NB][kInvCols], rinv[NB];
    pdl_wait();
    if (*info) return;
    const long long j0 = static_cast<long long>(blockIdx.x) * NB;
    const int r = threadIdx.x & 63, cl = threadIdx.x >> 6, first = blockIdx.y * kInvCols, c = first + cl;
    for (int k = first + cl; k < NB; k += kInvCols) t[NB * k + r] = r >= k ? L[(j0 + r) + (j0 + k) * lda] : 0.0;
    if (cl == 0 && r >= first) rinv[r] = 1.0 / L[(j0 + r) + (j0 + r) * lda];
    __syncthreads();
    double v = r == c ? 1.0 : 0.0;
    for (int k = first; k < NB; ++k) {  // (columns right of k: zeros)
        if (r == k) x[k][cl] = v = v * rinv[k];
        __syncthreads();
        if ((r | 31) > k && r > k) v -= t[NB * k + r] * x[k][cl];
    }
    if (r < c) return;
    PackedTile& o = out[blockIdx.x];
    double l = t[NB * c + r];
    if (r == c && isinf(l)) l = 0.0;  // weight infinity: x is 0 there, and so is its part of a residual
    const int at = packed_at(r, c), at_t = packed_at(63 - c, 63 - r);
    o.inv[at] = v;
    o.tile[at] = l;
    o.inv_t[at_t] = v;
    o.tile_t[at_t] = l;
}

// Products of packed tiles with a vector in shared memory, by the first four warps: lane
// p of warp q takes every fourth of its two rows' entries (17 FMAs; a thread per row
// and group of columns, with the zeros that share a warp with entries, 32).
constexpr int kPairT = 128, kPairN = 17;
__device__ __forceinline__ void load_packed(const double* __restrict__ M, double (&m)[kPairN]) {
    const int p = threadIdx.x & 31, q = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < kPairN; ++i) m[i] = q < 4 && q + 4 * i < 65 ? M[32 * (q + 4 * i) + p] : 0.0;
}
__device__ __forceinline__ void pair_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
// Row r of M b, for threads r < 64 (all four warps call it).
__device__ __forceinline__ double packed_row(const double (&m)[kPairN], const double* b, double (*part)[NB]) {
    const int p = threadIdx.x & 31, q = threadIdx.x >> 5;
    double s = 0.0, upper = 0.0;  // row 63 - p, row p
#pragma unroll
    for (int i = 0; i < kPairN; ++i) {
        const int e = q + 4 * i;
        if (e >= 65) continue;
        if (e > p && e - 4 <= p) {
            upper = s;
            s = 0.0;
        }
        s = fma(m[i], b[e > p ? e - p - 1 : e], s);
    }
    part[q][p] = upper;
    part[q][63 - p] = s;
    pair_sync();
    const int r = threadIdx.x & 63;
    return (part[0][r] + part[1][r]) + (part[2][r] + part[3][r]);
}
struct TileShared {
    double part[4][NB], b[NB], x[NB];
};
// x = T^-1 b (sm.b, overwritten) with T's inverse m and T itself (t), refined once.
// kReversed: b's rows and those of T are in reverse order, x's are not.
template <bool kReversed>
__device__ __forceinline__ void tile_solve(const double (&m)[kPairN], const double (&t)[kPairN], TileShared& sm,
                                           double* x) {
    if (threadIdx.x < kPairT) {
        const int r = threadIdx.x;
        const double x1 = packed_row(m, sm.b, sm.part);
        if (r < NB) sm.x[r] = x1;
        pair_sync();
        const double ax = packed_row(t, sm.x, sm.part);
        if (r < NB) sm.b[r] -= ax;
        pair_sync();
        const double v = x1 + packed_row(m, sm.b, sm.part);
        if (r < NB) x[kReversed ? 63 - r : r] = isfinite(v) ? v : x1;  // (x1 out of range: no residual)
    }
    __syncthreads();
}

constexpr int kSolT = 256;
constexpr int kSolRows = 16;  // rows (columns) of L per pass of a block

// Forward step j: y_j = L_jj^-1 b_j, b[j0 + 64 : r_end) -= L[.., j] y_j.
// blockIdx.y = 1: the second chain's tile, dj rows further on.
__global__ void __launch_bounds__(kSolT) forward_step(const double* __restrict__ L, int j0, int r_end, int dj, int lda,
                                                     const PackedTile* __restrict__ tiles, double* __restrict__ b,
                                                     double* __restrict__ y, const int* __restrict__ info) {
    __shared__ TileShared sm;
    __shared__ double x[NB], red[kSolRows][kSolT / kSolRows + 1];
    const int lr = threadIdx.x & (kSolRows - 1), kg = threadIdx.x / kSolRows;  // row, group of four columns
    j0 += blockIdx.y * dj;
    r_end += blockIdx.y * dj;
    double m[kPairN], t[kPairN], l[4] = {0.0, 0.0, 0.0, 0.0};
    load_packed(tiles[j0 / NB].inv, m);
    load_packed(tiles[j0 / NB].tile, t);
    int r = j0 + NB + blockIdx.x * kSolRows + lr;
    if (r < r_end) {
#pragma unroll
        for (int i = 0; i < 4; ++i) l[i] = L[r + static_cast<long long>(j0 + 4 * kg + i) * lda];
    }
    pdl_wait();
    pdl_trigger();
    if (*info) return;
    if (threadIdx.x < NB) sm.b[threadIdx.x] = b[j0 + threadIdx.x];
    __syncthreads();
    tile_solve<false>(m, t, sm, x);
    if (blockIdx.x == 0 && threadIdx.x < NB) y[j0 + threadIdx.x] = x[threadIdx.x];
    for (int base = j0 + NB + blockIdx.x * kSolRows; base < r_end; base += gridDim.x * kSolRows) {
        const int nr = base + gridDim.x * kSolRows + lr;
        const double s = fma(l[0], x[4 * kg], l[1] * x[4 * kg + 1]) + fma(l[2], x[4 * kg + 2], l[3] * x[4 * kg + 3]);
        if (nr < r_end) {
#pragma unroll
            for (int i = 0; i < 4; ++i) l[i] = L[nr + static_cast<long long>(j0 + 4 * kg + i) * lda];
        }
        red[lr][kg] = s;
        __syncthreads();
        // sixteen partial sums per row, added by a half-warp tree
        double v = red[kg][lr];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, 16);
        if (lr == 0 && base + kg < r_end) b[base + kg] -= v;
        __syncthreads();
    }
}

// Backward step j: x_j = L_jj^-T y_j (into b), y[i0 : i1) -= L[j, ..]^T x_j.
// known >= 0: x_j is there already, as b[known], b[known - 1], ...
struct BackwardTile {
    int j0, i0, i1, known;
};
__global__ void __launch_bounds__(kSolT) backward_step(const double* __restrict__ L, BackwardTile t0, BackwardTile t1,
                                                      int lda, const PackedTile* __restrict__ tiles,
                                                      double* __restrict__ y, double* __restrict__ b,
                                                      const int* __restrict__ info) {
    __shared__ TileShared sm;
    __shared__ double x[NB];
    const int kg = threadIdx.x & 15, lc = threadIdx.x >> 4;  // group of four rows, column
    const BackwardTile t = blockIdx.y ? t1 : t0;
    const int j0 = t.j0;
    double m[kPairN], d[kPairN], l[4] = {0.0, 0.0, 0.0, 0.0};
    if (t.known < 0) {
        load_packed(tiles[j0 / NB].inv_t, m);
        load_packed(tiles[j0 / NB].tile_t, d);
    }
    int c = t.i0 + blockIdx.x * kSolRows + lc;
    if (c < t.i1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) l[i] = L[j0 + 4 * kg + i + static_cast<long long>(c) * lda];
    }
    pdl_wait();
    pdl_trigger();
    if (*info) return;
    if (t.known >= 0) {
        if (threadIdx.x < NB) x[threadIdx.x] = b[t.known - threadIdx.x];
        __syncthreads();
    } else {
        if (threadIdx.x < NB) sm.b[63 - threadIdx.x] = y[j0 + threadIdx.x];
        __syncthreads();
        tile_solve<true>(m, d, sm, x);
        if (blockIdx.x == 0 && threadIdx.x < NB) b[j0 + threadIdx.x] = x[threadIdx.x];
    }
    for (; c - lc < t.i1; c += gridDim.x * kSolRows) {
        double v = fma(l[0], x[4 * kg], l[1] * x[4 * kg + 1]) + fma(l[2], x[4 * kg + 2], l[3] * x[4 * kg + 3]);
        const int nc = c + gridDim.x * kSolRows;
        if (nc < t.i1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) l[i] = L[j0 + 4 * kg + i + static_cast<long long>(nc) * lda];
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, 16);
        if (kg == 0 && c < t.i1) y[c] -= v;
    }
}

// The right-hand side of the two chains of band_potrf_twisted, and the solution back
// in the band's order. base: the second chain's first row, its last s rows copies.
__global__ void twist_rhs(const double* __restrict__ b, int n, int base, int s, double* __restrict__ bt) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n + s) bt[i] = i < base ? b[i] : i < n ? b[n - 1 - (i - base)] : 0.0;
}
__global__ void twist_merge_rhs(int n, int base, int s, double* __restrict__ bt) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // row base - s + i of the band
    if (i < s) bt[base - s + i] += bt[n + s - 1 - i];
}
__global__ void twist_solution(const double* __restrict__ bt, int n, int base, const int* __restrict__ info,
                               double* __restrict__ b) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && *info == 0) b[i] = bt[i < base ? i : base + n - 1 - i];
}

}  // namespace

// bt, lda: as for dense_potrf (chol.cu).
static void dense_potrf_fp64(double* A, int n, int lda, int bt, int* info, cudaStream_t s) {
    GBA_CUDA_CHECK(cudaMemsetAsync(info, 0, sizeof(int), s));
    static bool attr = false;
    const int smem = 2 * NB * kSP * sizeof(double);
    const int tsmem = 2 * NB * (NB + 1) * sizeof(double);
    if (!attr) {
        GBA_CUDA_CHECK(cudaFuncSetAttribute(syrk_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        GBA_CUDA_CHECK(cudaFuncSetAttribute(trsm_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tsmem));
        attr = true;
    }
    const int nt = n / NB;
    for (int jb = 0; jb < nt; ++jb) {
        const int j0 = jb * NB;
        potrf_diag_kernel<<<1, 256, 0, s>>>(A, j0, lda, info);
        GBA_LAUNCH_CHECK();
        const int below = std::min(nt - jb - 1, bt);
        if (below == 0) continue;
        // few panel tiles (a band, or the last steps): split them over more CTAs
        const int sms = device_sm_count();
        const int rows = below * 4 <= sms ? 16 : NB;
        trsm_panel_kernel<<<below * (NB / rows), 256, tsmem, s>>>(A, j0, lda, rows, info);
        GBA_LAUNCH_CHECK();
        const long long tiles = (long long)below * (below + 1) / 2;
        if (tiles * 2 <= sms)
            syrk_update_quad_kernel<<<static_cast<unsigned>(4 * tiles), 256, 0, s>>>(A, j0, below, lda, info);
        else
            syrk_update_kernel<<<static_cast<unsigned>(tiles), 256, smem, s>>>(A, j0, below, lda, info);
        GBA_LAUNCH_CHECK();
    }
}

// first: the step after tile_inverse.
static void launch_forward(bool first, dim3 grid, const double* L, int j0, int r_end, int dj, int lda,
                           const PackedTile* tiles, double* b, double* y, const int* info, cudaStream_t s) {
    if (first) {
        forward_step<<<grid, kSolT, 0, s>>>(L, j0, r_end, dj, lda, tiles, b, y, info);
        GBA_LAUNCH_CHECK();
    } else {
        launch_pdl(forward_step, grid, kSolT, 0, s, L, j0, r_end, dj, lda, tiles, b, y, info);
    }
}

// Of n rows: the packed tiles and a vector.
struct SolveWork {
    PackedTile* tiles;
    double* y;
    SolveWork(void* ws, int n) : tiles(static_cast<PackedTile*>(ws)), y(reinterpret_cast<double*>(tiles + n / NB)) {}
};
size_t dense_potrs_workspace(int n) { return n / NB * sizeof(PackedTile) + n * sizeof(double); }

static void invert_tiles(const double* L, int nt, int lda, const SolveWork& w, const int* info, cudaStream_t s) {
    launch_pdl(tile_inverse, dim3(nt, NB / kInvCols), kInvT, NB * NB * sizeof(double), s, L, lda, w.tiles, info);
}
// Blocks of a step over `rows` rows (columns) of each chain. Two passes of a block at
// most where the rows allow it: a further pass costs a block less than a further block
// costs the launch.
static dim3 step_grid(int rows, int chains) {
    return dim3(std::max(1, std::min(2 * device_sm_count(), ceil_div(rows, kSolRows))), chains);
}

void dense_potrs(const double* L, int n, int lda, int bt, double* b, const int* info, void* workspace,
                 cudaStream_t s) {
    if (n % NB != 0 || bt < 0 || (bt < n / NB - 1 ? lda + 1 < (bt + 2) * NB : lda < n))
        throw std::invalid_argument("dense_potrs: n must be a multiple of 64 and lda hold the band");
    const int nt = n / NB;
    const SolveWork w(workspace, n);
    invert_tiles(L, nt, lda, w, info, s);
    for (int jb = 0; jb < nt; ++jb) {
        const int j0 = jb * NB;
        const int r_end = static_cast<int>(std::min<long long>(n, j0 + NB + (long long)bt * NB));
        launch_forward(jb == 0, step_grid(r_end - j0 - NB, 1), L, j0, r_end, 0, lda, w.tiles, b, w.y, info, s);
    }
    for (int jb = nt - 1; jb >= 0; --jb) {
        const int j0 = jb * NB, i0 = std::max(0, j0 - bt * NB);
        const BackwardTile t{j0, i0, j0, -1};
        launch_pdl(backward_step, step_grid(j0 - i0, 1), kSolT, 0, s, L, t, t, lda, w.tiles, w.y, b, info);
    }
}

size_t band_twist_solve_workspace(int n, int bt) {
    return dense_potrs_workspace(n + NB * bt) + sizeof(double) * (n + static_cast<size_t>(NB) * bt);
}

void band_potrs_twisted(const double* F, int n, int lda, int bt, int ta, double* b, const int* info, void* workspace,
                        cudaStream_t s) {
    const int np = n + bt * NB, sep = bt * NB, a = ta * NB, base = a + sep, tb = n / NB - ta - bt;
    const SolveWork w(workspace, np);
    double* x = w.y + np;
    launch_pdl(twist_rhs, ceil_div(np, 256), 256, 0, s, b, n, base, sep, x);
    invert_tiles(F, n / NB, lda, w, info, s);  // not those of the copies
    for (int k = 0; k < std::max(ta, tb); ++k) {
        const int chains = k < ta && k < tb ? 2 : 1, j0 = k * NB + (k < ta ? 0 : base);
        launch_forward(k == 0, step_grid(sep, chains), F, j0, j0 + NB + sep, base, lda, w.tiles, x, w.y, info, s);
    }
    launch_pdl(twist_merge_rhs, ceil_div(sep, 256), 256, 0, s, n, base, sep, x);
    for (int k = 0; k < bt; ++k) {
        const int j0 = a + k * NB;
        launch_forward(false, step_grid(base - j0 - NB, 1), F, j0, base, 0, lda, w.tiles, x, w.y, info, s);
    }
    auto columns = [&](int j0, int first) { return std::max(first, j0 - sep); };
    for (int k = bt - 1; k >= 0; --k) {
        const int j0 = a + k * NB, i0 = columns(j0, 0);
        const BackwardTile t{j0, i0, j0, -1};
        launch_pdl(backward_step, step_grid(j0 - i0, 1), kSolT, 0, s, F, t, t, lda, w.tiles, w.y, x, info);
    }
    // chain 0's tiles above, beside chain 1's: the rows between (known now), then its own
    for (int k = 0; k < std::max(ta, tb + bt); ++k) {
        BackwardTile t[2];
        int m = 0;
        if (k < ta) {
            const int j0 = a - (k + 1) * NB;
            t[m++] = {j0, columns(j0, 0), j0, -1};
        }
        if (k < tb + bt) {
            const int j0 = np - (k + 1) * NB;
            // row j0 + i of chain 1 is row base + n - 1 - j0 - i of the band
            t[m++] = {j0, columns(j0, base), std::min(j0, n), k < bt ? base + n - 1 - j0 : -1};
        }
        launch_pdl(backward_step, step_grid(sep, m), kSolT, 0, s, F, t[0], t[m - 1], lda, w.tiles, w.y, x,
                   info);
    }
    launch_pdl(twist_solution, ceil_div(n, 256), 256, 0, s, x, n, base, info, b);
}

void Solver::ensure_schur_storage() {
    const int want = schur_layout_;
    if (S_.get() && schur_layout_planned_ == want) return;
    bool band = false;
    if (want == 2) {
        plan_schur_band();
        band = true;
    } else if (want == 0 && C_ >= 2 && 3ll * n_blocks_ <= static_cast<long long>(C_) * C_) {
        plan_schur_band();  // a band can only pay with at most ~1/3 of the blocks present
        band = band_beneficial_;
    }
    band_mode_ = band;
    S_.release();
    S_.alloc(static_cast<size_t>(n_pad_) * (band ? band_ldb_ : n_pad_));
    // A band that pays is factored from both ends (an explicitly chosen one leaves its
    // factor in S): 3 (bt + 2) <= nt, so at least bt + 3 of the nt panels run beside others.
    const int nt = n_pad_ / NB;
    twist_ta_ = band && want == 0 ? (nt - band_bt_ + 1) / 2 : 0;
    twist_.release();
    size_t ws = std::max(dense_potrf_workspace(n_pad_), dense_potrs_workspace(n_pad_));
    if (twist_ta_) {
        twist_.alloc(static_cast<size_t>(n_pad_ + NB * band_bt_) * band_ldb_);
        ws = std::max(ws, std::max(band_twist_workspace(n_pad_, band_bt_), band_twist_solve_workspace(n_pad_, band_bt_)));
    }
    if (chol_ws_.size() < ws) {
        chol_ws_.release();
        chol_ws_.alloc(ws);
    }
    schur_layout_planned_ = want;
}

static const char* const kWaitRanOut = "dense_potrf: a wait of the trailing update ran out";

int Solver::schur_dense(double lambda) {
    ensure_schur_storage();
    const int lda = band_mode_ ? band_ldb_ - 1 : n_pad_;
    const int bt = band_mode_ ? band_bt_ : n_pad_ / NB - 1;
    const int* perm = band_mode_ ? cam_perm_.get() : nullptr;
    // T_e bp (9 per observation) in the place of the camera pass's Jacobian records
    // (20 per observation), which are not read after it
    double* tb = JcR_.get();
    compute_T_kernel<<<ceil_div(9ll * E_, kTT), kTT, 0, stream_>>>(W_.get(), Vinv_.get(), bp_.get(), s_pt_.get(),
                                                                 cam_pos_.get(), E_, T_.get(), tb);
    GBA_LAUNCH_CHECK();
    GBA_CUDA_CHECK(cudaMemsetAsync(S_.get(), 0, S_.size() * sizeof(double), stream_));
    if (n_blocks_ > 0) {
        cudaEvent_t ev = prof_start();
        assemble_kernel<<<ceil_div(9ll * n_blocks_, 288), 288, 0, stream_>>>(
            block_off_.get(), block_ce_.get(), block_cf_.get(), pair_e_.get(), pair_f_.get(), T_.get(), W_.get(),
            n_blocks_, lda, perm, S_.get());
        GBA_LAUNCH_CHECK();
        if (n_long_ > 0) {
            const int4* chunks = reinterpret_cast<const int4*>(long_chunks_.get());
            assemble_chunks_kernel<<<n_long_chunks_, 9 * kSlices, 0, stream_>>>(chunks, pair_e_.get(), pair_f_.get(),
                                                                               T_.get(), W_.get(), long_part_.get());
            GBA_LAUNCH_CHECK();
            assemble_finalize_kernel<<<n_long_, 96, 0, stream_>>>(long_off_.get(), chunks, block_ce_.get(),
                                                                  block_cf_.get(), long_part_.get(), lda, perm,
                                                                  S_.get());
            GBA_LAUNCH_CHECK();
        }
        prof_stop("schur_assemble", ev);
    }
    add_damped_u_kernel<<<ceil_div(81ll * C_ + (n_pad_ - 9 * C_), 256), 256, 0, stream_>>>(U_.get(), lambda, C_,
                                                                                        n_pad_, lda, perm, S_.get());
    GBA_LAUNCH_CHECK();
    GBA_CUDA_CHECK(cudaMemsetAsync(rhs_.get(), 0, rhs_.size() * sizeof(double), stream_));
    if (n_cchunk_ > 0) {
        rhs_chunks_kernel<<<n_cchunk_, 9 * kRhsPos, 0, stream_>>>(cchunk_begin_.get(), cchunk_cam_.get(),
                                                                 cam_off_.get(), kCamChunkSlots, tb,
                                                                 cam_part_.get());
        GBA_LAUNCH_CHECK();
    }
    rhs_finalize_kernel<<<ceil_div(9ll * C_, 128), 128, 0, stream_>>>(cam_chunk_off_.get(), cam_part_.get(),
                                                                     bc_.get(), C_, rhs_.get());
    GBA_LAUNCH_CHECK();
    if (harvest_) {
        if (!Sdiag_.get()) Sdiag_.alloc(81ull * C_);
        extract_diag_blocks<<<ceil_div(81ll * C_, 256), 256, 0, stream_>>>(S_.get(), C_, lda, perm, Sdiag_.get());
        GBA_LAUNCH_CHECK();
    }
    bool twisted = twist_ta_ > 0;  // the factor is in twist_, not in S
    s_assembled_ = false;
    cudaEvent_t ev = prof_start();
    if (schur_layout_ != 0)
        dense_potrf_fp64(S_.get(), n_pad_, lda, bt, info_.get(), stream_);
    else if (twisted)
        band_potrf_twisted(S_.get(), n_pad_, lda, bt, twist_ta_, twist_.get(), info_.get(), chol_ws_.get(), stream_);
    else
        dense_potrf(S_.get(), n_pad_, lda, bt, info_.get(), chol_ws_.get(), stream_);
    prof_stop("dense_potrf", ev);
    int info = 0;
    read_back({{&info, info_.get(), sizeof info}});
    if (twisted && info > 0) {
        // Which chain meets its bad pivot first, and where, is not what the rows in their
        // order would say: ask them.
        twisted = false;
        dense_potrf(S_.get(), n_pad_, lda, bt, info_.get(), chol_ws_.get(), stream_);
        read_back({{&info, info_.get(), sizeof info}});
    }
    if (info < 0) throw std::runtime_error(kWaitRanOut);
    if (info != 0) return info;
    // solve in a copy so rhs stays the assembled right-hand side (in the band
    // layout the copy is in the renumbered camera order; the padding stays 0)
    if (band_mode_) {
        GBA_CUDA_CHECK(cudaMemsetAsync(pcg_x_.get(), 0, n_pad_ * sizeof(double), stream_));
        permute_cameras<<<ceil_div(9 * C_, 256), 256, 0, stream_>>>(perm, C_, true, rhs_.get(), pcg_x_.get());
        GBA_LAUNCH_CHECK();
    } else {
        GBA_CUDA_CHECK(cudaMemcpyAsync(pcg_x_.get(), rhs_.get(), n_pad_ * sizeof(double), cudaMemcpyDeviceToDevice,
                                       stream_));
    }
    s_assembled_ = twisted;
    if (twisted)
        band_potrs_twisted(twist_.get(), n_pad_, lda, bt, twist_ta_, pcg_x_.get(), info_.get(), chol_ws_.get(), stream_);
    else
        dense_potrs(S_.get(), n_pad_, lda, bt, pcg_x_.get(), info_.get(), chol_ws_.get(), stream_);
    if (band_mode_) {
        permute_cameras<<<ceil_div(9 * C_, 256), 256, 0, stream_>>>(perm, C_, false, pcg_x_.get(), dc_.get());
        GBA_LAUNCH_CHECK();
    } else {
        GBA_CUDA_CHECK(cudaMemcpyAsync(dc_.get(), pcg_x_.get(), 9ull * C_ * sizeof(double), cudaMemcpyDeviceToDevice,
                                       stream_));
    }
    if (s_wanted_) keep_factor();
    sync();
    return 0;
}

void Solver::keep_factor() {
    s_wanted_ = true;
    if (!s_assembled_) return;
    dense_potrf(S_.get(), n_pad_, band_ldb_ - 1, band_bt_, info_.get(), chol_ws_.get(), stream_);
    s_assembled_ = false;
    int info = 0;
    read_back({{&info, info_.get(), sizeof info}});  // (S is there, on any stream)
    if (info < 0) throw std::runtime_error(kWaitRanOut);
}

}  // namespace gba
