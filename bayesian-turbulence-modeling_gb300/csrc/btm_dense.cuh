// btm_dense.cuh - dense FP64 inverse of the coarsest multigrid level
// (Gauss-Jordan in place, no pivoting: the level matrices are SPD), shared by
// the FP64 and mixed-precision engines.
//
// Step k of the textbook scheme on [A | I]: the pivot row times 1 / A_kk, then
// every other row minus its column-k entry times the pivot row (one fma per
// element).  Of the 2n columns only n + 1 change in a step, and those with one
// place each in an n x n array: column k of A becomes a unit vector and column
// k of the right-hand side is born.  Both variants below do the same
// operations on every element in the same order as the sweep over all 2n
// columns, so the inverse is the same bits.
#pragma once
#include "btm_common.h"
#include "btm_team.cuh"
#include <type_traits>

namespace btm {

__device__ __forceinline__ bool bad_pivot(double piv) { return !(fabs(piv) > 1e-300); }

// n <= kCoarseDirect on one CTA, A [n][n] (shared or global).  The reciprocal of
// a pivot (8-9 dependent FP64 instructions, 550 clocks) is the longest part of a
// step: warp 0 forms the next pivot first and its reciprocal while the other
// warps update the matrix.  Returns false, with A half done, at a vanishing pivot.
template <class T>
__device__ __noinline__ bool dense_inverse_small(T &tm, double *A, int n) {
    static_assert(kCoarseDirect == 32, "a row to a warp");
    __shared__ double row[kCoarseDirect], col[kCoarseDirect], next;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    if (t == 0) next = A[0];
    __syncthreads();
    double piv = next;
    double rp = warp == 0 ? 1.0 / piv : 0.0;
    for (int k = 0; k < n; ++k) {
        if (bad_pivot(piv)) return false;   // the same on every thread
        if (warp == 0) {
            if (lane < n) row[lane] = lane == k ? rp : A[k * n + lane] * rp;
        } else if (warp == 1) {
            if (lane < n && lane != k) col[lane] = A[lane * n + k];
        }
        __syncthreads();
        if (warp == 0) {
            if (k + 1 < n) {
                piv = fma(-col[k + 1], row[k + 1], A[(k + 1) * n + k + 1]);
                if (lane == 0) next = piv;
                rp = 1.0 / piv;
            }
        } else {
            for (int i = warp - 1; i < n; i += nw - 1) {
                if (lane < n) {
                    double v = row[lane];
                    if (i != k) v = fma(-col[i], v, lane == k ? 0.0 : A[i * n + lane]);
                    // warp 0 reads the next pivot's old value meanwhile; its
                    // place is not read again before the pivot's own step
                    if (i != k + 1 || lane != k + 1) A[i * n + lane] = v;
                }
            }
        }
        __syncthreads();
        if (k + 1 < n) piv = next;
    }
    return true;
}

// Up to kCoarseDirectGrid rows on the whole team, A [n][n] in global memory,
// kPanel pivots at a time.  What the pivots of a panel do to the rest of the
// matrix depends only on the panel's multipliers (mult [n][kPanel]: a row's
// entry in the pivot column at the time of the pivot) and its scaled pivot rows
// (piv [kPanel][n]).  Both come from short recurrences: the kPanel x kPanel
// diagonal block, which every CTA works out for itself in shared memory, then
// 16 lanes per row (multipliers) or per column (pivot rows).  The rest of the
// matrix takes the kPanel updates of an element from registers in one pass:
// two grid barriers and one pass over the matrix per 16 pivots instead of one
// each per pivot, and half of the fused multiply-adds.  972 rows: 15.1 ms ->
// 2.6 ms (FP64 issue alone: 1.6 ms).
template <class T>
__device__ __noinline__ bool dense_inverse_panels(T &tm, double *A, double *mult, double *prow, int n) {
    __shared__ double D[kPanel][kPanel];     // diagonal block as it evolves
    __shared__ double Dm[kPanel][kPanel];    // [row][pivot] multipliers inside the block
    __shared__ double Dr[kPanel][kPanel];    // [pivot][column] scaled pivot rows inside the block
    __shared__ double Drp[kPanel];
    __shared__ int bad;
    const int t = threadIdx.x, lane = t & 31;
    const int half = lane >> 4, l = lane & 15;
    const unsigned full = 0xffffffffu;
    if (t == 0) bad = 0;
    __syncthreads();
    for (int k0 = 0; k0 < n; k0 += kPanel) {
        const int b = min(kPanel, n - k0);
        if (t < kPanel * kPanel) {
            const int i = t >> 4, j = t & 15;
            D[i][j] = i < b && j < b ? LD(A + (size_t)(k0 + i) * n + k0 + j) : 0.0;
        }
        __syncthreads();
        // four warps, one to an SMSP: a thread holds rows i and i + 8 of column j
        for (int k = 0; k < b; ++k) {
            const int i = t >> 4, j = t & 15;
            double rk = 0.0, m0 = 0.0, m1 = 0.0, v0 = 0.0, v1 = 0.0;
            if (t < 128) {
                const double piv = D[k][k];
                if (t == 0 && bad_pivot(piv)) bad = 1;
                const double rp = 1.0 / piv;
                rk = j == k ? rp : D[k][j] * rp;
                m0 = D[i][k];
                m1 = D[i + 8][k];
                v0 = j == k ? 0.0 : D[i][j];
                v1 = j == k ? 0.0 : D[i + 8][j];
                if (t == 0) Drp[k] = rp;
                if (i == (k & 7)) Dr[k][j] = rk;
                if (j == k) { Dm[i][k] = m0; Dm[i + 8][k] = m1; }
            }
            __syncthreads();
            if (t < 128) {
                D[i][j] = i == k ? rk : fma(-m0, rk, v0);
                D[i + 8][j] = i + 8 == k ? rk : fma(-m1, rk, v1);
            }
            __syncthreads();
        }
        if (bad) return false;   // the same in every CTA
        // multipliers of the rows outside the panel: 16 lanes hold a row's
        // panel columns; then the pivot rows' columns outside the panel, 16
        // lanes hold a column's panel rows.  Two of each to a warp.
        const int nOut = n - b, units = (nOut + 1) >> 1;
        for (int u = tm.spread() >> 5; u < 2 * units; u += tm.size() >> 5) {
            const bool rows = u < units;
            const int q = 2 * (rows ? u : u - units) + half;
            const bool on = q < nOut && l < b;
            const int o = q < k0 ? q : q + b;   // row or column outside the panel
            const size_t at = rows ? (size_t)o * n + k0 + l : (size_t)(k0 + l) * n + o;
            double v = on ? LD(A + at) : 0.0;
            if (rows) {
                for (int k = 0; k < b; ++k) {
                    const double m = __shfl_sync(full, v, (lane & 16) + k);
                    if (on && l == k) mult[(size_t)o * kPanel + k] = m;
                    v = fma(-m, Dr[k][l], l == k ? 0.0 : v);
                }
            } else {
                for (int k = 0; k < b; ++k) {
                    const double r = __shfl_sync(full, v, (lane & 16) + k) * Drp[k];
                    if (on && l == k) prow[(size_t)k * n + o] = r;
                    v = l == k ? r : fma(-Dm[l][k], r, v);
                }
            }
            if (on) A[at] = v;
        }
        tm.sync();
        // the diagonal block (every CTA has read its old values by now)
        if (tm.rank() < kPanel * kPanel) {
            const int i = t >> 4, j = t & 15;
            if (i < b && j < b) A[(size_t)(k0 + i) * n + k0 + j] = D[i][j];
        }
        // everything outside the panel's rows and columns
        const int strips = (n + 31) >> 5;
        const int warps = tm.size() >> 5, groups = max(1, warps / strips);
        for (int w = tm.rank() >> 5; w < strips * groups; w += warps) {
            const int g = w / strips, j = (w - g * strips) * 32 + lane;
            const bool on = j < n && (j < k0 || j >= k0 + b);
            double r[kPanel];
#pragma unroll
            for (int k = 0; k < kPanel; ++k) r[k] = on && k < b ? LD(prow + (size_t)k * n + j) : 0.0;
            for (int i = g; i < n; i += groups) {
                if (i >= k0 && i < k0 + b) continue;
                const double *m = mult + (size_t)i * kPanel;
                if (!on) continue;
                double v = LD(A + (size_t)i * n + j);
                if (b == kPanel) {
                    double mk[kPanel];
#pragma unroll
                    for (int k = 0; k < kPanel; ++k) mk[k] = LD(m + k);
#pragma unroll
                    for (int k = 0; k < kPanel; ++k) v = fma(-mk[k], r[k], v);
                } else {
#pragma unroll
                    for (int k = 0; k < kPanel; ++k)
                        if (k < b) v = fma(-LD(m + k), r[k], v);
                }
                A[(size_t)i * n + j] = v;
            }
        }
        tm.sync();
    }
    return true;
}

// Inverse of the n x n matrix in A (filled by the caller, every thread past a
// barrier); work [2 kPanel n] doubles; n <= kCoarseDirect on one CTA.  False: a
// pivot vanished.
template <class T>
__device__ __forceinline__ bool dense_inverse(T &tm, double *A, double *work, int n) {
    if constexpr (std::is_same<T, GridTeam>::value) {
        return dense_inverse_panels(tm, A, work, work + (size_t)kPanel * n, n);
    } else {
        return dense_inverse_small(tm, A, n);
    }
}

}  // namespace btm
