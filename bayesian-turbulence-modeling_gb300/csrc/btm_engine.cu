// btm_engine.cu - the GB300 SIMPLE / SST k-omega engine (sm_103a).
//
// One persistent launch runs a whole forward solve G(x, theta): every phase of
// the reference outer iteration (incompressible/src/SIMPLESolver.cpp:731-1036)
// is a device function templated on a "team":
//   * BlockTeam - one CTA owns one instance (small meshes; a batch of N
//     instances is a grid of N CTAs, each retiring when its solve ends);
//   * GridTeam  - every CTA of a cooperative launch owns one large instance,
//     phases separated by a bounded software grid barrier.
// Control flow is team-uniform: all decisions use values every thread of the
// team computed identically (deterministic fixed-order reductions).
//
// Floating point: the file is compiled with -fmad=false and every face sum is
// evaluated per cell in ascending face order, the order in which the
// reference's face loops scatter into that cell.  Assembly, gradients and the
// LDU mat-vec therefore round exactly like the reference; only dot products
// (parallel trees) and transcendental library calls differ in the last bits.
// There are no floating-point atomics anywhere.
#include "btm_common.h"
#include <type_traits>
#include "btm_team.cuh"
#include "btm_bc.cuh"
#include "btm_phases64.cuh"
#include "btm_observe.cuh"
#include "btm_ramg.cuh"
#include "btm_dense.cuh"
#include "btm_cycle.cuh"

#include <cuda_runtime.h>
#include <stdint.h>

namespace btm {

constexpr int kThreads = 512;

// ---- pressure AMG ---------------------------------------------------------
__device__ __forceinline__ double *lev_vals(DevInst &I, const DevMesh &M, int l) {
    return l == 0 ? I.diag : I.amgVal + M.lev[l].valOff;
}
__device__ __forceinline__ double *lev_x(DevInst &I, const DevMesh &M, int l) {
    return l == 0 ? I.s : I.amgX + M.lev[l].vecOff;
}
__device__ __forceinline__ double *lev_b(DevInst &I, const DevMesh &M, int l) {
    return l == 0 ? I.r : I.amgB + M.lev[l].vecOff;
}
__device__ __forceinline__ double *lev_r(DevInst &I, const DevMesh &M, int l) {
    return l == 0 ? I.t : I.amgR + M.lev[l].vecOff;
}
// Gauss-Seidel reciprocal diagonals: level 0 at [0, nC), level l at nC + vecOff
__device__ __forceinline__ double *lev_rd(DevInst &I, const DevMesh &M, int l) {
    return l == 0 ? I.amgRd : I.amgRd + M.nC + M.lev[l].vecOff;
}

// numeric Galerkin update of level l from level l-1 (fixed gather order)
template <class T>
__device__ void amg_galerkin(T &tm, const DevMesh &M, DevInst &I, int l) {
    const AmgLevelDev &L = M.lev[l];
    const double *fine = lev_vals(I, M, l - 1);
    double *val = lev_vals(I, M, l);
    for (int k = tm.spread(); k < L.nnz; k += tm.size()) {
        double s = 0.0;
        for (int q = L.gOff[k]; q < L.gOff[k + 1]; ++q) s += LD(fine + L.gIdx[q]);
        val[k] = s;
    }
}

// reciprocal diagonals of level l (after its values are final)
template <class T>
__device__ void amg_level_rd(T &tm, const DevMesh &M, DevInst &I, int l) {
    const AmgLevelDev &L = M.lev[l];
    double *rd = lev_rd(I, M, l);
    const double *val = lev_vals(I, M, l);
    for (int i = tm.spread(); i < L.n; i += tm.size()) {
        double d;
        if (l == 0) d = LD(I.diag + i);
        else d = L.diagPos[i] >= 0 ? LD(val + L.diagPos[i]) : 0.0;
        rd[i] = gs_rd(d);
    }
}

// Dense inverse of the coarsest level (Galerkin product of the pinned /
// Dirichlet-bounded pressure Laplacian: SPD).  A matrix with a vanishing pivot
// is no such product; its rows are passed over one by one, which needs the
// sweep over all 2n columns with ping-pong buffers.
template <class T>
__device__ __noinline__ void amg_coarse_inverse_sweep(T &tm, const DevMesh &M, DevInst &I) {
    const int l = M.nLevels - 1;
    const AmgLevelDev &L = M.lev[l];
    const int n = L.n, w2 = 2 * n;
    double *A = I.gj, *B = I.gj + (size_t)n * w2;
    const double *val = lev_vals(I, M, l);
    for (int i = tm.spread(); i < n; i += tm.size()) {
        double *row = A + (size_t)i * w2;
        for (int j = 0; j < w2; ++j) row[j] = 0.0;
        if (l == 0) {
            row[i] = LD(I.diag + i);  // level 0 as coarsest: LDU rows
            for (int e = M.cfOff[i]; e < M.cfOff[i + 1]; ++e) {
                const int f = M.cfFace[e], oth = M.cfOther[e];
                if (oth >= 0) row[oth] = LD(I.upper + f);
                else row[-(oth + 1)] = LD(I.lower + f);
            }
        } else {
            for (int q = L.rowPtr[i]; q < L.rowPtr[i + 1]; ++q) row[L.colIdx[q]] = LD(val + q);
        }
        row[n + i] = 1.0;
    }
    tm.sync();
    for (int k = 0; k < n; ++k) {
        const double piv = LD(A + (size_t)k * w2 + k);
        const bool skip = !(fabs(piv) > 1e-300);
        const double rp = skip ? 0.0 : 1.0 / piv;
        for (int idx = tm.spread(); idx < n * w2; idx += tm.size()) {
            const int i = idx / w2, j = idx - i * w2;
            const double akj = LD(A + (size_t)k * w2 + j) * rp;
            double v = LD(A + idx);
            if (!skip) {
                if (i == k) v = akj;
                else v = fma(-LD(A + (size_t)i * w2 + k), akj, v);
            }
            B[idx] = v;
        }
        tm.sync();
        double *tmp = A; A = B; B = tmp;
    }
    for (int idx = tm.spread(); idx < n * n; idx += tm.size()) {
        const int i = idx / n, j = idx - i * n;
        I.ainv[idx] = LD(A + (size_t)i * w2 + n + j);
    }
    tm.sync();
}

template <class T>
__device__ __noinline__ void amg_coarse_inverse(T &tm, const DevMesh &M, DevInst &I) {
    const int l = M.nLevels - 1, n = M.lev[l].n;
    const AmgLevelDev &L = M.lev[l];
    double *A = I.ainv;
    const double *val = lev_vals(I, M, l);
    // a large mesh's level on one CTA (the phase test hook)
    if (!std::is_same<T, GridTeam>::value && n > kCoarseDirect) {
        amg_coarse_inverse_sweep(tm, M, I);
        return;
    }
    for (int idx = tm.spread(); idx < n * n; idx += tm.size()) A[idx] = 0.0;
    tm.sync();
    for (int i = tm.spread(); i < n; i += tm.size()) {
        double *row = A + (size_t)i * n;
        if (l == 0) {
            row[i] = LD(I.diag + i);  // level 0 as coarsest: LDU rows
            for (int e = M.cfOff[i]; e < M.cfOff[i + 1]; ++e) {
                const int f = M.cfFace[e], oth = M.cfOther[e];
                if (oth >= 0) row[oth] = LD(I.upper + f);
                else row[-(oth + 1)] = LD(I.lower + f);
            }
        } else {
            for (int q = L.rowPtr[i]; q < L.rowPtr[i + 1]; ++q) row[L.colIdx[q]] = LD(val + q);
        }
    }
    tm.sync();
    if (!dense_inverse(tm, A, I.gj, n)) {
        tm.sync();
        amg_coarse_inverse_sweep(tm, M, I);
    }
}

// the arrays of an instance for the V-cycle (btm_cycle.cuh)
struct Cycle64 {
    using V = double;
    static constexpr double kWeight = 0.7;
    const DevMesh &M;
    DevInst &I;
    __device__ __forceinline__ int levels() const { return M.nLevels; }
    __device__ __forceinline__ bool direct() const { return M.coarseDirect != 0; }
    __device__ __forceinline__ const AmgLevelDev &lev(int l) const { return M.lev[l]; }
    __device__ __forceinline__ RowTab rows() const { return RowTab(M); }
    __device__ __forceinline__ double *x(int l) const { return lev_x(I, M, l); }
    __device__ __forceinline__ double *b(int l) const { return lev_b(I, M, l); }
    __device__ __forceinline__ double *r(int l) const { return lev_r(I, M, l); }
    __device__ __forceinline__ double *rd(int l) const { return lev_rd(I, M, l); }
    __device__ __forceinline__ double *val(int l) const { return lev_vals(I, M, l); }
    __device__ __forceinline__ const double *sys() const { return I.diag; }
    __device__ __forceinline__ const double *ainv() const { return I.ainv; }
};

// one colour-ordered Gauss-Seidel sweep (forward or reverse colour order)
template <class T, int W>
__device__ __noinline__ void amg_gs_rows(T &tm, const DevMesh &M, DevInst &I, int l, bool reverse) {
    // (locals: the descriptors are in shared memory, and every store has them read again)
    const CsrTab L(M.lev[l]);
    const RowTab R(M);
    double *x = lev_x(I, M, l);
    const double *b = lev_b(I, M, l);
    const double *val = lev_vals(I, M, l);
    const double *rd = lev_rd(I, M, l);
    const int32_t *off = M.lev[l].colorOff, *rows = M.lev[l].colorRows;
    const int nColors = M.lev[l].nColors;
    for (int cc = 0; cc < nColors; ++cc) {
        const int col = reverse ? nColors - 1 - cc : cc;
        const int q1 = off[col + 1];
        for (int q = off[col] + tm.rank(); q < q1; q += tm.size()) {
            const int i = rows[q];
            const double ri = LD(rd + i);
            if (!nonzero64(ri)) continue;
            double s = LD(b + i);
            if constexpr (W == 0) s = ldu_off<T, true>(R, val, (const double *)x, i, s);
            else s = csr_off<T, true, W>(L, val, (const double *)x, i, i, s);
            x[i] = s * ri;
        }
        tm.sync();
    }
}

// (W entries of a row at a time, as the level's longest row needs: levels of
// structured meshes have rows of 5, whose sweeps are a tenth faster than with 8)
template <class T>
__device__ void amg_gs_sweep(T &tm, const DevMesh &M, DevInst &I, int l, bool reverse) {
    const int widest = M.lev[l].widest;
    if (l == 0) amg_gs_rows<T, 0>(tm, M, I, l, reverse);
    else if (widest <= 5) amg_gs_rows<T, 5>(tm, M, I, l, reverse);
    else if (widest <= 6) amg_gs_rows<T, 6>(tm, M, I, l, reverse);
    else amg_gs_rows<T, 8>(tm, M, I, l, reverse);
}

// residual of level l and restriction into level l+1 (x_{l+1} = 0)
template <class T>
__device__ __noinline__ void amg_restrict(T &tm, const DevMesh &M, DevInst &I, int l) {
    const AmgLevelDev &L = M.lev[l];
    const double *x = lev_x(I, M, l), *b = lev_b(I, M, l), *val = lev_vals(I, M, l);
    double *r = lev_r(I, M, l);
    for (int i = tm.spread(); i < L.n; i += tm.size()) {
        double s;
        if (l == 0) {
            s = ldu_row<T>(M, I, x, i);
        } else {
            s = csr_off<T, false>(L, val, x, i, -1, 0.0);
        }
        r[i] = LD(b + i) - s;
    }
    tm.sync();
    const AmgLevelDev &C = M.lev[l + 1];
    double *bc = lev_b(I, M, l + 1), *xc = lev_x(I, M, l + 1);
    for (int J = tm.spread(); J < C.n; J += tm.size()) {
        double s = 0.0;
        for (int q = L.aggOff[J]; q < L.aggOff[J + 1]; ++q) s += LD(r + L.aggMem[q]);
        bc[J] = s;
        xc[J] = 0.0;
    }
    tm.sync();
}

template <class T>
__device__ void amg_prolong(T &tm, const DevMesh &M, DevInst &I, int l) {
    const AmgLevelDev &L = M.lev[l];
    double *x = lev_x(I, M, l);
    const double *xc = lev_x(I, M, l + 1);
    for (int i = tm.spread(); i < L.n; i += tm.size()) x[i] = LD(x + i) + LD(xc + L.map[i]);
    tm.sync();
}

template <class T>
__device__ void amg_coarse_solve(T &tm, const DevMesh &M, DevInst &I) {
    const int l = M.nLevels - 1;
    const int n = M.lev[l].n;
    if (M.coarseDirect) {
        const double *b = lev_b(I, M, l);
        double *x = lev_x(I, M, l);
        for (int i = tm.rank(); i < n; i += tm.size()) {
            double s = 0.0;
            for (int j = 0; j < n; ++j) s = fma(LD(I.ainv + (size_t)i * n + j), LD(b + j), s);
            x[i] = s;
        }
        tm.sync();
    } else {
        for (int s = 0; s < kCoarseSweeps; ++s) amg_gs_sweep(tm, M, I, l, (s & 1) != 0);
    }
}

// V-cycle on all levels, on one CTA (L1 keeps the rows there, and passes that
// fetch ahead of their barrier measured 20 % slower: the grid's are in
// btm_cycle.cuh): 2 pre-sweeps (colours ascending), 2 post sweeps
// (colours descending), symmetric so the preconditioner suits CG.
template <class T>
__device__ void amg_vcycle_gs(T &tm, const DevMesh &M, DevInst &I) {
    const int nl = M.nLevels;
    for (int l = 0; l < nl - 1; ++l) {
        amg_gs_sweep(tm, M, I, l, false);
        amg_gs_sweep(tm, M, I, l, false);
        amg_restrict(tm, M, I, l);
    }
    amg_coarse_solve(tm, M, I);
    for (int l = nl - 2; l >= 0; --l) {
        amg_prolong(tm, M, I, l);
        amg_gs_sweep(tm, M, I, l, true);
        amg_gs_sweep(tm, M, I, l, true);
    }
}

// Hierarchy refresh and V-cycle, the same on one CTA and on the cooperative
// grid (every level on the whole team; the grid's dense coarsest level has
// up to kCoarseDirectGrid rows and is inverted and applied by all CTAs).
template <class T> struct AmgDriver {
    __device__ static void setup(T &tm, const DevMesh &M, DevInst &I) {
        amg_level_rd(tm, M, I, 0);
        for (int l = 1; l < M.nLevels; ++l) {
            amg_galerkin(tm, M, I, l);
            tm.sync();
            amg_level_rd(tm, M, I, l);
        }
        tm.sync();
        if (M.coarseDirect) amg_coarse_inverse(tm, M, I);
    }
    __device__ static void vcycle(T &tm, const DevMesh &M, DevInst &I) {
        if constexpr (std::is_same<T, GridTeam>::value) Cycle<T, Cycle64>::run(tm, Cycle64{M, I});
        else amg_vcycle_gs(tm, M, I);
    }
};

// What the CG solvers take from the first squared residual norm: the norm,
// whether there is nothing to solve, and the limit of their stopping test.
__device__ __forceinline__ double cg_start(int lane, double rr, double tol) {
    const double r0 = sqrt(rr);
    const double limit = residual_limit(r0, tol);
    return pick(lane, r0, flag64(r0 < 1e-30), limit);
}

// AMGSolver::solve (LinearSolver.hpp:602-653) with the reference's own
// hierarchy rebuilt from this system (btm_ramg.cuh); one CTA.  r = I.r,
// z = I.s (the V-cycle's level-0 x), p = I.pv, Ap = I.v, level-0 residual I.t.
__device__ __noinline__ SolveResult team_ramg_pcg(BlockTeamRef &tm, const DevMesh &M, DevInst &I, double *x,
                                                  int maxIter, double tol) {
    SolveResult res = {0, 0.0, 0.0, 0};
    const int nC = M.nC;
    const uint64_t t0 = tm.leader() ? globaltimer_ns() : 0;
    const int nLev = ramg_setup(tm, M, I, x != I.pp);
    if (tm.leader()) I.rg.setupNs += globaltimer_ns() - t0;
    double a0[1] = {0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        const double rc = I.src[c] - ldu_row<BlockTeamRef>(M, I, x, c);
        I.r[c] = rc;
        I.s[c] = 0.0;
        a0[0] = fma(rc, rc, a0[0]);
    }
    double o[3];
    tm.template sum_then<1, 3>(a0, o, [tol](int lane, double rr, double) { return cg_start(lane, rr, tol); });
    const double r0 = o[0], limit = o[2];
    res.initialRes = r0;
    if (is_set(o[1])) { res.converged = 1; return res; }
    ramg_precondition(tm, M, I, nLev);
    double a1[1] = {0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        const double z = I.s[c];
        I.pv[c] = z;
        a1[0] = fma(I.r[c], z, a1[0]);
    }
    tm.template sum<1>(a1);
    double rz = a1[0];
    for (int it = 0; it < maxIter; ++it) {
        double a2[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            const double ap = ldu_row<BlockTeamRef>(M, I, I.pv, c);
            I.v[c] = ap;
            a2[0] = fma(I.pv[c], ap, a2[0]);
        }
        tm.template sum_then<1, 2>(a2, o, [rz](int lane, double pAp, double) {
            return pick(lane, flag64(fabs(pAp) < 1e-30), rz / pAp);
        });
        if (is_set(o[0])) break;
        const double alpha = o[1];
        double a3[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            x[c] = x[c] + alpha * I.pv[c];
            const double rc = I.r[c] - alpha * I.v[c];
            I.r[c] = rc;
            I.s[c] = 0.0;
            a3[0] = fma(rc, rc, a3[0]);
        }
        tm.template sum_then<1, 2>(a3, o, [=](int lane, double rr, double) {
            return pick(lane, rr, flag64(residual_below(rr, limit, r0, tol)));
        });
        res.iterations = it + 1;
        res.finalSq = o[0];
        if (is_set(o[1])) { res.converged = 1; return res; }
        ramg_precondition(tm, M, I, nLev);
        double a4[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) a4[0] = fma(I.r[c], I.s[c], a4[0]);
        tm.template sum_then<1, 2>(a4, o, [rz](int lane, double t, double) { return pick(lane, t, t / (rz + 1e-30)); });
        const double rzNew = o[0], beta = o[1];
        for (int c = tm.rank(); c < nC; c += tm.size()) I.pv[c] = I.s[c] + beta * I.pv[c];
        tm.sync();
        rz = rzNew;
    }
    return res;
}

// The reference-order AMG runs in the kernel instantiated for BlockTeamRef
// only (one CTA per instance); the other teams keep the per-case hierarchy.
template <class T> struct RefAmg {
    __device__ static bool on(const DevInst &) { return false; }
    __device__ static SolveResult run(T &, const DevMesh &, DevInst &, double *, int, double) {
        return {0, 0.0, 0.0, 0};
    }
};
template <> struct RefAmg<BlockTeamRef> {
    __device__ static bool on(const DevInst &I) { return I.S.refAmg != 0; }
    __device__ static SolveResult run(BlockTeamRef &tm, const DevMesh &M, DevInst &I, double *x, int maxIter,
                                      double tol) {
        return team_ramg_pcg(tm, M, I, x, maxIter, tol);
    }
};

// AMG-preconditioned CG (AMGSolver::solve, LinearSolver.hpp:602-653) on
// (I.diag, I.upper, I.lower, I.src), x in place (the pressure correction
// starts from zero).  Vectors: r = I.r, z = I.s (V-cycle level-0 x),
// p = I.pv, Ap = I.v, V-cycle scratch I.t.
template <class T>
__device__ __noinline__ SolveResult team_amg_pcg(T &tm, const DevMesh &M, DevInst &I, double *x, int maxIter, double tol) {
    if (RefAmg<T>::on(I)) return RefAmg<T>::run(tm, M, I, x, maxIter, tol);
    SolveResult res = {0, 0.0, 0.0, 0};
    const int nC = M.nC;
    AmgDriver<T>::setup(tm, M, I);
    double a0[1] = {0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        double rc = LD(I.src + c) - ldu_row<T>(M, I, x, c);
        I.r[c] = rc;
        I.s[c] = 0.0;
        a0[0] = fma(rc, rc, a0[0]);
    }
    double o[3];
    tm.template sum_then<1, 3>(a0, o, [tol](int lane, double rr, double) { return cg_start(lane, rr, tol); });
    const double r0 = o[0], limit = o[2];
    res.initialRes = r0;
    if (is_set(o[1])) { res.converged = 1; return res; }
    // The reference's breakdown guards (|p.Ap| < 1e-30, rz + 1e-30) are
    // absolute.  On grid meshes (above the one-CTA size) they are applied as
    // if the system had been scaled to a unit-norm right-hand side, as the
    // mixed engine scales it: the p' coefficients of the 2M-cell duct are so
    // small that the absolute guard ended the CG after about 0.6 iterations
    // per outer iteration.  One-CTA meshes (every parity case) keep the
    // reference's absolute guards.
    const double guard = std::is_same<T, GridTeam>::value ? 1e-30 * r0 * r0 : 1e-30;
    AmgDriver<T>::vcycle(tm, M, I);
    double a1[1] = {0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        double z = LD(I.s + c);
        I.pv[c] = z;
        a1[0] = fma(LD(I.r + c), z, a1[0]);
    }
    tm.template sum<1>(a1);
    double rz = a1[0];
    for (int it = 0; it < maxIter; ++it) {
        if (!tm.ok()) break;
        double a2[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            double ap = ldu_row<T>(M, I, I.pv, c);
            I.v[c] = ap;
            a2[0] = fma(LD(I.pv + c), ap, a2[0]);
        }
        tm.template sum_then<1, 2>(a2, o, [rz, guard](int lane, double pAp, double) {
            return pick(lane, flag64(fabs(pAp) < guard), rz / pAp);
        });
        if (is_set(o[0])) break;
        const double alpha = o[1];
        double a3[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            x[c] = fma(alpha, LD(I.pv + c), LD(x + c));
            double rc = fma(-alpha, LD(I.v + c), LD(I.r + c));
            I.r[c] = rc;
            I.s[c] = 0.0;
            a3[0] = fma(rc, rc, a3[0]);
        }
        tm.template sum_then<1, 2>(a3, o, [=](int lane, double rr, double) {
            return pick(lane, rr, flag64(residual_below(rr, limit, r0, tol)));
        });
        res.iterations = it + 1;
        res.finalSq = o[0];
        if (is_set(o[1])) { res.converged = 1; return res; }
        AmgDriver<T>::vcycle(tm, M, I);
        double a4[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) a4[0] = fma(LD(I.r + c), LD(I.s + c), a4[0]);
        tm.template sum_then<1, 2>(a4, o, [rz, guard](int lane, double t, double) {
            return pick(lane, t, t / (rz + guard));
        });
        const double rzNew = o[0], beta = o[1];
        for (int c = tm.rank(); c < nC; c += tm.size()) I.pv[c] = fma(beta, LD(I.pv + c), LD(I.s + c));
        tm.sync();
        rz = rzNew;
    }
    return res;
}

// Jacobi-preconditioned CG (PCGSolver::solve, LinearSolver.hpp:147-186) on
// (I.diag, I.upper, I.lower, I.src); x in place.  r = I.r, z = I.s, p = I.pv, Ap = I.v.
template <class T>
__device__ __noinline__ SolveResult team_pcg(T &tm, const DevMesh &M, DevInst &I, double *x, int maxIter, double tol) {
    SolveResult res = {0, 0.0, 0.0, 0};
    const int nC = M.nC;
    double a0[2] = {0.0, 0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        double rc = LD(I.src + c) - ldu_row<T>(M, I, x, c);
        double rdc = jac_rd(LD(I.diag + c));
        double z = rc * rdc;
        I.rd[c] = rdc;
        I.r[c] = rc; I.s[c] = z; I.pv[c] = z;
        a0[0] = fma(rc, rc, a0[0]);
        a0[1] = fma(rc, z, a0[1]);
    }
    double o[4];
    tm.template sum_then<2, 4>(a0, o, [tol](int lane, double rr, double t) {
        const double start = cg_start(lane, rr, tol);
        return lane == 3 ? t : start;
    });
    const double r0 = o[0], limit = o[2];
    res.initialRes = r0;
    if (is_set(o[1])) { res.converged = 1; return res; }
    double rz = o[3];
    for (int it = 0; it < maxIter; ++it) {
        if (!tm.ok()) break;
        double a2[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            double ap = ldu_row<T>(M, I, I.pv, c);
            I.v[c] = ap;
            a2[0] = fma(LD(I.pv + c), ap, a2[0]);
        }
        tm.template sum_then<1, 2>(a2, o, [rz](int lane, double pAp, double) {
            return pick(lane, flag64(fabs(pAp) < 1e-30), rz / pAp);
        });
        if (is_set(o[0])) break;
        const double alpha = o[1];
        double a3[2] = {0.0, 0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            x[c] = fma(alpha, LD(I.pv + c), LD(x + c));
            double rc = fma(-alpha, LD(I.v + c), LD(I.r + c));
            double z = rc * LD(I.rd + c);
            I.r[c] = rc;
            I.s[c] = z;
            a3[0] = fma(rc, rc, a3[0]);
            a3[1] = fma(rc, z, a3[1]);
        }
        tm.template sum_then<2, 4>(a3, o, [=](int lane, double rr, double t) {
            const double beta = t / (rz + 1e-30);
            return lane == 3 ? t : pick(lane, rr, flag64(residual_below(rr, limit, r0, tol)), beta);
        });
        res.iterations = it + 1;
        res.finalSq = o[0];
        if (is_set(o[1])) { res.converged = 1; return res; }
        const double beta = o[2];
        for (int c = tm.rank(); c < nC; c += tm.size()) I.pv[c] = fma(beta, LD(I.pv + c), LD(I.s + c));
        tm.sync();
        rz = o[3];
    }
    return res;
}

// GaussSeidelSolver::solve (LinearSolver.hpp:258-299) on (I.diag, I.upper,
// I.lower, I.src), x in place: in-place sweeps in row order, each row summing
// its neighbours in face order with the latest values, then a residual check
// against |source|.  A sweep runs wavefront by wavefront over the level-0
// row-order dependencies (M.wf0Off / M.wf0Rows): a row reads the new values
// of its lower-index neighbours and the old values of the others, exactly as
// the sequential sweep, with the reference's operation order per row.  Only
// the residual norm (a parallel reduction) differs in the last bits.
template <class T>
__device__ __noinline__ SolveResult team_gauss_seidel(T &tm, const DevMesh &M, DevInst &I, double *x, int maxIter,
                                                      double tol) {
    SolveResult res = {0, 0.0, 0.0, 0};
    const int nC = M.nC;
    double a0[1] = {0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        const double bc = LD(I.src + c);
        a0[0] = fma(bc, bc, a0[0]);
    }
    tm.template sum<1>(a0);
    double b0 = sqrt(a0[0]);
    res.initialRes = b0;
    if (b0 < 1e-30) b0 = 1.0;
    for (int it = 0; it < maxIter; ++it) {
        if (!tm.ok()) break;
        for (int w = 0; w < M.nWf0; ++w) {
            for (int q = M.wf0Off[w] + tm.rank(); q < M.wf0Off[w + 1]; q += tm.size()) {
                const int i = M.wf0Rows[q];
                const double d = LD(I.diag + i);
                if (fabs(d) <= 1e-30) continue;
                double sacc = LD(I.src + i);
                for (int e = M.cfOff[i]; e < M.cfOff[i + 1]; ++e) {
                    const int f = M.cfFace[e], oth = M.cfOther[e];
                    if (oth >= 0) sacc -= LD(I.upper + f) * LD(x + oth);
                    else sacc -= LD(I.lower + f) * LD(x + (-(oth + 1)));
                }
                x[i] = sacc / d;
            }
            tm.sync();
        }
        double a1[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            const double rc = LD(I.src + c) - ldu_row<T>(M, I, x, c);
            a1[0] = fma(rc, rc, a1[0]);
        }
        tm.template sum<1>(a1);
        res.iterations = it + 1;
        res.finalSq = a1[0];
        if (sqrt(a1[0]) / b0 < tol) { res.converged = 1; return res; }
    }
    return res;
}

// makeSolver semantics for the device (LinearSolver.hpp:659-665): AMG and
// PCG run the CG family, GaussSeidel the in-place sweep; every other name
// runs BiCGSTAB.
template <class T>
__device__ SolveResult team_solve(T &tm, const DevMesh &M, DevInst &I, int kind, double *x, int maxIter, double tol) {
    if (kind == 3) return team_amg_pcg(tm, M, I, x, maxIter, tol);
    if (kind == 0) return team_pcg(tm, M, I, x, maxIter, tol);
    if (kind == 2) return team_gauss_seidel(tm, M, I, x, maxIter, tol);
    return team_bicgstab(tm, M, I, x, maxIter, tol);
}

// ---------------------------------------------------------------------------
// initUniform (SIMPLESolver.cpp:23-51)
// ---------------------------------------------------------------------------
template <class T>
__device__ void phase_init_uniform(T &tm, const DevMesh &M, DevInst &I) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double U0 = I.init[0], U1 = I.init[1], U2 = I.init[2], p0 = I.init[3], k0 = I.init[4], w0 = I.init[5];
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        I.ux[c] = U0; I.uy[c] = U1; I.uz[c] = U2; I.p[c] = p0; I.k[c] = k0;
        I.f1[c] = 1.0; I.f2[c] = 1.0; I.pk[c] = 0.0; I.cdkw[c] = 0.0;
        double y = smax(M.wd[c], 1e-20);
        double omWall = 60.0 * nu / (cf.b1 * y * y);
        double om = smax(omWall, w0);
        I.om[c] = om;
        I.nut[c] = cf.a1 * k0 / smax(cf.a1 * om, 1e-20);
    }
    for (int b = tm.rank(); b < M.nB; b += tm.size()) {
        I.ubx[b] = U0; I.uby[b] = U1; I.ubz[b] = U2; I.pb[b] = p0; I.kb[b] = k0; I.omb[b] = w0;
    }
    tm.sync();
    phase_bc_u(tm, M, I);
    phase_bc_p(tm, M, I);
    phase_bc_k(tm, M, I, false);
    phase_bc_w(tm, M, I, 0.075, false);  // applyAllBCs uses applyOmegaBC's default beta1
    tm.sync();
}

// ---------------------------------------------------------------------------
// the SIMPLE outer loop (SIMPLESolver::solve, SIMPLESolver.cpp:696-1043)
// ---------------------------------------------------------------------------
template <class T>
__device__ void simple_solve(T &tm, const DevMesh &M, DevInst &I) {
    const DevSettings &S = I.S;
    const Coef cf = load_coef(I);
    const int nC = M.nC, nB = M.nB;
    const double nu = I.nu;
    if (I.initMode == 0) phase_init_uniform(tm, M, I);
    int turbEst = I.initMode == 0 ? 0 : I.turbEstIn;
    double lastKChange = 1.0, lastOmChange = 1.0;
    double normUx0 = 1, normUy0 = 1, normP0 = 1;
    int converged = 0, diverged = 0, finalIter = S.maxIter, ran = 0;
    int64_t inner = 0, innerMom = 0, innerP = 0, innerTurb = 0;
    double last[6] = {0, 0, 0, 0, 0, 0};
    const bool turbScheduled = S.turbStart < S.maxIter;
    PhaseClock clk;
    clk.start(tm.leader());
    const uint64_t tStart = tm.leader() ? globaltimer_ns() : 0;
    if (tm.leader()) I.rg.setupNs = 0;
    const bool d2 = M.is2d && !I.solveZ;   // no z normals, no z velocity
    // the momentum diffusion coefficients fit kold | omold (adjacent, idle until
    // the turbulence equations) on meshes of quadrilaterals
    double *keepD = (I.omold + nC) - I.kold >= M.nIF ? I.kold : nullptr;
    if (d2) {
        phase_grad_init(tm, M, I);
        tm.sync();
    }

    for (int iter = 0; iter < S.maxIter; ++iter) {
        if (!tm.ok()) break;
        ran = iter + 1;
        const bool turbActive = iter >= S.turbStart;
        const bool turbUpdate = turbActive && ((iter - S.turbStart) % S.turbInterval == 0);
        // 1. turbulence closure fields at the start-of-iteration U
        // (the injection source also reads the z gradients, which the packed rows
        // of the reference-order AMG may have replaced)
        if (d2 && I.inj) phase_grad_init(tm, M, I);
        if (d2) phase_grads<T, true>(tm, M, I, 15);
        else phase_grads<T, false>(tm, M, I, 15);
        tm.sync();
        if (turbUpdate) {
            if (!turbEst && iter >= S.turbStart + S.nutFloorIters) turbEst = 1;
            const double nutMin = turbEst ? 0.0 : 0.1 * nu;
            if (d2) phase_closure<T, true>(tm, M, I, nutMin);
            else phase_closure<T, false>(tm, M, I, nutMin);
            tm.sync();
        }
        clk.lap(0);
        // 2. momentum, component by component with the latest U
        SolveResult resU[3];
        resU[2].initialRes = 0.0; resU[2].iterations = 0;
        for (int comp = 0; comp < 3; ++comp) {
            if (comp == 2 && !I.solveZ) break;
            if (comp > 0) {
                if (d2) phase_grads<T, true>(tm, M, I, 1 << (comp - 1));
                else phase_grads<T, false>(tm, M, I, 1 << (comp - 1));
                tm.sync();
            }
            if (comp == 0 && I.inj) phase_inj(tm, M, I, I.g, I.nut, iter == 0);
            if (d2) phase_momq_faces<T, true>(tm, M, I, comp, comp == 0, keepD);
            else phase_momq_faces<T, false>(tm, M, I, comp, comp == 0, keepD);
            tm.sync();
            phase_momq_cells(tm, M, I, comp);
            tm.sync();
            clk.lap(1);
            double *x = comp == 0 ? I.ux : (comp == 1 ? I.uy : I.uz);
            resU[comp] = team_solve(tm, M, I, S.momSolver, x, S.innerIter, S.innerTol);
            innerMom += resU[comp].iterations;
            tm.sync();
            clk.lap(2);
        }
        phase_bc_u(tm, M, I);
        phase_dp(tm, M, I);
        tm.sync();
        // 3. pressure correction
        if (d2) phase_pq_faces<T, true>(tm, M, I);
        else phase_pq_faces<T, false>(tm, M, I);
        tm.sync();
        phase_pq_cells(tm, M, I);
        tm.sync();
        clk.lap(3);
        SolveResult resP = team_solve(tm, M, I, S.pSolver, I.pp, S.innerIter, S.innerTol);
        innerP += resP.iterations;
        tm.sync();
        clk.lap(5);
        for (int b = tm.rank(); b < nB; b += tm.size()) I.ppb[b] = M.bcPp[b] == 0 ? LD(I.pp + M.bown[b]) : 0.0;
        tm.sync();
        // 4. corrections (correctVelocity / correctPressure, SIMPLESolver.cpp:456-475)
        {
            const double *P[1] = {I.pp};
            const double *PB[1] = {I.ppb};
            const double alphaP = S.alphaP;
            for (int c = tm.rank(); c < nC; c += tm.size()) {
                double gx[1], gy[1], gz[1];
                if (d2) gq_cell<T, 1, true>(M, c, P, PB, gx, gy, gz);
                else gq_cell<T, 1, false>(M, c, P, PB, gx, gy, gz);
                const double aP = LD(I.aPx + c);
                double rAP = (fabs(aP) > 1e-30) ? 1.0 / aP : 0.0;
                double vol = M.vol[c];
                I.ux[c] = LD(I.ux + c) - rAP * gx[0] * vol;
                I.uy[c] = LD(I.uy + c) - rAP * gy[0] * vol;
                if (!d2) I.uz[c] = LD(I.uz + c) - rAP * gz[0] * vol;
                I.p[c] = LD(I.p + c) + alphaP * LD(I.pp + c);
            }
            tm.sync();
            phase_bc_u(tm, M, I);
            phase_bc_p(tm, M, I);
            tm.sync();
        }
        clk.lap(6);
        // 5. k and omega
        SolveResult resK = {0, 0, 0, 0}, resW = {0, 0, 0, 0};
        double change[4];   // largest k and omega, largest change of k and of omega
        if (turbUpdate) {
            for (int c = tm.rank(); c < nC; c += tm.size()) { I.kold[c] = LD(I.k + c); I.omold[c] = LD(I.om + c); }
            if (d2) phase_turbq_faces<T, true>(tm, M, I, 0, true);
            else phase_turbq_faces<T, false>(tm, M, I, 0, true);
            tm.sync();
            phase_turbq_cells(tm, M, I, 0);
            tm.sync();
            resK = team_solve(tm, M, I, S.turbSolver, I.k, S.innerIter, S.innerTol);
            innerTurb += resK.iterations;
            tm.sync();
            for (int c = tm.rank(); c < nC; c += tm.size()) I.k[c] = smax(S.kMin, smin(S.kMax, LD(I.k + c)));
            tm.sync();
            phase_bc_k(tm, M, I, true);
            tm.sync();
            if (d2) phase_turbq_faces<T, true>(tm, M, I, 1, false);
            else phase_turbq_faces<T, false>(tm, M, I, 1, false);
            tm.sync();
            phase_turbq_cells(tm, M, I, 1);
            tm.sync();
            resW = team_solve(tm, M, I, S.turbSolver, I.om, S.innerIter, S.innerTol);
            innerTurb += resW.iterations;
            tm.sync();
            for (int c = tm.rank(); c < nC; c += tm.size()) I.om[c] = smax(S.omegaMin, smin(1e15, LD(I.om + c)));
            tm.sync();
            phase_bc_w(tm, M, I, cf.b1, true);
            tm.sync();
            // wall re-pin (SIMPLESolver.cpp:884-908) and change norms (:910-922)
            double mx[4] = {1e-30, 1e-30, 0.0, 0.0};
            const double sbs = sqrt(cf.bstar);
            for (int c = tm.rank(); c < nC; c += tm.size()) {
                const int b = M.pinFace[c];
                double omc = LD(I.om + c);
                if (b >= 0) {
                    double y1 = M.bdeltaW[b];
                    double omRes = 60.0 * nu / (cf.b1 * y1 * y1);
                    if (S.useWallFn) {
                        double k_p = smax(LD(I.k + c), 1e-30);
                        double uTau = sqrt(sbs * k_p);
                        double omLog = uTau / (sbs * S.vonKarman * y1);
                        omc = sqrt(omRes * omRes + omLog * omLog);
                    } else {
                        omc = omRes;
                    }
                    I.om[c] = omc;
                }
                const double kc = LD(I.k + c);
                mx[0] = smax(mx[0], fabs(kc));
                mx[1] = smax(mx[1], fabs(omc));
                mx[2] = smax(mx[2], fabs(kc - LD(I.kold + c)));
                mx[3] = smax(mx[3], fabs(omc - LD(I.omold + c)));
            }
            tm.template maxr<4>(mx);
            for (int q = 0; q < 4; ++q) change[q] = mx[q];
        }
        clk.lap(7);
        // 6. residual bookkeeping and the convergence / divergence tests, by
        // one warp (the quotients side by side in its lanes): lastKChange,
        // lastOmChange, and how the iteration ends (0: on, 1: converged, 2: diverged)
        const double eUx = resU[0].initialRes, eUy = resU[1].initialRes, eUz = resU[2].initialRes;
        const double eP = resP.initialRes;
        if (I.normFixed) {
            normUx0 = I.normIn[0];
            normUy0 = I.normIn[1];
            normP0 = I.normIn[2];
        } else if (iter == 0) {
            normUx0 = smax(eUx, 1e-30);
            normUy0 = smax(eUy, 1e-30);
            normP0 = smax(eP, 1e-30);
        } else if (iter < 50) {
            normP0 = smax(normP0, eP);
        }
        double end[3];
        tm.template once<3>(end, [&](int lane) {
            const double normMom0 = smax(normUx0, normUy0);
            const double num = lane == 0 ? eUx : lane == 1 ? eUy : lane == 2 ? eP : change[lane == 3 ? 2 : 3];
            const double den = lane < 2 ? normMom0 : lane == 2 ? normP0 : change[lane == 3 ? 0 : 1];
            double q = num / den;
            if (lane < 3 && den < 1e-20) q = 0.0;
            const double nUx = __shfl_sync(0xffffffffu, q, 0), nUy = __shfl_sync(0xffffffffu, q, 1),
                         nP = __shfl_sync(0xffffffffu, q, 2), qK = __shfl_sync(0xffffffffu, q, 3),
                         qW = __shfl_sync(0xffffffffu, q, 4);
            const double dK = turbUpdate ? qK : lastKChange, dW = turbUpdate ? qW : lastOmChange;
            double maxRes = smax(smax(nUx, nUy), nP);
            if (turbActive) maxRes = smax(smax(maxRes, dK), dW);
            if (!isfinite(eUx) || !isfinite(eUy) || !isfinite(eUz) || !isfinite(eP) || !isfinite(dK) || !isfinite(dW))
                maxRes = INFINITY;
            double how = 0.0;
            if (maxRes < S.convTol && iter > 0 && (!turbScheduled || (turbActive && turbEst))) how = 1.0;
            else if (isnan(maxRes) || isinf(maxRes) || maxRes > S.divLimit) how = 2.0;
            return pick(lane, dK, dW, how);
        });
        lastKChange = end[0];
        lastOmChange = end[1];
        const double eK = turbActive ? lastKChange : 0.0, eW = turbActive ? lastOmChange : 0.0;
        last[0] = eUx; last[1] = eUy; last[2] = eUz; last[3] = eP; last[4] = eK; last[5] = eW;
        if (tm.leader() && I.hist && iter < I.histCap)
            for (int q = 0; q < 6; ++q) I.hist[6 * (size_t)iter + q] = last[q];
        if (is_set(end[2])) {
            converged = end[2] == 1.0;
            diverged = !converged;
            finalIter = iter;
            break;
        }
    }
    tm.sync();
    if (tm.leader()) {
        const bool aborted = !tm.ok();
        I.out[0] = aborted ? 4 : (diverged ? 2 : (converged ? 0 : 1));
        I.out[1] = converged;
        I.out[2] = diverged;
        I.out[3] = finalIter;
        I.out[4] = ran;
        I.out[5] = turbEst;
        I.out[6] = aborted ? 1 : 0;
        I.out[7] = -1;
        inner = innerMom + innerP + innerTurb;
        I.outInner[0] = inner;
        I.outInner[1] = innerMom;
        I.outInner[2] = innerP;
        I.outInner[3] = innerTurb;
        I.outInner[4] = 0;
        for (int q = 0; q < 6; ++q) I.outLast[q] = last[q];
        I.outLast[6] = normUx0;
        I.outLast[7] = normUy0;
        I.outLast[8] = normP0;
        if (I.S.refAmg && I.S.pSolver == 3 && clk.acc[5] >= I.rg.setupNs) {
            // hierarchy setups of the reference-order AMG count as AMG setup
            clk.acc[5] -= I.rg.setupNs;
            clk.acc[4] += I.rg.setupNs;
        }
        for (int q = 0; q < kPhaseSlots; ++q) I.outTime[q] = clk.acc[q];
        I.outTime[kPhaseSlots] = tStart;
        I.outTime[kPhaseSlots + 1] = globaltimer_ns();
        if (I.obsOut) observe_leader<T>(M, I);
        if (I.doneFlag) {
            __threadfence_system();
            *I.doneFlag = 1;
        }
    }
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
// One CTA per instance.  NT threads per CTA; small instances use NT = 256 so
// that two instances share an SM and hide each other's latency.
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_simple_block(DevInst *insts, int n) {
    __shared__ double red[NT > 2 * 32 * kRedSlots ? NT : 2 * 32 * kRedSlots];
    __shared__ double tot[2 * (NT / 32) + kRedResults];
    __shared__ DevMesh sM;
    __shared__ DevInst sI;
    if (blockIdx.x >= n) return;
    if (threadIdx.x == 0) {
        sI = insts[blockIdx.x];
        sM = *sI.M;
    }
    __syncthreads();
    BlockTeam tm{red, 0, tot, 0, live_warps(sM.nC)};
    simple_solve(tm, sM, sI);
}
template __global__ void k_simple_block<256>(DevInst *, int);
template __global__ void k_simple_block<512>(DevInst *, int);

// The same for launches that contain instances with the reference-order AMG;
// `xsCap` doubles of dynamic shared memory hold every level's x when they fit.
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_simple_block_ref(DevInst *insts, int n, int xsCap) {
    __shared__ double red[NT > 2 * 32 * kRedSlots ? NT : 2 * 32 * kRedSlots];
    __shared__ double tot[2 * (NT / 32) + kRedResults];
    __shared__ DevMesh sM;
    __shared__ DevInst sI;
    extern __shared__ __align__(16) double xsm[];
    if (blockIdx.x >= n) return;
    if (threadIdx.x == 0) {
        sI = insts[blockIdx.x];
        sM = *sI.M;
        sI.rg.xs = (sI.S.refAmg && (int64_t)sM.nC + sI.rg.rowPool <= xsCap) ? xsm : nullptr;
    }
    __syncthreads();
    BlockTeamRef tm;
    tm.red = red;
    tm.buf = 0;
    tm.tot = tot;
    tm.turn = 0;
    tm.live = live_warps(sM.nC);
    simple_solve(tm, sM, sI);
}
template __global__ void k_simple_block_ref<256>(DevInst *, int, int);
template __global__ void k_simple_block_ref<512>(DevInst *, int, int);

__global__ void __launch_bounds__(kThreads, 1) k_simple_grid(DevInst *inst) {
    __shared__ double red[2 * 32 * kRedSlots];
    __shared__ DevMesh sM;
    __shared__ DevInst sI;
    __shared__ int shAbort;
    if (threadIdx.x == 0) {
        sI = *inst;
        sM = *sI.M;
        shAbort = 0;
    }
    __syncthreads();
    GridTeam tm{red, 0, sI.gpart, sI.barrier, sI.err, &shAbort, 0u};
    simple_solve(tm, sM, sI);
}

// Test hook: one phase on one CTA with the state already on the device.
__global__ void __launch_bounds__(kThreads, 1) k_debug(DevInst *inst) {
    __shared__ double red[kThreads > 2 * 32 * kRedSlots ? kThreads : 2 * 32 * kRedSlots];
    __shared__ double tot[2 * (kThreads / 32) + kRedResults];
    __shared__ DevMesh sM;
    __shared__ DevInst sI;
    if (threadIdx.x == 0) {
        sI = *inst;
        sM = *sI.M;
    }
    __syncthreads();
    BlockTeamRef tm;
    tm.red = red;
    tm.buf = 0;
    tm.tot = tot;
    tm.turn = 0;
    tm.live = live_warps(sM.nC);
    const DevMesh &M = sM;
    DevInst &I = sI;
    const int ph = I.dbgPhase, arg = I.dbgArg;
    const bool d2 = M.is2d && !I.solveZ;
    auto grads = [&]() {
        if (d2) {
            phase_grad_init(tm, M, I);
            tm.sync();
            phase_grads<BlockTeamRef, true>(tm, M, I, 15);
        } else {
            phase_grads<BlockTeamRef, false>(tm, M, I, 15);
        }
        tm.sync();
    };
    SolveResult res = {0, 0.0, 0.0, 0};
    switch (ph) {
        case 1:  // greenGaussGrad of p -> gp
            grads();
            break;
        case 2:  // computeFields (no floor) + |S|
            grads();
            if (d2) phase_closure<BlockTeamRef, true>(tm, M, I, -1.0);
            else phase_closure<BlockTeamRef, false>(tm, M, I, -1.0);
            break;
        case 3:  // assembleMomentum(comp = arg)
            grads();
            if (d2) phase_momq_faces<BlockTeamRef, true>(tm, M, I, arg, true, nullptr);
            else phase_momq_faces<BlockTeamRef, false>(tm, M, I, arg, true, nullptr);
            tm.sync();
            phase_momq_cells(tm, M, I, arg);
            break;
        case 4:  // assemblePressureCorrection with I.aPx
            grads();
            phase_dp(tm, M, I);
            tm.sync();
            if (d2) phase_pq_faces<BlockTeamRef, true>(tm, M, I);
            else phase_pq_faces<BlockTeamRef, false>(tm, M, I);
            tm.sync();
            phase_pq_cells(tm, M, I);
            break;
        case 5:
        case 6:  // assembleKEquation / assembleOmegaEquation
            if (d2) phase_turbq_faces<BlockTeamRef, true>(tm, M, I, ph - 5, true);
            else phase_turbq_faces<BlockTeamRef, false>(tm, M, I, ph - 5, true);
            tm.sync();
            phase_turbq_cells(tm, M, I, ph - 5);
            break;
        case 7:  // v = A r
            for (int c = tm.rank(); c < M.nC; c += tm.size()) I.v[c] = ldu_row<BlockTeamRef>(M, I, I.r, c);
            break;
        case 8:  // BiCGSTAB on (diag,upper,lower,src), x = pp
            res = team_bicgstab(tm, M, I, I.pp, I.S.innerIter, I.S.innerTol);
            break;
        case 9:  // AMG-PCG on the same system, x = pp (starts at zero)
            for (int c = tm.rank(); c < M.nC; c += tm.size()) I.pp[c] = 0.0;
            tm.sync();
            res = team_amg_pcg(tm, M, I, I.pp, I.S.innerIter, I.S.innerTol);
            break;
        case 11:  // PCG (Jacobi)
            res = team_pcg(tm, M, I, I.pp, I.S.innerIter, I.S.innerTol);
            break;
        case 13:  // Gauss-Seidel
            res = team_gauss_seidel(tm, M, I, I.pp, I.S.innerIter, I.S.innerTol);
            break;
        case 12:  // reference-order AMG hierarchy of (diag, upper, lower)
            if (I.S.refAmg) res.iterations = ramg_setup(tm, M, I, true);
            break;
    }
    tm.sync();
    if (threadIdx.x == 0) {
        I.outLast[0] = res.iterations;
        I.outLast[1] = sqrt(res.finalSq) / (res.initialRes < 1e-30 ? 1.0 : res.initialRes);
        I.outLast[2] = res.initialRes;
        I.outLast[3] = res.converged;
    }
}

// ---------------------------------------------------------------------------
// Mesh::computeWallDistance (core/src/Mesh.cpp:345-373): minimum over the wall
// face centres of |c - w|.  Each thread owns one cell; the wall centres stream
// through shared memory in tiles.  The squared distance is formed exactly as
// (dx*dx + dy*dy) + dz*dz without contraction and the square root is taken
// once of the minimum: sqrt is correctly rounded and monotone, so the result
// is bit-identical to the reference's minimum of square roots.
//
// Nine FP64 instructions per pair at 1/64 of the FP32 rate bound the plain
// search (122,880 cells, 992 faces: the whole call, allocation and copies
// included, 2.89 ms; with what follows 1.96 ms).  A first pass finds each
// cell's least distance in FP32, a second one the faces whose FP32 distance is
// within twice its error of that, and only those are measured in FP64 (a
// handful per cell, kept in a list so that the lanes measure theirs together).
//
// Error of an FP32 distance: coordinates relative to the first wall centre are
// formed in FP64 and rounded once (|error| <= 2^-24 R, R the largest of them in
// the cell and the walls), their differences once more; with the rounding of
// the squares, sum and root the distance is off by less than 2^-20 R.  The
// pass allows 2^-18 R.  Non-finite or overflowing coordinates make the
// threshold infinite: every face is measured.
// ---------------------------------------------------------------------------
constexpr int kWallTile = 1024;
constexpr int kWallList = 8;
__device__ __forceinline__ double wall_d2(double x, double y, double z, const double *w) {
    const double dx = __dsub_rn(x, w[0]), dy = __dsub_rn(y, w[1]), dz = __dsub_rn(z, w[2]);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}
__global__ void __launch_bounds__(256) k_wall_distance(const double *cc, int nC, const double *wp, int nW,
                                                        double *out) {
    __shared__ float sx[kWallTile], sy[kWallTile], sz[kWallTile];
    __shared__ unsigned int reach;   // largest |wall coordinate|, as float bits (NaN and infinity largest)
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const double ox = wp[0], oy = wp[1], oz = wp[2];
    double x = ox, y = oy, z = oz;
    if (c < nC) { x = cc[3 * (size_t)c]; y = cc[3 * (size_t)c + 1]; z = cc[3 * (size_t)c + 2]; }
    const float fx = (float)(x - ox), fy = (float)(y - oy), fz = (float)(z - oz);
    if (threadIdx.x == 0) reach = 0;
    auto stage = [&](int t0, int n, bool measure) {
        __syncthreads();
        float m = 0.0f;
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const double *w = wp + 3 * (size_t)(t0 + j);
            const float ax = (float)(w[0] - ox), ay = (float)(w[1] - oy), az = (float)(w[2] - oz);
            sx[j] = ax; sy[j] = ay; sz[j] = az;
            if (measure) {
                const unsigned int big = max(__float_as_uint(fabsf(ax)),
                                             max(__float_as_uint(fabsf(ay)), __float_as_uint(fabsf(az))));
                m = __uint_as_float(max(__float_as_uint(m), big));
            }
        }
        if (measure) atomicMax(&reach, __float_as_uint(m));
        __syncthreads();
    };
    float least = INFINITY;
    for (int t0 = 0; t0 < nW; t0 += kWallTile) {
        const int n = min(kWallTile, nW - t0);
        stage(t0, n, true);
#pragma unroll 4
        for (int j = 0; j < n; ++j) {
            const float dx = fx - sx[j], dy = fy - sy[j], dz = fz - sz[j];
            least = fminf(least, fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
        }
    }
    float size = fmaxf(fmaxf(fabsf(fx), fabsf(fy)), fmaxf(fabsf(fz), __uint_as_float(reach)));
    if (isnan(fx) || isnan(fy) || isnan(fz) || isnan(__uint_as_float(reach))) size = INFINITY;
    const float edge = sqrtf(least) + 2.0f * 0x1p-18f * size;
    float limit = fmaf(edge, edge, 1e-37f) * 1.00001f;
    if (isnan(limit)) limit = INFINITY;
    double best = INFINITY;
    int list[kWallList], held = 0;
    auto measure = [&]() {
        int most = held;
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
        for (int q = 0; q < most; ++q) {
            if (q < held) {
                int j = list[0];
#pragma unroll
                for (int e = 1; e < kWallList; ++e) j = q == e ? list[e] : j;
                const double d2 = wall_d2(x, y, z, wp + 3 * (size_t)j);
                best = d2 < best ? d2 : best;
            }
        }
        held = 0;
    };
    for (int t0 = 0; t0 < nW; t0 += kWallTile) {
        const int n = min(kWallTile, nW - t0);
        if (nW > kWallTile) stage(t0, n, false);
        for (int j = 0; j < n; ++j) {
            const float dx = fx - sx[j], dy = fy - sy[j], dz = fz - sz[j];
            // (a NaN here is a NaN in FP64 too, which is never the least)
            if (!(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > limit)) {
#pragma unroll
                for (int e = 0; e < kWallList; ++e) list[e] = held == e ? t0 + j : list[e];
                ++held;
            }
            if (__any_sync(0xffffffffu, held == kWallList)) measure();
        }
    }
    measure();
    if (c < nC) out[c] = sqrt(best);
}

int engine_wall_distance(const double *dCentres, int nC, const double *dWall, int nW, double *dOut, void *stream) {
    if (nC <= 0) return 0;
    k_wall_distance<<<(nC + 255) / 256, 256, 0, (cudaStream_t)stream>>>(dCentres, nC, dWall, nW, dOut);
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Staging of a batch's results and start states.  A 219-instance batch took
// 4,600 copies of a few KB, 53 ms beside a 56 ms solve; gathered into one
// buffer it is one copy.  blockIdx.y: instance, x: cells in strides.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pack(const StageItem *items, double *stage) {
    const StageItem &S = items[blockIdx.y];
    double *o = stage + S.at;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    if (t < 9) o[t] = S.last[t];
    if (t == 9) o[t] = __longlong_as_double((long long)*S.err);
    if (t >= 10 && t < 14) {
        const unsigned int lo = (unsigned int)S.out[2 * (t - 10)], hi = (unsigned int)S.out[2 * (t - 10) + 1];
        o[t] = __longlong_as_double((long long)((unsigned long long)hi << 32 | lo));
    }
    if (t >= 14 && t < 19) o[t] = __longlong_as_double(S.inner[t - 14]);
    if (t >= 19 && t < 19 + kPhaseSlots + 2) o[t] = __longlong_as_double((long long)S.time[t - 19]);
    o += kStageHead;
    for (int q = t; q < S.nObs; q += nt) o[q] = S.obs[q];
    if (!S.state) return;
    o += S.nObs;
    const int nC = S.nC, nB = S.nB;
    double *cells = o + 3 * (size_t)nC, *bu = cells + kStageCells * (size_t)nC, *bs = bu + 3 * (size_t)nB;
    for (int c = t; c < nC; c += nt) {
        for (int i = 0; i < 3; ++i) o[3 * (size_t)c + i] = S.u[i][c];
        for (int k = 0; k < kStageCells; ++k) cells[k * (size_t)nC + c] = S.cell[k][c];
    }
    for (int b = t; b < nB; b += nt) {
        for (int i = 0; i < 3; ++i) bu[3 * (size_t)b + i] = S.ub[i][b];
        for (int k = 0; k < 3; ++k) bs[k * (size_t)nB + b] = S.bnd[k][b];
    }
}
__global__ void __launch_bounds__(256) k_unpack(const StageItem *items, const double *stage) {
    const StageItem &S = items[blockIdx.y];
    const double *o = stage + S.at;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const int nC = S.nC, nB = S.nB;
    const double *cells = o + 3 * (size_t)nC, *bu = cells + kStageCells * (size_t)nC, *bs = bu + 3 * (size_t)nB;
    for (int c = t; c < nC; c += nt) {
        for (int i = 0; i < 3; ++i) S.u[i][c] = o[3 * (size_t)c + i];
        for (int k = 0; k < kStageCells; ++k)
            if (S.cell[k]) S.cell[k][c] = cells[k * (size_t)nC + c];
    }
    for (int b = t; b < nB; b += nt) {
        for (int i = 0; i < 3; ++i) S.ub[i][b] = bu[3 * (size_t)b + i];
        for (int k = 0; k < 3; ++k) S.bnd[k][b] = bs[k * (size_t)nB + b];
    }
}
int engine_pack(const StageItem *dItems, int n, int maxCells, double *dStage, void *stream) {
    const dim3 grid(min(64, (maxCells + 255) / 256), n);
    k_pack<<<grid, 256, 0, (cudaStream_t)stream>>>(dItems, dStage);
    return (int)cudaGetLastError();
}
int engine_unpack(const StageItem *dItems, int n, int maxCells, const double *dStage, void *stream) {
    const dim3 grid(min(64, (maxCells + 255) / 256), n);
    k_unpack<<<grid, 256, 0, (cudaStream_t)stream>>>(dItems, dStage);
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------
int engine_block_threads() { return kThreads; }

// Dynamic shared memory of the reference-order kernel for the level vectors
// (every level's x: nC + 2 nC + 64 doubles) when they fit within this much.
constexpr int kRamgXsBytes256 = 96 * 1024;    // two CTAs per SM
constexpr int kRamgXsBytes512 = 192 * 1024;   // one CTA per SM

int engine_launch_block(DevInst *dInsts, int n, int threads, void *stream, bool refAmg, int maxCells) {
    if (n <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (refAmg) {
        const int cap = threads == 256 ? kRamgXsBytes256 : kRamgXsBytes512;
        // only what the level vectors need: the rest of the SM's shared
        // memory / L1 stays L1, which holds level 0's matrix
        const int64_t need = 8 * (3 * (int64_t)maxCells + 64);
        const int bytes = need <= cap ? (int)need : 0;
        cudaError_t e;
        if (threads == 256) {
            e = cudaFuncSetAttribute(k_simple_block_ref<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
            if (e != cudaSuccess) return (int)e;
            k_simple_block_ref<256><<<n, 256, bytes, st>>>(dInsts, n, bytes / 8);
        } else {
            e = cudaFuncSetAttribute(k_simple_block_ref<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
            if (e != cudaSuccess) return (int)e;
            k_simple_block_ref<512><<<n, 512, bytes, st>>>(dInsts, n, bytes / 8);
        }
    } else {
        if (threads == 256) k_simple_block<256><<<n, 256, 0, st>>>(dInsts, n);
        else k_simple_block<512><<<n, 512, 0, st>>>(dInsts, n);
    }
    return (int)cudaGetLastError();
}

int engine_grid_blocks(int *blocks_out) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_simple_grid, kThreads, 0);
    if (e != cudaSuccess) return (int)e;
    if (per < 1) per = 1;
    *blocks_out = sms * per;
    return 0;
}

int engine_launch_grid(DevInst *dInst, int blocks, void *stream) {
    void *args[] = {&dInst};
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_simple_grid, dim3(blocks), dim3(kThreads), args, 0,
                                                (cudaStream_t)stream);
    return (int)e;
}

int engine_launch_debug(DevInst *dInst, void *stream) {
    k_debug<<<1, kThreads, 0, (cudaStream_t)stream>>>(dInst);
    return (int)cudaGetLastError();
}

}  // namespace btm
