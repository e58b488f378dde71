// btm_cycle.cuh - the multigrid V-cycle of large meshes (one mesh on the
// cooperative grid) on the per-case hierarchy, shared by the FP64 and
// mixed-precision engines.
//
// A V-cycle is a chain of about 50 short passes, each a barrier and then one
// sparse row per thread: a barrier is 1.4 us and a row was 4 us, of which the
// multiply-adds take 0.3; the rest were dependent loads (row pointer, columns, x,
// then 1 / diagonal and the aggregate's members), all from L2, as a barrier's
// acquire empties L1.  But only x (or the residual) changes from pass to pass.
// Every pass here therefore begins with its loads of everything else, runs them
// inside its barrier (between arrival and wait), and then needs x only: the
// barrier's latency and those of the loads overlap.  74k-cell duct, FP32:
// pressure solve 1.66 -> 1.05 ms an outer iteration; 123k-cell step, FP64: 22.4
// -> 19.4 ms (there the FP64 multiply-adds weigh more).
//
// `A` presents the arrays of an engine: V (value type), lev(l), x(l), b(l),
// r(l), val(l), rd(l), sys() (diag | upper | lower of level 0), ainv().
#pragma once
#include "btm_common.h"
#include "btm_team.cuh"
#include <type_traits>

namespace btm {

// one sparse row with its coefficients, ready for x
template <class V, int W>
struct CycRow {
    int col[W], n, more;    // n: entries; the ones past W start at `more`
    V a[W];
};

template <class T, class A>
struct Cycle {
    using V = typename A::V;
    static constexpr int WC = 8;   // entries held of a coarse row; of level 0: 4 (quadrilaterals) or 6 (hexahedra)

    // ---- rows: level 0 from the position-major tables (off-diagonal part),
    // coarse levels from their CSR (all of it)
    template <int W0>
    __device__ __forceinline__ static void fetch(const A &a, const RowTab &R, int i, CycRow<V, W0> &r) {
        const V *sys = a.sys();
        r.n = R.width;
        r.more = W0;
#pragma unroll
        for (int k = 0; k < W0; ++k) {
            const bool in = k < R.width;
            const size_t at = (size_t)(in ? k : 0) * R.nC + i;
            r.col[k] = in ? R.col[at] : -1;
            r.a[k] = LD(sys + R.ent[at]);
        }
    }
    __device__ __forceinline__ static void fetch(const AmgLevelDev &L, const V *val, int i, CycRow<V, WC> &r) {
        const int q0 = L.rowPtr[i];
        r.n = L.rowPtr[i + 1] - q0;
        r.more = q0 + WC;
#pragma unroll
        for (int k = 0; k < WC; ++k) {
            const int at = q0 + min(k, r.n - 1);
            r.col[k] = k < r.n ? L.colIdx[at] : -1;
            r.a[k] = LD(val + at);
        }
    }
    // y + row x (Neg: y - row x), without column `skip`, in the row's order
    template <bool Neg, int W0>
    __device__ __forceinline__ static V apply(const A &a, const RowTab &R, const CycRow<V, W0> &r, const V *x, int i,
                                              V y) {
        V v[W0];
#pragma unroll
        for (int k = 0; k < W0; ++k) v[k] = LD(x + max(r.col[k], 0));
#pragma unroll
        for (int k = 0; k < W0; ++k)
            if (r.col[k] >= 0) y = fma_any(Neg ? -r.a[k] : r.a[k], v[k], y);
        for (int k = W0; k < R.width; ++k) {
            const size_t at = (size_t)k * R.nC + i;
            const int c = R.col[at];
            const V e = LD(a.sys() + R.ent[at]);
            if (c >= 0) y = fma_any(Neg ? -e : e, LD(x + c), y);
        }
        return y;
    }
    template <bool Neg>
    __device__ __forceinline__ static V apply(const AmgLevelDev &L, const V *val, const CycRow<V, WC> &r, const V *x,
                                              int skip, V y) {
        V v[WC];
#pragma unroll
        for (int k = 0; k < WC; ++k) v[k] = LD(x + max(r.col[k], 0));
#pragma unroll
        for (int k = 0; k < WC; ++k)
            if (r.col[k] >= 0 && r.col[k] != skip) y = fma_any(Neg ? -r.a[k] : r.a[k], v[k], y);
        for (int k = WC; k < r.n; ++k) {
            const int at = r.more + k - WC, c = L.colIdx[at];
            const V e = LD(val + at);
            if (c != skip) y = fma_any(Neg ? -e : e, LD(x + c), y);
        }
        return y;
    }

    // ---- one colour-ordered Gauss-Seidel sweep (colours ascending, or
    // descending).  `zero`: x is zero, and the first colour needs no x at all;
    // b may have been written in the pass before, so it waits for the barrier.
    // Without `zero` b is older than the last barrier.
    __device__ __noinline__ static void gs(T &tm, const A &a, int l, bool reverse, bool zero) {
        const AmgLevelDev &L = a.lev(l);
        const RowTab R = a.rows();
        V *x = a.x(l);
        const V *b = a.b(l), *rd = a.rd(l), *val = a.val(l);
        const int32_t *off = L.colorOff, *rowsOf = L.colorRows;
        const int nColors = L.nColors;
        if (l > 0) gs_level<false, WC>(tm, a, L, R, x, b, rd, val, off, rowsOf, nColors, reverse, zero);
        else if (R.width <= 4) gs_level<true, 4>(tm, a, L, R, x, b, rd, val, off, rowsOf, nColors, reverse, zero);
        else gs_level<true, 6>(tm, a, L, R, x, b, rd, val, off, rowsOf, nColors, reverse, zero);
    }
    template <bool L0, int W>
    __device__ __forceinline__ static void gs_level(T &tm, const A &a, const AmgLevelDev &L, const RowTab &R, V *x,
                                                    const V *b, const V *rd, const V *val, const int32_t *off,
                                                    const int32_t *rowsOf, int nColors, bool reverse, bool zero) {
        for (int cc = 0; cc < nColors; ++cc) {
            const int col = reverse ? nColors - 1 - cc : cc;
            const int q1 = off[col + 1];
            int q = off[col] + tm.spread();
            const bool on = q < q1, alone = zero && cc == 0;
            int i = 0;
            CycRow<V, W> r;
            V ri = 0, bi = 0;
            tm.arrive();
            if (on) {
                i = rowsOf[q];
                ri = LD(rd + i);
                if (!alone) {
                    bi = LD(b + i);
                    if constexpr (L0) fetch(a, R, i, r);
                    else fetch(L, val, i, r);
                }
            }
            tm.wait();
            if (on && ri != (V)0) {
                if (alone) bi = LD(b + i);
                else if constexpr (L0) bi = apply<true>(a, R, r, x, i, bi);
                else bi = apply<true>(L, val, r, x, i, bi);
                x[i] = bi * ri;
            }
            for (q += tm.size(); q < q1; q += tm.size()) {
                i = rowsOf[q];
                ri = LD(rd + i);
                if (ri == (V)0) continue;
                bi = LD(b + i);
                if (!alone) {
                    if constexpr (L0) {
                        fetch(a, R, i, r);
                        bi = apply<true>(a, R, r, x, i, bi);
                    } else {
                        fetch(L, val, i, r);
                        bi = apply<true>(L, val, r, x, i, bi);
                    }
                }
                x[i] = bi * ri;
            }
        }
    }

    template <int W0>
    __device__ __forceinline__ static void residual0(T &tm, const A &a, const RowTab &R, const V *x, const V *b, V *res,
                                                     int n) {
        const V *sys = a.sys();
        int i = tm.spread();
        CycRow<V, W0> r;
        V d = 0, bi = 0;
        auto get = [&](int j) {
            fetch(a, R, j, r);
            d = LD(sys + j);
            bi = LD(b + j);
        };
        tm.arrive();
        if (i < n) get(i);
        tm.wait();
        for (; i < n; i += tm.size()) {
            res[i] = bi - apply<false>(a, R, r, x, i, d * LD(x + i));
            if (i + tm.size() < n) get(i + tm.size());
        }
    }
    // ---- residual of level l and its restriction, b of level l + 1 (members in
    // order); with `smooth` also the first damped-Jacobi sweep of level l + 1,
    // which starts from zero and needs no neighbours, into that level's r (its
    // x is not read before the second sweep writes it), else its x = 0.  (One
    // pass over the coarse rows, each forming its members' residuals in turn,
    // leaves most lanes waiting for the row with the most members.)
    __device__ __noinline__ static void restrict_to(T &tm, const A &a, int l, bool smooth) {
        const AmgLevelDev &L = a.lev(l);
        {
            const RowTab R = a.rows();
            const V *x = a.x(l), *b = a.b(l), *val = a.val(l);
            V *res = a.r(l);
            const int n = L.n;
            if (l == 0) {
                if (R.width <= 4) residual0<4>(tm, a, R, x, b, res, n);
                else residual0<6>(tm, a, R, x, b, res, n);
            } else {
                int i = tm.spread();
                CycRow<V, WC> r;
                V bi = 0;
                tm.arrive();
                if (i < n) {
                    fetch(L, val, i, r);
                    bi = LD(b + i);
                }
                tm.wait();
                for (; i < n; i += tm.size()) {
                    res[i] = bi - apply<false>(L, val, r, x, -1, (V)0);
                    if (i + tm.size() < n) {
                        fetch(L, val, i + tm.size(), r);
                        bi = LD(b + i + tm.size());
                    }
                }
            }
        }
        constexpr int K = 4;
        const V *res = a.r(l);
        V *bc = a.b(l + 1), *xc = a.x(l + 1), *rc = a.r(l + 1);
        const V *rd = a.rd(l + 1);
        const int n = a.lev(l + 1).n;
        const int32_t *off = L.aggOff, *mem = L.aggMem;
        int J = tm.spread();
        bool ready = J < n;
        int o = 0, m = 0, at[K];
        V w = 0;
        auto members = [&]() {
            o = off[J];
            m = off[J + 1] - o;
#pragma unroll
            for (int k = 0; k < K; ++k) at[k] = mem[o + min(k, m - 1)];
            if (smooth) w = A::kWeight * LD(rd + J);
        };
        tm.arrive();
        if (ready) members();
        tm.wait();
        for (; J < n; J += tm.size()) {
            if (!ready) members();
            ready = false;
            V v[K], s = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] = LD(res + at[k]);
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < m) s += v[k];
            for (int k = K; k < m; ++k) s += LD(res + mem[o + k]);
            bc[J] = s;
            if (smooth) rc[J] = fma_any(w, s, (V)0);
            else xc[J] = 0;
        }
    }

    // ---- the correction of one row to the members of its aggregate on the finer
    // level (every finer row has one aggregate): the members' x are final since
    // the way down
    struct Up {
        static constexpr int K = 4;
        int o, m, at[K];
        V v[K];
        __device__ __forceinline__ void fetch(const A &a, int l, int J) {
            const AmgLevelDev &F = a.lev(l - 1);
            const V *x = a.x(l - 1);
            o = F.aggOff[J];
            m = F.aggOff[J + 1] - o;
#pragma unroll
            for (int k = 0; k < K; ++k) at[k] = F.aggMem[o + min(k, m - 1)];
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] = LD(x + at[k]);
        }
        __device__ __forceinline__ void add(const A &a, int l, V c) const {
            V *x = a.x(l - 1);
            const int32_t *mem = a.lev(l - 1).aggMem;
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < m) x[at[k]] = v[k] + c;
            for (int k = K; k < m; ++k) x[mem[o + k]] = LD(x + mem[o + k]) + c;
        }
    };

    // ---- one damped-Jacobi sweep on a coarse level: reads x, writes `out`, or
    // (UP) adds the result, the level's last, to the finer level.  `fresh`: b was
    // written in the pass before and waits for the barrier.
    template <bool UP>
    __device__ __noinline__ static void jacobi(T &tm, const A &a, int l, const V *x, V *out, bool fresh) {
        const AmgLevelDev &L = a.lev(l);
        const V *b = a.b(l), *val = a.val(l), *rd = a.rd(l);
        const int n = L.n;
        CycRow<V, WC> r;
        Up u;
        V bi = 0, w = 0;
        int i = tm.spread();
        auto get = [&](int j) {
            fetch(L, val, j, r);
            if (!fresh) bi = LD(b + j);
            w = A::kWeight * LD(rd + j);
            if (UP) u.fetch(a, l, j);
        };
        tm.arrive();
        if (i < n) get(i);
        tm.wait();
        for (; i < n; i += tm.size()) {
            const V xi = LD(x + i);
            if (fresh) bi = LD(b + i);
            const V v = fma_any(w, apply<true>(L, val, r, x, -1, bi), xi);
            if (UP) u.add(a, l, v);
            else out[i] = v;
            if (i + tm.size() < n) get(i + tm.size());
        }
    }

    // x += the coarser level's correction
    __device__ __noinline__ static void prolong(T &tm, const A &a, int l) {
        const AmgLevelDev &L = a.lev(l);
        V *x = a.x(l);
        const V *xc = a.x(l + 1);
        tm.sync();
        for (int i = tm.spread(); i < L.n; i += tm.size()) x[i] = LD(x + i) + LD(xc + L.map[i]);
    }

    // ---- coarsest level.  Dense inverse of more than kCoarseDirect rows (the
    // grid): one warp per row, lane-strided partial sums folded by a butterfly,
    // the correction straight to the finer level.
    __device__ __noinline__ static void dense_up(T &tm, const A &a) {
        const int l = a.levels() - 1, n = a.lev(l).n, lane = threadIdx.x & 31;
        const V *b = a.b(l);
        constexpr int K = 16;
        double m[K];
        int i = tm.spread() >> 5;
        Up u;
        auto get = [&](int j) {
            const double *row = a.ainv() + (size_t)j * n;
#pragma unroll
            for (int k = 0; k < K; ++k) m[k] = LD(row + min(lane + 32 * k, n - 1));
            u.fetch(a, l, j);
        };
        tm.arrive();
        if (i < n) get(i);
        tm.wait();
        for (; i < n; i += tm.size() >> 5) {
            const double *row = a.ainv() + (size_t)i * n;
            double s = 0.0;
            V v[K];
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] = LD(b + min(lane + 32 * k, n - 1));
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (lane + 32 * k < n) s = fma(m[k], (double)v[k], s);
            for (int j0 = lane + 32 * K; j0 < n; j0 += 32 * K) {
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    m[k] = LD(row + min(j0 + 32 * k, n - 1));
                    v[k] = LD(b + min(j0 + 32 * k, n - 1));
                }
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (j0 + 32 * k < n) s = fma(m[k], (double)v[k], s);
            }
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) u.add(a, l, (V)s);
            if (i + (tm.size() >> 5) < n) get(i + (tm.size() >> 5));
        }
    }
    __device__ __noinline__ static void coarse(T &tm, const A &a) {
        const int l = a.levels() - 1, n = a.lev(l).n;
        if (a.direct()) {
            const V *b = a.b(l);
            V *x = a.x(l);
            constexpr int K = 16;   // entries of a row held
            const int i = tm.rank();
            const double *row = a.ainv() + (size_t)i * n;
            double m[K];
            if (i < n)
#pragma unroll
                for (int k = 0; k < K; ++k) m[k] = LD(row + min(k, n - 1));
            tm.sync();
            if (i < n) {   // at most kCoarseDirect rows
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (k < n) s = fma(m[k], (double)LD(b + k), s);
                for (int j = K; j < n; ++j) s = fma(LD(row + j), (double)LD(b + j), s);
                x[i] = (V)s;
            }
        } else {
            // the sweeps fetch b inside their first barrier, and the restriction
            // (or the residual of a mesh without coarse levels) has just written
            // it: a barrier of its own, once a cycle of kCoarseSweeps sweeps
            tm.sync();
            for (int s = 0; s < kCoarseSweeps; ++s) gs(tm, a, l, (s & 1) != 0, false);
        }
    }

    // ---- the V-cycle: two smoothing sweeps of every level before and after the
    // coarse correction, on level 0 multicolour Gauss-Seidel (colours ascending
    // before, descending after: symmetric, so the preconditioner suits CG), on the
    // coarse levels a pair of damped-Jacobi sweeps (x -> r -> x): one barrier per
    // sweep rather than one per colour (6-11 colours on Galerkin levels), for
    // ~15-20 % more PCG iterations.  Starts from x(0) = 0, ends with a barrier.
    __device__ static void run(T &tm, const A &a) {
        const int nl = a.levels();
        const bool dense = nl > 1 && a.direct() && a.lev(nl - 1).n > kCoarseDirect;
        for (int l = 0; l < nl - 1; ++l) {
            if (l == 0) {
                gs(tm, a, l, false, true);
                gs(tm, a, l, false, false);
            } else {
                jacobi<false>(tm, a, l, a.r(l), a.x(l), true);
            }
            restrict_to(tm, a, l, l + 1 < nl - 1);
        }
        if (dense) {
            dense_up(tm, a);
        } else {
            coarse(tm, a);
            if (nl > 1) prolong(tm, a, nl - 2);
        }
        for (int l = nl - 2; l >= 0; --l) {
            if (l == 0) {
                gs(tm, a, l, true, false);
                gs(tm, a, l, true, false);
            } else {
                jacobi<false>(tm, a, l, a.x(l), a.r(l), false);
                jacobi<true>(tm, a, l, a.r(l), a.x(l), false);
            }
        }
        tm.sync();
    }
};

}  // namespace btm
