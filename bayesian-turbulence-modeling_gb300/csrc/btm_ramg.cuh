// btm_ramg.cuh - the reference's AMG-preconditioned CG (AMGSolver,
// core/include/LinearSolver.hpp:497-656) on one CTA, with the hierarchy
// rebuilt from the actual matrix at every solve and every Gauss-Seidel sweep
// in the reference's row order.
//
// The reference's setup and smoother are sequential loops over rows.  Both
// are evaluated here in parallel with the sequential results:
//
//   * Forward Gauss-Seidel (CSRMatrix::gaussSeidelSweep, :328-337): row i
//     reads the new x of its lower-index neighbours and the old x of the
//     higher-index ones.  Rows are grouped into wavefronts by the depth of
//     the "lower-index neighbour" DAG (depth(i) = 1 + max depth of its
//     lower-index neighbours); a wavefront's rows are independent, and every
//     row sums its terms in the reference's order.
//   * Greedy aggregation (buildAggregates, :407-443): a row becomes a seed
//     exactly when no lower-index seed claims it, and it is claimed by the
//     lowest-index seed whose row entry for it is strong.  That recursion runs
//     over the same wavefronts; aggregate ids are the seeds' prefix count in
//     row order.  (The reference's second pass never finds an unassigned row:
//     every row is a seed or claimed in the first.)  The aggregation maps are
//     therefore bit-identical to the reference's.
//   * Galerkin product (galerkinProduct, :446-485): an aggregate's members
//     are its seed and the rows its seed claimed, all in the seed's row; each
//     coarse entry sums its fine entries in (fine row ascending, fine column
//     ascending) order, as the reference's single pass over the fine rows.
//
// Levels of at most kRamgWarpRows rows run on warp 0 alone (warp barriers
// instead of CTA barriers).  Dot products of the CG loop are parallel trees,
// and the smoother multiplies by reciprocal diagonals where the reference
// divides: both differ from the reference in the last bits only.
//
// Coarse levels live in per-instance pools sized at twice the fine rows and
// three times the fine entries; a level that would not fit ends the
// hierarchy (it becomes the coarsest level, smoothed by the reference's 50
// sweeps), which typical 2-D and 3-D meshes never reach.
#pragma once
#include "btm_common.h"
#include "btm_team.cuh"

namespace btm {

constexpr int kRamgMinCoarse = 50;     // minCoarseSize_ (LinearSolver.hpp:509)
constexpr int kRamgCoarseSweeps = 50;  // coarseSweeps_
constexpr int kRamgMaxCoarsen = 20;    // maxLevels_
constexpr int kRamgWarpRows = 64;     // levels up to this size run on warp 0

// One level as the device functions see it.  Level 0 reads its values from
// the LDU system through entry ids (the lduToCSR layout built per case).
struct RLevel {
    int n, nWf;
    const int32_t *ptr, *col, *ent;
    const double *val, *dg, *ldu;
    const int32_t *wfOff, *wfRows;
    const double *rd;               // 1/diag where |diag| > 1e-30, else 0
    double *x, *b, *r;
    const int32_t *map;             // this level -> next level (null at the coarsest)
    const int32_t *memOff, *mem;    // next level's members in this level, ascending
    const double *rec, *rds;        // packed rows (null: not packed) and their 1/diag (not level 0)
    bool shared;                    // x is in shared memory
    __device__ __forceinline__ double v(int j) const { return ent ? ldu[ent[j]] : val[j]; }
    __device__ __forceinline__ double d(int i) const { return ent ? ldu[i] : dg[i]; }
};

__device__ __forceinline__ RLevel ramg_level(const DevMesh &M, const DevInst &I, int l) {
    const RamgWork &W = I.rg;
    const int32_t *t = W.lev + l * kRamgLevInts;
    RLevel L;
    L.n = t[RL_N];
    L.ldu = I.diag;
    if (l == 0) {
        L.ptr = M.lev[0].rowPtr; L.col = M.lev[0].colIdx; L.ent = M.r0Ent;
        L.val = nullptr; L.dg = nullptr;
        L.wfOff = M.wf0Off; L.wfRows = M.wf0Rows; L.nWf = M.nWf0;
        L.x = W.xs ? W.xs : I.s;
        L.b = I.r; L.r = I.t; L.rd = W.rd;
    } else {
        L.ptr = W.ptr + t[RL_PTR]; L.col = W.col + t[RL_ENT]; L.ent = nullptr;
        L.val = W.val + t[RL_ENT]; L.dg = W.dg + t[RL_VEC];
        L.wfOff = W.wfOff + t[RL_WFO]; L.wfRows = W.wfRows + t[RL_VEC]; L.nWf = t[RL_NWF];
        L.x = W.xs ? W.xs + M.nC + t[RL_VEC] : W.x + t[RL_VEC];
        L.b = W.b + t[RL_VEC]; L.r = W.r + t[RL_VEC]; L.rd = W.rd + M.nC + t[RL_VEC];
    }
    L.map = t[RL_MAP] >= 0 ? W.map + t[RL_MAP] : nullptr;
    L.memOff = t[RL_MAP] >= 0 ? W.memOff + t[RL_MOFF] : nullptr;
    L.mem = t[RL_MAP] >= 0 ? W.mem + t[RL_MEM] : nullptr;
    L.rec = t[RL_REC] < 0 ? nullptr : l == 0 ? I.g[0] : I.amgVal + t[RL_REC];
    L.rds = W.cv + (l == 0 ? 0 : t[RL_VEC]);
    L.shared = W.xs != nullptr;
    return L;
}

// ---- CTA helpers ------------------------------------------------------------
__device__ __forceinline__ int ramg_warp_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Exclusive prefix sum of a[0..n) in place over the CTA; returns the total.
__device__ int ramg_scan(int32_t *a, int n) {
    __shared__ int sh[33];
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, w = t >> 5, nw = nt >> 5;
    const int chunk = (n + nt - 1) / nt;
    const int lo = min(n, t * chunk), hi = min(n, lo + chunk);
    int s = 0;
    for (int i = lo; i < hi; ++i) s += a[i];
    const int inc = ramg_warp_scan(s);
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        const int v = lane < nw ? sh[lane] : 0;
        const int vi = ramg_warp_scan(v);
        if (lane < nw) sh[lane] = vi - v;
        if (lane == 31) sh[32] = vi;
    }
    __syncthreads();
    int run = sh[w] + inc - s;
    for (int i = lo; i < hi; ++i) {
        const int v = a[i];
        a[i] = run;
        run += v;
    }
    const int total = sh[32];
    __syncthreads();
    return total;
}

// ---- smoother, residual, transfer (the CTA, or warp 0 when `wm`) ------------
struct RGroup {
    int rank, size;
    bool wm;
    __device__ __forceinline__ void sync() const {
        if (wm) __syncwarp();
        else __syncthreads();
    }
};

// CSRMatrix::gaussSeidelSweep (LinearSolver.hpp:328-337), wavefront by
// wavefront.  The reference divides by the diagonal and subtracts products;
// the sweeps multiply by the reciprocal formed once per setup and use fused
// multiply-adds (at most a unit in the last place per operation), which keeps
// the FP64 division and half of the FP64 instructions off the chain of
// dependent operations every wavefront waits for.
//
// A wavefront is a short dependent step (a few rows per warp, 4 to 5 entries
// each, 64 clocks per multiply-add), 4 sweeps of about 12 of them per level and
// 50 sweeps of about 7 on the coarsest: read row by row from the CSR arrays,
// the index, value and vector loads in front of each multiply-add took 1.5 us
// (39 rows) to 4.7 us (1920 rows) a wavefront.  With one warp to an SMSP every
// instruction and every wait on a load between two barriers counts, so the rows
// are packed (ramg_pack) as records in wavefront order, read with three to five
// 16-byte loads, and the two halves of the CTA take turns: while one half
// computes a wavefront the other one fetches its rows of the next and works out
// where their x are.  Between two barriers are left the x loads, the
// multiply-adds and a store.  Rows are padded with zeros in their own column
// (no branch per entry).  A coarsest level of up to 64 rows stays in the
// registers of warp 0 for all its sweeps.  The entries of a row past the
// eighth, and rows past the CTA's size, are read in place.
constexpr int kRowRegs = 8;
constexpr int kRec = 10;   // doubles per record of a coarse level: 8 values, 8 columns, by 16-byte parts
// x of a level, in shared memory (addresses of 32 bits) or global memory
template <bool SM> struct RX;
template <> struct RX<true> {
    using At = uint32_t;
    uint32_t base;
    __device__ __forceinline__ RX(const RLevel &L) : base((uint32_t)__cvta_generic_to_shared(L.x)) {}
    __device__ __forceinline__ At at(int i) const { return base + 8u * (unsigned int)i; }
    __device__ __forceinline__ static double get(At a) {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
        return v;
    }
    __device__ __forceinline__ static void put(At a, double v) {
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
    }
};
template <> struct RX<false> {
    using At = double *;
    double *base;
    __device__ __forceinline__ RX(const RLevel &L) : base(L.x) {}
    __device__ __forceinline__ At at(int i) const { return base + i; }
    __device__ __forceinline__ static double get(At a) { return *a; }
    __device__ __forceinline__ static void put(At a, double v) { *a = v; }
};
template <int W, bool SM>
struct RRow {
    double b, rd, val[W];
    typename RX<SM>::At to, from[W];
    int row;       // -1: nothing to store
    bool wide;     // more entries than W
};
template <int W, bool SM>
__device__ __forceinline__ void ramg_record(const RX<SM> &x, const double *rec, const double *rds, int n, int slot,
                                            RRow<W, SM> &R) {
    const double2 *p = reinterpret_cast<const double2 *>(rec) + slot;
#pragma unroll
    for (int k = 0; k < W / 2; ++k) {
        const double2 v = p[k * n];
        R.val[2 * k] = v.x;
        R.val[2 * k + 1] = v.y;
    }
    const double2 c = p[W / 2 * n];
    const unsigned int col[4] = {(unsigned int)__double2loint(c.x), (unsigned int)__double2hiint(c.x),
                                 (unsigned int)__double2loint(c.y), (unsigned int)__double2hiint(c.y)};
    R.rd = W == 4 ? c.y : rds[slot];
    R.wide = col[0] >> 15 & 1;
#pragma unroll
    for (int k = 0; k < W; ++k) R.from[k] = x.at(k & 1 ? col[k >> 1] >> 16 : col[k >> 1] & 0x7fffu);
}
// entries of a wide row i past the first kRowRegs off-diagonal ones (columns
// ascend, so the diagonal is before entry j when its column is past i)
__device__ __forceinline__ double ramg_rest(const RLevel &L, int i, double s) {
    const int j0 = L.ptr[i], j1 = L.ptr[i + 1];
    for (int j = j0 + kRowRegs; j < j1; ++j) {
        const int c = L.col[j];
        if (c != i && j - j0 - (c > i ? 1 : 0) >= kRowRegs) s = fma(-L.val[j], L.x[c], s);
    }
    return s;
}
// b minus the products of the row's first N entries
template <int N, int W, bool SM>
__device__ __forceinline__ double ramg_sum_first(const RRow<W, SM> &R) {
    double x[N];
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = RX<SM>::get(R.from[k]);
    double s = R.b;
#pragma unroll
    for (int k = 0; k < N; ++k) s = fma(-R.val[k], x[k], s);
    return s;
}
template <int W, bool SM>
__device__ __forceinline__ double ramg_sum(const RRow<W, SM> &R) {
    return ramg_sum_first<W>(R);
}
template <int W, bool SM>
__device__ __forceinline__ void ramg_relax(const RLevel &L, const RRow<W, SM> &R) {
    double s = ramg_sum(R);
    if (W == kRowRegs && R.wide) s = ramg_rest(L, R.row, s);
    RX<SM>::put(R.to, s * R.rd);
}
// The wavefronts of a level in the lanes of a warp (at most 32 of them):
// first slot and number of rows
struct RWaves {
    int off, num;
    __device__ __forceinline__ RWaves(const RLevel &L) {
        const int w = threadIdx.x & 31;
        off = w < L.nWf ? L.wfOff[w] : 0;
        num = w < L.nWf ? L.wfOff[w + 1] - off : 0;
    }
    __device__ __forceinline__ static int of(int v, int w) { return __shfl_sync(0xffffffffu, v, w); }
};
// All sweeps of a level of at most 64 rows on one warp: slot s of the
// wavefront order belongs to lane s % 32.  Wide rows keep up to kRowMore further
// entries, which only their wavefronts spend instructions on.  False (and
// nothing done): a row has more.
constexpr int kRowMore = 6;
template <bool SM>
__device__ __noinline__ bool ramg_gs_resident(const RLevel &L, int sweeps) {
    const RWaves T(L);
    const int lane = threadIdx.x & 31, nWf = L.nWf, n = L.n;
    const RX<SM> x(L);
    RRow<8, SM> R[2];
    double more[2][kRowMore];
    typename RX<SM>::At moreAt[2][kRowMore];
    int wave[2] = {-1, -1};
    unsigned int used[2] = {0, 0};   // wavefronts with rows in slots 0-31 / 32-63
    unsigned int wide[2] = {0, 0};   // ... and wide rows among them
    unsigned int past4[2] = {0, 0}, past6[2] = {0, 0};   // ... and rows of more than 4, 6 entries
    bool fits = true;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int slot = min(lane + 32 * h, n - 1);
        ramg_record(x, L.rec, L.rds, n, slot, R[h]);
        const int i = R[h].row = L.wfRows[slot];
        R[h].to = x.at(i);
        R[h].b = L.b[i];
#pragma unroll
        for (int k = 0; k < kRowMore; ++k) { more[h][k] = 0.0; moreAt[h][k] = R[h].to; }
        if (R[h].wide) {
            int k = 0;
            for (int j = L.ptr[i]; j < L.ptr[i + 1]; ++j) {
                if (L.col[j] == i || k++ < kRowRegs) continue;
                if (k > kRowRegs + kRowMore) fits = false;
#pragma unroll
                for (int q = 0; q < kRowMore; ++q)
                    if (q == k - 1 - kRowRegs) { more[h][q] = L.val[j]; moreAt[h][q] = x.at(L.col[j]); }
            }
        }
    }
    if (!__all_sync(0xffffffffu, fits)) return false;
    for (int w = 0; w < nWf; ++w) {
        const int o = RWaves::of(T.off, w), num = RWaves::of(T.num, w);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (o < 32 * h + 32 && o + num > 32 * h) used[h] |= 1u << w;
            const int slot = lane + 32 * h;
            const bool mine = slot >= o && slot < o + num;
            if (mine && nonzero64(R[h].rd)) wave[h] = w;
            if (__any_sync(0xffffffffu, mine && R[h].wide)) wide[h] |= 1u << w;
            const bool four = nonzero64(R[h].val[4]) || nonzero64(R[h].val[5]);
            const bool six = nonzero64(R[h].val[6]) || nonzero64(R[h].val[7]);
            if (__any_sync(0xffffffffu, mine && (four || six))) past4[h] |= 1u << w;
            if (__any_sync(0xffffffffu, mine && six)) past6[h] |= 1u << w;
        }
    }
    for (int t = 0; t < sweeps; ++t) {
        for (int w = 0; w < nWf; ++w) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (used[h] >> w & 1) {
                    // (a position whose entries are all zero leaves the sums as they are)
                    double s = past6[h] >> w & 1   ? ramg_sum_first<8>(R[h])
                               : past4[h] >> w & 1 ? ramg_sum_first<6>(R[h])
                                                   : ramg_sum_first<4>(R[h]);
                    if (wide[h] >> w & 1) {
#pragma unroll
                        for (int k = 0; k < kRowMore; ++k) s = fma(-more[h][k], RX<SM>::get(moreAt[h][k]), s);
                    }
                    s = s * R[h].rd;
                    if (wave[h] == w) RX<SM>::put(R[h].to, s);
                }
            }
            __syncwarp();
        }
    }
    return true;
}
// sweeps of a level over the CTA; W = 4: level 0.  Thread r of a half takes row
// r of the wavefronts of its half's turn and row r + half of the others.
template <int W, bool SM>
__device__ __noinline__ void ramg_gs_packed(const RLevel &L, int sweeps) {
    const RWaves T(L);
    const int nWf = L.nWf, n = L.n, nt = blockDim.x, half = nt >> 1, t0 = threadIdx.x;
    const int rank[2] = {t0, t0 < half ? t0 + half : t0 - half};
    const RX<SM> x(L);
    const double *__restrict__ b = L.b, *__restrict__ rds = L.rds, *__restrict__ rec = L.rec;
    const int32_t *__restrict__ rows = L.wfRows;
    auto read = [&](int slot, RRow<W, SM> &R) {
        const int row = rows[slot];
        ramg_record(x, rec, rds, n, slot, R);
        R.b = b[row];
        R.to = x.at(row);
        R.row = nonzero64(R.rd) ? row : -1;
    };
    auto fetch = [&](int w, int r, RRow<W, SM> &R) {
        const int num = RWaves::of(T.num, w), o = RWaves::of(T.off, w);
        R.row = -1;
        if (r < num) read(o + r, R);
    };
    auto plus = [nWf](int w, int d) { w += d; return w >= nWf ? w - nWf : w; };
    const int steps = sweeps * nWf;
    RRow<W, SM> R[2];
    int w = 0;
    const int two = nWf > 1 ? 2 % nWf : 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) fetch(plus(0, h % nWf), rank[h], R[h]);
    for (int t = 0; t < steps; t += 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (t + h < steps) {
                const int num = RWaves::of(T.num, w);
                if (R[h].row >= 0) ramg_relax(L, R[h]);
                if (num > nt) {
                    const int o = RWaves::of(T.off, w);
                    for (int r = rank[h] + nt; r < num; r += nt) {
                        RRow<W, SM> more;
                        read(o + r, more);
                        if (more.row >= 0) ramg_relax(L, more);
                    }
                }
                __syncthreads();
                fetch(plus(w, two), rank[h], R[h]);
                w = plus(w, 1);
            }
        }
    }
}
template <bool SM>
__device__ __forceinline__ bool ramg_gs_records(const RGroup &g, const RLevel &L, int sweeps) {
    // (level 0 has records of its own kind; a mesh of at most kRamgWarpRows
    // cells sweeps it on warp 0 from its CSR rows)
    if (g.wm) return !L.ent && L.n <= 64 && ramg_gs_resident<SM>(L, sweeps);
    if (L.ent) ramg_gs_packed<4, SM>(L, sweeps);
    else ramg_gs_packed<8, SM>(L, sweeps);
    return true;
}
__device__ __noinline__ void ramg_gs(const RGroup &g, const RLevel &L, int sweeps) {
    if (L.rec && (L.shared ? ramg_gs_records<true>(g, L, sweeps) : ramg_gs_records<false>(g, L, sweeps))) return;
    for (int t = 0; t < sweeps; ++t) {
        for (int w = 0; w < L.nWf; ++w) {
            for (int q = L.wfOff[w] + g.rank; q < L.wfOff[w + 1]; q += g.size) {
                const int i = L.wfRows[q];
                double s = L.b[i];
                for (int j = L.ptr[i]; j < L.ptr[i + 1]; ++j) {
                    const int c = L.col[j];
                    if (c != i) s = fma(-L.v(j), L.x[c], s);
                }
                const double ri = L.rd[i];
                if (ri != 0.0) L.x[i] = s * ri;
            }
            g.sync();
        }
    }
}

// CSRMatrix::residual (:318-326), then the restriction of the V-cycle
// (:571-575): coarse b = sum of the members' residuals in ascending row
// order, coarse x = 0.  A row's entries are fetched together.
__device__ __noinline__ void ramg_restrict(const RGroup &g, const RLevel &L, const RLevel &Cl) {
    // (locals: a store through one of the pointers would have the others read again)
    const int32_t *__restrict__ ptr = L.ptr, *__restrict__ col = L.col, *__restrict__ ent = L.ent;
    const double *__restrict__ vals = ent ? L.ldu : L.val, *__restrict__ x = L.x, *__restrict__ b = L.b;
    double *res = L.r;
    const int n = L.n, size = g.size, nc = Cl.n;
    for (int i = g.rank; i < n; i += size) {
        double s = 0.0;
        const int j1 = ptr[i + 1];
        for (int j = ptr[i]; j < j1; j += kRowRegs) {
            int at[kRowRegs];
            double v[kRowRegs], xv[kRowRegs];
#pragma unroll
            for (int k = 0; k < kRowRegs; ++k) at[k] = min(j + k, j1 - 1);
#pragma unroll
            for (int k = 0; k < kRowRegs; ++k) xv[k] = x[col[at[k]]];
#pragma unroll
            for (int k = 0; k < kRowRegs; ++k) v[k] = vals[ent ? ent[at[k]] : at[k]];
#pragma unroll
            for (int k = 0; k < kRowRegs; ++k)
                if (j + k < j1) s = fma(v[k], xv[k], s);
        }
        res[i] = b[i] - s;
    }
    g.sync();
    const int32_t *__restrict__ memOff = L.memOff, *__restrict__ mem = L.mem;
    double *cb = Cl.b, *cx = Cl.x;
    for (int J = g.rank; J < nc; J += size) {
        double s = 0.0;
        for (int q = memOff[J]; q < memOff[J + 1]; ++q) s += res[mem[q]];
        cb[J] = s;
        cx[J] = 0.0;
    }
    g.sync();
}

__device__ __noinline__ void ramg_prolong(const RGroup &g, const RLevel &L, const RLevel &Cl) {
    for (int i = g.rank; i < L.n; i += g.size) L.x[i] = L.x[i] + Cl.x[L.map[i]];
    g.sync();
}

// AMGSolver::vcycle (:553-589) over levels [l0, l1] (l1 the coarsest)
__device__ void ramg_vcycle_range(const RGroup &g, const DevMesh &M, const DevInst &I, int l0, int l1, bool down,
                                  bool up) {
    if (down) {
        for (int l = l0; l < l1; ++l) {
            const RLevel L = ramg_level(M, I, l), Cl = ramg_level(M, I, l + 1);
            ramg_gs(g, L, 2);
            ramg_restrict(g, L, Cl);
        }
    }
    if (down && up) {
        const RLevel Lc = ramg_level(M, I, l1);
        ramg_gs(g, Lc, kRamgCoarseSweeps);
    }
    if (up) {
        for (int l = l1 - 1; l >= l0; --l) {
            const RLevel L = ramg_level(M, I, l), Cl = ramg_level(M, I, l + 1);
            ramg_prolong(g, L, Cl);
            ramg_gs(g, L, 2);
        }
    }
}

// ---- hierarchy setup (AMGSolver::setup, :516-551) ---------------------------
// Wavefronts of a coarse level: depth by relaxation (ping-pong), then rows
// bucketed by depth.  Returns the wavefront count.
template <class T>
__device__ int ramg_wavefronts(T &tm, const RamgWork &W, const int32_t *ptr, const int32_t *col, int n,
                               int32_t *wfOff, int32_t *wfRows) {
    int32_t *a = W.aux, *b = W.aux2;
    for (int i = tm.rank(); i < n; i += tm.size()) a[i] = 0;
    tm.sync();
    for (int it = 0; it <= n; ++it) {
        bool changed = false;
        for (int i = tm.rank(); i < n; i += tm.size()) {
            int dd = 0;
            for (int j = ptr[i]; j < ptr[i + 1]; ++j) {
                const int c = col[j];
                if (c < i) dd = max(dd, a[c] + 1);
            }
            b[i] = dd;
            changed = changed || dd != a[i];
        }
        const bool again = __syncthreads_or(changed);
        int32_t *tmp = a; a = b; b = tmp;
        if (!again) break;
    }
    // a holds the depths; count, scan and place
    __shared__ int deepest;
    if (tm.leader()) deepest = 0;
    tm.sync();
    int mx = 0;
    for (int i = tm.rank(); i < n; i += tm.size()) mx = max(mx, a[i]);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(&deepest, mx);
    tm.sync();
    const int nWf = deepest + 1;
    for (int q = tm.rank(); q <= nWf; q += tm.size()) wfOff[q] = 0;
    tm.sync();
    for (int i = tm.rank(); i < n; i += tm.size()) atomicAdd(&wfOff[a[i]], 1);
    tm.sync();
    ramg_scan(wfOff, nWf + 1);
    for (int q = tm.rank(); q < nWf; q += tm.size()) b[q] = wfOff[q];
    tm.sync();
    for (int i = tm.rank(); i < n; i += tm.size()) wfRows[atomicAdd(&b[a[i]], 1)] = i;
    tm.sync();
    return nWf;
}

// Packs the rows of every level as records in wavefront order (the coarsest
// level first: its 50 sweeps are the longest chain).  Nothing is allocated for
// them.  The coarse levels take the place of the other AMG form's arrays, which
// an instance with this one does not use (amgVal up to gpart is one stretch of
// the slab), with their 1/diag in that of the Galerkin contributions.  Level 0 of
// a mesh of quadrilaterals (records of 6 doubles: 4 values, 4 columns, 1/diag)
// takes that of the velocity gradients, which the pressure correction leaves free
// (formed anew at the start of every outer iteration; `vel`: they are still
// needed).  A level that does not fit, or has more than 32 wavefronts, is swept
// from its CSR rows.
template <class T>
__device__ void ramg_pack(T &tm, const DevMesh &M, DevInst &I, int nLev, bool vel) {
    const RamgWork &W = I.rg;
    const int64_t cap = I.gpart - I.amgVal;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    int64_t used = 0;
    for (int l = nLev - 1; l >= 0; --l) {
        const RLevel L = ramg_level(M, I, l);
        if (L.nWf > 32 || L.n > 32767) continue;
        const int vec = l == 0 ? 0 : W.lev[l * kRamgLevInts + RL_VEC];
        if (l == 0 ? vel || M.maxCellFaces > 4 : used + (int64_t)kRec * L.n > cap || vec + L.n > M.nnz0) continue;
        double *rec = l == 0 ? I.g[0] : I.amgVal + used;
        for (int w = warp; w < L.nWf; w += nw) {
            const int o = L.wfOff[w], rows = L.wfOff[w + 1] - o;
            for (int r = lane; r < rows; r += 32) {
                const int i = L.wfRows[o + r];
                // entry k and column k of the record
                const int W8 = l == 0 ? 4 : kRowRegs, slot = o + r;
                auto val = [&](int k) -> double & { return rec[2 * ((size_t)(k >> 1) * L.n + slot) + (k & 1)]; };
                uint16_t *col = reinterpret_cast<uint16_t *>(rec + 2 * ((size_t)(W8 >> 1) * L.n + slot));
                int k = 0;
                for (int j = L.ptr[i]; j < L.ptr[i + 1]; ++j) {
                    const int c = L.col[j];
                    if (c == i) continue;
                    if (k < W8) {
                        val(k) = L.v(j);
                        col[k] = (uint16_t)c;
                    }
                    ++k;
                }
                if (k > W8) col[0] |= 0x8000;
                for (; k < W8; ++k) {
                    val(k) = 0.0;
                    col[k] = (uint16_t)i;
                }
                if (l == 0) rec[2 * ((size_t)2 * L.n + slot) + 1] = L.rd[i];
                else W.cv[vec + slot] = L.rd[i];
            }
        }
        if (threadIdx.x == 0) W.lev[l * kRamgLevInts + RL_REC] = (int)used;
        if (l > 0) used += (int64_t)kRec * L.n;
    }
    tm.sync();
}

// Builds levels 1.. from level 0 (whose values are the current system) and
// every level's reciprocal diagonals.  Returns the level count.
template <class T>
__device__ __noinline__ int ramg_setup(T &tm, const DevMesh &M, DevInst &I, bool vel) {
    const RamgWork &W = I.rg;
    const int n0 = M.nC;
    if (tm.leader()) {
        int32_t *t = W.lev;
        t[RL_N] = n0; t[RL_PTR] = 0; t[RL_ENT] = 0; t[RL_VEC] = 0; t[RL_MAP] = -1; t[RL_NWF] = M.nWf0; t[RL_REC] = -1;
    }
    for (int i = tm.rank(); i < n0; i += tm.size()) {
        const double d = I.diag[i];
        W.rd[i] = fabs(d) > 1e-30 ? 1.0 / d : 0.0;
    }
    tm.sync();
    int nLev = 1;
    int rowsUsed = 0, entsUsed = 0, ptrUsed = 0, wfoUsed = 0, mapUsed = 0, moffUsed = 0, memUsed = 0;
    for (int l = 0; l < kRamgMaxCoarsen; ++l) {
        const RLevel L = ramg_level(M, I, l);
        const int n = L.n;
        if (n <= kRamgMinCoarse) break;
        int32_t *claim = W.seed;
        // 1. seeds and claims, wavefront by wavefront
        for (int w = 0; w < L.nWf; ++w) {
            for (int q = L.wfOff[w] + tm.rank(); q < L.wfOff[w + 1]; q += tm.size()) {
                const int i = L.wfRows[q];
                const double ajj = fabs(L.d(i));
                int cl = -1;
                for (int j = L.ptr[i]; j < L.ptr[i + 1] && cl < 0; ++j) {
                    const int c = L.col[j];
                    if (c >= i) break;
                    if (claim[c] != -1) continue;   // c is not a seed
                    // the seed's own row entry for i decides (every occurrence)
                    const double aii = fabs(L.d(c));
                    for (int jj = L.ptr[c]; jj < L.ptr[c + 1]; ++jj) {
                        if (L.col[jj] != i) continue;
                        const double strength = fabs(L.v(jj)) / sqrt(aii * ajj + 1e-30);
                        if (strength > 0.25) { cl = c; break; }
                    }
                }
                claim[i] = cl;
            }
            tm.sync();
        }
        // 2. aggregate ids: the seeds' prefix count in row order
        int32_t *aid = W.aux;
        for (int i = tm.rank(); i < n; i += tm.size()) aid[i] = claim[i] == -1 ? 1 : 0;
        tm.sync();
        const int nc = ramg_scan(aid, n);
        if (nc == 0 || nc >= n) break;
        // a level that does not fit the pools ends the hierarchy here
        if (rowsUsed + nc > W.rowPool || memUsed + n > W.rowPool + n0 || mapUsed + n > W.rowPool + n0 ||
            moffUsed + nc + 1 > W.rowPool + 64 || ptrUsed + nc + 1 > W.rowPool + 64 ||
            wfoUsed + nc + 1 > W.rowPool + 64)
            break;
        // 3. map, member counts (seed + the rows it claimed, adjacent duplicates once)
        int32_t *map = W.map + mapUsed;
        int32_t *moff = W.memOff + moffUsed;
        for (int i = tm.rank(); i < n; i += tm.size()) map[i] = claim[i] == -1 ? aid[i] : aid[claim[i]];
        for (int i = tm.rank(); i < n; i += tm.size()) {
            if (claim[i] != -1) continue;
            int cnt = 1;
            for (int j = L.ptr[i]; j < L.ptr[i + 1]; ++j) {
                const int c = L.col[j];
                if (c > i && claim[c] == i && !(j > L.ptr[i] && L.col[j - 1] == c)) ++cnt;
            }
            moff[aid[i]] = cnt;
        }
        if (tm.leader()) moff[nc] = 0;
        tm.sync();
        ramg_scan(moff, nc + 1);
        int32_t *mem = W.mem + memUsed;
        for (int i = tm.rank(); i < n; i += tm.size()) {
            if (claim[i] != -1) continue;
            int at = moff[aid[i]];
            mem[at++] = i;
            for (int j = L.ptr[i]; j < L.ptr[i + 1]; ++j) {
                const int c = L.col[j];
                if (c > i && claim[c] == i && !(j > L.ptr[i] && L.col[j - 1] == c)) mem[at++] = c;
            }
        }
        tm.sync();
        // 4. Galerkin contributions in (member ascending, column ascending) order
        int32_t *coff = W.coff;
        for (int J = tm.rank(); J < nc; J += tm.size()) {
            int cnt = 0;
            for (int q = moff[J]; q < moff[J + 1]; ++q) cnt += L.ptr[mem[q] + 1] - L.ptr[mem[q]];
            coff[J] = cnt;
        }
        if (tm.leader()) coff[nc] = 0;
        tm.sync();
        ramg_scan(coff, nc + 1);
        for (int J = tm.rank(); J < nc; J += tm.size()) {
            int k = coff[J];
            for (int q = moff[J]; q < moff[J + 1]; ++q) {
                const int m = mem[q];
                for (int j = L.ptr[m]; j < L.ptr[m + 1]; ++j) {
                    W.cj[k] = map[L.col[j]];
                    W.cv[k] = L.v(j);
                    ++k;
                }
            }
            // sum equal coarse columns in arrival order (0.0 + first, as the
            // reference's default-constructed map entry), then sort by column
            const int o = coff[J], e = coff[J + 1];
            int dcount = 0;
            for (int kk = o; kk < e; ++kk) {
                const int Jc = W.cj[kk];
                const double vv = W.cv[kk];
                int p = o;
                while (p < o + dcount && W.cj[p] != Jc) ++p;
                if (p < o + dcount) {
                    W.cv[p] += vv;
                } else {
                    W.cj[o + dcount] = Jc;
                    W.cv[o + dcount] = 0.0 + vv;
                    ++dcount;
                }
            }
            for (int a = o + 1; a < o + dcount; ++a) {
                const int kc = W.cj[a];
                const double kv = W.cv[a];
                int b = a - 1;
                while (b >= o && W.cj[b] > kc) {
                    W.cj[b + 1] = W.cj[b];
                    W.cv[b + 1] = W.cv[b];
                    --b;
                }
                W.cj[b + 1] = kc;
                W.cv[b + 1] = kv;
            }
            W.aux2[J] = dcount;
        }
        tm.sync();
        // 5. the coarse CSR into the pools
        int32_t *cptr = W.ptr + ptrUsed;
        for (int J = tm.rank(); J < nc; J += tm.size()) cptr[J] = W.aux2[J];
        if (tm.leader()) cptr[nc] = 0;
        tm.sync();
        const int nnzc = ramg_scan(cptr, nc + 1);
        if (entsUsed + nnzc > W.entPool) break;
        int32_t *ccol = W.col + entsUsed;
        double *cval = W.val + entsUsed, *cdg = W.dg + rowsUsed;
        for (int J = tm.rank(); J < nc; J += tm.size()) {
            const int o = coff[J];
            double dJ = 0.0;
            for (int q = cptr[J]; q < cptr[J + 1]; ++q) {
                const int Jc = W.cj[o + q - cptr[J]];
                const double vv = W.cv[o + q - cptr[J]];
                ccol[q] = Jc;
                cval[q] = vv;
                if (Jc == J) dJ = vv;
            }
            cdg[J] = dJ;
            W.rd[n0 + rowsUsed + J] = fabs(dJ) > 1e-30 ? 1.0 / dJ : 0.0;
        }
        tm.sync();
        // 6. the new level's wavefronts
        int32_t *cwfo = W.wfOff + wfoUsed;
        const int nWf = ramg_wavefronts(tm, W, cptr, ccol, nc, cwfo, W.wfRows + rowsUsed);
        if (tm.leader()) {
            int32_t *t = W.lev + l * kRamgLevInts;
            t[RL_MAP] = mapUsed; t[RL_MOFF] = moffUsed; t[RL_MEM] = memUsed;
            int32_t *u = W.lev + (l + 1) * kRamgLevInts;
            u[RL_N] = nc; u[RL_PTR] = ptrUsed; u[RL_ENT] = entsUsed; u[RL_VEC] = rowsUsed; u[RL_MAP] = -1;
            u[RL_WFO] = wfoUsed; u[RL_NWF] = nWf; u[RL_NNZ] = nnzc; u[RL_REC] = -1;
        }
        mapUsed += n; moffUsed += nc + 1; memUsed += n;
        ptrUsed += nc + 1; entsUsed += nnzc; rowsUsed += nc; wfoUsed += nWf + 1;
        ++nLev;
        tm.sync();
    }
    tm.sync();
    ramg_pack(tm, M, I, nLev, vel);
    return nLev;
}

template <class T>
__device__ void ramg_vcycle(T &tm, const DevMesh &M, const DevInst &I, int nLev) {
    const int32_t *lev = I.rg.lev;
    int lw = nLev - 1;
    while (lw > 0 && lev[(lw - 1) * kRamgLevInts + RL_N] <= kRamgWarpRows) --lw;
    if (lev[lw * kRamgLevInts + RL_N] > kRamgWarpRows) lw = nLev;   // no level small enough
    const RGroup all{(int)threadIdx.x, (int)blockDim.x, false};
    if (lw == 0) {
        // every level is small: all of it on warp 0
        if (threadIdx.x < 32) {
            const RGroup w0{(int)threadIdx.x, 32, true};
            ramg_vcycle_range(w0, M, I, 0, nLev - 1, true, true);
        }
        __syncthreads();
        return;
    }
    if (lw < nLev) {
        ramg_vcycle_range(all, M, I, 0, lw, true, false);
        if (threadIdx.x < 32) {
            const RGroup w0{(int)threadIdx.x, 32, true};
            ramg_vcycle_range(w0, M, I, lw, nLev - 1, true, true);
        }
        __syncthreads();
        ramg_vcycle_range(all, M, I, 0, lw, false, true);
    } else {
        ramg_vcycle_range(all, M, I, 0, nLev - 1, true, true);
    }
}

// The V-cycle preconditioner z = M r on levels [0, nLev): level 0's b is I.r
// and the result z is left in I.s.  Levels from the first one of at most
// kRamgWarpRows rows down to the coarsest run on warp 0.  With the
// shared-memory copy of the level vectors (W.xs), level 0's x starts at zero
// there and is copied to I.s at the end; otherwise the caller zeroes I.s.
template <class T>
__device__ void ramg_precondition(T &tm, const DevMesh &M, const DevInst &I, int nLev) {
    if (I.rg.xs) {
        for (int c = threadIdx.x; c < M.nC; c += blockDim.x) I.rg.xs[c] = 0.0;
        __syncthreads();
    }
    ramg_vcycle(tm, M, I, nLev);
    if (I.rg.xs) {
        for (int c = threadIdx.x; c < M.nC; c += blockDim.x) I.s[c] = I.rg.xs[c];
        __syncthreads();
    }
}

}  // namespace btm
