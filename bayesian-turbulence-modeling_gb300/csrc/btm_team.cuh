// btm_team.cuh - execution teams shared by the FP64 and mixed-precision
// engines: one CTA (BlockTeam) or a whole cooperative grid (GridTeam);
// deterministic fixed-order team reductions and a bounded software grid
// barrier.  Header-only device code.
#pragma once
#include "btm_common.h"

#include <cuda_runtime.h>
#include <stdint.h>

namespace btm {

// std::max / std::min selection semantics (first argument on ties and NaN)
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ float smaxf(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float sminf(float a, float b) { return (b < a) ? b : a; }

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr uint64_t kBarrierTimeoutNs = 2000000000ull;  // 2 s: a stuck barrier aborts the solve

// ---------------------------------------------------------------------------
// teams
// ---------------------------------------------------------------------------
// FP64 reductions over one CTA.  A GB300 SM sub-partition (SMSP) holds its
// FP64 unit for 64 clocks per warp instruction, whatever the number of active
// lanes and however independent the instructions are (measured: 63.9 clocks
// per dependent and per independent addition of one warp, 152 with two warps
// on the SMSP).  What a reduction costs is therefore its FP64 warp
// instructions, and a butterfly in every warp followed by a fold of all warp
// partials in every thread spends most of them on copies of the same sums.
// Here every warp does only the first step of its butterfly (two values at
// once: each half of the lanes goes on with one of them) and leaves the 16
// sums of each value in shared memory; half of the warps finish two source
// warps each (16 lanes per source, later 8 per value: no addition is done
// twice), and one warp adds the per-warp totals in warp order.  The additions,
// their pairing and their order are those of the butterfly and the fold, so
// the totals are the same bits.
//
// Shared memory: `red` [threads] doubles, shared with the FP32 reductions
// (hence the barrier in front), and `tot` [2][warps] + kRedResults: totals,
// results.
struct RedAdd {
    __device__ __forceinline__ static double op(double a, double b) { return a + b; }
    __device__ __forceinline__ static double first(const double *) { return 0.0; }
};
struct RedMax {   // smax: the first operand survives ties and NaN
    __device__ __forceinline__ static double op(double a, double b) { return smax(a, b); }
    __device__ __forceinline__ static double first(const double *p) { return __ldcg(p); }
};

// The folding warp goes on to `f(lane, t0, t1)`, the scalars that follow from
// the totals (all its lanes call it; lane q < NOUT leaves result q): a
// division costs 8 to 9 FP64 instructions, and formed in every warp of the
// CTA they took as long as the matrix products of a BiCGSTAB iteration.  Both
// together: 4x32 channel, one CTA, 13.4 -> 6.5 us a BiCGSTAB iteration.
constexpr int kRedResults = 6;
template <int N, class Op, int NOUT, class F>
__device__ __forceinline__ void block_reduce(double *red, double *tot, double *v, int turn, int live, double *out, F f) {
    static_assert((N == 1 || N == 2) && NOUT <= kRedResults, "one or two values at a time");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    double *res = tot + 2 * nw;
    double h;
    if (N == 2) {
        const bool second = lane >= 16;
        const double got = __shfl_xor_sync(0xffffffffu, second ? v[0] : v[1], 16);
        h = second ? Op::op(got, v[1]) : Op::op(v[0], got);
    } else {
        h = Op::op(v[0], __shfl_xor_sync(0xffffffffu, v[0], 16));
    }
    __syncthreads();
    if (N == 2 || lane < 16) red[warp * (16 * N) + lane] = h;   // [warp][value][16]
    __syncthreads();
    if (2 * warp < nw) {
        const int src = 2 * warp + (lane >> 4), l = lane & 15;
        double x;
        if (N == 2) {
            // lanes 0-7 of a source take the first value, 8-15 the second
            const double *e = red + src * 32 + (l >> 3) * 16 + (l & 7);
            x = Op::op(e[0], e[8]);
        } else {
            const double own = red[src * 16 + l];
            x = Op::op(own, __shfl_xor_sync(0xffffffffu, own, 8));
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) x = Op::op(x, __shfl_xor_sync(0xffffffffu, x, o));
        if (l == 0) tot[src] = x;
        if (N == 2 && l == 8) tot[nw + src] = x;
        // the folding warp (another one each time: a warp stays on its SMSP)
        // waits for the totals, the other warps for the result only
        asm volatile("bar.sync 1, %0;" ::"r"(nw << 4) : "memory");
        if (warp == (turn & 3)) {
            const double *t = tot + (lane < N ? lane * nw : 0);
            double s = t[0];
            for (int q = 1; q < live; ++q) s = Op::op(s, t[q]);
            const double t0 = __shfl_sync(0xffffffffu, s, 0), t1 = N == 2 ? __shfl_sync(0xffffffffu, s, 1) : 0.0;
            const double r = f(lane, t0, t1);
            if (lane < NOUT) res[lane] = r;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NOUT; ++j) out[j] = res[j];
}
template <int N, class Op>
__device__ __noinline__ void block_totals(double *red, double *tot, double *v, int turn, int live) {
    block_reduce<N, Op, N>(red, tot, v, turn, live, v, [](int lane, double t0, double t1) { return lane == 0 ? t0 : t1; });
}


__device__ __forceinline__ int live_warps(int nC) { return max(1, min((int)(blockDim.x >> 5), (nC + 31) >> 5)); }

struct BlockTeam {
    double *red;   // shared [max(threads, 2 * 32 * kRedSlots)]
    int buf;
    double *tot;   // shared [2 * warps + kRedResults]
    int turn;
    int live;      // warps that own cells: the others only ever add zeros to a sum
    __device__ __forceinline__ int rank() const { return threadIdx.x; }
    __device__ __forceinline__ int spread() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }
    __device__ __forceinline__ bool sync() { __syncthreads(); return true; }
    __device__ __forceinline__ bool ok() const { return true; }

    template <int N, class Op>
    __device__ __forceinline__ void reduce(double *v, int warps) {
        if constexpr (N > 2) {
            reduce<2, Op>(v, warps);
            reduce<N - 2, Op>(v + 2, warps);
        } else {
            block_totals<N, Op>(red, tot, v, turn++, warps);
        }
    }
    // Sum N values over the team; every thread receives the identical totals.
    template <int N>
    __device__ __forceinline__ void sum(double *v) { reduce<N, RedAdd>(v, live); }
    template <int N>
    __device__ __forceinline__ void maxr(double *v) { reduce<N, RedMax>(v, blockDim.x >> 5); }
    template <int N>
    __device__ __forceinline__ void sumd(double *v) { reduce<N, RedAdd>(v, live); }
    // Sums N values and leaves f(q, t0, t1) of the totals in out[q], q < NOUT,
    // in every thread; one warp evaluates f.
    template <int N, int NOUT, class F>
    __device__ __forceinline__ void sum_then(double *v, double *out, F f) {
        block_reduce<N, RedAdd, NOUT>(red, tot, v, turn++, live, out, f);
    }
    // The same for warp 0's values f(lane) that need no reduction
    template <int NOUT, class F>
    __device__ __forceinline__ void once(double *out, F f) {
        double *res = tot + 2 * (blockDim.x >> 5);
        __syncthreads();
        if (threadIdx.x < 32) {
            const double r = f((int)threadIdx.x);
            if (threadIdx.x < NOUT) res[threadIdx.x] = r;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NOUT; ++j) out[j] = res[j];
    }

    // FP32 sums (Krylov dot products of the mixed-precision engine): a warp
    // butterfly, then every warp re-reduces the per-warp partials with the
    // same butterfly, so all threads hold identical totals after one barrier.
    // The fold stays in FP32: on GB300 a chain of dependent FP64 additions per
    // reduction doubled the BiCGSTAB time, and pairwise FP32 summation of at
    // most 16k products is accurate to ~1e-6, far inside what the Krylov
    // scalars need (the equation defects themselves are FP64).
    template <int N>
    __device__ __forceinline__ void sumf(float *v) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        float *rb = reinterpret_cast<float *>(red + buf * 32 * kRedSlots);   // [slot][warp]
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < N; ++j) rb[j * 32 + warp] = v[j];
        __syncthreads();
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float s = lane < nw ? rb[j * 32 + lane] : 0.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            v[j] = s;
        }
        buf ^= 1;
    }
    // FP32 maxima with smax semantics (a NaN in the first operand survives)
    template <int N>
    __device__ __forceinline__ void maxf(float *v) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] = smaxf(v[j], __shfl_xor_sync(0xffffffffu, v[j], o));
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        float *rb = reinterpret_cast<float *>(red + buf * 32 * kRedSlots);
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < N; ++j) rb[warp * kRedSlots + j] = v[j];
        __syncthreads();
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float s = rb[j];
            for (int q = 1; q < nw; ++q) s = smaxf(s, rb[q * kRedSlots + j]);
            v[j] = s;
        }
        buf ^= 1;
    }
};

// One CTA per instance whose AMG solves use the reference-order AMG
// (btm_ramg.cuh).  A distinct type so that only the kernel instantiated for
// it carries that solver in its call graph (the plain kernel keeps its
// register allocation).
struct BlockTeamRef : BlockTeam {};

struct GridTeam {
    double *red;            // shared [2][32][kRedSlots]
    int buf;
    double *gpart;          // global [2][gridDim][kRedSlots]
    unsigned int *bar;      // arrivals since the launch (zeroed before it)
    int32_t *err;
    int *shAbort;           // shared flag
    unsigned int target;    // thread 0: arrivals that complete the next barrier
    __device__ __forceinline__ int rank() const { return blockIdx.x * blockDim.x + threadIdx.x; }
    // The same ranks dealt out warp by warp over the CTAs, for passes that end
    // in no reduction (a sum's bits depend on who owns what): with rank() a
    // 1,257-row level runs on 3 SMs, 16 warps deep in their FP64 units, and the
    // last pass over any array fills some SMs and leaves the others idle.
    __device__ __forceinline__ int spread() const {
        return (int)(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) << 5 | (threadIdx.x & 31));
    }
    __device__ __forceinline__ int size() const { return gridDim.x * blockDim.x; }
    __device__ __forceinline__ bool leader() const { return blockIdx.x == 0 && threadIdx.x == 0; }
    __device__ __forceinline__ bool ok() const { return *shAbort == 0; }

    // Software grid barrier for a cooperative launch (all CTAs co-resident):
    // one release arrival per CTA on a counter that only grows, acquire polls
    // of that counter (its wrap-around is harmless: the difference to the
    // target is what counts).  A barrier is nothing but latency, one L2
    // round trip for the arrival and one for the poll that sees the last; a
    // clock read, a nanosleep or a second flag in every poll adds its own.
    // Every wait is bounded: each kPollsPerCheck polls the CTA looks at the
    // error flag and the clock, and after kBarrierTimeoutNs it flags the error
    // and the whole team abandons the solve.  A CTA that has abandoned it no
    // longer arrives.
    //
    // 152 CTAs of 512 threads: 1.44 us a barrier.
    //
    // arrive() and wait() are its two halves: loads that do not depend on what
    // the other CTAs are still writing go between them.
    __device__ __noinline__ void arrive() {
        __syncthreads();
        if (threadIdx.x == 0 && *shAbort == 0) {
            target += gridDim.x;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        }
    }
    __device__ __noinline__ bool wait() {
        if (threadIdx.x == 0 && *shAbort == 0) {
            uint64_t t0 = 0;
            for (unsigned int polls = 1;; ++polls) {
                unsigned int now;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(bar) : "memory");
                if ((int)(now - target) >= 0) break;
                if ((polls & (kPollsPerCheck - 1)) == 0) {
                    if (*(volatile int32_t *)err) { *shAbort = 1; break; }
                    const uint64_t t = globaltimer_ns();
                    if (t0 == 0) {
                        t0 = t;
                    } else if (t - t0 > kBarrierTimeoutNs) {
                        atomicExch(err, 2);
                        *shAbort = 1;
                        break;
                    }
                }
            }
        }
        __syncthreads();
        return *shAbort == 0;
    }
    __device__ __forceinline__ bool sync() {
        arrive();
        return wait();
    }
    static constexpr unsigned int kPollsPerCheck = 256;

    // Totals of N values whose per-warp totals are in rb[warp][value] (shared,
    // visible after the first barrier here): warp 0 adds them in warp order,
    // lane j the j-th value; after the grid barrier warp j folds the CTAs'
    // partials of value j (each lane a fixed strided subset, then a
    // butterfly) for its CTA.  The order of the operations is that of a fold
    // in every thread; one warp does them, because an FP64 warp instruction
    // holds its SMSP for 64 clocks.
    template <int N, class Op, int NOUT, class F>
    __device__ __forceinline__ void fold_then(double *out, F f) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        double *rb = red + buf * 32 * kRedSlots;
        __syncthreads();
        if (warp == 0 && lane < N) {
            const int nw = blockDim.x >> 5;
            double s = rb[lane];
            for (int q = 1; q < nw; ++q) s = Op::op(s, rb[q * kRedSlots + lane]);
            gpart[((size_t)buf * gridDim.x + blockIdx.x) * kRedSlots + lane] = s;
        }
        sync();
        double *tot = rb + 31 * kRedSlots, *res = rb + 29 * kRedSlots;
        if (warp < N) {
            const double *gp = gpart + (size_t)buf * gridDim.x * kRedSlots + warp;
            double s = Op::first(gp);
            // all loads before the additions
            for (int q0 = lane; q0 < (int)gridDim.x; q0 += 32 * 8) {
                double p[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) p[i] = __ldcg(gp + (size_t)min(q0 + 32 * i, (int)gridDim.x - 1) * kRedSlots);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (q0 + 32 * i < (int)gridDim.x) s = Op::op(s, p[i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s = Op::op(s, __shfl_xor_sync(0xffffffffu, s, o));
            if (lane == 0) tot[warp] = s;
        }
        if (N > 1) __syncthreads();
        if (warp == 0) {
            __syncwarp();
            const double r = f(lane, tot[0], N > 1 ? tot[1] : 0.0);
            if (lane < NOUT) res[lane] = r;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NOUT; ++j) out[j] = res[j];
        buf ^= 1;
    }
    template <int N, class Op>
    __device__ __noinline__ void fold(double *v) {
        fold_then<N, Op, N>(v, [this](int lane, double, double) {
            return red[buf * 32 * kRedSlots + 31 * kRedSlots + (lane < N ? lane : 0)];
        });
    }
    // warp totals of N values into rb[warp][value]
    template <int N>
    __device__ __forceinline__ void leave(double *v) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int j = 0; j < N; ++j) red[buf * 32 * kRedSlots + (threadIdx.x >> 5) * kRedSlots + j] = v[j];
    }
    template <int N, int NOUT, class F>
    __device__ __forceinline__ void sum_then(double *v, double *out, F f) {
        leave<N>(v);
        fold_then<N, RedAdd, NOUT>(out, f);
    }
    template <int NOUT, class F>
    __device__ __forceinline__ void once(double *out, F f) {
        double *res = red + buf * 32 * kRedSlots + 29 * kRedSlots;
        __syncthreads();
        if (threadIdx.x < 32) {
            const double r = f((int)threadIdx.x);
            if (threadIdx.x < NOUT) res[threadIdx.x] = r;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NOUT; ++j) out[j] = res[j];
        buf ^= 1;
    }
    template <int N>
    __device__ void sum(double *v) {
        leave<N>(v);
        fold<N, RedAdd>(v);
    }
    template <int N>
    __device__ void maxr(double *v) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] = smax(v[j], __shfl_xor_sync(0xffffffffu, v[j], o));
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int j = 0; j < N; ++j) red[buf * 32 * kRedSlots + (threadIdx.x >> 5) * kRedSlots + j] = v[j];
        fold<N, RedMax>(v);
    }
    // FP32 values, FP64 accumulation from the warp totals up
    template <int N>
    __device__ void sumf(float *v) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int j = 0; j < N; ++j) red[buf * 32 * kRedSlots + (threadIdx.x >> 5) * kRedSlots + j] = (double)v[j];
        double d[N];
        fold<N, RedAdd>(d);
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = (float)d[j];
    }
    template <int N>
    __device__ void sumd(double *v) { sum<N>(v); }
    template <int N>
    __device__ void maxf(float *v) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] = smaxf(v[j], __shfl_xor_sync(0xffffffffu, v[j], o));
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int j = 0; j < N; ++j) red[buf * 32 * kRedSlots + (threadIdx.x >> 5) * kRedSlots + j] = (double)v[j];
        double d[N];
        fold<N, RedMax>(d);
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = (float)d[j];
    }
};

// Loads that must see writes made by other CTAs in the same launch (after a
// grid barrier) bypass L1: in grid mode every field read goes through __ldcg.
// In block mode one CTA owns the data and plain loads are coherent.
template <class T> struct Ld;
template <> struct Ld<BlockTeam> {
    __device__ __forceinline__ static double f(const double *p) { return *p; }
    __device__ __forceinline__ static float f(const float *p) { return *p; }
};
template <> struct Ld<BlockTeamRef> : Ld<BlockTeam> {};
template <> struct Ld<GridTeam> {
    __device__ __forceinline__ static double f(const double *p) { return __ldcg(p); }
    __device__ __forceinline__ static float f(const float *p) { return __ldcg(p); }
};
#define LD(ptr) (Ld<T>::f(ptr))

// ---------------------------------------------------------------------------
// Rows of the sparse systems.  y + sum_k a_k x_k (minus with Neg), one fused
// multiply-add per entry in the order of the row.  A row's entries are fetched
// W at a time: first all columns, then all coefficients and all x, then the
// chain of multiply-adds.  An entry at a time, every x waits for its column
// and the next entry for the branch on the side of the face: two cache (on the
// grid: L2) latencies per entry.  123k-cell step on the grid: V-cycle 0.44 ->
// 0.33 ms; 4x32 channel, one CTA: p' solve 165 -> 145 us an outer iteration.
// ---------------------------------------------------------------------------
// v != 0 (and not -0) without an FP64 comparison
__device__ __forceinline__ bool nonzero64(double v) { return (__double_as_longlong(v) << 1) != 0; }
__device__ __forceinline__ double fma_any(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_any(float a, float b, float c) { return fmaf(a, b, c); }

// The row tables of a mesh as locals: DevMesh and DevInst live in shared memory,
// where every store through a pointer has their fields read again.
struct RowTab {
    const int32_t *ent, *col;
    int nC, width;
    __device__ __forceinline__ explicit RowTab(const DevMesh &M)
        : ent(M.rowEnt), col(M.rowCol), nC(M.nC), width(M.rowW) {}
};

// Off-diagonal part of row c of an LDU system `sys` = diag | upper | lower, in
// ascending face order (entries and columns of all rows by position in the
// row, [rowW][nC], so neighbouring threads read neighbouring words; -1: no
// entry).
template <class T, bool Neg, int W, class V>
__device__ __forceinline__ V ldu_off_w(const RowTab &R, const V *sys, const V *x, int c, V y) {
    for (int w0 = 0; w0 < R.width; w0 += W) {
        int col[W], ent[W];
        V a[W], v[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const bool in = w0 + k < R.width;
            const size_t at = (size_t)(in ? w0 + k : 0) * R.nC + c;
            col[k] = in ? R.col[at] : -1;
            ent[k] = R.ent[at];
        }
#pragma unroll
        for (int k = 0; k < W; ++k) {
            a[k] = LD(sys + ent[k]);
            v[k] = LD(x + max(col[k], 0));
        }
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (col[k] >= 0) y = fma_any(Neg ? -a[k] : a[k], v[k], y);
    }
    return y;
}
template <class T, bool Neg, class V>
__device__ __forceinline__ V ldu_off(const RowTab &R, const V *sys, const V *x, int c, V y) {
    // quadrilaterals have up to 4 faces, hexahedra 6
    return R.width <= 4 ? ldu_off_w<T, Neg, 4>(R, sys, x, c, y) : ldu_off_w<T, Neg, 6>(R, sys, x, c, y);
}
template <class T, bool Neg, class V>
__device__ __forceinline__ V ldu_off(const DevMesh &M, const V *sys, const V *x, int c, V y) {
    return ldu_off<T, Neg>(RowTab(M), sys, x, c, y);
}

struct CsrTab {
    const int32_t *rowPtr, *colIdx;
    __device__ __forceinline__ CsrTab(const AmgLevelDev &L) : rowPtr(L.rowPtr), colIdx(L.colIdx) {}
};
// Row i of a CSR level without its column `skip` (-1: all of it), W entries at a
// time (an FP64 multiply-add that no lane needs takes its 64 clocks all the
// same: W should fit the level's longest row).
template <class T, bool Neg, int W = 8, class V>
__device__ __forceinline__ V csr_off(const CsrTab &L, const V *val, const V *x, int i, int skip, V y) {
    const int q1 = L.rowPtr[i + 1];
    for (int q = L.rowPtr[i]; q < q1; q += W) {
        int col[W];
        V a[W], v[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int at = min(q + k, q1 - 1);
            col[k] = L.colIdx[at];
            a[k] = LD(val + at);
        }
#pragma unroll
        for (int k = 0; k < W; ++k) v[k] = LD(x + col[k]);
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (q + k < q1 && col[k] != skip) y = fma_any(Neg ? -a[k] : a[k], v[k], y);
    }
    return y;
}

}  // namespace btm
