// Device functions of the engine behind plain entry points, for
// test_gpu_device_units.py: one function each, without a solve around it.
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_common.h"
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_team.cuh"
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_phases64.cuh"
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_dense.cuh"
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_cycle.cuh"

#include <cuda_runtime.h>
#include <vector>

using namespace btm;

__global__ void k_div(const double *x, const double *d, const double *r, double *q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = div_by(x[i], d[i], r[i]);
}

// below[i][j] = residual_below(sq[i][j], limit(r0[i], tol[i]), ...): one warp per i
__global__ void k_limit(const double *r0, const double *tol, const double *sq, int m, int *below, double *limit) {
    const int i = blockIdx.x, lane = threadIdx.x;
    const double l = residual_limit(r0[i], tol[i]);
    if (lane == 0) limit[i] = l;
    for (int j = lane; j < m; j += 32)
        below[(size_t)i * m + j] = residual_below(sq[(size_t)i * m + j], l, r0[i], tol[i]);
}

constexpr int kThreads = 512;
struct GridMem {
    double *gpart;
    unsigned int *bar;
    int32_t *err;
};
__global__ void __launch_bounds__(kThreads, 1) k_inverse_grid(double *A, double *work, int n, GridMem g, int *ok) {
    __shared__ double red[2 * 32 * kRedSlots];
    __shared__ int shAbort;
    if (threadIdx.x == 0) shAbort = 0;
    __syncthreads();
    GridTeam tm{red, 0, g.gpart, g.bar, g.err, &shAbort, 0u};
    const bool good = dense_inverse(tm, A, work, n);
    if (threadIdx.x == 0) ok[blockIdx.x] = good;
}
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_inverse_block(double *A, int n, int *ok) {
    __shared__ double red[NT > 2 * 32 * kRedSlots ? NT : 2 * 32 * kRedSlots];
    __shared__ double tot[2 * (NT / 32) + kRedResults];
    BlockTeam tm{red, 0, tot, 0, live_warps(n)};
    const bool good = dense_inverse(tm, A, nullptr, n);
    if (threadIdx.x == 0) ok[0] = good;
}

// a hierarchy as the V-cycle takes it, arrays of all levels one after the other
template <class VT>
struct Levels {
    using V = VT;
    static constexpr V kWeight = (V)0.7;
    DevMesh M;
    const V *matrix;               // diag | upper | lower of level 0
    V *xs, *bs, *rs, *rds, *vals;
    int at[kMaxLevels];            // a level's place in xs, bs, rs, rds
    const double *inverse;
    __device__ int levels() const { return M.nLevels; }
    __device__ bool direct() const { return M.coarseDirect != 0; }
    __device__ const AmgLevelDev &lev(int l) const { return M.lev[l]; }
    __device__ RowTab rows() const { return RowTab(M); }
    __device__ V *x(int l) const { return xs + at[l]; }
    __device__ V *b(int l) const { return bs + at[l]; }
    __device__ V *r(int l) const { return rs + at[l]; }
    __device__ V *rd(int l) const { return rds + at[l]; }
    __device__ V *val(int l) const { return vals + M.lev[l].valOff; }
    __device__ const V *sys() const { return matrix; }
    __device__ const double *ainv() const { return inverse; }
};
template <class V>
__global__ void __launch_bounds__(kThreads, 1) k_vcycle(const Levels<V> *levels, GridMem g) {
    __shared__ double red[2 * 32 * kRedSlots];
    __shared__ int shAbort;
    if (threadIdx.x == 0) shAbort = 0;
    __syncthreads();
    GridTeam tm{red, 0, g.gpart, g.bar, g.err, &shAbort, 0u};
    Cycle<GridTeam, Levels<V>>::run(tm, *levels);
}

namespace {
// device copies of a call's arrays, freed when it returns
struct Mem {
    std::vector<void *> all;
    cudaError_t e = cudaSuccess;
    template <class T>
    T *get(size_t n, const T *from = nullptr) {
        void *p = nullptr;
        const size_t bytes = sizeof(T) * (n ? n : 1);
        if (e == cudaSuccess) e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) return nullptr;
        all.push_back(p);
        e = from ? cudaMemcpy(p, from, sizeof(T) * n, cudaMemcpyHostToDevice) : cudaMemset(p, 0, bytes);
        return (T *)p;
    }
    template <class T>
    void back(T *to, const T *from, size_t n) {
        if (e == cudaSuccess) e = cudaMemcpy(to, from, sizeof(T) * n, cudaMemcpyDeviceToHost);
    }
    void launched() {
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    ~Mem() {
        for (void *p : all) cudaFree(p);
    }
};
}  // namespace

extern "C" {

int unit_div_by(int n, const double *x, const double *d, const double *r, double *q) {
    Mem M;
    double *dx = M.get(n, x), *dd = M.get(n, d), *dr = M.get(n, r), *dq = M.get<double>(n);
    if (M.e != cudaSuccess) return (int)M.e;
    k_div<<<(n + 255) / 256, 256>>>(dx, dd, dr, dq, n);
    M.launched();
    M.back(q, dq, n);
    return (int)M.e;
}

int unit_residual_limit(int n, int m, const double *r0, const double *tol, const double *sq, int *below,
                        double *limit) {
    Mem M;
    double *dr = M.get(n, r0), *dt = M.get(n, tol), *ds = M.get((size_t)n * m, sq), *dl = M.get<double>(n);
    int *db = M.get<int>((size_t)n * m);
    if (M.e != cudaSuccess) return (int)M.e;
    k_limit<<<n, 32>>>(dr, dt, ds, m, db, dl);
    M.launched();
    M.back(below, db, (size_t)n * m);
    M.back(limit, dl, n);
    return (int)M.e;
}

// A [n][n] to its inverse, in place.  blocks > 0: on a cooperative grid of that
// many CTAs (all co-resident: one to an SM); 0: on one CTA of `threads`.
// ok: the outcome of every CTA.
int unit_dense_inverse(int blocks, int threads, int n, double *A, int *ok) {
    Mem M;
    double *dA = M.get((size_t)n * n, A), *work = M.get<double>((size_t)2 * kPanel * n);
    int *dOk = M.get<int>(blocks > 0 ? blocks : 1);
    GridMem g{M.get<double>((size_t)2 * (blocks > 0 ? blocks : 1) * kRedSlots), M.get<unsigned int>(1),
              M.get<int32_t>(1)};
    if (M.e != cudaSuccess) return (int)M.e;
    if (blocks > 0) {
        void *args[] = {&dA, &work, &n, &g, &dOk};
        M.e = cudaLaunchCooperativeKernel((const void *)k_inverse_grid, dim3(blocks), dim3(kThreads), args, 0, 0);
    } else if (n > kCoarseDirect) {
        return -1;
    } else if (threads == 256) {
        k_inverse_block<256><<<1, 256>>>(dA, n, dOk);
    } else {
        k_inverse_block<512><<<1, 512>>>(dA, n, dOk);
    }
    M.launched();
    M.back(A, dA, (size_t)n * n);
    M.back(ok, dOk, blocks > 0 ? blocks : 1);
    int32_t err = 0;
    M.back(&err, g.err, 1);
    return M.e != cudaSuccess ? (int)M.e : err ? -2 : 0;
}

}  // extern "C"

namespace {
// sizes: nLevels, direct, nC, rowW; per level n, nColors
// and the places of rowPtr, colIdx, map, aggOff, aggMem, colorOff, colorRows in
// `ints` and of its values in `vals`; then those of rowEnt and rowCol.
template <class V>
int vcycle(int blocks, const int64_t *sizes, const int32_t *ints, int64_t nInts, const double *vals, int64_t nVals,
           const double *matrix, int64_t nMatrix, const double *rds, const double *inverse, int64_t nInverse,
           const double *b, double *x) {
    Mem M;
    auto as = [&](const double *p, int64_t n) { return std::vector<V>(p, p + n); };
    Levels<V> L{};
    DevMesh &D = L.M;
    const int nl = D.nLevels = (int)sizes[0];
    D.coarseDirect = (int)sizes[1];
    D.nC = (int)sizes[2];
    D.rowW = (int)sizes[3];
    const int32_t *di = M.get((size_t)nInts, ints);
    int64_t rows = 0;
    for (int l = 0; l < nl; ++l) {
        const int64_t *q = sizes + 4 + 10 * l;
        AmgLevelDev &v = D.lev[l];
        v.n = (int)q[0];
        v.nColors = (int)q[1];
        const int32_t **to[] = {&v.rowPtr, &v.colIdx, &v.map, &v.aggOff, &v.aggMem, &v.colorOff, &v.colorRows};
        for (int k = 0; k < 7; ++k) *to[k] = di + q[2 + k];
        v.valOff = q[9];
        L.at[l] = (int)rows;
        rows += v.n;
    }
    D.rowEnt = di + sizes[4 + 10 * nl];
    D.rowCol = di + sizes[5 + 10 * nl];
    const std::vector<V> hv = as(vals, nVals), hm = as(matrix, nMatrix), hr = as(rds, rows), hb = as(b, D.nC);
    L.vals = M.get(hv.size(), hv.data());
    L.matrix = M.get(hm.size(), hm.data());
    L.rds = M.get(hr.size(), hr.data());
    L.inverse = M.get((size_t)nInverse, inverse);
    L.xs = M.get<V>(rows);
    L.rs = M.get<V>(rows);
    L.bs = M.get<V>(rows);
    if (M.e == cudaSuccess) M.e = cudaMemcpy(L.bs, hb.data(), sizeof(V) * D.nC, cudaMemcpyHostToDevice);
    const Levels<V> *dL = M.get(1, &L);
    GridMem g{M.get<double>((size_t)2 * blocks * kRedSlots), M.get<unsigned int>(1), M.get<int32_t>(1)};
    if (M.e != cudaSuccess) return (int)M.e;
    void *args[] = {&dL, &g};
    M.e = cudaLaunchCooperativeKernel((const void *)k_vcycle<V>, dim3(blocks), dim3(kThreads), args, 0, 0);
    M.launched();
    std::vector<V> hx(D.nC);
    M.back(hx.data(), L.xs, D.nC);
    for (int i = 0; i < D.nC; ++i) x[i] = (double)hx[i];
    int32_t err = 0;
    M.back(&err, g.err, 1);
    return M.e != cudaSuccess ? (int)M.e : err ? -2 : 0;
}
}  // namespace

// x = one V-cycle on b from zero (x of level 0)
extern "C" int unit_vcycle(int fp32, int blocks, const int64_t *sizes, const int32_t *ints, int64_t nInts,
                           const double *vals, int64_t nVals, const double *matrix, int64_t nMatrix, const double *rds,
                           const double *inverse, int64_t nInverse, const double *b, double *x) {
    return fp32 ? vcycle<float>(blocks, sizes, ints, nInts, vals, nVals, matrix, nMatrix, rds, inverse, nInverse, b, x)
                : vcycle<double>(blocks, sizes, ints, nInts, vals, nVals, matrix, nMatrix, rds, inverse, nInverse, b, x);
}
