// Device functions of the engine behind plain entry points, for
// test_gpu_device_units.py: one function each, without a solve around it.
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_common.h"
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_team.cuh"
#include "../bayesian-turbulence-modeling_gb300/csrc/btm_phases64.cuh"

#include <cuda_runtime.h>
#include <vector>

using namespace btm;

__global__ void k_div(const double *x, const double *d, const double *r, double *q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = div_by(x[i], d[i], r[i]);
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

}  // extern "C"
