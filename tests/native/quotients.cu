// The kernels' quotients and wraps, value by value (see test_gpu_quotients.py).
#include "../../lbm_solver_3d_b200/csrc/k_stream.cuh"

#include <vector>

using namespace lbmgpu;

__global__ void k_div3(const double* a, const double* b, double* q, size_t n) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    div3(a[3 * k], a[3 * k + 1], a[3 * k + 2], b[k], q[3 * k], q[3 * k + 1], q[3 * k + 2]);
}
__global__ void k_min_image(const double* r, const int* m, double* t, size_t n) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k < n) t[k] = min_image(r[k], m[k]);
}

template <class B, class Kern>
static int apply(Kern kern, const double* a, size_t na, const B* b, double* out, size_t nout, size_t n) {
    double *da = nullptr, *dout = nullptr;
    B* db = nullptr;
    cudaError_t e = cudaMalloc(&da, na * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&db, n * sizeof(B));
    if (e == cudaSuccess) e = cudaMalloc(&dout, nout * sizeof(double));
    if (e == cudaSuccess) e = cudaMemcpy(da, a, na * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, n * sizeof(B), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        kern<<<(unsigned)((n + 255) / 256), 256>>>(da, db, dout, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, nout * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    return (int)e;
}

// q[3n] = a[3n] / b[n]; t[n] = the minimum image of r[n] on an axis of m[n]
extern "C" int quot_div3(const double* a, const double* b, double* q, size_t n) { return apply(k_div3, a, 3 * n, b, q, 3 * n, n); }
extern "C" int quot_min_image(const double* r, const int* m, double* t, size_t n) { return apply(k_min_image, r, n, m, t, n, n); }
