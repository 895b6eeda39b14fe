// The network kernels' reciprocal against the division (see test_gpu_quotients.py).
#include "../../lbm_solver_3d_b200/csrc/k_mlp.cu"

// bit patterns first, first + 1, ... (n of them) whose reciprocals differ from 1 / x
__global__ void k_recip(unsigned first, unsigned long long n, unsigned long long* wrong) {
    unsigned long long bad = 0;
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + (unsigned)k), y = recip_ge1(x), want = __fdiv_rn(1.0f, x);
        bad += __float_as_uint(y) != __float_as_uint(want) && !(isnan(y) && isnan(want));
    }
    if (bad) atomicAdd(wrong, bad);
}

extern "C" int recip_wrong(unsigned first, unsigned long long n, unsigned long long* wrong) {
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(*d));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(*d));
    if (e == cudaSuccess) {
        k_recip<<<1184, 256>>>(first, n, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(wrong, d, sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
