// child_weight(a, sigma_of(s)) and a / s of every pair, on the device.
#include "sbc_internal.cuh"

__global__ void k_pairs(int n, const double* a, const int64_t* s, double* w, double* q)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    w[i] = sbc::child_weight(a[i], sbc::sigma_of(s[i]));
    q[i] = a[i] / (double)s[i];
}

extern "C" int child_weights(int n, const double* a, const int64_t* s, double* w, double* q)
{
    double *da, *dw, *dq;
    int64_t* ds;
    const size_t b = sizeof(double) * (size_t)n;
    if (cudaMalloc(&da, b) || cudaMalloc(&ds, b) || cudaMalloc(&dw, b) || cudaMalloc(&dq, b)) return 1;
    cudaMemcpy(da, a, b, cudaMemcpyHostToDevice);
    cudaMemcpy(ds, s, b, cudaMemcpyHostToDevice);
    k_pairs<<<(n + 255) / 256, 256>>>(n, da, ds, dw, dq);
    cudaMemcpy(w, dw, b, cudaMemcpyDeviceToHost);
    cudaMemcpy(q, dq, b, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(ds);
    cudaFree(dw);
    cudaFree(dq);
    return (int)cudaDeviceSynchronize();
}
