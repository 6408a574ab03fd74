// Test helper (not part of the library): the chain kernel's FP64 division on the device, and the
// device's own quotient, for a batch of operands.
#include "achr_div.cuh"

__global__ void div_batch_kernel(int n, const double *a, const double *b, double *q, double *want) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    q[t] = achr::div_rn(a[t], b[t]);
    want[t] = __ddiv_rn(a[t], b[t]);
}

extern "C" int div_batch(int n, const double *a, const double *b, double *q, double *want) {
    double *d = nullptr;
    const size_t bytes = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 4 * bytes) != cudaSuccess) return 1;
    cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    div_batch_kernel<<<(n + 127) / 128, 128>>>(n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
    cudaError_t e = cudaMemcpy(q, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(want, d + 3 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
