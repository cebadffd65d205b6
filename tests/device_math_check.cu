// The branch-free FP64 helpers of device_math.cuh on arrays (tests/test_gpu_device_math.py).
#include <cuda_runtime.h>

#include "device_math.cuh"

namespace {
__global__ void apply(int op, const double *a, const double *b, double *out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const double x = a[i], y = b[i];
    double r = 0.0;
    switch(op) {
    case 0: r = bhcb::rcp_signed(y); break;
    case 1: r = bhcb::div_rn(x, y); break;
    case 2: r = bhcb::rcp_square(y * y, bhcb::rcp_rn(y)); break;
    case 3: r = bhcb::quot_rn(x, y * y, bhcb::rcp_square(y * y, bhcb::rcp_rn(y))); break;
    case 4: r = bhcb::sqrt_rn(x); break;
    case 5: r = x / y; break;
    case 6: r = sqrt(x); break;
    case 7: r = bhcb::rcp_rn(y); break;
    case 8: r = bhcb::sqrt_any(x); break;
    }
    out[i] = r;
}
} // namespace

extern "C" int device_math(int op, const double *a, const double *b, double *out, int n)
{
    double *da = nullptr, *db = nullptr, *dout = nullptr;
    const size_t bytes = sizeof(double) * (size_t)n;
    cudaError_t e = cudaMalloc(&da, bytes);
    if(e == cudaSuccess) e = cudaMalloc(&db, bytes);
    if(e == cudaSuccess) e = cudaMalloc(&dout, bytes);
    if(e == cudaSuccess) e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    if(e == cudaSuccess) e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    if(e == cudaSuccess) {
        apply<<<(n + 255) / 256, 256>>>(op, da, db, dout, n);
        e = cudaGetLastError();
    }
    if(e == cudaSuccess) e = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    return (int)e;
}
