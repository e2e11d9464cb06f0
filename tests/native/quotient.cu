// quotient.cu -- TEST HARNESS: the FP32 quotients of the cell models (dv and dvc of
// ucla_cmg_b200/csrc/common.cuh) on the device.  Not part of the library.
#include "../../ucla_cmg_b200/csrc/common.cuh"

__global__ void k_quotients(int n, const float *a, const float *b, float *y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = ep::dv(a[i], b[i]);
    y[n + i] = ep::dvc(a[i], b[i]);
}

extern "C" int quotients(int n, const float *a, const float *b, float *y) {
    k_quotients<<<(n + 255) / 256, 256>>>(n, a, b, y);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
