// The FP64 helpers of rf_device.cuh on arrays, for test_device_arithmetic.py.
#include "rf_device.cuh"

namespace {

// out: rows of n results
__global__ void helpers(int n, const double *a, const double *b, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    out[i] = rf::rcp_pos(y);
    out[n + i] = rf::rsqrt_pos(y);
    out[2 * n + i] = rf::sqrt_pos(y);
    out[3 * n + i] = rf::div_by(x, y, rf::rcp_pos(y));
    out[4 * n + i] = rf::div_const<3>(x);
    out[5 * n + i] = rf::div_const<-5>(x);
    out[6 * n + i] = rf::div_const<7>(x);
    out[7 * n + i] = rf::div_const<-10>(x);
    // the closed forms' largest product of reciprocals: 1 / (6 d u^3)
    const double u = rf::sqrt_pos(y), ru = rf::rcp_pos(u), d = fabs(x);
    const double den = rf::fmul(rf::fmul(6.0, d), rf::fmul(rf::fmul(u, u), u));
    const double r6 = rf::rcp_pos(d) * (1.0 / 6.0);
    out[8 * n + i] = den;
    out[9 * n + i] = rf::div_by(x, den, r6 * ru * ru * ru);
}

}  // namespace

extern "C" int device_arithmetic(int n, const double *a, const double *b, double *out) {
    double *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(double) * 12 * (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        helpers<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, sizeof(double) * 10 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
