// The correctly rounded reciprocals and quotients of rp_device.cuh beside the
// IEEE operators: out[0] .. out[kOut - 1], each of n values.
#include <cstdint>
#include "rp_device.cuh"

constexpr int kOut = 3;

__global__ void k_quot(int64_t n, const double* a, const double* b, double* out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v[kOut] = {rp_rcp(b[i]), rp_rcp_in(b[i]), rp_rcp3(b[i]).y};
    for (int k = 0; k < kOut; k++) out[k * n + i] = v[k];
}

extern "C" int quot_selftest(int64_t n, const double* a, const double* b, double* out) {
    double* d[3] = {};
    const size_t bytes = (size_t)n * 8;
    int err = 0;
    for (int i = 0; i < 3; i++) err |= cudaMalloc(&d[i], i == 2 ? kOut * bytes : bytes) != cudaSuccess;
    if (!err) {
        err |= cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice) != cudaSuccess;
        err |= cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice) != cudaSuccess;
        k_quot<<<(unsigned)((n + 255) / 256), 256>>>(n, d[0], d[1], d[2]);
        err |= cudaMemcpy(out, d[2], kOut * bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    for (int i = 0; i < 3; i++) cudaFree(d[i]);
    return err;
}
