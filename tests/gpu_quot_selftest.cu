// The correctly rounded reciprocals and quotients of rp_device.cuh beside the
// IEEE operators: out[0] .. out[kOut - 1], each of n values.
#include <cstdint>
#include "rp_device.cuh"

constexpr int kOut = 7;

__global__ void k_quot(int64_t n, const double* a, const double* b, double* out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double y0 = rp_rcp_near(b[i]);
    const double v[kOut] = {rp_rcp(b[i]),          rp_rcp_in(b[i]),
                            rp_rcp3(b[i]).y,       rp_quot(a[i], b[i]),
                            rp_div_by(a[i], b[i], 1.0 / b[i]),
                            rp_div_rcp(a[i], b[i], rp_rcp3(b[i])),
                            rp_div_fast(a[i], b[i], rp_rcp_round(b[i], y0), y0)};
    for (int k = 0; k < kOut; k++) out[k * n + i] = v[k];
}

// polintd at the nodes of P: rp_polintd2 of (u, v) -> r[0], r[1], rp_polintd of
// each -> r[2], r[3]; u, v three values each
__global__ void k_polint(int64_t n, const __grid_constant__ RpPolint P, const double* u, const double* v, double* r) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a[3] = {u[i], u[n + i], u[2 * n + i]}, b[3] = {v[i], v[n + i], v[2 * n + i]};
    double ra, rb;
    rp_polintd2(P, a, b, ra, rb);
    r[i] = ra;
    r[n + i] = rb;
    r[2 * n + i] = rp_polintd(P, a[0], a[1], a[2]);
    r[3 * n + i] = rp_polintd(P, b[0], b[1], b[2]);
}

// xa: the nodes, x the place, ns the nearest node (0-based)
extern "C" int polint_selftest(int64_t n, const double* xa, double x, int ns, const double* u, const double* v,
                               double* r) {
    RpPolint P;
    P.ns = ns;
    P.d1 = xa[1] - x;
    P.e12 = xa[1] - xa[2];
    P.e01 = xa[0] - xa[1];
    P.e02 = xa[0] - xa[2];
    P.dns = xa[ns] - x;
    P.b = (ns == 2) ? xa[2] - x : xa[0] - x;
    P.re12 = 1.0 / P.e12;
    P.re01 = 1.0 / P.e01;
    P.re02 = 1.0 / P.e02;
    double* d[3] = {};
    const size_t bytes = (size_t)n * 8;
    int err = 0;
    for (int i = 0; i < 3; i++) err |= cudaMalloc(&d[i], (i == 2 ? 4 : 3) * bytes) != cudaSuccess;
    if (!err) {
        err |= cudaMemcpy(d[0], u, 3 * bytes, cudaMemcpyHostToDevice) != cudaSuccess;
        err |= cudaMemcpy(d[1], v, 3 * bytes, cudaMemcpyHostToDevice) != cudaSuccess;
        k_polint<<<(unsigned)((n + 255) / 256), 256>>>(n, P, d[0], d[1], d[2]);
        err |= cudaMemcpy(r, d[2], 4 * bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    for (int i = 0; i < 3; i++) cudaFree(d[i]);
    return err;
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
