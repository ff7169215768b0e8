// The adjoint pair's fit on its own: the sum of squares and utru that the
// search for the smoothing parameter takes from a pass at p, of m columns of np
// resampled points (y[i * m + k]) with spacings h and parameters p.
#include <cstdint>
#include "rp_adjoint.cuh"

constexpr int kMax = 144;

__global__ void k_fit(int m, int np, double serr, const double* y, const double* h, const double* p, double* sum,
                      double* utru) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    using W = BFit<kMax, false>;
    double buf[W::kArrays * (kMax + 1)];
    const W w{buf};
    BPar B;
    B.np = np;
    B.sw = np;
    B.z1 = 0.0;
    B.hb = h[k];
    B.rh = 1.0 / h[k];
    B.serr = serr;
    const double r = serr / h[k];
    B.r2 = r * r;
    for (int i = 1; i <= np; i++) w.y(i) = y[(int64_t)(i - 1) * m + k];
    b_solve<false>(w, B, p[k]);
    sum[k] = b_sum(w, B);
    utru[k] = b_utru(w, B);
}

extern "C" int adj_fit(int m, int np, double serr, const double* y, const double* h, const double* p, double* sum,
                       double* utru) {
    double* d[5] = {};
    const size_t bm = (size_t)m * 8, by = bm * np;
    const double* src[3] = {y, h, p};
    const size_t sz[5] = {by, bm, bm, bm, bm};
    int err = 0;
    for (int i = 0; i < 5; i++) err |= cudaMalloc(&d[i], sz[i]) != cudaSuccess;
    for (int i = 0; i < 3 && !err; i++) err |= cudaMemcpy(d[i], src[i], sz[i], cudaMemcpyHostToDevice) != cudaSuccess;
    if (!err) {
        k_fit<<<(m + 63) / 64, 64>>>(m, np, serr, d[0], d[1], d[2], d[3], d[4]);
        err |= cudaMemcpy(sum, d[3], bm, cudaMemcpyDeviceToHost) != cudaSuccess;
        err |= cudaMemcpy(utru, d[4], bm, cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    for (int i = 0; i < 5; i++) cudaFree(d[i]);
    return err;
}
