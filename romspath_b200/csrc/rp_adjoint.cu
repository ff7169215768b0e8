// rp_adjoint.cu -- kernels of the adjoint pair (rp_forward / rp_backward),
// the tangent-linear reference and the replay used by finite differences.
// The steps run the generic step of rp_adjoint.cuh, with VTurb's displacements
// (and their derivatives) from kernels of their own; compiled without FMA
// contraction so that a replayed step takes its forward step's bits.
#include <cuda_runtime.h>

#include "rp_internal.h"
#include "rp_adjoint.cuh"

namespace rp {

constexpr int kAdjBlock = 128;
constexpr int kAdjVtBlock = 64;
constexpr int kAdjStepBlocks = 4;      // blocks of the steps in doubles and in dual numbers an SM
constexpr int kAdjReverseBlocks = 3;

__device__ __forceinline__ void adj_load(const AdjStateDev& s, int64_t n, double& x, double& y, double& z,
                                         AdjAux& a) {
    x = s.x[n];
    y = s.y[n];
    z = s.z[n];
    a.age = s.age[n];
    a.status = s.status[n];
    a.gid = s.gid[n];
    a.isin = s.isin[n];
}

__device__ __forceinline__ void adj_store_aux(const AdjStateDev& s, int64_t n, const AdjAux& a) {
    s.age[n] = a.age;
    s.status[n] = a.status;
    s.gid[n] = a.gid;
    s.isin[n] = a.isin;
}

// VTurb's displacements of a step in doubles (tv[n]); find: search p and
// record it in prec[n], else use prec[n].
//
// Bound by the fit's chains of dependent FP64 operations (a pivot, its
// reciprocal, the next pivot) and the traffic of the passes' factor and u:
// 64-thread blocks, eight an SM, hold 65,536 particles in one wave.  On the
// 130x98x20 grid with 65,536 particles a forward step (this kernel, 0.50 ms, and
// the rest) takes 0.57 ms, 1.5 in one kernel whose passes divided three times a
// row by the IEEE operator; a replayed step, one pass, 0.18 ms.
template <int NPMAX>
__global__ void __launch_bounds__(kAdjVtBlock, 512 / kAdjVtBlock)
    k_adj_vturb(const __grid_constant__ RpStepArgs A, const __grid_constant__ AdjFrames F, AdjStateDev s,
                double* __restrict__ prec, int find, double kappa, double* __restrict__ tv) {
    using W = BFit<NPMAX, false>;
    double buf[W::kArrays * (NPMAX + 1)];
    const W w{buf};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.p.n; i += stride) {
        const int64_t n = s.order ? s.order[i] : i;
        double p = find ? 0.0 : prec[n], t = 0.0;
        uint32_t fl = 0;
        if (a_active(A, A.p.dob[n], s.status[n], s.isin[n]))
            t = b_vturb(A, F, s.gid[n] - 1, s.x[n], s.y[n], s.z[n], kappa, A.p.pid[n], find != 0, p, fl, w);
        if (find) prec[n] = p;
        tv[n] = t;
    }
}

// The same with its derivatives in the start's x, y, z and in kappa: tv[q n],
// q = 0..4 (b_vturb_rev).  A reverse step (this kernel and k_adj_reverse) on
// the workload above takes 0.65 ms, 1.9 with the fit carried in dual numbers.
template <int NPMAX>
__global__ void __launch_bounds__(kAdjVtBlock, 512 / kAdjVtBlock)
    k_adj_vturb_rev(const __grid_constant__ RpStepArgs A, const __grid_constant__ AdjFrames F, AdjStateDev s,
                    const double* __restrict__ prec, double kappa, double* __restrict__ tv) {
    using W = BFit<NPMAX, true>;
    double buf[W::kArrays * (NPMAX + 1)];
    const W w{buf};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.p.n; i += stride) {
        const int64_t n = s.order ? s.order[i] : i;
        double t[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        uint32_t fl = 0;
        if (a_active(A, A.p.dob[n], s.status[n], s.isin[n]))
            b_vturb_rev(A, F, s.gid[n] - 1, s.x[n], s.y[n], s.z[n], kappa, A.p.pid[n], prec[n], fl, w, t);
#pragma unroll
        for (int q = 0; q < 5; q++) tv[q * A.p.n + n] = t[q];
    }
}

// one step of the model in doubles on state s; with VTurb on, tv holds
// k_adj_vturb's displacements.  Four stages of gathers; 65,536 particles 64 us
// at four blocks an SM (one wave) with levels bisected and particles taken by
// cell, 131 us at three, walked, as they lay.
__global__ void __launch_bounds__(kAdjBlock, kAdjStepBlocks) k_adj_step(const __grid_constant__ RpStepArgs A,
                                                         const __grid_constant__ AdjFrames F, AdjStateDev s,
                                                         const double* __restrict__ tv) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.p.n; i += stride) {
        const int64_t n = s.order ? s.order[i] : i;
        double x, y, z;
        AdjAux a;
        adj_load(s, n, x, y, z, a);
        uint32_t fl = 0;
        a_step<double>(A, F, A.p.dob[n], A.p.pid[n], x, y, z, a, fl,
                       [&](const AStage<double>&, bool, double) { return tv[n]; });
        s.x[n] = x;
        s.y[n] = y;
        s.z[n] = z;
        adj_store_aux(s, n, a);
    }
}

// VTurb in dual numbers within a step
template <class D, int NPMAX>
__device__ __forceinline__ D adj_vturb_dual(const RpStepArgs& A, const AdjFrames& F, int gid, const D& X, const D& Y,
                                            AStage<D>& S1, bool have_s1, const D& Zpar, const D& K, uint32_t pid,
                                            double p, uint32_t& fl, const AFit<D, NPMAX>& w) {
    if (!have_s1) b_stage(A, F, gid - 1, X, Y, S1, fl);
    return a_vturb(A, F, gid - 1, S1, Zpar, K, pid, p, w);
}

// one step in dual numbers carrying d/d(x0, y0, z0, kappa): tangent-linear
// propagation; t holds the 12 derivatives of (x, y, z) per particle
template <int NPMAX>
__global__ void __launch_bounds__(kAdjBlock) k_adj_tangent(const __grid_constant__ RpStepArgs A,
                                                            const __grid_constant__ AdjFrames F, AdjStateDev s,
                                                            double* __restrict__ t, const double* __restrict__ prec,
                                                            double kappa) {
    using D = Dual<4>;
    D buf[kAdjArrays * (NPMAX + 1)];
    const AFit<D, NPMAX> w{buf};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.p.n; i += stride) {
        const int64_t n = s.order ? s.order[i] : i;
        double x, y, z;
        AdjAux a;
        adj_load(s, n, x, y, z, a);
        D X(x), Y(y), Z(z), K(kappa);
        double* tn = t + n * 12;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            X.d[q] = tn[q];
            Y.d[q] = tn[4 + q];
            Z.d[q] = tn[8 + q];
        }
        K.d[3] = 1.0;
        const D X0 = X, Y0 = Y;
        const int gid = a.gid;
        uint32_t fl = 0;
        a_step<D>(A, F, A.p.dob[n], A.p.pid[n], X, Y, Z, a, fl, [&](AStage<D>& S1, bool have_s1, const D& Zpar) {
            return adj_vturb_dual<D, NPMAX>(A, F, gid, X0, Y0, S1, have_s1, Zpar, K, A.p.pid[n], prec[n], fl, w);
        });
#pragma unroll
        for (int q = 0; q < 4; q++) {
            tn[q] = X.d[q];
            tn[4 + q] = Y.d[q];
            tn[8 + q] = Z.d[q];
        }
        s.x[n] = X.v;
        s.y[n] = Y.v;
        s.z[n] = Z.v;
        adj_store_aux(s, n, a);
    }
}

// one reverse step: from the step's starting state s (read only), the
// step's Jacobian by dual numbers seeded on (x, y, z), VTurb's row of it from
// tv (k_adj_vturb_rev); then lambda <- J^T lambda for (x, y, z) and
// kbar += lambda . d(x,y,z)/dkappa (kappa enters z alone, through VTurb)
__global__ void __launch_bounds__(kAdjBlock, kAdjReverseBlocks) k_adj_reverse(const __grid_constant__ RpStepArgs A,
                                                            const __grid_constant__ AdjFrames F, AdjStateDev s,
                                                            const double* __restrict__ tv, double* __restrict__ lx,
                                                            double* __restrict__ ly, double* __restrict__ lz,
                                                            double* __restrict__ kbar) {
    using D = Dual<3>;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.p.n; i += stride) {
        const int64_t n = s.order ? s.order[i] : i;
        double x, y, z;
        AdjAux a;
        adj_load(s, n, x, y, z, a);
        D X(x), Y(y), Z(z);
        X.d[0] = 1.0;
        Y.d[1] = 1.0;
        Z.d[2] = 1.0;
        uint32_t fl = 0;
        const int vsign = a_step<D>(A, F, A.p.dob[n], A.p.pid[n], X, Y, Z, a, fl,
                                    [&](const AStage<D>&, bool, const D&) {
                                        D t(tv[n]);
#pragma unroll
                                        for (int q = 0; q < 3; q++) t.d[q] = tv[(q + 1) * A.p.n + n];
                                        return t;
                                    });
        const double bx = lx[n], by = ly[n], bz = lz[n];
        lx[n] = bx * X.d[0] + by * Y.d[0] + bz * Z.d[0];
        ly[n] = bx * X.d[1] + by * Y.d[1] + bz * Z.d[1];
        lz[n] = bx * X.d[2] + by * Y.d[2] + bz * Z.d[2];
        if (A.vturb_on && vsign) kbar[n] += bz * ((double)vsign * tv[4 * A.p.n + n]);
    }
}

// the same with the whole step in dual numbers seeded on (x, y, z, kappa), for
// runs with more sub-steps a step than k_adj_vturb_rev keeps
template <int NPMAX>
__global__ void __launch_bounds__(kAdjBlock) k_adj_reverse_dual(const __grid_constant__ RpStepArgs A,
                                                                 const __grid_constant__ AdjFrames F, AdjStateDev s,
                                                                 const double* __restrict__ prec, double kappa,
                                                                 double* __restrict__ lx, double* __restrict__ ly,
                                                                 double* __restrict__ lz, double* __restrict__ kbar) {
    using D = Dual<4>;
    D buf[kAdjArrays * (NPMAX + 1)];
    const AFit<D, NPMAX> w{buf};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.p.n; i += stride) {
        const int64_t n = s.order ? s.order[i] : i;
        double x, y, z;
        AdjAux a;
        adj_load(s, n, x, y, z, a);
        D X(x), Y(y), Z(z), K(kappa);
        X.d[0] = 1.0;
        Y.d[1] = 1.0;
        Z.d[2] = 1.0;
        K.d[3] = 1.0;
        const D X0 = X, Y0 = Y;
        const int gid = a.gid;
        uint32_t fl = 0;
        a_step<D>(A, F, A.p.dob[n], A.p.pid[n], X, Y, Z, a, fl, [&](AStage<D>& S1, bool have_s1, const D& Zpar) {
            return adj_vturb_dual<D, NPMAX>(A, F, gid, X0, Y0, S1, have_s1, Zpar, K, A.p.pid[n], prec[n], fl, w);
        });
        const double bx = lx[n], by = ly[n], bz = lz[n];
        lx[n] = bx * X.d[0] + by * Y.d[0] + bz * Z.d[0];
        ly[n] = bx * X.d[1] + by * Y.d[1] + bz * Z.d[1];
        lz[n] = bx * X.d[2] + by * Y.d[2] + bz * Z.d[2];
        kbar[n] += bx * X.d[3] + by * Y.d[3] + bz * Z.d[3];
    }
}

template <class K>
static unsigned adj_grid(K kernel, int64_t n, int num_sms, int block) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, 0) != cudaSuccess || occ < 1) occ = 1;
    int64_t b = (int64_t)num_sms * occ;
    const int64_t need = (n + block - 1) / block;
    if (need < b) b = need;
    return (unsigned)(b < 1 ? 1 : b);
}

template <int NPMAX>
static cudaError_t adj_launch_t(int kind, const RpStepArgs& A, const AdjFrames& F, const AdjStateDev& s,
                                double* prec, int find, double kappa, double* tv, double* t, double* lx, double* ly,
                                double* lz, double* kbar, cudaStream_t st, int num_sms, int64_t* nlaunch) {
    const int64_t n = A.p.n;
    if (kind == 0) {
        if (A.vturb_on) {
            k_adj_vturb<NPMAX><<<adj_grid(k_adj_vturb<NPMAX>, n, num_sms, kAdjVtBlock), kAdjVtBlock, 0, st>>>(
                A, F, s, prec, find, kappa, tv);
            *nlaunch += 1;
        }
        k_adj_step<<<adj_grid(k_adj_step, n, num_sms, kAdjBlock), kAdjBlock, 0, st>>>(A, F, s, tv);
    } else if (kind == 1) {
        k_adj_tangent<NPMAX><<<adj_grid(k_adj_tangent<NPMAX>, n, num_sms, kAdjBlock), kAdjBlock, 0, st>>>(
            A, F, s, t, prec, kappa);
    } else if (A.vturb_on && A.loop > NPMAX) {
        k_adj_reverse_dual<NPMAX><<<adj_grid(k_adj_reverse_dual<NPMAX>, n, num_sms, kAdjBlock), kAdjBlock, 0, st>>>(
            A, F, s, prec, kappa, lx, ly, lz, kbar);
    } else {
        if (A.vturb_on) {
            k_adj_vturb_rev<NPMAX><<<adj_grid(k_adj_vturb_rev<NPMAX>, n, num_sms, kAdjVtBlock), kAdjVtBlock, 0,
                                     st>>>(A, F, s, prec, kappa, tv);
            *nlaunch += 1;
        }
        k_adj_reverse<<<adj_grid(k_adj_reverse, n, num_sms, kAdjBlock), kAdjBlock, 0, st>>>(A, F, s, tv, lx, ly, lz,
                                                                                            kbar);
    }
    *nlaunch += 1;
    return cudaGetLastError();
}

cudaError_t launch_adj(int kind, const RpStepArgs& A, const AdjFrames& F, const AdjStateDev& s, double* prec, int find,
                       double kappa, double* tv, double* t, double* lx, double* ly, double* lz, double* kbar,
                       int npmax, cudaStream_t st, int num_sms, int64_t* nlaunch) {
    if (A.p.n <= 0) return cudaSuccess;
    if (npmax <= 88)
        return adj_launch_t<88>(kind, A, F, s, prec, find, kappa, tv, t, lx, ly, lz, kbar, st, num_sms, nlaunch);
    if (npmax <= 128)
        return adj_launch_t<128>(kind, A, F, s, prec, find, kappa, tv, t, lx, ly, lz, kbar, st, num_sms, nlaunch);
    return adj_launch_t<144>(kind, A, F, s, prec, find, kappa, tv, t, lx, ly, lz, kbar, st, num_sms, nlaunch);
}

// Fortran-ordered field (+ Stokes term, summed in FP64) -> [j][i][k] FP64
template <typename S>
__global__ void k_adj_store(const S* __restrict__ src, const S* __restrict__ add, double* __restrict__ dst, int ni,
                            int nj, int nk, int64_t e0, int64_t count) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const int64_t e = e0 + t;
    const int64_t plane = (int64_t)ni * nj;
    const int k = (int)(e / plane);
    const int64_t r = e - (int64_t)k * plane;
    const int j = (int)(r / ni);
    const int i = (int)(r - (int64_t)j * ni);
    double v = (double)src[t];
    if (add) v = v + (double)add[t];
    dst[((int64_t)j * ni + i) * nk + k] = v;
}

cudaError_t launch_adj_store(const double* src, const double* add, double* dst, int ni, int nj, int nk, int64_t e0,
                             int64_t count, cudaStream_t s) {
    const unsigned nb = (unsigned)((count + 255) / 256);
    if (nb == 0) return cudaSuccess;
    k_adj_store<double><<<nb, 256, 0, s>>>(src, add, dst, ni, nj, nk, e0, count);
    return cudaGetLastError();
}

// initial tangent: d(x, y, z)/d(x0, y0, z0, kappa) = [I 0]
__global__ void k_adj_tangent_init(double* t, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* tn = t + i * 12;
#pragma unroll
    for (int q = 0; q < 12; q++) tn[q] = 0.0;
    tn[0] = 1.0;
    tn[5] = 1.0;
    tn[10] = 1.0;
}

cudaError_t launch_adj_tangent_init(double* t, int64_t n, cudaStream_t s) {
    const unsigned nb = (unsigned)((n + 255) / 256);
    if (nb == 0) return cudaSuccess;
    k_adj_tangent_init<<<nb, 256, 0, s>>>(t, n);
    return cudaGetLastError();
}

}  // namespace rp
