// rp_step.cuh -- the per-particle step of update_particles
// (ROMSPath.f90:662-905) on the device: RK4 advection, HTurb, VTurb with
// the PPPACK smoothing spline, nest hand-off, vertical update and status.
#pragma once

#include "rp_device.cuh"

// --------------------------------------------------------------- noise

// Normal deviate `d` of particle `pid` at this step: the noise hook when
// set, else Philox4x32-10 at counter (pid, step, d/2) with Box-Muller's
// cosine branch (pdf_module.f90:26-40) on the uniforms (r+0.5)/2^32.
__device__ __forceinline__ double rp_normal(const RpStepArgs& A, uint32_t pid, uint32_t d) {
    if (A.hook) return A.hook[(int64_t)(pid - A.pid_base) * A.ndraw + d];
    uint32_t c[4] = {pid, (uint32_t)A.step_index, (uint32_t)(A.step_index >> 32), d >> 1};
    rp_philox(c, (uint32_t)A.seed, (uint32_t)(A.seed >> 32));
    const uint32_t a = (d & 1u) ? c[2] : c[0];
    const uint32_t b = (d & 1u) ? c[3] : c[1];
    const double u1 = ((double)a + 0.5) / 4294967296.0;
    const double u2 = ((double)b + 0.5) / 4294967296.0;
    return sqrt(-2.0 * rp_log_pos(u1)) * rp_cos2pi(u2);
}

// Normal deviates d and d+1 (d even) by one Philox call; d+1 only with
// `both` (the hook holds no more than the step's draws).
__device__ __forceinline__ void rp_normal2(const RpStepArgs& A, uint32_t pid, uint32_t d, bool both, double& n0,
                                           double& n1) {
    n1 = 0.0;
    if (A.hook) {
        const double* h = A.hook + (int64_t)(pid - A.pid_base) * A.ndraw + d;
        n0 = h[0];
        if (both) n1 = h[1];
        return;
    }
    uint32_t c[4] = {pid, (uint32_t)A.step_index, (uint32_t)(A.step_index >> 32), d >> 1};
    rp_philox(c, (uint32_t)A.seed, (uint32_t)(A.seed >> 32));
    const double u1 = ((double)c[0] + 0.5) / 4294967296.0;
    const double u2 = ((double)c[1] + 0.5) / 4294967296.0;
    n0 = sqrt(-2.0 * rp_log_pos(u1)) * rp_cos2pi(u2);
    if (both) {
        const double u3 = ((double)c[2] + 0.5) / 4294967296.0;
        const double u4 = ((double)c[3] + 0.5) / 4294967296.0;
        n1 = sqrt(-2.0 * rp_log_pos(u3)) * rp_cos2pi(u4);
    }
}

// Uniform k (0..4) of behave's draws: the hook's entry d0 + 2 + k (d0 =
// 2 + idt/deltat, after the HTurb and VTurb normals and behave's two), else
// Philox4x32-10 at counter (pid, step, 0x40000000 + k/4), word k%4.
__device__ __forceinline__ double rp_uniform(const RpStepArgs& A, uint32_t pid, uint32_t d0, uint32_t k) {
    if (A.hook) return A.hook[(int64_t)(pid - A.pid_base) * A.ndraw + d0 + 2 + k];
    uint32_t c[4] = {pid, (uint32_t)A.step_index, (uint32_t)(A.step_index >> 32), 0x40000000u + (k >> 2)};
    rp_philox(c, (uint32_t)A.seed, (uint32_t)(A.seed >> 32));
    return ((double)c[k & 3u] + 0.5) / 4294967296.0;
}

// laplace (pdf_module.f90:42-55) of one uniform: sign(dev2, dev1) with
// dev1 = u - 0.5, dev2 = -log(1 - 2|dev1|) / sqrt(2)
__device__ __forceinline__ double rp_laplace_of(double u) {
    const double dev1 = RP_SUB(u, 0.5);
    const double dev2 = RP_MUL(-1.0, rp_log(RP_SUB(1.0, RP_MUL(2.0, fabs(dev1))))) / sqrt(2.0);
    const double mag = fabs(dev2);
    return (dev1 >= 0.0) ? mag : -mag;
}

// ------------------------------------------------------- find_currents

struct StageState {
    RhoCell rc;
    double tdepth, zb, zc, zf, zeta;
};

// The u, v, w gathers of find_currents under WETDRY: each slot's value
// with that slot's wetdry masks (interpolation_module.f90:628-671, 710-757,
// 917-939).  Out of line: the step without WETDRY keeps its registers.
template <typename T>
__device__ __noinline__ void rp_gather_wd(const RpStepArgs& A, const RpGridDev& g, double X, double Y,
                                          const LevelPick& Lr, const LevelPick& Lw, const RhoCell& rc, double& Uad,
                                          double& Vad, double& Wad, uint32_t& fl) {
    const int N = g.N;
    const int ns = (A.ets == 1) ? 2 : 3;
    const int sl[3] = {g.sb, g.sc, g.sf};
    double u[3], v[3], w[3];
    for (int q = 0; q < ns; q++) {
        UVCell c;
        rp_u_cell(g, X, Y, c, fl, g.wd_u, RP_SLOTS, sl[q]);
        u[q] = rp_col_uv<T>(g.u, c, N, Lr, sl[q]);
        rp_v_cell(g, X, Y, c, fl, g.wd_v, RP_SLOTS, sl[q]);
        v[q] = rp_col_uv<T>(g.v, c, N, Lr, sl[q]);
        double cw[4];
        rp_rho_wd_weights(g, rc, sl[q], cw, fl);
        w[q] = rp_col_rho<T>(g.w, rc, cw, N + 1, Lw, sl[q]);
    }
    if (A.ets == 1) {                                      // advection_module.f90:277-287
        Uad = rp_polintd(A.pi, u[0], u[0], u[1]);
        Vad = rp_polintd(A.pi, v[0], v[0], v[1]);
        Wad = rp_polintd(A.pi, w[0], w[0], w[1]);
    } else {
        Uad = rp_polintd(A.pi, u[0], u[1], u[2]);
        Vad = rp_polintd(A.pi, v[0], v[1], v[2]);
        Wad = rp_polintd(A.pi, w[0], w[1], w[2]);
    }
}

// find_currents (advection_module.f90:129-350); Z is INOUT.
template <typename T>
__device__ __forceinline__ void rp_find_currents(const RpStepArgs& A, const RpGridDev& g, double X, double Y,
                                                 double& Z, double& Uad, double& Vad, double& Wad,
                                                 StageState& S, uint32_t& fl) {
    rp_rho_cell(g, X, Y, S.rc, fl);
    S.tdepth = -1.0 * rp_bil(g.h, S.rc);
    const RpSlots zt = rp_zeta3<T>(g, S.rc);
    S.zb = zt.b;
    S.zc = zt.c;
    S.zf = zt.f;
    if (Z < S.tdepth) Z = S.tdepth + RP_F_0P001;
    S.zeta = rp_polintd(A.pi, S.zb, S.zc, S.zf);
    if (Z > S.zeta) Z = S.zeta - RP_F_0P001;

    LevelPick Lr, Lw;
    rp_walk2(g, S.zeta, S.tdepth, Z, Lr, Lw, fl);
    if (A.wetdry) {
        rp_gather_wd<T>(A, g, X, Y, Lr, Lw, S.rc, Uad, Vad, Wad, fl);
        return;
    }
    const int N = g.N;
    // at ets == 1 the values are (b, b, c) (advection_module.f90:277-287)
    auto in_time = [&](const RpSlots& v) -> double {
        return (A.ets == 1) ? rp_polintd(A.pi, v.b, v.b, v.c) : rp_polintd(A.pi, v.b, v.c, v.f);
    };
    {
        UVCell cu;
        rp_u_cell(g, X, Y, cu, fl);
        Uad = in_time(rp_col3<T>(g, g.u, cu.o, cu.cff, cu.use, N, Lr));
    }
    {
        UVCell cv;
        rp_v_cell(g, X, Y, cv, fl);
        Vad = in_time(rp_col3<T>(g, g.v, cv.o, cv.cff, cv.use, N, Lr));
    }
    {
        const int64_t o[4] = {S.rc.o00, S.rc.o10, S.rc.o11, S.rc.o01};
        double cw[4];
#pragma unroll
        for (int k = 0; k < 4; k++) cw[k] = S.rc.wet4 ? S.rc.cb[k] : S.rc.ci[k];
        Wad = in_time(rp_col3<T>(g, g.w, o, cw, nullptr, N + 1, Lw));
    }
}

// ----------------------------------------------------------- spline
//
// The smoothing-spline fit of one particle.  Its arrays (1-based element i):
//   fitz  the breaks             y    the resampled data fitKH
//   qty   Q'y                    r12  the factor's two ratios v(i,2), v(i,3)
//   u     u(i)/v(i,1), then u(i)
// The column's lines (slope, intercept) sit in r12 and its levels z(k) in u
// until the fit overwrites them.

// A warp's fits in a private array each; SU: u in the warp's shared memory
// instead (element i of lane l at su[(i - 1) * 32 + l]: no bank conflicts).
template <int NPMAX, bool SU>
struct SplineLocal {
    static constexpr int kDoubles = (SU ? 5 : 6) * (NPMAX + 2);
    double* base;                  // kDoubles doubles, 16-byte aligned
    double* su;
    __device__ __forceinline__ double2* rr() const { return reinterpret_cast<double2*>(base); }
    __device__ __forceinline__ double2 r12(int i) const { return rr()[i]; }
    __device__ __forceinline__ void set_r12(int i, double a, double b) const { rr()[i] = make_double2(a, b); }
    __device__ __forceinline__ double& fitz(int i) const { return base[2 * (NPMAX + 2) + i]; }
    __device__ __forceinline__ double& y(int i) const { return base[3 * (NPMAX + 2) + i]; }
    __device__ __forceinline__ double& qty(int i) const { return base[4 * (NPMAX + 2) + i]; }
    __device__ __forceinline__ double& u(int i) const { return SU ? su[(i - 1) * 32] : base[5 * (NPMAX + 2) + i]; }
};

// The same with every array in a warp's shared memory (element i of array a
// of lane l at sm[(a * (NPMAX + 1) + i) * 32 + l]).
template <int NPMAX>
struct SplineShared {
    static constexpr size_t kBytes = (size_t)(NPMAX + 1) * 32 * 6 * sizeof(double);
    double* sm;                    // this lane's first element
    __device__ __forceinline__ double& at(int a, int i) const { return sm[(a * (NPMAX + 1) + i) * 32]; }
    __device__ __forceinline__ double2 r12(int i) const { return make_double2(at(0, i), at(1, i)); }
    __device__ __forceinline__ void set_r12(int i, double a, double b) const { at(0, i) = a; at(1, i) = b; }
    __device__ __forceinline__ double& fitz(int i) const { return at(2, i); }
    __device__ __forceinline__ double& y(int i) const { return at(3, i); }
    __device__ __forceinline__ double& qty(int i) const { return at(4, i); }
    __device__ __forceinline__ double& u(int i) const { return at(5, i); }
};

// What a fit's passes share.  The breaks are fitz(1) = z1, fitz(k) =
// fitz(k-1) + dz, fitz(np) = zend (ver_turb_module.f90:126-136); the passes
// re-form them by the same additions.  fitz(k-1) + dz rounds the same way
// while |fitz| stays in one binade, so v4(k) = fitz(k+1) - fitz(k) changes
// its value a handful of times down a column (4 on average at 124 points),
// and what is formed from v4 alone is formed again only there: at the rows
// flagged in chg, which holds the changes of every lane of the warp, so that
// the lanes take either path together (a lane whose v4 does not change forms
// the same values again).
constexpr int kChgWords = 5;       // 160 bits >= kMaxNp + 1 (rp_internal.h)
struct RpFit {
    int np;
    bool mono;                     // the breaks ascend: ppvalu may guess its piece
    double z1, dz, zend, rdz;      // rdz: about 1 / dz
    double f4;                     // fitz(4)
    double v1, v2, v3;             // v4(1..3)
    double r1, r2, r3;             // serr / v4(1..3)
    double y1;                     // 1 / v4(1), correctly rounded
    double serr, dy2;
    uint32_t chg[kChgWords];       // bit k: v4(k) != v4(k-1) in some lane, k >= 2
    // V1(2), V2(2), V1(3) of setupq's matrix
    __device__ __forceinline__ void first_rows(double p, double& a1, double& a2, double& b1) const {
        const double six1mp = 6.0 * (1.0 - p), twop = 2.0 * p;
        const double v2s2 = -r2 - r1, v2s3 = -r3 - r2;
        a1 = six1mp * (r1 * r1 + v2s2 * v2s2 + r2 * r2) + twop * (v1 + v2);
        a2 = six1mp * (v2s2 * r2 + r2 * v2s3) + p * v2;
        b1 = six1mp * (r2 * r2 + v2s3 * v2s3 + r3 * r3) + twop * (v2 + v3);
    }
    // bits i .. i + 31 of chg
    __device__ __forceinline__ uint32_t bits(int i) const {
        const int w = i >> 5;
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int q = 0; q < kChgWords; q++) {
            lo = (q == w) ? chg[q] : lo;
            hi = (q == w + 1) ? chg[q] : hi;
        }
        return __funnelshift_r(lo, hi, i & 31);
    }
};

// The pass below with every division left to the IEEE operator, for fits
// whose operands leave the shared-reciprocal division's range (NaN frames,
// subnormal diffusivities).
template <class W>
__device__ __noinline__ double rp_chol1d_ieee(const W w, const RpFit& F, double p) {
    const int np = F.np;
    const double six1mp = 6.0 * (1.0 - p), twop = 2.0 * p;
    double ri = F.r2, rn = F.r3, v4n = F.v3;
    double a1, a2, b1;
    F.first_rows(p, a1, a2, b1);
    double uprev = 0.0, ucur = w.qty(2), r2prev = 0.0;
    for (int i = 2; i <= np - 2; i++) {
        const bool in = i <= np - 3;             // rows with a third band
        const double v4nn = in ? w.fitz(i + 3) - w.fitz(i + 2) : 0.0;
        const double rnn = in ? F.serr / v4nn : 0.0;
        const double V3 = six1mp * (in ? ri * rn : 0.0);
        const double v2sn = -rn - ri, v2snn = -rnn - rn;
        const double ratio1 = a2 / a1, ratio2 = V3 / a1;
        w.set_r12(i, ratio1, ratio2);
        w.u(i) = ucur / a1;
        const double a1n = b1 - ratio1 * a2;
        a2 = (six1mp * (v2sn * rn + rn * v2snn) + p * v4n) - ratio1 * V3;
        b1 = (six1mp * (rn * rn + v2snn * v2snn + rnn * rnn) + twop * (v4n + v4nn)) - ratio2 * V3;
        a1 = a1n;
        const double unext = w.qty(i + 1) - ratio1 * ucur - r2prev * uprev;
        uprev = ucur;
        ucur = unext;
        r2prev = ratio2;
        ri = rn;
        rn = rnn;
        v4n = v4nn;
    }
    double up2 = 0.0, up1 = ucur / a1;
    w.u(np - 1) = up1;
    for (int i = np - 2; i >= 2; i--) {
        const double2 r = w.r12(i);
        const double ui = w.u(i) - up1 * r.x - up2 * r.y;
        w.u(i) = ui;
        up2 = up1;
        up1 = ui;
    }
    double prev = 0.0, sum = 0.0, ulast = 0.0;
    for (int i = 2; i <= np; i++) {
        const double ui = (i < np) ? w.u(i) : 0.0;
        const double raw = (ui - ulast) / (w.fitz(i) - w.fitz(i - 1));
        const double fin = raw - prev;
        sum = sum + (fin * fin) * F.dy2;
        prev = raw;
        ulast = ui;
    }
    return sum + (-prev * -prev) * F.dy2;
}

// chol1d (pppack.f90:1428-1566) for p.  With all data weights dy(i) = serr
// setupq's bands are v(i,1) = r(i-1), v(i,2) = -r(i) - r(i-1), v(i,3) = r(i);
// the band values of a row (V1, V2, V3 below) are formed by setupq's own
// operations.  Factorisation and forward substitution run in one ascending
// sweep that keeps v(i,2), v(i,3) and u(i)/v(i,1); back substitution runs
// descending; then Q u and sum_i qu(i)^2 dy(i)^2 are formed ascending (the
// reference's summation order).
//
// A row is one chain of dependent FP64 operations (pivot, reciprocal,
// quotient, next pivot: about 95 cycles at 8 a step on B200), so the rows
// hold no branch: the quotients share the pivot's reciprocal and are formed
// whether their operands are in range or not, and the pass is made again by
// the IEEE operator when one was not (with a test and a cold branch in each
// row a row took 320 cycles alone, without 190).  What the rows read from
// memory is loaded a group of rows ahead.
template <class W>
__device__ __forceinline__ double rp_chol1d(const W& w, const RpFit& F, double p) {
    const int np = F.np;
    const double six1mp = 6.0 * (1.0 - p);
    const double twop = 2.0 * p;
    double ri = F.r2;                            // r(i),   i = 2
    double rn = F.r3;                            // r(i+1)
    double v4n = F.v3;                           // v4(i+1)
    double a1, a2, b1;
    F.first_rows(p, a1, a2, b1);
    double uprev = 0.0, ucur = w.qty(2), r2prev = 0.0;
    double acc = F.f4;                           // the running sum of the breaks, fitz(i+2)
    double V3 = 0.0, V2n = 0.0, V1nn = 0.0;      // V3(i), V2(i+1), V1(i+2)
    uint32_t off = 0;                            // largest exponent distance of an operand
    uint32_t ones = 0;                           // all bits: a significand of all ones
    // the band values of row i, whose v4(i), v4(i+1) or v4(i+2) may be new
    auto bands = [&](int i) {
        const double f = (i + 3 == np) ? F.zend : acc + F.dz;
        const double v4nn = f - acc;             // v4(i+2)
        const double rnn = rp_div_rcp(F.serr, v4nn, rp_rcp3(v4nn));
        off = max(off, rp_exp_off(v4nn));
        ones = max(ones, rp_ones(v4nn));
        V3 = six1mp * (ri * rn);
        const double v2sn = -rn - ri;            // v(i+1,2) of setupq
        const double v2snn = -rnn - rn;          // v(i+2,2)
        V2n = six1mp * (v2sn * rn + rn * v2snn) + p * v4n;
        V1nn = six1mp * (rn * rn + v2snn * v2snn + rnn * rnn) + twop * (v4n + v4nn);
        ri = rn;
        rn = rnn;
        v4n = v4nn;
    };
    auto row = [&](int i, double qn) {
        acc = acc + F.dz;
        off = max(max(off, rp_exp_off(a1)), max(rp_exp_off(a2), rp_exp_off_z(ucur)));
        ones = max(ones, rp_ones(a1));
        const RpRcp y = rp_rcp3(a1);
        const double ratio1 = rp_div_rcp(a2, a1, y);
        const double ratio2 = rp_div_rcp(V3, a1, y);
        w.u(i) = rp_div_rcp(ucur, a1, y);        // u(i)/v(i,1)
        w.set_r12(i, ratio1, ratio2);
        const double a1n = b1 - ratio1 * a2;
        a2 = V2n - ratio1 * V3;
        b1 = V1nn - ratio2 * V3;
        a1 = a1n;
        const double unext = qn - ratio1 * ucur - r2prev * uprev;
        uprev = ucur;
        ucur = unext;
        r2prev = ratio2;
    };
    constexpr int G = 4;
    double q[G];
#pragma unroll
    for (int k = 0; k < G; k++) q[k] = w.qty(min(3 + k, np - 1));
    int i = 2;
    for (; i + G - 1 <= np - 3; i += G) {
        double qx[G];
#pragma unroll
        for (int k = 0; k < G; k++) qx[k] = w.qty(min(i + 1 + G + k, np - 1));
        // a change of v4 at k concerns rows k-2 .. k
        if (i == 2 || (F.bits(i) & ((1u << (G + 2)) - 1u))) {
#pragma unroll
            for (int k = 0; k < G; k++) {
                bands(i + k);
                row(i + k, q[k]);
            }
            off = max(off, rp_exp_off(V3));
        } else {
#pragma unroll
            for (int k = 0; k < G; k++) row(i + k, q[k]);
        }
#pragma unroll
        for (int k = 0; k < G; k++) q[k] = qx[k];
    }
    for (; i <= np - 3; i++) {
        bands(i);
        row(i, w.qty(i + 1));
    }
    off = max(off, rp_exp_off(V3));
    {                                             // row np-2: V3 = six1mp * 0
        const double ratio1 = a2 / a1;
        w.set_r12(np - 2, ratio1, (six1mp * 0.0) / a1);
        w.u(np - 2) = ucur / a1;
        a1 = b1 - ratio1 * a2;
        ucur = w.qty(np - 1) - ratio1 * ucur - r2prev * uprev;
    }
    // back substitution, the ratios read a group of rows ahead
    double up2 = 0.0, up1 = ucur / a1;            // u(np-1)/v(np-1,1)
    w.u(np - 1) = up1;
    constexpr int B = 8;
    double2 sa[B], sb[B];
    auto load = [&](double2(&t)[B], int j) {
#pragma unroll
        for (int k = 0; k < B; k++) t[k] = w.r12(max(j - k, 2));
    };
    auto solve = [&](const double2(&t)[B], int j) {
#pragma unroll
        for (int k = 0; k < B; k++) {
            const double ui = w.u(j - k) - up1 * t[k].x - up2 * t[k].y;
            w.u(j - k) = ui;
            up2 = up1;
            up1 = ui;
        }
    };
    int j = np - 2;
    load(sa, j);
    for (; j - 2 * B + 1 >= 2; j -= 2 * B) {
        load(sb, j - B);
        solve(sa, j);
        load(sa, j - 2 * B);
        solve(sb, j - B);
    }
    for (; j >= 2; j--) {
        const double2 t = w.r12(j);
        const double ui = w.u(j) - up1 * t.x - up2 * t.y;
        w.u(j) = ui;
        up2 = up1;
        up1 = ui;
    }
    // qu = Q u and the weighted sum of squares, i = 1..np in order
    // (u(1) = u(np) = 0)
    double prev = 0.0, sum = 0.0, ulast = 0.0;
    double v4 = F.v1, yv = F.y1;
    acc = F.z1;                                   // fitz(i-1)
    off = max(off, rp_exp_off(v4));
    constexpr int R = 8;                          // rows whose quotients are formed side by side
    for (i = 2; i + R - 1 < np; i += R) {
        double us[R + 1], du[R], raw[R];
        us[0] = ulast;
#pragma unroll
        for (int k = 0; k < R; k++) {
            us[k + 1] = w.u(i + k);
            du[k] = us[k + 1] - us[k];
            off = max(off, rp_exp_off_z(du[k]));
        }
        ulast = us[R];
        if (F.bits(i - 1) & ((1u << R) - 1u)) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                const double f = acc + F.dz;
                v4 = f - acc;                     // v4(i+k-1)
                acc = f;
                const RpRcp y = rp_rcp3(v4);
                yv = y.y;
                off = max(off, rp_exp_off(v4));
                ones = max(ones, rp_ones(v4));
                raw[k] = rp_div_rcp(du[k], v4, y);
            }
        } else {
#pragma unroll
            for (int k = 0; k < R; k++) {
                raw[k] = rp_div_fast(du[k], v4, yv, yv);
                acc = acc + F.dz;
            }
        }
#pragma unroll
        for (int k = 0; k < R; k++) {
            const double fin = raw[k] - prev;
            sum = sum + (fin * fin) * F.dy2;
            prev = raw[k];
        }
    }
    for (; i <= np; i++) {
        const double ui = (i < np) ? w.u(i) : 0.0;
        const double f = (i == np) ? F.zend : acc + F.dz;
        const double raw = rp_quot(ui - ulast, f - acc);
        acc = f;
        ulast = ui;
        const double fin = raw - prev;
        sum = sum + (fin * fin) * F.dy2;
        prev = raw;
    }
    const double finn = -prev;
    sum = sum + (finn * finn) * F.dy2;
    if (off >= kDivSpan || ones == 0xffffffffu) sum = rp_chol1d_ieee(w, F, p);
    return sum;
}

// utru (pppack.f90:5219-5223) of the pass just made
template <class W>
__device__ __forceinline__ double rp_utru(const W& w, const RpFit& F) {
    double utru = 0.0, ulast = 0.0, acc = F.z1;
    for (int i = 2; i <= F.np; i++) {
        const double ui = (i < F.np) ? w.u(i) : 0.0;
        const double f = (i == F.np) ? F.zend : acc + F.dz;
        utru = utru + (f - acc) * (ulast * (ulast + ui) + ui * ui);
        acc = f;
        ulast = ui;
    }
    return utru;
}

// smooth (pppack.f90:5108-5317) on the fit's Q'y; dy(i) = serr for all i.
// Returns p; w.u holds the final u; passes = chol1d passes made.
template <class W>
__device__ __forceinline__ double rp_smooth(const W& w, const RpFit& F, double s, int max_iter, uint32_t& fl,
                                            int& passes) {
    // one call site of chol1d: the passes of p = 1 (s <= 0), p = 0 and the
    // secant search follow one another in the same loop
    const double ooss = 1.0 / sqrt(s);
    double p = (s <= 0.0) ? 1.0 : 0.0;
    double q = 0.0, prevq = 0.0, prevsf = 0.0;
    passes = 0;
    for (int it = 0;; it++) {
        const double sum = rp_chol1d(w, F, p);
        passes++;
        if (s <= 0.0) break;
        if (it == 0) {
            const double sfq = 36.0 * sum;
            if (!(s < sfq)) break;
            const double oosf = 1.0 / sqrt(sfq);
            q = -(oosf - ooss) * sfq / (6.0 * rp_utru(w, F) * oosf);
            prevsf = oosf;
        } else {
            const double sfq = 36.0 * sum / ((1.0 + q) * (1.0 + q));
            if (fabs(sfq - s) <= 0.01 * s) break;
            if (it >= max_iter) { fl |= RP_FL_SPLINE; break; }
            const double oosf = 1.0 / sqrt(sfq);
            const double change = (q - prevq) / (oosf - prevsf) * (oosf - ooss);
            prevq = q;
            q = q - change;
            prevsf = oosf;
        }
        p = q / (1.0 + q);
    }
    return p;
}

// One piece of the fit: its breaks and the coefficients a(i,1..4) that
// smooth's epilogue forms (pppack.f90:5303-5316), kept between the sub-steps
// (consecutive positions mostly share their piece).
struct RpPiece {
    double x0, x1;                 // fitz(i), fitz(i+1); x0 > x1: none yet
    double a1, a2, a3, a4;
};

// interv (pppack.f90:3363-3576): the largest i <= np-1 with fitz(i) <= x,
// 1 below the first break (and for a NaN x)
template <class W>
__device__ __forceinline__ int rp_interv(const W& w, const RpFit& F, double x) {
    const int np = F.np;
    if (!(x >= w.fitz(1))) return 1;
    if (F.mono) {                  // ascending breaks: from the uniform guess to the piece
        const double t = (x - F.z1) * F.rdz;
        int i = (t < (double)(np - 2)) ? (int)t + 1 : np - 1;
        while (i > 1 && w.fitz(i) > x) i--;
        while (i < np - 1 && w.fitz(i + 1) <= x) i++;
        return i;
    }
    int lo = 1, hi = np;           // fitz(lo) <= x; answer in [lo, hi-1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (w.fitz(mid) <= x) lo = mid; else hi = mid;
    }
    return lo;
}

// ppvalu (pppack.f90:4246-4362) of the smoothing spline at x
template <class W>
__device__ __forceinline__ double rp_ppvalu(const W& w, const RpFit& F, double p, double x, int jderiv, RpPiece& pc) {
    if (!(x >= pc.x0 && x < pc.x1)) {
        const int np = F.np;
        const int i = rp_interv(w, F, x);
        const double K1 = 6.0 * (1.0 - p) * F.dy2;
        auto uu = [&](int k) -> double { return (k <= 1 || k >= np) ? 0.0 : w.u(k); };
        const double fm = w.fitz(max(i - 1, 1)), f0 = w.fitz(i), f1 = w.fitz(i + 1), f2 = w.fitz(min(i + 2, np));
        const double um = uu(i - 1), u0 = uu(i), u1 = uu(i + 1), u2 = uu(i + 2);
        const double y0 = w.y(i), y1 = w.y(i + 1);
        const double h4 = f1 - f0;
        const double yh = rp_rcp(h4);
        const double rm = rp_div_by(u1 - u0, h4, yh);                              // raw(i+1)
        const double fi = (i == 1) ? rm - 0.0 : rm - rp_quot(u0 - um, f0 - fm);
        const double fn = (i + 1 == np) ? -rm : rp_quot(u2 - u1, f2 - f1) - rm;
        const double a1i = y0 - K1 * fi;
        const double a1n = y1 - K1 * fn;
        const double a3i = u0 * 6.0 * p;
        const double a3n = u1 * 6.0 * p;
        const double a4i = rp_div_by(a3n - a3i, h4, yh);
        pc.a1 = a1i;
        pc.a2 = rp_div_by(a1n - a1i, h4, yh) - (a3i + rp_div_by(a4i, 3.0, 1.0 / 3.0) * h4) / 2.0 * h4;
        pc.a3 = a3i;
        pc.a4 = a4i;
        pc.x0 = f0;
        pc.x1 = f1;
    }
    // Horner loop of ppvalu with k = 4: value = (value/fmmjdr)*h + coef(m)
    const double h = x - pc.x0;
    double value = 0.0;
    if (jderiv == 0) {
        value = (value / 4.0) * h + pc.a4;
        value = rp_div_by(value, 3.0, 1.0 / 3.0) * h + pc.a3;
        value = (value / 2.0) * h + pc.a2;
        value = (value / 1.0) * h + pc.a1;
    } else {
        value = (value / 3.0) * h + pc.a4;
        value = (value / 2.0) * h + pc.a3;
        value = (value / 1.0) * h + pc.a2;
    }
    return value;
}

// ----------------------------------------------------------------- VTurb

// VTurb (ver_turb_module.f90:31-329).  The 2-D quantities at (Xpar, Ypar)
// are those of RK stage 1 (identical operations and operands).
template <typename T, class W>
__device__ __forceinline__ double rp_vturb(const RpStepArgs& A, const RpGridDev& g, const StageState& S, double Zpar,
                                           uint32_t pid, uint32_t& fl, const W& w) {
    const int sw = g.N + 1;
    const int np = (int)((double)sw * A.sub);
    const double tdepth = S.tdepth, zeta = S.zeta;
    const double h = -1.0 * tdepth;
    const ZCtx zx = rp_zctx(g.vtransform, g.hc, h);
    // column z(k), KH(k) (ver_turb_module.f90:100-124)
    const double* cw = S.rc.wet4 ? S.rc.cb : S.rc.ci;
    const int64_t o[4] = {S.rc.o00, S.rc.o10, S.rc.o11, S.rc.o01};
    bool asc = true;               // the levels ascend
    double z1 = 0.0, ztop = 0.0, k1 = 0.0, ktop = 0.0;
    // the corners' three slots of a level, loaded a level ahead of their use
    const T* aks = reinterpret_cast<const T*>(g.aks);
    const T* col[4];
#pragma unroll
    for (int q = 0; q < 4; q++) col[q] = aks + o[q] * sw * RP_SLOTS;
    T nb[4], nc[4], nf[4];
    double ns = __ldg(g.sw), ncs = __ldg(g.csw);
    auto fetch = [&](int k) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const T* c = col[q] + (k - 1) * RP_SLOTS;
            nb[q] = __ldg(c + g.sb);
            nc[q] = __ldg(c + g.sc);
            nf[q] = __ldg(c + g.sf);
        }
        ns = __ldg(g.sw + k - 1);
        ncs = __ldg(g.csw + k - 1);
    };
    fetch(1);
#pragma unroll 2
    for (int k = 1; k <= sw; k++) {
        const double s = ns, cs = ncs;
        double K3[3], z3[3];
        K3[0] = cw[0] * (double)nb[0] + cw[1] * (double)nb[1] + cw[2] * (double)nb[2] + cw[3] * (double)nb[3];
        K3[1] = cw[0] * (double)nc[0] + cw[1] * (double)nc[1] + cw[2] * (double)nc[2] + cw[3] * (double)nc[3];
        K3[2] = cw[0] * (double)nf[0] + cw[1] * (double)nf[1] + cw[2] * (double)nf[2] + cw[3] * (double)nf[3];
        fetch(min(k + 1, sw));
        if (g.vtransform == 2) {
            const double Sk = rp_div_by(g.hc * s + h * cs, zx.den, zx.yden);
            z3[0] = S.zb + (S.zb + h) * Sk;
            z3[1] = S.zc + (S.zc + h) * Sk;
            z3[2] = S.zf + (S.zf + h) * Sk;
        } else {
            z3[0] = rp_zlevel_c(zx, s, cs, S.zb);
            z3[1] = rp_zlevel_c(zx, s, cs, S.zc);
            z3[2] = rp_zlevel_c(zx, s, cs, S.zf);
        }
        double zk, kk;
        rp_polintd2(A.pi, z3, K3, zk, kk);
        w.u(k) = zk;
        if (k == 1) {
            z1 = zk;
            k1 = kk;
        } else {
            asc = asc && (zk > ztop);
            const double m = rp_quot(ktop - kk, ztop - zk);  // linint's line on [z(k-1), z(k)]
            w.set_r12(k - 1, m, ktop - m * ztop);
        }
        ztop = zk;
        ktop = kk;
    }
    // resample to np points (ver_turb_module.f90:126-136), linint per point;
    // setupq's Q'y (pppack.f90:4816-4822) on the way.  On
    // ascending levels linint's bisection ends on the last level at or below
    // the point, which the ascending points reach by walking up.
    const double dz = (ztop - z1) / (double)(np - 1);
    RpFit F;
    F.np = np;
    F.mono = asc && dz > 1e-9 * fmax(fabs(z1), fabs(ztop));
    F.z1 = z1;
    F.dz = dz;
    F.zend = ztop;
    F.rdz = 1.0 / dz;
    F.serr = A.serr;
    F.dy2 = A.serr * A.serr;
#pragma unroll
    for (int q = 0; q < kChgWords; q++) F.chg[q] = 0u;
    {
        w.fitz(1) = z1;
        w.y(1) = k1;
        int j = 1;                               // the point's bracket [z(j), z(j+1)]
        double zn = w.u(2);
        double2 ln = w.r12(1), ln2 = w.r12(2);   // its line and the next bracket's
        double x = z1, fprev = z1, yprev = k1, dprev = 0.0;
        double v4 = 0.0, yv = 0.0;
        for (int i = 2; i <= np; i++) {
            double yi;
            if (i < np) {
                x = x + dz;
                if (asc) {
                    while (j < sw - 1 && zn <= x) {
                        j++;
                        zn = w.u(j + 1);
                        ln = ln2;
                        ln2 = w.r12(j + 1);      // read a bracket ahead of its use
                    }
                } else {
                    int jlo = 1, jhi = sw;
                    for (;;) {
                        const int k = (jhi + jlo) / 2;
                        if (w.u(k) > x) jhi = k; else jlo = k;
                        if (jhi - jlo == 1) break;
                    }
                    ln = w.r12(jlo);
                }
                yi = ln.x * x + ln.y;
            } else {
                x = ztop;
                yi = ktop;
            }
            w.fitz(i) = x;
            w.y(i) = yi;
            const double v = x - fprev;          // v4(i-1)
            if (i == 2 || !(v == v4)) {
                v4 = v;
                yv = rp_rcp(v);
                if (i > 2) {
#pragma unroll
                    for (int q = 0; q < kChgWords; q++)
                        F.chg[q] |= (((i - 1) >> 5) == q) ? 1u << ((i - 1) & 31) : 0u;
                }
            }
            if (i == 2) {
                F.v1 = v;
                F.y1 = yv;
            }
            if (i == 3) F.v2 = v;
            if (i == 4) {
                F.v3 = v;
                F.f4 = x;
            }
            const double diff = rp_div_by(yi - yprev, v, yv);
            if (i > 2) w.qty(i - 1) = diff - dprev;
            dprev = diff;
            fprev = x;
            yprev = yi;
        }
        F.r1 = A.serr / F.v1;
        F.r2 = A.serr / F.v2;
        F.r3 = A.serr / F.v3;
        const unsigned lanes = __activemask();
#pragma unroll
        for (int q = 0; q < kChgWords; q++) F.chg[q] = __reduce_or_sync(lanes, F.chg[q]);
    }
    int passes;
    const double p = rp_smooth(w, F, A.smth, A.spline_max_iter, fl, passes);
    if (A.spl) rp_count_fit(A.spl, passes);

    // random displacement sub-steps (ver_turb_module.f90:231-293)
    const double deltat = A.deltat;
    double ParZc = Zpar, dev_next = 0.0;
    RpPiece pc;
    pc.x0 = 1.0;
    pc.x1 = 0.0;
#pragma unroll 1
    for (int i = 1; i <= A.loop; i++) {
        double DEV;                              // draw 1+i; pairs (2,3), (4,5), ...
        if (i & 1) rp_normal2(A, pid, (uint32_t)(1 + i), i < A.loop, DEV, dev_next);
        else DEV = dev_next;
        double Kprimec = 0.0;
        if (ParZc <= tdepth || ParZc >= zeta) Kprimec = 0.0;
        else Kprimec = rp_ppvalu(w, F, p, ParZc, 1, pc);
        const double KprimeZc = Kprimec * deltat;
        const double Z3rdc = ParZc + 0.5 * KprimeZc;
        double KH3rdc;
        if (Z3rdc < tdepth || Z3rdc > zeta) {
            KH3rdc = A.aksback;
        } else {
            KH3rdc = rp_ppvalu(w, F, p, Z3rdc, 0, pc);
            if (KH3rdc < A.aksback) KH3rdc = A.aksback;
        }
        const double r = 1.0;
        const double dTz = KprimeZc + DEV * sqrt(2.0 / r * KH3rdc * deltat);
        ParZc = ParZc + dTz;
        if (ParZc <= tdepth) ParZc = tdepth + fabs(ParZc - tdepth);
        if (ParZc >= zeta) ParZc = zeta - fabs(ParZc - zeta);
    }
    return ParZc - Zpar;
}

// ------------------------------------------------------------ one particle

// Skip tests of update_particles (ROMSPath.f90:672-690).
__device__ __forceinline__ bool rp_active(const RpStepArgs& A, int64_t n) {
    const RpParticlesDev& P = A.p;
    if (A.ix[2] <= P.dob[n]) return false;
    if (P.status[n] == 9.0) return false;
    if (A.oob && !P.isin[n]) return false;
    return true;
}

// VTurb of one particle on its own (the first kernel of the step):
// the stage-1 z clamp of find_currents (advection_module.f90:171-183) is
// applied first when RK4 runs, exactly as RKAdvect hands Zpar to VTurb.
template <typename T, class W>
__device__ void rp_vturb_one(const RpStepArgs& A, int64_t n, const W& w, double* turbv) {
    const RpParticlesDev& P = A.p;
    if (!rp_active(A, n)) return;
    uint32_t fl = 0;
    const int gid = P.gid[n];
    const RpGridDev& g = A.g[gid - 1];
    const double Xpar = P.x[n], Ypar = P.y[n];
    double Zpar = P.z[n];
    StageState S1;
    rp_rho_cell(g, Xpar, Ypar, S1.rc, fl);
    S1.tdepth = -1.0 * rp_bil(g.h, S1.rc);
    S1.zb = rp_zeta_at<T>(g, S1.rc, g.sb);
    S1.zc = rp_zeta_at<T>(g, S1.rc, g.sc);
    S1.zf = rp_zeta_at<T>(g, S1.rc, g.sf);
    S1.zeta = rp_polintd(A.pi, S1.zb, S1.zc, S1.zf);
    if (A.scheme == 1) {
        if (Zpar < S1.tdepth) Zpar = S1.tdepth + RP_F_0P001;
        if (Zpar > S1.zeta) Zpar = S1.zeta - RP_F_0P001;
    }
    turbv[n] = rp_vturb<T>(A, g, S1, Zpar, P.pid[n], fl, w);
    if (fl) P.flags[n] |= fl;
}

// getInterpStr (interpolation_module.f90:964-1174) of one slot on the u or
// v corner set: the same edge and dry-corner rules as u and v in getInterp3D.
template <typename T>
__device__ __forceinline__ double rp_str_at(const void* f, const UVCell& c, int slot) {
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = c.use[k] ? rp_ld<T>(f, c.o[k] * RP_SLOTS + slot) : 0.0;
    return c.cff[0] * v[0] + c.cff[1] * v[1] + c.cff[2] * v[2] + c.cff[3] * v[3];
}

// getInterp3D of salt or temp, ztype 1 (interpolation_module.f90:529-558,
// 769-809): the rho corner set (bilinear, inverse distance with a dry
// corner) on the rho levels of the slot's own zeta.
// wcf: under WETDRY the slot's weights from its wetdry_mask_rho
// (rp_rho_wd_weights, formed once per cell by the caller), else null.
template <typename T>
__device__ __forceinline__ double rp_tracer_at(const RpGridDev& g, const void* f, const RhoCell& c, double zeta,
                                               double depth, double zpar, int slot, const double* wcf) {
    LevelPick L;
    rp_walk_rho(g, zeta, depth, zpar, L);
    return rp_col_rho<T>(f, c, wcf ? wcf : (c.wet4 ? c.cb : c.ci), g.N, L, slot);
}

// The diagnostics that close update_particles' particle loop
// (ROMSPath.f90:935-986), at the particle's new position and grid, with
// the step's tdepth: height above bottom and, where it reaches a new
// minimum, the bottom stress (WriteBottom); salinity and temperature and
// their running sums (SaltTempOn, SaltTempMean).  Out of line: the step's
// registers are not spent on it when the diagnostics are off.
template <typename T>
__device__ __noinline__ void rp_diag_one(const RpStepArgs& A, int64_t n, double tdepth, uint32_t& fl) {
    const RpParticlesDev& P = A.p;
    const RpGridDev& g = A.g[P.gid[n] - 1];
    const double X = P.x[n], Y = P.y[n], Z = P.z[n];
    if (A.diag & RP_DIAG_BOTTOM_D) {                       // 935-952
        const double btemp = -1.0 * tdepth + Z;
        const double hob0 = P.hob[n];
        const double hob = (btemp < hob0) ? btemp : hob0;
        P.hob[n] = hob;
        if (btemp == hob) {
            const int sl[3] = {g.sb, g.sc, g.sf};
            double su[3], sv[3];
            UVCell c;
            if (A.wetdry) {                                // each slot's wetdry_mask_u / _v
                for (int q = 0; q < 3; q++) {
                    rp_u_cell(g, X, Y, c, fl, g.wd_u, RP_SLOTS, sl[q]);
                    su[q] = rp_str_at<T>(g.bustr, c, sl[q]);
                    rp_v_cell(g, X, Y, c, fl, g.wd_v, RP_SLOTS, sl[q]);
                    sv[q] = rp_str_at<T>(g.bvstr, c, sl[q]);
                }
            } else {
                rp_u_cell(g, X, Y, c, fl);
                for (int q = 0; q < 3; q++) su[q] = rp_str_at<T>(g.bustr, c, sl[q]);
                rp_v_cell(g, X, Y, c, fl);
                for (int q = 0; q < 3; q++) sv[q] = rp_str_at<T>(g.bvstr, c, sl[q]);
            }
            P.bustr[n] = rp_polintd(A.pi, su[0], su[1], su[2]);
            P.bvstr[n] = rp_polintd(A.pi, sv[0], sv[1], sv[2]);
        }
    }
    if (A.diag & RP_DIAG_SALTTEMP_D) {                     // 962-986
        RhoCell c;
        rp_rho_cell(g, X, Y, c, fl);
        const double zb = rp_zeta_at<T>(g, c, g.sb);
        const double zc = rp_zeta_at<T>(g, c, g.sc);
        const double zf = rp_zeta_at<T>(g, c, g.sf);
        double wcf[3][4];                                  // WETDRY: each slot's weights, once
        if (A.wetdry) {
            rp_rho_wd_weights(g, c, g.sb, wcf[0], fl);
            rp_rho_wd_weights(g, c, g.sc, wcf[1], fl);
            rp_rho_wd_weights(g, c, g.sf, wcf[2], fl);
        }
        const double* wb = A.wetdry ? wcf[0] : nullptr;
        const double* wc = A.wetdry ? wcf[1] : nullptr;
        const double* wf = A.wetdry ? wcf[2] : nullptr;
        const double s = rp_polintd(A.pi, rp_tracer_at<T>(g, g.salt, c, zb, tdepth, Z, g.sb, wb),
                                    rp_tracer_at<T>(g, g.salt, c, zc, tdepth, Z, g.sc, wc),
                                    rp_tracer_at<T>(g, g.salt, c, zf, tdepth, Z, g.sf, wf));
        const double t = rp_polintd(A.pi, rp_tracer_at<T>(g, g.temp, c, zb, tdepth, Z, g.sb, wb),
                                    rp_tracer_at<T>(g, g.temp, c, zc, tdepth, Z, g.sc, wc),
                                    rp_tracer_at<T>(g, g.temp, c, zf, tdepth, Z, g.sf, wf));
        P.salt[n] = s;
        P.temp[n] = t;
        if (A.diag & RP_DIAG_MEAN_D) {
            P.mean_salt[n] = P.mean_salt[n] + s;
            P.mean_temp[n] = P.mean_temp[n] + t;
        }
    }
}

// behave's response to the four standard deviations at the particle
// (behavior_module.f90:285-375): 4 laplace, 2 normal and 1 uniform draws,
// the Fuchs swim / sink choice into par(:,pAcc/pVort/pbehaveW/pSSF);
// returns the vertical velocity wb (cm/s).  Real powers are pinned as
// x**2.0D0 = x*x, r**3.0D0 = (r*r)*r, x**0.5D0 = sqrt(x); exp and log are
// this project's own.  Shared by both forms of the step.
__device__ __forceinline__ double rp_behave_swim(const RpStepArgs& A, int64_t n, uint32_t pid, double stdaccturbu,
                                                 double stdvortturb, double stdaccwaveu, double stdaccwavev) {
    const RpBehaviorDev& b = A.beh;
    const double G = 980.0, RHOF = 1.026, MU = 0.010260, RHOP = 1.06;   // ROMSPath.h:15-19
    double wb;
    const uint32_t d0 = 2u + (uint32_t)A.loop;
    const double vortturbu = RP_MUL(stdvortturb, rp_laplace_of(rp_uniform(A, pid, d0, 0)));
    const double vortturbv = RP_MUL(stdvortturb, rp_laplace_of(rp_uniform(A, pid, d0, 1)));
    const double vorttot = sqrt(RP_ADD(RP_MUL(vortturbu, vortturbu), RP_MUL(vortturbv, vortturbv)));
    const double accturbu = RP_MUL(stdaccturbu, rp_laplace_of(rp_uniform(A, pid, d0, 2)));
    const double accturbv = RP_MUL(stdaccturbu, rp_laplace_of(rp_uniform(A, pid, d0, 3)));
    const double accwaveu = RP_MUL(stdaccwaveu, rp_normal(A, pid, d0));
    const double accwavev = RP_MUL(stdaccwavev, rp_normal(A, pid, d0 + 1));
    const double au = RP_ADD(accturbu, accwaveu), av = RP_ADD(accturbv, accwavev);
    const double acctot = sqrt(RP_ADD(RP_MUL(au, au), RP_MUL(av, av)));
    const double c1v = 2.0 / rp_log(b.vort_cr / b.vort_sat);
    const double c2v = RP_MUL(c1v, rp_log(vorttot / sqrt(RP_MUL(b.vort_cr, b.vort_sat))));
    const double c1a = 2.0 / rp_log(b.acc_cr / b.acc_sat);
    const double c2a = RP_MUL(c1a, rp_log(acctot / sqrt(RP_MUL(b.acc_cr, b.acc_sat))));
    const double ev = rp_exp(RP_MUL(-2.0, c2v)), ea = rp_exp(RP_MUL(-2.0, c2a));
    const double pswimv = RP_ADD(RP_SUB(b.b1pv, b.b0pv) / RP_ADD(1.0, ev), b.b0pv);
    const double pswima = RP_ADD(RP_SUB(b.b1pa, b.b0pa) / RP_ADD(1.0, ea), b.b0pa);
    const double pswim = (b.va_flag == 1) ? pswimv : (b.va_flag == 2) ? pswima : ((pswima < pswimv) ? pswima : pswimv);
    const double wswimv = RP_ADD(RP_MUL(RP_SUB(b.b1w, b.b0wv), 1.0) / RP_ADD(1.0, ev), b.b0wv);
    const double wswima = RP_ADD(RP_MUL(RP_SUB(b.b1w, b.b0wa), 1.0) / RP_ADD(1.0, ea), b.b0wa);
    const double wswim = (b.va_flag == 1) ? wswimv : (b.va_flag == 2) ? wswima : RP_ADD(wswima, wswimv);
    const double r = b.initsize / 2.0e4;
    const double t1 = RP_MUL(RP_MUL(RP_MUL(RP_MUL(4.0 / 3.0, G), RP_MUL(RP_MUL(r, r), r)), RHOF), RHOP - RHOF);
    const double wsink = RP_SUB(RP_MUL(3.0, MU), sqrt(RP_ADD(t1, RP_MUL(9.0, RP_MUL(MU, MU))))) / RP_MUL(r, RHOF);
    double ssf;
    if (rp_uniform(A, pid, d0, 4) < pswim) {
        wb = wswim;
        ssf = 0.0;
    } else {
        wb = wsink;
        ssf = 1.0;
    }
    const RpParticlesDev& P = A.p;
    P.acc[n] = acctot / 100.0;
    P.vort[n] = vorttot;
    P.behavew[n] = wb;
    P.ssf[n] = ssf;
    return wb;
}

// ZBehav of behave (381-391) from the vertical velocity wb
__device__ __forceinline__ double rp_behave_z(const RpStepArgs& A, double wb) {
    if (A.beh.behavior == 1) return RP_MUL(A.beh.swimfast, (double)A.idt);
    if (A.beh.behavior == 10) return RP_MUL(wb, (double)A.idt) / 100.0;
    return 0.0;
}

// getInterp3D of a behave field, ztype 2 (the w levels) at one slot; wcf
// as for rp_tracer_at
template <typename T>
__device__ __forceinline__ double rp_wfield_at(const RpGridDev& g, const void* f, const RhoCell& c, double zeta,
                                               double depth, double zpar, int slot, const double* wcf, uint32_t& fl) {
    LevelPick L;
    rp_walk_w(g, zeta, depth, zpar, L, fl);
    return rp_col_rho<T>(f, c, wcf ? wcf : (c.wet4 ? c.cb : c.ci), g.N + 1, L, slot);
}

// behave (behavior_module.f90:186-393) at the step's (Xpar, Ypar, Zpar) in
// the particle's grid: with Process_VA / Process_WA the standard deviations
// of turbulent acceleration and vorticity and of wave acceleration at the
// particle (240-280), then the response; returns ZBehav.  Out of line: the
// passive step keeps its registers.
template <typename T>
__device__ __noinline__ double rp_behave(const RpStepArgs& A, int64_t n, const RpGridDev& g, double Xpar,
                                         double Ypar, double Zpar, uint32_t pid, uint32_t& fl) {
    const RpBehaviorDev& b = A.beh;
    double wb = 0.0;
    if (b.va || b.wa) {
        RhoCell c;
        rp_rho_cell(g, Xpar, Ypar, c, fl);
        const double depth = -1.0 * rp_bil(g.h, c);
        const double zt[3] = {rp_zeta_at<T>(g, c, g.sb), rp_zeta_at<T>(g, c, g.sc), rp_zeta_at<T>(g, c, g.sf)};
        const int sl[3] = {g.sb, g.sc, g.sf};
        double wcf[3][4];                                  // WETDRY: each slot's weights, once
        if (A.wetdry)
            for (int q = 0; q < 3; q++) rp_rho_wd_weights(g, c, sl[q], wcf[q], fl);
        auto wq = [&](int q) -> const double* { return A.wetdry ? wcf[q] : nullptr; };
        double ey[3], stdaccturbu = 0.0, stdvortturb = 0.0, stdaccwaveu = 0.0, stdaccwavev = 0.0;
        if (b.va) {
            for (int q = 0; q < 3; q++) ey[q] = rp_wfield_at<T>(g, g.turbaccel, c, zt[q], depth, Zpar, sl[q], wq(q), fl);
            stdaccturbu = rp_polintd(A.pi, ey[0], ey[1], ey[2]);
            for (int q = 0; q < 3; q++) ey[q] = rp_wfield_at<T>(g, g.turbvort, c, zt[q], depth, Zpar, sl[q], wq(q), fl);
            stdvortturb = rp_polintd(A.pi, ey[0], ey[1], ey[2]);
            stdaccturbu = RP_MUL(stdaccturbu, 100.0);
        }
        if (b.wa) {
            for (int q = 0; q < 3; q++) ey[q] = rp_wfield_at<T>(g, g.waveaccelu, c, zt[q], depth, Zpar, sl[q], wq(q), fl);
            stdaccwaveu = rp_polintd(A.pi, ey[0], ey[1], ey[2]);
            for (int q = 0; q < 3; q++) ey[q] = rp_wfield_at<T>(g, g.waveaccelv, c, zt[q], depth, Zpar, sl[q], wq(q), fl);
            stdaccwavev = rp_polintd(A.pi, ey[0], ey[1], ey[2]);
            stdaccwaveu = RP_MUL(stdaccwaveu, 100.0);
            stdaccwavev = RP_MUL(stdaccwavev, 100.0);
        }
        wb = rp_behave_swim(A, n, pid, stdaccturbu, stdvortturb, stdaccwaveu, stdaccwavev);
    }
    return rp_behave_z(A, wb);
}

// One particle of update_particles; with VTurb on, turbv holds the VTurb
// kernel's displacements.
template <typename T>
__device__ void rp_update_one(const RpStepArgs& A, int64_t n, const double* turbv) {
    const RpParticlesDev& P = A.p;
    if (!rp_active(A, n)) return;                          // ROMSPath.f90:672-690
    P.age[n] = P.age[n] + (double)(float)A.idt;            // 693

    uint32_t fl = 0;
    int gid = P.gid[n];
    const RpGridDev& g = A.g[gid - 1];
    const uint32_t pid = P.pid[n];
    const double Xpar = P.x[n], Ypar = P.y[n], z0 = P.z[n];
    double Zpar = z0;

    double pm, pn;                                         // 727-728
    {
        const int I = rp_ifloor(Xpar), J = rp_ifloor(Ypar);
        const double X = Xpar - (double)I, Y = Ypar - (double)J;
        const int i0 = rp_clamp(I, 1, g.nx, fl), i1 = rp_clamp(I + 1, 1, g.nx, fl);
        const int j0 = rp_clamp(J, 1, g.ny, fl), j1 = rp_clamp(J + 1, 1, g.ny, fl);
        const int64_t o00 = (int64_t)(j0 - 1) * g.nx + (i0 - 1), o10 = (int64_t)(j0 - 1) * g.nx + (i1 - 1);
        const int64_t o11 = (int64_t)(j1 - 1) * g.nx + (i1 - 1), o01 = (int64_t)(j1 - 1) * g.nx + (i0 - 1);
        const double c0 = (1 - X) * (1 - Y), c1 = X * (1 - Y), c2 = X * Y, c3 = (1 - X) * Y;
        pm = c0 * __ldg(g.pm + o00) + c1 * __ldg(g.pm + o10) + c2 * __ldg(g.pm + o11) + c3 * __ldg(g.pm + o01);
        pn = c0 * __ldg(g.pn + o00) + c1 * __ldg(g.pn + o10) + c2 * __ldg(g.pn + o11) + c3 * __ldg(g.pn + o01);
    }

    double AdvectX = 0.0, AdvectY = 0.0, AdvectZ = 0.0;
    if (A.scheme == 1) {                                   // RKAdvect, advection_module.f90:20-125
        // stages 2-4 start from the (stage-1 clamped) start position plus the
        // previous stage's slope times idt/2; a loop, so that the stage's code
        // (about 2,000 instructions) stays in the instruction cache
        const double didt = (double)A.idt;
        double Uad = 0.0, Vad = 0.0, Wad = 0.0, P_U = 0.0, P_V = 0.0, P_W = 0.0;
#pragma unroll 1
        for (int st = 0; st < 4; st++) {
            double xs = Xpar, ys = Ypar, zs = Zpar;
            if (st > 0) {
                xs = Xpar + Uad * pm * didt / 2.0;
                ys = Ypar + Vad * pn * didt / 2.0;
                zs = Zpar + Wad * didt / 2.0;
            }
            StageState St;
            rp_find_currents<T>(A, g, xs, ys, zs, Uad, Vad, Wad, St, fl);
            const double kn_u = Uad * pm, kn_v = Vad * pn, kn_w = Wad;
            if (st == 0) {
                Zpar = zs;                                 // Z is INOUT in find_currents
                P_U = kn_u;
                P_V = kn_v;
                P_W = kn_w;
            } else {
                const double c = (st == 3) ? 1.0 : 2.0;
                P_U = P_U + c * kn_u;
                P_V = P_V + c * kn_v;
                P_W = P_W + c * kn_w;
            }
        }
        AdvectX = didt * (P_U / 6.0);
        AdvectY = didt * (P_V / 6.0);
        AdvectZ = didt * (P_W / 6.0);
    }

    double TurbHx = 0.0, TurbHy = 0.0;
    if (A.hturb_on) {                                      // HTurb, hor_turb_module.f90:30-51
        const double r = 1.0;
        const double KM = A.khturb[gid - 1];
        const double devX = rp_normal(A, pid, 0u);
        const double devY = rp_normal(A, pid, 1u);
        TurbHx = devX * sqrt(2.0 / r * KM * (double)A.idt);
        TurbHy = devY * sqrt(2.0 / r * KM * (double)A.idt);
    }
    TurbHx = TurbHx * pm;
    TurbHy = TurbHy * pn;

    double TurbV = 0.0;
    if (A.vturb_on) TurbV = turbv[n];                      // VTurb, 783
    double ZBehav = 0.0;                                   // behave(), 800-804
    if (A.beh.behavior || A.beh.va || A.beh.wa) ZBehav = rp_behave<T>(A, n, g, Xpar, Ypar, Zpar, pid, fl);

    // new position and nest hand-off (821-836)
    const double newXpos = P.x[n] + AdvectX + TurbHx;
    const double newYpos = P.y[n] + AdvectY + TurbHy;
    double tempX = newXpos, tempY = newYpos;
    bool ingrid = false, obound = false;
    for (int i = 1; i <= A.ngrid; i++) {
        tempX = g.scl[i - 1][0] * newXpos + g.off[i - 1][0];
        tempY = g.scl[i - 1][1] * newYpos + g.off[i - 1][1];
        rp_bounds(A.g[i - 1], tempX, tempY, ingrid, obound);
        if (ingrid) { gid = i; break; }
    }
    const RpGridDev& gn = A.g[gid - 1];
    RhoCell rn;
    rp_rho_cell(gn, tempX, tempY, rn, fl);
    const double tdepth = -1.0 * rp_bil(gn.h, rn);         // 837
    const double e0 = 1.0 * rp_zeta_at<T>(gn, rn, gn.sb);
    const double e1 = 1.0 * rp_zeta_at<T>(gn, rn, gn.sc);
    const double e2 = 1.0 * rp_zeta_at<T>(gn, rn, gn.sf);
    const double P_zeta = rp_polintd(A.pi, e0, e1, e2);    // 843
    P.wd[n] = (-1.0 * tdepth) + P_zeta;
    P.zeta[n] = P_zeta;
    P.bath[n] = -1.0 * tdepth;
    bool hbot = false, htop = false;
    double newZpos;
    if (A.nsb == 0) {                                      // 852-872
        newZpos = z0 + AdvectZ + TurbV + ZBehav;
        if (newZpos < tdepth) { newZpos = tdepth + fabs(newZpos - tdepth); hbot = true; }
        if (newZpos > P_zeta) { newZpos = P_zeta - fabs(newZpos - P_zeta); htop = true; }
    } else if (A.nsb == 1) {
        newZpos = P_zeta - A.vertdist;
    } else {
        newZpos = tdepth + A.vertdist;
    }
    if (ingrid) {                                          // 874-892
        P.isin[n] = 1;
        P.x[n] = tempX;
        P.y[n] = tempY;
        P.z[n] = newZpos;
        double st = 1.0;
        if (htop) st = RP_F_1P1;
        if (hbot) st = RP_F_1P2;
        P.status[n] = st;
        P.gid[n] = gid;
    } else if (obound) {
        P.isin[n] = 0;
        P.gid[n] = A.ngrid;
        P.status[n] = -8.0;
    } else {
        P.isin[n] = 1;
        P.status[n] = -9.0;
    }
    if (A.diag) rp_diag_one<T>(A, n, tdepth, fl);
    if (fl) P.flags[n] |= fl;
}
