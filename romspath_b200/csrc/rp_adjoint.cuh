// rp_adjoint.cuh -- the particle step written once over a generic scalar S
// (double, or Dual<4> carrying derivatives with respect to the step's
// starting x, y, z and the diffusivity multiplier kappa), for the adjoint
// pair rp_forward / rp_backward and the tangent-linear reference.
//
// The model is the FP64 step of update_particles (ROMSPath.f90:662-905):
// RK4 with the reference's interpolation (bilinear, inverse-distance,
// level walk, polintd in time), HTurb, VTurb with the smoothing-spline
// fit, hand-off and reflections.  Differences from the exact form that
// make it differentiable and replayable:
//   * kappa multiplies the diffusivity data (AKs) the fit is made to; at a
//     fixed smoothing parameter the fit is linear in the data, so this is
//     the same as scaling the fitted K(z);
//   * the fit uses exactly uniform breaks (as the mixed form) and a given
//     smoothing parameter p: rp_forward finds p by smooth()'s secant search
//     (pppack.f90:5108-5317) and records it per particle and step; replay,
//     tangent and adjoint runs reuse the recorded p (the search is a
//     discrete iteration, treated like the reflections: piecewise);
//   * the noise is frozen (Philox draws keyed on particle id and step).
// Branches (level brackets, reflections, land rejection, hand-off, pieces
// of the spline) are taken on values, so derivatives are those of the
// piece the trajectory is on.
#pragma once

#include "rp_step.cuh"

// ------------------------------------------------------------ dual numbers

template <int N>
struct Dual {
    double v;
    double d[N];
    __device__ __forceinline__ Dual() {}
    __device__ __forceinline__ Dual(double x) : v(x) {
#pragma unroll
        for (int i = 0; i < N; i++) d[i] = 0.0;
    }
};

template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v + b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] + b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v - b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] - b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a) {
    Dual<N> r;
    r.v = -a.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = -a.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v * b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    const double ib = 1.0 / b.v;
    r.v = a.v * ib;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
    return r;
}
// mixed with double
template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, double b) {
    Dual<N> r = a;
    r.v = a.v + b;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator+(double a, const Dual<N>& b) { return b + a; }
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, double b) {
    Dual<N> r = a;
    r.v = a.v - b;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(double a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a - b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = -b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, double b) {
    Dual<N> r;
    r.v = a.v * b;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * b;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(double a, const Dual<N>& b) { return b * a; }
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, double b) {
    Dual<N> r;
    r.v = a.v / b;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] / b;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(double a, const Dual<N>& b) {
    return Dual<N>(a) / b;
}

__device__ __forceinline__ double aval(double x) { return x; }
template <int N>
__device__ __forceinline__ double aval(const Dual<N>& x) { return x.v; }

__device__ __forceinline__ double asqrt(double x) { return sqrt(x); }
template <int N>
__device__ __forceinline__ Dual<N> asqrt(const Dual<N>& a) {
    Dual<N> r;
    r.v = sqrt(a.v);
    const double k = (r.v > 0.0) ? 0.5 / r.v : 0.0;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * k;
    return r;
}
template <class S>
__device__ __forceinline__ S aabs(const S& a) {
    return (aval(a) < 0.0) ? -a : a;
}

// ------------------------------------------------------------- stencils

template <class S>
struct ARho {
    int64_t o[4];
    S cb[4];
    S ci[4];
    bool wet4;
};

template <class S>
__device__ __forceinline__ void a_rho_cell(const RpGridDev& g, const S& ip, const S& jp, ARho<S>& c, uint32_t& fl) {
    const int I = rp_ifloor(aval(ip)), J = rp_ifloor(aval(jp));
    const S X = ip - (double)I, Y = jp - (double)J;
    const int i0 = rp_clamp(I, 1, g.nx, fl), i1 = rp_clamp(I + 1, 1, g.nx, fl);
    const int j0 = rp_clamp(J, 1, g.ny, fl), j1 = rp_clamp(J + 1, 1, g.ny, fl);
    c.o[0] = (int64_t)(j0 - 1) * g.nx + (i0 - 1);
    c.o[1] = (int64_t)(j0 - 1) * g.nx + (i1 - 1);
    c.o[2] = (int64_t)(j1 - 1) * g.nx + (i1 - 1);
    c.o[3] = (int64_t)(j1 - 1) * g.nx + (i0 - 1);
    c.cb[0] = (1.0 - X) * (1.0 - Y);
    c.cb[1] = X * (1.0 - Y);
    c.cb[2] = X * Y;
    c.cb[3] = (1.0 - X) * Y;
    double m[4];
#pragma unroll
    for (int k = 0; k < 4; k++) m[k] = (double)__ldg(g.mrho + c.o[k]);
    c.wet4 = !((m[0] + m[1] + m[2] + m[3]) < 4.0);
    // getcoeff (interpolation_module.f90:1230-1273) with the exact-node pin
    S dist[4], W[4];
    dist[0] = asqrt(X * X + Y * Y);
    dist[1] = asqrt((1.0 - X) * (1.0 - X) + Y * Y);
    dist[2] = asqrt((1.0 - X) * (1.0 - X) + (1.0 - Y) * (1.0 - Y));
    dist[3] = asqrt(X * X + (1.0 - Y) * (1.0 - Y));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (aval(dist[k]) == 0.0) {
            fl |= RP_FL_NODE;
            if (m[k] != 0.0) {
#pragma unroll
                for (int q = 0; q < 4; q++) c.ci[q] = S((q == k) ? 1.0 : 0.0);
                return;
            }
            W[k] = S(0.0);
        } else {
            W[k] = m[k] / dist[k];
        }
    }
    const S WT = W[0] + W[1] + W[2] + W[3];
#pragma unroll
    for (int k = 0; k < 4; k++) c.ci[k] = (aval(WT) == 0.0) ? S(0.0) : W[k] / WT;
}

template <class S>
__device__ __forceinline__ S a_dot4(const double* a, const int64_t o[4], const S w[4]) {
    return w[0] * __ldg(a + o[0]) + w[1] * __ldg(a + o[1]) + w[2] * __ldg(a + o[2]) + w[3] * __ldg(a + o[3]);
}

// polintd (interpolation_module.f90:72-109) at the step's fixed nodes
template <class S>
__device__ __forceinline__ S a_polint(const RpPolint& P, const S& y0, const S& y1, const S& y2) {
    const S q12 = (y2 - y1) * P.re12;
    const S q01 = (y1 - y0) * P.re01;
    const S c = (P.d1 * q12 - P.d1 * q01) * P.re02;
    const S a = (P.ns == 2) ? q12 : q01;
    const S yns = (P.ns == 0) ? y0 : ((P.ns == 1) ? y1 : y2);
    return yns + P.dns * a + P.b * c;
}

template <class S>
struct AUV {
    int64_t o[4];
    S cff[4];
    bool use[4];
};

// u / v corner sets of getInterp3D (interpolation_module.f90:608-767)
template <class S>
__device__ __forceinline__ void a_uv_cell(const RpGridDev& g, const S& ip, const S& jp, bool is_u, AUV<S>& c,
                                          uint32_t& fl) {
    int ci[4], cj[4];
    double m[4];
    S X, Y;
    if (is_u) {
        const int xi_u = g.nx - 1, eta_u = g.ny;
        const int Jn = rp_ifloor(aval(jp));
        Y = jp - (double)Jn;
        const S uvI = ip - 0.5;
        const int In = rp_ifloor(aval(uvI));
        X = uvI - (double)In;
        const int j0 = rp_clamp(Jn, 1, eta_u, fl), j1 = rp_clamp(Jn + 1, 1, eta_u, fl);
        const int a = In >= xi_u ? xi_u : (In < 1 ? 1 : In);
        const int b = In >= xi_u ? xi_u : (In < 1 ? 1 : In + 1);
        ci[0] = a; ci[1] = b; ci[2] = b; ci[3] = a;
        cj[0] = j0; cj[1] = j0; cj[2] = j1; cj[3] = j1;
#pragma unroll
        for (int k = 0; k < 4; k++) c.o[k] = (int64_t)(cj[k] - 1) * xi_u + (ci[k] - 1);
#pragma unroll
        for (int k = 0; k < 4; k++) m[k] = (double)__ldg(g.mu + c.o[k]);
        if (In >= xi_u) { m[1] = 0.0; m[2] = 0.0; }
        else if (In < 1) { m[0] = 0.0; m[3] = 0.0; }
    } else {
        const int xi_v = g.nx, eta_v = g.ny - 1;
        int In = rp_ifloor(aval(ip));
        X = ip - (double)In;
        const S uvJ = jp - 0.5;
        int Jn = rp_ifloor(aval(uvJ));
        if (Jn < 1) Jn = 1;
        if (Jn > eta_v) In = eta_v;     // interpolation_module.f90:696
        Y = uvJ - (double)Jn;
        const int i0 = rp_clamp(In, 1, xi_v, fl), i1 = rp_clamp(In + 1, 1, xi_v, fl);
        ci[0] = i0; ci[1] = i1; ci[2] = i1; ci[3] = i0;
        if (Jn >= eta_v) { cj[0] = cj[1] = cj[2] = cj[3] = eta_v; }
        else { cj[0] = Jn; cj[1] = Jn; cj[2] = Jn + 1; cj[3] = Jn + 1; }
#pragma unroll
        for (int k = 0; k < 4; k++) c.o[k] = (int64_t)(cj[k] - 1) * xi_v + (ci[k] - 1);
#pragma unroll
        for (int k = 0; k < 4; k++) m[k] = (double)__ldg(g.mv + c.o[k]);
        if (Jn >= eta_v) { m[2] = 0.0; m[3] = 0.0; }
    }
    c.cff[0] = (1.0 - X) * (1.0 - Y);
    c.cff[1] = X * (1.0 - Y);
    c.cff[2] = X * Y;
    c.cff[3] = (1.0 - X) * Y;
    const double nwater = m[0] + m[1] + m[2] + m[3];
#pragma unroll
    for (int k = 0; k < 4; k++) c.use[k] = true;
    if (nwater < 4.0 && nwater > 0.0) {
#pragma unroll
        for (int k = 0; k < 4; k++) if (m[k] == 0.0) c.use[k] = false;
    } else if (nwater == 0.0) {
#pragma unroll
        for (int k = 0; k < 4; k++) { c.cff[k] = S(0.0); c.use[k] = false; }
    }
}

// getSlevel / getWlevel (grid_module.f90:513-598), h = -depth
template <class S>
__device__ __forceinline__ S a_zlev(int vt, double hc, double s, double cs, const S& zeta, const S& h) {
    if (vt == 2) {
        const S Sk = (hc * s + h * cs) / (hc + h);
        return zeta + (zeta + h) * Sk;
    } else if (vt == 1) {
        const S Sk = hc * s + (h - hc) * cs;
        return Sk + zeta * (1.0 + Sk / h);
    }
    return zeta * (1.0 + s) + hc * s + (h - hc) * cs;
}

template <class S>
struct APick {
    int ibot, itop;
    S z1, z2;
};

// level bracket of getInterp3D (interpolation_module.f90:529-582)
template <class S>
__device__ __forceinline__ void a_walk(const RpGridDev& g, bool wlev, const S& zeta, const S& depth, const S& zpar,
                                       APick<S>& L, uint32_t& fl) {
    const S h = -depth;
    const int nz = wlev ? g.N + 1 : g.N;
    const double* s = wlev ? g.sw : g.sr;
    const double* cs = wlev ? g.csw : g.csr;
    S zl1 = depth, zl2 = depth;
    int i;
    for (i = 1; i <= nz; i++) {
        zl2 = a_zlev(g.vtransform, g.hc, __ldg(s + i - 1), __ldg(cs + i - 1), zeta, h);
        if (aval(zl2) > aval(zpar)) break;
        zl1 = zl2;
    }
    if (i > nz) {
        if (wlev) fl |= RP_FL_WTOP;
        L.ibot = nz; L.itop = nz; L.z1 = S(0.5); L.z2 = S(0.5);
    } else if (i == 1) {
        if (wlev) fl |= RP_FL_WBOT;
        L.ibot = 1; L.itop = 1; L.z1 = S(0.5); L.z2 = S(0.5);
    } else {
        const S Z = (zpar - zl1) / (zl2 - zl1);
        L.ibot = i - 1; L.itop = i; L.z1 = 1.0 - Z; L.z2 = Z;
    }
}

// zcff1*zprof(Ibot) + zcff2*zprof(Itop) of one frame of a 3-D field
template <class S>
__device__ __forceinline__ S a_col(const double* f, const int64_t o[4], const S cff[4], const bool use[4], int nlev,
                                   const APick<S>& L) {
    S pb(0.0), pt(0.0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (use[k]) {
            pb = pb + cff[k] * __ldg(f + o[k] * nlev + L.ibot - 1);
            pt = pt + cff[k] * __ldg(f + o[k] * nlev + L.itop - 1);
        }
    }
    return L.z1 * pb + L.z2 * pt;
}

// The level at index k (1-based) as the picks above compare it, without
// derivatives and with 1 / (hc + h) formed once
struct ALevels {
    double hc, h, rden, zeta;
    __device__ __forceinline__ double at(const double* s, const double* cs, int k) const {
        return zeta + (zeta + h) * ((hc * __ldg(s + k - 1) + h * __ldg(cs + k - 1)) * rden);
    }
};

// The first of nz ascending levels above zpar (nz + 1: none), by bisection
__device__ __forceinline__ int a_above(const ALevels& v, const double* s, const double* cs, int nz, double zpar) {
    int lo = 0, hi = nz + 1;
#pragma unroll 1
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (v.at(s, cs, mid) > zpar) hi = mid; else lo = mid;
    }
    return hi;
}

template <class S>
__device__ __forceinline__ void a_bracket(const RpGridDev& g, const double* s, const double* cs, int nz, int i,
                                          const S& zeta, const S& h, const S& zpar, APick<S>& L) {
    if (i > nz || i == 1) {
        L.ibot = L.itop = (i == 1) ? 1 : nz;
        L.z1 = S(0.5);
        L.z2 = S(0.5);
        return;
    }
    const S z1 = a_zlev(2, g.hc, __ldg(s + i - 2), __ldg(cs + i - 2), zeta, h);
    const S z2 = a_zlev(2, g.hc, __ldg(s + i - 1), __ldg(cs + i - 1), zeta, h);
    const S Z = (zpar - z1) / (z2 - z1);
    L.ibot = i - 1;
    L.itop = i;
    L.z1 = 1.0 - Z;
    L.z2 = Z;
}

// Both brackets of getInterp3D.  Where the levels ascend (as in rp_walk2) by
// bisection on their values: walked level by level with a division each, the
// two walks were most of a stage.
template <class S>
__device__ __forceinline__ void a_walk2(const RpGridDev& g, const S& zeta, const S& depth, const S& zpar, APick<S>& Lr,
                                        APick<S>& Lw, uint32_t& fl) {
    const S h = -depth;
    const double hv = aval(h), zv = aval(zeta), pv = aval(zpar);
    if (!(g.asc && hv > 0.0 && hv < 1e30 && zv + hv > 0.0 && zv < 1e30 && pv == pv)) {
        a_walk(g, false, zeta, depth, zpar, Lr, fl);
        a_walk(g, true, zeta, depth, zpar, Lw, fl);
        return;
    }
    const ALevels v{g.hc, hv, 1.0 / (g.hc + hv), zv};
    const int N = g.N;
    a_bracket(g, g.sr, g.csr, N, a_above(v, g.sr, g.csr, N, pv), zeta, h, zpar, Lr);
    const int iw = a_above(v, g.sw, g.csw, N + 1, pv);
    if (iw > N + 1) fl |= RP_FL_WTOP;
    if (iw == 1) fl |= RP_FL_WBOT;
    a_bracket(g, g.sw, g.csw, N + 1, iw, zeta, h, zpar, Lw);
}

template <class S>
struct AStage {
    ARho<S> rc;
    S tdepth, zb, zc, zf, zeta;
};

template <class S>
__device__ __forceinline__ void a_stage_2d(const RpStepArgs& A, const AdjFrames& F, int gi, const RpGridDev& g,
                                           AStage<S>& St) {
    St.tdepth = -a_dot4(g.h, St.rc.o, St.rc.cb);
    St.zb = a_dot4(F.f[gi][0][0], St.rc.o, St.rc.ci);
    St.zc = a_dot4(F.f[gi][0][1], St.rc.o, St.rc.ci);
    St.zf = a_dot4(F.f[gi][0][2], St.rc.o, St.rc.ci);
    St.zeta = a_polint(A.pi, St.zb, St.zc, St.zf);
}

// find_currents (advection_module.f90:129-350); Z is INOUT
template <class S>
__device__ __forceinline__ void a_find_currents(const RpStepArgs& A, const AdjFrames& F, int gi, const S& X, const S& Y,
                                                S& Z, S& U, S& V, S& W, AStage<S>& St, uint32_t& fl) {
    const RpGridDev& g = A.g[gi];
    a_rho_cell(g, X, Y, St.rc, fl);
    a_stage_2d(A, F, gi, g, St);
    if (aval(Z) < aval(St.tdepth)) Z = St.tdepth + RP_F_0P001;
    if (aval(Z) > aval(St.zeta)) Z = St.zeta - RP_F_0P001;
    APick<S> Lr, Lw;
    a_walk2(g, St.zeta, St.tdepth, Z, Lr, Lw, fl);
    const int N = g.N;
    S val3[3];
    {
        AUV<S> cu;
        a_uv_cell(g, X, Y, true, cu, fl);
#pragma unroll
        for (int t = 0; t < 3; t++) val3[t] = a_col(F.f[gi][1][t], cu.o, cu.cff, cu.use, N, Lr);
        U = (A.ets == 1) ? a_polint(A.pi, val3[0], val3[0], val3[1]) : a_polint(A.pi, val3[0], val3[1], val3[2]);
    }
    {
        AUV<S> cv;
        a_uv_cell(g, X, Y, false, cv, fl);
#pragma unroll
        for (int t = 0; t < 3; t++) val3[t] = a_col(F.f[gi][2][t], cv.o, cv.cff, cv.use, N, Lr);
        V = (A.ets == 1) ? a_polint(A.pi, val3[0], val3[0], val3[1]) : a_polint(A.pi, val3[0], val3[1], val3[2]);
    }
    {
        const bool all[4] = {true, true, true, true};
        const S* cw = St.rc.wet4 ? St.rc.cb : St.rc.ci;
#pragma unroll
        for (int t = 0; t < 3; t++) val3[t] = a_col(F.f[gi][3][t], St.rc.o, cw, all, N + 1, Lw);
        W = (A.ets == 1) ? a_polint(A.pi, val3[0], val3[0], val3[1]) : a_polint(A.pi, val3[0], val3[1], val3[2]);
    }
}

// ------------------------------------------------------------- VTurb

// Workspace of one fit: column z(k), K(k) (k <= s_w) and the chol1d arrays
// (i <= np), NPMAX + 1 entries each.
template <class S, int NPMAX>
struct AFit {
    S* base;
    __device__ __forceinline__ S& zc(int k) const { return base[k]; }
    __device__ __forceinline__ S& kh(int k) const { return base[(NPMAX + 1) + k]; }
    __device__ __forceinline__ S& s1(int i) const { return base[2 * (NPMAX + 1) + i]; }
    __device__ __forceinline__ S& s2(int i) const { return base[3 * (NPMAX + 1) + i]; }
    __device__ __forceinline__ S& u(int i) const { return base[4 * (NPMAX + 1) + i]; }
    __device__ __forceinline__ S& y(int i) const { return base[5 * (NPMAX + 1) + i]; }
};
constexpr int kAdjArrays = 6;

// linint of the column at x (bisection on values; interpolation_module.f90:27-61)
template <class S, int NPMAX>
__device__ __forceinline__ S a_linint(const AFit<S, NPMAX>& w, int sw, const S& x) {
    int jlo = 1, jhi = sw;
    const double xv = aval(x);
    while (jhi - jlo > 1) {
        const int k = (jhi + jlo) / 2;
        if (aval(w.zc(k)) > xv) jhi = k; else jlo = k;
    }
    const S m = (w.kh(jlo) - w.kh(jhi)) / (w.zc(jlo) - w.zc(jhi));
    return m * x + (w.kh(jlo) - m * w.zc(jlo));
}

// chol1d (pppack.f90:1428-1566) on uniform breaks at a given p (the bands of
// the mixed form's m_chol1d).  Leaves u(1..np).
template <class S, int NPMAX>
__device__ void a_chol1d(const AFit<S, NPMAX>& w, int np, const S& hb, double p, double serr) {
    const S r = serr / hb;
    const S r2 = r * r;
    const double six1mp = 6.0 * (1.0 - p);
    const S D = six1mp * (6.0 * r2) + (4.0 * p) * hb;
    const S E = six1mp * (-4.0 * r2) + p * hb;
    const S F = six1mp * r2;
    const S rh = 1.0 / hb;
    S a1 = D, a2 = E, b1 = D;
    S uprev(0.0), ucur = (w.y(3) - 2.0 * w.y(2) + w.y(1)) * rh, r2prev(0.0);
    for (int i = 2; i <= np - 2; i++) {
        const S Fi = (i <= np - 3) ? F : S(0.0);
        const S ratio1 = a2 / a1;
        b1 = b1 - ratio1 * a2;
        const S c2 = E - ratio1 * Fi;
        const S ratio2 = Fi / a1;
        const S c1 = D - ratio2 * Fi;
        w.s1(i) = ratio1;
        w.s2(i) = ratio2;
        w.u(i) = ucur / a1;
        const S qn = (w.y(i + 2) - 2.0 * w.y(i + 1) + w.y(i)) * rh;      // qty(i+1)
        const S unext = qn - ratio1 * ucur - r2prev * uprev;
        uprev = ucur;
        ucur = unext;
        r2prev = ratio2;
        a1 = b1;
        a2 = c2;
        b1 = c1;
    }
    w.u(np) = S(0.0);
    w.u(np - 1) = ucur / a1;
    for (int i = np - 2; i >= 2; i--) w.u(i) = w.u(i) - w.u(i + 1) * w.s1(i) - w.u(i + 2) * w.s2(i);
    w.u(1) = S(0.0);
}

// ppvalu (pppack.f90:4246-4362) of the fit, piece formed as smooth's
// epilogue forms a(:,1..4) (pppack.f90:5303-5316)
template <class S, int NPMAX>
__device__ __forceinline__ S a_ppvalu(const AFit<S, NPMAX>& w, int np, const S& z1, const S& hb, double p,
                                      double serr, const S& x, int jderiv) {
    const double t = floor(aval((x - z1) / hb));
    const int i = (t >= 0.0 && t < (double)(np - 1)) ? (int)t + 1 : ((t >= (double)(np - 1)) ? np - 1 : 1);
    const S rh = 1.0 / hb;
    const S xi = z1 + (double)(i - 1) * hb;
    const S um = (i >= 2) ? w.u(i - 1) : S(0.0);
    const S u0 = w.u(i), u1 = w.u(i + 1);
    const S u2 = (i + 2 <= np) ? w.u(i + 2) : S(0.0);
    const S raw0 = (i >= 2) ? (u0 - um) * rh : S(0.0);
    const S raw1 = (u1 - u0) * rh;
    const S raw2 = (i + 2 <= np) ? (u2 - u1) * rh : S(0.0);
    const double K1 = 6.0 * (1.0 - p) * serr * serr;
    const S a1i = w.y(i) - K1 * (raw1 - raw0);
    const S a1n = w.y(i + 1) - K1 * (raw2 - raw1);
    const S a3i = u0 * (6.0 * p);
    const S a3n = u1 * (6.0 * p);
    const S a4i = (a3n - a3i) * rh;
    const S a2i = (a1n - a1i) * rh - (a3i + a4i * (1.0 / 3.0) * hb) * 0.5 * hb;
    const S hx = x - xi;
    if (jderiv == 0) return ((a4i * (1.0 / 3.0) * hx + a3i) * 0.5 * hx + a2i) * hx + a1i;
    return (a4i * 0.5 * hx + a3i) * hx + a2i;
}

// VTurb (ver_turb_module.f90:31-329) with the diffusivity data scaled by
// kappa, at the recorded smoothing parameter p, in any arithmetic S.
template <class S, int NPMAX>
__device__ S a_vturb(const RpStepArgs& A, const AdjFrames& F, int gi, const AStage<S>& St, const S& Zpar,
                     const S& kappa, uint32_t pid, double p, const AFit<S, NPMAX>& w) {
    const RpGridDev& g = A.g[gi];
    const int sw = g.N + 1;
    const int np = (int)((double)sw * A.sub);
    const S h = -St.tdepth;
    const S* cw = St.rc.wet4 ? St.rc.cb : St.rc.ci;
    for (int k = 1; k <= sw; k++) {
        const double s = __ldg(g.sw + k - 1), cs = __ldg(g.csw + k - 1);
        w.zc(k) = a_polint(A.pi, a_zlev(g.vtransform, g.hc, s, cs, St.zb, h),
                           a_zlev(g.vtransform, g.hc, s, cs, St.zc, h), a_zlev(g.vtransform, g.hc, s, cs, St.zf, h));
        S K3[3];
#pragma unroll
        for (int t = 0; t < 3; t++) {
            const double* a = F.f[gi][4][t];
            K3[t] = cw[0] * __ldg(a + St.rc.o[0] * sw + k - 1) + cw[1] * __ldg(a + St.rc.o[1] * sw + k - 1) +
                    cw[2] * __ldg(a + St.rc.o[2] * sw + k - 1) + cw[3] * __ldg(a + St.rc.o[3] * sw + k - 1);
        }
        w.kh(k) = kappa * a_polint(A.pi, K3[0], K3[1], K3[2]);
    }
    // resample to np uniform points (ver_turb_module.f90:126-136)
    const S z1 = w.zc(1);
    const S hb = (w.zc(sw) - z1) / (double)(np - 1);
    w.y(1) = w.kh(1);
    w.y(np) = w.kh(sw);
    for (int i = 2; i <= np - 1; i++) w.y(i) = a_linint(w, sw, z1 + (double)(i - 1) * hb);
    a_chol1d(w, np, hb, p, A.serr);
    // random displacement sub-steps (ver_turb_module.f90:231-293)
    const double deltat = A.deltat;
    const S tdepth = St.tdepth, zeta = St.zeta;
    S ParZc = Zpar;
    for (int i = 1; i <= A.loop; i++) {
        S Kprimec(0.0);
        if (!(aval(ParZc) <= aval(tdepth) || aval(ParZc) >= aval(zeta)))
            Kprimec = a_ppvalu(w, np, z1, hb, p, A.serr, ParZc, 1);
        const S KprimeZc = Kprimec * deltat;
        const S Z3rdc = ParZc + 0.5 * KprimeZc;
        S KH3rdc;
        if (aval(Z3rdc) < aval(tdepth) || aval(Z3rdc) > aval(zeta)) {
            KH3rdc = S(A.aksback);
        } else {
            KH3rdc = a_ppvalu(w, np, z1, hb, p, A.serr, Z3rdc, 0);
            if (aval(KH3rdc) < A.aksback) KH3rdc = S(A.aksback);
        }
        const double DEV = rp_normal(A, pid, (uint32_t)(1 + i));
        ParZc = ParZc + (KprimeZc + DEV * asqrt(2.0 * KH3rdc * deltat));
        if (aval(ParZc) <= aval(tdepth)) ParZc = tdepth + aabs(ParZc - tdepth);
        if (aval(ParZc) >= aval(zeta)) ParZc = zeta - aabs(ParZc - zeta);
    }
    return ParZc - Zpar;
}

// ------------------------------------- VTurb in doubles, and its reverse
//
// The forward and replayed steps' VTurb (k_adj_vturb) and the reverse step's
// (k_adj_vturb_rev), each a kernel of its own.  The reverse differentiates the
// displacement by hand: through the sub-steps backwards, one more solve with
// the fit's own factor (its matrix is symmetric), the bands, the resampling
// and the column.  Carried through the fit as dual numbers of four directions
// instead, every array holds five doubles a point (31 KB a thread).
//
// Arrays of one fit (1-based element i), NPMAX + 1 doubles each.  REV: the
// reverse's arrays too.
template <int NPMAX, bool REV>
struct BFit {
    static constexpr int kArrays = REV ? 11 : 6;
    double* base;                  // kArrays (NPMAX + 1) doubles
    __device__ __forceinline__ double& at(int a, int i) const { return base[a * (NPMAX + 1) + i]; }
    __device__ __forceinline__ double& zc(int k) const { return at(0, k); }    // column z(k), K(k)
    __device__ __forceinline__ double& kh(int k) const { return at(1, k); }
    __device__ __forceinline__ double& y(int i) const { return at(2, i); }     // resampled data
    __device__ __forceinline__ double& u(int i) const { return at(3, i); }
    __device__ __forceinline__ double& s1(int i) const { return at(4, i); }    // the factor's ratios
    __device__ __forceinline__ double& s2(int i) const { return at(5, i); }
    __device__ __forceinline__ double& inv(int i) const { return at(6, i); }   // 1 / pivot
    __device__ __forceinline__ double& ub(int i) const { return at(7, i); }    // adjoints of u, then M^-1 of them
    __device__ __forceinline__ double& yb(int i) const { return at(8, i); }    // adjoints of y
    __device__ __forceinline__ double& zt(int i) const { return at(9, i); }    // sub-step i's start and deviate
    __device__ __forceinline__ double& dev(int i) const { return at(10, i); }
    // adjoints of the column, over the sub-steps once they have been used
    __device__ __forceinline__ double& zcb(int k) const { return zt(k); }
    __device__ __forceinline__ double& khb(int k) const { return dev(k); }
};

// What the passes of a fit share
struct BPar {
    int np, sw;
    double z1, hb, rh, serr, r2;
    // chol1d's bands on uniform breaks
    __device__ __forceinline__ void bands(double p, double& D, double& E, double& F) const {
        const double six1mp = 6.0 * (1.0 - p);
        D = six1mp * (6.0 * r2) + 4.0 * p * hb;
        E = six1mp * (-4.0 * r2) + p * hb;
        F = six1mp * r2;
    }
};

// the column's level k: z(k) of the three slots' zeta, K(k) before kappa
template <class S>
__device__ __forceinline__ void b_level(const RpStepArgs& A, const AdjFrames& F, int gi, const AStage<S>& St, int k,
                                        S& z, S& K) {
    const RpGridDev& g = A.g[gi];
    const int sw = g.N + 1;
    const S h = -St.tdepth;
    const S* cw = St.rc.wet4 ? St.rc.cb : St.rc.ci;
    const double s = __ldg(g.sw + k - 1), cs = __ldg(g.csw + k - 1);
    S K3[3];
#pragma unroll
    for (int t = 0; t < 3; t++) {
        const double* a = F.f[gi][4][t] + k - 1;
        K3[t] = cw[0] * __ldg(a + St.rc.o[0] * sw) + cw[1] * __ldg(a + St.rc.o[1] * sw) +
                cw[2] * __ldg(a + St.rc.o[2] * sw) + cw[3] * __ldg(a + St.rc.o[3] * sw);
    }
    K = a_polint(A.pi, K3[0], K3[1], K3[2]);
    if (g.vtransform == 2) {                     // the slots share the stretching
        const S Sk = (g.hc * s + h * cs) / (g.hc + h);
        z = a_polint(A.pi, St.zb + (St.zb + h) * Sk, St.zc + (St.zc + h) * Sk, St.zf + (St.zf + h) * Sk);
    } else {
        z = a_polint(A.pi, a_zlev(g.vtransform, g.hc, s, cs, St.zb, h), a_zlev(g.vtransform, g.hc, s, cs, St.zc, h),
                     a_zlev(g.vtransform, g.hc, s, cs, St.zf, h));
    }
}

// linint's bracket of x in the column: from j up on ascending levels and
// points, else by its bisection
template <class W>
__device__ __forceinline__ int b_bracket(const W& w, int sw, bool asc, int j, double x) {
    if (asc) {
        while (j < sw - 1 && !(w.zc(j + 1) > x)) j++;
        return j;
    }
    int lo = 1, hi = sw;
    while (hi - lo > 1) {
        const int k = (hi + lo) / 2;
        if (w.zc(k) > x) hi = k; else lo = k;
    }
    return lo;
}

// column and resampled data (ver_turb_module.f90:100-136)
template <class W>
__device__ __forceinline__ void b_column(const RpStepArgs& A, const AdjFrames& F, int gi, const AStage<double>& St,
                                         double kappa, const W& w, BPar& B, bool& asc) {
    const int sw = A.g[gi].N + 1, np = (int)((double)sw * A.sub);
    asc = true;
    double zp = 0.0;
#pragma unroll 2
    for (int k = 1; k <= sw; k++) {
        double z, K;
        b_level(A, F, gi, St, k, z, K);
        w.zc(k) = z;
        w.kh(k) = kappa * K;
        asc = asc && (k == 1 || z > zp);
        zp = z;
    }
    B.sw = sw;
    B.np = np;
    B.z1 = w.zc(1);
    B.hb = (zp - B.z1) / (double)(np - 1);
    asc = asc && B.hb > 0.0;
    B.rh = 1.0 / B.hb;
    B.serr = A.serr;
    const double r = A.serr / B.hb;
    B.r2 = r * r;
    w.y(1) = w.kh(1);
    w.y(np) = w.kh(sw);
    int j = 0;
    double m = 0.0, b = 0.0;
    for (int i = 2; i <= np - 1; i++) {
        const double x = B.z1 + (double)(i - 1) * B.hb;
        const int jn = b_bracket(w, sw, asc, max(j, 1), x);
        if (jn != j) {
            j = jn;
            m = (w.kh(j) - w.kh(j + 1)) / (w.zc(j) - w.zc(j + 1));
            b = w.kh(j) - m * w.zc(j);
        }
        w.y(i) = m * x + b;
    }
}

// The pass below with every quotient left to the IEEE operator, for fits whose
// operands leave the shared-reciprocal division's range (NaN frames, a zero or
// a tiny data weight).
template <bool REV, class W>
__device__ __noinline__ void b_solve_ieee(const W w, const BPar& B, double p) {
    const int np = B.np;
    double D, E, F;
    B.bands(p, D, E, F);
    double a1 = D, a2 = E, b1 = D;
    double uc = (w.y(3) - 2.0 * w.y(2) + w.y(1)) * B.rh, up = 0.0, r2p = 0.0;
    for (int i = 2; i <= np - 2; i++) {
        const double Fi = (i <= np - 3) ? F : 0.0;
        const double q1 = a2 / a1, q2 = Fi / a1;
        w.s1(i) = q1;
        w.s2(i) = q2;
        w.u(i) = uc / a1;
        if (REV) w.inv(i) = 1.0 / a1;
        a1 = b1 - q1 * a2;
        a2 = E - q1 * Fi;
        b1 = D - q2 * Fi;
        const double qn = (w.y(i + 2) - 2.0 * w.y(i + 1) + w.y(i)) * B.rh;
        const double un = qn - q1 * uc - r2p * up;
        up = uc;
        uc = un;
        r2p = q2;
    }
    if (REV) w.inv(np - 1) = 1.0 / a1;
    w.u(np) = 0.0;
    w.u(np - 1) = uc / a1;
    for (int i = np - 2; i >= 2; i--) w.u(i) = w.u(i) - w.u(i + 1) * w.s1(i) - w.u(i + 2) * w.s2(i);
    w.u(1) = 0.0;
}

// chol1d (pppack.f90:1428-1566) at p: leaves u(1..np), the ratios and, REV,
// the pivots' reciprocals.
//
// The operations are a_chol1d's, in its order, the three quotients of a row
// correctly rounded on one reciprocal of the pivot; as in rp_chol1d a row holds
// no branch and the pass is made again by the IEEE operator where an operand
// was out of that division's range.  A row is one chain (pivot, reciprocal,
// ratio, pivot).
template <bool REV, class W>
__device__ __forceinline__ void b_solve(const W& w, const BPar& B, double p) {
    const int np = B.np;
    double D, E, F;
    B.bands(p, D, E, F);
    double a1 = D, a2 = E, b1 = D;
    double y0 = w.y(2), yp = w.y(3);
    double uc = (yp - 2.0 * y0 + w.y(1)) * B.rh, up = 0.0, r2p = 0.0;
    uint32_t off = rp_exp_off_z(F), ones = 0;
    auto row = [&](int i, double yn, double Fi) {
        off = max(max(off, rp_exp_off(a1)), max(rp_exp_off_z(a2), rp_exp_off_z(uc)));
        ones = max(ones, rp_ones(a1));
        const RpRcp y = rp_rcp3(a1);
        const double q1 = rp_div_rcp(a2, a1, y), q2 = rp_div_rcp(Fi, a1, y);
        w.s1(i) = q1;
        w.s2(i) = q2;
        w.u(i) = rp_div_rcp(uc, a1, y);
        if (REV) w.inv(i) = y.y;
        a1 = b1 - q1 * a2;
        a2 = E - q1 * Fi;
        b1 = D - q2 * Fi;
        const double qn = (yn - 2.0 * yp + y0) * B.rh;
        y0 = yp;
        yp = yn;
        const double un = qn - q1 * uc - r2p * up;
        up = uc;
        uc = un;
        r2p = q2;
    };
    int i = 2;
#pragma unroll 1
    for (; i + 3 <= np - 3; i += 4) {            // the rows' data read together
        const double ya = w.y(i + 2), yb = w.y(i + 3), yc = w.y(i + 4), yd = w.y(i + 5);
        row(i, ya, F);
        row(i + 1, yb, F);
        row(i + 2, yc, F);
        row(i + 3, yd, F);
    }
#pragma unroll 1
    for (; i <= np - 2; i++) row(i, w.y(i + 2), i <= np - 3 ? F : 0.0);
    if (off >= kDivSpan || ones == 0xffffffffu) {
        b_solve_ieee<REV>(w, B, p);
        return;
    }
    if (REV) w.inv(np - 1) = rp_rcp(a1);
    double u2 = 0.0, u1 = uc / a1;               // u(i+2), u(i+1)
    w.u(np) = 0.0;
    w.u(np - 1) = u1;
    w.u(1) = 0.0;
    i = np - 2;
#pragma unroll 1
    for (; i - 3 >= 2; i -= 4) {                 // four rows' values read together
        double v[4], q1[4], q2[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = w.u(i - k);
            q1[k] = w.s1(i - k);
            q2[k] = w.s2(i - k);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const double ui = v[k] - u1 * q1[k] - u2 * q2[k];
            w.u(i - k) = ui;
            u2 = u1;
            u1 = ui;
        }
    }
    for (; i >= 2; i--) {
        const double ui = w.u(i) - u1 * w.s1(i) - u2 * w.s2(i);
        w.u(i) = ui;
        u2 = u1;
        u1 = ui;
    }
}

// sum qu^2 dy^2 of the pass just made, qu = Q u, in the reference's order.
// (From the forward sweep alone, as (phi + p phi') / 6 of phi(p) = b'M^-1 b,
// it needs no back substitution but cancels: with the data's weight at 1e-4
// and spacings of 0.02 to 50 m its error was up to 4e-4 where this sum's is
// 1e-9, with 1e-6 up to 2.5.)
template <class W>
__device__ __forceinline__ double b_sum(const W& w, const BPar& B) {
    const int np = B.np;
    const double dy2 = B.serr * B.serr;
    double prev = 0.0, sum = 0.0, ul = 0.0;      // raw(i), u(i)
    auto term = [&](double ui) {
        const double raw = (ui - ul) * B.rh;
        const double fin = raw - prev;
        sum = sum + fin * fin * dy2;
        prev = raw;
        ul = ui;
    };
    int i = 2;
#pragma unroll 1
    for (; i + 3 <= np; i += 4) {
        const double ua = w.u(i), ub = w.u(i + 1), uc = w.u(i + 2), ud = w.u(i + 3);
        term(ua);
        term(ub);
        term(uc);
        term(ud);
    }
    for (; i <= np; i++) term(w.u(i));
    return sum + prev * prev * dy2;
}

// utru (pppack.f90:5219-5223) of the pass just made
template <class W>
__device__ __forceinline__ double b_utru(const W& w, const BPar& B) {
    double utru = 0.0, ul = 0.0;
    for (int i = 2; i <= B.np; i++) {
        const double ui = w.u(i);
        utru = utru + B.hb * (ul * (ul + ui) + ui * ui);
        ul = ui;
    }
    return utru;
}

// The fit at p; find: at the p of smooth()'s secant search (pppack.f90:
// 5108-5317, reference cold start).  Returns p; the last pass made is p's.
template <class W>
__device__ __forceinline__ double b_fit(const W& w, const BPar& B, bool find, double p, double s, int max_iter,
                                        uint32_t& fl) {
    if (find) p = (s <= 0.0) ? 1.0 : 0.0;
    const double ooss = 1.0 / sqrt(s);
    double q = 0.0, prevq = 0.0, prevsf = 0.0;
#pragma unroll 1
    for (int it = 0;; it++) {
        b_solve<false>(w, B, p);
        if (!find || s <= 0.0) return p;
        const double sfq = 36.0 * b_sum(w, B) / ((1.0 + q) * (1.0 + q));
        const double oosf = 1.0 / sqrt(sfq);
        if (it == 0) {
            if (!(s < sfq)) return p;
            q = -(oosf - ooss) * sfq / (6.0 * b_utru(w, B) * oosf);
        } else {
            if (fabs(sfq - s) <= 0.01 * s) return p;
            if (it >= max_iter) {
                fl |= RP_FL_SPLINE;
                return p;
            }
            const double change = (q - prevq) / (oosf - prevsf) * (oosf - ooss);
            prevq = q;
            q = q - change;
        }
        prevsf = oosf;
        p = q / (1.0 + q);
    }
}

// ppvalu's piece at x (a_ppvalu's terms)
struct BPiece {
    int i;
    double hx, c1, c2, c3, c4, a1n, a3n, d0, d1, d2;   // d: u(i)-u(i-1), u(i+1)-u(i), u(i+2)-u(i+1)
};
__device__ __forceinline__ int b_piece_at(const BPar& B, double x) {
    const double t = floor((x - B.z1) * B.rh);
    return (t >= 0.0 && t < (double)(B.np - 1)) ? (int)t + 1 : ((t >= (double)(B.np - 1)) ? B.np - 1 : 1);
}
// c: a piece of the same fit formed before (c.i = 0: none), formed again where
// x lies in another one
template <class W>
__device__ __forceinline__ void b_piece(const W& w, const BPar& B, double p, double x, BPiece& c) {
    const int np = B.np, i = b_piece_at(B, x);
    if (i != c.i) {
        const double u0 = w.u(i), u1 = w.u(i + 1);
        c.i = i;
        c.d0 = (i >= 2) ? u0 - w.u(i - 1) : 0.0;
        c.d1 = u1 - u0;
        c.d2 = (i + 2 <= np) ? w.u(i + 2) - u1 : 0.0;
        const double K1 = 6.0 * (1.0 - p) * B.serr * B.serr;
        c.c1 = w.y(i) - K1 * ((c.d1 - c.d0) * B.rh);
        c.a1n = w.y(i + 1) - K1 * ((c.d2 - c.d1) * B.rh);
        c.c3 = u0 * (6.0 * p);
        c.a3n = u1 * (6.0 * p);
        c.c4 = (c.a3n - c.c3) * B.rh;
        c.c2 = (c.a1n - c.c1) * B.rh - (c.c3 + c.c4 * (1.0 / 3.0) * B.hb) * 0.5 * B.hb;
    }
    c.hx = x - (B.z1 + (double)(i - 1) * B.hb);
}
__device__ __forceinline__ double b_value(const BPiece& c) {
    return ((c.c4 * (1.0 / 3.0) * c.hx + c.c3) * 0.5 * c.hx + c.c2) * c.hx + c.c1;
}
__device__ __forceinline__ double b_slope(const BPiece& c) { return (c.c4 * 0.5 * c.hx + c.c3) * c.hx + c.c2; }

// adjoint g of the piece's value (DERIV: of its slope) to x (returned), u, y,
// the spacing and the first break
template <bool DERIV, class W>
__device__ __forceinline__ double b_piece_rev(const W& w, const BPar& B, double p, const BPiece& c, double g,
                                              double& hbb, double& z1b) {
    const int np = B.np, i = c.i;
    const double hx = c.hx, hb = B.hb, rh = B.rh;
    const double xb = g * (DERIV ? c.c4 * hx + c.c3 : b_slope(c));
    double a1b = DERIV ? 0.0 : g, a2b = DERIV ? g : g * hx;
    double a3b = DERIV ? g * hx : g * 0.5 * hx * hx;
    double a4b = DERIV ? g * 0.5 * hx * hx : g * (1.0 / 6.0) * hx * hx * hx;
    double rhb = a2b * (c.a1n - c.c1);
    double a1nb = a2b * rh;
    a1b -= a2b * rh;
    hbb -= a2b * (0.5 * c.c3 + c.c4 * hb * (1.0 / 3.0));
    a3b -= 0.5 * hb * a2b;
    a4b -= hb * hb * (1.0 / 6.0) * a2b;
    const double a3nb = a4b * rh;
    a3b -= a4b * rh;
    rhb += a4b * (c.a3n - c.c3);
    const double K1 = 6.0 * (1.0 - p) * B.serr * B.serr;
    const double r0b = K1 * a1b, r1b = K1 * (a1nb - a1b), r2b = -K1 * a1nb;       // of raw(i), raw(i+1), raw(i+2)
    rhb += r0b * c.d0 + r1b * c.d1 + r2b * c.d2;
    if (i >= 2) w.ub(i - 1) -= r0b * rh;
    w.ub(i) += ((i >= 2 ? r0b : 0.0) - r1b) * rh + 6.0 * p * a3b;
    w.ub(i + 1) += (r1b - (i + 2 <= np ? r2b : 0.0)) * rh + 6.0 * p * a3nb;
    if (i + 2 <= np) w.ub(i + 2) += r2b * rh;
    w.yb(i) += a1b;
    w.yb(i + 1) += a1nb;
    hbb -= rhb * rh * rh + xb * (double)(i - 1);
    z1b -= xb;
    return xb;
}

// One sub-step of the random walk (ver_turb_module.f90:231-293) from z
struct BSub {
    bool in1, in2, bot, top;       // slope taken; diffusivity taken from the fit; reflected
    double kz, z3, sd, z;          // slope times deltat, z3, sqrt(2 K deltat), the new position
    BPiece c1, c2;                 // the pieces at the start and at z3
};
template <class W>
__device__ __forceinline__ BSub b_sub(const W& w, const BPar& B, const RpStepArgs& A, double p, double tdepth,
                                      double zeta, double z, double dev, const BPiece& last) {
    BSub s;
    s.c1 = last;
    s.in1 = !(z <= tdepth || z >= zeta);
    double kp = 0.0;
    if (s.in1) {
        b_piece(w, B, p, z, s.c1);
        kp = b_slope(s.c1);
    }
    s.kz = kp * A.deltat;
    s.z3 = z + 0.5 * s.kz;
    s.in2 = !(s.z3 < tdepth || s.z3 > zeta);
    double K = A.aksback;
    s.c2 = s.c1;
    if (s.in2) {
        b_piece(w, B, p, s.z3, s.c2);
        K = b_value(s.c2);
        if (K < A.aksback) {
            K = A.aksback;
            s.in2 = false;
        }
    }
    s.sd = sqrt(2.0 * K * A.deltat);
    double n = z + (s.kz + dev * s.sd);
    s.bot = n <= tdepth && n - tdepth < 0.0;
    if (n <= tdepth) n = tdepth + fabs(n - tdepth);
    s.top = n >= zeta;
    if (s.top) n = zeta - fabs(n - zeta);
    s.z = n;
    return s;
}

// RK stage 1's 2-D quantities and the z clamp find_currents applies there
// (advection_module.f90:171-183)
template <class S>
__device__ __forceinline__ void b_stage(const RpStepArgs& A, const AdjFrames& F, int gi, const S& X, const S& Y,
                                        AStage<S>& St, uint32_t& fl) {
    a_rho_cell(A.g[gi], X, Y, St.rc, fl);
    a_stage_2d(A, F, gi, A.g[gi], St);
}

// VTurb's displacement; find: p is searched and returned, else given
template <class W>
__device__ __forceinline__ double b_vturb(const RpStepArgs& A, const AdjFrames& F, int gi, double X, double Y,
                                          double Z, double kappa, uint32_t pid, bool find, double& p, uint32_t& fl,
                                          const W& w) {
    AStage<double> St;
    b_stage(A, F, gi, X, Y, St, fl);
    if (A.scheme == 1) {
        if (Z < St.tdepth) Z = St.tdepth + RP_F_0P001;
        if (Z > St.zeta) Z = St.zeta - RP_F_0P001;
    }
    BPar B;
    bool asc;
    b_column(A, F, gi, St, kappa, w, B, asc);
    p = b_fit(w, B, find, p, A.smth, A.spline_max_iter, fl);
    double z = Z, dev, dev_next = 0.0;
    BPiece c;
    c.i = 0;
#pragma unroll 1
    for (int i = 1; i <= A.loop; i++) {
        if (i & 1) rp_normal2(A, pid, (uint32_t)(1 + i), i < A.loop, dev, dev_next);
        else dev = dev_next;
        const BSub s = b_sub(w, B, A, p, St.tdepth, St.zeta, z, dev, c);
        z = s.z;
        c = s.c2;
    }
    return z - Z;
}

// VTurb's displacement t[0] and its derivatives t[1..4] in the start's x, y, z
// and in kappa, at the recorded p; A.loop <= NPMAX
template <class W>
__device__ __forceinline__ void b_vturb_rev(const RpStepArgs& A, const AdjFrames& F, int gi, double X, double Y,
                                            double Z, double kappa, uint32_t pid, double p, uint32_t& fl, const W& w,
                                            double t[5]) {
    BPar B;
    bool asc;
    int clamp = 0;                 // stage 1's z: 1 put on the bottom, 2 under the surface
    double hbb = 0.0, z1b = 0.0, tdb = 0.0, zeb = 0.0;   // adjoints of hb, z1, tdepth, zeta
    double zb = 1.0;                                     // of the position
    {
        AStage<double> St;
        b_stage(A, F, gi, X, Y, St, fl);
        if (A.scheme == 1) {
            if (Z < St.tdepth) {
                Z = St.tdepth + RP_F_0P001;
                clamp = 1;
            }
            if (Z > St.zeta) {
                Z = St.zeta - RP_F_0P001;
                clamp = 2;
            }
        }
        b_column(A, F, gi, St, kappa, w, B, asc);
        b_solve<true>(w, B, p);
        for (int i = 1; i <= B.np; i++) {
            w.ub(i) = 0.0;
            w.yb(i) = 0.0;
        }
        double z = Z, dev = 0.0, dev_next = 0.0;
        BPiece c;
        c.i = 0;
#pragma unroll 1
        for (int i = 1; i <= A.loop; i++) {
            if (i & 1) rp_normal2(A, pid, (uint32_t)(1 + i), i < A.loop, dev, dev_next);
            else dev = dev_next;
            w.zt(i) = z;
            w.dev(i) = dev;
            const BSub s = b_sub(w, B, A, p, St.tdepth, St.zeta, z, dev, c);
            z = s.z;
            c = s.c2;
        }
        t[0] = z - Z;
#pragma unroll 1
        for (int i = A.loop; i >= 1; i--) {
            const double zi = w.zt(i), d = w.dev(i);
            const BSub s = b_sub(w, B, A, p, St.tdepth, St.zeta, zi, d, c);
            c = s.c1;
            if (s.top) {
                zeb += 2.0 * zb;
                zb = -zb;
            }
            if (s.bot) {
                tdb += 2.0 * zb;
                zb = -zb;
            }
            double kzb = zb;
            if (s.in2) {
                const double Kb = zb * d * ((s.sd > 0.0) ? 0.5 / s.sd : 0.0) * 2.0 * A.deltat;
                const double z3b = b_piece_rev<false>(w, B, p, s.c2, Kb, hbb, z1b);
                zb += z3b;
                kzb += 0.5 * z3b;
            }
            if (s.in1) zb += b_piece_rev<true>(w, B, p, s.c1, kzb * A.deltat, hbb, z1b);
        }
    }
    const int np = B.np, sw = B.sw;
    // lambda = M^-1 ub by the fit's factor; u(1) = u(np) = 0.  Upwards first,
    // four rows' values read together
    {
        double w1 = 0.0, w2 = 0.0, q1 = 0.0, q2 = 0.0, q2p = 0.0;   // w(i-1), w(i-2), ratio1(i-1), ratio2(i-1), (i-2)
        int i = 2;
#pragma unroll 1
        for (; i + 3 <= np - 2; i += 4) {
            double v[4], r1[4], r2[4], iv[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v[k] = w.ub(i + k);
                r1[k] = w.s1(i + k);
                r2[k] = w.s2(i + k);
                iv[k] = w.inv(i + k);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double wi = fma(-q2p, w2, fma(-q1, w1, v[k]));
                w.ub(i + k) = wi * iv[k];
                w2 = w1;
                w1 = wi;
                q2p = q2;
                q1 = r1[k];
                q2 = r2[k];
            }
        }
        for (; i <= np - 1; i++) {
            const double wi = fma(-q2p, w2, fma(-q1, w1, w.ub(i)));
            w.ub(i) = wi * w.inv(i);
            w2 = w1;
            w1 = wi;
            q2p = q2;
            if (i <= np - 2) {
                q1 = w.s1(i);
                q2 = w.s2(i);
            }
        }
    }
    // Downwards, all that follows from lambda in one sweep: the bands and the
    // right-hand side b(i) = (y(i+1) - 2 y(i) + y(i-1)) / hb in hb, the data's
    // adjoints, and the resampling y(i) = K(j) + m (x - z(j)), x = z1 + (i-1) hb,
    // whose bracket's sums are put down where it changes
    for (int k = 1; k <= sw; k++) {
        w.zcb(k) = 0.0;
        w.khb(k) = 0.0;
    }
    {
        double sD = 0.0, sE = 0.0, sF = 0.0, sB = 0.0;
        double l1 = 0.0, l2 = 0.0, u1 = 0.0, u2 = 0.0;      // lambda and u of rows i+1, i+2
        double y1 = w.y(np), y0 = w.y(np - 1);              // y(i+1), y(i)
        int j = 0;
        double m = 0.0, rz = 0.0, z0 = 0.0, gK = 0.0, gm = 0.0;   // bracket; sums of g and of m's adjoint
        auto put = [&]() {
            if (j == 0) return;
            const double mb = gm * rz;
            w.khb(j) += gK + mb;
            w.khb(j + 1) -= mb;
            w.zcb(j) -= gK * m + mb * m;
            w.zcb(j + 1) += mb * m;
        };
        // adjoint g of y(i): the direct one and lambda's
        auto data = [&](int i, double g) {
            const double x = B.z1 + (double)(i - 1) * B.hb;
            const bool in = asc ? (j != 0 && (j == 1 || w.zc(j) <= x)) : false;
            if (!in) {
                put();
                if (asc) {
                    j = (j == 0) ? sw - 1 : j;
                    while (j > 1 && w.zc(j) > x) j--;
                } else {
                    j = b_bracket(w, sw, false, 1, x);
                }
                z0 = w.zc(j);
                rz = 1.0 / (z0 - w.zc(j + 1));
                m = (w.kh(j) - w.kh(j + 1)) * rz;
                gK = gm = 0.0;
            }
            gK += g;
            gm = fma(g, x - z0, gm);
            const double xb = g * m;
            z1b += xb;
            hbb = fma((double)(i - 1), xb, hbb);
        };
        // row i: lambda(i) from its forward value; y(i+1)'s adjoint is then complete
        auto row = [&](int i, double v, double q1, double q2, double ui, double ym, double yb1) {
            const double l = fma(-l1, q1, fma(-l2, q2, v));
            sD = fma(l, ui, sD);
            sE = fma(l, u1, fma(l1, ui, sE));
            sF = fma(l, u2, fma(l2, ui, sF));
            sB = fma(l, (y1 - 2.0 * y0 + ym) * B.rh, sB);
            const double g = fma((l - 2.0 * l1) + l2, B.rh, yb1);
            if (i + 1 < np) data(i + 1, g);
            else w.khb(sw) += g;
            l2 = l1;
            l1 = l;
            u2 = u1;
            u1 = ui;
            y1 = y0;
            y0 = ym;
        };
        row(np - 1, w.ub(np - 1), 0.0, 0.0, w.u(np - 1), w.y(np - 2), w.yb(np));
        int i = np - 2;
#pragma unroll 1
        for (; i - 3 >= 2; i -= 4) {
            double v[4], q1[4], q2[4], ui[4], ym[4], yb[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v[k] = w.ub(i - k);
                q1[k] = w.s1(i - k);
                q2[k] = w.s2(i - k);
                ui[k] = w.u(i - k);
                ym[k] = w.y(i - k - 1);
                yb[k] = w.yb(i - k + 1);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) row(i - k, v[k], q1[k], q2[k], ui[k], ym[k], yb[k]);
        }
#pragma unroll 1
        for (; i >= 2; i--) row(i, w.ub(i), w.s1(i), w.s2(i), w.u(i), w.y(i - 1), w.yb(i + 1));
        data(2, fma(l2 - 2.0 * l1, B.rh, w.yb(2)));         // lambda(1) = 0; l1 = lambda(2), l2 = lambda(3)
        put();
        w.khb(1) += fma(l1, B.rh, w.yb(1));
        const double six1mp = 6.0 * (1.0 - p), dr2 = -2.0 * B.r2 * B.rh;
        const double Dh = six1mp * 6.0 * dr2 + 4.0 * p, Eh = six1mp * -4.0 * dr2 + p, Fh = six1mp * dr2;
        hbb -= Dh * sD + Eh * sE + Fh * sF + sB * B.rh;
    }
    const double hr = hbb / (double)(np - 1);
    w.zcb(sw) += hr;
    w.zcb(1) += z1b - hr;
    // the column and the 2-D quantities in x and y, and K in kappa
    Dual<2> DX(X), DY(Y);
    DX.d[0] = 1.0;
    DY.d[1] = 1.0;
    AStage<Dual<2>> St;
    b_stage(A, F, gi, DX, DY, St, fl);
    // Z of the clamp: t = z - Z
    const double Zb = zb - 1.0;
    if (clamp == 1) tdb += Zb;
    if (clamp == 2) zeb += Zb;
    double gx = tdb * St.tdepth.d[0] + zeb * St.zeta.d[0], gy = tdb * St.tdepth.d[1] + zeb * St.zeta.d[1], gk = 0.0;
#pragma unroll 1
    for (int k = 1; k <= sw; k++) {
        Dual<2> z, K;
        b_level(A, F, gi, St, k, z, K);
        const double zk = w.zcb(k), kk = w.khb(k);
        gx += zk * z.d[0] + kk * (kappa * K.d[0]);
        gy += zk * z.d[1] + kk * (kappa * K.d[1]);
        gk += kk * K.v;
    }
    t[1] = gx;
    t[2] = gy;
    t[3] = (clamp == 0) ? Zb : 0.0;
    t[4] = gk;
}

// ----------------------------------------------------------- one step

// The state a step carries besides (x, y, z).
struct AdjAux {
    double age, status;
    int gid;
    int8_t isin;
};

// Skip tests of update_particles (ROMSPath.f90:672-690)
__device__ __forceinline__ bool a_active(const RpStepArgs& A, double dob, double status, int8_t isin) {
    return !(A.ix[2] <= dob || status == 9.0 || (A.oob && !isin));
}

// One particle-step of the model (ROMSPath.f90:672-892) from (X, Y, Z) with
// auxiliary state `a`; updates X, Y, Z, a.  vturb(St, have_s1, Zpar) is VTurb's
// displacement (S1: RK stage 1's quantities where have_s1), called with VTurb
// on.  Returns the sign the new Z carries VTurb's displacement with (0: not at
// all).
template <class S, class VT>
__device__ __forceinline__ int a_step(const RpStepArgs& A, const AdjFrames& F, double dob, uint32_t pid, S& X, S& Y,
                                      S& Z, AdjAux& a, uint32_t& fl, VT&& vturb) {
    if (!a_active(A, dob, a.status, a.isin)) return 0;
    a.age = a.age + (double)(float)A.idt;
    int gid = a.gid;
    const int gi = gid - 1;
    const RpGridDev& g = A.g[gi];
    const S Xpar = X, Ypar = Y, z0 = Z;
    S Zpar = Z;
    S pm, pn;
    {
        ARho<S> c;
        a_rho_cell(g, Xpar, Ypar, c, fl);
        pm = a_dot4(g.pm, c.o, c.cb);
        pn = a_dot4(g.pn, c.o, c.cb);
    }
    S AdvectX(0.0), AdvectY(0.0), AdvectZ(0.0);
    AStage<S> S1;
    bool have_s1 = false;
    if (A.scheme == 1) {                                  // RKAdvect
        const double didt = (double)A.idt;
        S U, V, Wv, kx(0.0), ky(0.0), kz(0.0), ax(0.0), ay(0.0), az(0.0);
        for (int st = 0; st < 4; st++) {
            S xs = Xpar, ys = Ypar, zs = Zpar;
            if (st > 0) {
                xs = Xpar + kx * didt / 2.0;
                ys = Ypar + ky * didt / 2.0;
                zs = Zpar + kz * didt / 2.0;
            }
            AStage<S> Sx;
            a_find_currents(A, F, gi, xs, ys, zs, U, V, Wv, Sx, fl);
            if (st == 0) {
                Zpar = zs;                                // INOUT z of stage 1
                S1 = Sx;
                have_s1 = true;
            }
            kx = U * pm;
            ky = V * pn;
            kz = Wv;
            const double wgt = (st == 0 || st == 3) ? 1.0 : 2.0;
            ax = ax + wgt * kx;
            ay = ay + wgt * ky;
            az = az + wgt * kz;
        }
        AdvectX = didt * (ax / 6.0);
        AdvectY = didt * (ay / 6.0);
        AdvectZ = didt * (az / 6.0);
    }
    S TurbHx(0.0), TurbHy(0.0);
    if (A.hturb_on) {                                     // HTurb
        const double sc = sqrt(2.0 * A.khturb[gi] * (double)A.idt);
        TurbHx = rp_normal(A, pid, 0u) * sc * pm;
        TurbHy = rp_normal(A, pid, 1u) * sc * pn;
    }
    S TurbV(0.0);
    if (A.vturb_on) TurbV = vturb(S1, have_s1, Zpar);
    // new position and hand-off (ROMSPath.f90:821-836)
    const S newX = X + AdvectX + TurbHx;
    const S newY = Y + AdvectY + TurbHy;
    S tX = newX, tY = newY;
    bool ingrid = false, obound = false;
    for (int i = 1; i <= A.ngrid; i++) {
        tX = g.scl[i - 1][0] * newX + g.off[i - 1][0];
        tY = g.scl[i - 1][1] * newY + g.off[i - 1][1];
        rp_bounds(A.g[i - 1], aval(tX), aval(tY), ingrid, obound);
        if (ingrid) { gid = i; break; }
    }
    const RpGridDev& gn = A.g[gid - 1];
    ARho<S> rn;
    a_rho_cell(gn, tX, tY, rn, fl);
    const S tdepth = -a_dot4(gn.h, rn.o, rn.cb);
    const S P_zeta = a_polint(A.pi, a_dot4(F.f[gid - 1][0][0], rn.o, rn.ci), a_dot4(F.f[gid - 1][0][1], rn.o, rn.ci),
                              a_dot4(F.f[gid - 1][0][2], rn.o, rn.ci));
    bool hbot = false, htop = false;
    S newZ;
    if (A.nsb == 0) {                                     // ROMSPath.f90:852-872
        newZ = z0 + AdvectZ + TurbV;
        if (aval(newZ) < aval(tdepth)) { newZ = tdepth + aabs(newZ - tdepth); hbot = true; }
        if (aval(newZ) > aval(P_zeta)) { newZ = P_zeta - aabs(newZ - P_zeta); htop = true; }
    } else if (A.nsb == 1) {
        newZ = P_zeta - A.vertdist;
    } else {
        newZ = tdepth + A.vertdist;
    }
    int vsign = 0;
    if (ingrid) {                                         // 874-892
        a.isin = 1;
        X = tX;
        Y = tY;
        Z = newZ;
        if (A.nsb == 0) vsign = (hbot != htop) ? -1 : 1;
        double st = 1.0;
        if (htop) st = RP_F_1P1;
        if (hbot) st = RP_F_1P2;
        a.status = st;
        a.gid = gid;
    } else if (obound) {
        a.isin = 0;
        a.gid = A.ngrid;
        a.status = -8.0;
    } else {
        a.isin = 1;
        a.status = -9.0;
    }
    return vsign;
}
