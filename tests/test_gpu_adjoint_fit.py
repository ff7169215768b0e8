"""The adjoint pair's fit and forward model against something independent.

* A pass of the fit (b_solve, b_sum, b_utru: the sum of squares and utru that
  the search for the smoothing parameter compares) against its restatement in
  numpy, whose FP64 operations in the same order give the same bits: over point
  counts around the row groups, spacings, data weights and p up to 1 and down
  to 0, and operands out of the shared-reciprocal division's range.
* rp_forward against the CPU oracle on the same noise, over smoothing
  parameters that take p from 1 to 0 and data weights.  The models differ in
  rounding (uniform breaks, polintd's divisions): 1e-9 relative in the sum of
  squares at worst (p near 0, 124 points), so about 1e-9 in the smoothing
  parameter and in the fitted diffusivity, below 1e-9 m a sub-step of up to a
  metre; 140 sub-steps that all add up and grow tenfold: 1e-6 m in z, and with
  shears below 0.1 / s on cells of 1000 m 1e-7 cells in x and y.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "romspath_b200", "csrc")
P = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fit") / "adjfit.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, os.path.join(HERE, "gpu_adj_fit_selftest.cu"), "-o", so],
                   check=True)
    L = C.CDLL(so)
    L.adj_fit.argtypes = [C.c_int, C.c_int, C.c_double] + [P] * 5
    return L


def _pass(y, h, p, serr):
    """chol1d on uniform breaks, its sum of squares and utru: y[i - 1] the data of point i of every column"""
    n = y.shape[0]
    rh = 1.0 / h
    r = serr / h
    r2 = r * r
    six = 6.0 * (1.0 - p)
    D, E, F = six * (6.0 * r2) + 4.0 * p * h, six * (-4.0 * r2) + p * h, six * r2
    a1, a2, b1 = D, E, D
    uc, up, r2p = (y[2] - 2.0 * y[1] + y[0]) * rh, np.zeros_like(h), np.zeros_like(h)
    u, s1, s2 = np.zeros((n + 1,) + h.shape), {}, {}
    for i in range(2, n - 1):
        Fi = F if i <= n - 3 else np.zeros_like(h)
        q1, q2 = a2 / a1, Fi / a1
        s1[i], s2[i], u[i] = q1, q2, uc / a1
        a1, a2, b1 = b1 - q1 * a2, E - q1 * Fi, D - q2 * Fi
        qn = (y[i + 1] - 2.0 * y[i] + y[i - 1]) * rh
        up, uc, r2p = uc, qn - q1 * uc - r2p * up, q2
    u[n - 1] = uc / a1
    for i in range(n - 2, 1, -1):
        u[i] = u[i] - u[i + 1] * s1[i] - u[i + 2] * s2[i]
    total, utru, prev = np.zeros_like(h), np.zeros_like(h), np.zeros_like(h)
    for i in range(2, n + 1):
        raw = (u[i] - u[i - 1]) * rh
        fin = raw - prev
        total = total + fin * fin * (serr * serr)
        prev = raw
        utru = utru + h * (u[i - 1] * (u[i - 1] + u[i]) + u[i] * u[i])
    return total + prev * prev * (serr * serr), utru


@pytest.mark.parametrize("serr", [1e-4, 1e-6, 1e-2, 0.0, 1e-160, 1e150])
@pytest.mark.parametrize("npt", [4, 5, 6, 7, 8, 9, 10, 28, 84, 124, 143, 144])
def test_pass_matches_its_restatement(lib, npt, serr):
    rng = np.random.default_rng(npt)
    m = 1000
    h = np.exp(rng.uniform(np.log(0.02), np.log(50.0), m))
    xi = np.linspace(0.0, 1.0, npt)[:, None]
    y = 10.0 ** rng.uniform(-4, 0, m) * 4 * xi * (1 - xi) * (1 + 0.2 * np.sin(xi * rng.uniform(3, 40, m))
                                                               + 0.02 * rng.normal(size=(npt, m)))
    y[:, :5] = 0.0
    y[npt // 2, 5:10] = np.nan
    y[:, 10:15] *= 1e-300
    q = 10.0 ** rng.uniform(-12, 8, m)
    q[::7] = 0.0
    p = q / (1.0 + q)
    p[::11] = 1.0
    got = [np.empty(m), np.empty(m)]
    y = np.ascontiguousarray(y)
    assert lib.adj_fit(m, npt, serr, *[a.ctypes.data_as(P) for a in (y, h, p, *got)]) == 0
    with np.errstate(all="ignore"):
        want = _pass(y, h, p, serr)
    for g, w in zip(got, want):
        assert np.array_equal(g, w, equal_nan=True)


@pytest.mark.parametrize("spec,param", [
    ({}, {}), ({}, {"sub": 1.1}), ({"N": 20}, {}), ({"N": 30}, {}), ({"N": 35}, {}), ({}, {"smth": 0.0}),
    ({}, {"smth": 1e-24, "serr": 1e-6}), ({}, {"smth": 1e-14, "serr": 1e-6}), ({}, {"smth": 1e-6}),
    ({}, {"smth": 10.0}), ({}, {"smth": 1e9}), ({}, {"serr": 1e-2}), ({"land": "islands"}, {"serr": 1.0}),
    ({"vtransform": 1}, {})])
def test_forward_matches_oracle(spec, param):
    from romspath_b200 import Tracker, schedule
    from romspath_b200.adjoint import Adjoint, step_table
    n, nsteps = 128, 14
    case = harness.make_case("tiny", n, seed=11, spec_over=spec, param_over=param, s_range=(-1.0, 0.0))
    want, _ = harness.run_oracle(case, nsteps)
    T = Tracker(case.specs, case.grids, case.params, numpar=n, field_dtype="f64", seed=7)
    for (k, slot) in schedule.initial_loads():
        T.upload_frame(1, slot, case.frame(k))
    T.locate(case.release, t_b=1)
    steps = step_table(2.0, int(case.params["dt"]), int(case.params["idt"]))[0][:nsteps]
    adj = Adjoint(T)
    adj.load_frames(max(max(s.frame_b, s.frame_c, s.frame_f) for s in steps), lambda ng, k: case.frame(k, ng))
    adj.forward(steps, checkpoint_every=4)
    got = T.get_particles()
    T.close()
    assert np.array_equal(got["status"], want["status"])
    for c, tol in (("x", 1e-7), ("y", 1e-7), ("z", 1e-6)):
        assert np.abs(got[c] - want[c]).max() <= tol, c


# kernels of the adjoint pair by what rp_kernel_launches tells: VTurb is a kernel of
# its own but in the tangent and where the sub-steps are more than its reverse keeps
@pytest.mark.parametrize("param,fwd,rev", [({}, 2, 2), ({"vturb_on": 0}, 1, 1), ({"deltat": 3.0}, 2, 1)])
def test_launches_are_counted(param, fwd, rev):
    from romspath_b200 import Tracker, schedule
    from romspath_b200.adjoint import Adjoint, step_table
    n = 128
    case = harness.make_case("tiny", n, seed=11, param_over=param)
    T = Tracker(case.specs, case.grids, case.params, numpar=n, field_dtype="f64", seed=7)
    for (k, slot) in schedule.initial_loads():
        T.upload_frame(1, slot, case.frame(k))
    T.locate(case.release, t_b=1)
    steps = step_table(2.0, int(case.params["dt"]), int(case.params["idt"]))[0][:6]
    adj = Adjoint(T)
    adj.load_frames(max(max(s.frame_b, s.frame_c, s.frame_f) for s in steps), lambda ng, k: case.frame(k, ng))
    z = np.zeros(n)

    def launches(f):
        l0 = T.kernel_launches()
        f()
        return T.kernel_launches() - l0

    assert launches(lambda: adj.forward(steps, checkpoint_every=3)) == 6 * fwd
    assert launches(lambda: adj.backward(z, z, z)) == 4 * fwd + 6 * rev
    assert launches(adj.replay) == 6 * fwd
    T.close()
