"""The division helpers of rp_device.cuh against IEEE division, bit for bit:
random operands over the range they claim, both sides of its ends 2^-498 and
2^498, powers of two, significands of all ones, zeros, subnormals, infinities and
NaN (the helpers that test their operands), exact quotients and halfway-close
ones.  Every helper is correctly rounded in its range, so the tolerance is 0."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "romspath_b200", "csrc")
P = C.POINTER(C.c_double)
OUT = ["rcp", "rcp_in", "rcp3", "quot", "div_by", "div_rcp", "div_fast"]


def _operands(rng, n):
    """(a, b): the first half spread over the exponents 2^-498 .. 2^498, the rest mixed with the special values."""
    def spread():
        return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-498, 498, n)) * rng.choice([-1.0, 1.0], n)

    a, b = spread(), spread()
    k = n // 16
    b[:k] = np.ldexp(np.nextafter(2.0, 0.0), rng.integers(-400, 400, k))             # all ones
    b[k:2 * k] = np.ldexp(1.0, rng.integers(-498, 498, k))
    b[2 * k:3 * k] = np.ldexp(1.0 + rng.integers(1, 64, k) * 2.0 ** -52, rng.integers(-400, 400, k))
    b[3 * k:4 * k] = np.ldexp(2.0 - rng.integers(1, 64, k) * 2.0 ** -52, rng.integers(-400, 400, k))
    m = rng.integers(-400, 400, k)
    a[4 * k:5 * k] = np.ldexp(rng.integers(1, 1 << 26, k) * 1.0, m) * rng.integers(1, 1 << 26, k)
    b[4 * k:5 * k] = np.ldexp(rng.integers(1, 1 << 26, k) * 1.0, m)
    a[5 * k:6 * k] = b[5 * k:6 * k]
    edge = np.concatenate([np.ldexp([1.0, np.nextafter(1.0, 0), np.nextafter(1.0, 2), 1.5, np.nextafter(2.0, 0)], e)
                           for e in (-499, -498, -497, 497, 498, 499)])
    odd = np.concatenate([edge, [0.0, 5e-324, 2.2e-308, 2.3e-308, 1e-200, 1e200, 1.7e308, np.inf, np.nan]])
    odd = np.concatenate([odd, -odd])
    h = n // 2
    a[h:h + n // 8] = rng.choice(odd, n // 8)
    b[h + n // 16:h + 3 * n // 16] = rng.choice(odd, n // 8)
    return a, b


def _in_range(b):
    """The helpers' range: a biased exponent within 2^-498 <= |b| < 2^498"""
    with np.errstate(invalid="ignore"):
        return (np.abs(b) >= np.ldexp(1.0, -498)) & (np.abs(b) < np.ldexp(1.0, 498))


def _all_ones(b):
    return (b.view(np.uint64) & np.uint64((1 << 52) - 1)) == np.uint64((1 << 52) - 1)


def _same(x, y):
    return (x.view(np.uint64) == y.view(np.uint64)) | (np.isnan(x) & np.isnan(y))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quot") / "quot.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, os.path.join(HERE, "gpu_quot_selftest.cu"), "-o", so],
                   check=True)
    L = C.CDLL(so)
    L.quot_selftest.argtypes = [C.c_int64, P, P, P]
    L.polint_selftest.argtypes = [C.c_int64, P, C.c_double, C.c_int, P, P, P]
    return L


@pytest.fixture(scope="module")
def run(lib):
    n = 1 << 22
    a, b = _operands(np.random.default_rng(17), n)
    out = np.empty((len(OUT), n))
    assert lib.quot_selftest(n, *[v.ctypes.data_as(P) for v in (a, b, out)]) == 0
    return a, b, dict(zip(OUT, out))


def test_reciprocals(run):
    a, b, out = run
    with np.errstate(all="ignore"):
        want = 1.0 / b
    assert _same(out["rcp"], want).all()
    ok = _in_range(b) & ~_all_ones(b)
    assert ok.sum() > b.size // 2
    for k in ("rcp_in", "rcp3"):
        assert _same(out[k][ok], want[ok]).all(), k


def test_quotients(run):
    a, b, out = run
    with np.errstate(all="ignore"):
        want = a / b
    assert _same(out["quot"], want).all()
    assert _same(out["div_by"], want).all()
    ok = _in_range(a) & _in_range(b) & ~_all_ones(b)
    assert ok.sum() > b.size // 2
    for k in ("div_rcp", "div_fast"):
        assert _same(out[k][ok], want[ok]).all(), k
    zero = (a == 0.0) & _in_range(b) & ~_all_ones(b)       # a zero of either sign
    assert zero.any()
    for k in ("div_rcp", "div_fast"):
        assert (out[k][zero] == 0.0).all(), k


# nodes and place as a run meets them (frames an hour apart, the nearest node each
# in turn), and frame times whose differences leave the helpers' range
@pytest.mark.parametrize("xa,x,ns", [
    ((0.0, 3600.0, 7200.0), 3900.0, 1), ((0.0, 3600.0, 7200.0), 300.0, 0), ((0.0, 3600.0, 7200.0), 6900.0, 2),
    ((3600.0, 7200.0, 10800.0), 7200.0, 1), ((0.0, 1e-160, 3e-160), 1.1e-160, 1), ((0.0, 3600.0, 7200.0), 3600.0, 1)])
def test_polintd_pair(lib, xa, x, ns):
    rng = np.random.default_rng(5)
    n = 1 << 18
    u = rng.uniform(-1.0, 1.0, (3, n)) * 10.0 ** rng.uniform(-8, 3, n)
    v = rng.uniform(-1.0, 1.0, (3, n)) * 10.0 ** rng.uniform(-8, 3, n)
    k = n // 8
    u[:, :k] = u[0, :k]                                     # no change in time
    v[1, k:2 * k] = v[0, k:2 * k]
    u[:, 2 * k:3 * k] = 0.0
    v[:, 3 * k:4 * k] *= 1e-200                             # one of the pair out of range
    u[2, 4 * k:4 * k + 9] = np.nan
    v[1, 4 * k + 9:4 * k + 18] = np.inf
    u[:, 5 * k:5 * k + 9] = 5e-324
    r = np.empty((4, n))
    t = np.array(xa)
    args = [np.ascontiguousarray(q) for q in (u, v)]
    assert lib.polint_selftest(n, t.ctypes.data_as(P), x, ns, *[q.ctypes.data_as(P) for q in args],
                               r.ctypes.data_as(P)) == 0
    for got, want in ((r[0], r[2]), (r[1], r[3])):
        assert np.array_equal(got, want, equal_nan=True)
