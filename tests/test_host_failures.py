"""Failures of the CUDA runtime on the host side of the C ABI (rp_api.cu), made by
a fake runtime whose memory is the host's and whose kernels do nothing
(fake_cudart.cpp, fake_launch.cu): no GPU takes part.  Allocations and launches fail where a test says;
what the launchers are then given, what a call returns and what it holds is
checked."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import harness
from romspath_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = str(tmp_path_factory.mktemp("fake"))
    csrc = os.path.join(ROOT, "romspath_b200", "csrc")
    objs = []
    for src in (os.path.join(csrc, "rp_api.cu"), os.path.join(HERE, "fake_launch.cu"),
                os.path.join(HERE, "fake_cudart.cpp")):
        objs.append(os.path.join(d, os.path.basename(src) + ".o"))
        subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
                        "-I", os.path.join(ROOT, "include"), "-I", csrc, "-c", src, "-o", objs[-1]], check=True)
    so = os.path.join(d, "libfake.so")
    # -Bsymbolic: a runtime already in the process must not take the fake's place
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, *objs], check=True)
    L = C.CDLL(so)
    _lib._declare(L)
    for f in ("bytes", "adj", "ordered", "sorts", "null_bufs"):
        getattr(L, "fake_" + f).restype = C.c_long
    L.fake_fail_malloc.argtypes = [C.c_long, C.c_int]
    L.fake_fail_adj.argtypes = [C.c_long]
    return L


@pytest.fixture
def tracker(fake, monkeypatch):
    """A Tracker on the fake runtime, n particles of the tiny grid set."""
    from romspath_b200 import Tracker
    monkeypatch.setattr(_lib, "_lib", fake)
    fake.fake_reset()
    made = []

    def make(n, **kw):
        case = harness.make_case("tiny", 16, seed=1)
        T = Tracker(case.specs, case.grids, case.params, numpar=n, **kw)
        made.append(T)
        for slot in (1, 2, 3):
            T.upload_frame(1, slot, case.frame(slot))
        z = np.zeros(n)
        T.set_particles(z, z, z, z, z, z, z + 1.0, np.ones(n, dtype=np.int32))
        fake.fake_reset()
        return T

    yield make
    fake.fake_reset()
    for T in made:
        T.close()


@pytest.mark.parametrize("k", range(5))
def test_resort_buffers_are_all_or_none(fake, tracker, k):
    T = tracker(64)
    held = fake.fake_bytes()
    fake.fake_fail_malloc(k, 0)
    with pytest.raises(Exception, match="NOMEM"):
        T.set_launch(12, 0)
    assert fake.fake_bytes() == held
    T.set_launch(2, 0)                                 # memory is there again
    for _ in range(3):
        T.step((0.0, 3600.0, 7200.0), (0.0, 300.0, 600.0), 2, 1, 2, 3)
    assert fake.fake_sorts() == 1 and fake.fake_null_bufs() == 0


def _adjoint(T, nsteps):
    from romspath_b200.adjoint import Adjoint, step_table
    case = harness.make_case("tiny", 16, seed=1)
    A = Adjoint(T)
    A.load_frames(3, lambda ng, k: case.frame(k, ng))
    return A, step_table(2.0, int(case.params["dt"]), int(case.params["idt"]))[0][:nsteps]


@pytest.mark.parametrize("where", ["first", "later", "second run"])
def test_failed_forward_leaves_no_record(fake, tracker, where):
    T = tracker(64)
    A, steps = _adjoint(T, 6)
    z = np.zeros(64)
    if where == "second run":
        A.forward(steps, checkpoint_every=3)
        A.backward(z, z, z)
    fake.fake_fail_adj(0 if where == "first" else 4)
    with pytest.raises(Exception, match="ERR_CUDA"):
        A.forward(steps, checkpoint_every=3)
    A.n = 64
    fake.fake_reset()
    for use in (lambda: A.backward(z, z, z), lambda: A.replay(kappa=1.0), lambda: A.tangent(1.0)):
        with pytest.raises(Exception, match="ERR_STATE.*call rp_forward first"):
            use()
    assert fake.fake_adj() == 0
    A.forward(steps, checkpoint_every=3)
    A.backward(z, z, z)


def test_refused_forward_keeps_the_record(fake, tracker):
    T = tracker(64)
    A, steps = _adjoint(T, 6)
    z = np.zeros(64)
    A.forward(steps, checkpoint_every=3)
    with pytest.raises(Exception, match="ERR_ARG"):
        A.forward(steps, checkpoint_every=0)
    A.backward(z, z, z)


# the order by cell is a speed-up: without the memory for it the particles are taken as they lie
@pytest.mark.parametrize("k", range(5))
def test_forward_goes_on_without_its_order(fake, tracker, k):
    n = 8192
    T = tracker(n)
    A, steps = _adjoint(T, 14)
    z = np.zeros(n)
    fake.fake_fail_malloc(10 + k, 1)                   # the run's ten buffers and k of the order's, then no more
    A.forward(steps, checkpoint_every=7)
    A.backward(z, z, z)
    A.replay()
    assert fake.fake_ordered() == 0 and fake.fake_sorts() == 0 and fake.fake_adj() == 14 + 12 + 14 + 14
    fake.fake_reset()
    A.forward(steps, checkpoint_every=7)               # memory is there again
    assert fake.fake_ordered() == 14 and fake.fake_null_bufs() == 0


# what a long run needed is not held through short ones: no more than twice what the run needs stays
@pytest.mark.parametrize("first,second", [((12, 12), (3, 3)), ((12, 1), (3, 1)), ((12, 12), (12, 1)), ((6, 3), (6, 3)),
                                          ((6, 3), (5, 3))])
def test_kept_adjoint_buffers_are_bounded(fake, tracker, first, second):
    n = 256
    T = tracker(n)
    A, steps = _adjoint(T, 12)
    z = np.zeros(n)
    empty = fake.fake_bytes()
    A.forward(steps[:second[0]], checkpoint_every=second[1])
    need = fake.fake_bytes() - empty
    A.forward(steps[:first[0]], checkpoint_every=first[1])
    A.forward(steps[:second[0]], checkpoint_every=second[1])
    A.backward(z, z, z)
    assert fake.fake_bytes() - empty <= 2 * need


def test_adjoint_launches_are_counted_as_told(fake, tracker):
    T = tracker(64)
    A, steps = _adjoint(T, 6)
    z = np.zeros(64)
    l0 = T.kernel_launches()
    A.forward(steps, checkpoint_every=3)               # each launcher call of the fake tells two kernels
    assert T.kernel_launches() - l0 == 2 * 6
    A.backward(z, z, z)
    assert T.kernel_launches() - l0 == 2 * (6 + 4 + 6)
    A.replay()
    A.tangent()
    assert T.kernel_launches() - l0 == 2 * (6 + 4 + 6 + 6 + 6) + 1    # the tangent's start is one more
