"""The reverse step's VTurb (differentiated by hand) where it can go wrong --
point counts around its row groups and workspace sizes, one, an odd number and
more sub-steps than it keeps, p = 1 and p = 0, no RK4 (so no clamp of z),
fixed depths, columns that reach the bottom and the surface, other Vtransforms
-- against the tangent-linear reference, which carries dual numbers through
the whole step.  Tolerance: two exact routes to one derivative, 1e-9 relative
(test_gpu_adjoint.py)."""
import numpy as np
import pytest

import harness
from test_gpu_adjoint import TARGET

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec,param", [
    ({}, {}), ({}, {"sub": 1.1}), ({}, {"sub": 1.2}), ({}, {"sub": 1.3}), ({}, {"sub": 1.5}), ({"N": 3}, {"sub": 1.1}),
    ({"N": 21}, {}), ({"N": 21}, {"sub": 4.05}), ({"N": 31}, {"sub": 4.04}), ({"N": 35}, {}),
    ({}, {"deltat": 300.0}), ({}, {"deltat": 100.0}), ({}, {"deltat": 4.0}), ({}, {"deltat": 3.0}),
    ({}, {"smth": 0.0}), ({}, {"smth": 1e9}), ({}, {"scheme": 0}), ({}, {"nsb": 1}), ({"vtransform": 1}, {}),
    ({"vtransform": 3}, {}), ({}, {"vturb_on": 0})])
def test_backward_matches_tangent_linear(spec, param):
    _check(spec, param, 129)


# enough particles for the kernels to take them by cell (the tangent-linear
# reference takes them as they lie), in segments of 4 and of 14 steps
@pytest.mark.parametrize("ckpt", [4, 14])
def test_ordered_by_cell(ckpt):
    _check({"land": "islands"}, {"hturb_on": 1, "constant_hturb": [1.0] * 5}, 8209, ckpt)


def _check(spec, param, n, ckpt=4):
    from romspath_b200 import Tracker, schedule
    from romspath_b200.adjoint import Adjoint, attribution_loss, step_table
    case = harness.make_case("tiny", n, seed=11, spec_over=spec, param_over=param, s_range=(-1.0, 0.0))
    T = Tracker(case.specs, case.grids, case.params, numpar=n, field_dtype="f64", seed=7)
    for (k, slot) in schedule.initial_loads():
        T.upload_frame(1, slot, case.frame(k))
    T.locate(case.release, t_b=1)
    steps = step_table(2.0, int(case.params["dt"]), int(case.params["idt"]))[0][:14]
    adj = Adjoint(T)
    adj.load_frames(max(max(s.frame_b, s.frame_c, s.frame_f) for s in steps), lambda ng, k: case.frame(k, ng))
    adj.forward(steps, kappa=1.25, checkpoint_every=ckpt)
    fin = T.get_particles()
    _, gx, gy = attribution_loss(fin["x"], fin["y"], TARGET)
    gz = np.linspace(-1.0, 1.0, n)
    got = adj.backward(gx, gy, gz)
    J = adj.tangent(kappa=1.25)
    T.close()
    want = np.einsum("ni,niq->nq", np.stack([gx, gy, gz], axis=1), J)
    for q in range(3):
        assert np.allclose(got[q], want[:, q], rtol=1e-9, atol=1e-12 * np.abs(want[:, q]).max()), q
    assert abs(got[3] - want[:, 3].sum()) <= 1e-9 * np.abs(want[:, 3]).sum()
