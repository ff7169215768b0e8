"""The exact form's VTurb kernel at the edges of its row groups (4, 8 and 16
rows), of its workspace sizes (88, 128, 144 points), of its division's range
and of its level search, and with the spline's u in shared and in local
memory, against the oracle: every particle column bit for bit, as everywhere
in the exact form."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


def _check(case, nsteps, **tracker):
    T = None
    if tracker:
        from romspath_b200 import Tracker
        T = Tracker(case.specs, case.grids, case.params, numpar=case.release.z.shape[0],
                    field_dtype=case.spec.field_dtype, stokes=case.spec.stokes, seed=7, **tracker)
    g, T = harness.run_gpu(case, nsteps, tracker=T)
    T.close()
    o, _ = harness.run_oracle(case, nsteps)
    bad = {k: v for k, v in harness.compare(g, o).items() if v}
    assert not bad, f"fields differing (particle counts): {bad}"


# int((N + 1) * sub) points: the smallest, the remainders of the row groups,
# both sides of each workspace size and the largest
@pytest.mark.parametrize("N,sub", [(3, 1.0), (4, 1.0), (3, 1.5), (6, 1.0), (8, 1.0), (9, 1.0), (10, 1.9), (6, 4.0),
                                   (21, 4.0), (21, 4.05), (31, 4.0), (31, 4.04), (35, 4.0)])
def test_point_counts(N, sub):
    _check(harness.make_case("tiny", 100, seed=5, spec_over={"N": N}, param_over={"sub": sub}), 3)


# diffusivity of 0 (a fit of zeros), subnormal (below the shared-reciprocal
# division's range: the IEEE pass), and scaled to its range's ends
@pytest.mark.parametrize("scale", [0.0, 1e-310, 1e-140, 1e-3, 1e140])
def test_diffusivity_range(scale):
    case = harness.make_case("tiny", 100, seed=6)
    plain = case.frame
    case.frame = lambda k, ng=1: dict(plain(k, ng), aks=np.asfortranarray(plain(k, ng)["aks"] * scale))
    _check(case, 3)


# levels whose depths do not ascend, equal levels, and the other Vtransforms
# (the linear walk)
@pytest.mark.parametrize("which", ["equal", "descend", "vt1", "vt3"])
def test_level_search(which):
    over = {"vt1": {"vtransform": 1}, "vt3": {"vtransform": 3}}.get(which)
    case = harness.make_case("tiny", 200, seed=8, spec_over=over, param_over={"vturb_on": int(which != "descend")})
    g = case.grids[0]
    if which == "equal":
        for k in ("s_rho", "cs_r", "s_w", "cs_w"):
            g[k] = g[k].copy()
            g[k][2] = g[k][3]
    if which == "descend":
        for k in ("s_rho", "cs_r"):
            g[k] = g[k].copy()
            g[k][[2, 3]] = g[k][[3, 2]]
    _check(case, 6)


# one block of four warps per SM: more particles than fit with u in shared
# memory, and as many as do
@pytest.mark.parametrize("n", [148 * 4 * 32, 148 * 4 * 32 + 1])
def test_shared_and_local_u(n):
    _check(harness.make_case("tiny", n, seed=9), 2, blocks_per_sm=1)
